"""Registers that the overlap of decode and Gram counts on, as the compiler
reports them: beside a Gram CTA (one per SM) the register file holds three
decode blocks, or one where the Gram runs 16 epilogue warps."""
import os
import re
import shutil
import subprocess
from concurrent.futures import ThreadPoolExecutor

import pytest

from ldsc_b200 import build

REGISTERS = 65536


def _registers(source):
    """{kernel (mangled name): registers a thread, as allocated (in eights)}"""
    r = subprocess.run([build.NVCC, "-c", os.path.join(build.CSRC, source), "-o", os.devnull, "-Xptxas", "-v"]
                       + build.CUFLAGS, capture_output=True, text=True, check=True)
    out, name = {}, None
    for line in r.stderr.splitlines():
        m = re.search(r"Compiling entry function '(\w+)'", line)
        name = m.group(1) if m else name
        m = re.search(r"Used (\d+) registers", line)
        if m and name:
            out[name] = (int(m.group(1)) + 7) // 8 * 8
            name = None
    return out


@pytest.mark.skipif(shutil.which(build.NVCC) is None, reason="needs nvcc")
def test_decode_blocks_fit_beside_a_gram_cta():
    with ThreadPoolExecutor(2) as ex:
        decode, gram = ex.map(_registers, ["decode.cu", "gram_tc.cu"])
    (decode,) = [v for k, v in decode.items() if "k_decode_i8" in k]
    tc = {k: v for k, v in gram.items() if "k_gram_tc" in k}
    (long_rows,) = [v for k, v in tc.items() if "ILi3ELi0ELi8ELi0E" in k]      # 8 epilogue warps: 320 threads
    (short_rows,) = [v for k, v in tc.items() if "ILi3ELi0ELi16ELi0E" in k]    # 16: 576 threads
    assert (REGISTERS - 320 * long_rows) // (256 * decode) >= 3
    assert (REGISTERS - 576 * short_rows) // (256 * decode) >= 1
