"""The context's host buffers against counting stand-ins of the runtime's calls: a
trim neither locks nor unlocks pages (that would stall the device's other
contexts), ordinary memory goes, and growth and release stay as they were."""
import os
import shutil
import subprocess

import pytest

from ldsc_b200 import build

SOURCE = r"""
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "hostbuf.h"

static int locked = 0, unlocked = 0;
static bool fail_lock = false;
extern "C" cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    if (fail_lock) return cudaErrorMemoryAllocation;
    locked++;
    *p = std::malloc(n);
    return cudaSuccess;
}
extern "C" cudaError_t cudaFreeHost(void* p) {
    unlocked++;
    std::free(p);
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }

int main() {
    using ldsc::HostBuf;
    HostBuf b;
    uint8_t* p = b.ensure(1000);
    assert(p && locked == 1 && b.ensure(10) == p && locked == 1);
    uint8_t* q = b.ensure(100000);
    assert(q != p && locked == 2 && b.cap >= 100000);
    std::memset(q, 1, 100000);
    b.trim();
    assert(locked == 2 && unlocked == 0 && b.ensure(100000) == q && locked == 2);   // nothing locked or unlocked
    uint8_t* big = b.ensure(HostBuf::PINNED_MAX + 1);   // ordinary memory
    assert(big && locked == 2 && b.cap > HostBuf::PINNED_MAX);
    std::memset(big, 1, HostBuf::PINNED_MAX + 1);
    b.trim();
    assert(unlocked == 0 && b.p == q && b.cap >= 100000 && b.cap < HostBuf::PINNED_MAX);
    assert(b.ensure(100000) == q);
    fail_lock = true;
    uint8_t* r = b.ensure(1 << 20);   // none can be locked
    assert(r && r != q && locked == 2);
    std::memset(r, 1, 1 << 20);
    fail_lock = false;
    b.release();
    assert(locked == unlocked && b.p == nullptr && b.cap == 0 && b.blocks.empty());
    b.trim();
    b.release();
    assert(unlocked == 2);
    // what growth leaves locked is bounded
    size_t total = 0;
    HostBuf g;
    for (size_t n = 1; n <= HostBuf::PINNED_MAX; n *= 2) g.ensure(n);
    for (const HostBuf::Block& x : g.blocks)
        if (x.pinned) total += x.cap;
    assert(total < 2 * HostBuf::PINNED_MAX);
    g.release();
    std::puts("ok");
}
"""


@pytest.mark.skipif(shutil.which(build.NVCC) is None, reason="needs the CUDA headers")
def test_trim_keeps_locked_pages(tmp_path):
    cuda = os.path.join(os.path.dirname(os.path.dirname(shutil.which(build.NVCC))), "include")
    src, exe = tmp_path / "hostbuf_test.cpp", tmp_path / "hostbuf_test"
    src.write_text(SOURCE)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I", cuda, "-I", build.CSRC, str(src), "-o", str(exe)])
    assert subprocess.check_output([str(exe)], text=True).strip() == "ok"
