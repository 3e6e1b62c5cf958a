"""The regression graphs are kept by a key.  A kernel's buffer that is not in it
could move (its size grows with another call's sizes) and leave a graph that
still writes to memory given back to the device's pool.  Running that is not a
test, so the source is read: every buffer the captured launches name is in the
key of their graph."""
import os
import re

import ldsc_b200

ABI = os.path.join(os.path.dirname(ldsc_b200.__file__), "csrc", "abi.cpp")


def _balanced(text, start, open_, close):
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == open_) - (text[i] == close)
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError("unbalanced")


def test_every_captured_buffer_is_in_its_graphs_key():
    src = re.sub(r"//[^\n]*", "", open(ABI).read())
    keys = [m.start() for m in re.finditer(r"gkey\{", src)]
    assert len(keys) == 2   # h2 and rg
    for at in keys:
        key = _balanced(src, src.index("{", at), "{", "}")
        launch = _balanced(src, src.index("(", src.index("graph_launch(ctx, gkey", at)), "(", ")")
        used = set(re.findall(r"ctx->(\w+)\.as<", launch))
        assert used
        assert used <= set(re.findall(r"ctx->(\w+)\.p", key)), used - set(re.findall(r"ctx->(\w+)\.p", key))
