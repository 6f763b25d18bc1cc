"""CPU tests of the single-launch and batched solvers' host rules and of what their kernels rely on."""

import os
import re

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
CSRC = os.path.join(ROOT, "jno_b200", "csrc")


def _code(name):
    """A source file without its comments."""
    src = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", src, flags=re.S))


def _body(code, head):
    """The braces' contents that follow the first match of `head`."""
    found = re.search(head, code)
    assert found, head
    at = code.index("{", found.end())
    depth, end = 0, at
    while True:
        depth += {"{": 1, "}": -1}.get(code[end], 0)
        end += 1
        if depth == 0:
            return code[at + 1:end - 1]


def test_a_cluster_has_started_before_any_block_stores_into_another():
    """A block of a cluster may touch another's shared memory only after a cluster-wide barrier has shown that all
    have started. The remote stores are BlockSum's, so the barrier belongs to what no kernel can leave out: its
    constructor, the only way to make one (a struct with a constructor takes no brace list of its fields)."""
    code = _code("femk_persist.cuh")
    struct = _body(code, r"struct BlockSum\b")
    made = _body(struct, r"BlockSum\([^)]*\)\s*:(?:\s*\w+\([^)]*\),?)*\s*(?=\{)")
    assert re.sub(r"\s+", " ", made).strip() == "if (SET == kOneCluster) cluster_sync();"
    assert "st_cluster(" in struct and "= default" not in struct
    for name in sorted(os.listdir(CSRC)):
        if name != "femk_persist.cuh":
            assert "st_cluster(" not in _code(name), name


def test_nothing_is_cleared_on_another_stream_than_the_call_s():
    """cudaMemset goes to the legacy default stream and does not wait: a solve on a non-blocking stream could run before
    the clearing of its counters, or beside it."""
    for name in sorted(os.listdir(CSRC)):
        assert not re.search(r"\bcudaMemset\s*\(", _code(name)), name
