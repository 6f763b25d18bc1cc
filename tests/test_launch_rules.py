"""CPU tests of the single-launch and batched solvers' host rules and of what their kernels rely on.

``launch_harness.cu`` runs the solvers' host code against a made-up CUDA runtime, which logs what is launched where and
fails the call it is told to."""

import os
import re
import subprocess

import pytest

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


def test_matrix_free_shares_lie_inside_the_partials_on_any_number_of_sms():
    """Where the product's block shares start and how many there are, against the buffer's length, from one SM (a
    partition of a GPU) to more than the whole one has."""
    internal, cg = _code("femk_internal.cuh"), _code("femk_cg.cu")
    values = dict(re.findall(r"\b(k\w+) = (\d+)[,;]", internal))
    length = re.search(r"cudaMalloc\(&p->partials, sizeof\(double\) \* ([^)]*\)?[^)]*)\)", cg).group(1)
    start = re.search(r"p->partials \+ ((?:\(int64_t\))?k\w+(?: \* p->n_sm)?)", cg)
    assert start, "no start of the shares"
    blocks = re.search(r"blocks_for\(std::max\(a\.count, a\.ndir\), 128, (.*?)\);", cg).group(1)

    def at(expr, n_sm):
        expr = expr.replace("(int64_t)", "").replace("p->n_sm", str(n_sm))
        for table in (values, dict(re.findall(r"\b(k\w+) = (\d+)[,;]", cg))):
            expr = re.sub(r"\bk\w+", lambda m: table.get(m.group(0), m.group(0)), expr)
        return eval(expr, {}, {})

    for n_sm in (1, 8, 16, 34, 60, 68, 69, 148, 160):
        # the reductions before the shares: three values of at most 16 blocks an SM
        assert 3 * 16 * n_sm <= at(start.group(1), n_sm), n_sm
        assert at(start.group(1), n_sm) + at(blocks, n_sm) <= at(length, n_sm), n_sm


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    from jno_b200 import _build

    _build.build()
    out = str(tmp_path_factory.mktemp("harness") / "harness")
    objs = [os.path.join(ROOT, "_build", o) for o in ("femk_batch_sets.o", "femk_persist.o")]
    subprocess.run([_build._nvcc(), *_build.ARCH, "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-diag-suppress",
                    "177,550", "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-o", out,
                    os.path.join(ROOT, "tests", "launch_harness.cu"), *objs, "-cudart", "none"], check=True)

    def run(*args):
        return subprocess.run([out, *map(str, args)], check=True, capture_output=True, text=True).stdout.splitlines()

    return run


@pytest.mark.parametrize("largest", [16, 8, 4, 2, 1])
def test_devices_without_large_clusters_get_another_form(harness, largest):
    """A part of a GPU may hold no cluster of 16 blocks, or none at all: the solvers ask and use the grid."""
    for rows in (300, 1000, 1500, 4000, 16000, 17000):
        log = harness(largest, 0, "-", "solve", rows, 15)
        launches = [line for line in log if line.startswith("launch")]
        assert len(launches) == 2 and not any(line.startswith("refused") for line in log), log
        for line in launches:
            _, _, _, blocks, _, cluster, _, cooperative = line.split()
            assert int(cluster) <= largest and (int(blocks) == 1 or int(cluster) or cooperative == "1")
    log = harness(largest, 0, "-", "batch", 100, 1000, 1500, 5000, 9000, 16000, 30000, 120000)
    assert not any(line.startswith("refused") for line in log), log


@pytest.mark.parametrize("name", ["cudaLaunchKernelExC", "cudaStreamWaitEvent", "cudaEventRecord", "cudaMemsetAsync"])
def test_a_batch_that_fails_half_way_waits_for_what_it_launched(harness, name):
    """Classes of problems run on streams of their own beside the caller's. Whichever call fails, each of these streams
    is joined into the caller's (or waited for) after its last launch, before the call returns."""
    batch = ("batch", 100, 1000, 1500, 5000, 9000, 30000, 120000)
    assert sum(line.startswith("launch") for line in harness(16, 0, "-", *batch)) == 4
    for at in range(1, 10):
        log = harness(16, at, name, *batch)
        busy, marks = set(), {}
        for line in log:
            word = line.split()
            if word[0] == "launch" and word[1] != "1":
                busy.add(word[1])
            elif word[0] == "record":
                marks[word[1]] = word[2]  # the event now stands for this stream
            elif word[0] == "wait" and word[1] == "1":
                busy.discard(marks[word[2]])
            elif word[0] == "synchronize":
                busy.discard(word[1])
        assert not busy, (at, log)
        if any(line.startswith("failed") for line in log):
            assert "status 2" in log, (at, log)


def test_the_single_launch_bicgstab_looks_at_its_index_checks(harness):
    """The bounds-checked build's kernels record a bad index and skip the access; the call has to report it."""
    for rows in (300, 4000, 17000):
        log = harness(16, 0, "-", "solve", rows, 15)
        second = [i for i, line in enumerate(log) if line.startswith("launch")][1]
        assert "checked" in log[second:], log
