"""What every kernel that overlaps its neighbours in the stream keeps to, read from the sources: such a mistake is a
hang or a stale read on the GPU now and then, which no run on one can be trusted to show."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "nnops_b200" / "csrc"


def _code(path):
    """The file without its comments."""
    return re.sub(r"/\*.*?\*/", "", re.sub(r"//[^\n]*", "", path.read_text()), flags=re.S)


def _sources():
    return {p.name: _code(p) for p in sorted(CSRC.glob("*.cu*"))}


def _body(text, at):
    """The braced block that opens at or after ``at``."""
    start = at = text.index("{", at)
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(text[at], 0)
        at += 1
        if depth == 0:
            return text[start:at]


def test_no_kernel_lets_its_successor_start_before_its_own_wait():
    """Or three kernels are in flight, two of them holding what they have while they wait."""
    for name, text in _sources().items():
        assert ("griddepcontrol" in text) == (name == "ptx.cuh"), name
    ptx = _sources()["ptx.cuh"]
    assert ptx.count("griddepcontrol.launch_dependents") == 1
    body = _body(ptx, ptx.index("void let_next_kernel_start("))
    assert body.index("griddepcontrol.wait;") < body.index("griddepcontrol.launch_dependents;")


def test_tensor_memory_is_allocated_before_the_successor_may_start():
    """A producer warp that has not met the allocating warp does so first."""
    for name, text in _sources().items():
        for at in (m.start() for m in re.finditer(r"named_barrier_arrive\(1, ", text)):
            kernel_end = text.find("__global__", at)
            kernel = text[at:kernel_end if kernel_end > 0 else len(text)]
            assert kernel.index("tmem_alloc(") < kernel.index("named_barrier_arrive(2, 64)"), name
            assert kernel.index("named_barrier_sync(2, 64)") < kernel.index("let_next_kernel_start()"), name


def test_what_the_previous_kernel_may_still_write_is_read_coherently():
    """A kernel that is resident before the previous one has completed must not read through the non-coherent path, nor
    leave the compiler free to: a const __restrict__ pointer, an intrinsic that may move ahead of the wait."""
    overlapped = 0
    for name, text in _sources().items():
        if name in ("ptx.cuh", "ptx_pair.cuh", "internal.cuh") or "previous_kernel_done()" not in text:
            continue
        assert "__ldg(" not in text and "global.nc" not in text, name
        for at in (m.end() for m in re.finditer(r"__global__", text)):
            signature = text[at:text.index("{", at)]
            if "previous_kernel_done()" in _body(text, at):
                overlapped += 1
                assert not re.search(r"const [\w:]+\* __restrict__", signature), (name, signature)
    assert overlapped >= 18


def test_what_is_read_from_another_cta_has_come_before_it_may_leave():
    """In the few-row engine's exchange the CTAs part at a barrier that orders no memory, so every load has to be waited
    for: those of rows and channels that are not stored by a vote on their values."""
    kernel = _sources()["gemm_i8_skinny.cu"]
    kernel = kernel[kernel.index("gemm_i8_skinny_kernel(const"):]
    loads, stores = kernel.index("theirs[p][j] = ld_shared_cluster_u32("), kernel.index("finish_rows<KIND, 4>(")
    parting = kernel.index("cluster_sync_all_relaxed()", stores)
    assert kernel.count("ld_shared_cluster_u32(") == 1 and loads < stores < parting
    after = kernel[stores:parting]
    vote = _body(after, after.index("if (r + 4 > row_end || !all_ok)"))
    assert "v[0] | v[1] | v[2] | v[3]" in vote and re.search(r"row_end = __any_sync\(0xFFFFFFFFu, \(seen & never\) != 0\)", vote)
    assert "all_ok = __all_sync(0xFFFFFFFFu, n_ok)" in kernel[:loads]
