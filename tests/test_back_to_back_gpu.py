"""Streams of calls with nothing between them: kernels overlap the end of the one before, so each must find what that one
wrote, and must not write what it still reads.  The same calls with a synchronisation after each give the same bytes."""
import numpy as np
import pytest
import torch

from nnops_b200 import ops, synth

pytestmark = pytest.mark.gpu


def _same_with_and_without_waiting(chain, times=4):
    """``chain(after)`` runs its calls, ``after()`` behind each, and returns tensors."""
    want = [t.clone() for t in chain(torch.cuda.synchronize)]
    torch.cuda.synchronize()
    for _ in range(times):
        got = chain(lambda: None)
        assert all(torch.equal(g.view(torch.uint8), w.view(torch.uint8)) for g, w in zip(got, want, strict=True))
    return want


@pytest.mark.parametrize("m,engines", [(1, ("gemv_dsq", "gemv_mma", "gemv_dsq")), (4, ("gemv_mma", "rows", "gemv_dsq")),
                                       (16, ("rows", "rows", "rows"))])
@pytest.mark.parametrize("n", [1024, 9600])
def test_flagged_q4_1_calls_among_others(cuda_device, nnb200_lib, m, engines, n):
    """Calls that fetch their weights ahead of the kernel before them, in a row and between kernels that do not."""
    rng = np.random.default_rng(m + n)
    k = 1024
    wide = torch.from_numpy(synth.q4_1_weights(rng, n, k)).to(cuda_device)
    back = torch.from_numpy(synth.q4_1_weights(rng, k, (n + 127) // 128 * 128)).to(cuda_device)
    w8 = torch.from_numpy(rng.integers(-127, 128, (k, k), dtype=np.int8)).to(cuda_device)
    x0 = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float16)).to(cuda_device)
    scale, zp = torch.full((m,), 0.05, device=cuda_device), torch.zeros(m, dtype=torch.int8, device=cuda_device)
    flagged = dict(overlap_previous=True, min_clip=-4.0, max_clip=4.0)

    def chain(after):
        x, seen = x0, []
        for e in engines:
            up = ops.linear_q4_1(x, wide, k, engine=e, alpha=0.3, **flagged)
            after()
            down = ops.linear_q4_1(up, back, n, engine=e, alpha=0.3, **flagged)
            after()
            ops.linear_q4_1(x, wide, k, engine=e, alpha=0.6, out=up, **flagged)   # over what `down` is made from
            after()
            q = ops.quantize_linear(down, scale, zp)
            after()
            x = ops.gemm_i8(q, w8, out_kind="f16", scale_w=2e-4)
            after()
            seen += [up, down, q, x]
        return seen

    want = _same_with_and_without_waiting(chain)
    assert all(torch.isfinite(t.float()).all() and t.float().abs().max() > 0 for t in want)
