"""A batch of products in one launch, and operands off the 16-byte rule: byte for byte against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from nnops_b200 import capi, ops

pytestmark = pytest.mark.gpu


def _store(x: np.ndarray, transposed: bool, device, offset: int = 0):
    """x [..., R, C] on the device, stored [..., C, R] when ``transposed``, ``offset`` bytes into its allocation."""
    y = np.ascontiguousarray(np.swapaxes(x, -1, -2)) if transposed else x
    flat = torch.empty(y.size + offset, dtype=torch.from_numpy(y).dtype, device=device)
    t = flat[offset:].view(y.shape)
    t.copy_(torch.from_numpy(y))
    return t.transpose(-1, -2) if transposed else t


def _check(device, batch, m, n, k, *, pose="nt", out_kind="s8", shared_a=False, shared_w=False, unsigned=False, zero_points=False,
           offset=0, launches=None, seed=0, min_workspace=False):
    rng = np.random.default_rng(seed)
    a = rng.integers(0, 256, ((1 if shared_a else batch), m, k)).astype(np.uint8) if unsigned else \
        rng.integers(-127, 128, ((1 if shared_a else batch), m, k), dtype=np.int8)
    w = rng.integers(-127, 128, ((1 if shared_w else batch), n, k), dtype=np.int8)
    kw = {"scale_a": rng.uniform(0.001, 0.02, m).astype(np.float32), "scale_w": rng.uniform(0.001, 0.02, n).astype(np.float32)}
    if out_kind in ("s8", "u8"):
        kw.update(out_scale=1.7, out_zp=3)
    if zero_points:
        kw.update(zp_a=rng.integers(-9, 10, m).astype(np.int32), zp_w=rng.integers(-3, 4, n).astype(np.int32))
    if batch == 1:
        a, w = a[0], w[0]
    ta = _store(a, pose[0] == "t", device, offset)
    tw = _store(w, pose[1] == "n", device, offset)
    if batch > 1:
        ta, tw = (ta[0] if shared_a else ta), (tw[0] if shared_w else tw)
    before = capi.lib().nnb200_launch_count()
    got = ops.gemm_i8(ta, tw, out_kind=out_kind, min_workspace=min_workspace, **kw).cpu().numpy()
    if launches is not None:
        assert capi.lib().nnb200_launch_count() - before == launches
    if batch == 1:
        want = oracle.gemm_i8(a, w, out_kind=out_kind, **kw)
        assert np.array_equal(got, want)
        return
    for b in range(batch):
        want = oracle.gemm_i8(a[0 if shared_a else b], w[0 if shared_w else b], out_kind=out_kind, **kw)
        assert np.array_equal(got[b], want), b


@pytest.mark.parametrize("shape", [(2, 16, 16, 16), (5, 128, 128, 128), (3, 144, 272, 208), (40, 129, 65, 144), (9, 300, 528, 1024)])
@pytest.mark.parametrize("pose", ["nt", "nn", "tn", "tt"])
def test_batch_is_one_launch(cuda_device, nnb200_lib, shape, pose):
    """Every tile width, ragged last tiles, all poses whose pitches TMA can address."""
    batch, m, n, k = shape
    if (pose[0] == "t" and m % 16) or (pose[1] == "n" and n % 16):
        m, n = (m + 15) // 16 * 16, (n + 15) // 16 * 16
    _check(cuda_device, batch, m, n, k, pose=pose, launches=1, seed=batch + m)


@pytest.mark.parametrize("out_kind", ["s32", "s8", "u8", "f32", "f16"])
@pytest.mark.parametrize("shared", ["", "a", "w"])
@pytest.mark.parametrize("zero_points", [False, True])
def test_batch_destinations_and_shared_operands(cuda_device, nnb200_lib, out_kind, shared, zero_points):
    _check(cuda_device, 4, 96, 200, 272, out_kind=out_kind, shared_a=shared == "a", shared_w=shared == "w", zero_points=zero_points,
           unsigned=out_kind == "u8", seed=7)


def test_batch_writes_interleaved_outputs(cuda_device, nnb200_lib):
    """Heads side by side in one row ([M, heads, N] storage): the batch step is smaller than a product."""
    rng = np.random.default_rng(3)
    a, w = (rng.integers(-127, 128, (6, 80, 160), dtype=np.int8) for _ in range(2))
    out = torch.full((80, 6, 80), -1, dtype=torch.int32, device=cuda_device)
    ops.gemm_i8(torch.from_numpy(a).to(cuda_device), torch.from_numpy(w).to(cuda_device), out=out.permute(1, 0, 2))
    got = out.cpu().numpy()
    for b in range(6):
        assert np.array_equal(got[:, b], oracle.gemm_i8(a[b], w[b])), b


@pytest.mark.parametrize("case", [
    # k, offset, pose, batch
    (2049, 0, "nt", 1), (2050, 1, "nt", 1), (2047, 3, "nt", 1), (2052, 13, "nt", 1), (2048, 5, "nt", 1),
    (2049, 0, "nn", 1), (2053, 0, "tt", 1), (2048, 7, "tn", 1), (700, 0, "nt", 3), (701, 2, "nn", 3)])
@pytest.mark.parametrize("zero_points", [False, True])
def test_operands_off_the_tma_rule(cuda_device, nnb200_lib, case, zero_points):
    """Sizes from which the operands are copied into aligned rows: odd K, odd bases, each pose, batches."""
    k, offset, pose, batch = case
    _check(cuda_device, batch, 257, 301, k, pose=pose, offset=offset, zero_points=zero_points, unsigned=k % 2 == 0, seed=k)


@pytest.mark.parametrize("m", [1, 7, 17])
def test_few_rows_off_the_tma_rule(cuda_device, nnb200_lib, m):
    _check(cuda_device, 1, m, 9001, 1500 if m > 7 else 15001, zero_points=True, seed=m)


@pytest.mark.parametrize("shape", [(1, 512, 1024), (16, 12800, 256), (24, 10000, 128), (8, 513, 1024), (5, 1001, 1000), (24, 10001, 200)])
@pytest.mark.parametrize("pose", ["nn", "tn"])
def test_few_rows_with_k_by_n_weights(cuda_device, nnb200_lib, shape, pose):
    """Few rows whose operands are not k-contiguous, as they lie and through aligned copies."""
    m, n, k = shape
    if pose[0] == "t" and n % 16 == 0:
        m = (m + 15) // 16 * 16
    _check(cuda_device, 1, m, n, k, pose=pose, zero_points=True, seed=n)


@pytest.mark.parametrize("case", [
    # m, n, k, pose: rows of one turn and more a warp, few long rows a block each, both with and without sums
    (300, 300, 2100, "nt"), (300, 300, 9001, "nt"), (2, 1100, 2049, "nt"), (33, 5001, 260, "nn"), (40, 9999, 300, "tn"),
    # K too short for the copies to pay: the generic engine
    (2, 9000, 33, "nt"), (64, 1001, 64, "nn"), (16, 1000, 129, "nt")])
@pytest.mark.parametrize("zero_points", [False, True])
def test_copies_of_few_long_rows_and_short_k(cuda_device, nnb200_lib, case, zero_points):
    m, n, k, pose = case
    copied = k > 160
    _check(cuda_device, 1, m, n, k, pose=pose, zero_points=zero_points, seed=m + k, out_kind="s32",
           launches=None if zero_points else (2 if copied else 1))


@pytest.mark.parametrize("batch,m,n,k,launches", [(2, 1, 512, 4096, 2), (3, 8, 256, 4096, 3), (2, 16, 1024, 1024, 2), (6, 4, 64, 16384, 6),
                                                  (8, 8, 512, 1024, 1), (2, 17, 512, 4096, 1), (16, 1, 64, 16384, 1)])
def test_few_rows_in_a_small_batch(cuda_device, nnb200_lib, batch, m, n, k, launches):
    """A launch of the streaming engine each until one launch of the tile kernel is shorter."""
    _check(cuda_device, batch, m, n, k, launches=launches, seed=k)


@pytest.mark.parametrize("case", [(2049, 0, "nt", 1), (2050, 1, "nn", 1), (700, 0, "nt", 3)])
@pytest.mark.parametrize("zero_points", [False, True])
def test_operands_off_the_tma_rule_with_the_least_scratch(cuda_device, nnb200_lib, case, zero_points):
    """No room for copies: the generic engine, a launch a product."""
    k, offset, pose, batch = case
    _check(cuda_device, batch, 65, 301, k, pose=pose, offset=offset, zero_points=zero_points, min_workspace=True, seed=k,
           launches=None if zero_points else batch)
