"""The few-row engine on layers with few channels: clusters of CTAs share a tile's K and add up their sums through
distributed shared memory.  Byte for byte against the oracle at the edges of rows, channels, K shares and cluster sizes."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from nnops_b200 import capi, ops

pytestmark = pytest.mark.gpu

KINDS = ("s32", "s8", "u8", "f32", "f16")


def _case(device, m, n, k, kind, *, engine, seed, zero_points=False, a_unsigned=False, pad=0):
    rng = np.random.default_rng(seed)
    a = rng.integers(0, 256, (m, k), dtype=np.uint8) if a_unsigned else rng.integers(-127, 128, (m, k), dtype=np.int8)
    w = rng.integers(-127, 128, (n, k), dtype=np.int8)
    kw = dict(out_kind=kind, scale_a=rng.uniform(0.01, 0.03, m).astype(np.float32),
              scale_w=rng.uniform(0.001, 0.02, n).astype(np.float32))
    if kind in ("s8", "u8"):
        kw.update(out_scale=0.6 * k ** 0.5, out_zp=3)
    if kind in ("s32", "s8", "u8"):
        kw.update(relu=True, bias=rng.integers(-1000, 1001, n).astype(np.int32))
    else:
        kw["bias"] = rng.normal(size=n).astype(np.float32 if kind == "f32" else np.float16)
    if zero_points:
        kw.update(zp_a=rng.integers(-9, 10, m).astype(np.int32), zp_w=rng.integers(-9, 10, n).astype(np.int32))
    held = torch.full((m + 2, n + pad), 77, dtype=ops._OUT_TORCH[kind], device=device)
    out = held[1:m + 1, :n]
    ops.gemm_i8(torch.from_numpy(a).to(device), torch.from_numpy(w).to(device), out=out, engine=engine, **kw)
    want = oracle.gemm_i8(a, w, **kw)
    assert np.array_equal(out.cpu().numpy().view(np.uint8), want.view(np.uint8))
    # Nothing around the window was touched.
    assert bool((held[0] == 77).all()) and bool((held[m + 1] == 77).all()) and bool((held[:, n:] == 77).all())
    assert capi.take_device_error() == 0


@pytest.mark.parametrize("m", [1, 8, 9, 31, 32, 33, 64, 65, 127, 128])
@pytest.mark.parametrize("shape", [(64, 1024), (130, 4096), (2500, 528), (4096, 2064), (9300, 1040)])
def test_clusters_share_k(cuda_device, nnb200_lib, m, shape):
    """One to 73 tiles: clusters of eight down to two, K blocks that do not divide by them, a ragged last block."""
    n, k = shape
    i = m + n
    _case(cuda_device, m, n, k, KINDS[i % 5], engine="skinny", seed=i, zero_points=i % 2 == 0, a_unsigned=i % 3 == 0, pad=i % 4)


@pytest.mark.parametrize("shape", [(9, 8192, 512), (16, 1024, 4096), (16, 96, 8192), (24, 4096, 1024), (32, 64, 512), (64, 4096, 2048),
                                   (64, 9472, 8192), (128, 2048, 4096), (128, 4736, 4096),
                                   (1, 6400, 512), (1, 64, 8192), (1, 11008, 2048), (4, 11008, 2112), (8, 19000, 512)])
def test_calls_routed_to_clusters(cuda_device, nnb200_lib, shape):
    """The smallest K of each row of the rule, one row to a handful, and a call with only the minimum workspace."""
    m, n, k = shape
    args = capi.GemmI8Args(a=4096, w=4096, out=4096, m=m, n=n, k=k, a_stride_m=k, a_stride_k=1, w_stride_n=k, w_stride_k=1, ldc=n, batch=1,
                           scale_a_scalar=1.0, scale_w_scalar=1.0, out_scale=1.0)
    assert capi.ENGINE_NAMES[nnb200_lib.nnb200_gemm_i8_engine(ctypes.byref(args))] == "skinny"
    _case(cuda_device, m, n, k, "f16", engine="auto", seed=m + k)
    a = torch.randint(-127, 128, (m, k), dtype=torch.int8, device=cuda_device)
    w = torch.randint(-127, 128, (n, k), dtype=torch.int8, device=cuda_device)
    got = ops.gemm_i8(a, w, zp_a=3, min_workspace=True)
    assert torch.equal(got, ops.gemm_i8(a, w, zp_a=3, engine="generic"))
