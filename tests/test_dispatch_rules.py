"""Which engine a call runs on, asked without a GPU: the blocks carry addresses that nothing dereferences."""
import ctypes as C

import pytest

BASE = 0x7000_0000_0000


def _i8(lib, m, n, k, pose="nt", *, batch=1, offset=0):
    """A block of aligned operands in the given pose, rows padded to 16 bytes."""
    from nnops_b200 import capi
    up = lambda v: (v + 15) // 16 * 16 + offset
    a = capi.GemmI8Args(a=BASE, w=BASE + (1 << 32), out=BASE + (2 << 32), m=m, n=n, k=k, ldc=n, batch=batch,
                        scale_a_scalar=1.0, scale_w_scalar=1.0, out_scale=1.0)
    a.a_stride_m, a.a_stride_k = (1, up(m)) if pose[0] == "t" else (up(k), 1)
    a.w_stride_n, a.w_stride_k = (1, up(n)) if pose[1] == "n" else (up(k), 1)
    if batch > 1:
        a.a_batch_stride, a.w_batch_stride, a.out_batch_stride = m * up(k), n * up(k), m * n
    return a


@pytest.mark.parametrize("pose", ["nn", "tn", "tt"])
@pytest.mark.parametrize("shape", [(1, 512, 1024), (8, 4096, 4096), (16, 12800, 256), (24, 10000, 128), (64, 28672, 8192)])
def test_few_rows_engine_takes_k_contiguous_operands_only(nnb200_lib, shape, pose):
    """The few-row engine's tensor maps have one pose: the others belong to the square engine."""
    from nnops_b200 import capi
    a = _i8(nnb200_lib, *shape, pose)
    assert capi.ENGINE_NAMES[nnb200_lib.nnb200_gemm_i8_engine(C.byref(a))] == "umma"
