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


def _q4(m, n, k, f16, *, ldw=None, force=0, workspace=None):
    from nnops_b200 import capi
    blocks = (k + 31) // 32
    return capi.Q41Args(a=BASE, w_blocks=BASE + (1 << 32), out=BASE + (2 << 32), m=m, n=n, k=k, lda=(k + 7) // 8 * 8,
                        ldw_blocks=ldw or blocks, ldc=n, a_f16=int(f16), out_f16=0, alpha=1.0, force_engine=force,
                        workspace=BASE + (3 << 32) if workspace else None, workspace_bytes=workspace or 0)


@pytest.mark.parametrize("k,ldw", [(1000, None), (352, None), (4128, None), (8992, None), (1024, 33)])
def test_q4_1_calls_held_in_f32_stay_on_the_engine_that_does(nnb200_lib, k, ldw):
    """K off the 128 rule, or rows off the 16-byte rule: few rows run on the CUDA-core GEMV, whose weights and
    activations are f32, whatever scratch there is."""
    engine = lambda q: nnb200_lib.nnb200_q4_1_engine(C.byref(q))
    for n in (64, 11008, 40000):
        for m, f16 in [(2, True), (8, True), (2, False), (16, False)]:
            assert nnb200_lib.nnb200_q4_1_workspace_bytes(C.byref(_q4(m, n, k, f16, ldw=ldw))) == 0
            assert engine(_q4(m, n, k, f16, ldw=ldw, workspace=1 << 33)) == 3, (m, n, f16)
        # Where the other engine rounds the weights to f16 too, the weights go to tensor memory ...
        assert engine(_q4(9, n, k, True, ldw=ldw)) == 7
        need = nnb200_lib.nnb200_q4_1_workspace_bytes(C.byref(_q4(17, n, k, False, ldw=ldw)))
        assert engine(_q4(17, n, k, False, ldw=ldw, workspace=need)) == 7
        # ... for 17 and more f32 rows only with the scratch that brings them off the CUDA cores.
        assert engine(_q4(17, n, k, False, ldw=ldw, workspace=need - 1)) == 3
    for m, f16 in [(16, True), (128, True), (5, False), (64, False)]:
        q = _q4(m, 4096, 4096, f16)
        assert engine(_q4(m, 4096, 4096, f16, workspace=nnb200_lib.nnb200_q4_1_workspace_bytes(C.byref(q)))) == 7


@pytest.mark.parametrize("call,pays", [
    # Time falls from six generic steps of K up, from four with more than 16 rows, and with outputs enough.
    ((1, 28672, 8191), True), ((16, 1000, 257), True), ((16, 1000, 129), False), ((33, 1000, 129), True), ((64, 10001, 129), False),
    ((1, 100000, 33), False), ((2, 100000, 17), False), ((64, 100000, 65), True), ((1024, 1000, 17), True), ((64, 1000, 65), False),
    ((3, 100, 300), False)])
def test_copies_into_aligned_rows_only_where_they_pay(nnb200_lib, call, pays):
    """The scratch asked for beyond the least is the copies' (K is off the 16-byte rule in every case)."""
    m, n, k = call
    a = _i8(nnb200_lib, m, n, k)
    a.a_stride_m = a.w_stride_n = k
    copies = nnb200_lib.nnb200_gemm_i8_workspace_bytes(C.byref(a)) - nnb200_lib.nnb200_gemm_i8_min_workspace_bytes(C.byref(a))
    up = lambda v, to: -(-v // to) * to
    want = sum(up(rows * up(k, 16), 256) for rows in (m, n)) if pays else 0
    assert copies >= want and (copies == 0) == (want == 0)


@pytest.mark.parametrize("m,n,k,f16,engine", [
    # parts of a cluster to add up: K beyond one unit has to pay for it
    (33, 4096, 384, True, 7), (64, 4096, 256, True, 7), (64, 4096, 384, True, 1), (64, 4096, 512, True, 7), (65, 4096, 256, True, 1),
    (128, 4096, 384, True, 1), (128, 4096, 512, True, 7), (128, 9472, 640, True, 1), (128, 9472, 768, True, 7),
    (33, 4096, 288, True, 1), (64, 4096, 672, True, 7), (9, 4096, 128, True, 7),
    # a tile a CTA
    (128, 14336, 256, True, 7), (64, 14336, 288, True, 1), (64, 28672, 416, True, 7),
    (3, 1024, 1024, False, 4), (4, 4096, 1024, False, 4), (5, 1024, 1024, False, 7), (3, 4096, 4096, False, 7), (3, 14336, 256, False, 7),
    (64, 2048, 256, False, 5), (64, 2048, 384, False, 7), (64, 14336, 256, False, 7)])
def test_q4_1_weights_in_tensor_memory_where_k_is_long_enough(nnb200_lib, m, n, k, f16, engine):
    need = nnb200_lib.nnb200_q4_1_workspace_bytes(C.byref(_q4(m, n, k, f16)))
    q = _q4(m, n, k, f16, workspace=need or 1 << 33)
    assert nnb200_lib.nnb200_q4_1_engine(C.byref(q)) == engine
    q.activation = 3   # the other GEMMs' epilogues fetch it cold
    assert nnb200_lib.nnb200_q4_1_engine(C.byref(q)) == (7 if engine in (1, 5) else engine)


def test_q4_gemv_knob_comes_before_the_weights_in_tensor_memory(nnb200_lib, knobs):
    engine = lambda m, f16: nnb200_lib.nnb200_q4_1_engine(C.byref(_q4(m, 28672, 4096, f16, workspace=1 << 33)))
    assert (engine(4, True), engine(4, False), engine(1, True)) == (7, 7, 6)
    knobs("q4_gemv", 2)
    assert (engine(4, True), engine(4, False), engine(1, True)) == (6, 6, 6)
    knobs("q4_gemv", 1)
    assert (engine(4, True), engine(4, False), engine(1, True)) == (7, 7, 4)


@pytest.mark.parametrize("m,n,k,engine", [
    # from the streaming engine (up to 16 rows): by tiles per SM, by K, from 9 rows by both
    (1, 6272, 512, "decode"), (1, 6273, 512, "skinny"), (8, 6272, 4096, "decode"), (8, 6273, 4096, "skinny"),
    (1, 64, 8128, "decode"), (1, 64, 8192, "skinny"), (8, 1024, 4096, "decode"), (9, 1024, 4096, "skinny"), (9, 1023, 4096, "decode"),
    (9, 1024, 4032, "decode"), (16, 6272, 512, "decode"), (16, 6273, 512, "skinny"),
    # one row of a long K where tiles are too many for clusters and too few for the SMs stays there
    (1, 9472, 4096, "skinny"), (1, 9473, 4096, "decode"), (1, 9473, 2048, "skinny"), (2, 9473, 4096, "skinny"),
    (1, 14208, 4096, "decode"), (1, 14209, 4096, "skinny"),
    # from the square engine: up to 32 rows, up to 64 with a long K, beyond with few channels too
    (17, 64, 64, "skinny"), (32, 9472, 512, "skinny"), (33, 4096, 2032, "umma"), (33, 6272, 2048, "skinny"), (33, 6273, 2048, "umma"),
    (64, 6273, 8176, "umma"), (64, 9472, 8192, "skinny"), (64, 9473, 512, "skinny"),
    (65, 4736, 4080, "umma"), (65, 4736, 4096, "skinny"), (65, 4737, 4096, "umma"), (128, 4736, 4096, "skinny"), (129, 4096, 8192, "umma"),
    (89, 6400, 16384, "skinny"), (90, 6400, 16384, "umma"), (72, 9472, 16384, "umma"), (72, 9472, 32768, "skinny")])
def test_few_rows_engine_by_tiles_and_k(nnb200_lib, m, n, k, engine):
    """Both sides of each line of the rule, for 148 SMs; the query answers what the call runs on."""
    from nnops_b200 import capi
    a = _i8(nnb200_lib, m, n, k)
    assert capi.ENGINE_NAMES[nnb200_lib.nnb200_gemm_i8_engine(C.byref(a))] == engine
    a.force_engine = capi.ENGINES["umma"]
    assert capi.ENGINE_NAMES[nnb200_lib.nnb200_gemm_i8_engine(C.byref(a))] == "umma"
