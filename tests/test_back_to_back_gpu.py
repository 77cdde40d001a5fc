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


def _s8(rng, device, *shape):
    return torch.from_numpy(rng.integers(-127, 128, shape, dtype=np.int8)).to(device)


def _producers(rng, device):
    """Every kernel that lets its successor start before its epilogue: three inputs each, and a call into ``out``."""
    def i8(m, n, k, engine):
        w, sw = _s8(rng, device, n, k), torch.rand(n, device=device) * 0.02 + 0.001
        xs = [_s8(rng, device, m, k) for _ in range(3)]
        out = torch.empty((m, n), dtype=torch.int8, device=device)
        return xs, lambda x: ops.gemm_i8(x, w, out_kind="s8", out=out, out_scale=0.6 * k ** 0.5, scale_w=sw, engine=engine)

    def q4(m, n, k, engine, dtype=torch.float16, **kw):
        w = torch.from_numpy(synth.q4_1_weights(rng, n, k)).to(device)
        xs = [torch.from_numpy(rng.standard_normal((m, k)).astype(np.float16)).to(device) for _ in range(3)]
        out = torch.empty((m, n), dtype=dtype, device=device)
        return xs, lambda x: ops.linear_q4_1(x, w, k, out=out, alpha=0.05, engine=engine, **kw)

    return {"few rows, clusters": lambda: i8(16, 2048, 1024, "skinny"), "few rows, tiles": lambda: i8(16, 19456, 256, "skinny"),
            "tile": lambda: i8(200, 2048, 512, "umma"), "pair": lambda: i8(512, 6144, 2048, "umma"),
            "dense f16": lambda: q4(256, 2048, 512, "gemm_two_pass"), "dense f16, pair": lambda: q4(1024, 6144, 512, "gemm_two_pass"),
            "rows": lambda: q4(16, 2048, 1024, "rows"), "rows, f32": lambda: q4(16, 2048, 1024, "rows", torch.float32),
            "rows, flagged": lambda: q4(16, 19456, 256, "rows", overlap_previous=True)}


def _consumers(rng, device, x):
    """Calls that read ``x``, by kernel: as activations, as weights, as an image, as elements."""
    m, n = x.shape
    few = min(m, 8)
    i32 = lambda c: torch.from_numpy(rng.integers(-9, 10, c).astype(np.int32)).to(device)
    f32 = lambda c: torch.rand(c, device=device) * 0.02 + 0.001
    if x.dtype == torch.int8:
        w, a, zp_m, zp_n = _s8(rng, device, 256, n), _s8(rng, device, 8, n), i32(m), i32(256)
        wide, scales, zeros = _s8(rng, device, 256 * 24, n), f32(m), torch.zeros(m, dtype=torch.int8, device=device)
        image, planes = x.view(m, n // 256, 8, 32), x.view(m, n // 512, 4, 128)
        small, large = ops.prepack_conv2d_i8(_s8(rng, device, 3, 3, 32, 48)), ops.prepack_conv2d_i8(_s8(rng, device, 3, 3, 128, 128))
        calls = {
            "decode": lambda: ops.gemm_i8(x[:few], w, engine="decode"), "few rows": lambda: ops.gemm_i8(x[:few], w, engine="skinny"),
            "tile": lambda: ops.gemm_i8(x, w, engine="umma"), "generic": lambda: ops.gemm_i8(x, w[:33], engine="generic"),
            "narrow": lambda: ops.gemm_i8(x[:few], w, engine="narrow"),
            "sums": lambda: ops.gemm_i8(x, w, zp_a=zp_m, zp_w=zp_n), "sums, other operands": lambda: ops.gemm_i8(x, w, zp_a=5, zp_w=zp_n),
            "realign": lambda: ops.gemm_i8(x[:, 3:-2], w[:, 3:-2], zp_w=zp_n),
            "weights, decode": lambda: ops.gemm_i8(a, x, engine="decode"), "weights, few rows": lambda: ops.gemm_i8(a, x, engine="skinny"),
            "weights, tile": lambda: ops.gemm_i8(w, x, engine="umma"), "weights, realign": lambda: ops.gemm_i8(a[:, 1:], x[:, 1:], zp_a=3),
            "batch": lambda: ops.gemm_i8(x.view(4, m // 4, n), x.view(4, m // 4, n)),
            "gather": lambda: ops.conv2d_i8(image, small, padding=(1, 1), out_kind="f32", zp_x=3),
            "implicit": lambda: ops.conv2d_i8(planes, large, padding=(1, 1), out_kind="f32", zp_x=3),
            "dequantize": lambda: ops.dequantize_linear(x, scales, zeros),
        }
        if m >= 256:
            calls["pair"] = lambda: ops.gemm_i8(x, wide, engine="umma")
        return calls
    blocks = torch.from_numpy(synth.q4_1_weights(rng, 512, n)).to(device)
    scales, zeros = f32(m), torch.zeros(m, dtype=torch.int8, device=device)
    w8 = _s8(rng, device, 256, n)
    half = x.dtype == torch.float16
    calls = {
        "quantize": lambda: ops.quantize_linear(x, scales, zeros), "fp_act": lambda: ops.linear_fp_act(x, w8, scale_a=0.02),
        "deferred scaling": lambda: ops.linear_q4_1(x[:1], blocks, n, engine="gemv_dsq"),
        "deferred scaling, early": lambda: ops.linear_q4_1(x[:1], blocks, n, engine="gemv_dsq", overlap_previous=True),
        "warp MMA": lambda: ops.linear_q4_1(x[:few // 2], blocks, n, engine="gemv_mma"),
        "warp MMA, early": lambda: ops.linear_q4_1(x[:few // 2], blocks, n, engine="gemv_mma", overlap_previous=True),
        "CUDA cores": lambda: ops.linear_q4_1(x[:few], blocks, n, engine="gemv_simt"),
        "rows": lambda: ops.linear_q4_1(x[:16], blocks, n, engine="rows"),
        "rows, early": lambda: ops.linear_q4_1(x[:16], blocks, n, engine="rows", overlap_previous=True),
        "two passes": lambda: ops.linear_q4_1(x, blocks, n, engine="gemm_two_pass"),
    }
    if half:
        calls["fused"] = lambda: ops.linear_q4_1(x, blocks, n, engine="gemm")
    return calls


@pytest.mark.parametrize("producer", ["few rows, clusters", "few rows, tiles", "tile", "pair", "dense f16", "dense f16, pair", "rows",
                                      "rows, f32", "rows, flagged"])
def test_what_a_kernel_wrote_just_before(cuda_device, nnb200_lib, producer):
    """Each call reads what the one before has written and the one after writes over it at once, with other values; calls
    that need scratch get the one the call before them had."""
    rng = np.random.default_rng(11)
    torch.manual_seed(3)
    xs, produce = _producers(rng, cuda_device)[producer]()
    calls = _consumers(rng, cuda_device, produce(xs[0]))

    def chain(after):
        seen = []
        for i, call in enumerate(calls.values()):
            for step in range(2):
                produce(xs[(i + step) % 3])
                after()
                seen.append(call())
                after()
        return seen

    want = _same_with_and_without_waiting(chain)
    for i in range(0, len(want), 2):   # the two inputs do not give the same, or nothing would show
        assert not torch.equal(want[i], want[i + 1])


@pytest.mark.parametrize("captured", [False, True])
def test_forks_and_joins(cuda_device, nnb200_lib, captured):
    """Calls on two streams that wait for each other by events, eager and in a CUDA graph: a kernel that may overlap the one
    before it in its stream still comes after what its stream has waited for."""
    rng = np.random.default_rng(5)
    w1, w2, wide = _s8(rng, cuda_device, 2048, 1024), _s8(rng, cuda_device, 1024, 2048), _s8(rng, cuda_device, 6144, 1024)
    blocks = torch.from_numpy(synth.q4_1_weights(rng, 2048, 1024)).to(cuda_device)
    x0 = _s8(rng, cuda_device, 300, 1024)
    outs = {n: torch.empty(s, dtype=t, device=cuda_device) for n, s, t in [
        ("a", (300, 2048), torch.int8), ("b", (16, 2048), torch.int8), ("c", (300, 1024), torch.int8), ("d", (16, 1024), torch.int8),
        ("e", (16, 2048), torch.float16), ("f", (300, 6144), torch.int8)]}
    x = torch.empty_like(x0)
    half = torch.empty((16, 1024), dtype=torch.float16, device=cuda_device)
    scale, zp = torch.full((300,), 0.02, device=cuda_device), torch.zeros(300, dtype=torch.int8, device=cuda_device)
    side = torch.cuda.Stream()
    kw = dict(out_kind="s8", out_scale=20.0, scale_w=0.01)

    def work():
        main = torch.cuda.current_stream()
        for _ in range(3):
            ops.gemm_i8(x, w1, out=outs["a"], engine="umma", **kw)
            side.wait_stream(main)
            with torch.cuda.stream(side):
                ops.gemm_i8(outs["a"][:16, :1024], w1, out=outs["b"], engine="skinny", **kw)     # reads what main wrote
                ops.dequantize_linear(outs["b"][:, :1024].contiguous(), scale[:16], zp[:16], out=half)
                ops.linear_q4_1(half, blocks, 1024, out=outs["e"], engine="rows")
            ops.gemm_i8(outs["a"], w2, out=outs["c"], engine="umma", **kw)
            main.wait_stream(side)
            ops.gemm_i8(outs["b"], w2, out=outs["d"], engine="skinny", **kw)      # behind c on main, reads what side wrote
            ops.gemm_i8(outs["c"], wide, out=outs["f"], engine="umma", **kw)
            x[:16].copy_(outs["d"])
            x[16:].copy_(outs["c"][16:])

    def serial():
        x.copy_(x0)
        work()
        torch.cuda.synchronize()
        return {n: t.clone() for n, t in outs.items()}

    want = serial()
    for _ in range(3):
        x.copy_(x0)
        for t in outs.values():
            t.zero_()
        if captured:
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                work()
            graph.replay()
        else:
            work()
        torch.cuda.synchronize()
        assert all(torch.equal(outs[n].view(torch.uint8), want[n].view(torch.uint8)) for n in outs)
