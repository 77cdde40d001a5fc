"""Q4_1 weights as the 128-row operand in tensor memory, a few to 128 activation rows, against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from nnops_b200 import ops, synth

pytestmark = pytest.mark.gpu


def _check(device, m, n, k, a_dtype, out_dtype, **kw):
    rng = np.random.default_rng(m * 7 + n + k)
    wb = synth.q4_1_weights(rng, n, k)
    a = rng.standard_normal((m, k)).astype(a_dtype)
    want = oracle.q4_1_matmul(a.astype(np.float32), wb, k, out_dtype="f32", w_round_f16=True).astype(np.float64)
    ta, tw = torch.from_numpy(a).to(device), torch.from_numpy(wb).to(device)
    got = [ops.linear_q4_1(ta, tw, k, out_dtype=out_dtype, engine="rows", **kw).cpu().numpy().astype(np.float64) for _ in range(2)]
    assert np.array_equal(got[0], got[1])   # a fixed order of additions
    # Weights rounded to f16 on both sides and exact products: what is left is the order of f32 sums
    # (sqrt(K) roundings of 2^-24 of the running sum, K up to 8320), the remainder of an f32
    # activation's two f16 parts (2^-22) and the f16 result's own rounding (2^-11).
    rms = float(np.sqrt(np.mean(want ** 2)))
    tol = 2e-5 * (rms + np.abs(want)) + (2.0 ** -11 * np.abs(want) + 2.0 ** -25 if out_dtype == torch.float16 else 0.0)
    assert (np.abs(got[0] - want) <= tol).all(), float((np.abs(got[0] - want) - tol).max())


@pytest.mark.parametrize("shape", [
    # m, n, k: K of half a unit, clusters that share K (few channels), whole waves, several tiles a CTA
    (2, 128, 128), (16, 1, 256), (9, 130, 384), (5, 1000, 2048), (17, 4096, 1152), (33, 129, 8320), (16, 9500, 640),
    (64, 14336, 512), (65, 1000, 384), (128, 300, 4096), (100, 19000, 256), (3, 45000, 128), (7, 40000, 1152),
    # rows of 8- and 4-byte pitch, K padded to 128 (and within a block)
    (16, 3000, 1088), (82, 500, 8992), (11, 128, 4128), (20, 19000, 288), (128, 700, 352), (5, 260, 1000), (70, 300, 40)])
@pytest.mark.parametrize("out_dtype", [torch.float16, torch.float32])
def test_rows_f16(cuda_device, nnb200_lib, shape, out_dtype):
    _check(cuda_device, *shape, np.float16, out_dtype)


@pytest.mark.parametrize("shape", [(1, 300, 256), (2, 1000, 2048), (8, 9500, 640), (9, 4096, 1152), (33, 130, 384), (64, 260, 4096),
                                   (50, 19000, 256), (13, 700, 1056), (40, 192, 1100), (64, 300, 68)])
@pytest.mark.parametrize("out_dtype", [torch.float16, torch.float32])
def test_rows_f32(cuda_device, nnb200_lib, shape, out_dtype):
    _check(cuda_device, *shape, np.float32, out_dtype)


@pytest.mark.parametrize("n", [1000, 9500])
@pytest.mark.parametrize("act", ["none", "silu", "gelu"])
def test_rows_epilogue(cuda_device, nnb200_lib, n, act):
    """alpha, bias, clip and activation, with and without a split of K: the same engine's plain product, finished in f64."""
    rng = np.random.default_rng(n)
    m, k = 18, 768
    wb = torch.from_numpy(synth.q4_1_weights(rng, n, k)).to(cuda_device)
    a = torch.from_numpy(rng.standard_normal((m, k)).astype(np.float16)).to(cuda_device)
    bias = rng.standard_normal(n).astype(np.float32)
    plain = ops.linear_q4_1(a, wb, k, out_dtype=torch.float32, engine="rows").double().cpu()
    x = (plain * 0.5 + torch.from_numpy(bias).double()).clamp(-1.5, 2.0)
    want = {"none": lambda v: v, "silu": torch.nn.functional.silu,
            "gelu": lambda v: torch.nn.functional.gelu(v, approximate="tanh")}[act](x).numpy()
    got = ops.linear_q4_1(a, wb, k, out_dtype=torch.float32, engine="rows", alpha=0.5, bias=bias, min_clip=-1.5, max_clip=2.0,
                          activation=act).cpu().numpy()
    assert np.abs(got - want).max() <= 2e-6 * 4


def test_rows_pitched_and_chosen_by_itself(cuda_device, nnb200_lib):
    """Pitched activations and outputs; the automatic choice from two rows up."""
    rng = np.random.default_rng(1)
    m, n, k = 20, 700, 512
    wb = torch.from_numpy(synth.q4_1_weights(rng, n, k)).to(cuda_device)
    a = torch.from_numpy(rng.standard_normal((m, k + 40)).astype(np.float16)).to(cuda_device)[:, 8:8 + k]
    assert ops.q4_1_engine(a, wb, k, out_dtype=torch.float16) == 7
    out = torch.full((m, n + 24), 7.0, dtype=torch.float16, device=cuda_device)
    ops.linear_q4_1(a, wb, k, out=out[:, 8:8 + n])
    assert torch.equal(out[:, 8:8 + n], ops.linear_q4_1(a.contiguous(), wb, k, engine="rows"))
    assert (out[:, :8] == 7).all() and (out[:, 8 + n:] == 7).all()


@pytest.mark.parametrize("shape,dtype,magnitude", [
    ((2, 300, 1000), np.float32, 1e-6), ((8, 129, 352), np.float32, 1e5), ((13, 200, 4128), np.float32, 1e-6),
    ((16, 64, 1004), np.float32, 1e5), ((5, 260, 1000), np.float32, 1.0),
    ((2, 260, 1000), np.float16, 1.0), ((8, 130, 4128), np.float16, 1.0)])
def test_few_rows_off_the_128_rule_are_computed_in_f32(cuda_device, nnb200_lib, shape, dtype, magnitude):
    """The automatic choice against unrounded weights, over magnitudes that two f16 parts could not hold."""
    m, n, k = shape
    rng = np.random.default_rng(k)
    wb = synth.q4_1_weights(rng, n, k)
    a = (rng.standard_normal((m, k)) * magnitude).astype(dtype)
    blocks = wb.reshape(n, -1, 20)
    d, low = (blocks[:, :, i:i + 2].copy().view(np.float16).astype(np.float64) for i in (0, 2))
    nibbles = np.concatenate([blocks[:, :, 4:] & 15, blocks[:, :, 4:] >> 4], axis=2).astype(np.float64)
    w = (d * nibbles + low).reshape(n, -1)[:, :k]
    got = ops.linear_q4_1(torch.from_numpy(a).to(cuda_device), torch.from_numpy(wb).to(cuda_device), k,
                          out_dtype=torch.float32).cpu().numpy()
    # f32 throughout: a rounding of the weight, a lane's chain of fused multiply-adds (32 to a block, every
    # 32nd block its own), five additions over the lanes: that many times 2^-24 of the sum of magnitudes.
    # (Weights rounded to f16 are off by up to 2^-11 of a term: 50 times as much.)
    chain = 32 * -(-((k + 31) // 32) // 32) + 6
    x = a.astype(np.float64)
    assert (np.abs(got - x @ w.T) <= chain * 2.0 ** -24 * (np.abs(x) @ np.abs(w).T)).all()


@pytest.mark.parametrize("n", [1024, 9600])   # clusters that share K; a tile a CTA
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_overlap_with_the_preceding_kernel(cuda_device, nnb200_lib, n, dtype):
    """Each call reads what the one before wrote, and what a kernel without the attribute wrote."""
    rng = np.random.default_rng(n)
    wb = torch.from_numpy(synth.q4_1_weights(rng, n, n)).to(cuda_device)
    x0 = torch.from_numpy(rng.standard_normal((16, n))).to(device=cuda_device, dtype=dtype)

    def chain(overlap):
        x, seen = x0 * 1.0, []
        for step in range(6):
            x = ops.linear_q4_1(x, wb, n, alpha=0.02, out_dtype=dtype, engine="rows", overlap_previous=overlap)
            if step == 2:
                x = x * 1.5
            seen.append(x)
        return torch.stack(seen)

    want = chain(False)
    assert torch.isfinite(want).all() and want.abs().max() > 0
    for _ in range(5):
        assert torch.equal(chain(True), want)
