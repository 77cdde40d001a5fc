"""The 8-bit epilogues of the tile kernel: two groups of warps that take the tiles in turn, four column parts on
wide tiles.  Byte for byte against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from nnops_b200 import capi, ops

pytestmark = pytest.mark.gpu


def _check(device, m, n, k, *, out_kind="s8", relu=True, out_zp=0, negative="", per_token=False, zero_points=False, bn=None, knobs=None):
    rng = np.random.default_rng(m + n + k)
    a = rng.integers(-127, 128, (m, k), dtype=np.int8)
    w = rng.integers(-127, 128, (n, k), dtype=np.int8)
    scale_w = rng.uniform(0.001, 0.02, n).astype(np.float32)
    if negative == "column":
        scale_w[rng.integers(0, n, 3)] *= -1.0
    scale_a = rng.uniform(0.01, 0.03, m).astype(np.float32) if per_token else 0.02
    if negative == "row":
        scale_a = np.full(m, 0.02, np.float32) if not per_token else scale_a
        scale_a[m // 2] *= -1.0
    kw = dict(out_kind=out_kind, relu=relu, out_zp=out_zp, bias=rng.integers(-1000, 1001, n).astype(np.int32), scale_a=scale_a,
              scale_w=scale_w, out_scale=float(np.sqrt(k)) * 73 * 73 * 0.02 * 0.0105 / 45)
    if zero_points:
        kw.update(zp_a=rng.integers(-5, 6, m).astype(np.int32), zp_w=rng.integers(-3, 4, n).astype(np.int32))
    if bn is not None:
        knobs("i8_bn", bn)
    knobs("i8_pair", 0)
    got = ops.gemm_i8(torch.from_numpy(a).to(device), torch.from_numpy(w).to(device), engine="umma", **kw).cpu().numpy()
    assert capi.take_device_error() == 0
    assert np.array_equal(got, oracle.gemm_i8(a, w, **kw))


@pytest.mark.parametrize("bn", [64, 128, 192, 224, 256, 320, 384, 448, 512])
@pytest.mark.parametrize("out_kind", ["s8", "u8"])
def test_every_tile_width(cuda_device, nnb200_lib, knobs, bn, out_kind):
    """One tile, an odd and an even number of tiles a CTA (with 148 SMs: 19700 rows are 154 tiles of 128), ragged edges."""
    for m, n, k in [(100, bn - 7, 160), (19700, bn, 128), (129, 3 * bn + 40, 144)]:
        if bn > 256 and m > 148 * 128:
            m = 148 * 128 - 5    # the widest tiles are for single waves
        _check(cuda_device, m, n, k, out_kind=out_kind, bn=bn, knobs=knobs)


@pytest.mark.parametrize("relu", [True, False])
@pytest.mark.parametrize("out_zp", [0, 7])
@pytest.mark.parametrize("negative", ["", "column", "row"])
@pytest.mark.parametrize("out_kind", ["s8", "u8"])
def test_relu_zero_point_and_signs(cuda_device, nnb200_lib, knobs, relu, out_zp, negative, out_kind):
    _check(cuda_device, 300, 520, 256, out_kind=out_kind, relu=relu, out_zp=out_zp, negative=negative, knobs=knobs)


@pytest.mark.parametrize("zero_points", [False, True])
@pytest.mark.parametrize("per_token", [False, True])
def test_many_tiles_per_cta(cuda_device, nnb200_lib, knobs, zero_points, per_token):
    _check(cuda_device, 9000, 2070, 96, per_token=per_token, zero_points=zero_points, knobs=knobs)


@pytest.mark.parametrize("n", [64, 68, 72, 94, 97, 99, 1000, 1001, 1002])
@pytest.mark.parametrize("out_kind", ["s8", "f16"])
def test_rows_of_any_pitch(cuda_device, nnb200_lib, n, out_kind):
    """Destination rows at every byte (half) offset, whole and cut chunks; nothing beside them is written."""
    rng = np.random.default_rng(n)
    m, k = 200, 144
    a = rng.integers(-127, 128, (m, k), dtype=np.int8)
    w = rng.integers(-127, 128, (n, k), dtype=np.int8)
    kw = dict(out_kind=out_kind, out_scale=900.0) if out_kind == "s8" else dict(out_kind=out_kind, scale_a=0.02, scale_w=0.01)
    want = oracle.gemm_i8(a, w, **kw)
    dtype = torch.int8 if out_kind == "s8" else torch.float16
    for lead, pitch in [(0, n), (1, n + 3), (3, n + 7)]:
        flat = torch.full((m * pitch + lead,), 77, dtype=dtype, device=cuda_device)
        out = flat[lead:].as_strided((m, n), (pitch, 1))
        ops.gemm_i8(torch.from_numpy(a).to(cuda_device), torch.from_numpy(w).to(cuda_device), out=out, engine="umma", **kw)
        assert np.array_equal(out.cpu().numpy(), want)
        rest = flat.clone()
        rest[lead:].as_strided((m, n), (pitch, 1)).fill_(77)
        assert (rest == 77).all()
