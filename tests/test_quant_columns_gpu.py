"""QuantizeLinear / DequantizeLinear with one parameter per innermost element, bit for bit against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from nnops_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 8), (3, 8), (5, 64), (33, 72), (7, 2048), (130, 2056), (1000, 264), (2, 3, 40), (9, 100), (17, 1843)])
@pytest.mark.parametrize("dtype", [np.float32, np.float16])
@pytest.mark.parametrize("unsigned", [False, True])
def test_per_column(cuda_device, nnb200_lib, shape, dtype, unsigned):
    rng = np.random.default_rng(sum(shape))
    qt = np.uint8 if unsigned else np.int8
    cols = shape[-1]
    x = rng.standard_normal(shape).astype(dtype)
    flat = x.reshape(-1)
    odd = np.array([np.inf, -np.inf, np.nan, 60000.0, -60000.0, 0.5], dtype)[:flat.size]
    flat[:odd.size] = odd
    scale = rng.uniform(0.01, 0.05, cols).astype(np.float32)
    zp = rng.integers(100, 140, cols).astype(np.uint8) if unsigned else rng.integers(-20, 21, cols).astype(np.int8)
    axis = len(shape) - 1
    want = oracle.quantize_linear(x, scale, zp, axis=axis, out_dtype=qt)
    tx = torch.from_numpy(x).to(cuda_device)
    got = ops.quantize_linear(tx, scale, torch.from_numpy(zp), axis=axis, out_dtype=torch.uint8 if unsigned else torch.int8)
    assert np.array_equal(got.cpu().numpy(), want)
    q = rng.integers(0, 256, shape).astype(np.uint8) if unsigned else rng.integers(-128, 128, shape).astype(np.int8)
    back = ops.dequantize_linear(torch.from_numpy(q).to(cuda_device), scale, torch.from_numpy(zp), axis=axis,
                                 out_dtype=torch.float32 if dtype is np.float32 else torch.float16)
    assert np.array_equal(back.cpu().numpy(), oracle.dequantize_linear(q, scale, zp, axis=axis, out_dtype=dtype))
