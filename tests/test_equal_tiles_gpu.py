"""The few-row engine on more 128-channel tiles than SMs: equal, narrower tiles.  Byte for byte against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from nnops_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [33, 64, 65])
def test_few_rows_in_equal_tiles(cuda_device, nnb200_lib, m):
    """More 128-channel tiles than SMs without shared K: equal, narrower tiles."""
    rng = np.random.default_rng(m)
    a = rng.integers(-127, 128, (m, 272), dtype=np.int8)
    w = rng.integers(-127, 128, (20011, 272), dtype=np.int8)
    got = ops.gemm_i8(torch.from_numpy(a).to(cuda_device), torch.from_numpy(w).to(cuda_device), engine="skinny", min_workspace=True)
    assert np.array_equal(got.cpu().numpy(), oracle.gemm_i8(a, w))
