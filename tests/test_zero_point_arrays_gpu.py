"""Arrays of zero points that the caller has not looked at: the sweeps over the operands look on the device."""
import numpy as np
import pytest
import torch

import oracle
from nnops_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 300, 512), (7, 9001, 528), (5, 4000, 200), (40, 130, 1024), (3000, 33, 2064), (60, 5000, 1024), (2100, 260, 128)])
@pytest.mark.parametrize("live_a", [None, "first", "last"])
@pytest.mark.parametrize("live_w", [None, "last"])
@pytest.mark.parametrize("out_kind", ["s8", "f32"])
def test_zero_arrays_read_no_operand(cuda_device, nnb200_lib, shape, live_a, live_w, out_kind):
    m, n, k = shape
    rng = np.random.default_rng(m + n)
    a, w = rng.integers(-127, 128, (m, k), dtype=np.int8), rng.integers(-127, 128, (n, k), dtype=np.int8)
    za, zw = np.zeros(m, np.int32), np.zeros(n, np.int32)
    for z, live in ((za, live_a), (zw, live_w)):
        if live:
            z[0 if live == "first" else -1] = 3
    kw = {"scale_a": 0.02, "scale_w": rng.uniform(0.001, 0.02, n).astype(np.float32), "zp_a": za, "zp_w": zw}
    if out_kind == "s8":
        kw["out_scale"] = 0.5
    untouched = 0x5A5A5A5A
    workspace = torch.full((1 << 22,), untouched, dtype=torch.int32, device=cuda_device)
    ta, tw = torch.from_numpy(a).to(cuda_device), torch.from_numpy(w).to(cuda_device)
    got = ops.gemm_i8(ta, tw, out_kind=out_kind, workspace=workspace.view(torch.uint8), **kw).cpu().numpy()
    assert np.array_equal(got, oracle.gemm_i8(a, w, out_kind=out_kind, **kw))
    if k % 16:
        return   # copied into aligned rows, and the sums ride along
    # The workspace starts with the sums of A's rows (wanted by zero points of W), then those of W's; a sweep
    # that is shorter than its blocks' looks at the array goes ahead without.
    most = 16 * torch.cuda.get_device_properties(cuda_device).multi_processor_count
    at_w = (m + 63) // 64 * 64
    for start, x, count, live in ((0, a, n, live_w), (at_w, w, m, live_a)):
        sums = workspace[start:start + len(x)].cpu().numpy()
        looks = x.size >= 16 * min(-(-len(x) // 4), most) * count
        assert (sums == untouched).all() if looks and not live else np.array_equal(sums, x.sum(axis=1, dtype=np.int32))
