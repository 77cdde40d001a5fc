"""The compiled half of the tensor front end against the Python code that stands behind it: the same bytes where it
takes the call, the same errors where it does not."""
import numpy as np
import pytest
import torch

from nnops_b200 import capi, ops

pytestmark = pytest.mark.gpu


class _Recorder:
    """The compiled front end, noting of each call whether it took it."""

    def __init__(self, front):
        self.front, self.taken = front, []

    def __getattr__(self, name):
        def call(*args):
            made = getattr(self.front, name)(*args)
            self.taken.append((name, made is not None))
            return made
        return call


# What the Python code does instead, and the calls of its own that the compiled code then takes or not.
LEFT_TO_PYTHON = {
    "numpy parameters": [("gemm_i8", False)], "engine, least scratch": [("gemm_i8", False)],
    "quantize by one, from lists": [("quantize_linear", False)], "conv, zero points": [("conv2d_i8", False)], "conv, raw filter": [],
}


def _calls(dev):
    g = torch.Generator(device=dev).manual_seed(7)
    s8 = lambda *s: torch.randint(-127, 128, s, generator=g, device=dev, dtype=torch.int8)
    i32 = lambda n: torch.randint(-9, 10, (n,), generator=g, device=dev, dtype=torch.int32)
    f32 = lambda *s: torch.rand(s, generator=g, device=dev) * 0.02 + 0.001
    a, w, x = s8(33, 96), s8(70, 96), torch.randn((33, 96), generator=g, device=dev)
    q4 = torch.randint(0, 256, (70, 3, 20), generator=g, device=dev, dtype=torch.uint8)
    q4[:, :, :4] = torch.tensor([0, 36, 0, 168], dtype=torch.uint8, device=dev)   # d = 1/64, m = -1/32
    q4 = q4.reshape(70, 60)
    packed = ops.prepack_i8(w, scale_w=f32(70), zp_w=i32(70))
    q41 = ops.prepack_q4_1(torch.cat([q4[:, :40], q4[:, :40]], 1), 128)
    image, filt = torch.randint(0, 256, (2, 9, 8, 32), generator=g, device=dev, dtype=torch.uint8), s8(3, 3, 32, 48)
    pf, raw = ops.prepack_conv2d_i8(filt), torch.empty((35, 80), dtype=torch.float16, device=dev)
    zp8 = torch.randint(-9, 10, (33,), generator=g, device=dev, dtype=torch.int8)
    return {
        "plain": lambda: ops.gemm_i8(a, w),
        "options": lambda: ops.gemm_i8(a, w, out_kind="s8", bias=i32(70), relu=True, scale_a=f32(33), scale_w=0.01, zp_a=3, zp_w=i32(70),
                                       out_scale=0.7, out_zp=-5),
        "u8 into f16, window": lambda: ops.gemm_i8(a.view(torch.uint8), w, out_kind="f16", out=raw[1:34, 5:75], activation="gelu",
                                                   scale_w=f32(70), min_clip=-1, max_clip=2.5, act_alpha=0.5),
        "batch, transposed": lambda: ops.gemm_i8(s8(3, 33, 96), s8(96, 70).t(), out_kind="f32", scale_a=0.02),
        "numpy parameters": lambda: ops.gemm_i8(a, w, out_kind="f32", scale_w=np.full(70, 0.5, np.float32), zp_a=[2] * 33),
        "engine, least scratch": lambda: ops.gemm_i8(a, w, engine="generic", min_workspace=True, zp_a=3),
        "packed": lambda: ops.gemm_i8_packed(a, packed, out_kind="s8", zp_a=2),
        "off the 16-byte rule": lambda: ops.gemm_i8(s8(64, 200)[:, 1:190], s8(500, 200)[:, 3:192], out_kind="f32", zp_a=i32(64)),
        "q4_1": lambda: ops.linear_q4_1(x, q4, 96, bias=f32(70), activation="silu", alpha=0.5),
        "q4_1 f16": lambda: ops.linear_q4_1(x.half(), q4, 96, out_dtype=torch.float32),
        "q4_1 packed": lambda: ops.linear_q4_1(torch.ones((1, 128), device=dev, dtype=torch.float16), q41, 128),
        "quantize": lambda: ops.quantize_linear(x, f32(33), zp8),
        "quantize along 0 to u8": lambda: ops.quantize_linear(x.half(), f32(33), zp8, axis=0, out_dtype=torch.uint8),
        "quantize by one, from lists": lambda: ops.quantize_linear(x, 0.02, np.int8(3)),
        "dequantize along 1": lambda: ops.dequantize_linear(a.t().contiguous(), f32(33), zp8, axis=1, out_dtype=torch.float16),
        "fp_act": lambda: ops.linear_fp_act(x, w, scale_a=f32(33), scale_w=f32(70), bias=f32(70)),
        "fp_act, one scale": lambda: ops.linear_fp_act(x.half(), w, scale_a=0.02, zp_a=-4, scale_w=f32(70), activation="relu"),
        "fp_act, zero points": lambda: ops.linear_fp_act(x, w, scale_a=f32(33), zp_a=i32(33), act_dtype=torch.uint8),
        "fp_act, one zero point": lambda: ops.linear_fp_act(x, w, scale_a=f32(33), zp_a=130, act_dtype=torch.uint8, zp_w=i32(70)),
        "conv": lambda: ops.conv2d_i8(image, pf, stride=(2, 1), padding=(1, 1), bias=i32(48), relu=True, zp_x=128, scale_w=f32(48), out_scale=0.5),
        "conv, zero points": lambda: ops.conv2d_i8(image, pf, out_kind="f32", zp_w=i32(48), scale_x=0.5),
        "conv, raw filter": lambda: ops.conv2d_i8(image, filt, dilation=(2, 2)),
    }


@pytest.mark.parametrize("name", [
    "plain", "options", "u8 into f16, window", "batch, transposed", "numpy parameters", "engine, least scratch", "packed",
    "off the 16-byte rule", "q4_1", "q4_1 f16", "q4_1 packed", "quantize", "quantize along 0 to u8", "quantize by one, from lists",
    "dequantize along 1", "fp_act", "fp_act, one scale", "fp_act, zero points", "fp_act, one zero point", "conv", "conv, zero points",
    "conv, raw filter"])
def test_same_bytes_as_the_python_path(cuda_device, nnb200_lib, monkeypatch, name):
    calls = _calls(cuda_device)
    recorder = _Recorder(ops._front())
    monkeypatch.setattr(ops, "_native", recorder)
    got = calls[name]().clone()
    if name in LEFT_TO_PYTHON:
        assert recorder.taken == LEFT_TO_PYTHON[name]
    else:
        assert len(recorder.taken) == 1 and recorder.taken[0][1], recorder.taken
    calls = _calls(cuda_device)   # the same inputs again
    monkeypatch.setattr(ops, "_native", ops._NoFront())
    want = calls[name]()
    assert got.dtype == want.dtype and got.shape == want.shape and torch.equal(got.view(torch.uint8), want.contiguous().view(torch.uint8))


def test_mistakes_are_reported_where_they_were(cuda_device, nnb200_lib):
    a = torch.ones((4, 32), dtype=torch.int8, device=cuda_device)
    w = torch.ones((8, 48), dtype=torch.int8, device=cuda_device)
    with pytest.raises(ValueError, match="K mismatch"):
        ops.gemm_i8(a, w)
    with pytest.raises(ValueError, match="expected 8 quantization entries"):
        ops.gemm_i8(a, w[:, :32], scale_w=torch.ones(7, device=cuda_device))
    with pytest.raises(TypeError):
        ops.gemm_i8(a, w[:, :32], no_such_option=1)
    with pytest.raises(KeyError):
        ops.gemm_i8(a, w[:, :32], out_kind="s16")
    with pytest.raises(RuntimeError, match="CUDA"):
        ops.gemm_i8(a.cpu(), w.cpu()[:, :32])
    with pytest.raises(capi.Nnb200Error, match="nnb200_gemm_i8: invalid_argument"):
        ops.gemm_i8(a, w.as_strided((5, 32), (64, 2), 0))   # neither stride is 1
    with pytest.raises(ValueError):
        ops.quantize_linear(a, 1.0, 0)


def test_calls_on_a_side_stream_and_under_capture(cuda_device, nnb200_lib):
    a = torch.randint(-9, 10, (8, 256), dtype=torch.int8, device=cuda_device)
    w = torch.randint(-9, 10, (512, 256), dtype=torch.int8, device=cuda_device)
    want = ops.gemm_i8(a, w)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        got = ops.gemm_i8(a, w)
    got.zero_()
    graph.replay()
    assert torch.equal(got, want)
