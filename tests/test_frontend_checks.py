"""What the Python front end refuses before it calls the library; no GPU, the blocks are never run."""
import pytest
import torch

from nnops_b200 import capi, ops


def _args(a, w, out, **kw):
    return ops.gemm_i8_args(torch.zeros(a, dtype=torch.int8), torch.zeros(w, dtype=torch.int8), torch.zeros(out, dtype=torch.int32),
                            out_kind="s32", **kw)


@pytest.mark.parametrize("a,w,out", [((2, 3, 16, 64), (32, 64), (16, 32)), ((16, 64), (2, 3, 32, 64), (16, 32)),
                                     ((16, 64), (32, 64), (1, 2, 16, 32)), ((64,), (32, 64), (1, 32)), ((16, 64), (64,), (16, 1))])
def test_only_matrices_and_batches_of_them(nnb200_lib, a, w, out):
    with pytest.raises(ValueError):
        _args(a, w, out)
    assert _args((16, 64), (32, 64), (16, 32)).batch == 1
    assert _args((3, 16, 64), (32, 64), (3, 16, 32)).batch == 3


def test_batches_agree_or_are_one(nnb200_lib):
    """The kernels would walk the shorter batch past its end."""
    for a, w in [(2, 3), (3, 2)]:
        with pytest.raises(ValueError):
            _args((a, 16, 64), (w, 32, 64), (3, 16, 32))
    assert _args((1, 16, 64), (3, 32, 64), (3, 16, 32)).a_batch_stride == 0


@pytest.mark.parametrize("zp_a", [0, 7])
def test_scratch_beyond_the_least_may_fail_to_be_had(nnb200_lib, monkeypatch, zp_a):
    """A weight off the 16-byte rule asks for scratch of its own size; without it the call has what it needs."""
    empty = torch.empty

    def short_of_memory(n, *args, **kw):
        if n > limit:
            raise torch.OutOfMemoryError("out of memory")
        return empty(n, *args, **kw)

    limit = 1 << 40
    monkeypatch.setattr(torch, "empty", short_of_memory)
    keep = []
    full = _args((3, 2049), (5000, 2049), (3, 5000), zp_a=zp_a, keep=keep)
    assert full.workspace_bytes > 5000 * 2049
    limit = 1 << 20
    least = _args((3, 2049), (5000, 2049), (3, 5000), zp_a=zp_a, keep=keep)
    need = nnb200_lib.nnb200_gemm_i8_min_workspace_bytes(least)
    assert least.workspace_bytes == need and bool(least.workspace) == (need > 0) == (zp_a != 0)
    limit = 0
    if zp_a:
        with pytest.raises(torch.OutOfMemoryError):
            _args((3, 2049), (5000, 2049), (3, 5000), zp_a=zp_a, keep=keep)


def test_the_compiled_front_end_is_looked_up_by_torch_and_interpreter():
    import sysconfig
    import torch
    name = capi.front_path().name
    assert torch.__version__ in name and str(torch.version.cuda) in name and sysconfig.get_config_var("SOABI") in name


def test_without_the_compiled_front_end_the_python_code_does_the_calls(nnb200_lib, monkeypatch, tmp_path):
    """Not built, or built for another torch: a warning, once, and every function declines every call."""
    for path, content in ((tmp_path / "missing.so", None), (tmp_path / "broken.so", b"not a library")):
        if content is not None:
            path.write_bytes(content)
        monkeypatch.setattr(capi, "front_path", lambda: path)
        monkeypatch.setattr(ops, "_native", None)
        with pytest.warns(RuntimeWarning, match="through the interpreter"):
            assert ops._front().gemm_i8(None, None, "s32", None, {}) is None
        assert ops._native.conv2d_i8() is None
