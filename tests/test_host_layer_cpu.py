"""The host layer in front of the kernels, as far as it goes without a device."""

import ctypes
import glob
import os
import re
import subprocess

import pytest
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "flash-topk-attention_b200", "csrc")


@pytest.fixture(scope="module")
def lib():
    from flash_topk_attn_v2 import _lib
    return _lib.lib


def _score_code(lib, sb, sn, sh, B=2, H=2, N=128, D=64):
    """Return code of ftk_block_score for tensors of these strides.  The pointers are host
    memory that nothing reads: without a driver a call whose arguments are in order ends
    at the encoding of its tensor maps (-5)."""
    buf = ctypes.create_string_buffer(1 << 16)
    p = (ctypes.addressof(buf) + 255) // 256 * 256
    return lib.ftk_block_score(p, p, 1, B, H, N, D, sb, sn, sh, sb, sn, sh, 0, B * H, 64, 0, 0, 0.125,
                               p, p, 1 << 40, None, None)


@pytest.mark.skipif(torch.cuda.is_available(), reason="host pointers: only without a device")
def test_tensor_maps_refuse_a_repeated_dimension(lib):
    """Stride 0 along an extent above 1 (an expanded tensor) cannot be encoded; along an
    extent of 1 the stride means nothing."""
    ok, bad = -5, -1
    assert _score_code(lib, 128 * 128, 128, 64) == ok
    assert _score_code(lib, 0, 128, 64) == bad
    assert _score_code(lib, 128 * 128, 0, 64) == bad
    assert _score_code(lib, 128 * 128, 128, 0) == bad
    assert _score_code(lib, 0, 128, 64, B=1) == ok
    assert _score_code(lib, 128 * 64, 64, 0, H=1) == ok


def test_expanded_tensors_are_copied():
    """The gradient of a sum over tokens has strides (C, 0, 1); one key head shared by all
    heads, or one batch entry by all, is an expanded tensor too."""
    from flash_topk_attn_v2 import ops
    from flash_topk_attn_v2._lib import native
    o = torch.zeros(2, 64, 128, requires_grad=True)
    seen = []
    o.register_hook(seen.append)
    (o.sum(dim=1) * torch.ones(2, 128)).sum().backward()
    grad = seen[0]
    assert grad.stride(1) == 0 and grad.stride(2) == 1
    flat = torch.randn(1, 64, 128)
    heads = torch.randn(2, 1, 64, 64)
    for x, four_d, D in ((grad, False, 64), (flat.expand(2, 64, 128), False, 64),
                         (heads.expand(2, 4, 64, 64), True, 64)):
        H = x.shape[1] if four_d else x.shape[2] // D
        assert not native.in_place(x, four_d, D)
        y, sb, sn, sh = ops._as_bnhd(x, four_d, H, D)
        assert y.data_ptr() != x.data_ptr() and torch.equal(y, x)
        assert min(sb, sn, sh) > 0
        assert native.in_place(y, four_d, D)
    # a dimension of one may have any stride that is aligned
    assert native.in_place(flat, False, 64)
    assert native.in_place(torch.zeros(1, 64, 128).as_strided((1, 64, 128), (0, 128, 1)), False, 64)


def _fake(shape, dtype=torch.float16, device="cuda:0"):
    return torch.empty(shape, dtype=dtype, device=device)


def test_mismatched_arguments_are_refused_on_the_host():
    """Tensors on another device, of another type or of fewer heads than the kernels would
    read, shown with tensors that have no memory: every call ends before a launch."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    import flash_topk_attn_v2 as ftk
    with FakeTensorMode():
        x, cpu, other = _fake((1, 128, 128)), _fake((1, 128, 128), device="cpu"), \
            _fake((1, 128, 128), device="cuda:1")
        bf, f32 = _fake((1, 128, 128), torch.bfloat16), _fake((1, 128, 128), torch.float32)
        lists = _fake((1, 2, 2, 4), torch.int32)

        def attn(q=x, k=x, v=x, m=lists):
            return ftk.flash_topk_attn(q, k, v, m, None, 2, 64, 64)

        for args in (dict(k=cpu), dict(v=other), dict(q=f32, k=f32, v=cpu.float()),
                     dict(m=_fake((1, 2, 2, 4), torch.int32, "cpu")),
                     dict(m=_fake((1, 2, 2, 4), torch.int32, "cuda:1"))):
            with pytest.raises(ValueError, match="must be on cuda:0"):
                attn(**args)
        for args in (dict(k=bf), dict(v=bf), dict(k=f32, v=f32), dict(k=f32), dict(q=bf)):
            with pytest.raises(ValueError, match="type of q"):
                attn(**args)
        for shape in ((1, 1, 2, 4), (2, 2, 2, 4)):
            with pytest.raises(ValueError, match=r"\[B, H\]"):
                attn(m=_fake(shape, torch.int32))

        idx, scores = _fake((1, 2, 128, 4), torch.int32), _fake((1, 2, 128, 4), torch.float32)
        with pytest.raises(ValueError, match="shape of"):
            ftk.flash_qblock_merge(idx, _fake((1, 2, 128, 3), torch.float32), 64, 8, 8)
        with pytest.raises(ValueError, match="must be on cuda:0"):
            ftk.flash_qblock_merge(idx, scores.cpu(), 64, 8, 8)
        with pytest.raises(ValueError, match="shape of"):
            ftk.build_qblock_topk_indices(idx, 64, (0, 0), _fake((1, 1, 128, 4)), None, 8)
        with pytest.raises(ValueError, match="must be on cuda:0"):
            ftk.flash_topk_score(x, cpu, 2)
        with pytest.raises(ValueError, match="must be on cuda:0"):
            ftk.flash_block_score(x, other, 2, 64)
        with pytest.raises(ValueError, match="counts must be"):
            ftk.flash_build_reverse_indices_cuda(lists, _fake((1, 1, 2), torch.int32), 2)
        with pytest.raises(ValueError, match="must be on cuda:0"):
            ftk.flash_build_reverse_indices_cuda(lists, _fake((1, 2, 2), torch.int32, "cpu"), 2)


def test_the_native_layer_belongs_to_one_pytorch(tmp_path, monkeypatch):
    """Another PyTorch or interpreter makes the built object stale, and an object that was
    built for another is refused at import."""
    import importlib.util
    import os
    import types
    from flash_topk_attn_v2 import _lib
    path = os.path.join(os.path.dirname(os.path.dirname(_lib._HERE)), "flash-topk-attention_b200",
                        "build.py")
    spec = importlib.util.spec_from_file_location("ftk_build_under_test", path)
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    assert _lib.native.built_for == build.built_for()
    _lib.check_native(_lib.native)
    with pytest.raises(ImportError, match="build it again"):
        _lib.check_native(types.SimpleNamespace(built_for="torch 1.0.0, cpython-38"))

    for name in ("NATIVE", "NATIVE_STAMP"):
        monkeypatch.setattr(build, name, str(tmp_path / name))
    assert not build.native_is_current()               # no object
    (tmp_path / "NATIVE").write_text("x")
    assert not build.native_is_current()               # nobody knows what it was built for
    (tmp_path / "NATIVE_STAMP").write_text(build.built_for())
    assert build.native_is_current()
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    assert not build.native_is_current()
    monkeypatch.undo()
    for name in ("NATIVE", "NATIVE_STAMP"):
        monkeypatch.setattr(build, name, str(tmp_path / name))
    os.utime(tmp_path / "NATIVE", (0, 0))              # older than its sources
    assert not build.native_is_current()


@pytest.mark.parametrize("which", ["q", "k", "v"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_forward_mode_is_refused(which, dtype):
    """The attention has no forward-mode derivative: a tangent on an input raises, as a
    custom function without one does, instead of being dropped."""
    import torch.autograd.forward_ad as fw
    from torch._subclasses.fake_tensor import FakeTensorMode
    import flash_topk_attn_v2 as ftk
    with FakeTensorMode(), fw.dual_level():
        x = {n: _fake((1, 128, 128), dtype) for n in "qkv"}
        x[which] = fw.make_dual(x[which], _fake((1, 128, 128), dtype))
        with pytest.raises(NotImplementedError, match="forward-mode"):
            ftk.flash_topk_attn(*x.values(), _fake((1, 2, 2, 4), torch.int32), None, 2, 64, 64)


def test_threads_that_raise_a_kernels_shared_memory(tmp_path):
    """Two threads ask for two sizes of one kernel's dynamic shared memory at once: the limit ends
    at the larger one, as the record has it, whichever call is held up inside the runtime
    (native/smem_limit_probe.cpp).  No launcher sets the limit by itself."""
    exe = str(tmp_path / "probe")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", "/usr/local/cuda/include",
                    os.path.join(HERE, "native", "smem_limit_probe.cpp"), "-o", exe, "-lpthread"], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=60).stdout
    assert out.split() == ["0", "214016", "0"]      # refused, limit, calls for sizes on record
    text = "".join(re.sub(r"//[^\n]*", "", open(f).read()) for f in glob.glob(os.path.join(CSRC, "*.cu*")))
    assert len(re.findall(r"\bcudaFuncSetAttribute\b", text)) == 1
