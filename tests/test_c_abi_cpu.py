"""CPU-side checks of the boundary: the shared library loads without a GPU,
exports every symbol include/ftk_api.h declares, and the Python mirror raises
the reference's exceptions before touching the device."""

import ctypes
import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "ftk_api.h")


@pytest.fixture(scope="module")
def ftk():
    import flash_topk_attn_v2 as m
    return m


def test_library_exports_every_declared_symbol(ftk):
    from flash_topk_attn_v2 import _lib
    text = open(HEADER).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    declared = set(re.findall(r"\b(ftk_\w+)\s*\(", text))
    assert len(declared) >= 15
    raw = ctypes.CDLL(_lib.LIB_PATH)
    for name in declared:
        assert hasattr(raw, name), f"{name} declared in ftk_api.h but not exported"
    assert declared == set(_lib.SIGNATURES), declared ^ set(_lib.SIGNATURES)


def test_version_and_error_text(ftk):
    from flash_topk_attn_v2 import _lib
    assert _lib.lib.ftk_version() >= 100
    for code in (0, -1, -2, -3, -4, -5, 101, 105):
        assert _lib.error_text(code) != "unknown code"
    assert _lib.error_text(12345) == "unknown code"
    with pytest.raises(ValueError):
        _lib.check(-1, "x")
    with pytest.raises(NotImplementedError):
        _lib.check(-2, "x")
    with pytest.raises(RuntimeError):
        _lib.check(-4, "x")


def test_workspace_queries_need_no_gpu(ftk):
    from flash_topk_attn_v2 import _lib
    lib = _lib.lib
    a = lib.ftk_score_topk_workspace(2, 1024, 16)
    b = lib.ftk_block_score_workspace(2, 1024)
    assert a >= b + 2 * 1024 * 16 * 4 and b >= 2 * 2 * 1024 * 4
    assert lib.ftk_build_reverse_workspace(4, 64, 64) >= 4 * 64 * 2 * 4
    assert lib.ftk_sort_by_count_workspace(5000, 10) >= 11 * 3 * 4


def test_api_names_and_signatures(ftk):
    import inspect
    assert ftk.__all__ == ["flash_topk_score", "build_qblock_topk_indices", "flash_topk_attn"]
    s = inspect.signature(ftk.flash_topk_score)
    assert list(s.parameters) == ["q", "k", "num_heads", "score_block_size", "topk", "padding",
                                  "threshold"]
    assert s.parameters["score_block_size"].default == 64 and s.parameters["topk"].default == 16
    s = inspect.signature(ftk.build_qblock_topk_indices)
    # the reference's five parameters in its order, then this package's optional extension
    assert list(s.parameters) == ["topk_indices", "q_block_size", "q_padding", "topk_scores",
                                  "qblock_topk", "num_score_blocks"]
    assert s.parameters["num_score_blocks"].default is None
    s = inspect.signature(ftk.flash_topk_attn)
    assert list(s.parameters) == ["q", "k", "v", "merged_indices", "counts", "num_heads",
                                  "q_block_size", "kv_block_size", "scale", "num_kv_heads",
                                  "kv_padding", "q_padding", "S_MAX"]


def test_reference_exceptions_before_any_launch(ftk):
    x = torch.zeros(1, 128, 64)
    with pytest.raises(ValueError, match="requires CUDA"):
        ftk.flash_topk_score(x, x, num_heads=1)
    with pytest.raises(ValueError, match="num_heads is required"):
        ftk.flash_topk_score(x, x)
    with pytest.raises(ValueError, match="3D"):
        ftk.flash_topk_score(x[0], x[0], num_heads=1)
    x4 = torch.zeros(1, 2, 128, 32)
    with pytest.raises(ValueError, match="num_heads"):
        ftk.flash_topk_score(x4, x4, num_heads=3)
    idx = torch.zeros(1, 1, 100, 4, dtype=torch.int32)
    with pytest.raises(ValueError, match="divisible"):
        ftk.build_qblock_topk_indices(idx, 64)
    with pytest.raises(ValueError, match="q_pad_head"):
        ftk.build_qblock_topk_indices(idx, 64, q_padding=(64, 0))
    with pytest.raises(ValueError, match="non-negative"):
        ftk.build_qblock_topk_indices(idx, 64, q_padding=(-1, 0))
    with pytest.raises(ValueError, match=r"\[B, H, N, K\]"):
        ftk.build_qblock_topk_indices(idx[0], 64)
    with pytest.raises(ValueError, match="requires CUDA"):
        ftk.flash_topk_attn(x, x, x, idx, None, 1, 64, 64)


def test_no_fallback_when_library_missing(tmp_path, monkeypatch):
    """The package must refuse to import without its CUDA library."""
    from flash_topk_attn_v2 import _lib
    monkeypatch.setattr(os.path, "exists", lambda p, _e=os.path.exists: False
                        if p == _lib.LIB_PATH else _e(p))
    with pytest.raises(ImportError, match="no fallback"):
        _lib._load()


class _Attn(ctypes.Structure):
    """struct ftk_attn of include/ftk_attn.h"""
    _fields_ = ([(n, ctypes.c_void_p) for n in "qkv"] + [("dtype", ctypes.c_int), ("out_f32", ctypes.c_int)]
                + [(n, ctypes.c_int64) for n in ("B", "H", "Hkv", "N", "D")]
                + [(f"s{t}_{x}", ctypes.c_int64) for t in "qkv" for x in "bnh"]
                + [("lists", ctypes.c_void_p)]
                + [(n, ctypes.c_int) for n in ("list_rows", "W", "q_block", "kv_block", "q_pad_head",
                                               "kv_pad_head")]
                + [("scale", ctypes.c_float)])


def test_large_block_lists_split_into_half_blocks(ftk):
    """q / kv blocks of 65..128 rows are worked on as half-size blocks, the lists read in
    place: every query row must keep exactly the same set of key tokens, whatever the pad
    heads cover, and with blocks halved once or twice."""
    import numpy as np
    from flash_topk_attn_v2 import _lib

    def block_tokens(j, kvb, kph, N):
        return range(max(j * kvb - kph, 0), min((j + 1) * kvb - kph, N))

    rng = np.random.default_rng(0)
    for limit, N, g, kvb, qpad, kpad in [(64, 1000, 128, 128, (70, 82), (100, 52)),
                                         (64, 1000, 128, 64, (10, 14), (8, 16)),
                                         (64, 1000, 64, 128, (24, 0), (0, 24)),
                                         (64, 1000, 96, 96, (20, 36), (50, 6)),
                                         (64, 100, 128, 128, (14, 14), (27, 1)),
                                         (64, 1000, 64, 32, (24, 0), (0, 24)),
                                         (32, 1000, 128, 128, (70, 82), (100, 52)),
                                         (32, 1000, 128, 64, (10, 14), (8, 16)),
                                         (32, 1000, 128, 128, (127, 25), (33, 119)),
                                         (32, 100, 64, 128, (28, 0), (27, 1))]:
        QM, M = (qpad[0] + N + qpad[1]) // g, (kpad[0] + N + kpad[1]) // kvb
        lists = [rng.permutation(M)[:int(rng.integers(0, 5))].tolist() for _ in range(QM)]
        a = _Attn(q=64, k=64, v=64, dtype=1, B=1, H=1, Hkv=1, N=N, D=64, lists=64, list_rows=QM, W=4,
                  q_block=g, kv_block=kvb, q_pad_head=qpad[0], kv_pad_head=kpad[0], scale=1.0)
        out = (ctypes.c_int32 * 10)()
        assert _lib.lib.ftk_attn_parts(ctypes.addressof(a), limit, ctypes.addressof(out)) == 0
        pg, pkv, qph, kph, pqm, pm, q_shift, q_off, kv_shift, kv_off = out
        assert pg <= limit and pkv <= limit and 0 <= qph < pg and 0 <= kph < pkv
        assert pqm * pg >= qph + N and pm * pkv >= kph + N
        got = {}
        for m in range(pqm):
            row = (m + q_off) >> q_shift
            assert 0 <= row < QM
            tokens = set()
            for j in lists[row]:
                for x in range((j << kv_shift) - kv_off, ((j + 1) << kv_shift) - kv_off):
                    if 0 <= x < pm:
                        tokens.update(block_tokens(x, pkv, kph, N))
            for r in block_tokens(m, pg, qph, N):
                got[r] = tokens
        for m in range(QM):
            tokens = set()
            for j in lists[m]:
                tokens.update(block_tokens(j, kvb, kpad[0], N))
            for r in block_tokens(m, g, qpad[0], N):
                assert got[r] == tokens, (limit, N, g, kvb, r)
        assert len(got) == N


def test_first_generation_api_names_and_signatures():
    """The older package name keeps the reference's three signatures
    (flash_topk_attn/__init__.py:1-4, scoring.py:1289-1299, attention.py:70-74,
    :423-437) and refuses CPU tensors before any launch."""
    import inspect
    import flash_topk_attn as v1
    assert v1.__all__ == ["flash_topk_score", "flash_topk_attn", "build_qblock_topk_indices"]
    s = inspect.signature(v1.flash_topk_score)
    assert list(s.parameters) == ["q", "k", "v", "num_heads", "score_block_size", "topk",
                                  "padding", "score_only", "backend"]
    assert s.parameters["score_only"].default is False
    assert s.parameters["backend"].default == "triton"
    assert list(inspect.signature(v1.build_qblock_topk_indices).parameters) == [
        "topk_indices", "q_block_size", "q_padding"]
    assert list(inspect.signature(v1.flash_topk_attn).parameters) == [
        "q", "k", "v", "merged_indices", "counts", "num_heads", "q_block_size", "kv_block_size",
        "scale", "num_kv_heads", "kv_padding", "q_padding", "S_MAX"]
    x = torch.zeros(1, 128, 64)
    with pytest.raises(ValueError, match="requires CUDA"):
        v1.flash_topk_score(x, x, x, 1, topk=2)
    with pytest.raises(ValueError, match="topk"):
        v1.flash_topk_score(x, x, x, 1)
    with pytest.raises(ValueError, match="unsupported backend"):
        v1.flash_topk_score(x, x, x, 1, backend="cuda")
    with pytest.raises(ValueError, match="requires CUDA"):
        v1.build_qblock_topk_indices(torch.zeros(1, 1, 128, 2, dtype=torch.int32), 32)
    with pytest.raises(AssertionError):
        v1.flash_topk_attn(x, x, x, None, None, 1, 32, 64)
