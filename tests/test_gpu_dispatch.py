"""Branches that a size rule chooses: each at the sizes where it can go wrong,
against the oracle or against the other branch on the same inputs."""

import numpy as np
import pytest
import torch

import cases
import tolerance
from oracle import ftk_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ftk():
    import flash_topk_attn_v2 as m
    return m


def _lists(rng, heads, QM, M, W):
    """Random lists with empty rows and -1 tails."""
    out = np.full((heads, QM, W), -1, dtype=np.int32)
    for h in range(heads):
        for m in range(QM):
            n = int(rng.integers(0, min(W, M) + 1))
            out[h, m, :n] = rng.permutation(M)[:n]
    return out


def _grads(ftk, t, merged, H, g, kvb, **kw):
    q, k, v = (t[n].cuda().requires_grad_(True) for n in "qkv")
    o, lse = ftk.flash_topk_attn(q, k, v, torch.from_numpy(merged).cuda(), None, H, g, kvb, **kw)
    dq, dk, dv = torch.autograd.grad(o, (q, k, v), t["do"].cuda())
    ftk.check_errors()
    return o.detach(), lse, dq, dk, dv


@pytest.mark.parametrize("N,D,bsz,pad", [
    (512, 64, 64, (0, 0)),       # four key tiles
    (600, 128, 64, (20, 20)),    # five: the two accumulators take turns unevenly
    (768, 128, 256, (0, 0)),     # score blocks of two tiles: one group drains them all
    (640, 256, 128, (0, 0)),     # head dim in two slices
])
def test_score_overflow_is_redone_by_the_cta_that_saw_it(ftk, N, D, bsz, pad):
    """Logits far above the first key tile's in the query rows of one CTA only:
    that CTA walks the keys again (exact maximum, then sums), the others do not.
    Bound as for the exact oracle comparison of overflowing rows: fp32 logits of a
    few thousand carry 2^-24 relative error, 2e-4 in the exponential."""
    gen = torch.Generator().manual_seed(7)
    q = torch.randn(1, N, D, generator=gen)
    k = torch.randn(1, N, D, generator=gen)
    k[:, 300:] *= 40.0
    q[:, :256] *= 3.0
    q[:, 256:] *= 0.02
    qh, kh = q.half(), k.half()
    want = orc.block_score(qh.float().numpy(), kh.float().numpy(), 1, bsz, pad)
    got = ftk.flash_block_score(qh.cuda(), kh.cuda(), 1, bsz, pad).cpu().numpy()
    ftk.check_errors()
    assert np.isfinite(got).all()
    np.testing.assert_allclose(got, want, rtol=2e-4, atol=1e-7)


@pytest.mark.parametrize("D,g", [(128, 64), (64, 32)])
def test_redo_of_more_tiles_than_ctas(ftk, monkeypatch, D, g):
    """Every tile of the pipelined forward leaves the safe exponent range: the redo
    kernel's CTAs (one per SM) do more than one tile each, bit for bit as the
    exact kernel alone."""
    H, N, kvb = 80, 512, 64
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype="fp16", seed=21, do_seed=22))
    t["k"][:, 256:] *= 4.0
    t["q"] *= 2.0
    merged = np.tile(np.arange(8, dtype=np.int32), (1, H, N // g, 1))
    merged[0, 1] = -1
    args = (t["q"].cuda(), t["k"].cuda(), t["v"].cuda(), torch.from_numpy(merged).cuda(), None, H, g,
            kvb)
    o, lse = ftk.flash_topk_attn(*args)
    monkeypatch.setenv("FTK_FWD_PIPE", "0")
    o2, lse2 = ftk.flash_topk_attn(*args)
    ftk.check_errors()
    flagged = torch.ones(H, dtype=torch.bool, device="cuda")
    flagged[1] = False
    a, b = (x.view(N, H, D)[:, flagged] for x in (o, o2))
    assert torch.equal(a, b) and torch.equal(lse[0][flagged], lse2[0][flagged])
    assert not o.view(N, H, D)[:, 1].any() and torch.isinf(lse[0, 1]).all()


@pytest.mark.parametrize("H,marked", [(5001, [0, 1, 777, 3413, 3414, 5000]), (300, [299]), (100, [0, 49, 99]),
                                       (7, [])])
def test_redo_finds_the_marked_tiles(ftk, monkeypatch, H, marked):
    """Few tiles among many leave the safe exponent range, three of every head that is marked: the
    redo kernel finds those at the end of the words, of a round of looks (10240 words) and of a
    16-byte load, does each of them, and no other."""
    N, D, g = 300, 64, 64
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype="fp16", seed=25, do_seed=26))
    t["q"].view(N, H, D)[:, marked] *= 2.0
    t["k"].view(N, H, D)[64:, marked] *= 8.0
    merged = torch.arange(5, dtype=torch.int32).cuda().expand(1, H, 5, 5).contiguous()
    args = (t["q"].cuda(), t["k"].cuda(), t["v"].cuda(), merged, None, H, g, 64)
    pads = dict(q_padding=(0, 20), kv_padding=(0, 20))
    o, lse = ftk.flash_topk_attn(*args, **pads)
    monkeypatch.setenv("FTK_FWD_PIPE", "0")
    o2, lse2 = ftk.flash_topk_attn(*args, **pads)
    ftk.check_errors()
    same = (o.view(N, H, D) == o2.view(N, H, D)).all(-1).all(0)
    assert set(torch.nonzero(same).flatten().tolist()) == set(marked)
    assert torch.equal(lse[0, marked], lse2[0, marked])
    # the other heads: two roundings of P and O, values of V up to about 5
    torch.testing.assert_close(o, o2, atol=5 * 2 * 2.0 ** -11, rtol=2.0 ** -9)


@pytest.mark.parametrize("B,N,H,Hkv,D,g,kvb,dtype,f32", [
    (2, 4736, 4, 2, 128, 64, 64, "bf16", False),   # 148 kv tiles: heads walked, pairs of SMs
    (2, 4700, 4, 2, 64, 64, 64, "fp16", False),    # the same in one-CTA kernels, ragged
    (1, 4736, 16, 4, 128, 64, 32, "bf16", True),   # four heads, float32 results
    (1, 300, 6, 2, 128, 64, 64, "bf16", False),    # few tiles: one result per head, summed after
    (1, 300, 6, 2, 96, 32, 64, "bf16", True),
    (2, 4700, 4, 2, 256, 64, 64, "bf16", False),   # head dim 256 on pairs of SMs, walked
    (1, 300, 6, 2, 160, 64, 64, "fp16", True),
])
def test_grouped_heads_sum(ftk, B, N, H, Hkv, D, g, kvb, dtype, f32):
    """dK / dV of grouped kv heads against the same call with K / V repeated per
    query head, its dK / dV added up per group.  Either side rounds: the walk
    rounds the sum once, the other path each head's share and the sum, so the two
    differ by at most half an ulp of every share plus one ulp of the sum (eps / 2
    and eps relative, eps = 2^-7 or 2^-10), and by fp32 noise."""
    grp = H // Hkv
    tail_q, tail_k = -N % g, -N % kvb
    t = cases.make_inputs(dict(B=B, N=N, H=H, D=D, dtype=dtype, seed=5, do_seed=6))
    for n in "kv":
        t[n] = t[n].view(B, N, Hkv, grp, D)[:, :, :, 0].reshape(B, N, Hkv * D).clone()
    if f32:
        t = {n: x.float() for n, x in t.items()}
    QM, M = (N + tail_q) // g, (N + tail_k) // kvb
    W = M if N < 1000 else 6
    merged = _lists(np.random.default_rng(3), B * H, QM, M, W).reshape(B, H, QM, W)
    kw = dict(q_padding=(0, tail_q), kv_padding=(0, tail_k))
    got = _grads(ftk, t, merged, H, g, kvb, num_kv_heads=Hkv, **kw)
    rep = dict(t)
    for n in "kv":
        rep[n] = t[n].view(B, N, Hkv, 1, D).expand(B, N, Hkv, grp, D).reshape(B, N, H * D)
    want = _grads(ftk, rep, merged, H, g, kvb, **kw)
    for i in range(3):
        assert torch.equal(got[i], want[i])
    eps = 2.0 ** -10 if dtype == "fp16" and not f32 else 2.0 ** -7   # float32 is computed in bf16
    for i in (3, 4):
        assert got[i].dtype == (torch.float32 if f32 else want[i].dtype)
        share = want[i].double().view(B, N, Hkv, grp, D)
        total = share.sum(3).reshape(B, N, Hkv * D)
        slack = (0.5 * eps * share.abs().sum(3).reshape(B, N, Hkv * D) + eps * total.abs() + 1e-6)
        assert ((got[i].double() - total).abs() <= slack).all()


@pytest.mark.parametrize("H,D,g,kvb", [(16, 64, 64, 64), (16, 64, 32, 16), (8, 128, 32, 32)])
def test_dkv_tile_order(ftk, monkeypatch, H, D, g, kvb):
    """Several waves of dK / dV tiles are sorted by the work they have; the order
    decides when a tile runs, never what it computes."""
    B, N = 2, 2500
    tail_q, tail_k = -N % g, -N % kvb
    t = cases.make_inputs(dict(B=B, N=N, H=H, D=D, dtype="bf16", seed=8, do_seed=9))
    QM, M = (N + tail_q) // g, (N + tail_k) // kvb
    merged = _lists(np.random.default_rng(4), B * H, QM, M, 6).reshape(B, H, QM, 6)
    merged[:, :, :, 0] = M - 1          # one kv block that everybody reads
    merged[:, :, :, 1:] = np.where(merged[:, :, :, 1:] == M - 1, -1, merged[:, :, :, 1:])
    kw = dict(q_padding=(0, tail_q), kv_padding=(0, tail_k))
    sorted_ = _grads(ftk, t, merged, H, g, kvb, **kw)
    monkeypatch.setenv("FTK_DKV_ORDER", "0")
    plain = _grads(ftk, t, merged, H, g, kvb, **kw)
    for a, b in zip(sorted_, plain):
        assert torch.equal(a, b)


@pytest.mark.parametrize("D,g,kvb,N,qpad,kvpad,W,dtype", [
    (128, 32, 32, 1000, (9, 15), (20, 4), 24, "bf16"),    # wide lists: pairs of SMs, 8 + 8 groups
    (128, 32, 32, 1000, (9, 15), (20, 4), 3, "fp16"),     # narrow lists: one CTA per tile
    (128, 64, 32, 777, (0, 55), (31, 24), 20, "bf16"),    # odd number of kv blocks
    (128, 32, 64, 700, (20, 16), (60, 8), 8, "bf16"),
    (64, 32, 32, 500, (5, 7), (0, 12), 6, "bf16"),
    (64, 64, 32, 330, (0, 54), (11, 11), 11, "fp16"),
    (256, 32, 32, 520, (24, 0), (8, 16), 5, "bf16"),
    (256, 32, 64, 300, (10, 10), (40, 44), 6, "fp16"),
    (160, 64, 32, 384, (0, 0), (0, 0), 7, "bf16"),
])
def test_blocks_of_32_rows(ftk, D, g, kvb, N, qpad, kvpad, W, dtype):
    """Blocks of 32 rows are walked as 64-row tiles with a mask per half: one half
    listed, the other not, last tile half empty, several groups per tile, against
    the oracle (fp16: the plain bound; bf16: with the rounding envelope)."""
    H = 2
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype=dtype, seed=33, do_seed=34))
    x = {k: v.float().numpy() for k, v in t.items()}
    QM, M = (qpad[0] + N + qpad[1]) // g, (kvpad[0] + N + kvpad[1]) // kvb
    merged = _lists(np.random.default_rng(7), H, QM, M, W)[None]
    o, lse, *grads = _grads(ftk, t, merged, H, g, kvb, q_padding=qpad, kv_padding=kvpad)
    og = o.float().cpu().numpy()
    ora = tolerance.attention_oracles(orc, x, merged, H, g, kvb, dtype, og, qpad, kvpad)
    np.testing.assert_allclose(lse.cpu().numpy(), ora["lse"], atol=2e-3, rtol=1e-2)
    for nm, y in zip(("O", "dQ", "dK", "dV"), (o, *grads)):
        got = y.float().cpu().numpy()
        if dtype == "fp16":
            assert (tolerance.rel_err(got, ora["exact"][nm]) <= 1).all(), nm
        else:
            tolerance.check_rounded(got, ora["exact"][nm], ora["rounded"][nm],
                                    ora["envelope"][nm], nm)


@pytest.mark.parametrize("g,kvb", [(32, 32), (32, 64)])
def test_forward_reference_needs_more_than_four_tiles(ftk, g, kvb):
    """Eight q-blocks of a pair with disjoint lists, too many for the four tiles that
    give the rows their reference exponents: the tiles concerned go to the exact
    kernel, the others do not."""
    H, D, N = 2, 128, 512
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype="bf16", seed=35, do_seed=36))
    x = {k: v.float().numpy() for k, v in t.items()}
    QM, M = N // g, N // kvb
    merged = np.full((1, H, QM, M), -1, dtype=np.int32)
    for m in range(QM):
        merged[0, 0, m, 0] = (m * (64 // kvb)) % M
        merged[0, 1, m, :M] = np.random.default_rng(m).permutation(M)
    o, lse = ftk.flash_topk_attn(t["q"].cuda(), t["k"].cuda(), t["v"].cuda(),
                                 torch.from_numpy(merged).cuda(), None, H, g, kvb)
    ftk.check_errors()
    wo, wl = orc.sparse_attn_fwd(x["q"], x["k"], x["v"], merged, H, g, kvb)
    np.testing.assert_allclose(lse.cpu().numpy(), wl, atol=2e-3, rtol=1e-2)
    # one block of 32 or 64 keys per row: a bf16 P and a bf16 O, 2^-8 of the value each, and
    # the values of V are at most about 4
    np.testing.assert_allclose(o.float().cpu().numpy(), wo, atol=4 * 2 * 2.0 ** -8, rtol=2.0 ** -7)


@pytest.mark.parametrize("N,D,bsz,topk", [(3000, 128, 64, 8), (2050, 64, 128, 6), (1024, 256, 256, 4)])
def test_scoring_does_not_depend_on_the_split_of_the_keys(ftk, N, D, bsz, topk):
    """Few tiles of query rows: clusters share one and split its keys; many: none does.
    One slice alone and the same slice among 64 others give the same bits."""
    pad = (0, -N % bsz)
    t = cases.make_inputs(dict(B=64, N=N, H=1, D=D, dtype="bf16", seed=55, do_seed=56))
    q, k = t["q"].cuda(), t["k"].cuda()
    many = ftk.flash_topk_score(q, k, 1, bsz, topk, pad, 0.9)
    for b in (0, 63):
        one = ftk.flash_topk_score(q[b:b + 1], k[b:b + 1], 1, bsz, topk, pad, 0.9)
        for a, x in zip(one, many):
            assert torch.equal(a[0], x[b])
    ftk.check_errors()


@pytest.mark.parametrize("D,g", [(64, 64), (64, 32), (64, 128), (128, 64)])
def test_forward_ring(ftk, D, g):
    """Lists of 0, 1, 2, ... 13 tiles: fewer than the softmax groups, fewer than the
    stages of the ring, and more than one turn of it, on grids whose CTAs share an SM
    and on those where they do not (fp16: the plain bound)."""
    B, H, N, kvb = 2, 8, 1024, 64
    M, QM = N // kvb, N // g
    t = cases.make_inputs(dict(B=B, N=N, H=H, D=D, dtype="fp16", seed=51, do_seed=52))
    merged = np.full((B, H, QM, M), -1, dtype=np.int32)
    for m in range(QM):
        n = (m * g // 128) % 14      # as long for every q-block of a tile: the union's size
        for h in range(H):
            merged[:, h, m, :n] = (np.arange(n) + 3 * h) % M
    o, lse = ftk.flash_topk_attn(t["q"].cuda(), t["k"].cuda(), t["v"].cuda(),
                                 torch.from_numpy(merged).cuda(), None, H, g, kvb)
    ftk.check_errors()
    want_o, want_lse = orc.sparse_attn_fwd(t["q"].float().numpy(), t["k"].float().numpy(),
                                           t["v"].float().numpy(), merged, H, g, kvb)
    np.testing.assert_allclose(lse.cpu().numpy(), want_lse, atol=2e-3, rtol=1e-2)
    assert (tolerance.rel_err(o.float().cpu().numpy(), want_o) <= 1).all()


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("D,kvb,N,W,hot", [(128, 64, 1000, 7, 1.0), (128, 32, 1000, 9, 1.0), (96, 64, 900, 14, 1.0),
                                           (128, 64, 1024, 16, 6.0), (80, 64, 700, 2, 1.0)])
def test_forward_of_two_ctas_per_sm(ftk, dtype, D, kvb, N, W, hot):
    """Head dim 128, several waves of tiles: two forward CTAs share an SM.  One head of one batch
    entry alone is a grid of one wave and has the SM to itself; the row sums have the same parts and
    the same tiles give the references, so O and lse are the same bit for bit: lists of none to all
    blocks, odd and even numbers of tiles, rows for the exact kernel (fp16, hot)."""
    B, H, g = 2, 20, 64
    t = cases.make_inputs(dict(B=B, N=N, H=H, D=D, dtype=dtype, seed=63, do_seed=64))
    t["k"][:, N // 2:] *= hot
    QM, M = -(-N // g), -(-N // kvb)
    merged = _lists(np.random.default_rng(10), B * H, QM, M, W).reshape(B, H, QM, W)
    merged[0, 0, :, :] = -1
    merged[0, 0, :, 0] = M - 1          # one tile each
    pads = dict(q_padding=(0, QM * g - N), kv_padding=(0, M * kvb - N))
    call = lambda x, m, h: ftk.flash_topk_attn(x["q"].cuda(), x["k"].cuda(), x["v"].cuda(),
                                               torch.from_numpy(m).cuda(), None, h, g, kvb, **pads)
    o, lse = call(t, merged, H)
    for b, h in ((0, 0), (0, 7), (1, 19)):
        part = {k: v.view(B, N, H, D)[b:b + 1, :, h].contiguous() for k, v in t.items()}
        o1, lse1 = call(part, merged[b:b + 1, h:h + 1].copy(), 1)
        assert torch.equal(o1[0], o.view(B, N, H, D)[b, :, h]) and torch.equal(lse1[0, 0], lse[b, h])
    ftk.check_errors()


@pytest.mark.parametrize("D,kvb,W,dtype", [(128, 64, 101, "bf16"), (128, 64, 77, "fp16"), (96, 64, 101, "fp16"),
                                           (128, 32, 201, "fp16"), (128, 32, 160, "fp16")])
def test_forward_of_long_lists(ftk, monkeypatch, D, kvb, W, dtype):
    """More than 96 tiles of 64 keys and lists of three quarters of the blocks: the forward runs on
    pairs of SMs.  Where all blocks are listed the tiles are those of a single SM, bit for bit;
    else fp16 holds the plain bound against float64."""
    N, H, g = 6401, 2, 64
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype=dtype, seed=65, do_seed=66))
    QM, M = -(-N // g), -(-N // kvb)
    rng = np.random.default_rng(11)
    merged = np.stack([rng.permutation(M)[:W] for _ in range(H * QM)]).reshape(1, H, QM, W).astype(np.int32)
    merged[0, 1, 3] = -1
    pads = ((0, QM * g - N), (0, M * kvb - N))
    call = lambda: ftk.flash_topk_attn(t["q"].cuda(), t["k"].cuda(), t["v"].cuda(), torch.from_numpy(merged).cuda(),
                                       None, H, g, kvb, q_padding=pads[0], kv_padding=pads[1])
    o, lse = call()
    if W >= M:
        monkeypatch.setenv("FTK_FWD_2CTA", "0")
        o2, lse2 = call()
        assert torch.equal(o, o2) and torch.equal(lse, lse2)
    else:
        x = {n: v.float().numpy() for n, v in t.items()}
        wo, wl = orc.sparse_attn_fwd(x["q"], x["k"], x["v"], merged, H, g, kvb, None, *pads)
        np.testing.assert_allclose(lse.cpu().numpy(), wl, atol=2e-3, rtol=1e-2)
        assert (tolerance.rel_err(o.float().cpu().numpy(), wo) <= 1).all()
    ftk.check_errors()


@pytest.mark.parametrize("D,g,kvb", [(128, 64, 64), (128, 32, 64), (128, 48, 64), (128, 16, 32),
                                     (96, 64, 32), (64, 64, 64), (64, 32, 32)])
def test_dkv_rounds(ftk, D, g, kvb):
    """dK / dV of kv tiles that 0, 1, 2, ... 9 q-blocks list, or half of their rows: no round, one
    that has no successor, odd and even numbers, and more than a turn of the ring, with whole and
    masked tiles.  Lists below half of the blocks: the kernels of single SMs.  fp16: the plain
    bound."""
    H, N = 2, 48 * 60
    M, QM = -(-N // kvb), N // g
    per = 128 // kvb
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype="fp16", seed=53, do_seed=54))
    merged = np.full((1, H, QM, 10 * per), -1, dtype=np.int32)
    for m in range(QM):
        ids = [tile * per + b for tile in range(10) for b in range(per)
               if 3 * m < 3 * tile - (b % 2)]
        merged[0, 0, m, :len(ids)] = ids
        merged[0, 1, m, :len(ids[::2])] = ids[::2]      # every other block: half of a tile's rows
    assert 2 * merged.shape[-1] < M
    pads = dict(q_padding=(0, QM * g - N), kv_padding=(0, M * kvb - N))
    o, _, dq, dk, dv = _grads(ftk, t, merged, H, g, kvb, **pads)
    x = {n: v.float().numpy() for n, v in t.items()}
    args = (x["q"], x["k"], x["v"])
    _, lse = orc.sparse_attn_fwd(*args, merged, H, g, kvb, None, (0, QM * g - N), (0, M * kvb - N))
    want = orc.sparse_attn_bwd(*args, o.float().cpu().numpy(), lse, x["do"], merged, H, g, kvb, None,
                               (0, QM * g - N), (0, M * kvb - N))
    for got, w in zip((dq, dk, dv), want):
        assert (tolerance.rel_err(got.float().cpu().numpy(), w) <= 1).all()


@pytest.mark.parametrize("g,kvb,W", [(64, 64, 9), (32, 64, 4), (64, 32, 20), (64, 16, 30)])
def test_dq_of_two_ctas_per_sm(ftk, g, kvb, W):
    """Head dim 64, 256 tiles of query rows: two dQ CTAs share an SM.  Two heads of one
    batch entry alone fill no wave and take the SM each; both add up the tiles of a row
    in the same order, so dQ is the same bit for bit."""
    B, H, N, D = 2, 16, 1000, 64
    t = cases.make_inputs(dict(B=B, N=N, H=H, D=D, dtype="bf16", seed=61, do_seed=62))
    QM, M = -(-N // g), -(-N // kvb)
    merged = _lists(np.random.default_rng(9), B * H, QM, M, W).reshape(B, H, QM, W)
    pads = dict(q_padding=(0, QM * g - N), kv_padding=(0, M * kvb - N))
    dq = _grads(ftk, t, merged, H, g, kvb, **pads)[2]
    for b, h in ((0, 0), (1, 14)):
        part = {k: v.view(B, N, H, D)[b:b + 1, :, h:h + 2].reshape(1, N, 2 * D).contiguous()
                for k, v in t.items()}
        alone = _grads(ftk, part, merged[b:b + 1, h:h + 2].copy(), 2, g, kvb, **pads)[2]
        assert torch.equal(alone, dq.view(B, N, H, D)[b:b + 1, :, h:h + 2].reshape(1, N, 2 * D))


@pytest.mark.parametrize("D", [64, 128])
def test_redo_kernel_directly_before_the_backward(ftk, monkeypatch, D):
    """Every tile is flagged, and the gradient kernel follows the redo kernel with nothing
    in between: both allocate TMEM, and the results are those of the exact kernel alone."""
    B, H, N, g, kvb = 2, 16, 1024, 64, 64
    t = cases.make_inputs(dict(B=B, N=N, H=H, D=D, dtype="fp16", seed=23, do_seed=24))
    t["k"][:, 512:] *= 4.0
    t["q"] *= 2.0
    merged = np.tile(np.arange(N // kvb, dtype=np.int32), (B, H, N // g, 1))
    got = [_grads(ftk, t, merged, H, g, kvb) for _ in range(3)]
    monkeypatch.setenv("FTK_FWD_PIPE", "0")
    want = _grads(ftk, t, merged, H, g, kvb)
    for run in got:
        for a, b in zip(run, want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("M", [20, 64, 200, 1000, 1100, 2048, 2100])
def test_select_of_values_that_are_no_scores(ftk, M):
    """Rows with NaN, infinities, negative values and zeros: an average that is not >= 0
    counts as 0, the order is that of the averages with ties to the lower block, the cut is
    where the running sum of the raw values first reaches the threshold (never, once it is
    NaN)."""
    rng = np.random.default_rng(M)
    x = rng.random((24, M)).astype(np.float32)
    x /= x.sum(-1, keepdims=True)
    x[1, ::3] = np.nan
    x[2, 1::5] = np.inf
    x[3, ::2] *= -1
    x[4] = 0
    x[5] = np.nan
    x[6, 3], x[6, 4] = np.nan, np.inf
    x[7] = -1
    x[8, :M // 2] = -np.inf
    x[9] = np.float32(1e-45) * rng.integers(0, 3, M)
    x[10] = 3.0e38
    scores = torch.from_numpy(x).cuda().view(1, 1, 24, M)
    for k, thr, b, pad in ((8, 0.5, 64, (0, 0)), (32, 1.5, 64, (10, 3)), (64, 0.1, 48, (0, 0)),
                           (1, 0.0, 64, (0, 5)), (70, 0.9, 64, (0, 0))):
        width = min(k, M)
        count = np.full(M, b, np.float32)
        count[0] -= pad[0]
        count[-1] -= pad[1]
        with np.errstate(all="ignore"):
            avg = x / count
            avg = np.where(avg >= 0, avg, np.float32(0))
            order = np.argsort(-avg, axis=1, kind="stable")[:, :width]
            raw = np.take_along_axis(x, order, 1)
            cum = np.zeros(24, np.float32)
            cut = np.zeros(24, bool)
            want = np.full((24, width), -1, np.int32), np.zeros((24, width), np.float32), \
                np.zeros((24, width), np.float32)
            for r in range(width):
                on = ~cut
                want[0][on, r] = order[on, r]
                want[1][on, r] = raw[on, r]
                want[2][on, r] = np.take_along_axis(avg, order, 1)[on, r]
                cum = np.where(on, cum + raw[:, r], cum)
                cut |= cum >= np.float32(thr)
        got = ftk.flash_topk_select(scores, thr, k, b, pad)
        for g, w in zip(got, want):
            np.testing.assert_array_equal(g[0, 0].cpu().numpy(), w, err_msg=f"{k} {thr} {b} {pad}")
    ftk.check_errors()


@pytest.mark.parametrize("M,k,b,pad,offset", [
    (1, 1, 64, (3, 2), 0), (2, 1, 64, (0, 5), 0), (4, 4, 64, (0, 0), 0), (15, 3, 64, (0, 0), 0),
    (16, 16, 64, (0, 0), 1), (17, 16, 64, (9, 9), 0), (32, 8, 32, (20, 0), 0), (33, 32, 64, (0, 0), 0),
    (47, 16, 64, (8, 8), 0), (64, 17, 64, (0, 0), 0), (96, 32, 128, (0, 1), 1), (100, 24, 48, (5, 0), 0),
    (118, 24, 128, (40, 20), 0), (128, 16, 64, (0, 0), 0), (128, 32, 64, (0, 0), 1), (128, 30, 80, (0, 0), 0),
])
def test_select_with_a_row_per_lane(ftk, M, k, b, pad, offset):
    """Enough rows for the kernel that gives each lane a row (the last batch is not full): the
    order is exact where keys of 32 bits are not, with averages that tie, that differ by their last
    bit around the cut, far above the smallest one, zero, infinite, negative and NaN."""
    rng = np.random.default_rng(100 * M + k)
    rows = 150 * (96 + 2 * 128) * 3 // 2 + 5
    x = rng.random((rows, M)).astype(np.float32)
    ulp = np.float32(2.0 ** -23)
    kind = np.arange(rows) % 16
    x[kind == 1] = 1 + ulp * rng.integers(0, 6, (int((kind == 1).sum()), M))          # ties and last bits
    far = 1 + ulp * rng.integers(0, 400, (int((kind == 2).sum()), M)).astype(np.float32)
    far[:, 0] = 1e-6                                                                  # ... far above the first
    x[kind == 2] = far
    x[kind == 3] = np.float32(0.25)                                                   # all the same
    x[kind == 4] = 0
    x[kind == 5, ::3] = np.nan
    x[kind == 6, 1::5] = np.inf
    x[kind == 7, ::2] *= -1
    x[kind == 8] = rng.integers(0, 4, (int((kind == 8).sum()), M)) / 8                # many ties
    x[kind == 9] = np.exp(20 * x[kind == 9])
    x[kind == 10] = np.sort(x[kind == 10], axis=1)
    x[kind == 11] = -np.sort(-x[kind == 11], axis=1)
    x[kind == 12] = np.float32(1e-45) * rng.integers(0, 3, (int((kind == 12).sum()), M))
    x[kind == 13] = 0.015 * (1 + 0.02 * rng.standard_normal((int((kind == 13).sum()), M)))
    buf = torch.empty(rows * M + offset, device="cuda")
    scores = buf[offset:].view(1, 1, rows, M)                   # offset 1: rows that 16-byte copies cannot take
    scores.copy_(torch.from_numpy(x).view(1, 1, rows, M))
    count = np.full(M, b, np.float32)
    count[0] -= pad[0]
    count[-1] -= pad[1]
    with np.errstate(all="ignore"):
        avg = x / count
        avg = np.where(avg >= 0, avg, np.float32(0))
        order = np.argsort(-avg, axis=1, kind="stable")[:, :k]
        raw = np.take_along_axis(x, order, 1)
        picked = np.take_along_axis(avg, order, 1)
        for thr in (2.0 * M, 0.4 * k):
            cum, cut = np.zeros(rows, np.float32), np.zeros(rows, bool)
            keep = np.zeros((rows, k), bool)
            for r in range(k):
                keep[:, r] = ~cut
                cum = cum + raw[:, r]
                cut |= cum >= np.float32(thr)
            got = ftk.flash_topk_select(scores, thr, k, b, pad)
            for g, w, none in zip(got, (order, raw, picked), (-1, 0, 0)):
                w = np.where(keep, w, none).astype(g.cpu().numpy().dtype)
                np.testing.assert_array_equal(g[0, 0].cpu().numpy(), w, err_msg=f"threshold {thr}")
    ftk.check_errors()


@pytest.mark.parametrize("M,k,b,pad", [
    (4, 3, 64, (0, 0)), (17, 16, 64, (0, 0)), (32, 8, 64, (5, 0)), (33, 32, 64, (0, 0)), (47, 15, 64, (0, 9)),
    (64, 17, 48, (0, 0)), (100, 24, 64, (0, 0)), (128, 16, 64, (0, 0)), (128, 32, 64, (0, 0)), (16, 7, 48, (3, 0)),
])
def test_select_of_rows_that_tie_at_the_cut(ftk, M, k, b, pad):
    """Batches of 32 rows in which up to all tie where the last pick is cut: equal averages that have
    a place to themselves or not, averages that differ by last bits far above the row's smallest one,
    ties below everything that the first entries hold, and all of these among rows that do not
    tie, with one to 32 of a batch: the order is exact, and the lower block goes first."""
    rng = np.random.default_rng(1000 * M + k)
    rows = 128 * 150 * 4
    ulp = np.float32(2.0 ** -23)
    x = rng.random((rows, M)).astype(np.float32)
    batch, lane = np.arange(rows) // 32, np.arange(rows) % 32
    kind = batch % 12
    tied = lane < 1 + (batch // 12) % 32                    # 1 .. 32 rows of a batch

    def put(which, values):
        at = (kind == which) & tied
        x[at] = values(int(at.sum()))
    put(0, lambda n: np.full((n, M), 0.25))
    put(1, lambda n: np.zeros((n, M)))
    put(2, lambda n: rng.integers(0, 9, (n, M)) / 8)
    put(3, lambda n: np.where(np.arange(M) % 3 == 0, 1e-4, 1.0) * np.ones((n, 1)))
    put(4, lambda n: np.where(rng.random((n, M)) < 0.2, 1e-6, 1 + ulp * rng.integers(0, 3, (n, M))))
    put(5, lambda n: np.where(rng.random((n, M)) < 0.2, 1e-6, 1 + ulp * rng.integers(0, 400, (n, M))))
    put(6, lambda n: np.where(np.arange(M) < 2, 8.0, 0.125 * rng.integers(1, 3, (n, M))))
    put(7, lambda n: np.where(np.arange(M) < min(16, k), 1e6, 1 + ulp * rng.integers(0, 2, (n, M))))
    put(8, lambda n: np.where(rng.random((n, M)) < 0.3, np.inf, rng.integers(0, 2, (n, M)) / 2))
    put(9, lambda n: np.float32(1e-45) * rng.integers(0, 4, (n, M)))
    put(10, lambda n: np.where(np.arange(M) % 2 == 0, np.nan, -0.0) + 0.5 * rng.integers(0, 2, (n, M)))
    put(11, lambda n: np.exp2(rng.integers(-30, 4, (n, M)).astype(np.float32)))
    count = np.full(M, b, np.float32)
    count[0] -= pad[0]
    count[-1] -= pad[1]
    with np.errstate(all="ignore"):
        avg = x / count
        avg = np.where(avg > 0, avg, np.float32(0))
        order = np.argsort(-avg, axis=1, kind="stable")[:, :k]
    got = ftk.flash_topk_select(torch.from_numpy(x).cuda().view(1, 1, rows, M), float("inf"), k, b, pad)
    ftk.check_errors()
    # a sum that is infinite reaches any threshold: such rows end there
    raw = np.take_along_axis(x, order, 1)
    with np.errstate(all="ignore"):
        cut = np.cumsum(raw, axis=1) >= np.inf
    keep = ~np.concatenate([np.zeros((rows, 1), bool), cut[:, :-1]], axis=1)
    for g, w, none in zip(got, (order, raw, np.take_along_axis(avg, order, 1)), (-1, 0, 0)):
        w = np.where(keep, w, none).astype(g.cpu().numpy().dtype)
        np.testing.assert_array_equal(g[0, 0].cpu().numpy(), w)


@pytest.mark.parametrize("N,M,k,g,pad,W", [
    (200, 4, 3, 32, 0, 96), (100, 1, 1, 16, 0, 16), (512, 33, 8, 64, 5, 7), (700, 128, 32, 64, 0, 2048),
    (300, 127, 40, 32, 31, 130), (600, 64, 64, 128, 0, 50), (40, 100, 24, 64, 60, 30), (1000, 8, 8, 200, 0, 3),
])
def test_merge_with_a_cta_per_q_block(ftk, N, M, k, g, pad, W):
    """Few q-blocks go to CTAs of their own, the same ones repeated often to a warp each: lists,
    scores and counts agree bit for bit, with rows that name a block twice, entries of -1, scores
    that are negative, zero or NaN, sums that tie, and lists cut short."""
    rng = np.random.default_rng(N + M)
    idx = np.stack([rng.permutation(M)[:k] for _ in range(2 * N)]).reshape(1, 2, N, k).astype(np.int32)
    scr = rng.random((1, 2, N, k)).astype(np.float32)
    idx[0, 0, ::7, k // 2:] = -1
    scr[0, 0, 1::9] = 0.5
    scr[0, 0, 2::11, 0] = -1
    if k > 1:
        idx[0, 1, 3::50, 1] = idx[0, 1, 3::50, 0]        # a block twice in a row
    scr[0, 1, 5::90, 0] = np.nan
    idx, scr = torch.from_numpy(idx).cuda(), torch.from_numpy(scr).cuda()
    rep = min(3000, int(1e8) // (2 * N * k))
    for s in (scr, None):
        call = lambda i, s: ftk.flash_qblock_merge(i, s, g, W, M, q_padding=(pad, -(N + pad) % g),
                                                   return_counts=True, want_scores=True)
        few = call(idx, s)
        many = call(idx.repeat(rep, 1, 1, 1), None if s is None else s.repeat(rep, 1, 1, 1))
        for a, b in zip(few, many):
            if a is not None:
                assert torch.equal(a[0], b[0]) and torch.equal(a[0], b[-1])
    ftk.check_errors()


@pytest.mark.parametrize("N,M,k,g,W", [
    (700, 128, 128, 32, 128), (600, 64, 50, 64, 64), (300, 127, 33, 16, 40), (500, 16, 7, 100, 16), (90, 3, 3, 30, 2),
    (400, 1, 1, 200, 3),
])
def test_merge_of_rows_that_name_blocks_twice(ftk, N, M, k, g, W):
    """Rows of picks with replacement, absent ones among them, beside rows that name no block twice: a
    CTA per q-block adds a row's entries of one block in their order, as a warp per q-block (the same
    q-blocks repeated often) does.  Scores of several magnitudes, so that another order shows."""
    rng = np.random.default_rng(7 * N + M)
    idx = rng.integers(-1, M, (1, 2, N, k)).astype(np.int32)
    for n in range(0, N, 3):
        idx[0, :, n] = rng.permutation(M)[:k]
    scr = np.exp(6 * rng.standard_normal((1, 2, N, k))).astype(np.float32)
    idx, scr = torch.from_numpy(idx).cuda(), torch.from_numpy(scr).cuda()
    rep = min(3000, int(1e8) // (2 * N * k))
    call = lambda i, s: ftk.flash_qblock_merge(i, s, g, W, M, q_padding=(0, -N % g), return_counts=True,
                                               want_scores=True)
    few, many = call(idx, scr), call(idx.repeat(rep, 1, 1, 1), scr.repeat(rep, 1, 1, 1))
    for a, b in zip(few, many):
        assert torch.equal(a[0], b[0]) and torch.equal(a[0], b[-1])
    want = torch.zeros(2, -(-N // g), M + 1, dtype=torch.float64)
    block = (torch.arange(N) // g).view(1, N, 1).expand(2, N, k)
    at = torch.where(idx[0] < 0, M, idx[0]).long().cpu()
    want.index_put_((torch.arange(2).view(2, 1, 1).expand_as(at), block, at), scr[0].double().cpu(), accumulate=True)
    top = want[..., :M].sort(-1, descending=True).values[..., :W]
    torch.testing.assert_close(few[1][0][..., :top.shape[-1]].double().cpu(), top, rtol=g * k * 2.0 ** -24, atol=0)
    ftk.check_errors()


@pytest.mark.parametrize("D,g,kvb,N,W", [
    (64, 64, 16, 9600, 37),      # 600 blocks: more than one entry a thread of 18 warps
    (64, 16, 64, 1000, 5),       # eight groups per tile
    (128, 64, 64, 4200, 9),
    (128, 32, 32, 2100, 11),     # tiles of two listed blocks
    (128, 128, 128, 7000, 6),    # lists over blocks of twice the size
])
def test_lists_of_any_width(ftk, D, g, kvb, N, W):
    """The same lists, as they are, behind one more and with a tail that lets them be read
    16 bytes at a time: the union is the same, so are all results, bit for bit (the widths
    are all short enough for the one-CTA kernels)."""
    H = 2
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype="bf16", seed=71, do_seed=72))
    QM, M = -(-N // g), -(-N // kvb)
    lists = _lists(np.random.default_rng(11), H, QM, M, W)[None]
    pads = dict(q_padding=(0, QM * g - N), kv_padding=(0, M * kvb - N))
    want = None
    for width in (W, W + 1, -(-W // 4) * 4, -(-W // 4) * 4 + 4):
        wider = np.full((1, H, QM, width), -1, np.int32)
        wider[..., width - W if width == W + 1 else 0:][..., :W] = lists
        got = _grads(ftk, t, wider, H, g, kvb, **pads)
        if want is None:
            want = got
        for a, b in zip(got, want):
            assert torch.equal(a, b), width


@pytest.mark.parametrize("D,W", [(64, 16), (128, 16), (128, 3), (256, 16)])
def test_rows_that_do_not_exist(ftk, D, W):
    """Tiles with rows before the first and behind the last token, and with keys that are
    infinite and listed by nobody: the rows that are listed come out as they do alone."""
    H, N, g = 2, 960, 64
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype="bf16", seed=73, do_seed=74))
    M = N // g
    lists = _lists(np.random.default_rng(12), H, M, M, min(W, M))[None]
    want = _grads(ftk, t, lists, H, g, g)
    # the same problem behind four blocks (so that the same blocks share a tile) of 40 virtual
    # and 216 real rows, and before one that ends in 24 virtual ones
    pre, post = 4 * g - 40, g - 24
    n2 = pre + N + post
    t2 = {}
    for k, x in t.items():
        y = torch.zeros(1, n2, H * D, dtype=x.dtype)
        y[:, pre:pre + N] = x
        if k == "k":
            y[:, :pre] = float("inf")
        t2[k] = y
    wider = np.full((1, H, M + 5, lists.shape[-1]), -1, np.int32)
    wider[:, :, 4:M + 4] = np.where(lists >= 0, lists + 4, -1)
    got = _grads(ftk, t2, wider, H, g, g, q_padding=(40, 24), kv_padding=(40, 24))
    for i in (0, 2, 3, 4):
        assert torch.equal(got[i][:, pre:pre + N], want[i])
        assert not got[i][:, :pre].any() and not got[i][:, pre + N:].any()
    assert torch.equal(got[1][..., pre:pre + N], want[1])


@pytest.mark.parametrize("H,g,kvb,groups", [(16, 64, 64, 1), (16, 32, 32, 2)])
def test_dkv_pair_order(ftk, monkeypatch, H, g, kvb, groups):
    """Short lists at head dim 256: the tiles of the pairs of SMs are sorted by the work they
    have, the heaviest of all slices first, which changes when a tile runs and nothing else."""
    B, N, D = 2, 2600, 256
    tail_q, tail_k = -N % g, -N % kvb
    t = cases.make_inputs(dict(B=B, N=N, H=H, D=D, dtype="bf16", seed=8, do_seed=9))
    Hkv = H // groups
    for n in "kv":
        t[n] = t[n].view(B, N, H, D)[:, :, :Hkv].reshape(B, N, Hkv * D).clone()
    QM, M = (N + tail_q) // g, (N + tail_k) // kvb
    merged = _lists(np.random.default_rng(4), B * H, QM, M, 6).reshape(B, H, QM, 6)
    merged[..., 0] = np.where((merged == 1).any(-1), merged[..., 0], 1)   # a block that everybody reads
    kw = dict(q_padding=(0, tail_q), kv_padding=(0, tail_k), num_kv_heads=Hkv)
    sorted_ = _grads(ftk, t, merged, H, g, kvb, **kw)
    monkeypatch.setenv("FTK_DKV_ORDER", "0")
    plain = _grads(ftk, t, merged, H, g, kvb, **kw)
    for a, b in zip(sorted_, plain):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("D,g,kvb,N,W", [
    (64, 64, 64, 2000, 8),       # two tiles in flight
    (64, 32, 64, 1000, 6),       # four
    (128, 64, 64, 4200, 9),
    (128, 32, 32, 2100, 11),     # tiles of two listed blocks
    (128, 64, 64, 1000, 12),     # pairs of SMs
    (256, 64, 64, 1000, 5),
])
def test_order_of_a_list(ftk, dtype, D, g, kvb, N, W):
    """A list names a set of blocks: written backwards, or with entries that are left out
    ahead of it, it gives the same results bit for bit."""
    H = 2
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype=dtype, seed=75, do_seed=76))
    t["q"] *= 2.0                # rows whose blocks are far apart in score
    QM, M = -(-N // g), -(-N // kvb)
    lists = _lists(np.random.default_rng(13), H, QM, M, W)[None]
    pads = dict(q_padding=(0, QM * g - N), kv_padding=(0, M * kvb - N))
    want = _grads(ftk, t, lists, H, g, kvb, **pads)
    late = np.concatenate([np.full((1, H, QM, 4), -1, np.int32), lists], -1)
    for other in (lists[..., ::-1].copy(), late):
        for a, b in zip(_grads(ftk, t, other, H, g, kvb, **pads), want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("D,W", [(64, 8), (128, 3), (128, 8), (256, 8)])
@pytest.mark.parametrize("x", [14.9, 15.5, 16.5])
def test_fp16_rows_near_the_bound(ftk, monkeypatch, D, W, x):
    """One key of a block leads the rows' reference by 2^x.  Sums of a tile up to 2^15 are the
    pipelined kernel's, those above come out as the exact kernel gives them, bit for bit."""
    N, g = 512, 64
    M = N // g
    gen = torch.Generator().manual_seed(5)
    q, k = torch.zeros(1, N, D), torch.zeros(1, N, D)
    q[..., 0] = 8.0
    k[:, 5 * g + 7, 0] = x / (8.0 * D ** -0.5 * 1.4426950408889634)
    v = torch.randn(1, N, D, generator=gen)
    merged = np.full((1, 1, M, W), -1, np.int32)
    merged[0, 0, :, :3] = [0, 2, 5]
    if W == M:
        merged[0, 0] = np.arange(M)
    args = (q.half().cuda(), k.half().cuda(), v.half().cuda(), torch.from_numpy(merged).cuda(), None, 1,
            g, g)
    o, lse = ftk.flash_topk_attn(*args)
    monkeypatch.setenv("FTK_FWD_PIPE", "0")
    o2, lse2 = ftk.flash_topk_attn(*args)
    ftk.check_errors()
    if x < 15.0:
        # P up to 2^15 and O are rounded to fp16 (2^-11 relative) in both kernels, O is below 4
        assert (o.float() - o2.float()).abs().max().item() <= 4 * 4 * 2.0 ** -11
        torch.testing.assert_close(lse, lse2, rtol=1e-6, atol=1e-6)
    else:
        assert torch.equal(o, o2) and torch.equal(lse, lse2)


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("side", ["first", "last"])
def test_partial_score_tiles_add_up_in_order(ftk, D, side):
    """Key tiles that are not all there (the first one behind a pad head, the last one) add up
    a block's exponentials column by column: fifteen of 2^-24.3 behind a 1 vanish one after the
    other, since each is below half of the last place of 1, and 1 it stays."""
    bsz = 64
    pad, N = ((16, 0), 240) if side == "first" else ((0, 48), 208)
    start = 48 if side == "first" else 128   # first key of a whole block in the partial tile
    lone = 117 if side == "first" else 5     # a key of a block in a tile that is all there
    unit = 8.0 * D ** -0.5 * 1.4426950408889634
    q, k = torch.zeros(1, N, D), torch.zeros(1, N, D)
    q[..., 0] = 8.0
    k[..., 0] = -500.0 / unit                # 2^-500: nothing
    k[:, start + 1:start + 16, 0] = -24.3 / unit
    k[:, [start, lone], 0] = 0.0
    got = ftk.flash_block_score(q.half().cuda(), k.half().cuda(), 1, bsz, pad)
    ftk.check_errors()
    a, b = got[..., (start + pad[0]) // bsz], got[..., (lone + pad[0]) // bsz]
    assert torch.equal(a, b) and (a == 0.5).all()


def _coherent_lists(rng, M, QM, W, kind):
    """One slice's lists of W blocks: a window around the row, aligned runs of blocks, few blocks at random
    (each several times)."""
    out = np.empty((QM, W), np.int32)
    for m in range(QM):
        if kind == "window":
            first = min(max(m * M // QM - W // 2, 0), M - W)
            out[m] = np.arange(first, first + W)
        elif kind == "runs":
            out[m] = (rng.permutation(M // 8)[:W // 8, None] * 8 + np.arange(8)).reshape(-1)
        else:
            out[m] = np.resize(rng.permutation(M)[:W // 4], W)
    return out


@pytest.mark.parametrize("N,W,H,Hkv", [
    (6300, 40, 16, 16), (8192, 32, 12, 12),      # widest and narrowest of the lists that do
    (6300, 40, 16, 4),                           # one result per head, added up after both kernels
    (6300, 40, 4, 2), (4096, 16, 16, 16)])       # none: one wave and a half; fan-in 16
def test_lists_choose_the_dkv_kernel(ftk, monkeypatch, N, W, H, Hkv):
    """Lists of a quarter to a half of the blocks, blocks of many readers: slice by slice the
    pairs of SMs do dK / dV where four kv blocks are listed by few more q-blocks than two (their
    unions together below 1.2 of those), the one-CTA kernel the rest; the results are those of
    the latter alone."""
    import ctypes as C
    from flash_topk_attn_v2 import _lib
    g = kvb = 64
    D, QM = 128, -(-N // g)
    M = QM
    assert M <= 4 * W and 2 * W < M
    chosen = W >= 32 and H > 4
    rng = np.random.default_rng(21)
    kinds = ["window", "few", "runs", "few"] * (H // 4)
    lists = np.stack([_coherent_lists(rng, M, QM, W, k) for k in kinds])[None]
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype="bf16", seed=77, do_seed=78))
    for n in "kv":
        t[n] = t[n][..., :Hkv * D].contiguous()
    pads = dict(q_padding=(0, QM * g - N), kv_padding=(0, M * kvb - N), num_kv_heads=Hkv)
    lib = _lib.lib
    before = lib.ftk_launch_count()
    got = _grads(ftk, t, lists, H, g, kvb, **pads)
    launches = lib.ftk_launch_count() - before
    monkeypatch.setenv("FTK_DKV_2CTA", "0")
    before = lib.ftk_launch_count()
    want = _grads(ftk, t, lists, H, g, kvb, **pads)
    assert launches == lib.ftk_launch_count() - before + chosen
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    if not chosen or Hkv < H:
        return
    monkeypatch.delenv("FTK_DKV_2CTA")

    class Attn(C.Structure):
        _fields_ = ([(n, C.c_void_p) for n in "qkv"] + [("dtype", C.c_int), ("out_f32", C.c_int)]
                    + [(n, C.c_int64) for n in ("B", "H", "Hkv", "N", "D")]
                    + [(f"s{x}_{y}", C.c_int64) for x in "qkv" for y in "bnh"]
                    + [("lists", C.c_void_p)]
                    + [(n, C.c_int) for n in ("list_rows", "W", "q_block", "kv_block", "q_pad_head",
                                              "kv_pad_head")] + [("scale", C.c_float)])

    x = {n: y.cuda() for n, y in t.items()}
    dev_lists = torch.from_numpy(lists).cuda()
    s = (N * H * D, H * D, D)
    a = Attn(*(x[n].data_ptr() for n in "qkv"), _lib.dtype_code(x["q"]), 0, 1, H, H, N, D, *s, *s, *s,
             dev_lists.data_ptr(), QM, W, g, kvb, 0, 0, D ** -0.5)
    size = lib.ftk_attn_bwd_workspace(C.byref(a))
    ws = torch.zeros(size, dtype=torch.uint8, device="cuda")
    dq, dk, dv = (torch.empty_like(x["q"]) for _ in range(3))
    o, lse = got[0], got[1]
    assert lib.ftk_attn_bwd_dq(C.byref(a), o.data_ptr(), *s, x["do"].data_ptr(), *s, lse.data_ptr(),
                               ws.data_ptr(), size, dq.data_ptr(), *s, 0, 0) == 0
    assert lib.ftk_attn_bwd_dkv(C.byref(a), x["do"].data_ptr(), *s, lse.data_ptr(), ws.data_ptr(), size,
                                dk.data_ptr(), *s, dv.data_ptr(), *s, 0, 0) == 0
    torch.cuda.synchronize()
    for y, z in zip((dq, dk, dv), got[2:]):
        assert torch.equal(y, z)
    pick = ws[-256:].view(torch.int32)[:H].tolist()       # the last thing in the workspace
    per = 128 // kvb
    for h in range(H):
        on = np.zeros((QM, -(-M // (2 * per)) * 2 * per), bool)
        np.put_along_axis(on, lists[0, h], True, 1)
        single = on.reshape(QM, -1, per).any(-1).sum()
        pairs = on.reshape(QM, -1, 2 * per).any(-1).sum()
        assert pick[h] == (10 * pairs < 6 * single), (h, kinds[h], pairs / single)
    assert 0 < sum(pick) < H


@pytest.mark.parametrize("D,dtype", [(80, "fp16"), (96, "bf16"), (112, "fp16")])
def test_head_dims_below_128_where_lists_choose_pairs(ftk, monkeypatch, D, dtype):
    """Slices whose lists are windows have their dK / dV done by pairs of SMs, also with a head dim
    that is padded: the bits of the one-CTA kernel."""
    N, W, H, g = 6300, 40, 12, 64
    QM = M = -(-N // g)
    rng = np.random.default_rng(22)
    lists = np.stack([_coherent_lists(rng, M, QM, W, k) for k in ("window", "few", "runs", "window") * (H // 4)])[None]
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype=dtype, seed=81, do_seed=82))
    pads = dict(q_padding=(0, QM * g - N), kv_padding=(0, M * g - N))
    before = ftk._lib.lib.ftk_launch_count()
    got = _grads(ftk, t, lists, H, g, g, **pads)
    launches = ftk._lib.lib.ftk_launch_count() - before
    monkeypatch.setenv("FTK_DKV_2CTA", "0")
    before = ftk._lib.lib.ftk_launch_count()
    want = _grads(ftk, t, lists, H, g, g, **pads)
    assert launches == ftk._lib.lib.ftk_launch_count() - before + 1
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("N,H,W,groups", [
    (8192, 4, 4, 1), (8192, 4, 16, 1), (8192, 4, 64, 2), (8192, 8, 128, 2),   # two waves of pairs
    (2048, 8, 32, 2), (1024, 32, 16, 1),                                     # one wave; short lists
])
def test_dq_goes_by_the_faster_kernel(ftk, N, H, W, groups):
    """Head dim 64: two CTAs of one group per SM or one of two, whichever was measured to be
    the faster in these passes (by 1 to 20 %; the two give the same results)."""
    from torch.profiler import ProfilerActivity, profile
    M = N // 64
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=64, dtype="bf16", seed=79, do_seed=80))
    lists = np.stack([_coherent_lists(np.random.default_rng(h), M, M, W, "window") for h in range(H)])[None]
    q, k, v = (t[n].cuda().requires_grad_(True) for n in "qkv")
    o, _ = ftk.flash_topk_attn(q, k, v, torch.from_numpy(lists).cuda(), None, H, 64, 64)
    do = t["do"].cuda()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        torch.autograd.grad(o, (q, k, v), do)
        torch.cuda.synchronize()
    names = [e.key for e in prof.key_averages() if "sparse_bwd_dq_kernel" in e.key]
    assert len(names) == 1 and f"sparse_bwd_dq_kernel<64, {groups}>" in names[0], names


@pytest.mark.parametrize("bsz", [16, 48, 64, 80, 128, 192])
@pytest.mark.parametrize("D", [64, 128, 256])
def test_score_blocks_end_on_and_off_the_64_column_grid(ftk, D, bsz):
    """Full key tiles are asked for the end of a score block every 16 columns, or every 64 where
    the block size is a multiple of that.  Bound: sums of up to 192 exponentials of 2 ulp whose
    arguments, below 16, are rounded at 2^-21, and a row total of the same."""
    N = 1152   # six blocks of 192, whole key tiles at the other sizes that divide 128
    gen = torch.Generator().manual_seed(bsz + D)
    q, k = (torch.randn(1, N, D, generator=gen).bfloat16() for _ in range(2))
    pad = (0, -N % bsz)
    want = orc.block_score(q.float().numpy(), k.float().numpy(), 1, bsz, pad)
    got = ftk.flash_block_score(q.cuda(), k.cuda(), 1, bsz, pad).cpu().numpy()
    ftk.check_errors()
    np.testing.assert_allclose(got, want, rtol=5e-6, atol=0)


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("hot", [False, True])
def test_score_tiles_of_the_last_wave(ftk, D, hot):
    """192 tiles of 256 rows: those behind the last full wave of 148 SMs are split over clusters
    in a launch of their own (a launch more than one head at a time, a grid of 16 tiles), also
    where rows overflow there and the keys are walked again.  Same bits as one head at a time."""
    from flash_topk_attn_v2 import ops
    H, N, bsz = 12, 4096, 64
    gen = torch.Generator().manual_seed(D)
    q, k = (torch.randn(1, N, H, D, generator=gen).half() for _ in range(2))
    if hot:
        k[:, 300:, 10:] *= 40.0
        q[:, 1800:, 10:] *= 3.0
    q, k = q.cuda(), k.cuda()
    before = ops.launch_count()
    got = ftk.flash_block_score(q.view(1, N, H * D), k.view(1, N, H * D), H, bsz, (0, 0))
    launches = ops.launch_count() - before
    for h in range(H):
        before = ops.launch_count()
        one = ftk.flash_block_score(q[:, :, h].contiguous(), k[:, :, h].contiguous(), 1, bsz, (0, 0))
        assert ops.launch_count() - before == launches - 1
        assert torch.equal(got[:, h], one[:, 0])
    ftk.check_errors()


@pytest.mark.parametrize("D", [64, 128, 256])
def test_select_behind_two_scoring_launches(ftk, D):
    """Scoring in two launches, select overlapped behind them: several calls in a row, whose
    scratch is the same memory, and the same calls replayed from a graph, give what one head
    at a time does."""
    from flash_topk_attn_v2 import ops
    H, N, bsz, topk = 12, 4096, 64, 8
    gen = torch.Generator(device="cuda").manual_seed(D)
    sets = [[torch.randn(1, N, H, D, generator=gen, device="cuda").bfloat16() for _ in range(2)]
            for _ in range(3)]

    def calls():
        return [ftk.flash_topk_score(q.view(1, N, H * D), k.view(1, N, H * D), H, bsz, topk, (0, 0), 0.9)
                for q, k in sets]

    want = [[torch.cat(x, 1) for x in zip(*(
        ftk.flash_topk_score(q[:, :, h].contiguous(), k[:, :, h].contiguous(), 1, bsz, topk, (0, 0), 0.9)
        for h in range(H)))] for q, k in sets]
    before = ops.launch_count()
    eager = [calls() for _ in range(4)]
    assert ops.launch_count() - before == 4 * len(sets) * 3
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        calls()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        replayed = calls()
    for x in replayed:
        for y in x:
            y.zero_()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    ftk.check_errors()
    for got in eager + [replayed]:
        for a, b in zip(got, want):
            for x, y in zip(a, b):
                assert torch.equal(x, y)


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("D", [80, 96, 112])
def test_head_dims_below_128_on_pairs(ftk, D, dtype):
    """Wide lists: the backward's pair kernels leave out the k-steps and columns that are
    padding of the head dim.  Same bits as with the padding written out as zeros."""
    H, N, g = 3, 700, 64
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype=dtype, seed=D, do_seed=D + 1))
    M = -(-N // g)
    lists = np.tile(np.arange(M, dtype=np.int32), (1, H, M, 1))
    lists[0, 1, 3:, 2:] = -1
    pads = dict(q_padding=(0, M * g - N), kv_padding=(0, M * g - N), scale=D ** -0.5)
    got = _grads(ftk, t, lists, H, g, g, **pads)
    wide = {k: torch.nn.functional.pad(x.view(1, N, H, D), (0, 128 - D)).reshape(1, N, H * 128)
            for k, x in t.items()}
    want = _grads(ftk, wide, lists, H, g, g, **pads)
    assert torch.equal(got[1], want[1])
    for i in (0, 2, 3, 4):
        assert torch.equal(got[i].view(1, N, H, D), want[i].view(1, N, H, 128)[..., :D])


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("D", [72, 88, 104, 120])
def test_odd_multiples_of_8_on_pairs(ftk, D, dtype):
    """The C interface takes head dims that are multiples of 8, of which the Python layer refuses
    the odd ones: on the pair kernels as well, the same bits as with the padding written out as zeros
    and nothing is stored from column D on (the results' rows are wider, to see that)."""
    import ctypes as C
    from flash_topk_attn_v2 import _lib
    from test_c_abi_cpu import _Attn
    lib, H, N, g = _lib.lib, 3, 700, 64
    M = -(-N // g)
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype=dtype, seed=D, do_seed=D + 1))
    lists = np.tile(np.arange(M, dtype=np.int32), (1, H, M, 1))
    lists[0, 1, 3:, 2:] = -1
    lists = torch.from_numpy(lists).cuda()

    def attend(d):
        x = {n: torch.nn.functional.pad(y.view(N, H, D), (0, d - D)).cuda() for n, y in t.items()}
        s = (N * H * d, H * d, d)
        a = _Attn(*(x[n].data_ptr() for n in "qkv"), _lib.dtype_code(x["q"]), 0, 1, H, H, N, d, *s, *s, *s,
                  lists.data_ptr(), M, M, g, g, 0, 0, D ** -0.5)
        a = C.byref(a)
        size = max(lib.ftk_attn_fwd_workspace(a), lib.ftk_attn_bwd_workspace(a))
        ws = torch.zeros(size, dtype=torch.uint8, device="cuda")
        o, dq, dk, dv = (torch.full((N, H, d + 8), 7.0, dtype=x["q"].dtype, device="cuda") for _ in range(4))
        so = (N * H * (d + 8), H * (d + 8), d + 8)
        lse = torch.empty(H, N, device="cuda")
        assert lib.ftk_attn_fwd(a, o.data_ptr(), *so, lse.data_ptr(), ws.data_ptr(), size, 0, 0) == 0
        ws.zero_()
        assert lib.ftk_attn_bwd_dq(a, o.data_ptr(), *so, x["do"].data_ptr(), *s, lse.data_ptr(),
                                   ws.data_ptr(), size, dq.data_ptr(), *so, 0, 0) == 0
        assert lib.ftk_attn_bwd_dkv(a, x["do"].data_ptr(), *s, lse.data_ptr(), ws.data_ptr(), size,
                                    dk.data_ptr(), *so, dv.data_ptr(), *so, 0, 0) == 0
        torch.cuda.synchronize()
        return lse, o, dq, dk, dv

    got, want = attend(D), attend(128)
    assert torch.equal(got[0], want[0])
    for x, y in zip(got[1:], want[1:]):
        assert torch.equal(x[..., :D], y[..., :D])
        assert (x[..., D:] == 7.0).all()
        assert torch.isfinite(x).all() and x[..., :D].any()


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("at", [64 + 0, 64 + 1, 64 + 2, 64 + 9])
@pytest.mark.parametrize("what", [float("nan"), float("inf"), 3.0e4])
def test_forward_values_that_are_no_probabilities(ftk, monkeypatch, dtype, at, what):
    """A key of NaN or infinities, or one that overflows, sends its tile to the exact kernel
    whichever column it stands in; the rows whose logit of it is as far below are as if it was
    not there.  Bound of the latter: two roundings of P and of O."""
    H, N, D, g = 2, 512, 64, 64
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype=dtype, seed=91, do_seed=92))
    t["q"].view(1, N, H, D)[..., 0] = 1.0
    t["q"].view(1, N, H, D)[:, 300:, :, 0] = -1.0   # rows 300 on: -inf, or far below
    key = t["k"].view(1, N, H, D)[:, at]
    key.zero_()
    key[..., 0] = what
    merged = np.tile(np.arange(N // g, dtype=np.int32), (1, H, N // g, 1))
    args = [t[n].cuda() for n in "qkv"] + [torch.from_numpy(merged).cuda(), None, H, g, g]
    o, lse = ftk.flash_topk_attn(*args)
    monkeypatch.setenv("FTK_FWD_PIPE", "0")
    want, lse_want = ftk.flash_topk_attn(*args)
    ftk.check_errors()
    rows = slice(None, 256)   # the tiles of these rows all overflow
    for x, y in ((o[:, rows], want[:, rows]), (lse[..., rows], lse_want[..., rows])):
        assert torch.equal(torch.isnan(x), torch.isnan(y))
        assert torch.equal(torch.nan_to_num(x), torch.nan_to_num(y))
    eps = 2.0 ** -10 if dtype == "fp16" else 2.0 ** -7
    if what == 3.0e4:
        assert torch.isfinite(o[:, 384:]).all()
        bound = 2 * eps * want[:, 384:].abs().float() + 2 * eps
        assert ((o[:, 384:].float() - want[:, 384:].float()).abs() <= bound).all()


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("D,g,W", [(32, 64, 8), (64, 64, 8), (64, 64, 3), (64, 32, 16), (128, 64, 3),
                                   (128, 64, 8), (256, 64, 8)])
def test_rows_without_a_finite_logit(ftk, monkeypatch, dtype, D, g, W):
    """Query rows whose logits are all -inf (full tiles, and the last one, which is not): O = 0
    and lse = -inf, as from the exact kernel.  The rows beside them are not touched by that.
    Bound of those: P and O, below 4, are rounded in both kernels, at different references."""
    H, N = 2, 500
    M = -(-N // g)
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype=dtype, seed=93, do_seed=94))
    t["k"].view(1, N, H, D)[..., 0] = 1.0
    gone = torch.zeros(N, dtype=torch.bool)
    gone[[0, 7, 63, 200, 499]] = True
    gone[64:128] = True
    t["q"].view(1, N, H, D)[:, gone, :, 0] = -float("inf")
    lists = np.full((1, H, M, W), -1, np.int32)
    for m in range(M):
        lists[:, :, m] = np.sort((np.arange(W) + m) % M)
    pads = dict(q_padding=(0, M * g - N), kv_padding=(0, M * g - N))
    args = [t[n].cuda() for n in "qkv"] + [torch.from_numpy(lists).cuda(), None, H, g, g]
    o, lse = ftk.flash_topk_attn(*args, **pads)
    monkeypatch.setenv("FTK_FWD_PIPE", "0")
    o2, lse2 = ftk.flash_topk_attn(*args, **pads)
    ftk.check_errors()
    gone = gone.cuda()
    for x, y in ((o, lse), (o2, lse2)):
        assert not x[:, gone].any()
        assert (y[..., gone] == -float("inf")).all()
    eps = 2.0 ** -10 if dtype == "fp16" else 2.0 ** -7
    assert torch.isfinite(o[:, ~gone]).all()
    assert (o - o2)[:, ~gone].abs().max().item() <= 4 * 2 * eps
    torch.testing.assert_close(lse[..., ~gone], lse2[..., ~gone], rtol=1e-6, atol=1e-6)


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("pipe", [True, False])
@pytest.mark.parametrize("D,g,W", [(64, 64, 8), (64, 32, 16), (128, 64, 3), (128, 64, 8), (256, 64, 8),
                                   (64, 48, 4), (128, 128, 3)])
@pytest.mark.parametrize("level", [0.0, -30.0, -110.0])
def test_tiles_of_minus_infinity_before_finite_ones(ftk, monkeypatch, dtype, pipe, D, g, W, level):
    """All blocks but the last give logits of -inf, so a row's first tile, and the one that its
    reference is taken from, say nothing about the last one's logits, which lie around `level`.
    Bound: P and O, below 4, are rounded to 16 bits; a logit is a sum of D float32 products."""
    H, N = 2, 480 if g == 48 else 512
    M = N // g
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype=dtype, seed=95, do_seed=96))
    t["q"].view(1, N, H, D)[..., 0] = 8.0
    t["k"].view(1, N, H, D)[:, :-g, :, 0] = -float("inf")
    t["k"].view(1, N, H, D)[:, -g:, :, 0] = level * D ** 0.5 / 8.0
    lists = np.full((1, H, M, W), -1, np.int32)
    for m in range(M):
        lists[:, :, m] = np.append((np.arange(W - 1) + m) % (M - 1), M - 1)
    if not pipe:
        monkeypatch.setenv("FTK_FWD_PIPE", "0")
    o, lse = ftk.flash_topk_attn(*(t[n].cuda() for n in "qkv"), torch.from_numpy(lists).cuda(), None, H, g, g)
    ftk.check_errors()
    q, k, v = (t[n].view(N, H, D).transpose(0, 1).double() for n in "qkv")
    logits = q @ k[:, -g:].transpose(1, 2) * D ** -0.5
    want = (logits.softmax(-1) @ v[:, -g:]).transpose(0, 1).reshape(1, N, H * D)
    eps = 2.0 ** -10 if dtype == "fp16" else 2.0 ** -7
    assert (o.cpu().double() - want).abs().max().item() <= 4 * 2 * eps
    assert (lse[0].cpu().double() - logits.logsumexp(-1)).abs().max().item() <= D * 2.0 ** -24 * (8 - level)
