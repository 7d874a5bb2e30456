"""The kernels that work on pairs of SMs at head dim 128 with 64-row q-blocks.

The forward takes them for more than 96 tiles of 64 keys and lists that can name three quarters of
the blocks, dQ for such lists at any length.  Every test here also looks which kernel ran, so
that a line that moves does not leave it with another one."""

import numpy as np
import pytest
import torch

import cases
import tolerance
from oracle import ftk_oracle as orc

pytestmark = pytest.mark.gpu

G = 64
FORWARD, DQ = "sparse_fwd_pipe2_kernel", "sparse_bwd_dq2_kernel"


@pytest.fixture(scope="module")
def ftk():
    import flash_topk_attn_v2 as m
    return m


def _kernels(call):
    """Names of the kernels that the call launches, from a graph that it is captured into."""
    from cuda.bindings import driver

    def ok(result):
        assert result[0] == driver.CUresult.CUDA_SUCCESS, result[0]
        return result[1:] if len(result) > 2 else result[1]
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        call()
    stream.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        call()
    handle = driver.CUgraph(graph.raw_cuda_graph())
    nodes, count = ok(driver.cuGraphGetNodes(handle, 0))
    nodes, count = ok(driver.cuGraphGetNodes(handle, count))
    names = []
    for node in nodes:
        if ok(driver.cuGraphNodeGetType(node)) == driver.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            params = ok(driver.cuGraphKernelNodeGetParams(node))
            name = ok(driver.cuFuncGetName(params.func)) if int(params.func) else ok(driver.cuKernelGetName(params.kern))
            names.append(name.decode())
    return names


def _run(kernel, call, there=True):
    """The call's result; `kernel` is among the ones that it launches, or is not."""
    names = _kernels(call)
    assert any("sparse_" in n for n in names)
    assert any(kernel in n for n in names) == there, names
    return call()


def _lists(rng, H, QM, M, W):
    """Random lists; of every four q-blocks that a pair of SMs takes all, one, two or three are empty
    here and there."""
    out = np.full((1, H, QM, W), -1, dtype=np.int32)
    for h in range(H):
        for m in range(QM):
            if (m // 4) % 6 == 5 or ((m // 4) % 6 == 3 and m % 4 != 1 + h % 2):
                continue
            n = W if m % 7 == 0 else int(rng.integers(1, W + 1))
            out[0, h, m, :n] = rng.permutation(M)[:n]
    return out


def _attend(ftk, t, lists, H, **kw):
    args = [t[n].cuda() for n in "qkv"] + [torch.from_numpy(lists).cuda(), None, H, G, G]
    return lambda: ftk.flash_topk_attn(*args, **kw)


def _grads(ftk, t, lists, H, **kw):
    q, k, v = (t[n].cuda().requires_grad_(True) for n in "qkv")
    do, lists = t["do"].cuda(), torch.from_numpy(lists).cuda()

    def call():
        o, lse = ftk.flash_topk_attn(q, k, v, lists, None, H, G, G, **kw)
        return (o.detach(), lse) + torch.autograd.grad(o, (q, k, v), do)
    return call


@pytest.mark.parametrize("D,dtype", [(128, "fp16"), (128, "bf16"), (96, "fp16")])
def test_forward(ftk, monkeypatch, D, dtype):
    """Ragged length, virtual rows at either end, empty lists beside others, against float64 (fp16: the
    plain bound) and against one CTA per tile and the exact kernel.  Bound between kernels:
    P and O, below 6, are rounded in both, at other references."""
    H, N, W = 2, 6420, 80
    qpad, kvpad = (24, 20), (20, 24)
    QM = M = 101
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype=dtype, seed=41, do_seed=42))
    lists = _lists(np.random.default_rng(3), H, QM, M, W)
    call = _attend(ftk, t, lists, H, kv_padding=kvpad, q_padding=qpad)
    o, lse = _run(FORWARD, call)
    if dtype == "fp16":
        x = {n: v.float().numpy() for n, v in t.items()}
        wo, wl = orc.sparse_attn_fwd(x["q"], x["k"], x["v"], lists, H, G, G, None, qpad, kvpad)
        assert (tolerance.rel_err(o.float().cpu().numpy(), wo) <= 1).all()
        np.testing.assert_allclose(lse.cpu().numpy(), wl, atol=2e-3, rtol=1e-2)
    eps = 2.0 ** -10 if dtype == "fp16" else 2.0 ** -7
    for name in ("FTK_FWD_2CTA", "FTK_FWD_PIPE"):
        monkeypatch.setenv(name, "0")
        o2, lse2 = _run(FORWARD, call, there=False)
        assert (o.float() - o2.float()).abs().max().item() <= 6 * 2 * eps
        torch.testing.assert_close(lse, lse2, rtol=1e-5, atol=1e-5)
        assert torch.equal(lse == -float("inf"), lse2 == -float("inf"))
    ftk.check_errors()


@pytest.mark.parametrize("x", [14.9, 15.5, 16.5])
def test_fp16_rows_near_the_bound(ftk, monkeypatch, x):
    """One key of a block leads the rows' reference by 2^x: sums of a tile up to 2^15 are the pair
    kernel's, those above come out as the exact kernel gives them, bit for bit."""
    M, D = 97, 128
    N = M * G
    gen = torch.Generator().manual_seed(5)
    q, k = torch.zeros(1, N, D), torch.zeros(1, N, D)
    q[..., 0] = 8.0
    k[:, 5 * G + 7, 0] = x / (8.0 * D ** -0.5 * 1.4426950408889634)
    t = dict(q=q.half(), k=k.half(), v=torch.randn(1, N, D, generator=gen).half())
    call = _attend(ftk, t, np.tile(np.arange(M, dtype=np.int32), (1, 1, M, 1)), 1)
    o, lse = _run(FORWARD, call)
    monkeypatch.setenv("FTK_FWD_PIPE", "0")
    o2, lse2 = call()
    ftk.check_errors()
    if x < 15.0:
        # P up to 2^15 and O are rounded to fp16 (2^-11 relative) in both kernels, O is below 4
        assert (o.float() - o2.float()).abs().max().item() <= 4 * 4 * 2.0 ** -11
        torch.testing.assert_close(lse, lse2, rtol=1e-6, atol=1e-6)
    else:
        assert torch.equal(o, o2) and torch.equal(lse, lse2)


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
def test_rows_without_a_finite_logit(ftk, monkeypatch, dtype):
    """Query rows whose logits are all -inf: O = 0 and lse = -inf, and the rows beside them are not
    touched by that.  Bound of those: P and O, below 4, are rounded in both kernels."""
    H, N, D, W = 2, 6420, 128, 80
    M = -(-N // G)
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype=dtype, seed=93, do_seed=94))
    t["k"].view(1, N, H, D)[..., 0] = 1.0
    gone = torch.zeros(N, dtype=torch.bool)
    gone[[0, 7, 63, 200, 499, 3000, 6419]] = True
    gone[64:128] = True
    gone[1024:1280] = True
    t["q"].view(1, N, H, D)[:, gone, :, 0] = -float("inf")
    lists = np.stack([np.sort((np.arange(W) + m) % M) for m in range(M)]).astype(np.int32)
    call = _attend(ftk, t, np.tile(lists, (1, H, 1, 1)), H, q_padding=(0, -N % G), kv_padding=(0, -N % G))
    o, lse = _run(FORWARD, call)
    monkeypatch.setenv("FTK_FWD_PIPE", "0")
    o2, lse2 = call()
    ftk.check_errors()
    gone = gone.cuda()
    for x, y in ((o, lse), (o2, lse2)):
        assert not x[:, gone].any()
        assert (y[..., gone] == -float("inf")).all()
    eps = 2.0 ** -10 if dtype == "fp16" else 2.0 ** -7
    assert torch.isfinite(o[:, ~gone]).all()
    assert (o.float() - o2.float())[:, ~gone].abs().max().item() <= 4 * 2 * eps
    torch.testing.assert_close(lse[..., ~gone], lse2[..., ~gone], rtol=1e-6, atol=1e-6)


def test_marked_tiles(ftk, monkeypatch):
    """Rows of some heads leave the exponent range: their tiles, which are a pair's halves, come out of
    the exact kernel, bit for bit, and no other head's do."""
    H, N, D, W = 24, 6300, 128, 99
    M = -(-N // G)
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype="fp16", seed=25, do_seed=26))
    hot = [0, 7, 23]
    t["q"].view(1, N, H, D)[:, :, hot] *= 2.0
    t["k"].view(1, N, H, D)[:, 64:, hot] *= 8.0
    lists = np.tile(np.arange(M, dtype=np.int32), (1, H, M, 1))
    call = _attend(ftk, t, lists, H, q_padding=(0, -N % G), kv_padding=(0, -N % G))
    o, lse = _run(FORWARD, call)
    monkeypatch.setenv("FTK_FWD_PIPE", "0")
    o2, lse2 = call()
    ftk.check_errors()
    same = (o.view(N, H, D) == o2.view(N, H, D)).all(-1).all(0)
    assert torch.nonzero(same).flatten().tolist() == hot
    assert torch.equal(lse[0, hot], lse2[0, hot])
    # P and O are rounded to fp16 in both kernels, O is below 6
    assert (o.float() - o2.float()).abs().max().item() <= 6 * 2 * 2.0 ** -10


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
def test_order_of_a_list(ftk, dtype):
    """A list written backwards, or with entries that are left out ahead of it, gives the same
    results bit for bit."""
    H, N, D, W = 2, 6300, 128, 80
    M = -(-N // G)
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype=dtype, seed=75, do_seed=76))
    t["q"] *= 2.0
    lists = _lists(np.random.default_rng(13), H, M, M, W)
    pads = dict(q_padding=(0, -N % G), kv_padding=(0, -N % G))
    call = _grads(ftk, t, lists, H, **pads)
    want = _run(FORWARD, call)
    _run(DQ, call)
    late = np.concatenate([np.full((1, H, M, 4), -1, np.int32), lists], -1)
    for other in (lists[..., ::-1].copy(), late):
        for a, b in zip(_grads(ftk, t, other, H, **pads)(), want):
            assert torch.equal(a, b)
    ftk.check_errors()


@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
@pytest.mark.parametrize("D", [80, 96, 112])
def test_padded_head_dims(ftk, D, dtype):
    """Head dims below 128: the bits of the same rows with the padding written out as zeros."""
    H, N = 2, 6200
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=128, dtype=dtype, seed=D, do_seed=D + 1))
    t = {n: x.view(1, N, H, 128)[..., :D].contiguous() for n, x in t.items()}
    M = -(-N // G)
    lists = np.tile(np.arange(M, dtype=np.int32), (1, H, M, 1))
    lists[0, 1, 3:60, 2:] = -1
    pads = dict(q_padding=(0, M * G - N), kv_padding=(0, M * G - N), scale=D ** -0.5)
    flat = lambda x: x.reshape(1, N, -1)
    got = _run(FORWARD, _grads(ftk, {n: flat(x) for n, x in t.items()}, lists, H, **pads))
    wide = {n: flat(torch.nn.functional.pad(x, (0, 128 - D))) for n, x in t.items()}
    want = _run(DQ, _grads(ftk, wide, lists, H, **pads))
    assert torch.equal(got[1], want[1])
    for i in (0, 2, 3, 4):
        assert torch.equal(got[i].view(1, N, H, D), want[i].view(1, N, H, 128)[..., :D])
    ftk.check_errors()


@pytest.mark.parametrize("N,W,dtype", [(1900, 24, "fp16"), (1900, 30, "bf16"), (1000, 12, "fp16")])
def test_dq(ftk, monkeypatch, N, W, dtype):
    """Lists that can name three quarters of the blocks: dQ on pairs of SMs, beside one CTA per tile, whose
    arithmetic per element is the same in another order of the blocks, and (fp16) against float64."""
    H, D = 3, 128
    qpad, kvpad = (24, -(N + 24) % G), (20, -(N + 20) % G)
    QM, M = (sum(qpad) + N) // G, (sum(kvpad) + N) // G
    t = cases.make_inputs(dict(B=1, N=N, H=H, D=D, dtype=dtype, seed=51, do_seed=52))
    lists = _lists(np.random.default_rng(17), H, QM, M, W)
    assert 4 * W >= 3 * M
    call = _grads(ftk, t, lists, H, q_padding=qpad, kv_padding=kvpad)
    got = _run(DQ, call)
    if dtype == "fp16":
        x = {n: v.float().numpy() for n, v in t.items()}
        _, lse = orc.sparse_attn_fwd(x["q"], x["k"], x["v"], lists, H, G, G, None, qpad, kvpad)
        want = orc.sparse_attn_bwd(x["q"], x["k"], x["v"], got[0].float().cpu().numpy(), lse, x["do"], lists, H, G,
                                   G, None, qpad, kvpad)
        for a, w in zip(got[2:], want):
            assert (tolerance.rel_err(a.float().cpu().numpy(), w) <= 1).all()
    monkeypatch.setenv("FTK_DQ_2CTA", "0")
    single = _run(DQ, call, there=False)
    ftk.check_errors()
    for i in (0, 1, 3, 4):
        assert torch.equal(got[i], single[i])
    # sums of the same products, rounded once: next to each other in the result's type
    eps = 2.0 ** -10 if dtype == "fp16" else 2.0 ** -7
    torch.testing.assert_close(got[2].float(), single[2].float(), rtol=eps, atol=eps * got[2].abs().max().item() * 2.0 ** -5)
