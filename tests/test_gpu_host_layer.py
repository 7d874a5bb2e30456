"""The host layer in front of the kernels: layouts of the inputs, the autograd node, the
route of a call."""

import numpy as np
import pytest
import torch

import cases

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ftk():
    import flash_topk_attn_v2 as m
    return m


def _full_lists(B, H, QM, M, seed=0):
    rng = np.random.default_rng(seed)
    lists = np.stack([rng.permutation(M) for _ in range(B * H * QM)]).astype(np.int32)
    return torch.from_numpy(lists.reshape(B, H, QM, M)).cuda()


@pytest.mark.parametrize("dtype,D", [("bf16", 128), ("fp16", 64), ("fp32", 64)])
def test_gradient_of_a_sum_over_tokens(ftk, dtype, D):
    """o.sum(dim=1) hands the node a gradient with stride 0 over the tokens; the same
    numbers laid out give the same bits."""
    B, N, H = 2, 512, 2
    t = cases.make_inputs(dict(B=B, N=N, H=H, D=D, dtype="bf16" if dtype == "fp32" else dtype,
                               seed=71, do_seed=72))
    if dtype == "fp32":
        t = {n: x.float() for n, x in t.items()}
    merged = _full_lists(B, H, N // 64, N // 64)
    w = t["do"][:, 0].cuda()

    def grads(pool):
        q, k, v = (t[n].cuda().requires_grad_(True) for n in "qkv")
        o, _ = ftk.flash_topk_attn(q, k, v, merged, None, H, 64, 64)
        pool(o)
        return q.grad, k.grad, v.grad

    pooled = grads(lambda o: o.sum(dim=1).backward(w))
    dense = grads(lambda o: o.backward(w.unsqueeze(1).expand(B, N, H * D).contiguous()))
    ftk.check_errors()
    for a, b in zip(pooled, dense):
        assert torch.equal(a, b)


def test_expanded_inputs(ftk):
    """One key head for all heads in scoring, one batch entry's keys and values for all in
    the attention: as the same tensors laid out."""
    B, N, H, D = 2, 512, 4, 64
    t = cases.make_inputs(dict(B=B, N=N, H=H, D=D, dtype="bf16", seed=73, do_seed=74))
    q4 = t["q"].cuda().view(B, N, H, D).permute(0, 2, 1, 3)
    k4 = t["k"].cuda().view(B, N, H, D).permute(0, 2, 1, 3)[:, :1].expand(B, H, N, D)
    for a, b in zip(ftk.flash_topk_score(q4, k4, topk=4),
                    ftk.flash_topk_score(q4, k4.contiguous(), topk=4)):
        assert torch.equal(a, b)
    assert torch.equal(ftk.flash_block_score(q4, k4, H, 64),
                       ftk.flash_block_score(q4, k4.contiguous(), H, 64))
    k, v = (t[n].cuda()[:1].expand(B, N, H * D) for n in "kv")
    merged = _full_lists(B, H, N // 64, N // 64)
    for a, b in zip(ftk.flash_topk_attn(t["q"].cuda(), k, v, merged, None, H, 64, 64),
                    ftk.flash_topk_attn(t["q"].cuda(), k.contiguous(), v.contiguous(), merged, None,
                                        H, 64, 64)):
        assert torch.equal(a, b)
    ftk.check_errors()


# ------------------------------------------------------------------ the autograd node
def _problem(dtype="bf16", B=1, N=384, H=4, Hkv=2, D=64):
    t = cases.make_inputs(dict(B=B, N=N, H=H, D=D, dtype="bf16" if dtype == "fp32" else dtype,
                               seed=75, do_seed=76))
    t["k"], t["v"] = (t[n][..., :Hkv * D].contiguous() for n in "kv")
    if dtype == "fp32":
        t = {n: x.float() for n, x in t.items()}
    leaves = [t[n].cuda().requires_grad_(True) for n in "qkv"]
    merged = _full_lists(B, H, N // 64, N // 64, seed=1)[..., :4].contiguous()
    return leaves, merged, t["do"].cuda(), dict(H=H, Hkv=Hkv)


def _attend(ftk, leaves, merged, c):
    return ftk.flash_topk_attn(*leaves, merged, None, c["H"], 64, 64, num_kv_heads=c["Hkv"])[0]


def _expected(ftk, leaves, merged, do, c):
    return torch.autograd.grad(_attend(ftk, leaves, merged, c), leaves, do)


def _same(a, b):
    assert len(a) == len(b) and all(torch.equal(x, y) for x, y in zip(a, b))


def test_backward_twice_with_a_retained_graph(ftk):
    leaves, merged, do, c = _problem()
    want = _expected(ftk, leaves, merged, do, c)
    o = _attend(ftk, leaves, merged, c)
    _same(torch.autograd.grad(o, leaves, do, retain_graph=True), want)
    _same(torch.autograd.grad(o, leaves, do), want)
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad(o, leaves, do)


def test_only_some_inputs_want_a_gradient(ftk):
    leaves, merged, do, c = _problem()
    want = _expected(ftk, leaves, merged, do, c)
    for wanted in ((0,), (1,), (2,), (0, 2)):
        part = [x.detach().requires_grad_(i in wanted) for i, x in enumerate(leaves)]
        o, lse = ftk.flash_topk_attn(*part, merged, None, c["H"], 64, 64, num_kv_heads=c["Hkv"])
        assert o.requires_grad and not lse.requires_grad
        _same(torch.autograd.grad(o, [part[i] for i in wanted], do), [want[i] for i in wanted])


@pytest.mark.parametrize("dtype", ["bf16", "fp32"])
def test_saved_tensor_hooks(ftk, dtype):
    """What the node keeps goes through the hooks: offloaded to the host and back, with no
    copy left on the device, the gradients are the same."""
    leaves, merged, do, c = _problem(dtype)
    want = _expected(ftk, leaves, merged, do, c)
    kept = []

    def pack(x):
        kept.append((tuple(x.shape), x.dtype))
        return x.cpu()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda x: x.cuda()):
        o = _attend(ftk, leaves, merged, c)
    assert len(kept) == 6                      # q, k, v, O, lse, lists
    _same(torch.autograd.grad(o, leaves, do), want)


@pytest.mark.parametrize("reentrant", [False, True])
def test_checkpointing(ftk, reentrant):
    from torch.utils.checkpoint import checkpoint
    leaves, merged, do, c = _problem()
    want = _expected(ftk, leaves, merged, do, c)
    o = checkpoint(lambda q, k, v: _attend(ftk, (q, k, v), merged, c), *leaves,
                   use_reentrant=reentrant)
    o.backward(do)
    _same([x.grad for x in leaves], want)


@pytest.mark.parametrize("which", ["q", "o", "lists"])
def test_a_changed_saved_tensor_is_noticed(ftk, which):
    leaves, merged, do, c = _problem()
    o = _attend(ftk, leaves, merged, c)
    with torch.no_grad():
        {"q": leaves[0], "o": o, "lists": merged}[which].mul_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(o, leaves, do)


def test_backward_from_another_thread_and_stream(ftk):
    """The backward runs on the stream of its forward, whichever thread and stream asks."""
    import threading
    leaves, merged, do, c = _problem()
    want = _expected(ftk, leaves, merged, do, c)
    got, errors = [], []

    def work():
        try:
            side = torch.cuda.Stream()
            side.wait_stream(torch.cuda.default_stream())
            with torch.cuda.stream(side):
                o = _attend(ftk, leaves, merged, c)
                o.record_stream(torch.cuda.default_stream())
            torch.cuda.current_stream().wait_stream(side)
            with torch.cuda.stream(torch.cuda.Stream()):
                torch.cuda.current_stream().wait_stream(side)
                torch.autograd.backward(o, do, inputs=own[len(got)])
                torch.cuda.current_stream().synchronize()
            got.append([x.grad for x in own[len(got)]])
        except Exception as e:                 # noqa: BLE001  (shown below)
            errors.append(e)

    own = []
    for _ in range(2):
        leaves = [x.detach().clone().requires_grad_(True) for x in leaves]
        own.append(leaves)
        torch.cuda.synchronize()
        t = threading.Thread(target=work)
        t.start()
        t.join(60)
        assert not errors, errors
    torch.cuda.synchronize()
    for g in got:
        _same(g, want)


def test_gradients_carry_no_graph(ftk):
    """There is no second derivative: create_graph gives gradients without one."""
    leaves, merged, do, c = _problem()
    want = _expected(ftk, leaves, merged, do, c)
    got = torch.autograd.grad(_attend(ftk, leaves, merged, c), leaves, do, create_graph=True)
    _same(got, want)
    assert not any(g.requires_grad for g in got)


# ------------------------------------------------------------ the two routes of a call
def _forms(seed):
    """Calls of random form, ordinary and odd ones."""
    import random
    rng = random.Random(seed)
    pick = rng.choice
    D, H = pick([16, 48, 64, 96, 128, 160]), pick([1, 2, 4])
    g, block = pick([16, 32, 48, 64, 96, 128]), pick([16, 32, 48, 64, 96, 128])
    N = rng.randrange(200, 600)
    ph, kh = pick([0, rng.randrange(g)]), pick([0, rng.randrange(block)])
    return dict(B=pick([1, 2]), N=N, H=H, Hkv=pick([H, 1]), D=D, g=g, block=block,
                dtype=pick(["fp16", "bf16", "fp32"]), topk=pick([0, 1, 3, 8]),
                threshold=pick([1.0, 0.7]), qpad=(ph, -(ph + N) % g), kpad=(kh, -(kh + N) % block),
                width=pick([None, 1, 5]), four_d=pick([False, True]), scores=pick([True, False]),
                scale=pick([None, 0.25]), grad=pick([True, False]), strided=pick([False, True]))


@pytest.mark.parametrize("seed", range(40))
def test_both_routes_of_a_call_agree(ftk, seed):
    """Ordinary calls pass one check in the native layer; timed calls, and those that this
    check does not take, go through the checks of the operators first.  Either way a call
    gives the same bits, or the same exception."""
    from flash_topk_attn_v2 import ops
    f = _forms(seed)
    B, N, H, Hkv, D = f["B"], f["N"], f["H"], f["Hkv"], f["D"]
    dt = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}[f["dtype"]]
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def rand(*shape):
        wide = (*shape[:-1], shape[-1] + (8 if f["strided"] else 0))
        return torch.randn(wide, generator=gen, device="cuda").to(dt)[..., :shape[-1]]

    qk = [rand(B, H, N, D) for _ in range(2)] if f["four_d"] else [rand(B, N, H * D) for _ in range(2)]
    q, k, v, do = rand(B, N, H * D), rand(B, N, Hkv * D), rand(B, N, Hkv * D), rand(B, N, H * D)

    def chain():
        out = list(ftk.flash_topk_score(*qk, None if f["four_d"] else H, f["block"], f["topk"],
                                        f["kpad"], f["threshold"]))
        merged, counts, width = ftk.build_qblock_topk_indices(
            out[0], f["g"], f["qpad"], out[2] if f["scores"] else None, f["width"])
        leaves = [x.detach().requires_grad_(f["grad"]) for x in (q, k, v)]
        out += [merged, counts, torch.tensor(width)]
        try:
            out += ftk.flash_topk_attn(*leaves, merged, counts, H, f["g"], f["block"], f["scale"],
                                       Hkv, f["kpad"], f["qpad"])
            if f["grad"]:
                out += torch.autograd.grad(out[-2], leaves, do)
        except NotImplementedError as e:
            out.append(str(e))
        return out

    direct = chain()
    ops.enable_event_timing(True)
    try:
        checked = chain()
    finally:
        ops.enable_event_timing(False)
    ftk.check_errors()
    assert len(direct) == len(checked)
    for a, b in zip(direct, checked):
        assert a == b if isinstance(a, str) else torch.equal(a, b)


@pytest.mark.parametrize("D,g,kvb,H,Hkv,N", [
    (128, 64, 64, 2, 2, 512),        # pairs
    (64, 48, 48, 2, 2, 480),         # exact forward alone
    (64, 64, 64, 16, 16, 4736),      # dK/dV tiles sorted first
    (128, 64, 64, 6, 2, 320),        # one result per query head, summed by a kernel of its own
    (256, 64, 64, 2, 2, 512),        # dV and dK in two launches
])
def test_launch_count_is_what_a_capture_holds(ftk, D, g, kvb, H, Hkv, N):
    """Kernel nodes of a captured pass against the library's own count."""
    from cuda.bindings import runtime as rt
    from flash_topk_attn_v2 import ops
    gen = torch.Generator(device="cuda").manual_seed(1)
    q, do = (torch.randn(1, N, H * D, generator=gen, device="cuda").bfloat16() for _ in range(2))
    k, v = (torch.randn(1, N, Hkv * D, generator=gen, device="cuda").bfloat16() for _ in range(2))
    leaves = [x.requires_grad_(True) for x in (q, k, v)]
    qh = q.detach()
    pads = dict(kv_padding=(0, -N % kvb), q_padding=(0, -N % g))

    def step():
        idx, _, avg = ftk.flash_topk_score(qh, qh, H, kvb, 4, pads["kv_padding"], 0.9)
        merged, counts, _ = ftk.build_qblock_topk_indices(idx, g, pads["q_padding"], avg)
        o, _ = ftk.flash_topk_attn(*leaves, merged, counts, H, g, kvb, num_kv_heads=Hkv, **pads)
        torch.autograd.grad(o, leaves, do)

    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    before = ops.launch_count()
    with torch.cuda.graph(graph, stream=stream):
        step()
    counted = ops.launch_count() - before
    raw = rt.cudaGraph_t(graph.raw_cuda_graph())
    err, _, n = rt.cudaGraphGetNodes(raw, 0)
    err, nodes, _ = rt.cudaGraphGetNodes(raw, n)
    assert err == rt.cudaError_t.cudaSuccess
    kernel = rt.cudaGraphNodeType.cudaGraphNodeTypeKernel
    kernels = sum(rt.cudaGraphNodeGetType(x)[1] == kernel for x in nodes[:n])
    ftk.check_errors()
    assert counted == kernels > 0
