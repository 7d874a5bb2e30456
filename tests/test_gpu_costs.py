"""What uncommon inputs cost beside ordinary ones of the same size.

Both sides are timed here, on one device, so that a bound is a ratio.  Each is the ratio that the
work itself has, or that of the plain kernels, with room for noise; the inputs are ones that some
kernel once took several times longer over."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ftk():
    import flash_topk_attn_v2 as m
    return m


def _us(call, calls=5, rounds=7):
    """Device time of a call: the shortest of some rounds, the calls of a round back to back."""
    call()
    torch.cuda.synchronize()
    times = []
    for _ in range(rounds):
        a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
        torch.cuda._sleep(500000)      # the calls are enqueued by then
        a.record()
        for _ in range(calls):
            call()
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b) * 1e3 / calls)
    return min(times)


def _random_lists(H, QM, M, W, gen):
    return torch.rand(1, H, QM, M, generator=gen, device="cuda").topk(W, dim=-1).indices.to(torch.int32)


@pytest.mark.parametrize("D", [64, 128])
def test_backward_of_48_row_blocks(ftk, D):
    """48 rows of 64 and 96 of 128 make 16 / 9 times the tiles of 64-row blocks, whose pairs cost
    the same otherwise; 1.3 for half a warp that lists a block where the other half does not."""
    N, H = 4032, 16
    gen = torch.Generator(device="cuda").manual_seed(1)
    q, k, v, do = (torch.randn(1, N, H * D, generator=gen, device="cuda").bfloat16() for _ in range(4))
    for x in (q, k, v):
        x.requires_grad_(True)
    us = {}
    for g in (64, 48):
        M = N // g
        merged = _random_lists(H, M, M, M // 2, gen)
        o, _ = ftk.flash_topk_attn(q, k, v, merged, None, H, g, g)
        us[g] = _us(lambda: torch.autograd.grad(o, (q, k, v), do, retain_graph=True))
    ftk.check_errors()
    assert us[48] <= 1.3 * 16 / 9 * us[64], us


@pytest.mark.parametrize("D,W", [(64, 2), (64, 8), (128, 2), (256, 2)])
def test_forward_that_is_all_for_the_exact_kernel(ftk, monkeypatch, D, W):
    """fp16 rows beyond the pipelined kernel's range in every one of 1024 tiles: the forward is both
    kernels one after the other, and that is what it costs (1.3 of the sum); the bits are the exact
    kernel's."""
    N, H, g = 8192, 16, 64
    gen = torch.Generator(device="cuda").manual_seed(2)
    q, k, v = (torch.randn(1, N, H * D, generator=gen, device="cuda").half() for _ in range(3))
    merged = _random_lists(H, N // g, N // g, W, gen)
    hot = k * 12.0
    run = lambda keys: ftk.flash_topk_attn(q, keys, v, merged, None, H, g, g)
    ordinary, marked = _us(lambda: run(k)), _us(lambda: run(hot))
    o, lse = run(hot)
    monkeypatch.setenv("FTK_FWD_PIPE", "0")
    exact = _us(lambda: run(hot))
    o2, lse2 = run(hot)
    ftk.check_errors()
    same = (o.view(N, H, D) == o2.view(N, H, D)).all(-1).float().mean().item()
    assert torch.equal(lse, lse2) and same == 1.0
    assert marked <= 1.3 * (ordinary + exact), (marked, ordinary, exact)


@pytest.mark.parametrize("blocks,M,k,g", [(512, 64, 64, 64), (256, 64, 32, 64), (32, 128, 16, 32)])
def test_merge_of_rows_that_name_a_block_twice(ftk, blocks, M, k, g):
    """One block twice in every row takes its entries out of the order-free table: a warp that walks
    all entries in order takes 2 to 5 times as long as the table, so 8."""
    gen = torch.Generator(device="cuda").manual_seed(3)
    idx = torch.rand(1, 1, blocks * g, M, generator=gen, device="cuda").topk(k, -1).indices.to(torch.int32)
    scr = torch.rand(1, 1, blocks * g, k, generator=gen, device="cuda")
    us = []
    for _ in range(2):
        us.append(_us(lambda: ftk.flash_qblock_merge(idx, scr, g, M, M, q_padding=(0, 0), return_counts=True), 20))
        idx[..., 1] = idx[..., 0]
    ftk.check_errors()
    assert us[1] <= 8 * us[0], us


@pytest.mark.parametrize("rows,M,k", [(131072, 128, 32), (131072, 128, 16), (33000, 32, 8), (33000, 17, 16), (12000, 4, 3)])
@pytest.mark.parametrize("what,most", [("equal", 1.5), ("zero", 1.5), ("eighths", 3.0)])
def test_select_of_rows_that_tie(ftk, rows, M, k, what, most):
    """Rows of equal scores, as zero or padded queries leave them, are sorted like any others.  Ties at
    the cut that are not told apart at once take a second pass, and their averages are compared in
    full: not more than a third one."""
    gen = torch.Generator(device="cuda").manual_seed(4)
    x = torch.rand(1, 1, rows, M, generator=gen, device="cuda")
    y = {"equal": torch.full_like(x, 0.25), "zero": torch.zeros_like(x), "eighths": (x * 8).round() / 8}[what]
    us = [_us(lambda: ftk.flash_topk_select(s, 2.0 * M, k, 64, (0, 0)), 20) for s in (x, y)]
    ftk.check_errors()
    assert us[1] <= most * us[0], us
