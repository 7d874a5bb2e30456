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
