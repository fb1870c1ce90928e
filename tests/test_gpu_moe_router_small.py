"""Router product, choices and arrangement in one launch (csrc/moe.cu, `moe_router_small`) against the three launches it replaces:
one token and the most, fewer router rows than blocks and more than warps, groups, corrections, always-chosen experts."""

import pytest
import torch

from test_gpu_kernels import K, rnd

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


@pytest.mark.parametrize("T,H", [(1, 64), (3, 200), (16, 2048), (9, 4096)])
@pytest.mark.parametrize("experts,rows,top,groups,keep,always", [(5, 8, 2, 1, 1, 0), (16, 24, 2, 4, 2, 1), (34, 40, 3, 1, 1, 0), (96, 96, 8, 8, 3, 2)])
@pytest.mark.parametrize("softmax,renormalize,corrected", [(False, False, False), (True, False, True), (False, True, True)])
def test_one_launch_is_the_three(T, H, experts, rows, top, groups, keep, always, softmax, renormalize, corrected):
    k = K()
    x = rnd(T, H + 8, seed=41, dtype=torch.bfloat16)[:, :H]
    w = rnd(rows, H, seed=42, dtype=torch.bfloat16, scale=2.0 * H ** -0.5)
    corr = rnd(experts, seed=43, scale=0.05) if corrected else None
    E, P = experts + always - 1, T * (top + always)  # (the last router output stands for no expert)

    def outputs():
        i = dict(dtype=torch.int32, device="cuda")
        return [torch.zeros(T, rows, device="cuda"), torch.zeros(P, **i), torch.zeros(P, device="cuda"), torch.zeros(E + 1, **i),
                torch.full((P,), -7, **i), torch.zeros(P, **i)]

    lg, ch, wt, off, order, place = outputs()
    assert k.moe_router_small(x, w, lg, ch, wt, top, softmax, renormalize, corr, experts, groups, keep, 1.5, always, E, off, order, place)
    ref = x.float() @ w.float().t()
    # products of order one, sums of at most 4,096 of them in another order
    assert (lg - ref).abs().max().item() < 1e-4
    lg2, ch2, wt2, off2, order2, place2 = outputs()
    k.moe_route(lg, ch2, wt2, top, softmax, renormalize, correction=corr, experts=experts, groups=groups, keep=keep, scale=1.5,
                always=always)
    k.moe_arrange(ch2, P, E, off2, order2, place2)
    assert torch.equal(ch, ch2) and torch.equal(wt, wt2) and torch.equal(off, off2)
    # inside an expert's group the order is free: every pair at its place, once
    live = ch < E
    n = int(live.sum())
    assert int(off[-1]) == n and sorted(order[:n].tolist()) == live.nonzero().view(-1).tolist()
    for p in live.nonzero().view(-1).tolist():
        at = int(place[p])
        assert int(order[at]) == p and int(off[ch[p]]) <= at < int(off[ch[p] + 1])
    k.raise_on_status()


def test_steps_it_does_not_take():
    k = K()
    for x in (rnd(17, 64, dtype=torch.bfloat16), rnd(4, 64)):
        T = x.shape[0]
        i = dict(dtype=torch.int32, device="cuda")
        assert not k.moe_router_small(x, rnd(8, 64, dtype=x.dtype), torch.zeros(T, 8, device="cuda"), torch.zeros(T, **i),
                                      torch.zeros(T, device="cuda"), 1, False, False, None, 8, 1, 1, 1.0, 0, 8, torch.zeros(9, **i),
                                      torch.zeros(T, **i), torch.zeros(T, **i))
