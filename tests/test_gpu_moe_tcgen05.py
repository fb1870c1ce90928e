"""The routed experts' grouped product on tcgen05 (csrc/moe_tcgen05.cu) against a 32-bit reference and the mma.sync kernel, where
its tiles end: experts with no rows, one row, a row less and more than a tile; columns and k that fill no whole tile; choices that
name no expert; weights on the input; every activation."""

import pytest
import torch

from test_gpu_kernels import K, rnd

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


def reference(x, w, choice, weight, top, from_pairs, gated, act, limit, alpha, rows_of):
    out = {}
    for p in range(choice.numel()):
        e = int(choice.view(-1)[p])
        if e >= w.shape[0]:
            continue
        out.setdefault(e, []).append(p)
    n = w.shape[1] // 2 if gated else w.shape[1]
    full = torch.zeros(choice.numel(), n, dtype=torch.float32, device=x.device)
    for e, pairs in out.items():
        p = torch.tensor(pairs, device=x.device)
        v = (x[p // top] if from_pairs else x[rows_of[p]]).float() @ w[e].float().t()
        if weight is not None:
            v = v * weight.view(-1)[p][:, None]
        if gated:
            g, u = v[:, :n], v[:, n:]
            if act == 2:
                g, u = g.clamp(max=limit), u.clamp(-limit, limit)
                v = g * torch.sigmoid(alpha * g) * (u + 1)
            else:
                v = (torch.nn.functional.silu(g) if act == 0 else torch.nn.functional.gelu(g, approximate="tanh")) * u
        elif act == 3:
            v = v.clamp(min=0) ** 2
        full[p] = v
    return full


@pytest.mark.parametrize("counts,top", [([0, 1, 127, 128, 129, 3], 1), ([257, 0, 0, 1], 2), ([5] * 40, 3), ([1, 0, 16, 0], 1), ([2], 1)])
@pytest.mark.parametrize("n_out,k", [(128, 64), (264, 200), (72, 512), (520, 1032)])
@pytest.mark.parametrize("gated,act,weighted", [(True, 0, True), (True, 1, False), (True, 2, False), (False, 3, False), (False, -1, True)])
def test_grouped_product_matches_the_reference(counts, top, n_out, k, gated, act, weighted):
    kk = K()
    E = len(counts)
    total = -(-sum(counts) // top) * top
    flat = [e for e, n in enumerate(counts) for _ in range(n)] + [E + 1] * (total - sum(counts))  # (E + 1: no expert's)
    g = torch.Generator().manual_seed(5)
    choice = torch.tensor(flat, dtype=torch.int32)[torch.randperm(total, generator=g)].view(-1, top).contiguous().cuda()
    T = total // top
    offsets = torch.empty(E + 1, dtype=torch.int32, device="cuda")
    order, place = torch.zeros(T, top, dtype=torch.int32, device="cuda"), torch.zeros(T, top, dtype=torch.int32, device="cuda")
    kk.moe_arrange(choice, total, E, offsets, order, place)
    w = rnd(E, (2 if gated else 1) * n_out, k, seed=6, dtype=torch.bfloat16, scale=k ** -0.5)
    weight = (rnd(T, top, seed=7).abs() + 0.1) if weighted else None
    for from_pairs in (True, False):
        x = rnd(T if from_pairs else total, k, seed=8, dtype=torch.bfloat16)
        out = torch.full((total, n_out), 9.0, dtype=torch.bfloat16, device="cuda")
        old = kk.moe_tcgen05_rows
        try:
            kk.moe_tcgen05_rows = 0
            gathered = torch.empty(total, k, dtype=torch.bfloat16, device="cuda") if from_pairs else None
            kk.moe_grouped_linear(x, w, offsets, order, weight, out, top, from_pairs, gated, act, 3.0, 1.702, gathered=gathered)
            other = torch.full_like(out, 9.0)
            kk.moe_tcgen05_rows = 1 << 30
            kk.moe_grouped_linear(x, w, offsets, order, weight, other, top, from_pairs, gated, act, 3.0, 1.702)
        finally:
            kk.moe_tcgen05_rows = old
        kk.raise_on_status()
        live = choice.view(-1).cpu() < E
        at = place.view(-1).long()
        ref = reference(x, w, choice.cpu(), weight, top, from_pairs, gated, act, 3.0, 1.702, at)
        used = int(live.sum())
        got, gen = out[at][live.cuda()].float(), other[at][live.cuda()].float()
        ref = ref[live.cuda()]
        s = ref.abs().max().item()
        # one rounding to bfloat16 (2^-9 of the value) behind 32-bit sums of at most 1,032 products of order k^-1/2
        assert (got - ref).abs().max().item() <= (2 ** -8 + 1e-4) * s
        assert (got - gen).abs().max().item() <= (2 ** -7 + 1e-4) * s
        assert (out[used:] == 9.0).all()  # (places that belong to no expert stay as they were)


@pytest.mark.parametrize("gated,act", [(True, 0), (False, 3)])
def test_blocks_with_many_tiles_use_their_accumulators_again(gated, act):
    """More than four tiles per block (two accumulators in turn, each handed over several times), experts without places between
    full ones."""
    kk, n_out, k = K(), 2056 if gated else 4112, 136
    counts = [260, 0, 256, 129, 0, 250, 270, 128, 1, 0, 255, 257, 300, 0, 264, 127]
    tiles = sum(-(-c // 128) for c in counts) * -(-n_out // (128 if gated else 256))
    assert tiles > 2.5 * torch.cuda.get_device_properties(0).multi_processor_count
    E, total = len(counts), sum(counts)
    g = torch.Generator().manual_seed(9)
    flat = torch.tensor([e for e, n in enumerate(counts) for _ in range(n)], dtype=torch.int32)
    choice = flat[torch.randperm(total, generator=g)].view(-1, 1).contiguous().cuda()
    offsets = torch.empty(E + 1, dtype=torch.int32, device="cuda")
    order, place = (torch.zeros(total, 1, dtype=torch.int32, device="cuda") for _ in range(2))
    kk.moe_arrange(choice, total, E, offsets, order, place)
    w = rnd(E, (2 if gated else 1) * n_out, k, seed=6, dtype=torch.bfloat16, scale=k ** -0.5)
    x = rnd(total, k, seed=8, dtype=torch.bfloat16)
    out, gathered = (torch.full((total, n), 9.0, dtype=torch.bfloat16, device="cuda") for n in (n_out, k))
    launches = kk.launches
    kk.moe_grouped_linear(x, w, offsets, order, None, out, 1, True, gated, act, gathered=gathered)
    kk.raise_on_status()
    assert kk.launches == launches + 2  # (the rows gathered, the product)
    at = place.view(-1).long()
    ref = reference(x, w, choice.cpu(), None, 1, True, gated, act, 0.0, 1.0, at)
    # (one rounding to bfloat16 behind 32-bit sums of 136 products, as above)
    assert (out[at].float() - ref).abs().max().item() <= (2 ** -8 + 1e-4) * ref.abs().max().item()


@pytest.mark.parametrize("act", [0, 2])
def test_gates_that_are_almost_shut(act):
    """Denominators 1 + e^-z up to the largest 32-bit number: silu(-88) is -5.3e-37 and no zero, as in the mma.sync kernel."""
    kk, n_out, k, rows = K(), 64, 64, 20
    z = torch.tensor([-86.0, -87.0, -87.5, -88.0, -88.5, -90.0, -1.0, 3.0]).repeat(n_out // 8)  # (bfloat16 holds them)
    w = torch.zeros(1, 2 * n_out, k)
    w[0, :n_out, 0], w[0, n_out:, 0] = z, 1024.0
    w, x = w.to(torch.bfloat16).cuda(), torch.zeros(rows, k, dtype=torch.bfloat16, device="cuda")
    x[:, 0] = 1
    choice = torch.zeros(rows, 1, dtype=torch.int32, device="cuda")
    offsets = torch.empty(2, dtype=torch.int32, device="cuda")
    order, place = (torch.zeros(rows, 1, dtype=torch.int32, device="cuda") for _ in range(2))
    kk.moe_arrange(choice, rows, 1, offsets, order, place)
    outs, old = [], kk.moe_tcgen05_rows
    try:
        for kk.moe_tcgen05_rows in (0, 1 << 30):
            outs.append(torch.full((rows, n_out), 9.0, dtype=torch.bfloat16, device="cuda"))
            kk.moe_grouped_linear(x, w, offsets, order, None, outs[-1], 1, True, True, act, 2000.0, 1.0, gathered=torch.empty_like(x))
    finally:
        kk.moe_tcgen05_rows = old
    kk.raise_on_status()
    z64 = z.double().cuda()
    ref = torch.where(z64 < -88.72, 0.0, z64 / (1 + torch.exp(-z64)) * (1024 + (act == 2)))
    # one rounding to bfloat16, whose 8 bits make half a unit up to 2^-8 of a value, behind a 32-bit gate (some units of 2^-24)
    for out in outs:
        assert ((out.double() - ref).abs() <= (2 ** -8 + 1e-6) * ref.abs()).all()
