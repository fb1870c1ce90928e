"""Which form a step takes where two of them do the same work: the lines, and the forms on both sides of them against each other."""

from types import SimpleNamespace

import pytest
import torch

from conftest import device
from test_gpu_kernels import K

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


def portions(*lens):
    k = K()
    cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
    ctx = SimpleNamespace(cu_q_host=cu, num_requests=len(lens), shared={})
    p = k.long_portions(ctx, 16)
    assert k.long_portions(ctx, 16) is p  # (formed once per step)
    return p


def test_long_portions():
    assert portions(1, 16) == (0, 0, 0, 0, 2)
    assert portions(1, 17, 64, 16, 200) == (3, 281, 200, 1 + 1 + 4, 2)


@pytest.mark.parametrize("lens,sizes,matrix,decays", [
    ((17,), (8, 128, 256), False, False), ((64,), (8, 128, 256), False, False), ((150,), (8, 128, 256), True, False),
    ((800,), (8, 128, 256), True, True), ((17,), (8, 256, 512), False, False), ((100,), (8, 256, 512), False, False),
    ((256,), (8, 256, 512), True, False), ((100,) * 16, (8, 128, 256), True, False), ((24,) * 4, (4, 64, 64), False, False),
    ((1, 2048), (8, 128, 256), True, True), ((1, 16), (8, 128, 256), False, False)])
def test_recurrences_run_in_chunks_where_that_was_faster(lens, sizes, matrix, decays):
    k, p = K(), portions(*lens)
    assert k.mlstm_chunk_pays(p, *sizes) is matrix and k.gla_chunk_pays(p, *sizes) is decays


def test_float32_products_that_stay_with_the_library():
    k = K()
    for (M, N, K_), split in (((511, 4096, 1024), True), ((17, 4096, 1024), True), ((17, 32768, 1024), False), ((17, 4096, 768), False),
                              ((48, 6144, 1024), True), ((300, 256, 64), False), ((256, 1024, 256), False), ((1024, 1024, 256), True)):
        x, w = torch.empty(M, K_, device="meta"), torch.empty(N, K_, device="meta")
        assert k._split_pays(x, w) is split, (M, N, K_)


@pytest.mark.parametrize("heads,n_state,pdim,groups", [(4, 128, 64, 1), (8, 64, 48, 2), (2, 256, 32, 1), (3, 32, 16, 3), (32, 128, 64, 1)])
@pytest.mark.parametrize("lens", [[17], [64], [65, 3, 200], [150, 16, 1], [40] * 5])
@pytest.mark.parametrize("single_row", [False, True])
def test_short_and_long_walks_agree(heads, n_state, pdim, groups, lens, single_row):
    """The form that keeps the states in registers against the one that leaves them between its kernels; a row of steps and decays
    per token and one row for all."""
    from ullm_b200.engine import Workspace

    kk, d = K(), device()
    g = torch.Generator().manual_seed(91)
    T, B = sum(lens), len(lens)
    xbc = torch.randn(T, heads * pdim + 2 * groups * n_state, generator=g).bfloat16().to(d)
    rows = 1 if single_row else T
    dt, log_decay = (0.1 + torch.rand(rows, heads, generator=g)).to(d), (-0.2 * torch.rand(rows, heads, generator=g)).to(d)
    skip = torch.randn(heads, generator=g).to(d)
    state0 = torch.randn(B + 1, heads * pdim * n_state, generator=g).to(d)
    slots = torch.randperm(B + 1, generator=g)[:B].int().to(d)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=d)
    req = torch.cat([torch.full((n,), r, dtype=torch.int32) for r, n in enumerate(lens)]).to(d)
    outs, old = [], kk.lib.ullm_ssd_chunk_short_pays
    for short in (1, 0):
        kk.lib.ullm_ssd_chunk_short_pays = lambda *a: short
        try:
            out, state = torch.full((T, heads * pdim), 5.0, device=d), state0.clone()
            scores, launches = torch.empty(T, kk.ssd_chunk_floats(1, groups), device=d), kk.launches
            kk.ssd_chunk(xbc, heads * pdim, heads * pdim + groups * n_state, dt, log_decay, skip, scores, state, cu, slots, req, out, B, heads,
                         n_state, pdim, groups, 16, Workspace(d, T, B), portions(*lens))
            assert kk.launches - launches == (2 if short else 3)
        finally:
            kk.lib.ullm_ssd_chunk_short_pays = old
        kk.raise_on_status()
        outs.append((out.double(), state.double()))
    # both keep 16 bits of every 32-bit operand, in other orders: 2^-16 of the values each
    for a, b in zip(*outs):
        assert float((a - b).norm() / b.norm()) < 2.0 ** -15


def paged(q_lens, kv_lens, page=16):
    """Block table, page count and the step's arrays of requests that hold `kv_lens` tokens behind `q_lens` new ones."""
    per, bt, used = [-(-n // page) for n in kv_lens], torch.full((len(q_lens), max(-(-n // page) for n in kv_lens) + 1), -1, dtype=torch.int32), 0
    for r, n in enumerate(per):
        bt[r, :n] = torch.arange(used, used + n)
        used += n
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32)
    req = torch.cat([torch.full((n,), r, dtype=torch.int32) for r, n in enumerate(q_lens)])
    ctx = SimpleNamespace(decode_only=False, num_requests=len(q_lens), max_q_len=max(q_lens), max_kv_len=max(kv_lens), cu_q_host=cu.tolist(),
                          shared={}, start_positions_host=[b - a for a, b in zip(q_lens, kv_lens)])
    i = dict(dtype=torch.int32, device="cuda")
    return bt.cuda(), used, torch.arange(len(q_lens), **i), cu.cuda(), torch.tensor(kv_lens, **i), req.cuda(), ctx


@pytest.mark.parametrize("H,dk,dv,n,kv,window,path", [
    (16, 448, 384, 17, 17, 0, "latent_tcgen05"), (16, 448, 384, 17, 2000, 0, "window_mma"), (16, 448, 384, 64, 2000, 0, "window_mma"),
    (16, 448, 384, 200, 2000, 0, "latent_tcgen05"), (16, 448, 384, 600, 600, 0, "latent_tcgen05"), (8, 192, 128, 200, 2000, 1024, "window_mma"),
    (8, 192, 128, 400, 2000, 1024, "latent_tcgen05"), (32, 448, 384, 64, 2000, 1024, "window_mma")])
def test_latent_attention_by_rows_and_keys_in_sight(H, dk, dv, n, kv, window, path):
    k, outs = K(), []
    bt, pages, slots, cu, lens, req, ctx = paged([n], [kv])
    g = torch.Generator().manual_seed(95)
    kp, q = (torch.randn(*s, generator=g).bfloat16().cuda() for s in ((pages, 16, 1, dk), (n, H * dk)))
    for on in (True, False):
        k.latent_attention_on = on
        outs.append(torch.zeros(n, H * dv, dtype=torch.bfloat16, device="cuda"))
        try:
            k.windowed_attention(q, outs[-1], kp, None, bt, slots, cu, lens, req, H, 1, dk, dv, 16, window, dk ** -0.5, num_requests=1, ctx=ctx)
        finally:
            k.latent_attention_on = True
        assert k.attention_path == (path if on else "window_mma")
    k.raise_on_status()
    # (weights rounded to bfloat16 and one rounding of values of order one, on either side)
    assert (outs[0].float() - outs[1].float()).abs().max().item() <= 2.0 ** -6


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("q_lens,kv_lens,tiles", [([2], [2], False), ([8, 16], [8, 16], False), ([16] * 33, [16] * 33, True), ([17], [17], True), ([8], [300], True), ([1, 1], [5, 9], True)])
def test_32_bit_attention_of_a_few_keys_stays_with_the_general_kernel(dtype, q_lens, kv_lens, tiles):
    k, calls, outs = K(), [], []
    bt, pages, slots, cu, lens, req, ctx = paged(q_lens, kv_lens)
    g = torch.Generator().manual_seed(96)
    kp, vp, qkv = (torch.randn(*s, generator=g).to(dtype).cuda() for s in ((pages, 16, 2, 64), (pages, 16, 2, 64), (sum(q_lens), 8 * 64)))
    real = k.lib.ullm_attention_plain
    for on in (True, False):
        outs.append(torch.zeros(sum(q_lens), 4 * 64, dtype=dtype, device="cuda"))
        k.lib.ullm_attention_plain, k.plain_attention_on = (lambda *a: calls.append(0) or real(*a)), on
        try:
            k.paged_attention(qkv, outs[-1], kp, vp, bt, slots, cu, lens, req, 4, 2, 64, 16, 0, 0.125, ctx=ctx)
        finally:
            k.lib.ullm_attention_plain, k.plain_attention_on = real, True
    assert bool(calls) is tiles
    # (32-bit sums in another order, a last place of float16)
    assert (outs[0].float() - outs[1].float()).abs().max() < (4e-5 if dtype == torch.float32 else 4e-3)


@pytest.mark.parametrize("k_dim,n_out,launches", [(128, 256, 1), (256, 512, 1), (512, 512, 2), (1024, 256, 2)])
def test_small_experts_stay_with_mma_sync(k_dim, n_out, launches):
    kk, E, T = K(), 4, 40
    x, w = torch.randn(T, k_dim, device="cuda").bfloat16(), (torch.randn(E, n_out, k_dim, device="cuda") * k_dim ** -0.5).bfloat16()
    choice = (torch.arange(T, device="cuda") % E).int().view(T, 1)
    offsets, order, place = (torch.zeros(n, dtype=torch.int32, device="cuda") for n in (E + 1, T, T))
    kk.moe_arrange(choice, T, E, offsets, order, place)
    out, gathered, before = torch.zeros(T, n_out, dtype=torch.bfloat16, device="cuda"), torch.zeros_like(x), kk.launches
    kk.moe_grouped_linear(x, w, offsets, order, None, out, 1, True, False, gathered=gathered)
    assert kk.launches - before == launches
    ref = torch.stack([x[t].float() @ w[t % E].float().t() for t in range(T)])
    # (one rounding to bfloat16 behind 32-bit sums)
    assert (out[place.long()].float() - ref).abs().max() <= 2.0 ** -7 * ref.abs().max()
