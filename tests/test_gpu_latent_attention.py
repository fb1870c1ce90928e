"""Prompt attention over latent key rows on tcgen05 (csrc/attention_latent_tcgen05.cu) against a 32-bit reference and the mma.sync
kernel: blocks that end early, key tiles that end in the middle of a page, windows and stretches that begin inside a tile, pages
given back in front of the window, decoded tokens at the head of the step, garbage behind a request's last key."""

from types import SimpleNamespace

import pytest
import torch

from test_gpu_kernels import K, rnd

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


def reference(q, kp, bt, slots, q_lens, kv_lens, H, dk, dv, page, window, scale):
    out, t0 = [], 0
    for r, (n, kv) in enumerate(zip(q_lens, kv_lens)):
        rows = kp.view(-1, dk)[(bt[slots[r], torch.arange(kv) // page].long() * page + torch.arange(kv) % page).to(kp.device)]
        for j in range(n):
            pos = kv - n + j
            lo = max(0, pos - window + 1) if window > 0 else (pos - pos % -window if window < 0 else 0)
            k = rows[lo:pos + 1]
            p = torch.softmax((q[t0 + j].view(H, dk) @ k.t()) * scale, -1)
            out.append(p @ k[:, :dv])
        t0 += n
    return torch.stack(out)


@pytest.mark.parametrize("H,dk,dv", [(16, 448, 384), (32, 448, 384), (8, 192, 128), (1, 64, 64), (128, 320, 320), (4, 448, 256)])
@pytest.mark.parametrize("page,window", [(16, 0), (16, 100), (64, -128), (8, 0)])
@pytest.mark.parametrize("q_lens,kv_lens", [([130], [130]), ([1, 1, 1, 1, 9, 33], [70, 129, 1, 64, 9, 200]), ([8, 7, 65], [64, 71, 321])])
def test_latent_rows_match_the_reference(H, dk, dv, page, window, q_lens, kv_lens):
    k, scale = K(), dk ** -0.5
    T, B, dtype = sum(q_lens), len(q_lens), torch.bfloat16
    g = torch.Generator().manual_seed(31)
    pages = sum(-(-n // page) for n in kv_lens) + 2
    perm, slots = torch.randperm(pages, generator=g), torch.randperm(B + 1, generator=g)[:B]
    bt = torch.full((B + 1, max(-(-n // page) for n in kv_lens) + 1), -1, dtype=torch.int32)
    used = 0
    kp = rnd(pages, page, 1, dk, seed=32, dtype=dtype)
    for r, kl in enumerate(kv_lens):
        n = -(-kl // page)
        bt[slots[r], :n] = perm[used:used + n].int()
        if kl % page:
            kp[int(perm[used + n - 1]), kl % page:] = float("nan")  # (slots behind the last key may hold anything)
        used += n
    ref_bt = bt.clone()
    if window > 0:  # pages that lie wholly in front of every window have been given back
        for r, (n, kl) in enumerate(zip(q_lens, kv_lens)):
            bt[slots[r], :max(0, kl - n - window + 1) // page] = -1
    q = rnd(T, H * dk + 8, seed=33, dtype=dtype)[:, :H * dk]
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32).cuda()
    req = torch.cat([torch.full((n,), r, dtype=torch.int32) for r, n in enumerate(q_lens)]).cuda()
    ctx = SimpleNamespace(decode_only=False, num_requests=B, max_kv_len=max(kv_lens), cu_q_host=cu.tolist(), shared={},
                          start_positions_host=[a - b for a, b in zip(kv_lens, q_lens)])

    def run(on):
        out = torch.full((T, H * dv), 3.0, dtype=dtype, device="cuda")
        k.latent_attention_on = on
        try:
            k.windowed_attention(q, out, kp, None, bt.cuda(), slots.int().cuda(), cu, torch.tensor(kv_lens, dtype=torch.int32).cuda(),
                                 req, H, 1, dk, dv, page, window, scale, num_requests=B, ctx=ctx)
        finally:
            k.latent_attention_on = True
        k.raise_on_status()
        return out

    got, path = run(True), k.attention_path
    ref = reference(q.float(), torch.nan_to_num(kp.float()), ref_bt, slots.tolist(), q_lens, kv_lens, H, dk, dv, page, window, scale)
    # weights rounded to bfloat16 (2^-9 of each; they sum to one, the values are of order one) and one rounding of the result
    err = (got.float().view(T, H, dv) - ref).abs().max().item()
    assert err <= 2 ** -7 * max(1.0, ref.abs().max().item()), err
    if len(q_lens) != 6:
        assert path == "latent_tcgen05"
    if page in (8, 16, 32, 64) and not (kp.isnan().any()):
        assert (got.float() - run(False).float()).abs().max().item() <= 2 ** -6 * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("window", [0, 40, -64])
def test_a_missing_page_is_reported_where_a_row_sees_it(window):
    """A page that a row sees and the table does not hold is an error, as in the mma.sync kernel; one that only lies in a key tile
    with seen keys is not."""
    k, H, dk, dv, page, n, kv = K(), 16, 192, 128, 8, 20, 150  # positions 130 to 149; 40 positions: from 91 on, a stretch: from 128
    first = {0: 0, 40: 91, -64: 128}[window]
    kp, q = rnd(40, page, 1, dk, seed=42, dtype=torch.bfloat16), rnd(n, H * dk, seed=43, dtype=torch.bfloat16)
    cu, lens, req = (torch.tensor(x, dtype=torch.int32).cuda() for x in ([0, n], [kv], [0] * n))
    ctx = SimpleNamespace(decode_only=False, num_requests=1, max_kv_len=kv, cu_q_host=[0, n], shared={}, start_positions_host=[kv - n])

    def run(gone, value, on):
        bt = torch.arange(24, dtype=torch.int32).view(1, 24)
        bt[0, gone] = value
        k.latent_attention_on = on
        try:
            out = torch.zeros(n, H * dv, dtype=torch.bfloat16, device="cuda")
            k.windowed_attention(q, out, kp, None, bt.cuda(), torch.zeros(1, dtype=torch.int32).cuda(), cu, lens, req, H, 1, dk, dv, page,
                                 window, 0.07, num_requests=1, ctx=ctx)
        finally:
            k.latent_attention_on = True
        k.raise_on_status()

    for on in (True, False):
        for value in (-1, 40):
            for gone in {first // page, (first + 8) // page, 140 // page, (kv - 1) // page}:
                with pytest.raises(Exception, match="page id out of range"):
                    run(gone, value, on)
            for gone in {max(0, first // page - 1)} if window else {}:
                run(gone, value, on)


def test_a_long_decoded_request_does_not_decide_the_kernel_of_a_short_portion():
    """The kernel goes by the keys that the portions see, not by those of the decoded tokens in front of them."""
    k, H, dk, dv, page = K(), 16, 192, 128, 16
    q_lens, kv_lens = [1, 1, 1, 1, 24], [2500, 17, 900, 64, 40]
    T, B = sum(q_lens), len(q_lens)
    bt, used = torch.full((B, 160), -1, dtype=torch.int32), 0
    for r, kl in enumerate(kv_lens):
        n = -(-kl // page)
        bt[r, :n] = torch.arange(used, used + n)
        used += n
    kp, q = rnd(used, page, 1, dk, seed=52, dtype=torch.bfloat16), rnd(T, H * dk, seed=53, dtype=torch.bfloat16)
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32)
    req = torch.cat([torch.full((n,), r, dtype=torch.int32) for r, n in enumerate(q_lens)]).cuda()
    ctx = SimpleNamespace(decode_only=False, num_requests=B, max_kv_len=max(kv_lens), cu_q_host=cu.tolist(), shared={},
                          start_positions_host=[a - b for a, b in zip(kv_lens, q_lens)])
    out, launches = torch.zeros(T, H * dv, dtype=torch.bfloat16, device="cuda"), k.launches
    k.windowed_attention(q, out, kp, None, bt.cuda(), torch.arange(B, dtype=torch.int32).cuda(), cu.cuda(),
                         torch.tensor(kv_lens, dtype=torch.int32).cuda(), req, H, 1, dk, dv, page, 0, 0.07, num_requests=B, ctx=ctx)
    k.raise_on_status()
    assert k.launches == launches + 2  # (the portion's kernel, and the one of the decoded tokens)
    ref = reference(q.float(), kp.float(), bt, list(range(B)), q_lens, kv_lens, H, dk, dv, page, 0, 0.07)
    assert (out.float().view(T, H, dv) - ref).abs().max().item() <= 2 ** -7 * max(1.0, ref.abs().max().item())
