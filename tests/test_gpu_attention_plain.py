"""32-bit attention by row tiles (csrc/attention_plain.cu) against the plain reference and against the general kernel, at the
edges of its tiles: rows of a tile (32, shared by the query heads of a kv head), 32 keys of two groups, windows and stretches that begin inside
a tile, single tokens beside prompt portions, padding rows."""

import pytest
import torch

from test_gpu_kernels import K, attention_reference, close, rnd

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


def case(dtype, Hq, Hkv, D, page, q_lens, kv_lens, pad=0, behind=0):
    B, T = len(q_lens), sum(q_lens) + behind
    max_pages = max(-(-k // page) for k in kv_lens) + 1
    g = torch.Generator().manual_seed(21)
    pages = sum(-(-k // page) for k in kv_lens) + 2
    perm = torch.randperm(pages, generator=g)
    slots = torch.randperm(B + 2, generator=g)[:B].tolist()
    bt = torch.full((B + 2, max_pages), -1, dtype=torch.int32)
    used = 0
    for r, kl in enumerate(kv_lens):
        n = -(-kl // page)
        bt[slots[r], :n] = perm[used:used + n].int()
        used += n
    kp, vp = rnd(pages, page, Hkv, D, seed=22, dtype=dtype), rnd(pages, page, Hkv, D, seed=23, dtype=dtype)
    qkv = rnd(T, (Hq + 2 * Hkv) * D + pad, seed=24, dtype=dtype)
    cu = torch.tensor([0] + list(torch.tensor(q_lens).cumsum(0)), dtype=torch.int32).cuda()
    req = torch.cat([torch.full((n,), r, dtype=torch.int32) for r, n in enumerate(q_lens)]
                    + [torch.full((behind,), -1, dtype=torch.int32)]).cuda()
    return dict(qkv=qkv, kp=kp, vp=vp, bt=bt, slots=slots, cu=cu, req=req, q_lens=q_lens, kv_lens=kv_lens, T=T)


def run(c, Hq, Hkv, D, page, window, scale, on=True):
    k = K()
    out = torch.full((c["T"], Hq * D), 7.0, dtype=c["qkv"].dtype, device="cuda")
    k.plain_attention_on = on
    try:
        k.paged_attention(c["qkv"], out, c["kp"], c["vp"], c["bt"].cuda(), torch.tensor(c["slots"], dtype=torch.int32).cuda(),
                          c["cu"], torch.tensor(c["kv_lens"], dtype=torch.int32).cuda(), c["req"], Hq, Hkv, D, page, window, scale)
    finally:
        k.plain_attention_on = True
    k.raise_on_status()
    return out


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("Hq,Hkv,D", [(4, 4, 64), (4, 2, 128), (12, 4, 64), (8, 2, 128), (5, 1, 64), (16, 2, 128), (32, 1, 64)])
@pytest.mark.parametrize("window", [0, 33, -64])
@pytest.mark.parametrize("q_lens,kv_lens", [
    ([1, 31, 32, 33], [64, 31, 32, 97]), ([65, 1, 2], [65, 129, 66]), ([1, 1, 1], [1, 33, 260]), ([17], [81]),
    ([2, 40], [193, 223])])
def test_row_tiles_match_the_reference_and_the_general_kernel(dtype, Hq, Hkv, D, window, q_lens, kv_lens):
    scale, page = D ** -0.5, 16
    c = case(dtype, Hq, Hkv, D, page, q_lens, kv_lens)
    out = run(c, Hq, Hkv, D, page, window, scale)
    ref = attention_reference(c["qkv"][:, : Hq * D].float().cpu().view(c["T"], Hq, D), c["kp"].float().cpu().view(-1, Hkv, D),
                              c["vp"].float().cpu().view(-1, Hkv, D), c["bt"].long(), c["slots"], q_lens, kv_lens, Hq, Hkv, D,
                              page, window, scale)
    # (float16: a last place, 2^-11 of the value, beside the reference's 32 bits)
    close(out.view(c["T"], Hq, D).float() if dtype == torch.float32 else out.view(c["T"], Hq, D).float() / 25,
          ref if dtype == torch.float32 else ref / 25, torch.float32, None if dtype == torch.float32 else ref.abs().max().item())
    general = run(c, Hq, Hkv, D, page, window, scale, on=False)
    # both are 32-bit sums of at most 128 + 260 terms of order one in another order, rounded once to the dtype: 400 x 2^-24 of
    # order one, and a last place of float16
    assert (out.float() - general.float()).abs().max() < (4e-5 if dtype == torch.float32 else 4e-3)


def test_rows_on_other_borders_and_unknown_pages():
    """A row stride that 16-byte reads cannot take goes to the general kernel; an unknown page is reported and skipped."""
    c = case(torch.float32, 4, 2, 64, 16, [3, 1], [40, 20], pad=2)
    close(run(c, 4, 2, 64, 16, 0, 0.125), run(c, 4, 2, 64, 16, 0, 0.125, on=False).float().cpu(), torch.float32)
    c = case(torch.float32, 4, 2, 64, 16, [3, 1], [40, 20])
    c["bt"][c["slots"][0], 1] = 10 ** 6
    with pytest.raises(Exception, match="page id out of range"):
        run(c, 4, 2, 64, 16, 0, 0.125)


def test_padding_rows_are_zeros():
    c = case(torch.float32, 4, 2, 64, 16, [1, 1, 1], [9, 30, 4])
    c["req"][1] = -1
    out = run(c, 4, 2, 64, 16, 0, 0.125)
    assert torch.count_nonzero(out[1]) == 0 and torch.isfinite(out).all() and (out[[0, 2]] != 7.0).all()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("Hq,Hkv,D", [(4, 2, 64), (16, 1, 128)])
@pytest.mark.parametrize("q_lens,behind", [([0, 2], 0), ([0, 0, 2], 0), ([2, 0, 1], 0), ([1, 0, 0, 70], 0), ([1, 0], 1), ([1], 1), ([1, 1], 40),
                                           ([33, 1], 3), ([32, 32], 32), ([0, 0], 2)])
def test_requests_without_tokens_and_rows_behind_the_last(dtype, Hq, Hkv, D, q_lens, behind):
    """A batch row may bring no token, whatever the rows and requests count, and rows behind the last request's are zeros: as the
    general kernel has it."""
    c = case(dtype, Hq, Hkv, D, 16, q_lens, [n + 19 for n in q_lens], behind=behind)
    out, general = run(c, Hq, Hkv, D, 16, 0, D ** -0.5), run(c, Hq, Hkv, D, 16, 0, D ** -0.5, on=False)
    # (as above: 32-bit sums in another order, a last place of float16)
    assert (out.float() - general.float()).abs().max() < (4e-5 if dtype == torch.float32 else 4e-3)
    assert torch.count_nonzero(out[c["T"] - behind:]) == 0


def test_rows_of_a_portion_that_belong_to_no_request_or_lie_in_front_of_its_first_position():
    """Rows marked as padding inside a portion, and rows whose position would be negative, are zeros in both kernels."""
    c = case(torch.float32, 4, 2, 64, 16, [40, 12], [40, 12])
    c["req"][3], c["req"][37], c["kv_lens"] = -1, -1, [40, 7]
    out, general = run(c, 4, 2, 64, 16, 0, 0.125), run(c, 4, 2, 64, 16, 0, 0.125, on=False)
    assert torch.count_nonzero(general[[3, 37, 40, 44]]) == 0 and (out - general).abs().max() < 4e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("window", [0, 33, -64])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_values_that_a_row_does_not_see_do_not_reach_it(dtype, window, value):
    """An infinite or NaN value of a later token, or of one in front of a row's window, changes the rows that see it and no others."""
    Hq, Hkv, D, q_lens, kv_lens = 4, 2, 64, [90, 1], [150, 140]
    c = case(dtype, Hq, Hkv, D, 16, q_lens, kv_lens)
    clean = run(c, Hq, Hkv, D, 16, window, D ** -0.5)
    for at in (75, 90, 149):  # key positions of the first request, whose rows stand at 60 to 149
        v = c["vp"].clone()
        page = int(c["bt"][c["slots"][0], at // 16])
        c["vp"][page, at % 16, 1, 3] = value
        out, general = run(c, Hq, Hkv, D, 16, window, D ** -0.5), run(c, Hq, Hkv, D, 16, window, D ** -0.5, on=False)
        pos = torch.arange(60, 150)
        first = {0: 0 * pos, 33: (pos - 32).clamp(min=0), -64: pos - pos % 64}[window]
        hit = torch.zeros(c["T"], Hq, D, dtype=torch.bool)
        hit[:90, 2:, 3] = ((pos >= at) & (first <= at))[:, None]
        hit = hit.view(c["T"], -1).cuda()
        assert torch.equal(~torch.isfinite(out), hit) and torch.equal(~torch.isfinite(general), hit)
        assert (out - clean)[~hit].abs().max() <= (2e-5 if dtype == torch.float32 else 2e-3)  # (sums in another order, see above)
        c["vp"] = v
