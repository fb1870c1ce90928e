"""Windows that keep first positions on the tcgen05 prompt kernel (csrc/attention_prefill_pair.cu) against a 32-bit reference and the
mma.sync kernel: kept positions that fill part of a tile, a whole one, more than one, and reach into the window; windows that begin
inside a tile; pages between that were given back; values out of sight that are not finite; one-token entries in front."""

from types import SimpleNamespace

import pytest
import torch

from test_gpu_kernels import K, rnd

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]
D = 128


def case(Hq, Hkv, page, q_lens, kv_lens, window, keep, odd=False):
    pages = sum(-(-n // page) for n in kv_lens) + 1
    perm, used = torch.randperm(pages, generator=torch.Generator().manual_seed(1)), 0
    kp, vp = rnd(pages, page, Hkv, D, seed=2, dtype=torch.bfloat16), rnd(pages, page, Hkv, D, seed=3, dtype=torch.bfloat16)
    bt = torch.full((len(q_lens), max(-(-n // page) for n in kv_lens)), -1, dtype=torch.int32)
    for r, (n, q) in enumerate(zip(kv_lens, q_lens)):
        for i in range(-(-n // page)):
            bt[r, i] = perm[used]
            used += 1
        hidden = range(keep, max(keep, n - q - window + 1))  # (positions that no row of the request sees)
        for at in hidden:
            if odd:
                vp[bt[r, at // page].item(), at % page] = float("inf")
                kp[bt[r, at // page].item(), at % page] = float("nan")
            elif at % page == 0 and at + page <= max(keep, n - q - window + 1):
                bt[r, at // page] = -1  # (given back)
    T = sum(q_lens)
    cu = [0]
    for q in q_lens:
        cu.append(cu[-1] + q)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32).cuda()
    ctx = SimpleNamespace(decode_only=False, num_requests=len(q_lens), max_q_len=max(q_lens), max_kv_len=max(kv_lens), cu_q_host=cu,
                          start_positions_host=[n - q for n, q in zip(kv_lens, q_lens)], shared={},
                          workspace=SimpleNamespace(max_requests=8, get=lambda name, rows, cols, dtype, reserve=0: torch.empty(
                              rows, cols, dtype=dtype, device="cuda")))
    return dict(qkv=rnd(T, (Hq + 2 * Hkv) * D, seed=4, dtype=torch.bfloat16), kp=kp, vp=vp, bt=bt, cu=i32(cu), kl=i32(kv_lens),
                req=i32([r for r, q in enumerate(q_lens) for _ in range(q)]), rs=i32(list(range(len(q_lens)))), ctx=ctx, T=T)


def run(c, Hq, Hkv, page, window, keep, rows):
    kk = K()
    out = torch.full((c["T"], Hq * D), 7.0, dtype=torch.bfloat16, device="cuda")
    old, kk.kept_pair_rows = kk.kept_pair_rows, rows
    try:
        kk.paged_attention(c["qkv"], out, c["kp"], c["vp"], c["bt"].cuda(), c["rs"], c["cu"], c["kl"], c["req"], Hq, Hkv, D, page,
                           window, D ** -0.5, c["ctx"], keep_first=keep)
        path = kk.attention_path
    finally:
        kk.kept_pair_rows = old
    kk.raise_on_status()
    return out.float(), path


def reference(c, Hq, Hkv, page, q_lens, kv_lens, window, keep):
    out, t = torch.empty(c["T"], Hq, D), 0
    k, v, q = c["kp"].float().cpu(), c["vp"].float().cpu(), c["qkv"][:, :Hq * D].float().cpu().view(-1, Hq, D)
    for r, (n, ql) in enumerate(zip(kv_lens, q_lens)):
        for i in range(ql):
            pos = n - ql + i
            seen = [j for j in range(pos + 1) if j < keep or j > pos - window]
            at = [(c["bt"][r, j // page].item(), j % page) for j in seen]
            ks = torch.stack([k[a, b] for a, b in at]).repeat_interleave(Hq // Hkv, 1)
            vs = torch.stack([v[a, b] for a, b in at]).repeat_interleave(Hq // Hkv, 1)
            w = torch.softmax(torch.einsum("hd,jhd->hj", q[t], ks) * D ** -0.5, -1)
            out[t] = torch.einsum("hj,jhd->hd", w, vs)
            t += 1
    return out.view(c["T"], Hq * D)


@pytest.mark.parametrize("keep,window", [(4, 100), (1, 1), (128, 300), (129, 130), (200, 64), (40, 1000)])
@pytest.mark.parametrize("Hq,Hkv,page,q_lens,kv_lens", [(4, 2, 16, [65, 3], [520, 3]), (8, 1, 64, [33, 40], [700, 40]),
                                                       (2, 2, 16, [300], [300]), (4, 2, 32, [1, 1, 1, 1, 70], [600, 5, 130, 299, 470])])
@pytest.mark.parametrize("odd", [False, True])
def test_kept_positions_on_the_tcgen05_kernel(keep, window, Hq, Hkv, page, q_lens, kv_lens, odd):
    c = case(Hq, Hkv, page, q_lens, kv_lens, window, keep, odd)
    got, path = run(c, Hq, Hkv, page, window, keep, 1)
    other, plain = run(c, Hq, Hkv, page, window, keep, 1 << 30)
    assert path == "prefill_tcgen05" and plain == "prefill"
    ref = reference(c, Hq, Hkv, page, q_lens, kv_lens, window, keep).cuda()
    # weights and results rounded to bfloat16 (2^-9 each, of values up to the largest value), sums of at most 1,200 weights
    s = ref.abs().max().item()
    assert (got - ref).abs().max().item() <= 2 ** -7 * s
    assert (got - other).abs().max().item() <= 2 ** -6 * s


@pytest.mark.parametrize("Hq,Hkv,page,q_lens,kv_lens,window,keep", [
    (16, 8, 16, [2048], [2048], 1024, 4), (16, 8, 16, [17], [1800], 1024, 4), (8, 2, 16, [700, 401, 33], [700, 900, 1500], 512, 130),
    (16, 16, 16, [511], [2000], 128, 8)])
@pytest.mark.parametrize("peak", [1.0, 3.0])
def test_no_further_from_64_bits_than_the_mma_sync_kernel(Hq, Hkv, page, q_lens, kv_lens, window, keep, peak):
    """Both round a weight and a result to bfloat16; the weight of a row's largest score is exact in both."""
    c = case(Hq, Hkv, page, q_lens, kv_lens, window, keep)
    c["qkv"] = (c["qkv"] * peak).to(torch.bfloat16)
    ref, t = [], 0
    for r, (n, ql) in enumerate(zip(kv_lens, q_lens)):
        at, pos = torch.arange(n, device="cuda"), torch.arange(n - ql, n, device="cuda")[:, None]
        place = c["bt"].cuda()[r, at // page].clamp(min=0).long(), at % page
        k, v = (x[place].double().repeat_interleave(Hq // Hkv, 1) for x in (c["kp"], c["vp"]))
        s = torch.einsum("thd,jhd->htj", c["qkv"][t:t + ql, :Hq * D].double().view(ql, Hq, D), k) * D ** -0.5
        w = torch.softmax(s.masked_fill((at > pos) | ((at >= keep) & (at <= pos - window)), -float("inf")), -1)
        ref.append(torch.einsum("htj,jhd->thd", w, v).reshape(ql, Hq * D))
        t += ql
    ref = torch.cat(ref)
    error = [float((run(c, Hq, Hkv, page, window, keep, rows)[0].double() - ref).norm() / ref.norm()) for rows in (1, 1 << 30)]
    # (the roundings of at least 34,000 results: their norm varies by half a percent from one set of them to another)
    assert error[0] <= 1.01 * error[1]
