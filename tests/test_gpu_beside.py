"""Decode attention that runs beside the prompt attention of the same step's other rows (csrc/decode_core.cuh): the same bits as with
the launches one after the other, for even and uneven contexts, many times over, and in steps of the latent layers."""

from types import SimpleNamespace

import pytest
import torch

from test_gpu_kernels import K, rnd

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


def batch(q_lens, kv_lens, page, key_dim, kv_heads):
    bt, used = torch.full((len(q_lens), max(-(-n // page) for n in kv_lens)), -1, dtype=torch.int32), 0
    for r, n in enumerate(kv_lens):
        m = -(-n // page)
        bt[r, :m] = torch.arange(used, used + m)
        used += m
    cu = [0]
    for q in q_lens:
        cu.append(cu[-1] + q)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32).cuda()
    buffers = {}

    def get(name, rows, cols, dtype, reserve=0):
        key = (name, cols)
        if key not in buffers or buffers[key].shape[0] < rows:
            buffers[key] = torch.empty(max(rows, reserve), cols, dtype=dtype, device="cuda")
        return buffers[key][:rows]

    ws = SimpleNamespace(max_requests=len(q_lens), get=get)
    ctx = SimpleNamespace(decode_only=False, num_requests=len(q_lens), max_q_len=max(q_lens), max_kv_len=max(kv_lens), cu_q_host=cu,
                          start_positions_host=[n - q for n, q in zip(kv_lens, q_lens)], shared={}, workspace=ws)
    pages = rnd(used, page, kv_heads, key_dim, seed=3, dtype=torch.bfloat16)
    return ctx, bt.cuda(), i32(cu), i32(kv_lens), i32([r for r, q in enumerate(q_lens) for _ in range(q)]), i32(range(len(q_lens))), pages


@pytest.mark.parametrize("q_lens,kv_lens,kernel", [
    ([1] * 4 + [200], [700, 650, 690, 700, 200], "decode"),
    ([1] * 9 + [33, 300], [9, 40, 2000, 100, 30, 700, 64, 5, 1200, 33, 410], "decode_balanced"),
    ([1] * 40 + [17], [300 + i for i in range(40)] + [17], "decode")])
@pytest.mark.parametrize("Hq,Hkv", [(16, 8), (8, 1)])
@pytest.mark.parametrize("window", [0, 128])
def test_rows_beside_prompts(monkeypatch, q_lens, kv_lens, kernel, Hq, Hkv, window):
    kk, taken = K(), []
    rows_of = kk._decode_rows

    def watched(*a, beside=False, **kw):
        rows_of(*a, beside=beside, **kw)
        taken.append((kk.attention_path, beside))

    monkeypatch.setattr(kk, "_decode_rows", watched)
    ctx, bt, cu, kl, req, rs, kp = batch(q_lens, kv_lens, 16, 128, Hkv)
    vp = rnd(*kp.shape, seed=4, dtype=torch.bfloat16)
    T = sum(q_lens)
    source = rnd(T, (Hq + 2 * Hkv) * 128, seed=5, dtype=torch.bfloat16)
    qkv, weight = torch.empty_like(source), torch.ones(128, device="cuda")

    def run(pdl):
        kk.set_pdl(pdl)
        qkv.copy_(source)
        out = torch.full((T, Hq * 128), 7.0, dtype=torch.bfloat16, device="cuda")
        kk.qk_norm_in_place(qkv, Hq, Hkv, 128, weight, weight, 1e-6)  # (what the attention reads is written right in front of it)
        kk.paged_attention(qkv, out, kp, vp, bt, rs, cu, kl, req, Hq, Hkv, 128, 16, window, 128 ** -0.5, ctx)
        assert kk.attention_path == "prefill_tcgen05" and taken.pop() == (kernel, True) and not taken
        return out

    on = kk.pdl
    try:
        want = run(False)
        for _ in range(20):
            assert torch.equal(run(True), want)
    finally:
        kk.set_pdl(on)
    kk.raise_on_status()


def test_latent_rows_beside_prompts(monkeypatch):
    kk, Hq, dk, dv = K(), 16, 448, 384
    taken, attention = [], kk.windowed_attention

    def watched(*a, **kw):
        attention(*a, **kw)
        taken.append((kk.attention_path, kw.get("beside", False)))

    monkeypatch.setattr(kk, "windowed_attention", watched)
    q_lens, kv_lens = [1] * 12 + [900, 600], [60 + 150 * i for i in range(12)] + [900, 600]
    ctx, bt, cu, kl, req, rs, kp = batch(q_lens, kv_lens, 16, dk, 1)
    T = sum(q_lens)
    q = rnd(T, Hq * dk, seed=5, dtype=torch.bfloat16)

    def run(pdl):
        kk.set_pdl(pdl)
        out = torch.full((T, Hq * dv), 7.0, dtype=torch.bfloat16, device="cuda")
        kk.windowed_attention(q, out, kp, None, bt, rs, cu, kl, req, Hq, 1, dk, dv, 16, 0, 0.07, num_requests=len(q_lens),
                              workspace=ctx.workspace, ctx=ctx)
        # (the call for the rows ends before the call that it is part of)
        assert taken == [("window_mma", True), ("latent_tcgen05", False)] and kk.attention_path == "latent_tcgen05"
        taken.clear()
        return out

    on = kk.pdl
    try:
        want = run(False)
        for _ in range(20):
            assert torch.equal(run(True), want)
    finally:
        kk.set_pdl(on)
    kk.raise_on_status()
