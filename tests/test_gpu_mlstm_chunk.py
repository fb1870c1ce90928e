"""The chunked matrix-memory recurrence (csrc/mlstm_chunk.cu) against the recurrence in 64 bits and against the token-by-token
kernel: chunks that end early, several requests beside short ones, state carried from portion to portion, gates that forget at
once and never, a maximum that stays and one that moves."""

import pytest
import torch

from conftest import device
from test_gpu_kernels import K

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


def recurrence(q, k, v, gi, gf, S, n, m):
    out = torch.zeros(q.shape[0], q.shape[1], v.shape[2], dtype=q.dtype, device=q.device)
    for t in range(q.shape[0]):
        m2 = torch.maximum(gf[t] + m, gi[t])
        keep, take = torch.exp(gf[t] + m - m2), torch.exp(gi[t] - m2)
        m = m2
        S = keep[:, None, None] * S + take[:, None, None] * v[t][:, :, None] * k[t][:, None, :]
        n = keep[:, None] * n + take[:, None] * k[t]
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
        out[t] = (S * q[t][:, None, :]).sum(-1) / den[:, None]
    return out, S, n, m


@pytest.mark.parametrize("heads,dim,vdim", [(2, 16, 16), (3, 128, 256), (1, 48, 144), (2, 256, 512)])
@pytest.mark.parametrize("lens", [[64], [65, 3, 1, 130], [17, 16, 63, 200]])
@pytest.mark.parametrize("forget", [-6.0, 0.0, 6.0])
def test_chunks_match_the_recurrence(heads, dim, vdim, lens, forget):
    from ullm_b200.engine import Workspace

    kk, least, cap, scale = K(), 16, 15.0, dim ** -0.5
    g = torch.Generator().manual_seed(3)
    T, B = sum(lens), len(lens)
    size = 2 * heads * dim + heads * vdim
    qkv = torch.randn(T, size + 16, generator=g).bfloat16().to(device())
    gates = (2.0 * torch.randn(T, 2 * heads, generator=g)).to(device())
    bi, bf = torch.randn(heads, generator=g).to(device()), (forget + torch.randn(heads, generator=g)).to(device())
    floats = heads * dim * (vdim + 1) + heads
    stride = -(-floats // 4) * 4
    state0 = torch.randn(B + 1, stride, generator=g).to(device())
    slots = torch.randperm(B + 1, generator=g)[:B].int().to(device())
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=device())
    req = torch.cat([torch.full((n,), r, dtype=torch.int32) for r, n in enumerate(lens)]).to(device())

    def run(chunked):
        state, out = state0.clone(), torch.full((T, heads * vdim), 5.0, device=device())
        args = (qkv, 0, heads * dim, 2 * heads * dim, gates, bi, bf, state, cu, slots, req, out, B, heads, dim, vdim, scale, cap)
        if chunked:
            assert kk.mlstm_chunk(*args, Workspace(device(), T, B), least)
            kk.mlstm_recurrence(*args, most_tokens=least)
        else:
            kk.mlstm_recurrence(*args)
        kk.raise_on_status()
        return out.double().cpu(), state.double().cpu()

    got, state = run(True)
    plain, state_p = run(False)
    x = qkv.double().cpu()
    q = x[:, :heads * dim].view(T, heads, dim) * scale
    k = x[:, heads * dim:2 * heads * dim].view(T, heads, dim)
    v = x[:, 2 * heads * dim:size].view(T, heads, vdim)
    gd = gates.double().cpu()
    gi = cap * torch.tanh((gd[:, :heads] + bi.double().cpu()) / cap)
    gf = torch.nn.functional.logsigmoid(cap * torch.tanh((gd[:, heads:] + bf.double().cpu()) / cap))
    ref, worst = torch.zeros(T, heads, vdim, dtype=torch.float64), 0.0
    for r, n in enumerate(lens):
        a, s = int(cu[r]), state0[int(slots[r])].double().cpu()
        S, nn, m = s[:heads * dim * vdim].view(heads, vdim, dim), s[heads * dim * vdim:heads * dim * (vdim + 1)].view(heads, dim), \
            s[heads * dim * (vdim + 1):floats]
        ref[a:a + n], S, nn, m = recurrence(q[a:a + n], k[a:a + n], v[a:a + n], gi[a:a + n], gf[a:a + n], S, nn, m)
        want = torch.cat([S.reshape(-1), nn.reshape(-1), m])
        have = state[int(slots[r])][:floats]
        worst = max(worst, float((have - want).norm() / want.norm()))
    untouched = [i for i in range(B + 1) if i not in slots.tolist()]
    assert torch.equal(state[untouched], state0.double().cpu()[untouched])

    def err(o):
        return float((o.view(T, heads, vdim) - ref).norm() / ref.norm())

    print(f"chunks {err(got):.2e}, token by token {err(plain):.2e}, state {worst:.2e}")
    # 32-bit sums: 1e-6 where nothing cancels.  Where the terms of the denominator cancel (long memories: up to 2e-5 here) the
    # loss is the inputs' and the token-by-token kernel has it too: at most twice its distance
    assert err(got) < 2.0 * err(plain) + 1e-6 and worst < 2e-6


def inputs(heads, dim, vdim, lens, seed=3, forget=2.0):
    g = torch.Generator().manual_seed(seed)
    T, B = sum(lens), len(lens)
    qkv = torch.randn(T, 2 * heads * dim + heads * vdim, generator=g).bfloat16().to(device())
    gates = (2.0 * torch.randn(T, 2 * heads, generator=g)).to(device())
    bi, bf = torch.randn(heads, generator=g).to(device()), (forget + torch.randn(heads, generator=g)).to(device())
    state = torch.randn(B, heads * dim * (vdim + 1) + heads, generator=g).to(device())
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=device())
    req = torch.cat([torch.full((n,), r, dtype=torch.int32) for r, n in enumerate(lens)]).to(device())
    return qkv, gates, bi, bf, state, torch.arange(B, dtype=torch.int32, device=device()), cu, req


@pytest.mark.parametrize("heads,dim,vdim", [(8, 128, 256), (4, 256, 512), (2, 40, 300)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("lens", [[1] * 70, [300, 150, 40], [9, 2, 14] * 20, [120] * 6 + [3] * 12])
def test_token_by_token_does_not_depend_on_the_other_requests(heads, dim, vdim, dtype, lens):
    """More blocks than the chip holds at once: a block that starts behind others of its request and head that are done already
    begins from the same state as they.  Every request alone gives the same bits."""
    from ullm_b200.engine import Workspace

    kk = K()
    qkv, gates, bi, bf, state0, slots, cu, req = inputs(heads, dim, vdim, lens)
    qkv = qkv.to(dtype)
    T, B, ws = sum(lens), len(lens), Workspace(device(), sum(lens), len(lens))

    def run(lo, hi, which, workspace):
        n = len(which)
        out, state = torch.empty(hi - lo, heads * vdim, device=device()), state0.clone()
        kk.mlstm_recurrence(qkv[lo:hi], 0, heads * dim, 2 * heads * dim, gates[lo:hi], bi, bf, state, (cu[which[0]:which[-1] + 2] - lo),
                            slots[which[0]:which[-1] + 1], req[lo:hi] - which[0], out, n, heads, dim, vdim, dim ** -0.5, 15.0,
                            workspace=workspace)
        kk.raise_on_status()
        return out, state

    for workspace in (ws, ws, None):  # (the counters are zeros again behind a launch)
        out, state = run(0, T, list(range(B)), workspace)
        for r in {0, 1, B // 2, B - 2, B - 1}:
            a, b = int(cu[r]), int(cu[r + 1])
            one, one_state = run(a, b, [r], None)
            assert torch.equal(out[a:b], one) and torch.equal(state[r], one_state[r])


@pytest.mark.parametrize("heads,dim,vdim", [(8, 128, 256), (4, 256, 512)])
@pytest.mark.parametrize("lens", [[700], [500, 130]])
def test_error_against_64_bits_is_not_above_the_token_by_token_kernels(heads, dim, vdim, lens):
    """Long memories at the sizes of whole models: the typical error of an output row (a median, which the few rows whose denominator
    cancels do not decide) is not above the one of ordinary 32-bit sums."""
    from ullm_b200.engine import Workspace

    kk = K()
    for forget in (2.0, 6.0):
        qkv, gates, bi, bf, state0, slots, cu, req = inputs(heads, dim, vdim, lens, forget=forget)
        T, B, cap, scale = sum(lens), len(lens), 15.0, dim ** -0.5
        x, gd = qkv.double(), gates.double()
        q, k = (x[:, i * heads * dim:(i + 1) * heads * dim].view(T, heads, dim) for i in (0, 1))
        v = x[:, 2 * heads * dim:].view(T, heads, vdim)
        gi = cap * torch.tanh((gd[:, :heads] + bi.double()) / cap)
        gf = torch.nn.functional.logsigmoid(cap * torch.tanh((gd[:, heads:] + bf.double()) / cap))
        ref = torch.zeros(T, heads, vdim, dtype=torch.float64, device=device())
        for r in range(B):
            a, b, s = int(cu[r]), int(cu[r + 1]), state0[r].double()
            parts = s[:heads * dim * vdim].view(heads, vdim, dim), s[heads * dim * vdim:-heads].view(heads, dim), s[-heads:]
            ref[a:b] = recurrence(q[a:b] * scale, k[a:b], v[a:b], gi[a:b], gf[a:b], *parts)[0]
        typical = []
        for chunked in (True, False):
            state, out = state0.clone(), torch.empty(T, heads * vdim, device=device())
            args = (qkv, 0, heads * dim, 2 * heads * dim, gates, bi, bf, state, cu, slots, req, out, B, heads, dim, vdim, scale, cap)
            if chunked:
                assert kk.mlstm_chunk(*args, Workspace(device(), T, B), 16)
            else:
                kk.mlstm_recurrence(*args)
            d = (out.double().view(T, heads, vdim) - ref).norm(dim=-1) / ref.norm(dim=-1)
            typical.append(float(d.median()))
        print(f"forget {forget}: chunks {typical[0]:.2e}, token by token {typical[1]:.2e}")
        # (a tenth: the spread of the median between seeds)
        assert typical[0] <= 1.1 * typical[1]


@pytest.mark.parametrize("where", ["v inf", "v nan", "k nan", "forget gate nan", "input gate nan"])
@pytest.mark.parametrize("at", [20, 21, 63, 64, 75])
def test_what_is_not_finite_does_not_reach_earlier_tokens(where, at):
    from ullm_b200.engine import Workspace

    kk, heads, dim, vdim, lens = K(), 2, 32, 48, [100]
    qkv, gates, bi, bf, state0, slots, cu, req = inputs(heads, dim, vdim, lens)

    def run():
        out = torch.empty(100, heads * vdim, device=device())
        assert kk.mlstm_chunk(qkv, 0, heads * dim, 2 * heads * dim, gates, bi, bf, state0.clone(), cu, slots, req, out, 1, heads, dim, vdim,
                              dim ** -0.5, 15.0, Workspace(device(), 100, 1), 16)
        return out.view(100, heads, vdim)

    clean, value = run(), float("inf" if where == "v inf" else "nan")
    if where[0] == "v":
        qkv[at, 2 * heads * dim + vdim + 5] = value  # head 1, column 5
    elif where[0] == "k":
        qkv[at, heads * dim + dim + 5] = value
    else:
        gates[at, (heads if where[0] == "f" else 0) + 1] = value
    out = run()
    # (the sums of a chunk that holds such a value run in another order)
    assert torch.isfinite(out[:at]).all() and float((out[:at] - clean[:at]).norm() / clean[:at].norm()) < 1e-5
    assert torch.equal(out[:, 0], clean[:, 0]) or where[0] == "v" and torch.isfinite(out[:, 0]).all()
    assert not torch.isfinite(out[at, 1, 5])
