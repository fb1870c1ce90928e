"""The chunked recurrence with a decay per key channel (csrc/gla_chunk.cu) at sizes whose value columns go to several blocks, and
whose last block of columns is narrower, against the token-by-token kernel."""

import pytest
import torch

from conftest import device
from test_gpu_kernels import K

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


@pytest.mark.parametrize("heads,dim,vdim", [(2, 128, 256), (1, 256, 512), (2, 128, 208), (1, 240, 272), (3, 64, 256)])
@pytest.mark.parametrize("lens", [[64, 17], [130, 3, 65]])
def test_value_tiles_match_the_recurrence(heads, dim, vdim, lens):
    from ullm_b200.engine import Workspace

    kk, least = K(), 16
    assert kk.gla_chunk_applies(torch.bfloat16, heads, dim, vdim)
    g = torch.Generator().manual_seed(71)
    T, B = sum(lens), len(lens)
    size = 2 * heads * dim + heads * vdim
    y = torch.randn(T, size, generator=g).bfloat16().to(device())
    z = (2.0 + torch.randn(T, heads * dim, generator=g)).to(device())
    bias = torch.randn(heads * dim, generator=g).to(device())
    state0 = torch.randn(B + 1, heads * dim * vdim, generator=g).to(device())
    slots = torch.randperm(B + 1, generator=g)[:B].int().to(device())
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=device())
    req = torch.cat([torch.full((n,), r, dtype=torch.int32) for r, n in enumerate(lens)]).to(device())
    outs, states = [], []
    for chunked in (True, False):
        w, state, out = z.clone(), state0.clone(), torch.full((T, heads * vdim), 5.0, device=device())
        args = (y, 0, heads * dim, 2 * heads * dim)
        if chunked:
            kk.gla_decay(w, bias, 1 / 8.0)
            assert (w - torch.exp(torch.nn.functional.logsigmoid(z + bias) / 8.0)).abs().max().item() < 1e-6
            kk.gla_chunk(*args, w, dim ** -0.5, kk.gla_chunk_scratch(Workspace(device(), T, B), T, B, heads, dim, vdim), state, cu,
                         slots, req, out, B, heads, dim, vdim, least)
            kk.gla_recurrence(*args, w, None, 0.0, dim ** -0.5, state, cu, slots, req, out, B, heads, dim, vdim, most_tokens=least)
        else:
            kk.gla_recurrence(*args, w, bias, 1 / 8.0, dim ** -0.5, state, cu, slots, req, out, B, heads, dim, vdim)
        kk.raise_on_status()
        outs.append(out.double())
        states.append(state.double())
    # three bfloat16 terms keep 24 bits of every 32-bit operand: both sides differ by the rounding of 32-bit sums and products (2^-24
    # each): of up to 130 decays one after the other, of sums over up to 256 channels and 130 tokens, at most sqrt(130 + 256 + 130)
    # roundings' worth when they are independent
    assert float((outs[0] - outs[1]).norm() / outs[1].norm()) < 2.0 ** -24 * 516 ** 0.5
    assert float((states[0] - states[1]).norm() / states[1].norm()) < 2.0 ** -24 * 516 ** 0.5


@pytest.mark.parametrize("bonus", [False, True])
@pytest.mark.parametrize("at,value", [(20, float("inf")), (21, float("nan")), (63, float("inf")), (64, float("nan")), (75, float("inf"))])
def test_a_value_that_is_not_finite_does_not_reach_earlier_tokens(bonus, at, value):
    from ullm_b200.engine import Workspace

    kk, heads, dim, vdim, T = K(), 2, 32, 144, 100
    g = torch.Generator().manual_seed(72)
    y = torch.randn(T, 2 * heads * dim + heads * vdim, generator=g).bfloat16().to(device())
    w = torch.sigmoid(2.0 + torch.randn(T, heads * dim, generator=g)).to(device())
    u = torch.randn(heads * dim, generator=g).to(device()) if bonus else None
    cu, req = torch.tensor([0, T], dtype=torch.int32, device=device()), torch.zeros(T, dtype=torch.int32, device=device())

    def run():
        out, state = torch.empty(T, heads * vdim, device=device()), torch.zeros(1, heads * dim * vdim, device=device())
        kk.gla_chunk(y, 0, heads * dim, 2 * heads * dim, w, dim ** -0.5, kk.gla_chunk_scratch(Workspace(device(), T, 1), T, 1, heads, dim, vdim),
                     state, cu, req[:1], req, out, 1, heads, dim, vdim, 16, bonus=u)
        return out.view(T, heads, vdim)

    clean = run()
    y[at, 2 * heads * dim + vdim + 133] = value  # head 1, column 133
    out = run()
    # (the sums of a warp's own tokens run in another order; two terms of an operand with a bonus)
    assert torch.isfinite(out[:at]).all() and float((out[:at] - clean[:at]).norm() / clean[:at].norm()) < (1e-4 if bonus else 1e-5)
    other = torch.ones(heads, vdim, dtype=torch.bool)
    other[1, 133] = False
    assert torch.isfinite(out[:, other]).all() and not torch.isfinite(out[at:, 1, 133]).any()
