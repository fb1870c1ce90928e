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
