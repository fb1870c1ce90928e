"""The chunked state-space recurrence without a workspace: scratch of the call's own is 32-bit whatever the program's default type."""

import pytest
import torch

from conftest import device
from test_gpu_kernels import K

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


@pytest.mark.parametrize("default", [torch.bfloat16, torch.float64])
def test_scratch_of_a_call_without_a_workspace(default):
    from ullm_b200.engine import Workspace

    kk, heads, n_state, pdim, T = K(), 4, 64, 32, 200
    f, d = torch.float32, device()
    g = torch.Generator().manual_seed(81)
    xbc = torch.randn(T, heads * pdim + 2 * n_state, generator=g).bfloat16().to(d)
    dt, log_decay = torch.rand(T, heads, generator=g).to(d), -0.1 * torch.rand(T, heads, generator=g).to(d)
    cu, req = torch.tensor([0, T], dtype=torch.int32, device=d), torch.zeros(T, dtype=torch.int32, device=d)

    def run(workspace):
        out, state = torch.empty(T, heads * pdim, dtype=f, device=d), torch.zeros(1, heads * pdim * n_state, dtype=f, device=d)
        scores = torch.empty(T, kk.ssd_chunk_floats(1, 1), dtype=f, device=d)
        kk.ssd_chunk(xbc, heads * pdim, heads * pdim + n_state, dt, log_decay, torch.ones(heads, dtype=f, device=d), scores, state, cu,
                     req[:1], req, out, 1, heads, n_state, pdim, 1, 16, workspace)
        return out, state

    ref = run(Workspace(d, T, 1))
    torch.set_default_dtype(default)
    try:
        got = run(None)
    finally:
        torch.set_default_dtype(torch.float32)
    assert all(torch.equal(a, b) for a, b in zip(got, ref))
