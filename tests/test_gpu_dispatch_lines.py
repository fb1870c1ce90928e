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
