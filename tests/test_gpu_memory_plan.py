"""The memory set aside for a step's scratch (`Part.step_scratch`) against what the workspace reserves at the first prompt, for every
mixer with a chunked form; the planes of a 32-bit product's rows."""

import pytest
import torch

import borosun_helpers as bh
import ludalix_helpers as lh
import mafarax_helpers as mh
import ninelix_helpers as nh
import plain_ludalix as pl
from helpers import random_ids

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


def ludalix(*sizes):
    cfg = lh.config(64, 97, [("mlstm", lh.mlstm(*size, 7.5), None) for size in sizes])
    return cfg, {n: t.bfloat16() for n, t in pl.random_weights(cfg, seed=5).items()}, 16


MODELS = {"one size": (lh, lambda: ludalix((2, 32, 48), (2, 32, 48))), "two sizes": (lh, lambda: ludalix((2, 32, 48), (1, 64, 80))),
          "borosun": (bh, lambda: bh.weights_for("D", "bfloat16")), "mafarax": (mh, lambda: mh.weights_for("E", "bfloat16")),
          "ninelix": (nh, lambda: nh.weights_for("F", "bfloat16"))}


@pytest.fixture
def always_chunks():
    """Every form with scratch at every size (steps as short as these take others)."""
    from test_gpu_kernels import K

    k = K()
    old = k.mlstm_chunk_on, k.gla_chunk_on, k.lib.ullm_ssd_chunk_short_pays
    k.mlstm_chunk_on, k.gla_chunk_on, k.lib.ullm_ssd_chunk_short_pays = 2, 2, lambda *a: 0
    yield
    k.mlstm_chunk_on, k.gla_chunk_on, k.lib.ullm_ssd_chunk_short_pays = old


@pytest.mark.parametrize("name", MODELS)
@pytest.mark.parametrize("max_requests", [1, 3, 9])
@pytest.mark.usefixtures("always_chunks")
def test_prompt_steps_reserve_what_the_plan_holds(tmp_path, name, max_requests):
    helpers, make = MODELS[name]
    cfg, w, page = make()
    r = helpers.make_runner(tmp_path, cfg, w, page, "bfloat16", max_requests=max_requests)
    planned = {}
    for (buffer, *_), size in r.model.step_scratch(64, max_requests).items():
        planned[buffer] = planned.get(buffer, 0) + size
    assert planned and r._activation_bytes() >= sum(planned.values()) + (512 << 20)

    def made():
        out = {}
        for (buffer, _cols, _dtype), t in r.workspace.buffers.items():
            if buffer.endswith(".chunks"):
                out[buffer] = out.get(buffer, 0) + t.numel() * t.element_size()
        return out

    # one short prompt, then the steps with the most chunks: one long prompt, and as many portions as bring more than 16 tokens
    most = min(max_requests, 64 // 17)
    shares = [64 // most + (1 if i < 64 % most else 0) for i in range(most)]
    for plan in ([("a", 20)], [("b", 64)], [(f"c{i}", n) for i, n in enumerate(shares)]):
        lh.replay(r, {rid: random_ids(cfg["vocab"], n, 3 + n) for rid, n in plan}, [plan])
        assert all(size <= planned[buffer] for buffer, size in made().items())
    if name == "one size":
        assert made() == planned
    # (rows of Borosun's input product whose length is no multiple of eight run token by token: reserved for, not made)
    assert made() or name == "borosun"


def test_planes_of_a_32_bit_product(tmp_path):
    from test_gpu_kernels import K

    M, k, N = 300, 132, 256
    x, w, out = (torch.randn(a, b, device="cuda") for a, b in ((M, k), (N, k), (M, N)))
    torch.cuda.synchronize()
    before = torch.cuda.memory_stats()["requested_bytes.all.allocated"]
    assert K().linear_f32_split(x, w, out)
    # rows of the planes end on 16-byte borders: up to four numbers more in each
    assert torch.cuda.memory_stats()["requested_bytes.all.allocated"] - before <= 6 * M * (k + 4)
    cfg, weights, page = bh.weights_for("D", "float32")
    r = bh.make_runner(tmp_path, cfg, weights, page, "float32")
    longest = max(t.shape[-1] for t in r.model.all_tensors().values() if t.dim() >= 2)
    assert r._activation_bytes() >= 64 * 6 * longest + (512 << 20)
