"""Steps of every model with programmatic dependent launch give the bits of steps whose kernels wait for one another's ends: prompts,
portions of prompts, prompts beside decoded tokens, decoded tokens alone."""

import importlib

import pytest
import torch

import tiny_configs
from helpers import random_ids
from test_gpu_kernels import K

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]

WIDE = dict(tiny_configs.TINY_A, num_hidden_layers=6, hidden_size=256, head_dim=128, intermediate_size=512, vocab_size=1000,
            max_position_embeddings=1024)
MODELS = [("qwen3", "wide")] + [("qwen3", tag) for tag in sorted(tiny_configs.ALL)]
for _name in ("borosun", "finosun", "ludalix", "mafarax", "ninelix", "pidenex"):
    # (ninelix B, C and D take the size of their distance table from a checkpoint)
    MODELS += [(_name, tag) for tag in sorted(importlib.import_module(_name + "_helpers").CONFIGS) if _name != "ninelix" or tag not in "BCD"]


def config(name, tag):
    if name != "qwen3":
        return importlib.import_module(name + "_helpers").CONFIGS[tag]
    return (WIDE, 16) if tag == "wide" else (tiny_configs.ALL[tag][0], tiny_configs.ALL[tag][2])


def steps(cfg, page, dtype):
    from ullm_b200.engine import ModelRunner, StepEntry

    r = ModelRunner(config=cfg, dtype=dtype, page_size=page, num_pages=8 * -(-128 // page), max_requests=6, max_context=110,
                    max_step_tokens=256, load_format="random", seed=3, random_std=0.05)
    vocab = r.spec.vocab_size
    ids = [random_ids(vocab, 110, 7 + i) for i in range(6)]
    at, out = [0] * 6, []

    def step(*lengths):
        entries = []
        for i, n in lengths:
            entries.append(StepEntry(str(i), ids[i][at[i]:at[i] + n], [n - 1]))
            at[i] += n
        out.append(r.step(entries).clone())

    for i in range(6):
        r.add_request(str(i))
    step((0, 70), (1, 33))
    step((2, 20))
    step((0, 1), (1, 1), (2, 1), (3, 90))
    step((3, 1), (4, 17), (5, 64), (2, 30))
    for _ in range(3):
        step(*((i, 1) for i in range(6)))
    r.check_device_status()
    return out


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("name,tag", MODELS)
def test_the_bits_do_not_depend_on_it(name, tag, dtype):
    kk, (cfg, page) = K(), config(name, tag)
    on = kk.pdl
    try:
        kk.set_pdl(False)
        want = steps(cfg, page, dtype)
        kk.set_pdl(True)
        for _ in range(2):
            for a, b in zip(steps(cfg, page, dtype), want):
                assert torch.equal(a, b)
    finally:
        kk.set_pdl(on)
