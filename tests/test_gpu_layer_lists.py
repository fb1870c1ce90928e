"""Layers that run from another layer's list of launches: the same logits, bit for bit, as layers that launch for themselves, and
lists only where nothing else runs between the launches."""

import pytest
import torch

from helpers import random_ids

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


def config(layers=6, **more):
    return dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=layers, hidden_size=256, num_attention_heads=4,
                num_key_value_heads=2, head_dim=128, intermediate_size=512, vocab_size=1000, rope_theta=10000.0, rms_norm_eps=1e-6,
                attention_bias=False, tie_word_embeddings=True, max_position_embeddings=1024, torch_dtype="bfloat16", **more)


def steps(cfg, on, dtype="bfloat16"):
    """Prompts, a portion of one, and mixed steps with few and many decoded rows in front; (logits, layers that ran from a list)."""
    from ullm_b200.csrc import kernels
    from ullm_b200.engine import ModelRunner, StepEntry

    K = kernels()
    r = ModelRunner(config=cfg, dtype=dtype, page_size=16, num_pages=120, max_requests=8, max_context=256, max_step_tokens=512,
                    load_format="random", seed=3, random_std=0.05)
    ids = [random_ids(cfg["vocab_size"], 200, 7 + i) for i in range(7)]
    K.layer_lists, before, launches = on, K.listed_layers, K.launches
    out = []
    try:
        for i in range(7):
            r.add_request(str(i))
        out.append(r.step([StepEntry(str(i), ids[i][:40 + 9 * i], [39 + 9 * i]) for i in range(3)]).clone())
        out.append(r.step([StepEntry("3", ids[3][:20], [19])]).clone())
        out.append(r.step([StepEntry(str(i), [ids[i][100 + i]], [0]) for i in range(3)] + [StepEntry("4", ids[4][:150], [149])]).clone())
        out.append(r.step([StepEntry(str(i), [ids[i][120 + i]], [0]) for i in range(5)] + [StepEntry("5", ids[5][:33], [32]),
                                                                                         StepEntry("6", ids[6][:190], [3, 189])]).clone())
        out.append(r.step([StepEntry("6", [ids[6][190]], [0])]).clone())  # (a decode step: no list)
        r.check_device_status()
    finally:
        K.layer_lists = True
    return out, K.listed_layers - before, K.launches - launches


@pytest.mark.parametrize("layers,listed", [(6, 12), (5, 8), (4, 0)])
def test_listed_layers_form_the_same_logits(layers, listed):
    own, none, launches = steps(config(layers), False)
    got, ran, same = steps(config(layers), True)
    assert none == 0 and ran == listed and same == launches
    for a, b in zip(own, got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("cfg,dtype,listed", [(config(), "float32", 0), (dict(config(), attention_bias=True), "bfloat16", 3)])
def test_layers_with_other_work_between_the_launches_run_for_themselves(cfg, dtype, listed):
    """float32 products allocate their planes, and products with a bias are torch's (but for the step of 20 tokens: the stream
    kernel's)."""
    own, _, _ = steps(cfg, False, dtype)
    got, ran, _ = steps(cfg, True, dtype)
    assert ran == listed and all(torch.equal(a, b) for a, b in zip(own, got))


def test_no_lists_while_a_measurement_runs():
    from ullm_b200.csrc import kernels

    K = kernels()
    K.skip_groups = frozenset({"sampling"})
    try:
        assert steps(config(), True)[1] == 0
    finally:
        K.skip_groups = frozenset()
