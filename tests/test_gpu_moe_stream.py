"""The routed experts' products of few tokens (csrc/moe_stream.cu) against a 32-bit reference and the mma.sync kernel: one token and
sixteen, every token at one expert and all at different ones, experts without tokens, choices that name no expert, weights on the
input, every activation, k that ends inside a block."""

import pytest
import torch

from test_gpu_kernels import K, rnd
from test_gpu_moe_tcgen05 import reference

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


@pytest.mark.parametrize("T,E,top,spread", [(1, 4, 2, True), (8, 16, 2, True), (9, 3, 3, True), (16, 40, 2, False), (16, 2, 1, False)])
@pytest.mark.parametrize("n_out,k", [(32, 64), (1024, 2048), (96, 832)])
@pytest.mark.parametrize("gated,act,weighted", [(True, 0, True), (True, 1, False), (True, 2, False), (False, 3, False), (False, -1, True)])
def test_streamed_experts_match_the_reference(T, E, top, spread, n_out, k, gated, act, weighted):
    kk = K()
    g = torch.Generator().manual_seed(61)
    choice = torch.stack([torch.randperm(E + 1, generator=g)[:top] if spread else (torch.arange(top) + 1) % E for _ in range(T)])
    choice = choice.int().cuda()  # (E: no expert's)
    total = T * top
    offsets = torch.empty(E + 1, dtype=torch.int32, device="cuda")
    order, place = torch.zeros(T, top, dtype=torch.int32, device="cuda"), torch.zeros(T, top, dtype=torch.int32, device="cuda")
    kk.moe_arrange(choice, total, E, offsets, order, place)
    w = rnd(E, (2 if gated else 1) * n_out, k, seed=62, dtype=torch.bfloat16, scale=k ** -0.5)
    weight = (rnd(T, top, seed=63).abs() + 0.1) if weighted else None
    live, at = (choice.view(-1) < E), place.view(-1).long()
    for from_pairs in (True, False):
        x = rnd(T if from_pairs else total, k, seed=64, dtype=torch.bfloat16)
        outs = []
        old = kk.moe_stream_tokens, kk.moe_tcgen05_rows
        try:
            for kk.moe_stream_tokens in (16, 0):
                kk.moe_tcgen05_rows = 1 << 30
                outs.append(torch.full((total, n_out), 9.0, dtype=torch.bfloat16, device="cuda"))
                kk.moe_grouped_linear(x, w, offsets, order, weight, outs[-1], top, from_pairs, gated, act, 3.0, 1.702)
        finally:
            kk.moe_stream_tokens, kk.moe_tcgen05_rows = old
        kk.raise_on_status()
        ref = reference(x, w, choice.cpu(), weight, top, from_pairs, gated, act, 3.0, 1.702, at)[live]
        got, gen = (o[at][live].float() for o in outs)
        s = max(ref.abs().max().item() if ref.numel() else 0.0, 1e-6)
        # one rounding to bfloat16 (2^-9 of the value) behind 32-bit sums of at most 2,048 products of order k^-1/2
        if ref.numel():
            assert (got - ref).abs().max().item() <= (2 ** -8 + 1e-4) * s
            assert (got - gen).abs().max().item() <= (2 ** -7 + 1e-4) * s
        assert (outs[0][int(live.sum()):] == 9.0).all()


@pytest.mark.parametrize("T,top,n_out,k", [(1, 4, 32, 64), (1, 9, 96, 192), (7, 3, 64, 128), (16, 2, 64, 320), (16, 32, 32, 64)])
@pytest.mark.parametrize("gated,act,weighted", [(True, 0, True), (False, -1, True), (False, 3, False)])
@pytest.mark.parametrize("kind", ["one expert", "repeated", "mixed"])
def test_a_token_may_name_an_expert_more_than_once(T, top, n_out, k, gated, act, weighted, kind):
    """The product is defined for any choices: places of one token at one expert, and more places of an expert than tokens."""
    kk, E = K(), 5
    g = torch.Generator().manual_seed(67)
    choice = {"one expert": torch.full((T, top), 3), "repeated": torch.randint(0, 2, (T, top), generator=g),
              "mixed": torch.randint(0, E + 1, (T, top), generator=g)}[kind].int().cuda()
    total = T * top
    offsets = torch.empty(E + 1, dtype=torch.int32, device="cuda")
    order, place = torch.zeros(T, top, dtype=torch.int32, device="cuda"), torch.zeros(T, top, dtype=torch.int32, device="cuda")
    kk.moe_arrange(choice, total, E, offsets, order, place)
    w = rnd(E, (2 if gated else 1) * n_out, k, seed=62, dtype=torch.bfloat16, scale=k ** -0.5)
    weight = (rnd(T, top, seed=63).abs() + 0.1) if weighted else None
    live, at = (choice.view(-1) < E), place.view(-1).long()
    for from_pairs in (True, False):
        x = rnd(T if from_pairs else total, k, seed=64, dtype=torch.bfloat16)
        out = torch.full((total, n_out), 9.0, dtype=torch.bfloat16, device="cuda")
        kk.moe_grouped_linear(x, w, offsets, order, weight, out, top, from_pairs, gated, act, 3.0, 1.702)
        kk.raise_on_status()
        ref = reference(x, w, choice.cpu(), weight, top, from_pairs, gated, act, 3.0, 1.702, at)[live]
        # (one rounding to bfloat16 behind sums of at most 320 products, as above)
        assert (out[at][live].float() - ref).abs().max().item() <= (2 ** -8 + 1e-4) * max(ref.abs().max().item(), 1e-6)
        assert (out[int(live.sum()):] == 9.0).all()
