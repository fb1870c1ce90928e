"""Which layers may run from another layer's list of launches: those of the parts as they are written, and no others (no GPU: the lists
themselves are a stand-in's)."""

from types import SimpleNamespace

import pytest

from cpu_kernels import CpuKernels
from helpers import random_ids
from ullm_b200 import csrc
from ullm_b200.csrc import ops, set_kernels
from ullm_b200.parts.mlp import GatedMLP
from ullm_b200.parts.model import _same
from ullm_b200.parts.norm import RMSNorm
from ullm_b200.parts.registry import FEED_FORWARDS, NORMS


class Listing(CpuKernels):
    """Runs a list by running the layer it stands for, so that the results stay right, and counts."""

    def __init__(self):
        super().__init__()
        self.listed = 0

    def lists_apply(self):
        return True

    def record_launches(self, run):
        return run(), "list"

    def lists_alike(self, a, tensors_a, b, tensors_b):
        return [t.shape for t in tensors_a] == [t.shape for t in tensors_b]

    def run_list(self, listed, tensors):
        self.listed += 1
        return True


CONFIG = dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=6, hidden_size=64, num_attention_heads=2, num_key_value_heads=1,
              head_dim=32, intermediate_size=96, vocab_size=200, rope_theta=10000.0, rms_norm_eps=1e-6, attention_bias=False,
              tie_word_embeddings=True, max_position_embeddings=256, torch_dtype="float32")


def run(prepare=None):
    """Layers that ran from a list in a step of one prompt."""
    from ullm_b200.engine import ModelRunner, StepEntry

    K, before = Listing(), csrc._KERNELS
    set_kernels(K)
    try:
        r = ModelRunner(config=CONFIG, dtype="float32", page_size=16, num_pages=16, max_requests=2, max_context=64, max_step_tokens=64,
                        load_format="random", seed=3, device="cpu")
        if prepare is not None:
            prepare(r.model)
        r.add_request("a")
        r.step([StepEntry("a", random_ids(200, 9, 1), [8])])
        return K.listed
    finally:
        set_kernels(before)


def test_layers_of_plain_parts_run_from_a_list():
    assert run() == 3


@pytest.mark.parametrize("table,kind,cls", [(FEED_FORWARDS, "gated_mlp", GatedMLP), (NORMS, "rmsnorm", RMSNorm)])
def test_a_subclass_runs_itself(monkeypatch, table, kind, cls):
    """It may do more than launch kernels, also where it leaves `forward` as it is."""
    ran = []

    class More(cls):
        def forward(self, *a, **kw):
            ran.append(self)
            return super().forward(*a, **kw)

    class Same(cls):
        pass

    for sub in (More, Same):
        monkeypatch.setitem(table, kind, sub)
        assert run() == 0
    assert len({id(p) for p in ran}) >= 6  # (every layer's)


def test_a_forward_put_in_its_place_is_called():
    called = []

    def replace(model):
        part = model.blocks[4].feed_forward
        forward = part.forward
        part.forward = lambda *a, **kw: called.append(4) or forward(*a, **kw)

    assert run(replace) == 1 and called == [4]  # (layer 3 runs from the list, 4 and what is behind it run themselves)


def test_a_forward_put_on_the_class_is_called(monkeypatch):
    called = []
    forward = GatedMLP.forward
    monkeypatch.setattr(GatedMLP, "forward", lambda self, *a, **kw: called.append(self) or forward(self, *a, **kw))
    assert run() == 0 and len(called) == 6


def test_specs_differ_in_fields_that_their_comparison_leaves_out():
    import dataclasses

    @dataclasses.dataclass
    class S:
        a: int
        b: int = dataclasses.field(default=0, compare=False)

    assert _same([S(1, 2)], [S(1, 2)]) and not _same([S(1, 2)], [S(1, 3)])
    assert not _same({"x": (S(1, 2),)}, {"x": (S(1, 3),)}) and not _same({"x": 1}, {"y": 1})


def test_a_list_that_is_refused_leaves_the_layer_to_itself(monkeypatch):
    monkeypatch.setattr(Listing, "run_list", lambda self, listed, tensors: False)
    called = []
    forward = GatedMLP.forward
    monkeypatch.setattr(GatedMLP, "forward", lambda self, *a, **kw: called.append(self) or forward(self, *a, **kw))
    monkeypatch.setattr(GatedMLP, "written_forward", GatedMLP.forward)
    assert run() == 0 and len(called) == 6


@pytest.mark.parametrize("code,says", [(4, ops._ERRORS[4]), (-7, "cublasGemmEx answered 7"), (99, "error 99")])
def test_a_list_that_fails_says_whose_error_it_was(monkeypatch, code, says):
    monkeypatch.setattr(ops, "_native", SimpleNamespace(replay=lambda tape, tensors: code))
    k = ops.Kernels.__new__(ops.Kernels)
    with pytest.raises(ops.KernelError) as e:
        k.run_list(("list", 3), ())
    assert says in str(e.value)
