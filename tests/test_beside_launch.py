"""Decode attention beside the prompt attention of the same step: launched so only where the prompt kernel is the launch right in
front of it (csrc/decode_core.cuh)."""

from types import SimpleNamespace

import torch

from ullm_b200.csrc import ops


def test_a_call_that_fills_its_scratch_first_does_not_run_beside(monkeypatch):
    """The first call of a head shape makes and clears its arrays, behind the prompt kernel: it waits as always."""
    queue = []
    monkeypatch.setattr(ops, "_ptr", lambda t: 0 if t is None else t.data_ptr())
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    empty, zeros = torch.empty, torch.zeros
    monkeypatch.setattr(torch, "empty", lambda *size, device=None, **kw: empty(*size, **kw))
    monkeypatch.setattr(torch, "zeros", lambda *size, device=None, **kw: queue.append("fill") or zeros(*size, **kw))
    k = ops.Kernels.__new__(ops.Kernels)
    k._decb, k.launches, k.status = {}, 0, empty(4, dtype=torch.int32)
    k._decode_choice = lambda *a: "balanced"
    k.lib = SimpleNamespace(ullm_decode_attention_balanced=lambda *a: queue.append(a[-1]) or 0,
                            ullm_decode_attention_balanced_scratch_floats=lambda *a: 8, ullm_decode_attention_tcgen05_scratch_floats=lambda *a: 8)
    t = empty(4, 512)
    for beside in (True, True, False):
        queue.clear()
        k._decode_rows(t, t, t, t, t, t, t, 2, 1, 128, 16, 0, 1.0, 4, True, None, rows=2, beside=beside)
        assert queue[-1] == int(beside and "fill" not in queue)
    assert queue == [0]
