"""The norm-and-add row kernel with a row in registers and with a row in shared memory (csrc/sandwich_norm.cu) against 64 bits: rows of
one piece, of a part of a warp, of the longest block, beyond it, and of no whole pieces; every norm on either side."""

import pytest
import torch

from test_gpu_kernels import K, rnd

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


def norm(v, w, eps, center):
    v = v - v.mean(-1, keepdim=True) if center else v
    return w * v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps)


@pytest.mark.parametrize("cols,shift", [(8, 0), (264, 0), (2048, 0), (8192, 0), (8200, 0), (100, 0), (256, 1)])
@pytest.mark.parametrize("dtype,out_dtype", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32),
                                             (torch.float32, torch.bfloat16), (torch.float32, torch.float32), (torch.float16, torch.float16)])
def test_rows(cols, shift, dtype, out_dtype):
    rows, eps, limit = 3, 1e-5, {torch.float32: 3e-6, torch.bfloat16: 2 ** -8, torch.float16: 2 ** -10}[out_dtype]
    w, w2, b2, vec, al = rnd(cols, seed=1), rnd(cols, seed=2), rnd(cols, seed=3), rnd(cols, seed=4), torch.tensor([0.3], device="cuda")
    for first in ("rms", "center", "plain", "scale", None):
        for second in (0, 1, 2, 3, None):
            a = rnd(rows * cols + shift, seed=5, dtype=dtype)[shift:].view(rows, cols) if first else None
            stream, extra = rnd(rows, cols, seed=6), rnd(rows, cols, seed=7) if second else None
            out = torch.full((rows, cols), 9.0, dtype=out_dtype, device="cuda")
            ref = stream.double()
            if first:
                ad = a.double()
                ref = ref + 0.5 * {"rms": lambda: norm(ad, w.double(), eps, False), "center": lambda: norm(ad, w.double(), eps, True),
                                   "plain": lambda: ad, "scale": lambda: ad * w.double()}[first]()
            args = {}
            if extra is not None:
                ref, args = ref + extra.double() + vec.double(), dict(extra_rows=extra, extra_vec=vec)
            follow = {0: (w2, eps, 0, out), 1: (w2, eps, 1, out), 2: (w2, 0.0, 2, al, b2, out), 3: (None, 0.0, 3, out), None: None}[second]
            K().norm_add_norm(stream, a, w if first in ("rms", "center", "scale") else None, eps, 0.5, center=first == "center",
                              plain=first in ("plain", "scale"), next_norm=follow, **args)
            assert (stream.double() - ref).abs().max().item() <= 3e-6 * max(1.0, ref.abs().max().item()), (first, second)
            if second is not None:
                want = {0: lambda: norm(ref, w2.double(), eps, False), 1: lambda: norm(ref, w2.double(), eps, True),
                        2: lambda: torch.tanh(0.3 * ref) * w2.double() + b2.double(), 3: lambda: ref}[second]()
                assert (out.double() - want).abs().max().item() <= limit * max(1.0, want.abs().max().item()), (first, second)
