"""The clamped gate, xielu and the gated add in 16-byte pieces against references, where lengths or addresses allow pieces and where
not; the gated add with gates at infinities."""

import pytest
import torch

from test_gpu_kernels import K, rnd

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


def apply(kind, z, pq):
    if kind == "clamped":
        g, u = z.chunk(2, -1)
        g, u = g.clamp(max=1.5), u.clamp(-1.5, 1.5)
        return g * torch.sigmoid(1.702 * g) * (u + 1)
    a = torch.nn.functional.softplus(pq)
    neg = z.clamp(max=0)
    return torch.where(z > 0, a[0] * z * z + 0.5 * z, (0.5 + a[1]) * (torch.expm1(neg) - neg) + 0.5 * z)


@pytest.mark.parametrize("dtype,limit", [(torch.float32, 2e-6), (torch.bfloat16, 2 ** -8), (torch.float16, 2 ** -10)])
@pytest.mark.parametrize("rows,cols,shift", [(1, 8, 0), (3, 7, 0), (5, 96, 0), (2, 100, 0), (4, 64, 1)])
def test_row_kernels_in_pieces(dtype, limit, rows, cols, shift):
    kk, pq = K(), rnd(2, seed=54)
    x = rnd(rows * 2 * cols + shift, seed=55, dtype=dtype)[shift:].view(rows, 2 * cols)  # (shift: off the 16-byte border)
    out = torch.empty(rows, cols, dtype=dtype, device="cuda")
    kk.act_mul_clamped(x, out, 1.5, 1.702)
    ref = apply("clamped", x.float(), pq)
    assert (out.float() - ref).abs().max().item() <= limit * max(1.0, ref.abs().max().item())
    out = torch.empty_like(x)
    kk.xielu(x, pq, out)
    ref = apply("xielu", x.float(), pq)
    assert (out.float() - ref).abs().max().item() <= limit * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("dtype,limit", [(torch.float32, 2e-6), (torch.bfloat16, 2 ** -8), (torch.float16, 2 ** -10)])
@pytest.mark.parametrize("rows,cols,shift", [(1, 8, 0), (3, 7, 0), (5, 264, 0), (2, 100, 0), (4, 64, 1)])
@pytest.mark.parametrize("both", [True, False])
def test_gated_add(dtype, limit, rows, cols, shift, both):
    a, f = (rnd(rows * cols + shift, seed=s, dtype=dtype)[shift:].view(rows, cols) for s in (61, 62))
    n = 2 if both else 1
    g, b1, b2 = 4 * rnd(rows, n * cols, seed=63), rnd(cols, seed=64), rnd(cols, seed=65)
    stream, copy = rnd(rows, cols, seed=66), torch.empty(rows, cols, dtype=dtype, device="cuda")
    g[0, 0], g[0, 1], g[0, 2], g[0, 3] = 200.0, -200.0, float("inf"), float("-inf")
    ref = stream.double() + a.double() * torch.sigmoid(g[:, :cols].double() + b1.double())
    if both:
        ref += f.double() * torch.sigmoid(g[:, cols:].double() + b2.double())
    K().gated_add_f32(a, f if both else None, g, b1, b2 if both else None, stream, copy)
    assert (stream.double() - ref).abs().max().item() <= 1e-6 * max(1.0, ref.abs().max().item())
    assert (copy.double() - ref).abs().max().item() <= limit * max(1.0, ref.abs().max().item())


@pytest.mark.parametrize("shift", [0, 1])
def test_gated_add_through_gates_that_are_almost_shut(shift):
    """Denominators 1 + e^-z up to the largest 32-bit number: the quotient is that of a division (infinite ones give zero)."""
    z = torch.tensor([-60.0, -87.0, -87.3, -87.4, -87.5, -88.0, -88.5, -88.7, -89.0, -200.0], dtype=torch.float64).repeat(4)
    a = torch.tensor([1.0, -3.0, 1e30, -3e38], dtype=torch.float32).repeat_interleave(10)
    g, a = (torch.cat([torch.zeros(shift), v.float()]).cuda()[shift:].view(1, 40) for v in (z, a))  # (shift: off the 16-byte border)
    stream = torch.zeros(1, 40, device="cuda")
    K().gated_add_f32(a, None, g, torch.zeros(40, device="cuda"), None, stream)
    z64 = g.double()
    ref = torch.where(z64 < -88.72, 0.0, a.double() / (1 + torch.exp(-z64)))
    # a 32-bit exponential (2 units) and a quotient (2 more), 2^-24 each; results under 2^-126 by its smallest steps
    assert ((stream.double() - ref).abs() <= 4e-7 * ref.abs() + 3e-45).all()
