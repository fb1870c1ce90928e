"""float32 products in three bfloat16 terms per operand (csrc/linear_f32_split.cu) against products in 64 bits: edges of the tiles
of rows, columns and k, a bias, operands of very different size, infinities and NaN."""

import pytest
import torch

from conftest import device
from test_gpu_kernels import K

pytestmark = [pytest.mark.gpu, pytest.mark.needs_cuda]


def run(x, w, bias=None):
    kk, out = K(), torch.full((x.shape[0], w.shape[0]), 9.0, device=device())
    old, kk.f32_split_rows, kk.f32_split_results = (kk.f32_split_rows, kk.f32_split_results), 1, 0
    try:
        assert kk.linear_f32_split(x, w, out, bias)
    finally:
        kk.f32_split_rows, kk.f32_split_results = old
    kk.raise_on_status()
    return out


@pytest.mark.parametrize("M,N,k", [(1, 4, 4), (128, 128, 64), (129, 132, 68), (511, 1024, 3072), (300, 6144, 1024), (40, 100, 60),
                                   (512, 4096, 1024), (257, 2052, 132), (1000, 32, 2048)])
@pytest.mark.parametrize("spread", [0.0, 6.0])
def test_error_against_64_bits(M, N, k, spread):
    check_error(M, N, k, spread)


# every width of a tile, with k blocks well past the ring's stages and the block sums in tensor memory, k and columns that end
# inside a block and a tile (148 SMs, which the choice of the width goes by)
WIDTHS = [(32, 511, 1028, 836), (64, 200, 4100, 1028), (96, 400, 6148, 900), (128, 300, 6148, 708)]


@pytest.mark.parametrize("width,M,N,k", WIDTHS)
def test_every_width_wraps_its_rings(width, M, N, k):
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert K().lib.ullm_linear_f32_split_columns(M, N) == width
    check_error(M, N, k, 0.0)


def check_error(M, N, k, spread):
    g = torch.Generator(device=device()).manual_seed(M + N)
    x, w = (torch.randn(r, k, generator=g, device=device()) * torch.exp(spread * torch.randn(r, k, generator=g, device=device()))
            for r in (M, N))
    bias = torch.randn(N, generator=g, device=device())
    got = run(x, w, bias)
    ref = x.double() @ w.double().t() + bias.double()
    size = (x.double().abs() @ w.double().abs().t()) + bias.double().abs()
    # per result, of the sum of sizes: 2^-24 for the terms left out and for the bias; k / 64 rounded additions; and in a k block four
    # tensor instructions at full size (the others work 2^-8 below), each of which cuts its 16 products and the sum so far at 2^-24 of
    # the largest of them: 70 cuts
    assert ((got.double() - ref).abs() <= 2.0 ** -24 * (72 + k / 64) * size).all()
    lib = torch.addmm(bias, x, w.t()).double()
    err, err_lib = float((got.double() - ref).norm() / ref.norm()), float((lib - ref).norm() / ref.norm())
    print(f"error {err:.2e}, the library's {err_lib:.2e}")
    assert err <= err_lib * 1.1 + 1e-7


@pytest.mark.parametrize("N", [160] + [n for _, _, n, _ in WIDTHS[1:]])
def test_infinities_and_nan_as_in_float32(N):
    M = {160: 200}.get(N) or next(m for _, m, n, _ in WIDTHS if n == N)
    x, w = torch.randn(M, 256, device=device()), torch.randn(N, 256, device=device())
    x[3, 7], x[5, 9], x[199, 255], w[17, 3], w[20, 4] = float("inf"), float("nan"), 3.4e38, float("-inf"), 0.0
    x[8] = 0.0
    x[8, 4], x[9, 100] = float("inf"), -3.4028e38
    got, ref = run(x, w), x @ w.t()
    big = ref.isnan() | ref.isinf() | (ref.abs() > 1e30)
    assert torch.equal(got.isnan(), ref.isnan()) and torch.equal(got[ref.isinf()], ref[ref.isinf()])
    assert torch.allclose(got[big & ~ref.isnan()], ref[big & ~ref.isnan()], rtol=1e-5)
    assert (got[~big] - ref[~big]).abs().max() < 1e-4


def test_what_it_does_not_take():
    kk, out = K(), torch.empty(300, 256, device=device())
    w = torch.randn(256, 64, device=device())
    assert kk.linear_f32_split(torch.randn(300, 64, device=device()), w, out)
    assert not kk.linear_f32_split(torch.randn(300, 66, device=device()), torch.randn(256, 66, device=device()), out)  # k % 4
    y = torch.randn(300 * 64 + 1, device=device())[1:].view(300, 64)
    assert not kk.linear_f32_split(y, w, out)  # off the 16-byte border
    assert not kk.linear_f32_split(torch.randn(300, 128, device=device())[:, :64], w, out)  # rows with gaps
    assert not kk.linear_f32_split(torch.randn(200, 64, device=device()), w, out[:200])  # fewer than 2^16 results


@pytest.mark.parametrize("low,other", [(-126, 0), (0, -126), (-126, 20), (20, -126), (-70, -50), (-112, 0), (-100, 60)])
def test_operands_near_the_smallest_exponent_keep_24_bits(low, other):
    """Operands down to 2^-126 keep all their bits: the errors are those of operands of order one, and the library's at most."""
    M, N, k = 200, 512, 260
    g = torch.Generator(device=device()).manual_seed(3)
    x, w = (torch.randn(r, k, generator=g, device=device()).clamp(-8, 8) for r in (M, N))
    x, w = (torch.where(v.abs() < 1, v.sign() + v, v).ldexp(torch.tensor(e, device=device())) for v, e in ((x, low), (w, other)))
    got, ref = run(x, w).double(), x.double() @ w.double().t()
    size = x.double().abs() @ w.double().abs().t()
    # (as above, and half a unit of the smallest float)
    assert ((got - ref).abs() <= 2.0 ** -24 * (72 + k / 64) * size + 2.0 ** -150).all()
    lib = (x @ w.t()).double()
    assert float((got - ref).norm()) <= 1.1 * float((lib - ref).norm()) + 1e-7 * float(ref.norm()) + 2.0 ** -149 * (M * N) ** 0.5


def test_operands_and_sums_that_the_factor_takes_to_infinity():
    """Operands from 2^104 on and sums from 2^80 on are formed by multiply-adds: finite where float32 is."""
    x, w = torch.randn(140, 128, device=device()), torch.randn(600, 128, device=device())
    x[1], x[2, 5], x[3], w[7], w[9, 0] = x[1] * 2.0 ** 60, 2.0 ** 110, x[3] * 2.0 ** 104, w[7] * 2.0 ** 22, -(2.0 ** 120)
    got, ref = run(x, w).double(), x.double() @ w.double().t()
    size = x.double().abs() @ w.double().abs().t()
    fits = size < 2.0 ** 127
    assert torch.isfinite(got[fits]).all() and ((got - ref).abs() <= 2.0 ** -24 * 200 * size)[fits].all()


def test_a_product_over_no_columns_is_the_bias():
    kk, bias = K(), torch.randn(512, device=device())
    out = torch.full((300, 512), 9.0, device=device())
    kk.linear(torch.empty(300, 0, device=device()), torch.empty(512, 0, device=device()), out, bias)
    assert torch.equal(out, bias.expand(300, 512))
    kk.linear(torch.empty(300, 0, device=device()), torch.empty(512, 0, device=device()), out)
    assert torch.count_nonzero(out) == 0
