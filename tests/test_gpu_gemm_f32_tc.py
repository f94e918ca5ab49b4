"""Float products on the tensor cores (csrc/gemm_f32_tc.cu) against 64 bits: edges of tiles, slices and ranks, numbers of very different
sizes, and numbers that have no bfloat16 pieces."""
import pytest
import torch

from qwen_triton_b200.ops import kernels
from qwen_triton_b200.ops.kernels import GemmOut
from test_gpu_kernels import DEV, rand

pytestmark = pytest.mark.gpu


def both(a, w):
    out = [torch.full((1, a.shape[0], w.shape[0]), float("nan"), device=DEV) for _ in range(2)]
    kernels.gemm_f32_tc(a, w, GemmOut(out[0]))
    kernels.gemm_f32(a, w, GemmOut(out[1]))
    kernels.check_status(DEV)
    return out[0][0], out[1][0]


@pytest.mark.parametrize("m, n, k", [(1, 1, 4), (9, 64, 4), (128, 128, 64), (129, 130, 68), (33, 200, 2052), (300, 131, 1000), (549, 1024, 1024), (40, 513, 12288)])
@pytest.mark.parametrize("kind", ["normal", "positive", "wide"])
def test_errors_against_64_bits(m, n, k, kind):
    a, w = rand(m, k, seed=1), rand(n, k, seed=2, scale=0.02)
    if kind == "positive":
        a, w = a.abs(), w.abs()
    if kind == "wide":
        a = a * torch.exp(6 * rand(m, k, seed=3))
    want = a.double() @ w.double().T
    got, _ = both(a, w)
    # Products are exact but for pieces below 2^-25 of them.  An instruction adds 16 products to the sum so far and cuts each of the 17 below 2^-24 of the
    # largest; four of a slice's 24 add the large products (the others are 2^-8 of them and less), and slices are added rounded to nearest: no element is
    # further off than 4 x 17 x 2^-24 of its absolute sums.  Over all elements these cuts are independent, and far smaller than that.
    assert bool(((got.double() - want).abs() <= 68 * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)).all())
    assert float((got.double() - want).norm()) <= 2e-7 * float(want.norm())


def test_numbers_without_pieces_are_multiplied_as_floats():
    a, w = rand(140, 256, seed=4), rand(200, 256, seed=5)
    a[3, 5], a[7, 9], a[130, 3], w[150, 7], w[151, 3] = float("inf"), float("nan"), 3.4e38, -float("inf"), 1.0
    got, want = both(a, w)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    finite = torch.isfinite(want)
    assert torch.equal(finite, torch.isfinite(got))
    assert torch.equal(got[~finite & ~torch.isnan(want)], want[~finite & ~torch.isnan(want)])
    exact = a.double() @ w.double().T
    assert bool(((got.double() - exact).abs()[finite] <= 2.0 ** -20 * (a.double().abs() @ w.double().abs().T)[finite]).all())


def guarded(a, w):
    """The product, written ahead of a row that nothing may touch."""
    m, n = a.shape[0], w.shape[0]
    held = torch.full((m + 1, n), 7.25, device=DEV)
    kernels.gemm_f32_tc(a, w, GemmOut(held[:m].unsqueeze(0)))
    kernels.check_status(DEV)
    assert bool((held[m] == 7.25).all())
    return held[:m]


@pytest.mark.parametrize("m, n, k", [(33, 3, 4), (129, 131, 64), (40, 70, 68), (300, 129, 1000), (35, 513, 2052), (130, 1024, 4096)])
def test_what_can_be_exact_is(m, n, k):
    """Sums of one number, and of whole numbers below 2^24, in one slice, several, and several ranks."""
    a = rand(m, k, seed=1) * torch.exp(3 * rand(m, k, seed=2))                       # all 24 bits of a mantissa
    places = torch.arange(n, device=DEV) * 7 % k
    w = torch.zeros(n, k, device=DEV)
    w[torch.arange(n, device=DEV), places] = torch.exp2((torch.arange(n, device=DEV) % 19 - 9).float())
    assert torch.equal(guarded(a, w), a[:, places] * w.sum(1))
    assert torch.equal(guarded(w, a), (a[:, places] * w.sum(1)).T)
    whole, signs = (rand(m, k, seed=3) * 30).round(), (rand(n, k, seed=4) * 20).round()
    assert torch.equal(guarded(whole, signs), (whole.double() @ signs.double().T).float())
    large = (rand(m, k, seed=5) * 2 ** 21).round()                                   # three pieces each
    assert torch.equal(guarded(large, torch.sign(w)), large[:, places])


@pytest.mark.parametrize("k", [64, 1024, 4096])
def test_operands_of_one_sign_lose_no_more_than_the_pipe_cuts(k):
    """Cuts go towards zero: of a slice's four large instructions each takes half a unit of the sum so far (a quarter of the slice's to all of it) on average, at
    most 2.5 x 2^-24 together; what is rounded to nearest has no mean."""
    a, w = rand(300, k, seed=1).abs(), rand(500, k, seed=2).abs()
    want = a.double() @ w.double().T
    mean = float(((guarded(a, w).double() - want) / want).mean())
    assert -2.5 * 2.0 ** -24 <= mean <= 2.0 ** -28
