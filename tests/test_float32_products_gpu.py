"""float32 products lose nothing against chains of float32 multiply-adds: every finite number comes through the cutting in three parts
whole, the error over operands of several kinds is no larger than that of chains of 16 fmaf with a compensated running sum
(emulated here), and outputs that are not finite are what the chains give."""

import pytest
import torch

from clockwork_b200 import ops
from tests.gpu_tools import DEV

pytestmark = pytest.mark.gpu

KINDS = {
    "normal": lambda g, *s: torch.randn(*s, generator=g),
    "spread over e": lambda g, *s: torch.randn(*s, generator=g) * torch.exp(torch.randn(*s, generator=g)),
    "spread over e^3": lambda g, *s: torch.randn(*s, generator=g) * torch.exp(3 * torch.randn(*s, generator=g)),
    "one sign": lambda g, *s: torch.randn(*s, generator=g).abs(),
    "between 0 and 1": lambda g, *s: torch.rand(*s, generator=g),
}


def chains(a, w):
    """16 fmaf at a time (a product of two float32 is exact in float64, its sum with a float32 is rounded there and then once to
    float32), the chains' results added with their rounding errors carried along."""
    total = torch.zeros(a.shape[0], w.shape[0])
    lost = torch.zeros_like(total)
    for k0 in range(0, a.shape[1], 16):
        chain = torch.zeros_like(total)
        for k in range(k0, min(k0 + 16, a.shape[1])):
            chain = (a[:, k : k + 1].double() * w[:, k].double() + chain.double()).float()
        y = chain - lost
        t = total + y
        lost = (t - total) - y
        total = t
    return total


@pytest.mark.parametrize("k", [4, 64, 1536, 1800])
@pytest.mark.parametrize("kind", KINDS)
def test_error_is_no_larger_than_that_of_chains(kind, k):
    g = torch.Generator().manual_seed(11)
    a, w = KINDS[kind](g, 80, k), KINDS[kind](g, 500, k)
    want, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    error = lambda x: (((x.double() - want) / size) ** 2).mean().sqrt().item()  # noqa: E731
    assert error(ops.gemm_ref(a.to(DEV), w.to(DEV)).cpu()) <= error(chains(a, w))


@pytest.mark.parametrize("k", [4, 64, 1536])
@pytest.mark.parametrize("x,w", [(0x8080, 0xFFFF), (0x7F80, 0x7FFF), (0x1FFFF, 0x20000), (0x2FDFF, 0x3FFFF), (0x7FFFFF, 0x7FFFFF), (0x5F7DF, 0x23F7F)])
def test_numbers_whose_parts_are_largest(k, x, w):
    """One product over and over: 2^-24 for the result's rounding, up to 2^-25 cut off the sums of the second parts' products
    (8 additions of at most 2^-5 of the whole, 2^-23 each, none beyond the first at K of 4), 2^-29 left out."""
    x, w = 1 + x * 2.0**-23, 1 + w * 2.0**-23
    got = ops.gemm_ref(torch.full((17, k), x, device=DEV), torch.full((33, k), w, device=DEV)).double()
    assert (got / (k * x * w) - 1).abs().max().item() <= 1.6 * 2.0**-24


@pytest.mark.parametrize("n", [4, 40, 64, 200])
def test_every_finite_number_comes_through_whole(n):
    g = torch.Generator().manual_seed(n)
    bits = torch.randint(-(2**31), 2**31, (70, n), generator=g).to(torch.int32)
    small = torch.where(torch.rand(70, n, generator=g) < 0.3, bits & 0x00FFFFFF | bits & -(2**31), bits)  # (many below the smallest normal number)
    a = small.view(torch.float32)
    a = torch.where(a.isfinite(), a, torch.ones(()))
    for weights in (torch.eye(n), -torch.eye(n)):
        got = ops.gemm_ref(a.to(DEV), weights.to(DEV)).cpu()
        assert torch.equal(got, a @ weights if n == 1 else a * weights[0, 0])
        got = ops.gemm_ref(weights.to(DEV), a.to(DEV)).cpu()
        assert torch.equal(got, (a * weights[0, 0]).T)


def test_small_numbers_keep_their_bits():
    g = torch.Generator().manual_seed(5)
    a, w = torch.randn(40, 1536, generator=g), torch.randn(300, 1536, generator=g)
    want, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    for scale in (2.0**-110, 2.0**-118):
        got = ops.gemm_ref(a.to(DEV), (w * scale).to(DEV)).cpu().double() / scale
        assert (((got - want) / size) ** 2).mean().sqrt() <= (((chains(a, w).double() - want) / size) ** 2).mean().sqrt()


@pytest.mark.parametrize("k", [5, 16, 40, 1536, 8960])
@pytest.mark.parametrize("gated", [False, True])
def test_numbers_that_are_not_finite(k, gated):
    g = torch.Generator().manual_seed(k)
    a, w, up = torch.randn(20, k, generator=g), torch.randn(90, k, generator=g), torch.randn(90, k, generator=g)
    clean = a.clone()
    a[3, k - 1], a[5, 0], a[7, k - 1], a[9, :] = float("inf"), float("nan"), -float("inf"), 2.0**126
    a[11, 0], a[11, 1:] = torch.finfo(torch.float32).max, 0.0
    w[4] *= 2.0**-40
    run = lambda x: (ops.gemm_ref_swiglu(x.to(DEV), w.to(DEV), up.to(DEV)) if gated else ops.gemm_ref(x.to(DEV), w.to(DEV))).cpu()  # noqa: E731
    got, untouched = run(a), run(clean)
    rows = [r for r in range(20) if r not in (3, 5, 7, 9, 11)]
    assert torch.equal(got[rows], untouched[rows])  # (whatever stands in other rows)
    if gated:
        assert got[5].isnan().all()
        return
    want = chains(a, w)
    assert (got[3] == float("inf")).equal(w[:, -1] > 0) and (got[7] == float("inf")).equal(w[:, -1] < 0)
    torch.testing.assert_close(got[[3, 5, 7, 11]], want[[3, 5, 7, 11]], rtol=0, atol=0, equal_nan=True)
    finite = got[9].isfinite()  # (numbers so large that some sums fit and some do not: those that fit are as exact as any)
    exact, size = a[9].double() @ w.double().T, a[9].double().abs() @ w.double().abs().T
    assert ((got[9].double() - exact).abs() <= 19 * 2.0**-24 * size)[finite].all()
    torch.testing.assert_close(got[9][~finite], want[9][~finite], rtol=0, atol=0, equal_nan=True)


@pytest.mark.parametrize("rows", [1, 16, 17, 32])
@pytest.mark.parametrize("offset", [0, 1])
def test_few_rows_over_a_long_inner_dimension(rows, offset):
    """1,536 features over an inner dimension of five segments: tiles of 64 weight rows, whose sums are those of tiles of 128."""
    g = torch.Generator().manual_seed(rows)
    a, w = torch.randn(200, 8960 + offset, generator=g).to(DEV)[:, offset:], torch.randn(1500, 8960, generator=g).to(DEV)
    assert torch.equal(ops.gemm_ref(a[:rows], w), ops.gemm_ref(a, w)[:rows])
