"""Column means and O^T x of FP32 rows (vmc_sr_center, vmc_sr_update): no less
accurate than sums in FP64, over FP32's and FP64's whole ranges."""

from fractions import Fraction

import numpy as np
import pytest
import torch

from vmc_torch_gb300 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"
U = 2.0 ** -53


def update(O, x):
    ns, npar = O.shape
    dp = torch.full((npar,), 7.0, dtype=torch.float64, device=DEV)
    _lib.call("vmc_sr_update", _lib.ptr(O), 1, ns, npar, O.stride(0), _lib.ptr(x), _lib.ptr(dp), _lib.stream_of(DEV))
    return dp.cpu().numpy()


def center(O):
    ns, npar = O.shape
    out = torch.empty((ns, npar), device=DEV)
    mean = torch.empty(npar, dtype=torch.float64, device=DEV)
    _lib.call("vmc_sr_center", _lib.ptr(O), 1, ns, npar, O.stride(0), _lib.ptr(out), out.stride(0), _lib.ptr(mean),
              _lib.stream_of(DEV))
    return out.cpu().numpy(), mean.cpu().numpy()


def exact_sum(terms):
    return sum((Fraction(float(a)) * Fraction(float(b)) for a, b in terms), Fraction(0))


@pytest.mark.parametrize("npar", [1, 33, 1000, 38912, 39001])
def test_update_of_one_row_is_the_rounded_product(npar):
    """One row: every entry is one product.  Two roundings are allowed (the
    product's parts are joined in FP64): 2^-52 of it."""
    g = torch.Generator().manual_seed(npar)
    O = torch.randn(1, npar, generator=g) * torch.exp(4 * torch.randn(1, npar, generator=g))
    x = torch.randn(1, generator=g, dtype=torch.float64)
    dp = update(O.to(DEV), x.to(DEV))
    ref = (O[0].double() * x).numpy()
    assert (np.abs(dp - ref) <= 2 * U * np.abs(ref)).all()


@pytest.mark.parametrize("ns,npar", [(2, 40), (100, 70), (129, 38915), (1031, 40), (5000, 33)])
def test_update_against_exact_sums(ns, npar):
    """Each of eight warps sums its rows far below u of the sum S of magnitudes
    and rounds it into FP64 (three roundings); their sums are added in FP64
    (eight): 11 u S at the most, whatever the number of rows; a chain of FP64
    additions over them has ns u S."""
    rng = np.random.default_rng(ns)
    cols = np.unique(np.concatenate([[0, 31, npar - 1], rng.integers(0, npar, 5)]))
    O = (rng.standard_normal((ns, npar)) * np.exp(2 * rng.standard_normal((1, npar)))).astype(np.float32)
    x = rng.standard_normal(ns) * np.exp(rng.standard_normal(ns))
    dp = update(torch.as_tensor(O, device=DEV), torch.as_tensor(x, device=DEV))
    for c in cols:
        ref = exact_sum(zip(O[:, c], x))
        S = float(np.abs(O[:, c].astype(np.float64) * x).sum())
        assert abs(float(Fraction(float(dp[c])) - ref)) <= (11 * U + 2.0 ** -62) * S


# factors of O's columns and of x: products below and above FP32's range, x outside it, and both mixed
@pytest.mark.parametrize("fo,fx", [(1e-30, 1.0), (1e-38, 1e-5), (1e-42, 1e-3), (1.0, 1e-60), (1.0, 1e-300), (1e30, 1e20),
                                   (1e37, 1.0), (1.0, 1e200), (1e-40, 1e250), (3.0, 1e39)])
@pytest.mark.parametrize("ns,npar", [(1, 5), (70, 40), (140, 38920)])
def test_update_over_the_ranges(fo, fx, ns, npar):
    """Outside the range of the split products FP64 does the sums: ns + 11
    roundings of the sum of magnitudes."""
    rng = np.random.default_rng(ns + npar)
    O = (rng.standard_normal((ns, npar)) * fo).astype(np.float32)
    x = rng.standard_normal(ns) * fx
    if ns > 1:
        O[::3, ::2] = 0.0
        O[1::5] = (rng.standard_normal((len(O[1::5]), npar))).astype(np.float32)   # ordinary rows between the others
        x[2::7] = 0.0
    dp = update(torch.as_tensor(O, device=DEV), torch.as_tensor(x, device=DEV))
    for c in sorted({0, 1, npar // 2, npar - 1}):
        ref = exact_sum(zip(O[:, c], x))
        S = float(sum(abs(Fraction(float(a)) * Fraction(float(b))) for a, b in zip(O[:, c], x)))
        assert abs(float(Fraction(float(dp[c])) - ref)) <= (ns + 11) * U * S + 5e-324


@pytest.mark.parametrize("ns,npar", [(1, 3), (100, 33), (129, 38915), (3000, 40)])
def test_means_against_exact_sums(ns, npar):
    """As for the update, and one rounding of the division: 12 u of the mean magnitude."""
    rng = np.random.default_rng(ns)
    O = (rng.standard_normal((ns, npar)) * np.exp(3 * rng.standard_normal((ns, npar)))).astype(np.float32)
    _, mean = center(torch.as_tensor(O, device=DEV))
    for c in sorted({0, npar // 2, npar - 1}):
        ref = exact_sum(zip(O[:, c], np.ones(ns))) / ns
        S = float(np.abs(O[:, c].astype(np.float64)).sum()) / ns
        assert abs(float(Fraction(float(mean[c])) - ref)) <= (12 * U + 2.0 ** -62) * S


def test_infinite_entries_stay_in_their_columns():
    """As in FP64: an infinite entry makes its column's sum infinite (NaN with
    both signs) and leaves the others alone."""
    O = torch.randn(300, 70, generator=torch.Generator().manual_seed(1))
    O[17, 3] = float("inf")
    O[18, 5], O[190, 5] = float("inf"), -float("inf")
    O[2, 7] = float("nan")
    x = torch.rand(300, dtype=torch.float64, generator=torch.Generator().manual_seed(2)) + 0.1
    dp = update(O.to(DEV), x.to(DEV))
    _, mean = center(O.to(DEV))
    for v in (dp, mean):
        assert v[3] == np.inf and np.isnan(v[5]) and np.isnan(v[7])
        assert np.isfinite(np.delete(v, [3, 5, 7])).all()


@pytest.mark.parametrize("f", [1e-44, 1e-38, 1e-30, 1e-25, 1e30, 2e38])
@pytest.mark.parametrize("ns,npar", [(3, 20), (100, 33), (129, 38915)])
def test_centring_over_the_range(f, ns, npar):
    """Means that FP32 cannot sum (entries near its largest) and entries whose
    scaled remainder underflows it: the FP64 expression rounded, as elsewhere."""
    rng = np.random.default_rng(ns)
    O = (rng.uniform(0.1, 1.5, (ns, npar)) * f).astype(np.float32)
    O[:, ::3] = (rng.uniform(-1.5, 1.5, (ns, len(range(0, npar, 3)))) * f).astype(np.float32)
    out, mean = center(torch.as_tensor(O, device=DEV))
    ref = O.astype(np.float64).mean(0)
    assert (np.abs(mean - ref) <= (ns + 2) * U * np.abs(O.astype(np.float64)).mean(0)).all()
    want = ((O.astype(np.float64) - mean) * (1.0 / ns ** 0.5)).astype(np.float32)
    assert np.array_equal(out, want)
