"""The FP64 digit products where a level's sum is largest and on rows of disjoint
large entries."""

import numpy as np
import pytest
import torch

import vmc_torch_gb300 as vg
from vmc_torch_gb300 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def gram(X):
    T = torch.empty((X.shape[0],) * 2, dtype=torch.float64, device=DEV)
    solver = vg.MinSRGB300()
    solver._tc_gram_f64(X.to(DEV), T, 0.0, torch.device(DEV))
    solver._check_tc()
    return T.cpu().numpy()


@pytest.mark.parametrize("n,K", [(64, 256), (130, 250)])
def test_levels_of_digits_that_share_a_sign(n, K):
    """Digits near +127 throughout: the sums of the five products of level 4
    pass 2^24.  Levels 0 to 4 are summed exactly all the same; levels 5 and 6 (6
    and 7 products, units 2^-54 and 2^-62) lose at most 2 units of theirs in
    each addition past 2^24 (at most 16 x 7 additions); the 64-bit integer is
    rounded to FP64 once."""
    rng = np.random.default_rng(n)
    d = rng.integers(120, 128, (7, n, K))
    d[6] &= ~3                                    # 53 significant bits
    v = np.zeros((n, K), dtype=np.int64)
    for p in range(7):
        v = v * 256 + d[p]
    X = v.astype(np.float64) * 2.0 ** -55
    assert (X < 1).all() and ((X * 2.0 ** 55).astype(np.int64) == v).all() and X.max(1).min() > 0.5
    S = [sum(d[p] @ d[q - p].T for p in range(q + 1)) for q in range(7)]
    assert S[4].max() > 2 ** 24
    hi = ((S[0] * 256 + S[1]) * 256 + S[2]) * 256 + S[3]
    lo = (S[4] * 256 + S[5]) * 256 + S[6]
    t = hi * 65536 + ((lo + 128) >> 8)            # units of 2^-54
    T = gram(torch.as_tensor(X))
    err = np.abs(T * 2.0 ** 54 - t.astype(np.float64))
    assert (err <= t * 2.0 ** -53 + 16 * 7 * 2 + 2).all()


def test_rows_with_large_entries_in_different_columns():
    """Entries of 2^-30 of their row's largest, which stand in different columns
    of different rows: the error is bounded by the rows' largest entries (per
    term 36 x 2^-56 of their product, and the FP64 sums' roundings), not by the
    sum of magnitudes as on the FP64 cores."""
    n, K = 100, 700
    rng = np.random.default_rng(3)
    X = rng.standard_normal((n, K)) * 2.0 ** -30
    X[np.arange(n), 7 * np.arange(n)] = rng.uniform(0.5, 2.0, n)
    Xd = torch.as_tensor(X)
    ref = (Xd @ Xd.t()).numpy()
    m = np.abs(X).max(1)
    scale = np.outer(m, m)
    T = gram(Xd)
    sums = np.abs(X) @ np.abs(X).T
    assert (np.abs(T - ref) <= K * 36 * 2.0 ** -56 * scale + 8 * 2.0 ** -53 * np.maximum(sums, scale) +
            K * 2.0 ** -53 * sums).all()
    # relative to sqrt(T_ii T_jj), what the factorisation that follows commits by itself
    d = np.sqrt(np.diag(ref))
    assert (np.abs(T - ref) <= 2.0 ** -48 * np.outer(d, d)).all()
    C = torch.zeros((n, n), dtype=torch.float64, device=DEV)
    Xg = Xd.to(DEV)
    _lib.call("vmc_sr_gram", _lib.ptr(Xg), 0, n, K, K, _lib.ptr(C), n, 0.0, 0, _lib.stream_of(DEV))
    assert (np.abs(C.cpu().numpy() - ref) <= 2 * (K + 2) * 2.0 ** -53 * sums).all()     # gram="cuda": componentwise
