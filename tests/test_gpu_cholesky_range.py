"""Reciprocals of the Cholesky tile's pivots over FP64's range."""

import numpy as np
import pytest
import torch

from vmc_torch_gb300 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"



@pytest.mark.parametrize("d", [1e-310, 4e-309, 1e-300, 1e-150, 1.0, 1e150, 1e300, 1.7e308])
@pytest.mark.parametrize("n", [2, 65, 130])
def test_cholesky_of_extreme_diagonals(d, n):
    """A diagonal matrix: square roots, and zeros beside them."""
    A = torch.ones(n, dtype=torch.float64)
    A[::2] = d
    L = torch.diag(A).to(DEV)
    flag = torch.zeros(2, dtype=torch.int32, device=DEV)
    _lib.call("vmc_sr_cholesky", _lib.ptr(L), n, n, _lib.ptr(flag), _lib.stream_of(DEV))
    assert flag.tolist() == [0, 0]
    ref = torch.diag(A.sqrt()).numpy()
    assert (np.abs(torch.tril(L).cpu().numpy() - ref) <= 2.0 ** -52 * ref).all()


def test_reciprocals_of_the_pivots():
    """Column entries divided by a pivot's square root over mantissas and
    exponents: the reciprocal (2^-53 and the seed's step), the root, their
    product and the entry's own, half a unit each: 2^-51."""
    n = 64
    rng = np.random.default_rng(9)
    for e in (-1060, -1022, -1001, -999, -500, -126, -1, 0, 1, 127, 500, 999, 1001, 1020):
        m = np.concatenate([[1.0, np.nextafter(2.0, 1.0), 1.0 + 2.0 ** -52, 1.5], rng.uniform(1, 2, 28)])
        d = np.ldexp(m, e)
        a = np.sqrt(d) * rng.uniform(-1, 1, 32)
        A = np.zeros((n, n))
        i = np.arange(32)
        A[2 * i, 2 * i] = d
        A[2 * i + 1, 2 * i] = a
        A[2 * i + 1, 2 * i + 1] = 4.0
        L = torch.as_tensor(A, device=DEV)
        flag = torch.zeros(2, dtype=torch.int32, device=DEV)
        _lib.call("vmc_sr_cholesky", _lib.ptr(L), n, n, _lib.ptr(flag), _lib.stream_of(DEV))
        assert flag.tolist() == [0, 0], e
        Lc = L.cpu().numpy()
        root = np.sqrt(d)
        assert (np.abs(Lc[2 * i, 2 * i] - root) <= 2.0 ** -52 * root).all(), e
        ref = a / root
        assert (np.abs(Lc[2 * i + 1, 2 * i] - ref) <= 2.0 ** -51 * np.abs(ref)).all(), e
