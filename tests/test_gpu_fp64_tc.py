"""FP64 Gram matrices and the Cholesky factorisation on the tensor cores
(vmc_split_f64, vmc_sr_gram_f64_tc, vmc_sr_cholesky_tc) against FP64 on the
CPU, at the edges of the 128 x 64 tiles, the 32-column atoms, the 256-column
drains and the 64- and 256-column panels."""
import ctypes

import pytest
import torch

import vmc_torch_gb300 as vg
from vmc_torch_gb300 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rows(Ns, K, seed):
    """Rows and columns of very different sizes."""
    g = torch.Generator().manual_seed(seed)
    X = torch.randn(Ns, K, generator=g, dtype=torch.float64)
    return X * torch.exp(3 * torch.randn(Ns, 1, generator=g, dtype=torch.float64)) * \
        torch.exp(torch.randn(1, K, generator=g, dtype=torch.float64))


@pytest.mark.parametrize("Ns,K", [(1, 1), (2, 31), (63, 33), (64, 256), (65, 257), (128, 512), (129, 100), (300, 1025)])
def test_gram_f64(Ns, K):
    X = rows(Ns, K, Ns + K)
    T = torch.full((Ns, Ns), 7.0, dtype=torch.float64, device=DEV)
    solver = vg.MinSRGB300()
    solver._tc_gram_f64(X.to(DEV), T, 1e-3, torch.device(DEV))
    solver._check_tc()
    ref = X @ X.t() + 1e-3 * torch.eye(Ns, dtype=torch.float64)
    m = X.abs().amax(1)
    # per term: the operands' 2^-56 and the levels left out, at most 9 units of 2^-56 of 2^(E_i + E_j) <= 4 m_i m_j;
    # FP64 sums of the drains and of the reference: (K + 2) 2^-53 of the sum of magnitudes <= K m_i m_j
    tol = K * (36 * 2.0 ** -56 + 2 * (K + 2) * 2.0 ** -53) * (m[:, None] * m[None, :]) + 2.0 ** -52
    assert (T.cpu() - ref).abs().le(tol).all()
    assert torch.equal(T, T.t())


def test_gram_f64_slabs_and_nan():
    X = rows(130, 900, 5).to(DEV)
    one, many = vg.MinSRGB300(), vg.MinSRGB300()
    many.SLAB_BYTES = 1    # slabs of 256 columns
    A, B = (torch.empty((130, 130), dtype=torch.float64, device=DEV) for _ in range(2))
    one._tc_gram_f64(X, A, 0.5, torch.device(DEV))
    many._tc_gram_f64(X, B, 0.5, torch.device(DEV))
    n = X.norm(dim=1)
    assert ((A - B).abs() <= 2.0 ** -46 * n[:, None] * n[None, :]).all()
    X[70, 3] = float("nan")
    X[5, 899] = float("inf")
    one._tc_gram_f64(X, A, 0.5, torch.device(DEV))
    one._check_tc()
    bad = torch.zeros(130, dtype=torch.bool, device=DEV)
    bad[5] = bad[70] = True
    assert torch.equal(A.isnan(), bad[:, None] | bad[None, :])


@pytest.mark.parametrize("n", [1, 63, 64, 65, 129, 256, 257, 513, 769, 1100])
@pytest.mark.parametrize("tc", [False, True])
def test_cholesky(n, tc):
    g = torch.Generator().manual_seed(n)
    X = torch.randn(n, n + 8, generator=g, dtype=torch.float64)
    A = X @ X.t() / n + 1e-3 * torch.eye(n, dtype=torch.float64)
    e = torch.exp(torch.randn(n, generator=g, dtype=torch.float64))
    A = A * (e[:, None] * e[None, :])     # rows of different sizes, still positive definite
    s = _lib.stream_of(torch.device(DEV, 0))
    L = A.to(DEV)
    flag = torch.zeros(2, dtype=torch.int32, device=DEV)
    nbytes = ctypes.c_int64(0)
    _lib.call("vmc_sr_cholesky_tc_work_bytes", n, ctypes.byref(nbytes))
    work = torch.empty(nbytes.value, dtype=torch.uint8, device=DEV)

    def factor(M):
        if tc:
            _lib.call("vmc_sr_cholesky_tc", _lib.ptr(M), n, n, _lib.ptr(flag), _lib.ptr(work), _lib.ptr(flag[1:]), s)
        else:
            _lib.call("vmc_sr_cholesky", _lib.ptr(M), n, n, _lib.ptr(flag), s)

    factor(L)
    assert flag.tolist() == [0, 0]
    Lc = torch.tril(L.cpu())
    d = A.diagonal().sqrt()
    # backward error of a Cholesky factorisation, (n + 1) u |L| |L|^T <= (n + 1) u sqrt(A_ii A_jj), with the
    # unit of the double-float products (2^-45) or of the digits (2^-50) in place of u
    tol = (n + 8) * (2.0 ** -50 if tc else 2.0 ** -45) * d[:, None] * d[None, :]
    assert ((Lc @ Lc.t() - A).abs() <= tol).all()
    b = torch.randn(n, generator=g, dtype=torch.float64)
    x = b.to(DEV)
    _lib.call("vmc_sr_cholesky_solve", _lib.ptr(L), n, n, _lib.ptr(x), s)
    r = Lc @ (Lc.t() @ x.cpu()) - b
    # the solves' own backward error, n u |L| (|L|^T |x|) for each of the two
    scale = Lc.abs() @ (Lc.abs().t() @ x.cpu().abs())
    assert (r.abs() <= 2 * (n + 8) * 2.0 ** -52 * scale).all()
    # a pivot that is not positive sets the flag
    A[n - 1, n - 1] = -1.0
    factor(A.to(DEV))
    assert flag.tolist() == [1, 0]
