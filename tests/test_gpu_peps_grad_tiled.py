"""The register-tiled FP32 log-derivatives (D = 4, six rows, any number of
columns) against the per-output kernel, which a workspace that is not 16-byte
aligned selects, and the FP64 adjoint."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import lattice, peps
import vmc_torch_gb300 as vg
from vmc_torch_gb300 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"
Lx, D = 6, 4


def rows(T, Ly, occ, precision, offset=0):
    dt = torch.float64 if precision == "fp64" else torch.float32
    m = vg.FPEPS_GB300(Lx, Ly, D, precision=precision, tensors=torch.as_tensor(T), dtype=dt).to(DEV)
    B = occ.shape[0]
    O = torch.full((B, m.n_params + 3), 7.0, dtype=dt, device=DEV)
    n = 5 * (Ly + 1) * 16 * 16 * 16      # five walkers at a time
    work = torch.empty(n + 4, dtype=dt, device=DEV)
    _lib.call("vmc_peps_logpsi_grad", m._prec, _lib.ptr(m._tensors(O.device)), Lx, Ly, D, _lib.ptr(occ), B, _lib.ptr(O),
              O.stride(0), ctypes.c_void_p(work.data_ptr() + offset), 5, _lib.stream_of(O.device))
    assert (O[:, m.n_params:] == 7.0).all()
    return O[:, :m.n_params].cpu().numpy()


@pytest.mark.parametrize("Ly", [1, 2, 3, 5, 6, 7, 10])
def test_against_the_per_output_kernel_and_fp64(Ly):
    """Both FP32 kernels divide by the same amplitude, whose cancellation sets
    their error: the tiled one's is at most four times the other's, or 1e-5 of
    the row.  Rows without an amplitude (odd electron number) are zero in all."""
    N, B = Lx * Ly, 12
    T = peps.init_tensors(Lx, Ly, D, seed=40 + Ly).astype(np.float32).astype(np.float64)
    k = max(1, (2 * N) // 5)
    X = np.concatenate([lattice.random_initial_configs(B - 3, N, k, k, seed=Ly),
                        lattice.random_initial_configs(3, N, k, k - 1, seed=Ly + 1)])[np.random.default_rng(Ly).permutation(B)]
    occ = vg.pack(torch.as_tensor(X, device=DEV))
    a, b, c = rows(T, Ly, occ, "fp32"), rows(T, Ly, occ, "fp32", 4), rows(T, Ly, occ, "fp64")
    odd = (np.isin(X, [1, 2]).sum(1) % 2) == 1
    assert odd.sum() == 3 and not a[odd].any() and not b[odd].any() and not c[odd].any()
    n = np.linalg.norm(c[~odd], axis=1)
    ea, eb = (np.linalg.norm(v[~odd] - c[~odd], axis=1) / n for v in (a, b))
    assert np.isfinite(ea).all() and (ea <= 4 * eb + 1e-5).all(), (ea, eb)
    assert np.array_equal(a != 0, b != 0) or np.abs(a[(a != 0) != (b != 0)]).max() <= 1e-6 * np.abs(a).max()


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_tensors_that_are_not_finite(bad):
    """A configuration meets the tensors of its own site states only: the rows
    that are finite, and the others, are those of the per-output kernel."""
    Ly, B = 4, 40
    T = peps.init_tensors(Lx, Ly, D, seed=3).astype(np.float32).astype(np.float64)
    T[2, 1, 3][T[2, 1, 3] != 0] = bad
    X = lattice.random_initial_configs(B, Lx * Ly, 10, 10, seed=5)
    occ = vg.pack(torch.as_tensor(X, device=DEV))
    a, b = rows(T, Ly, occ, "fp32"), rows(T, Ly, occ, "fp32", 4)
    hit = X[:, 2 * Ly + 1] == 3
    assert 0 < hit.sum() < B
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    assert np.isfinite(a[~hit]).all() and (np.abs(a[~hit]).max(1) > 0).all()
    assert not a[hit].any() and not b[hit].any()
