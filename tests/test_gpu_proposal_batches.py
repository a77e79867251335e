"""Training gradients of the learned proposal over several row tiles, row ranges
of the bias sums and splits of the batch."""

import numpy as np
import pytest
import torch

from oracle import lattice, proposal as op
import vmc_torch_gb300 as vg
from vmc_torch_gb300.proposal import LearnedProposal

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("Lx,Ly,nup,R", [(4, 4, 8, 63), (4, 4, 8, 128), (4, 4, 8, 129), (4, 2, 3, 300), (4, 4, 8, 2049)])
def test_gradient_matches_autograd(Lx, Ly, nup, R):
    """A weight's gradient is an FP32 sum of R products of FP32 chains of at most
    512 terms: (R + 3 x 512) 2^-24 of the magnitudes at the most, 2.2e-4 at 2049
    samples; 5e-4 of the gradient's norm, block by block."""
    N = Lx * Ly
    H = vg.spinful_Fermi_Hubbard_square_lattice_torch(Lx, Ly, 1.0, 8.0, 2 * nup, n_fermions_per_spin=(nup, nup))
    H.precompute_hops_gpu(DEV)
    prop = LearnedProposal(N, H.edges_on(DEV), device=DEV, seed=R)
    with torch.no_grad():
        prop.params.mul_(3.0)
    prop.t += 1
    edges = H.graph.edges()
    X = lattice.random_initial_configs(R, N, nup, nup, seed=R + 1)
    rng = np.random.default_rng(R)
    tgt = (rng.random((R, 2 * len(edges))) ** 3).astype(np.float32)
    kt = np.array([0.4, 0.3, 0.2, 0.1], np.float32)
    loss_ref, g_ref = op.loss_and_grad(prop.params.cpu().numpy().astype(np.float64), X, tgt, kt, 0.1, edges, N)
    prop.buf_occ[:R] = vg.pack(torch.as_tensor(X, device=DEV))
    prop.buf_tgt[:R] = torch.as_tensor(tgt, device=DEV)
    prop.n_buf = R
    prop.k_target = lambda: torch.as_tensor(kt, device=DEV)
    prop.lr = 0.0
    loss = prop.train(epochs=1, batch=R, generator=torch.Generator(device=DEV).manual_seed(0))
    g = prop.grad.cpu().numpy().astype(np.float64)
    assert abs(loss - loss_ref) < 1e-4 * max(1.0, abs(loss_ref))
    Kin, off = prop.Kin, 0
    for n in (512 * Kin, 512, 512 * 512, 512, g.size - 512 * Kin - 512 * 512 - 1024 - 256, 256):
        a, b = g[off:off + n], g_ref[off:off + n]
        off += n
        assert np.linalg.norm(a - b) <= 5e-4 * np.linalg.norm(b) + 1e-12, n
    assert off == g.size
