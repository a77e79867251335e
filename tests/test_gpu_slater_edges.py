"""Slater determinants at the edges of the register tiles and warps."""

import numpy as np
import pytest
import torch

import vmc_torch_gb300 as vg

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("Lx,Ly,nu,nd", [(2, 2, 1, 0), (2, 2, 1, 1), (4, 2, 4, 4), (4, 4, 8, 8), (4, 4, 9, 8),
                                         (6, 4, 16, 15), (6, 4, 16, 16), (6, 6, 17, 16), (6, 6, 24, 24),
                                         (6, 6, 25, 24), (8, 8, 32, 31), (8, 8, 32, 32)])
@pytest.mark.parametrize("B", [1, 37])
def test_carried_state_after_sweeps(Lx, Ly, nu, nd, B):
    """Electron numbers on both sides of the 16-row tiles and of one and two
    warps a walker.  The state carried through two sweeps of inverse updates
    equals the determinants of the final configurations: an update's error is
    ~2^-52 times the conditions it has met (below 1e5 for these M), over up to
    two hundred accepted moves."""
    N, nf = Lx * Ly, nu + nd
    g = np.random.default_rng(nf)
    M = g.normal(size=(2 * N, nf))
    m = vg.SlaterDeterminant_GB300(2 * N, nf).to(DEV)
    with torch.no_grad():
        next(iter(m.parameters())).copy_(torch.as_tensor(M))
    m.invalidate()
    x0 = vg.init_walkers(B, N, nu, nd, seed=nf, device=DEV)
    s = vg.MetropolisExchangeSpinfulSamplerGB300()
    graph = vg.SquareLattice(Lx, Ly)
    fx, (sg, la) = s.step(x0, m, graph, use_log_amp=True)
    fx, (sg, la) = s.step(fx, m, graph, use_log_amp=True)
    assert tuple(fx.shape) == (B, N)
    x = fx.cpu().numpy()
    from oracle import models as om
    occ = np.asarray(om.quimb_to_netket(x))
    for b in range(B):
        rs, rl = np.linalg.slogdet(M[np.flatnonzero(occ[b])])
        assert float(sg[b]) == rs
        assert abs(float(la[b]) - rl) <= 200 * 2.0 ** -52 * 1e5
