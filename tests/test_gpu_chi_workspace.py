"""The chi-truncated model's workspace: what a walker state keeps."""
import ctypes

import pytest
import torch

import vmc_torch_gb300 as vg
from vmc_torch_gb300 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_local_energy_gives_its_workspace_back():
    """Local energies build hop terms thousands at a time; a state of a few
    walkers keeps the workspace of those walkers only."""
    Lx, Ly, D, chi, B = 4, 4, 4, 8, 20
    m = vg.FPEPS_GB300(Lx, Ly, D, max_bond=chi, generator=torch.Generator().manual_seed(3)).to(DEV)
    H = vg.spinful_Fermi_Hubbard_square_lattice_torch(Lx, Ly, 1.0, 8.0, 8, n_fermions_per_spin=(4, 4))
    H.precompute_hops_gpu(DEV)
    fx = vg.init_walkers(B, Lx * Ly, 4, 4, seed=2, device=DEV)
    nb = ctypes.c_int64(0)
    _lib.call("vmc_peps_chi_work_bytes", 0, Lx, Ly, D, chi, B, ctypes.byref(nb))
    st = m.bind_state(fx)
    _, e0 = vg.evaluate_energy(fx, m, H)
    assert st.extra["chi_work"].numel() == nb.value
    m.chi_rows = 7       # fewer walkers and terms at a time: the same sums
    _, e1 = vg.evaluate_energy(fx, m, H)
    assert st.extra["chi_work"].numel() == nb.value
    assert torch.equal(e0, e1)
