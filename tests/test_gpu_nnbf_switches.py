"""NNBF sweeps with the parallel parts switched off by the environment: the
chunk pipeline on one group of walkers, and chunks back to back."""
import os
import subprocess
import sys

import pytest
import torch

from oracle import models as om
import vmc_torch_gb300 as vg

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run(L, nf, B):
    N = L * L
    m = vg.NNBF_GB300(N, nf, precision="mixed").to(DEV)
    with torch.no_grad():
        for p, v in zip(m.params, om.nnbf_init(N, nf, 256, 2, seed=6)):
            p.copy_(torch.as_tensor(v))
    m.invalidate()
    H = vg.spinful_Fermi_Hubbard_square_lattice_torch(L, L, 1.0, 8.0, nf, n_fermions_per_spin=(nf // 2, nf // 2))
    H.precompute_hops_gpu(DEV)
    x0 = vg.init_walkers(B, N, nf // 2, nf // 2, seed=B, device=DEV)
    fx, (s, l) = vg.MetropolisExchangeSpinfulSamplerGB300(seed=5).step(x0.clone(), m, vg.SquareLattice(L, L),
                                                                       use_log_amp=True)
    _, e = vg.evaluate_energy(fx, m, H)
    assert not torch.equal(fx, x0)
    return [t.cpu() for t in (fx, s, l, e)]


@pytest.mark.parametrize("L,nf,B", [(8, 64, 6000), (6, 32, 9000)])
@pytest.mark.parametrize("switch", ["VMC_GB300_SWEEP_LANES", "VMC_GB300_SERIAL_CHUNKS"])
def test_switches_change_no_result(L, nf, B, switch, tmp_path):
    f = str(tmp_path / "out.pt")
    code = "import sys, torch; sys.path[:0] = [%r, %r]; import test_gpu_nnbf_switches as t; torch.save(t.run(%d, %d, %d), %r)" % (
        ROOT, os.path.join(ROOT, "tests"), L, nf, B, f)
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, env=dict(os.environ, **{switch: "1"}), cwd=ROOT)
    for a, b in zip(torch.load(f), run(L, nf, B)):
        assert torch.equal(a, b)
