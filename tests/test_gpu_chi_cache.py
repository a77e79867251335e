"""The row-by-row cached side states of chi-truncated sweeps in FP32: after a
sweep every walker's amplitude is that of its configuration contracted afresh."""

import pytest
import torch

import vmc_torch_gb300 as vg

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("Lx,Ly,D,chi,n", [(6, 6, 4, 16, 16), (4, 4, 4, 8, 4), (4, 6, 4, 8, 6), (6, 4, 4, 8, 6), (8, 8, 2, 4, 28)])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_swept_states_equal_fresh_ones(Lx, Ly, D, chi, n, precision):
    """The same rows absorbed in the same order from the same numbers, wherever
    the sweep took them up: equality."""
    dt = torch.float64 if precision == "fp64" else torch.float32
    m = vg.FPEPS_GB300(Lx, Ly, D, max_bond=chi, precision=precision, dtype=dt,
                       generator=torch.Generator().manual_seed(Lx + Ly)).to(DEV)
    assert m.truncated
    B = 23
    m.chi_rows = 9           # several chunks
    x0 = vg.init_walkers(B, Lx * Ly, n, n, seed=7, device=DEV)
    g = vg.SquareLattice(Lx, Ly)
    fx, (s, la) = vg.MetropolisExchangeSpinfulSamplerGB300(seed=3, sweeps_per_step=2).step(x0.clone(), m, g,
                                                                                          use_log_amp=True)
    assert not torch.equal(fx, x0)
    with torch.inference_mode():
        st = m._eval_state(fx)
        m._refresh(st, 0)
    assert torch.equal(m._state.sign, st.sign)
    assert torch.equal(m._state.logabs, st.logabs)
