"""Chi-truncated boundary states of low rank and their overlap, on tensors whose
amplitude is known in advance."""
import math

import pytest
import torch

import vmc_torch_gb300 as vg

pytestmark = pytest.mark.gpu
DEV = "cuda"


def overlap_model(a, b, c, precision):
    """4x4, D = 4, empty and doubly occupied sites only, states that are products
    over the columns: top (1, a) (1, a) (1, 0) (1e20, 0), bottom (0, 1) (0, 1)
    (b, 1) (c, 0) in the two even bond values; psi = a^2 b c 1e20."""
    T = torch.zeros(4, 4, 4, 4, 4, 4, 4, dtype=torch.float64)
    for s in (0, 3):
        T[0, :, s, 0, 0, 0, 0] = 1.0
        T[3, :, s, 0, 0, 0, 0] = 1.0
        T[1, :, s, 0, 0, 0, 0] = 1.0
        T[1, 0, s, 0, 0, 0, 2] = a
        T[1, 1, s, 0, 0, 0, 2] = a
        T[1, 3, s, 0, 0, 0, 0] = 1e20
        T[2, 0, s, 0, 2, 0, 0] = 1.0
        T[2, 1, s, 0, 2, 0, 0] = 1.0
        T[2, 2, s, 0, 0, 0, 0] = b
        T[2, 2, s, 0, 2, 0, 0] = 1.0
        T[2, 3, s, 0, 0, 0, 0] = c
    m = vg.FPEPS_GB300(4, 4, 4, max_bond=8, precision=precision, tensors=T,
                       dtype=torch.float64 if precision == "fp64" else torch.float32).to(DEV)
    assert m.truncated
    return m


@pytest.mark.parametrize("a,b,c", [(1.0, 1.0, 1.0), (0.5, 2.0, -1.0), (1e-2, 1e-3, 1.0), (1e-6, 1e-8, 1.0)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_states_of_rank_one(a, b, c, precision):
    """Fewer singular values than chi: nothing is truncated.  FP32 tensors (2^-24
    relative each, four of them) and a few FP32 roundings: 1e-5 in the
    log-amplitude."""
    x = torch.zeros(1, 16, dtype=torch.int64, device=DEV)
    x[0, [0, 5, 10]] = 3
    st = overlap_model(a, b, c, precision).bind_state(x)
    assert float(st.sign[0]) == math.copysign(1.0, c)
    assert abs(float(st.logabs[0]) - math.log(a * a * b * 1e20)) <= 1e-5


@pytest.mark.parametrize("a,b,c", [(1e-13, 1e-25, 1.0), (1e-18, 1e-3, 1.0),
                                   (1e-12, 1e-30, -1.0)])
def test_small_overlaps_of_normalised_states(a, b, c):
    """FP32 tensors (2^-24 relative each, four of them), a few FP32 roundings of
    the truncation: 1e-5 in the log-amplitude."""
    x = torch.zeros(1, 16, dtype=torch.int64, device=DEV)
    x[0, [0, 5, 10]] = 3
    for precision in ("fp64", "fp32"):
        st = overlap_model(a, b, c, precision).bind_state(x)
        assert float(st.sign[0]) == math.copysign(1.0, c), precision
        assert abs(float(st.logabs[0]) - math.log(a * a * b * 1e20)) <= 1e-5, precision
