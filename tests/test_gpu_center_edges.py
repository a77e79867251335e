"""The FP32 centring is the FP64 expression rounded to FP32, entry by entry."""

import pytest
import torch

from vmc_torch_gb300 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("ns,npar", [(1, 1), (2, 33), (63, 31), (64, 32), (1000, 129), (257, 8192), (130, 20001)])
@pytest.mark.parametrize("inplace", [False, True])
def test_center_rounds_the_fp64_expression(ns, npar, inplace):
    """The device mean (returned) is the one subtracted, so nothing but the
    rounding of ((double)x - mean) * scale is left: equality, on smooth data,
    constant columns, sparse columns and entries next to the mean."""
    g = torch.Generator(device="cpu").manual_seed(ns * npar)
    O = torch.randn(ns, npar + 5, generator=g) * torch.exp(3 * torch.randn(npar + 5, generator=g))
    O[:, ::7] = O[:1, ::7]
    O[:, 1::7] *= (torch.rand(ns, (npar + 5 + 5) // 7, generator=g) < 0.1)
    O[:, 2::7] = O[:1, 2::7] * (1 + 1e-6 * torch.randn(ns, (npar + 5 + 4) // 7, generator=g))
    O[:, 3::7] = torch.randint(-3, 4, (ns, (npar + 5 + 3) // 7), generator=g).float()
    O = O.to(DEV)[:, :npar]
    out = O.clone() if inplace else torch.full((ns, npar + 2), 7.0, device=DEV)[:, :npar]
    src = out if inplace else O
    ref_src = O.double()
    mean = torch.zeros(npar, dtype=torch.float64, device=DEV)
    _lib.call("vmc_sr_center", _lib.ptr(src), 1, ns, npar, src.stride(0), _lib.ptr(out), out.stride(0),
              _lib.ptr(mean), _lib.stream_of(DEV))
    scale = 1.0 / (ns ** 0.5)
    assert torch.allclose(mean, ref_src.mean(0), rtol=1e-12, atol=1e-14 * float(O.abs().max()))
    want = ((ref_src - mean) * scale).float()
    assert torch.equal(out, want)
