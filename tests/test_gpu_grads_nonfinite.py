"""Non-finite output weights in the batched FP32 adjoint: a configuration meets
those of its occupied orbitals only, as in the one-CTA-per-configuration kernel."""

import numpy as np
import pytest
import torch

import vmc_torch_gb300 as vg
from test_gpu_grads_batched import run

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("N,nf,B,rows", [(9, 9, 40, 40), (36, 32, 30, 7), (40, 64, 12, 12)])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_weights_of_empty_orbitals(N, nf, B, rows, bad):
    g = torch.Generator().manual_seed(N)
    model = vg.NNBF_GB300(N, nf, precision="mixed", generator=g)
    with torch.no_grad():
        model.params[5][3 * nf + 1, 17] = bad      # out_w row of orbital 3 (site 3, spin up), column 1
    model = model.to(DEV)
    rng = np.random.default_rng(nf)
    occ = np.zeros((B, 2), dtype=np.uint64)
    for b in range(B):
        free = np.array([o for o in range(2 * N) if o != 3])
        pick = list(rng.choice(free, nf, replace=False))
        if b % 3 == 2:
            pick[0] = 3                            # every third configuration holds orbital 3
        for o in pick:
            occ[b, 0 if o < N else 1] |= np.uint64(1) << np.uint64(o % N)
    empty = torch.as_tensor((occ[:, 0] >> np.uint64(3)) & np.uint64(1) == 0, device=DEV)
    occ = torch.as_tensor(occ.view(np.int64), device=DEV)
    a, c = run(model, occ, None, False), run(model, occ, rows, False)
    assert torch.isfinite(a["dense"][empty]).all()
    for k in ("dense", "g", "h", "logabs", "sign"):
        assert torch.equal(torch.isfinite(a[k]), torch.isfinite(c[k])), k
    assert torch.isfinite(a["logabs"][empty]).all() and torch.isnan(a["logabs"][~empty]).all()
    nout = 2 * N * nf
    sizes = [nout, 256 * 2 * N, 256, 256 * 256, 256, nout, 1]
    x, y = (torch.split(t["dense"], sizes, 1) for t in (a, c))
    # dh2: nf^2 terms in another order, 2 nf^2 2^-24 of the magnitudes, times |gelu'| <= 1.13
    ow = model.params[5].detach().abs().nan_to_num(0.0, 0.0)
    mag = 0.01 * 1.13 * (x[0].double().abs() @ ow)
    assert ((x[4].double() - y[4].double()).abs() <= (4 * nf * nf + 16) * 2.0 ** -24 * mag + 1e-37).all()
    assert torch.equal(x[0], y[0]) and torch.equal(x[5], y[5])
