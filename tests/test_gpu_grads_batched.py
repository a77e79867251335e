"""The batched FP32 adjoint (vmc_nnbf_logpsi_grad_ws) against the one-CTA-per-
configuration kernel (vmc_nnbf_logpsi_grad) and the row floor (vmc_floor_rows)
against masked_fill, at every matrix tile (16, 32, 48, 64) and its edges, with
blocks that do not divide the batch."""
import ctypes

import numpy as np
import pytest
import torch

import vmc_torch_gb300 as vg
from vmc_torch_gb300 import _lib
from vmc_torch_gb300.models import LOG_MIN

pytestmark = pytest.mark.gpu
DEV = "cuda"


def run(model, occ, rows, full):
    B, N, nf = occ.shape[0], model.n_sites, model.n_fermions
    _, arr = model.grad_net(torch.device(DEV, 0))
    s = _lib.stream_of(torch.device(DEV, 0))
    nout = 2 * N * nf
    nd = model.n_params - 256 * nout
    new = lambda *sh, dt=torch.float32: torch.full(sh, 7.0, dtype=dt, device=DEV)  # noqa: E731
    out = {"dense": new(B, nd + 1), "g": new(B, nout), "h": new(B, 256), "logabs": new(B, dt=torch.float64),
           "sign": new(B, dt=torch.float64)}
    if full:
        out["full"] = new(B, model.n_params)
    f = out.get("full")
    args = (arr, N, nf, 256, 0.01, _lib.ptr(occ), B, _lib.ptr(f), 0 if f is None else f.stride(0),
            _lib.ptr(out["dense"]), nd + 1, _lib.ptr(out["g"]), _lib.ptr(out["h"]), _lib.ptr(out["logabs"]),
            _lib.ptr(out["sign"]))
    if rows is None:
        _lib.call("vmc_nnbf_logpsi_grad", 0, *args, s)
    else:
        nb = ctypes.c_int64(0)
        _lib.call("vmc_nnbf_grad_work_bytes", N, nf, rows, ctypes.byref(nb))
        work = torch.empty(nb.value, dtype=torch.uint8, device=DEV)
        _lib.call("vmc_nnbf_logpsi_grad_ws", *args, _lib.ptr(work), rows, s)
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("N,nf,B,rows", [(1, 1, 3, 2), (8, 8, 130, 130), (9, 16, 5, 2), (16, 17, 20, 7), (36, 32, 131, 129),
                                         (25, 33, 9, 4), (30, 48, 6, 6), (36, 49, 7, 3), (64, 64, 140, 128)])
def test_batched_adjoint(N, nf, B, rows):
    g = torch.Generator().manual_seed(N * 100 + nf)
    model = vg.NNBF_GB300(N, nf, precision="mixed", generator=g)
    with torch.no_grad():
        for p in model.params:
            p.copy_(torch.randn(p.shape, generator=g, dtype=torch.float64) * (0.5 if p.dim() == 1 else 1.0) /
                    max(1, p.shape[-1]) ** 0.5)
    model = model.to(DEV)
    rng = np.random.default_rng(nf)
    occ = np.zeros((B, 2), dtype=np.uint64)
    for b in range(B):
        k = nf - 1 if b == 1 else nf       # one configuration with the wrong electron number
        for o in rng.choice(2 * N, k, replace=False):
            occ[b, 0 if o < N else 1] |= np.uint64(1) << np.uint64(o % N)
    occ = torch.as_tensor(occ.view(np.int64), device=DEV)
    full = N <= 16
    a, c = run(model, occ, None, full), run(model, occ, rows, full)
    nout, n_orb = 2 * N * nf, 2 * N
    for k in ("g", "h", "logabs", "sign"):
        assert torch.equal(a[k], c[k]), k
    sizes = [nout, 256 * n_orb, 256, 256 * 256, 256, nout, 1]
    x, y = (torch.split(t["dense"], sizes, 1) for t in (a, c))
    assert torch.equal(x[0], y[0]) and torch.equal(x[5], y[5]) and torch.equal(y[6], torch.full_like(y[6], 7.0))
    # dh2 is a sum of nf^2 terms in another order: 2 nf^2 2^-24 of the sum of magnitudes, both ways, times
    # s |gelu'| <= 1.13 s and a few roundings; dz0 is the same through |W1| and 256 more terms
    ow, w1 = model.params[5].detach().abs(), model.params[3].detach().abs()
    mag = 0.01 * 1.13 * (x[0].double().abs() @ ow)
    tol1 = (4 * nf * nf + 16) * 2.0 ** -24 * mag + 1e-37
    assert ((x[4].double() - y[4].double()).abs() <= tol1).all()
    tol0 = 1.13 * (tol1 @ w1 + 600 * 2.0 ** -24 * (mag @ w1)) + 1e-37
    assert ((x[2].double() - y[2].double()).abs() <= tol0).all()
    # the outer products are those of the batch's own dz0, dz1
    site = torch.arange(N, device=DEV)
    bits = torch.cat([(occ[:, :1] >> site) & 1, (occ[:, 1:] >> site) & 1], 1).float()
    assert torch.equal(y[1].view(B, 256, n_orb), y[2][:, :, None] * bits[:, None, :])
    w1a, w1b = x[3].view(B, 256, 256).double(), y[3].view(B, 256, 256).double()
    l, r = w1b * x[4].double()[:, :, None], w1a * y[4].double()[:, :, None]
    assert ((l - r).abs() <= 2.0 ** -22 * (l.abs() + r.abs()) + 1e-60).all()
    if full:
        k = (c["g"][:, :, None] * c["h"][:, None, :]).view(B, -1)
        assert torch.equal(c["full"], torch.cat([y[0], y[1], y[2], y[3], y[4], k, y[5]], 1))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_floor_rows(dtype):
    O = torch.randn(7, 300, device=DEV, dtype=dtype)
    la = torch.tensor([0.0, LOG_MIN, LOG_MIN - 1e-9, -float("inf"), float("nan"), 5.0, -200.0], device=DEV,
                      dtype=torch.float64)
    tail = O[:, 257:].clone()
    ref = O.clone().masked_fill_((la < LOG_MIN).unsqueeze(1), 0)
    view = O[:, :257]
    _lib.call("vmc_floor_rows", _lib.ptr(la), LOG_MIN, 7, _lib.ptr(view), 0 if dtype == torch.float64 else 1, 257,
              view.stride(0), _lib.stream_of(O.device))
    assert torch.equal(O[:, :257], ref[:, :257]) and torch.equal(O[:, 257:], tail)
