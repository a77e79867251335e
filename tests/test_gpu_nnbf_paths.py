"""Edges of the mixed-precision NNBF kernels: row remainders of the hidden
layer's tiles, determinants whose value is known in advance, and sweeps whose
walker number decides between one stream of overlapping launches and several
streams."""

import numpy as np
import pytest
import torch

from oracle import lattice, models as om
import vmc_torch_gb300 as vg
from vmc_torch_gb300 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def model(ps, N, nf):
    m = vg.NNBF_GB300(N, nf, precision="mixed").to(DEV)
    with torch.no_grad():
        for p, v in zip(m.params, ps):
            p.copy_(torch.as_tensor(v))
    m.invalidate()
    return m


@pytest.mark.parametrize("R", [1, 31, 127, 128, 129, 513])
def test_hidden_layer_rows(R):
    """BF16 products are exact in FP32; what is left is the output's BF16
    rounding (half an ulp: 2^-8 relative) and the order of 256 FP32 sums."""
    g = torch.Generator(device="cpu").manual_seed(R)
    H1 = (torch.randn(R, 256, generator=g) * 0.5).to(torch.bfloat16).to(DEV)
    W1 = (torch.randn(256, 256, generator=g) / 16).to(torch.bfloat16).to(DEV)
    b1 = (torch.randn(256, generator=g) * 0.1).to(DEV)
    H2 = torch.full((R + 1, 256), 3.0, dtype=torch.bfloat16, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    _lib.call("vmc_nnbf_hidden_layer", _lib.ptr(H1), R, _lib.ptr(W1), _lib.ptr(b1), _lib.ptr(H2), 0, 0,
              _lib.ptr(err), _lib.stream_of(DEV))
    assert int(err.item()) == 0
    ref = torch.nn.functional.gelu(H1.double() @ W1.double().t() + b1.double())
    assert ((H2[:R].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-4).all()
    assert (H2[R] == 3.0).all()


@pytest.mark.parametrize("Lx,Ly,nf", [(8, 8, 64), (6, 6, 32)])
@pytest.mark.parametrize("kind", ["permutation", "singular", "nan"])
def test_determinants_known_in_advance(Lx, Ly, nf, kind):
    """Scaled permutations have no elimination error: the sign is the
    permutation's times the scales', |det| the scales' product up to the FP32
    rounding of one product per step (nf x 2^-24) and of the logarithm.  A zero
    column is a zero amplitude, a NaN entry a NaN one, wherever it stands."""
    N = Lx * Ly
    rng = np.random.default_rng(nf)
    X = lattice.random_initial_configs(5, N, nf // 2, nf // 2, seed=nf)
    occ = np.flatnonzero(np.asarray(om.quimb_to_netket(X[:1]))[0])
    assert occ.size == nf
    for trial in range(6):
        ps = om.nnbf_init(N, nf, 256, 2, seed=trial)
        ps[-2][:] = 0.0
        perm = rng.permutation(nf)
        if trial == 0:
            perm = np.arange(nf)
        if trial == 1:   # one transposition of the first and last rows
            perm = np.arange(nf)
            perm[[0, -1]] = perm[[-1, 0]]
        scale = rng.choice([-1.0, 1.0], nf) * rng.uniform(0.25, 4.0, nf)
        rows = np.zeros((nf, nf))
        rows[np.arange(nf), perm] = scale.astype(np.float32)
        if kind == "singular":
            rows[:, perm[(7 * trial) % nf]] = 0.0
        if kind == "nan":
            rows[(11 * trial) % nf, (5 * trial) % nf] = np.nan
        ps[0][occ] = rows
        s, la = model(ps, N, nf).forward_log(torch.as_tensor(X, device=DEV))
        s, la = float(s[0]), float(la[0])
        if kind == "permutation":
            ref_s, ref_l = np.linalg.slogdet(rows)
            assert s == ref_s
            assert abs(la - ref_l) <= nf * 2.0 ** -24 + 1e-6
        elif kind == "singular":
            assert s == 0.0 and la <= np.log(1e-45)
        else:
            assert np.isnan(s) and np.isnan(la)


@pytest.mark.parametrize("Lx,Ly,nf", [(8, 8, 64), (6, 6, 32)])
@pytest.mark.parametrize("B", [4095, 4096, 6149])
def test_sweep_does_not_depend_on_the_batch(Lx, Ly, nf, B):
    """Walkers are independent: the first 257 of a batch (one stream up to
    4095 walkers, two and three groups above) end exactly as they do alone,
    with the random numbers replayed."""
    N, b = Lx * Ly, 257
    m = model(om.nnbf_init(N, nf, 256, 2, seed=5), N, nf)
    g = vg.SquareLattice(Lx, Ly)
    E = len(g.sweep_edges())
    rng = np.random.default_rng(B)
    rp = (rng.random((1, E, B), dtype=np.float32), rng.integers(0, 2, (1, E, B)).astype(np.uint8),
          rng.random((1, E, B), dtype=np.float32))
    x0 = vg.init_walkers(B, N, nf // 2, nf // 2, seed=B, device=DEV)
    out = []
    for sl in (slice(0, B), slice(0, b), slice(B - b, B)):
        fx, (s, l) = vg.MetropolisExchangeSpinfulSamplerGB300().step(
            x0[sl].clone(), m, g, use_log_amp=True,
            replay=tuple(torch.as_tensor(np.ascontiguousarray(a[:, :, sl]), device=DEV) for a in rp))
        out.append((fx.clone(), s.clone(), l.clone()))
    assert not torch.equal(out[0][0], x0)
    for x, first, last in zip(*out):
        assert torch.equal(x[:b], first)
        assert torch.equal(x[B - b:], last)


@pytest.mark.parametrize("Lx,Ly,nf", [(8, 8, 64), (6, 6, 32)])
@pytest.mark.parametrize("B", [257, 4096])
def test_captured_sweep_equals_eager(Lx, Ly, nf, B):
    """One stream of overlapping launches (257) and walker groups (4096) keep
    their order in a CUDA graph."""
    N = Lx * Ly
    m = model(om.nnbf_init(N, nf, 256, 2, seed=9), N, nf)
    g = vg.SquareLattice(Lx, Ly)
    x0 = vg.init_walkers(B, N, nf // 2, nf // 2, seed=B, device=DEV)
    with torch.inference_mode():   # as the sampler runs it
        st = m.bind_state(x0)
        occ0 = st.occ.clone()
        m.sweep(st, g, 1, 11, 0)
        torch.cuda.synchronize()
        want = [t.clone() for t in (st.occ, st.sign, st.logabs, st.n_acc)]
        assert not torch.equal(st.occ, occ0)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            m.sweep(st, g, 1, 11, 0)
        for _ in range(2):
            st.occ.copy_(occ0)
            graph.replay()
            torch.cuda.synchronize()
            for a, b in zip(want, (st.occ, st.sign, st.logabs, st.n_acc)):
                assert torch.equal(a, b)
