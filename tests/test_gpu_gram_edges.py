"""Tile, chunk and padding edges of the tensor-core FP32 Gram matrix."""

import pytest
import torch

from vmc_torch_gb300 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def gram(T, X, alpha, D, shift, accumulate):
    ns, K = X.shape
    rp, kp = -(-ns // 128) * 128, -(-K // 64) * 64
    planes = torch.full((3, rp, kp), 7.0, dtype=torch.bfloat16, device=DEV)
    rexp = torch.full((rp,), 99, dtype=torch.int32, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    s = _lib.stream_of(DEV)
    _lib.call("vmc_split_bf16x3", _lib.ptr(X), ns, K, X.stride(0), _lib.ptr(planes), rp, kp, _lib.ptr(rexp), s)
    _lib.call("vmc_sr_gram_tc", _lib.ptr(planes), _lib.ptr(rexp), ns, rp, kp, float(alpha), _lib.ptr(T), T.stride(0),
              None if D is None else _lib.ptr(D), float(shift), int(accumulate), _lib.ptr(err), s)
    assert int(err.item()) == 0


@pytest.mark.parametrize("ns,K", [(1, 1), (31, 64), (127, 65), (128, 2048), (129, 2049), (257, 4097), (385, 8200)])
@pytest.mark.parametrize("hadamard", [False, True])
def test_gram_edges(ns, K, hadamard):
    """A row is rounded to 2^-20 of its largest entry (half a unit of 2^-20 of
    the next power of two above it), which bounds an entry's error by
    K 2^-19 of the two rows' largest entries; the sums themselves add ~2^-30."""
    g = torch.Generator(device="cpu").manual_seed(ns + K)
    X = torch.randn(ns, K + 3, generator=g) * torch.exp(8 * torch.randn(ns, 1, generator=g))
    X[ns // 2] = 0.0 if ns > 1 else X[0]
    X = X.to(DEV)[:, :K]                       # a row stride that is not the width
    D = torch.randn(ns, ns, generator=g, dtype=torch.float64).to(DEV) if hadamard else None
    D = None if D is None else (D + D.t())
    T0 = torch.randn(ns, ns, generator=g, dtype=torch.float64).to(DEV)
    T0 = T0 + T0.t()
    ref = 0.25 * (X.double() @ X.double().t()) * (1.0 if D is None else D)
    m = X.abs().amax(1).double()
    tol = 0.25 * K * 2.0 ** -19 * m[:, None] * m[None] * (1.0 if D is None else D.abs())
    eye = torch.eye(ns, dtype=torch.float64, device=DEV)
    for accumulate in (0, 1):
        T = T0.clone()
        gram(T, X, 0.25, D, 1.5, accumulate)
        want = ref + 1.5 * eye + (T0 if accumulate else 0.0)
        assert ((T - want).abs() <= tol + 1e-12 * (1.0 + want.abs())).all()
        assert torch.equal(T, T.t())


def test_gram_range_of_exponents():
    """Rows at both ends of FP32, and a row that is not finite."""
    X = torch.ones(5, 200, device=DEV)
    X[0] *= 1e-44
    X[1] *= 3e38
    X[3, 77] = float("nan")
    T = torch.zeros(5, 5, dtype=torch.float64, device=DEV)
    gram(T, X, 1.0, None, 0.0, 0)
    fin = [0, 1, 2, 4]
    ref = X[fin].double() @ X[fin].double().t()
    got = T[fin][:, fin]
    assert ((got - ref).abs() <= ref.abs() * 2.0 ** -18).all()
    assert torch.isnan(T[3]).all()
