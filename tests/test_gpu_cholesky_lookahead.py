"""The Cholesky's trailing updates on two streams against the same on one."""

import ctypes
import threading

import pytest
import torch

from vmc_torch_gb300 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def spd(n, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    X = torch.randn(n, n + 8, generator=g, device=DEV, dtype=torch.float64) / n ** 0.5
    A = X @ X.t()
    A.diagonal().add_(1e-3)
    return A


def factor(A, stream):
    n = A.shape[0]
    nbytes = ctypes.c_int64(0)
    _lib.call("vmc_sr_cholesky_tc_work_bytes", n, ctypes.byref(nbytes))
    work = torch.empty(nbytes.value, dtype=torch.uint8, device=DEV)
    flag = torch.zeros(2, dtype=torch.int32, device=DEV)
    L = A.clone()
    return L, flag, work, lambda: _lib.call("vmc_sr_cholesky_tc", _lib.ptr(L), n, n, _lib.ptr(flag), _lib.ptr(work),
                                            _lib.ptr(flag[1:]), stream)


@pytest.mark.parametrize("n", [2560, 2561, 2815, 3073])
def test_lookahead_equals_one_stream(n):
    """Panels of 256 columns, orders that leave a last panel of 256, 1, 255 and
    1; a call under capture takes one stream throughout.  The same tiles in the
    same order of sums: equality."""
    A = spd(n, n)
    L, flag, _, run = factor(A, _lib.stream_of(torch.device(DEV, 0)))
    run()
    assert flag.tolist() == [0, 0]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        Lg, flag_g, _, run_g = factor(A, ctypes.c_void_p(side.cuda_stream))
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            run_g()
        Lg.copy_(A)
        graph.replay()
        side.synchronize()
    assert flag_g.tolist() == [0, 0]
    assert torch.equal(torch.tril(L), torch.tril(Lg))
    Lc = torch.tril(L)
    d = A.diagonal().sqrt()
    assert ((Lc @ Lc.t() - A).abs() <= (n + 8) * 2.0 ** -50 * d[:, None] * d[None]).all()


def test_two_threads_two_streams():
    mats = [spd(2600, 1), spd(2700, 2)]
    torch.cuda.synchronize()
    out = [None, None]

    def work(i):
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            for _ in range(4):
                L, flag, ws, run = factor(mats[i], ctypes.c_void_p(st.cuda_stream))
                run()
                st.synchronize()
                out[i] = (torch.tril(L), flag.tolist())

    ths = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in ths:
        t.start()
    for t in ths:
        t.join()
    for i in range(2):
        L, flag, _, run = factor(mats[i], _lib.stream_of(torch.device(DEV, 0)))
        run()
        assert out[i][1] == [0, 0]
        assert torch.equal(out[i][0], torch.tril(L))
