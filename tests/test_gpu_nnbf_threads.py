"""NNBF sweeps and local energies of several host threads, each on its own
stream, and beside another thread's capture."""

import threading

import pytest
import torch

from oracle import models as om
import vmc_torch_gb300 as vg

pytestmark = pytest.mark.gpu
DEV = "cuda"
L, NF = 6, 32
N = L * L


def model(seed):
    m = vg.NNBF_GB300(N, NF, precision="mixed").to(DEV)
    with torch.no_grad():
        for p, v in zip(m.params, om.nnbf_init(N, NF, 256, 2, seed=seed)):
            p.copy_(torch.as_tensor(v))
    m.invalidate()
    return m


def setup(B, seed):
    m = model(seed)
    H = vg.spinful_Fermi_Hubbard_square_lattice_torch(L, L, 1.0, 8.0, NF, n_fermions_per_spin=(NF // 2, NF // 2))
    H.precompute_hops_gpu(DEV)
    x0 = vg.init_walkers(B, N, NF // 2, NF // 2, seed=seed, device=DEV)
    with torch.inference_mode():
        st = m.bind_state(x0)
    fields = [st.occ, st.sign, st.logabs, st.n_acc, st.extra["z0"]]
    start = [t.clone() for t in fields]

    def run():
        """A sweep from the start and the local energies after it."""
        with torch.inference_mode():
            for t, v in zip(fields, start):
                t.copy_(v)
            m.sweep(st, vg.SquareLattice(L, L), 1, 11, 0)
            e = m.local_energy(st, H)
            return [t.clone() for t in fields] + [e]

    return m, st, fields, start, run


def test_threads_on_their_own_streams():
    """Few walkers whose connected configurations run in groups side by side,
    and walker groups: each thread's results are those of the calls alone."""
    sizes = [200, 300, 4096, 5000, 150, 4200]
    jobs = [setup(B, i + 1)[-1] for i, B in enumerate(sizes)]
    want = [j() for j in jobs]
    torch.cuda.synchronize()
    bad, errors = [0] * len(jobs), []

    def work(i):
        try:
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                for _ in range(12):
                    out = jobs[i]()
                    st.synchronize()
                    bad[i] += not all(torch.equal(a, b) for a, b in zip(out, want[i]))
        except Exception as e:   # reported in the test's thread
            errors.append((i, repr(e)))

    ths = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in ths:
        t.start()
    for t in ths:
        t.join()
    assert errors == []
    assert bad == [0] * len(jobs)


def test_eager_calls_beside_a_capture():
    """A capture holds the streams that its sweep has joined until it ends; a
    thread that sweeps meanwhile gets other ones."""
    m, st, fields, start, _ = setup(4100, 1)
    m2, st2, fields2, start2, _ = setup(4500, 2)
    g = vg.SquareLattice(L, L)

    def sweep(mm, s, f, v):
        with torch.inference_mode():
            for a, b in zip(f, v):
                a.copy_(b)
            mm.sweep(s, g, 1, 11, 0)

    want = []
    for mm, s, f, v in ((m, st, fields, start), (m2, st2, fields2, start2)):
        sweep(mm, s, f, v)
        torch.cuda.synchronize()
        want.append([t.clone() for t in f])
    out, errors = [], []

    def eager():
        try:
            side = torch.cuda.Stream()
            with torch.cuda.stream(side):
                sweep(m2, st2, fields2, start2)
                side.synchronize()
        except Exception as e:   # reported in the test's thread
            errors.append(repr(e))

    graph = torch.cuda.CUDAGraph()
    with torch.inference_mode():
        with torch.cuda.graph(graph, capture_error_mode="thread_local"):
            for a, b in zip(fields, start):
                a.copy_(b)
            m.sweep(st, g, 1, 11, 0)
            th = threading.Thread(target=eager)
            th.start()
            th.join()
            m.sweep(st, g, 1, 12, 1)
    assert errors == []
    assert all(torch.equal(a, b) for a, b in zip(fields2, want[1]))
    sweep(m, st, fields, start)
    with torch.inference_mode():
        m.sweep(st, g, 1, 12, 1)
    torch.cuda.synchronize()
    two = [t.clone() for t in fields]
    for _ in range(2):
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(fields, two))
