"""Workspaces whose size is a choice shrink where memory does not allow them."""

import pytest
import torch

from vmc_torch_gb300 import _lib


@pytest.mark.parametrize("limit,rows,least,want", [(100, 64, 1, 64), (100, 1000, 1, 62), (100, 1000, 90, 90), (5, 7, 2, 3)])
def test_rows_are_halved(limit, rows, least, want):
    tried = []

    def alloc(n):
        tried.append(n)
        if n > limit:
            raise torch.OutOfMemoryError("full")
        return "w%d" % n

    assert _lib.most_rows(alloc, rows, least) == (want, "w%d" % want)
    assert tried[0] == rows and tried == sorted(tried, reverse=True)


def test_least_is_the_end():
    def alloc(n):
        raise torch.OutOfMemoryError("full")

    with pytest.raises(torch.OutOfMemoryError):
        _lib.most_rows(alloc, 50, 10)


def test_other_errors_pass():
    def alloc(n):
        raise ValueError("no")

    with pytest.raises(ValueError):
        _lib.most_rows(alloc, 50)


@pytest.mark.gpu
def test_calls_beside_little_free_memory():
    """64 MB left to this process: local energies of few walkers, log-derivatives
    and an FP64 Gram matrix, which take 84, 100 and 290 MB by choice, give what
    they give otherwise."""
    import vmc_torch_gb300 as vg
    dev = torch.device("cuda", 0)
    L, nf, B = 6, 32, 200
    g = torch.Generator().manual_seed(1)
    m = vg.NNBF_GB300(L * L, nf, precision="mixed", generator=g).to(dev)
    H = vg.spinful_Fermi_Hubbard_square_lattice_torch(L, L, 1.0, 8.0, nf, n_fermions_per_spin=(nf // 2, nf // 2))
    H.precompute_hops_gpu(dev)
    x0 = vg.init_walkers(B, L * L, nf // 2, nf // 2, seed=3, device=dev)
    X = torch.randn(1000, 20000, generator=g, dtype=torch.float64).to(dev)
    big = vg.init_walkers(3000, L * L, nf // 2, nf // 2, seed=4, device=dev)
    with torch.inference_mode():
        st, st2 = m.bind_state(x0), m._eval_state(big)
        out = torch.empty((3000, m.n_params - m.n_params_out_w), device=dev)
        kg, kh = torch.empty((3000, 2 * L * L * nf), device=dev), torch.empty((3000, 256), device=dev)

    def run():
        T = torch.empty((1000, 1000), dtype=torch.float64, device=dev)
        solver = vg.MinSRGB300()
        with torch.inference_mode():
            e = m.local_energy(st, H)
            m._adjoint(st2, dense=out, g=kg, h=kh)
        solver._tc_gram_f64(X, T, 0.0, dev)
        solver._check_tc()
        return e.clone(), out.clone().cpu(), T.cpu()

    want = run()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hold = torch.empty(out.numel() * 4 + (8 << 20), dtype=torch.uint8, device=dev)   # room for run()'s own copies
    total = torch.cuda.get_device_properties(0).total_memory
    try:
        limit = torch.cuda.memory_reserved() + (64 << 20)
        del hold
        torch.cuda.set_per_process_memory_fraction(limit / total)
        with pytest.raises(torch.OutOfMemoryError):
            torch.empty(limit, dtype=torch.uint8, device=dev)
        got = run()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(want[0], got[0])
    n = X.norm(dim=1).cpu()
    assert ((want[2] - got[2]).abs() <= 2.0 ** -46 * n[:, None] * n[None]).all()
    assert torch.equal(torch.isfinite(want[1]), torch.isfinite(got[1]))
    assert (want[1] - got[1]).abs().max() <= 1e-3 * want[1].abs().max()
