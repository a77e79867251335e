"""Weights written by the kernel queued right before a sweep: the sweep's first
launches are ordered after it although later ones overlap their predecessors."""

import pytest
import torch

from oracle import models as om
import vmc_torch_gb300 as vg

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("Lx,Ly,nf", [(6, 6, 32), (8, 8, 64)])
@pytest.mark.parametrize("B", [100, 4100])
def test_weights_written_before_the_sweep(Lx, Ly, nf, B):
    N = Lx * Ly
    m = vg.NNBF_GB300(N, nf, precision="mixed").to(DEV)
    with torch.no_grad():
        for p, v in zip(m.params, om.nnbf_init(N, nf, 256, 2, seed=4)):
            p.copy_(torch.as_tensor(v))
    m.invalidate()
    g = vg.SquareLattice(Lx, Ly)
    x0 = vg.init_walkers(B, N, nf // 2, nf // 2, seed=B, device=DEV)
    with torch.inference_mode():   # as the sampler runs it
        st = m.bind_state(x0)
        w1 = m.net(st.device)[0][2]
        sets = [w1.clone(), torch.randn(256, 256, device=DEV).mul_(0.1).to(torch.bfloat16)]
        fields = [st.occ, st.sign, st.logabs, st.n_acc, st.extra["z0"]]
        start = [t.clone() for t in fields]

        def sweep(k, wait):
            for t, v in zip(fields, start):
                t.copy_(v)
            w1.copy_(sets[k])
            if wait:
                torch.cuda.synchronize()
            m.sweep(st, g, 1, 5, 0)
            return [t.clone() for t in fields]

        want = [sweep(k, True) for k in range(2)]
        assert not torch.equal(want[0][2], want[1][2])
        for _ in range(10):
            for k in range(2):
                for a, b in zip(sweep(k, False), want[k]):
                    assert torch.equal(a, b)
