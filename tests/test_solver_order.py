"""The solver queues everything that does not depend on the factorisation's
outcome before it first waits for the GPU (recorded calls, no GPU)."""

import types

import pytest
import torch

from vmc_torch_gb300 import optimizer as opt


@pytest.mark.parametrize("Ns", [8, 600])
def test_waits_come_after_the_solves(monkeypatch, Ns):
    log = []

    def call(name, *args):
        log.append(name)
        if name == "vmc_sr_cholesky_tc_work_bytes":
            args[1]._obj.value = 256

    monkeypatch.setattr(opt, "_lib", types.SimpleNamespace(
        call=call, ptr=lambda t: t, stream_of=lambda d: None, message=str))

    def gram(T, shift):
        log.append("gram")

    gram.check = lambda: log.append("wait: gram status")
    tolist = torch.Tensor.tolist

    def noted(t):
        log.append("wait: flags")
        return tolist(t)

    monkeypatch.setattr(torch.Tensor, "tolist", noted)
    E = torch.zeros(Ns, dtype=torch.float64)
    x, info = opt.MinSRGB300._factor_solve(gram, E, 0.0, Ns, 1e-3, torch.device("cpu"), opt._Stages(False))
    assert info == 0 and x.shape == (Ns,)
    first = min(i for i, n in enumerate(log) if n.startswith("wait"))
    assert "wait: gram status" in log and "wait: flags" in log
    for name in ("gram", "vmc_sr_cholesky" if Ns == 8 else "vmc_sr_cholesky_tc", "vmc_sr_rhs", "vmc_sr_cholesky_solve"):
        assert log.index(name) < first, log


def test_a_failed_gram_raises_before_its_factor_is_used(monkeypatch):
    monkeypatch.setattr(opt, "_lib", types.SimpleNamespace(
        call=lambda *a: None, ptr=lambda t: t, stream_of=lambda d: None, message=str))

    def gram(T, shift):
        pass

    def fail():
        raise ValueError("vmc_sr_gram_tc: timeout")

    gram.check = fail
    E = torch.zeros(4, dtype=torch.float64)
    with pytest.raises(ValueError, match="vmc_sr_gram_tc"):
        opt.MinSRGB300._factor_solve(gram, E, 0.0, 4, 1e-3, torch.device("cpu"), opt._Stages(False))


def test_the_first_of_two_gram_products_is_not_forgotten(monkeypatch):
    """The factored form makes two products; a status set by either is raised."""
    calls = []

    def call(name, *args):
        if name == "vmc_sr_gram_tc":
            calls.append(args[-2])
            if len(calls) == 1:
                args[-2][0] = 7

    monkeypatch.setattr(opt, "_lib", types.SimpleNamespace(
        call=call, ptr=lambda t: t, stream_of=lambda d: None, message=lambda v: "status %d" % v))
    solver = opt.MinSRGB300()
    dev = torch.device("cpu")
    X, T = torch.ones(3, 5), torch.zeros(3, 3, dtype=torch.float64)
    for _ in range(2):
        solver._tc_gram(X, T, 1.0, None, 0.0, 0, dev)
    assert len(calls) == 2
    with pytest.raises(ValueError, match="status 7"):
        solver._check_tc()
