"""The work that a program built on this package has it do, as cases that can be timed.

A variational Monte Carlo run samples configurations, measures their local
energies, differentiates their log-amplitudes and solves for the parameter
update, over and over, with one of three wavefunctions.  Each kind of case
below is one such call (or, for ``vmc_step``, the whole iteration), made
through the package's public classes and functions:

  vmc_step       one iteration of ``VMC_GB300.run_vmc_loop`` with the Slater model
  slater_sweep   ``MetropolisExchangeSpinfulSamplerGB300.step``, Slater
  slater_measure parameter update, then local energies and log-derivatives, Slater
  nnbf_sweep     the sampler's step, neural backflow
  nnbf_energy    local energies, neural backflow
  nnbf_grads     log-derivatives, neural backflow: full rows or Kronecker factors
  minsr_dense    ``MinSRGB300.solve`` on a matrix of log-derivatives
  minsr_factored ``MinSRGB300.solve`` on Kronecker-factored log-derivatives
  peps_sweep     the sampler's step, fermionic PEPS (chi-truncated or exact)
  peps_energy    local energies, fermionic PEPS
  peps_grads     log-derivatives, fermionic PEPS
  proposal_train one training epoch of the learned proposal
"""
import math

import numpy as np
import torch

DEV = "cuda"

# Lattices and electron numbers of the repository's tests, examples and benchmark:
# 4x2 at half filling, 4x4, 6x6 with 16+16, 8x8 at and below half filling.
HALF = 2          # n_up = n_dn = N/2
SLATER_LATTICES = [(4, 2), (4, 4), (6, 4), (6, 6), (8, 8)]
# the mixed-precision backflow kernels take 32 or 64 electrons
MIXED_SYSTEMS = [(8, 4, 16, 16), (6, 6, 16, 16), (8, 8, 16, 16), (8, 8, 32, 32)]


def listed():
    return [
        # the package's first example: a small system, where a step is launches and host time
        {"name": "vmc-step-slater-4x2", "kind": "vmc_step", "Lx": 4, "Ly": 2, "nu": 4, "nd": 4, "B": 512},
        # sampling of the largest Slater determinant, 64 orbitals
        {"name": "slater-sweep-8x8", "kind": "slater_sweep", "Lx": 8, "Ly": 8, "nu": 32, "nd": 32, "B": 4096},
        # a doped lattice with an odd electron number and an odd number of walkers, after a parameter update
        {"name": "slater-measure-8x8-doped", "kind": "slater_measure", "Lx": 8, "Ly": 8, "nu": 28, "nd": 27,
         "B": 1501},
        # the benchmark's headline: one 112-edge sweep of 16384 walkers
        {"name": "nnbf-sweep-8x8", "kind": "nnbf_sweep", "Lx": 8, "Ly": 8, "nu": 32, "nd": 32, "B": 16384},
        # local energies of the doped 6x6 lattice (32 electrons), odd number of walkers
        {"name": "nnbf-energy-6x6", "kind": "nnbf_energy", "Lx": 6, "Ly": 6, "nu": 16, "nd": 16, "B": 1501},
        # log-derivatives of the benchmark's model at scale: the output layer as Kronecker factors
        {"name": "nnbf-grads-8x8", "kind": "nnbf_grads", "Lx": 8, "Ly": 8, "nu": 32, "nd": 32, "B": 8192,
         "precision": "mixed", "factored": True},
        # double-precision log-derivatives of a small model, full rows
        {"name": "nnbf-grads-4x2-fp64", "kind": "nnbf_grads", "Lx": 4, "Ly": 2, "nu": 4, "nd": 4, "B": 301,
         "precision": "fp64", "factored": False},
        # natural-gradient step of the 8x8 Slater model (8192 parameters, FP64)
        {"name": "minsr-slater-8x8", "kind": "minsr_dense", "Ns": 2049, "Np": 8192, "dtype": "float64"},
        # natural-gradient step of the 8x8 backflow model (2.2 million parameters)
        {"name": "minsr-nnbf-8x8", "kind": "minsr_factored", "Lx": 8, "Ly": 8, "nf": 64, "Ns": 8192},
        # sampling of the 6x6 PEPS with the boundary truncated to 16
        {"name": "peps-sweep-6x6-chi16", "kind": "peps_sweep", "Lx": 6, "Ly": 6, "nu": 16, "nd": 16, "D": 4,
         "chi": 16, "B": 1024},
        # log-derivatives of the 6x6 PEPS, exact contraction
        {"name": "peps-grads-6x6", "kind": "peps_grads", "Lx": 6, "Ly": 6, "nu": 16, "nd": 16, "D": 4, "chi": 0,
         "B": 512},
        # one epoch of the learned proposal over recorded samples of the 8x8 model
        {"name": "proposal-train-8x8", "kind": "proposal_train", "Lx": 8, "Ly": 8, "nu": 32, "nd": 32, "n": 16384,
         "batch": 16384},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _filling(rng, Lx, Ly):
    """Half filling, or up to a fifth fewer electrons, one spin possibly odd one out."""
    n = Lx * Ly // HALF
    nu = n if rng.random() < 0.5 else rng.randint(max(1, int(0.8 * n)), n)
    return nu, max(1, nu - rng.randint(0, 1))


def draw(rng):
    kind = rng.choice(["vmc_step", "slater_sweep", "slater_measure", "nnbf_sweep", "nnbf_energy", "nnbf_grads",
                       "minsr_dense", "minsr_factored", "peps_sweep", "peps_energy", "peps_grads", "proposal_train"])
    c = {"kind": kind}
    if kind == "vmc_step":
        c.update(Lx=4, Ly=rng.choice([2, 4]), B=_log_int(rng, 128, 512))
        c["nu"], c["nd"] = _filling(rng, c["Lx"], c["Ly"])
    elif kind in ("slater_sweep", "slater_measure"):
        c["Lx"], c["Ly"] = rng.choice(SLATER_LATTICES)
        c["nu"], c["nd"] = _filling(rng, c["Lx"], c["Ly"])
        c["B"] = _log_int(rng, 128, 4096 if kind == "slater_sweep" else 2048)
    elif kind in ("nnbf_sweep", "nnbf_energy"):
        c["Lx"], c["Ly"], c["nu"], c["nd"] = rng.choice(MIXED_SYSTEMS)
        c["B"] = _log_int(rng, 256, 16384 if kind == "nnbf_sweep" else 4096)
    elif kind == "nnbf_grads":
        if rng.random() < 0.7:
            c["Lx"], c["Ly"], c["nu"], c["nd"] = rng.choice(MIXED_SYSTEMS)
            c.update(precision="mixed", factored=rng.random() < 0.75)
            c["B"] = _log_int(rng, 128, 8192) if c["factored"] else _log_int(rng, 16, 256)
        else:
            c["Lx"], c["Ly"] = rng.choice([(4, 2), (4, 4)])
            c["nu"], c["nd"] = _filling(rng, c["Lx"], c["Ly"])
            c.update(precision="fp64", factored=rng.random() < 0.5, B=_log_int(rng, 64, 512))
    elif kind == "minsr_dense":
        c["dtype"] = rng.choice(["float64", "float32"])
        c["Ns"] = _log_int(rng, 128, 2049)
        c["Np"] = _log_int(rng, 2 * c["Ns"], 8192 if c["dtype"] == "float64" else 32768)
    elif kind == "minsr_factored":
        Lx, Ly, nu, nd = rng.choice(MIXED_SYSTEMS)
        c.update(Lx=Lx, Ly=Ly, nf=nu + nd, Ns=_log_int(rng, 512, 8192))
    elif kind in ("peps_sweep", "peps_energy", "peps_grads"):
        Lx, Ly, nu, nd, D, chi = rng.choice([(6, 6, 16, 16, 4, 16), (6, 6, 16, 16, 4, 0), (4, 4, 8, 8, 4, 8),
                                             (4, 4, 7, 7, 4, 0), (6, 6, 18, 18, 2, 0)])
        c.update(Lx=Lx, Ly=Ly, nu=nu, nd=nd, D=D, chi=chi)
        c["B"] = _log_int(rng, 64, 1024 if kind == "peps_sweep" else 512)
    else:
        c["Lx"], c["Ly"], c["nu"], c["nd"] = rng.choice([(6, 6, 16, 16), (8, 8, 32, 32)])
        c["batch"] = _log_int(rng, 1024, 16384)
        c["n"] = c["batch"]
    return c


# ---- inputs ------------------------------------------------------------------------------------

def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(1000003 * int(seed) + salt)


def _configs(c, seed, B=None):
    """(B, N) int64 configurations (0 empty, 1 down, 2 up, 3 both), uniform over the sector."""
    g = _gen(seed, 1)
    B = c["B"] if B is None else B
    N = c["Lx"] * c["Ly"]
    up = torch.rand(B, N, generator=g, device=DEV).argsort(1) < c["nu"]
    dn = torch.rand(B, N, generator=g, device=DEV).argsort(1) < c["nd"]
    return 2 * up.long() + dn.long()


def _lattice(c):
    import vmc_torch_gb300 as vg
    H = vg.spinful_Fermi_Hubbard_square_lattice_torch(c["Lx"], c["Ly"], 1.0, 8.0, c["nu"] + c["nd"],
                                                      n_fermions_per_spin=(c["nu"], c["nd"]))
    H.precompute_hops_gpu(DEV)
    return H


def _slater(c, seed):
    import vmc_torch_gb300 as vg
    g = torch.Generator().manual_seed(int(seed))
    return vg.SlaterDeterminant_GB300(2 * c["Lx"] * c["Ly"], c["nu"] + c["nd"], init_std=0.1, generator=g).to(DEV)


def _nnbf(c, seed):
    import vmc_torch_gb300 as vg
    g = torch.Generator().manual_seed(int(seed))
    return vg.NNBF_GB300(c["Lx"] * c["Ly"], c["nu"] + c["nd"], precision=c.get("precision", "mixed"),
                         generator=g).to(DEV)


def _peps(c, seed):
    import vmc_torch_gb300 as vg
    g = torch.Generator().manual_seed(int(seed))
    return vg.FPEPS_GB300(c["Lx"], c["Ly"], c["D"], max_bond=c["chi"] or None, precision="fp32", generator=g).to(DEV)


def _sampled(c, seed, model, H, sweeps):
    """Walkers as a run has them: a few sweeps from uniform configurations."""
    import vmc_torch_gb300 as vg
    fxs = _configs(c, seed)
    return vg.MetropolisExchangeSpinfulSamplerGB300(seed=int(seed)).burn_in(fxs, model, H.graph, sweeps)


def _logderiv_like(Ns, Np, seed, salt, dtype):
    """Rows as log-derivatives have them: a mean, 64 correlated directions of falling weight, noise."""
    g = _gen(seed, salt)
    r = min(64, Np)
    w = torch.arange(1, r + 1, device=DEV, dtype=torch.float32) ** -0.5
    Z = torch.randn(Ns, r, generator=g, device=DEV)
    out = torch.empty(Ns, Np, dtype=dtype, device=DEV)
    for a in range(0, Np, 16384):       # blocks of columns, so that no second matrix of this size is held
        b = min(Np, a + 16384)
        W = torch.randn(r, b - a, generator=g, device=DEV) * w[:, None]
        mean = 0.1 * torch.randn(b - a, generator=g, device=DEV)
        blk = torch.zeros(Ns, b - a, device=DEV)
        for k in range(0, r, 8):        # elementwise sums: the same values on every run
            for q in range(k, min(r, k + 8)):
                blk.addcmul_(Z[:, q:q + 1], W[q:q + 1])
        out[:, a:b] = 0.3 * blk + mean + 0.3 * torch.randn(Ns, b - a, generator=g, device=DEV)
    return out, Z


def _energies(Z, seed):
    g = _gen(seed, 7)
    return (Z[:, :4].double().sum(1) + torch.randn(Z.shape[0], generator=g, device=DEV, dtype=torch.float64) - 30.0)


def prepare(case, seed):
    import vmc_torch_gb300 as vg
    c, k, seed = case, case["kind"], int(seed)
    s = {"case": c, "kind": k}
    if k == "vmc_step":
        s["H"] = _lattice(c)
        s["model"] = _slater(c, seed)
        s["fxs"] = _configs(c, seed)
        s["vmc"] = vg.VMC_GB300(vg.MetropolisExchangeSpinfulSamplerGB300(seed=seed), vg.MinSRGB300(),
                                vg.SGDGB300(learning_rate=0.02))
        s["cfg"] = vg.VMCLoopConfig(vmc_steps=1, ns_per_rank=c["B"], grad_batch_size=c["B"],
                                    n_params=s["model"].n_params, nsites=c["Lx"] * c["Ly"], learning_rate=0.02,
                                    diag_shift=1e-3, use_log_amp=True)
    elif k == "slater_sweep":
        s["H"] = _lattice(c)
        s["model"] = _slater(c, seed)
        s["fxs"] = _configs(c, seed)
        s["sampler"] = vg.MetropolisExchangeSpinfulSamplerGB300(seed=seed)
    elif k == "slater_measure":
        s["H"] = _lattice(c)
        s["model"] = _slater(c, seed)
        s["fxs"] = _sampled(c, seed, s["model"], s["H"], 4)
        s["opt"] = vg.SGDGB300(learning_rate=1e-4)
        s["dp"] = torch.randn(s["model"].n_params, generator=_gen(seed, 3), device=DEV, dtype=torch.float64)
    elif k in ("nnbf_sweep", "nnbf_energy", "nnbf_grads"):
        s["H"] = _lattice(c)
        s["model"] = _nnbf(c, seed)
        if k == "nnbf_sweep":
            s["fxs"] = _configs(c, seed)
            s["sampler"] = vg.MetropolisExchangeSpinfulSamplerGB300(seed=seed)
        else:
            s["fxs"] = _sampled(c, seed, s["model"], s["H"], 4)
    elif k == "minsr_dense":
        s["O"], Z = _logderiv_like(c["Ns"], c["Np"], seed, 11, getattr(torch, c["dtype"]))
        s["E"] = _energies(Z, seed)
        s["E_mean"] = float(s["E"].mean())
        s["solver"] = vg.MinSRGB300()
    elif k == "minsr_factored":
        n_orb = 2 * c["Lx"] * c["Ly"]
        Ng, Nh = n_orb * c["nf"], 256
        Nd = 2 * Ng + Nh * n_orb + Nh + Nh * Nh + Nh   # M_base, W0, b0, W1, b1, out_b
        dense, Z = _logderiv_like(c["Ns"], Nd, seed, 12, torch.float32)
        g, _ = _logderiv_like(c["Ns"], Ng, seed, 13, torch.float32)
        g *= 0.01                                        # the backflow's scale
        # rows of unoccupied orbitals carry no derivative
        occ = torch.rand(c["Ns"], n_orb, generator=_gen(seed, 14), device=DEV).argsort(1) < c["nf"]
        g.view(c["Ns"], n_orb, c["nf"]).mul_(occ[:, :, None])
        h = torch.nn.functional.gelu(torch.randn(c["Ns"], Nh, generator=_gen(seed, 15), device=DEV))
        s["O"] = vg.FactoredO(dense, g, h, Nd - Ng)
        s["E"] = _energies(Z, seed)
        s["E_mean"] = float(s["E"].mean())
        s["solver"] = vg.MinSRGB300()
    elif k in ("peps_sweep", "peps_energy", "peps_grads"):
        s["H"] = _lattice(c)
        s["model"] = _peps(c, seed)
        s["fxs"] = _sampled(c, seed, s["model"], s["H"], 2)
        s["sampler"] = vg.MetropolisExchangeSpinfulSamplerGB300(seed=seed + 1)
    else:
        from vmc_torch_gb300.proposal import LearnedProposal
        s["H"] = _lattice(c)
        model = _nnbf(c, seed)
        p = LearnedProposal(c["Lx"] * c["Ly"], s["H"].edges_on(DEV), device=DEV, seed=seed, buffer=c["n"])
        fxs = _configs(c, seed, c["n"])
        vg.evaluate_energy(fxs, model, s["H"])
        p.record(model)
        s["p"], s["gen"] = p, _gen(seed, 5)
    return s


def run(s):
    import vmc_torch_gb300 as vg
    c, k = s["case"], s["kind"]
    if k == "vmc_step":
        hist, fxs = s["vmc"].run_vmc_loop(s["fxs"], s["model"], s["H"], s["H"].graph, s["cfg"])
        return {"energy": hist[0], "fxs": fxs, "params": s["model"].params[0].data}
    if k in ("slater_sweep", "nnbf_sweep", "peps_sweep"):
        fxs, (sign, logabs) = s["sampler"].step(s["fxs"], s["model"], s["H"].graph, use_log_amp=True)
        return {"fxs": fxs, "sign": sign, "logabs": logabs}
    if k == "slater_measure":
        s["opt"].step(s["model"], s["dp"], DEV)
        E, eloc = vg.evaluate_energy(s["fxs"], s["model"], s["H"], use_log_amp=True)
        O, (sign, logabs) = vg.compute_grads_gpu(s["fxs"], s["model"], use_log_amp=True)
        return {"E": E, "eloc": eloc, "O": O, "sign": sign, "logabs": logabs}
    if k in ("nnbf_energy", "peps_energy"):
        E, eloc = vg.evaluate_energy(s["fxs"], s["model"], s["H"], use_log_amp=True)
        return {"E": E, "eloc": eloc}
    if k == "nnbf_grads" and c["factored"]:
        O, (sign, logabs) = vg.compute_grads_factored(s["fxs"], s["model"])
        return {"dense": O.dense, "g": O.g, "h": O.h, "sign": sign, "logabs": logabs}
    if k in ("nnbf_grads", "peps_grads"):
        O, (sign, logabs) = vg.compute_grads_gpu(s["fxs"], s["model"], use_log_amp=True)
        return {"O": O, "sign": sign, "logabs": logabs}
    if k in ("minsr_dense", "minsr_factored"):
        dp, _, info = s["solver"].solve(local_o=s["O"], local_energies=s["E"], energy_mean=s["E_mean"],
                                        total_samples=c["Ns"], n_params=s["O"].shape[1], diag_shift=1e-3,
                                        device=DEV, run_sr=True)
        return {"dp": dp, "info": info}
    p = s["p"]
    loss = p.train(epochs=1, batch=c["batch"], generator=s["gen"])
    return {"params": p.params, "m1": p.m1, "m2": p.m2, "loss": loss}


# ---- what a pass cannot do without --------------------------------------------------------------

def work(case):
    c, k = case, case["kind"]
    if "Lx" in c:
        N = c["Lx"] * c["Ly"]
        E = c["Lx"] * (c["Ly"] - 1) + c["Ly"] * (c["Lx"] - 1)
        nf = c.get("nf") or c["nu"] + c["nd"]
        n_orb = 2 * N
    B = c.get("B", 0)
    changed, accepted = 0.75, 0.25      # proposals that change a walker; that are accepted (random to half filling)
    hops = 1.0                          # non-zero hops per edge and walker (two spins, half of them blocked)
    if k == "vmc_step" or k == "slater_sweep":
        # ratio of a proposal: one nf-long product (two for an exchange); accepted: rank-1/2 update of nf^2
        f = B * E * (changed * 1.5 * 2 * nf + accepted * 1.5 * 4 * nf * nf)
        by = 16 * B * N + 16 * B + 8 * n_orb * nf
        if k == "vmc_step":
            Np = n_orb * nf
            f += B * (8 / 3 * nf ** 3 + E * hops * 2 * nf) + B * B * Np + B ** 3 / 3 + 4 * B * Np
            by += 8 * 2 * Np
        return {"bytes": by, "flops": f}
    if k == "slater_measure":
        return {"bytes": 8 * B * N + 8 * B * n_orb * nf + 24 * B + 16 * n_orb * nf,
                "flops": B * (2 * nf ** 3 + E * hops * 2 * nf)}
    if k.startswith("nnbf"):
        mlp = 2 * 256 * 256 + 2 * 256 * nf * nf                 # second layer, rows of the occupied orbitals
        lu = 2 / 3 * nf ** 3
        wb = 2 * (256 * n_orb + 256 * 256 + 256 * n_orb * nf)   # weights once, 16 bits
        if k == "nnbf_sweep":
            return {"bytes": 16 * B * N + 16 * B + wb, "flops": B * E * changed * (mlp + lu) + B * (mlp + lu)}
        if k == "nnbf_energy":
            return {"bytes": 8 * B * N + 8 * B + wb, "flops": B * E * hops * (mlp + lu)}
        e = 4 if c["precision"] == "mixed" else 8
        Ng = n_orb * nf
        Nd = 2 * Ng + 256 * n_orb + 256 + 256 * 256 + 256
        cols = Nd + Ng + 256 if c["factored"] else Nd + 256 * Ng
        return {"bytes": 8 * B * N + e * B * cols + e * (256 * n_orb + 256 * 256 + 256 * Ng),
                "flops": B * (3 * 2 * 256 * 256 + 2 * 2 * 256 * nf * nf + 2 * nf ** 3)}
    if k == "minsr_dense":
        e = 8 if c["dtype"] == "float64" else 4
        Ns, Np = c["Ns"], c["Np"]
        return {"bytes": e * Ns * Np + 8 * Ns + 8 * Np, "flops": Ns * Ns * Np + Ns ** 3 / 3 + 4 * Ns * Np}
    if k == "minsr_factored":
        Ns, Ng = c["Ns"], n_orb * nf
        Nd = 2 * Ng + 256 * n_orb + 256 + 256 * 256 + 256
        return {"bytes": 4 * Ns * (Nd + Ng + 256) + 8 * (Nd + 256 * Ng),
                "flops": Ns * Ns * (Nd + Ng + 256) + Ns ** 3 / 3 + 4 * Ns * Nd + 3 * 2 * Ns * Ng * 256}
    if k.startswith("peps"):
        D = c["D"]
        site = 2 * D ** c["Ly"] * D * D / 2                     # a site absorbed into a boundary of D^Ly, even half
        amp = N * site
        tb = 4 * N * 4 * D ** 4
        if k == "peps_sweep":
            return {"bytes": 16 * B * N + 16 * B + tb, "flops": B * E * changed * 2 * c["Ly"] * site}
        if k == "peps_energy":
            return {"bytes": 8 * B * N + 8 * B + tb, "flops": B * E * hops * 2 * c["Ly"] * site}
        return {"bytes": 8 * B * N + 4 * B * N * 4 * D ** 4 + 16 * B + tb, "flops": 3 * B * amp}
    Kin = ((n_orb + 63) // 64) * 64
    params = 512 * Kin + 512 * 512 + 512 * 256
    return {"bytes": c["n"] * (16 + 8 * E) + 4 * 6 * params, "flops": 6 * c["n"] * params}


# ---- the same in 64 bits, in plain torch ---------------------------------------------------------

def _edges(Lx, Ly):
    out = []
    for r in range(Lx):
        for q in range(Ly):
            if q + 1 < Ly:
                out.append((r * Ly + q, r * Ly + q + 1))
            if r + 1 < Lx:
                out.append((r * Ly + q, (r + 1) * Ly + q))
    return out


def _bits(fxs):
    """(B, 2N) occupations, spin up then spin down."""
    return torch.cat([(fxs >> 1) & 1, fxs & 1], 1)


def _orbs(bits, nf):
    """(B, nf) occupied orbitals, ascending."""
    return bits.nonzero()[:, 1].view(bits.shape[0], nf)


def _local_energy(fxs, Lx, Ly, amp, chunk):
    """U * doublons + sum over hops of -t * phase * psi(x')/psi(x); amp(configs) -> (sign, log|psi|)."""
    B, N = fxs.shape
    s0, l0 = amp(fxs)
    e = 8.0 * (fxs == 3).sum(1).double()
    b = _bits(fxs)
    # position of each mode (site, spin) in the order down_0, up_0, down_1, up_1, ...
    who, conf, sgn = [], [], []
    for i, j in _edges(Lx, Ly):
        for spin in (0, 1):                       # 0: down, 1: up
            v = 2 if spin else 1
            oi, oj = (fxs[:, i] // v) % 2, (fxs[:, j] // v) % 2
            w = (oi != oj).nonzero()[:, 0]
            y = fxs[w].clone()
            y[:, i] += v * (oj - oi)[w]
            y[:, j] += v * (oi - oj)[w]
            mid = b[w][:, i + 1:j].sum(1) + b[w][:, N + i + 1:N + j].sum(1)
            mid = mid + (b[w][:, N + j] if spin else b[w][:, i])
            who.append(w)
            conf.append(y)
            sgn.append(-1.0 * (1 - 2 * (mid % 2)).double())
    who, conf, sgn = torch.cat(who), torch.cat(conf), torch.cat(sgn)
    for a in range(0, who.numel(), chunk):
        w = who[a:a + chunk]
        s, l = amp(conf[a:a + chunk])
        e.index_add_(0, w, sgn[a:a + chunk] * s * s0[w] * torch.exp(l - l0[w]))
    return e


def _gelu(x):
    return 0.5 * x * (1 + torch.erf(x / math.sqrt(2.0)))


def _dgelu(x):
    return 0.5 * (1 + torch.erf(x / math.sqrt(2.0))) + x * torch.exp(-0.5 * x * x) / math.sqrt(2 * math.pi)


def _nnbf_forward(ps, fxs, nf):
    Mb, w0, b0, w1, b1, ow, ob = ps
    n_orb = Mb.shape[0]
    bits = _bits(fxs)
    z0 = bits.double() @ w0.t() + b0
    h1 = _gelu(z0)
    z1 = h1 @ w1.t() + b1
    h2 = _gelu(z1)
    M = Mb + 0.01 * (h2 @ ow.t() + ob).view(-1, n_orb, nf)
    orbs = _orbs(bits, nf)
    A = torch.gather(M, 1, orbs[:, :, None].expand(-1, -1, nf))
    return bits, z0, h1, z1, h2, A, orbs


def _minsr_exact(X, b, extra=None):
    """(O~^T x, x) for centred and scaled rows X, with the Gram matrix `extra` of further columns."""
    T = X @ X.t()
    if extra is not None:
        T += extra
    T.diagonal().add_(1e-3)
    x = torch.cholesky_solve(b[:, None], torch.linalg.cholesky(T))[:, 0]
    return X.t() @ x, x


def _peps_sites(T, fxs, Lx, Ly):
    """The walkers' site tensors with the fermionic signs: list of (B, l, u, r, d)."""
    D = T.shape[-1]
    par = torch.arange(D, device=T.device) % 2
    cnt = torch.tensor([0, 1, 1, 2], device=T.device)[fxs].view(-1, Lx, Ly)
    out = []
    for r in range(Lx):
        for q in range(Ly):
            t = T[r, q][fxs[:, r * Ly + q]]
            if r > 0:
                left = cnt[:, r, :q].sum(1)
                odd = (par[None, None, :] * ((par[None, :, None] + left[:, None, None]) % 2)) % 2   # (B, l, u)
                t = t * (1 - 2 * odd).to(t.dtype)[:, :, :, None, None]
            out.append(t)
    return out


def _peps_contract(sites, Lx, Ly):
    """Row by row into the full vector over the Ly vertical legs; returns (sign, log|.|) of the plain contraction."""
    D = sites[0].shape[-1]
    B = sites[0].shape[0]
    S = torch.zeros(B, D ** Ly, dtype=torch.float64, device=sites[0].device)
    S[:, 0] = 1
    log = torch.zeros(B, dtype=torch.float64, device=S.device)
    for r in range(Lx):
        W = torch.nn.functional.pad(S[:, None], (0, 0, 0, D - 1))          # (B, h, legs), h = 0 to begin with
        for q in range(Ly):
            W = W.reshape(B, D, D ** q, D, D ** (Ly - q - 1))
            W = torch.einsum("bhpuq,bhurd->brpdq", W, sites[r * Ly + q])
        S = W.reshape(B, D, D ** Ly)[:, 0]
        m = S.detach().abs().amax(1)
        S = S / m[:, None]
        log = log + torch.log(m)
    z = S[:, 0]
    return torch.sign(z.detach()), log + torch.log(z.abs())


def _peps_amp(T, Lx, Ly, chunk=512):
    def amp(fxs):
        s, l = [], []
        for a in range(0, fxs.shape[0], chunk):
            x = fxs[a:a + chunk]
            sg, lg = _peps_contract(_peps_sites(T, x, Lx, Ly), Lx, Ly)
            k = ((x == 1) | (x == 2)).sum(1)
            s.append(sg * (1 - 2 * ((k * (k - 1) // 2) % 2)).double())
            l.append(lg)
        return torch.cat(s), torch.cat(l)
    return amp


def exact(case, seed):
    c, k = case, case["kind"]
    if k in ("vmc_step", "slater_sweep", "nnbf_sweep", "peps_sweep"):
        return None                               # a chain of accepted moves has no other form
    if k != "minsr_dense" and k != "minsr_factored" and c.get("chi"):
        return None                               # the truncated contraction is defined by its own truncations
    s = prepare(case, seed)
    if k == "minsr_dense":
        O = s["O"].double()
        X = (O - O.mean(0)) / math.sqrt(c["Ns"])
        dp, _ = _minsr_exact(X, (s["E"] - s["E"].mean()) / math.sqrt(c["Ns"]))
        return {"dp": dp, "info": None}
    if k == "minsr_factored":
        Ns = c["Ns"]
        F = s["O"]
        if Ns * Ns * F.dense.shape[1] > 2e12:
            return None                           # FP64 products of that size take too long
        G, Hh = F.g.double(), F.h.double()
        mu = G.t() @ Hh / Ns
        v = ((G @ mu) * Hh).sum(1)
        K = ((G @ G.t()) * (Hh @ Hh.t()) - v[:, None] - v[None, :] + (mu * mu).sum()) / Ns
        X = F.dense.double()
        X = (X - X.mean(0)) / math.sqrt(Ns)
        dpd, x = _minsr_exact(X, (s["E"] - s["E"].mean()) / math.sqrt(Ns), K)
        dpk = ((G * x[:, None]).t() @ Hh - x.sum() * mu) / math.sqrt(Ns)
        return {"dp": torch.cat([dpd[:F.offset], dpk.reshape(-1), dpd[F.offset:]]), "info": None}
    if k == "proposal_train":
        p, n, b = s["p"], c["n"], c["batch"]
        perm = torch.randperm(n, device=DEV, generator=s["gen"])[:b]
        occ, tgt = p.buf_occ[perm], p.buf_tgt[perm].double()
        N, E = c["Lx"] * c["Ly"], tgt.shape[1] // 2
        site = torch.arange(N, device=DEV)
        up, dn = (occ[:, :1] >> site) & 1, (occ[:, 1:] >> site) & 1
        X = torch.zeros(b, p.Kin, dtype=torch.float64, device=DEV)
        X[:, :N], X[:, N:2 * N] = up.double(), dn.double()
        flat = p.params.double().requires_grad_(True)
        sizes = [512 * p.Kin, 512, 512 * 512, 512, 256 * 512, 256]
        W1, b1, W2, b2, Wo, bo = torch.split(flat, sizes)
        h = _gelu(X @ W1.view(512, -1).t() + b1)
        h = _gelu(h @ W2.view(512, 512).t() + b2)
        lg = h @ Wo.view(256, 512).t() + bo
        e = s["H"].edges_on(DEV).long()
        valid = torch.stack([up[:, e[:, 0]] != up[:, e[:, 1]], dn[:, e[:, 0]] != dn[:, e[:, 1]]], 2).view(b, 2 * E)
        logp = torch.log_softmax(lg[:, :2 * E].masked_fill(~valid, -1e300), 1).masked_fill(~valid, 0.0)
        t = tgt.masked_fill(~valid, 0.0)
        t = t / t.sum(1, keepdim=True)
        kt = torch.arange(1, 5, device=DEV, dtype=torch.float64) / 10
        kt = kt.float().double()
        loss = (-(t * logp).sum(1) - p.kweight * (kt * torch.log_softmax(lg[:, 2 * E:2 * E + 4], 1)).sum(1)).mean()
        g, = torch.autograd.grad(loss, flat)
        f32 = np.float32
        b1_, b2_, lr, eps = float(f32(0.9)), float(f32(0.999)), float(f32(p.lr)), float(f32(1e-8))
        m1, m2 = (1 - b1_) * g, (1 - b2_) * g * g
        new = flat.detach() - lr * (m1 / (1 - b1_)) / (torch.sqrt(m2 / (1 - b2_)) + eps)
        return {"params": new, "m1": m1, "m2": m2, "loss": float(loss)}
    fxs = s["fxs"]
    B, N = fxs.shape
    nf = c["nu"] + c["nd"]
    ps = [q.detach().double() for q in s["model"].params]
    if k == "slater_measure":
        M = ps[0] - 1e-4 * s["dp"].view_as(ps[0])
        orbs = _orbs(_bits(fxs), nf)
        A = M[orbs]
        sign, logabs = torch.linalg.slogdet(A)
        G = torch.linalg.inv(A).transpose(1, 2)
        O = torch.zeros(B, 2 * N, nf, dtype=torch.float64, device=DEV)
        O.scatter_(1, orbs[:, :, None].expand(-1, -1, nf), G)
        eloc = _local_energy(fxs, c["Lx"], c["Ly"], lambda x: torch.linalg.slogdet(M[_orbs(_bits(x), nf)]), 16384)
        return {"E": eloc.mean(), "eloc": eloc, "O": O.view(B, -1), "sign": sign, "logabs": logabs}
    if k == "nnbf_energy":
        eloc = _local_energy(fxs, c["Lx"], c["Ly"], lambda x: torch.linalg.slogdet(_nnbf_forward(ps, x, nf)[5]), 4096)
        return {"E": eloc.mean(), "eloc": eloc}
    if k == "nnbf_grads":
        ow = ps[5]
        rows = []
        for a in range(0, B, 512):
            bits, z0, h1, z1, h2, A, orbs = _nnbf_forward(ps, fxs[a:a + 512], nf)
            n = bits.shape[0]
            G = torch.zeros(n, 2 * N, nf, dtype=torch.float64, device=DEV)
            G.scatter_(1, orbs[:, :, None].expand(-1, -1, nf), torch.linalg.inv(A).transpose(1, 2))
            G = G.view(n, -1)
            dz1 = 0.01 * (G @ ow) * _dgelu(z1)
            dz0 = (dz1 @ ps[3]) * _dgelu(z0)
            parts = [G, (dz0[:, :, None] * bits[:, None, :].double()).reshape(n, -1), dz0,
                     (dz1[:, :, None] * h1[:, None, :]).reshape(n, -1), dz1]
            if c["factored"]:
                rows.append((torch.cat(parts + [0.01 * G], 1).float(), 0.01 * G, h2))
            else:
                parts += [(0.01 * G[:, :, None] * h2[:, None, :]).reshape(n, -1), 0.01 * G]
                rows.append((torch.cat(parts, 1),))
        if c["factored"]:
            d, g, h = (torch.cat(x) for x in zip(*rows))
            return {"dense": d, "g": g, "h": h, "sign": None, "logabs": None}
        return {"O": torch.cat([r[0] for r in rows]), "sign": None, "logabs": None}
    T = ps[0]
    if k == "peps_energy":
        eloc = _local_energy(fxs, c["Lx"], c["Ly"], _peps_amp(T, c["Lx"], c["Ly"]), 4096)
        return {"E": eloc.mean(), "eloc": eloc}
    O = torch.zeros(B, N, 4, c["D"] ** 4, dtype=torch.float64, device=DEV)
    logs, signs = [], []
    for a in range(0, B, 64):
        x = fxs[a:a + 64]
        sites = [t.clone().requires_grad_(True) for t in _peps_sites(T, x, c["Lx"], c["Ly"])]
        sg, lg = _peps_contract(sites, c["Lx"], c["Ly"])
        grads = torch.autograd.grad(lg.sum(), sites)
        unsigned = _peps_sites(torch.ones_like(T), x, c["Lx"], c["Ly"])      # the sign of every entry
        for i, (g, u) in enumerate(zip(grads, unsigned)):
            O[a + torch.arange(x.shape[0], device=DEV), i, x[:, i]] = (g * u).reshape(x.shape[0], -1)
        kk = ((x == 1) | (x == 2)).sum(1)
        signs.append(sg * (1 - 2 * ((kk * (kk - 1) // 2) % 2)).double())
        logs.append(lg.detach())
    mask = s["model"].structure_mask(c["Lx"], c["Ly"], c["D"]).to(DEV).view(1, N, 4, -1)
    return {"O": (O * mask).reshape(B, -1), "sign": torch.cat(signs), "logabs": torch.cat(logs)}
