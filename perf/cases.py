"""Performance cases of the propagators: what their users have them do, one
public call (or forward plus backward call) per pass.

``kind`` names the call:

* ``evolve``    one system through ``Lindblad_solver.evolve`` with host arrays
* ``host``      a batch in page-locked host memory through the same call
* ``ensemble``  a batch on the device through ``engine.propagate`` (generator kept)
* ``uneven``    chains of several dimensions through ``engine.ragged_enqueue`` (groups kept)
* ``gradient``  ``adjoint.chain_observables`` forward and backward
* ``redfield``  one initial state through ``Redfield_solver.evolve`` (tensor kept)
* ``block``     a block of initial states under a dense generator, ``redfield.propagate_vec_split``
* ``spectrum``  ``spectra.correlation_spectrum`` of a batch of correlation functions

``model`` names the physical system: ``chain`` (nearest-neighbour exciton
chain with site dephasing, the disorder ensemble of ``lime_gb300.chains``),
``coupled`` (the same with long-range r^-3 couplings), ``relax`` (``coupled``
plus downhill relaxation |k><k+1|) and ``open`` (chain plus a small random
Hermitian part and three dense complex collapse operators, the chains of the
uneven batch).
"""
import math

import numpy as np
import torch

from lime_gb300 import engine, redfield, spectra
from lime_gb300.adjoint import chain_observables
from lime_gb300.oqs import Lindblad_solver

DT = 0.05
CDT = torch.complex128


def listed():
    return [
        # the smallest call: a few steps of a four-level system, latency of the whole host call counts
        dict(name="evolve_n4", kind="evolve", model="relax", n=4, steps=20, precision="fp64", states=True),
        # the single exciton chain of the reference's own example, full horizon, default precision
        dict(name="evolve_chain16", kind="evolve", model="chain", n=16, steps=2000, precision="fp64", states=False),
        # the same on the tensor-core path (time-loop latency of one instance)
        dict(name="evolve_chain16_split", kind="evolve", model="chain", n=16, steps=2000, precision="split",
             states=False),
        # static-disorder ensemble in double precision, the default of every solver
        dict(name="ensemble_fp64", kind="ensemble", model="chain", n=64, batch=512, steps=8, precision="fp64"),
        # chains with dense collapse operators in double precision, an odd size
        dict(name="open_fp64", kind="ensemble", model="open", n=37, batch=48, steps=20, precision="fp64"),
        # the disorder ensemble of the benchmark, generators on the device
        dict(name="ensemble_split", kind="ensemble", model="chain", n=64, batch=4096, steps=20, precision="split"),
        # a smaller ensemble given in host memory, results back in host memory
        dict(name="host_split", kind="host", model="chain", n=64, batch=1900, steps=20, precision="split"),
        # chains of six dimensions with dense collapse operators in one call
        dict(name="uneven_split", kind="uneven", largest=256, odd=0, chains=192, steps=8),
        # absorption: dipole correlation and its gradients, 129 levels
        dict(name="absorption_gradient", kind="gradient", n=128, batch=32, steps=32, checkpoint=16,
             precision="split"),
        # Redfield populations and states of one initial state, the reference's own call
        dict(name="redfield_evolve", kind="redfield", n=20, steps=100),
        # a block of initial states under a 9216-dimensional Redfield generator
        dict(name="redfield_block", kind="block", n=96, rhs=512, steps=4),
        # spectra of an ensemble's correlation functions
        dict(name="spectrum", kind="spectrum", n=4096, batch=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["evolve", "evolve", "host", "ensemble", "ensemble", "ensemble", "uneven", "gradient",
                       "gradient", "redfield", "redfield", "block", "spectrum"])
    if kind == "evolve":
        n = _log(rng, 2, 64)
        precision = rng.choice(["fp64", "fp64", "split"])
        model = rng.choice(["chain", "coupled", "relax"])
        if model == "relax":
            n = min(n, 24)
            model = "relax" if precision == "fp64" else "coupled"
        most = max(10, min(2000, int(2000 * (16 / n) ** 3 / (1 if model != "relax" else 2 * n - 1))))
        steps = _log(rng, 10, max(11, most))
        states = precision == "fp64" and rng.random() < 0.5
        return dict(kind=kind, model=model, n=n, steps=steps, precision=precision, states=states)
    if kind == "host":
        return dict(kind=kind, model="chain", n=rng.randint(24, 64), batch=rng.randint(920, 2048),
                    steps=rng.randint(10, 40), precision="split")
    if kind == "ensemble":
        precision = rng.choice(["fp64", "split"])
        model = rng.choice(["chain", "coupled", "open"])
        n = _log(rng, 4, 64)
        steps = rng.randint(4, 24)
        pad = n if precision == "fp64" else 64
        most = int(4096 * (64 / pad) ** 3 / steps)
        if precision == "split":
            most = 4096 if model != "open" else 1024
        elif model == "open":
            most = most // 7
        return dict(kind=kind, model=model, n=n, batch=_log(rng, 16, max(17, min(4096, most))), steps=steps,
                    precision=precision)
    if kind == "uneven":
        return dict(kind=kind, largest=rng.choice([64, 128, 256]), odd=rng.choice([0, 1, 3, 5]),
                    chains=_log(rng, 24, 256), steps=rng.randint(4, 10))
    if kind == "gradient":
        precision = rng.choice(["fp64", "split"])
        n = _log(rng, 6, 128 if precision == "split" else 40)
        steps = rng.randint(8, 32)
        return dict(kind=kind, n=n, batch=_log(rng, 4, 32), steps=steps, checkpoint=rng.choice([8, 16, 64]),
                    precision=precision)
    if kind == "redfield":
        return dict(kind=kind, n=_log(rng, 3, 22), steps=_log(rng, 20, 100))
    if kind == "block":
        return dict(kind=kind, n=_log(rng, 12, 80), rhs=_log(rng, 8, 512), steps=rng.randint(2, 6))
    n = rng.choice([_log(rng, 64, 4096), 1 << rng.randint(6, 12)])
    return dict(kind=kind, n=n, batch=_log(rng, 8, 256 if n & (n - 1) == 0 else 128))


# ------------------------------------------------------------------ inputs
def _gen(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(int(seed))


def _chain(eps, J=-0.1):
    """(B, n) site energies -> (B, n, n) nearest-neighbour Hamiltonians."""
    n = eps.shape[-1]
    H = torch.diag_embed(eps)
    k = torch.arange(n - 1, device=eps.device)
    H[:, k, k + 1] = J
    H[:, k + 1, k] = J
    return H


def _system(case, batch, seed, device="cuda"):
    """H (B, n, n), site-dephasing rates (B, n) or None, collapse operators (list of (B, n, n))."""
    n, model = case["n"], case["model"]
    g = _gen(seed, device)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device=device, dtype=torch.float64)

    eps = 0.05 * normal(batch, n)
    if model in ("chain", "open"):
        H = _chain(eps)
    else:
        k = torch.arange(n, device=device, dtype=torch.float64)
        far = (k[:, None] - k[None, :]).abs()
        H = torch.diag_embed(eps) - 0.1 * torch.where(far > 0, far.clamp(min=1.0) ** -3, torch.zeros_like(far))
    rates, ops = None, []
    if model == "open":
        X = normal(batch, n, n) / math.sqrt(n)
        H = H + 0.01 * (X + X.mT) / 2
        for _ in range(3):
            L = torch.complex(normal(batch, n, n), normal(batch, n, n))
            ops.append(L * (0.1 / (2 * math.sqrt(2 * n))))
    else:
        u = torch.rand(batch, 1, generator=g, device=device, dtype=torch.float64)
        rates = (0.005 + 0.015 * u).expand(batch, n).contiguous()
        if model == "relax":
            for k in range(n - 1):
                L = torch.zeros(batch, n, n, dtype=CDT, device=device)
                L[:, k, k + 1] = 0.1
                ops.append(L)
    return H.to(CDT), rates, ops


def _mixed_states(batch, n, seed, device="cuda"):
    """(B, n, n) random density matrices of rank one."""
    g = _gen(seed + 77, device)
    psi = torch.complex(torch.randn(batch, n, generator=g, device=device, dtype=torch.float64),
                        torch.randn(batch, n, generator=g, device=device, dtype=torch.float64))
    psi = psi / psi.norm(dim=1, keepdim=True)
    r = psi[:, :, None] * psi[:, None, :].conj()
    return (r + r.mH) / 2                            # Hermitian bit for bit


def _uneven_sizes(case):
    sizes = [s for s in (8, 16, 32, 64, 128, 256) if s <= case["largest"]]
    sizes = [s - case["odd"] for s in sizes]
    return [sizes[i % len(sizes)] for i in range(case["chains"])]


def _uneven(case, seed):
    """Per-size stacked (H, ops, rho0), in increasing size."""
    out = {}
    for n in sorted(set(_uneven_sizes(case))):
        c = dict(n=n, model="open")
        b = _uneven_sizes(case).count(n)
        H, _, ops = _system(c, b, seed * 1000 + n)
        out[n] = (H, ops, _mixed_states(b, n, seed * 1000 + n))
    return out


def _projector(n, k, device="cuda"):
    E = torch.zeros(n, n, dtype=CDT, device=device)
    E[k, k] = 1
    return E


def _absorption(case, seed):
    n, B = case["n"], case["batch"]
    g = _gen(seed)
    eps = 0.05 * torch.randn(B, n, generator=g, device="cuda", dtype=torch.float64)
    bond = torch.full((B, n - 1), -0.1, dtype=torch.float64, device="cuda")
    gamma = torch.full((B, n), 0.01, dtype=torch.float64, device="cuda")
    d = 1 + 0.1 * torch.randn(B, n, generator=g, device="cuda", dtype=torch.float64)
    mu = torch.zeros(B, n + 1, n + 1, dtype=CDT, device="cuda")
    mu[:, 0, 1:] = d.to(CDT)
    mu[:, 1:, 0] = d.to(CDT)
    rho0 = torch.zeros_like(mu)
    rho0[:, 1:, 0] = d.to(CDT)                      # mu |g><g|
    w = torch.complex(torch.randn(B, case["steps"], 1, generator=g, device="cuda", dtype=torch.float64),
                      torch.randn(B, case["steps"], 1, generator=g, device="cuda", dtype=torch.float64))
    return eps, bond, gamma, mu, rho0, w


def _ohmic(w, lam=0.05, omega_c=0.1, kT=0.025):
    """S(w) of an Ohmic bath with exponential cutoff (detailed balance)."""
    w = np.asarray(w, dtype=np.float64)
    eta = np.pi * lam / omega_c
    small = np.abs(w) < 1e-12
    ws = np.where(small, 1.0, w)
    val = 2 * eta * ws * np.exp(-np.abs(ws) / omega_c) / (-np.expm1(-ws / kT))
    return np.where(small, 2 * eta * kT, val)


def _redfield_system(n, seed):
    """H, its eigenbasis and Lambda_k = V (S(-w) o (V^dag |k><k| V)) V^dag in the site basis, on the host."""
    rng = np.random.default_rng(seed)
    H = np.diag(rng.normal(0.0, 0.05, size=n)).astype(np.complex128)
    k = np.arange(n - 1)
    H[k, k + 1] = H[k + 1, k] = -0.1
    E, V = np.linalg.eigh(H)
    C = _ohmic(-(E[:, None] - E[None, :]))
    A = V.conj()[:, :, None] * V[:, None, :]         # A[k] = V^dag |k><k| V
    return H, E, V, C, A


def _correlations(case, seed):
    g = _gen(seed)
    B, n = case["batch"], case["n"]
    t = DT * torch.arange(1, n + 1, device="cuda", dtype=torch.float64)
    out = torch.zeros(B, n, dtype=CDT, device="cuda")
    for _ in range(6):
        w = 0.2 * torch.randn(B, 1, generator=g, device="cuda", dtype=torch.float64)
        a = torch.rand(B, 1, generator=g, device="cuda", dtype=torch.float64)
        out += a * torch.exp(torch.complex((-0.01 - 0.02 * a) * t, -w * t))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "evolve":
        H, rates, ops = (x[0].numpy() if isinstance(x, torch.Tensor) else x
                         for x in _system(case, 1, seed, "cpu"))
        n = case["n"]
        c_ops = [L[0].numpy() for L in ops]
        for k in range(n):
            L = np.zeros((n, n), dtype=np.complex128)
            L[k, k] = np.sqrt(rates[k])
            c_ops.append(L)
        e_ops = [_projector(n, k, "cpu").numpy() for k in range(n)]
        return dict(case=case, H=H, c_ops=c_ops, e_ops=e_ops, rho0=_mixed_states(1, n, seed, "cpu")[0].numpy())
    if kind == "host":
        H, rates, _ = _system(case, case["batch"], seed)
        rho0 = _mixed_states(case["batch"], case["n"], seed)
        return dict(case=case, **{k: torch.empty(v.shape, dtype=v.dtype, pin_memory=True).copy_(v)
                                  for k, v in dict(H=H, rates=rates, rho0=rho0).items()})
    if kind == "ensemble":
        H, rates, ops = _system(case, case["batch"], seed)
        c_ops = ops if rates is None else ops + [engine.SiteDephasing(rates)]
        return dict(case=case, gen=engine.LindbladGenerator.build(H, c_ops),
                    rho0=_mixed_states(case["batch"], case["n"], seed), e_ops=engine.Populations(case["n"]))
    if kind == "uneven":
        sizes, stacks = _uneven_sizes(case), _uneven(case, seed)
        seen, Hs, R0, Cs, Es = {}, [], [], [], []
        for n in sizes:
            b = seen.get(n, 0)
            seen[n] = b + 1
            H, ops, rho = stacks[n]
            Hs.append(H[b])
            Cs.append([L[b] for L in ops])
            R0.append(rho[b])
            Es.append([_projector(n, 0), _projector(n, n - 1)])
        return dict(case=case, groups=engine.ragged_groups(Hs, R0, Cs, Es, "split", torch.device("cuda")))
    if kind == "gradient":
        eps, bond, gamma, mu, rho0, w = _absorption(case, seed)
        N = case["n"] + 1
        for x in (eps, bond, gamma):
            x.requires_grad_(True)
        return dict(case=case, eps=eps, bond=bond, gamma=gamma, mu=mu, rho0=rho0, w=w,
                    H0=torch.zeros(N, N, dtype=CDT, device="cuda"))
    if kind == "redfield":
        n = case["n"]
        H = _redfield_system(n, seed)[0]
        pops = [_projector(n, k, "cpu").numpy() for k in range(n)]
        rs = redfield.Redfield_solver(H, c_ops=pops, spectra=[_ohmic] * n)
        rs.redfield_tensor()
        return dict(case=case, solver=rs, rho0=_mixed_states(1, n, seed, "cpu")[0].numpy(), e_ops=pops)
    if kind == "block":
        n = case["n"]
        _, E, V, C, A = _redfield_system(n, seed)
        dev = dict(dtype=CDT, device="cuda")
        A, C, E, V = (torch.as_tensor(x, **dev) for x in (A, C, E, V))
        Lam = C * A
        P = (A @ Lam).sum(0)
        D = n * n
        U = torch.cat([A.reshape(n, D), Lam.reshape(n, D)]).T                       # [(a, c), k]
        W = torch.cat([Lam.conj().mT.reshape(n, D), A.reshape(n, D)])               # [k, (d, b)]
        R = (U @ W).reshape(n, n, n, n).permute(0, 3, 1, 2).contiguous()             # [a, b, c, d]
        i = torch.arange(n, device="cuda")
        R[:, i, :, i] -= P                                                           # - d_bd P[a, c]
        R[i, :, i, :] -= P.conj()                                                    # - d_ac conj(P[b, d])
        R[i[:, None], i[None, :], i[:, None], i[None, :]] -= 1j * (E[:, None] - E[None, :])
        rho0 = V.mH @ _mixed_states(case["rhs"], n, seed) @ V
        e_ops = [V.mH[:, k, None] * V[None, k, :] for k in range(n)]
        return dict(case=case, R=(R.reshape(D, D), n), rho0=rho0, e_ops=e_ops)
    if kind == "spectrum":
        return dict(case=case, cor=_correlations(case, seed))
    raise ValueError(kind)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "evolve":
        res = Lindblad_solver(s["H"], c_ops=s["c_ops"], precision=case["precision"]).evolve(
            s["rho0"], dt=DT, Nt=case["steps"], e_ops=s["e_ops"], store_states=case["states"])
        return dict(observables=res.observables, states=np.stack(res.rholist))
    if kind == "host":
        res = Lindblad_solver(s["H"], c_ops=[engine.SiteDephasing(s["rates"])], precision=case["precision"]).evolve(
            s["rho0"], dt=DT, Nt=case["steps"], e_ops=engine.Populations(case["n"]), store_states=False)
        return dict(observables=res.observables, states=res.rholist)
    if kind == "ensemble":
        obs, _, rho = engine.propagate(s["gen"], s["rho0"], DT, case["steps"], s["e_ops"],
                                       precision=case["precision"])
        return dict(observables=obs, states=rho)
    if kind == "uneven":
        fins = engine.ragged_enqueue(s["groups"], DT, case["steps"], "split", engine.UNEVEN_DEFAULT)
        out = [fin(True) for fin in fins]
        return dict(observables=[o for o, _, _ in out], states=[r for _, _, r in out])
    if kind == "gradient":
        obs = chain_observables(s["H0"], s["eps"], s["bond"], s["gamma"], s["rho0"], [s["mu"]], DT, case["steps"],
                                site0=1, checkpoint=case["checkpoint"], precision=case["precision"])
        grads = torch.autograd.grad(obs, [s["eps"], s["bond"], s["gamma"]], grad_outputs=s["w"])
        return dict(observables=obs, grads=list(grads))
    if kind == "redfield":
        res = s["solver"].evolve(s["rho0"], DT, case["steps"], e_ops=s["e_ops"])
        return dict(observables=res.observables, states=np.stack(res.rholist))
    if kind == "block":
        obs, _, rho = redfield.propagate_vec_split(s["R"], s["rho0"], DT, case["steps"], s["e_ops"])
        return dict(observables=obs, states=rho)
    if kind == "spectrum":
        g, freq = spectra.correlation_spectrum(s["cor"], DT)
        return dict(spectrum=g, freq=freq)
    raise ValueError(kind)


# ------------------------------------------------------------------ work
def _rhs_flops(n, model):
    """One evaluation of a Lindblad right-hand side of dimension n: Hermitian, so X = Heff rho once."""
    couplings = 2 * (n - 1) if model == "chain" else n * (n - 1)
    flops = 4 * couplings * n + 8 * n * n            # real couplings, complex diagonal
    if model == "relax":
        flops += 8 * (n - 1)
    if model == "open":
        flops += 3 * (8 + 4) * n ** 3                # L rho, then the Hermitian half of (L rho) L^dag
    return flops


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    if kind in ("evolve", "host", "ensemble"):
        B = case.get("batch", 1)
        steps = case["steps"]
        ops = 3 * n * n if case["model"] == "open" else n
        out = steps * n + n * n * (steps if case.get("states") else 1)
        return dict(bytes=16 * B * (2 * n * n + ops + out),
                    flops=4 * steps * B * (_rhs_flops(n, case["model"]) + 6 * n * n))
    if kind == "uneven":
        sizes = _uneven_sizes(case)
        return dict(bytes=16 * sum(6 * m * m + 2 * case["steps"] for m in sizes),
                    flops=4 * case["steps"] * sum(_rhs_flops(m, "open") for m in sizes))
    if kind == "gradient":
        # two Hermitian chains per sample; forward, adjoint (with its recomputed stages) and gradient sums
        N = n + 1
        return dict(bytes=16 * case["batch"] * (3 * N * N + 2 * case["steps"]),
                    flops=2 * 4 * case["steps"] * case["batch"] * (3 * _rhs_flops(N, "chain") + 24 * N * N))
    if kind in ("redfield", "block"):
        D, R = n * n, case.get("rhs", 1)
        return dict(bytes=16 * (D * D + 2 * D * R + case["steps"] * R * n),
                    flops=4 * case["steps"] * 8 * D * D * R)
    B = case["batch"]
    return dict(bytes=32 * B * n, flops=5 * B * n * math.log2(n))


# ------------------------------------------------------------------ 64-bit results
def _rk4(f, rho, steps, each):
    for _ in range(steps):
        k1 = f(rho)
        k2 = f(rho + DT / 2 * k1)
        k3 = f(rho + DT / 2 * k2)
        k4 = f(rho + DT * k3)
        rho = rho + DT / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
        each(rho)
    return rho


def _lindblad(H, rates, ops):
    S = sum((L.mH @ L for L in ops), torch.zeros_like(H))
    if rates is not None:
        S = S + torch.diag_embed(rates).to(CDT)
    heff = H - 0.5j * S

    def f(rho):
        X = heff @ rho
        Y = rho @ heff.mH
        out = -1j * (X - Y)
        if rates is not None:
            out = out + torch.diag_embed(rates * torch.diagonal(rho, dim1=-2, dim2=-1))
        for L in ops:
            out = out + L @ rho @ L.mH
        return out
    return f


def exact(case, seed):
    kind = case["kind"]
    if kind in ("evolve", "host", "ensemble"):
        dev = "cpu" if kind == "evolve" else "cuda"
        B = case.get("batch", 1)
        H, rates, ops = _system(case, B, seed, dev)
        rho = _mixed_states(B, case["n"], seed, dev)
        H, rho, ops = H.cuda(), rho.cuda(), [L.cuda() for L in ops]
        f = _lindblad(H, None if rates is None else rates.cuda(), ops)
        pops, states = [], []

        def each(r):
            pops.append(torch.diagonal(r, dim1=-2, dim2=-1))
            if case.get("states"):
                states.append(r)
        rho = _rk4(f, rho, case["steps"], each)
        obs = torch.stack(pops, 1)
        if kind == "evolve":
            return dict(observables=obs[0].cpu().numpy(),
                        states=torch.stack([s[0] for s in states]).cpu().numpy() if states else rho.cpu().numpy())
        if kind == "host":
            return dict(observables=obs.cpu().numpy(), states=rho.cpu().numpy())
        return dict(observables=obs, states=rho)
    if kind == "uneven":
        observables, states = [], []
        for n, (H, ops, rho) in _uneven(case, seed).items():
            # chains of dimension <= 32 come back 64 // n to an instance, block-diagonal
            p = 64 // n if 2 * n <= 64 else 1
            B = H.shape[0]
            G = -(-B // p)
            ends = []
            rho = _rk4(_lindblad(H, None, ops), rho, case["steps"],
                       lambda r: ends.append(torch.stack([r[:, 0, 0], r[:, n - 1, n - 1]], -1)))
            obs = torch.zeros(G * p, case["steps"], 2, dtype=CDT, device="cuda")
            obs[:B] = torch.stack(ends, 1)
            full = torch.zeros(G * p, n, n, dtype=CDT, device="cuda")
            full[:B] = rho
            packed = torch.zeros(G, p * n, p * n, dtype=CDT, device="cuda")
            for q in range(p):
                packed[:, q * n:(q + 1) * n, q * n:(q + 1) * n] = full.reshape(G, p, n, n)[:, q]
            observables.append(obs.reshape(G, p, case["steps"], 2).permute(0, 2, 1, 3).reshape(G, case["steps"], 2 * p))
            states.append(packed)
        return dict(observables=observables, states=states)
    if kind == "gradient":
        eps, bond, gamma, mu, rho0, w = _absorption(case, seed)
        params = [x.requires_grad_(True) for x in (eps, bond, gamma)]
        N, B = case["n"] + 1, case["batch"]
        k = torch.arange(case["n"], device="cuda") + 1
        H = torch.zeros(B, N, N, dtype=CDT, device="cuda")
        H = H.index_put((torch.arange(B, device="cuda")[:, None], k, k), eps.to(CDT))
        off = torch.zeros(B, N, N, dtype=CDT, device="cuda")
        off = off.index_put((torch.arange(B, device="cuda")[:, None], k[:-1], k[1:]), bond.to(CDT))
        rates = torch.cat([torch.zeros(B, 1, dtype=torch.float64, device="cuda"), gamma], 1)
        out = []
        _rk4(_lindblad(H + off + off.mT, rates, []), rho0, case["steps"],
             lambda r: out.append(torch.einsum("bij,bji->b", mu, r)))
        obs = torch.stack(out, 1)[:, :, None]
        grads = torch.autograd.grad(obs, params, grad_outputs=w)
        return dict(observables=obs.detach(), grads=[g.detach() for g in grads])
    if kind in ("redfield", "block"):
        n, R = case["n"], case.get("rhs", 1)
        _, E, V, C, A = _redfield_system(n, seed)
        E, V, C, A = (torch.as_tensor(x, dtype=CDT, device="cuda") for x in (E, V, C, A))
        Lam = V @ (C * A) @ V.mH                                                     # site basis
        H = V @ torch.diag(E) @ V.mH
        P = torch.diagonal(Lam, dim1=0, dim2=1).mT                                   # sum_k |k><k| Lam_k
        rho = _mixed_states(R, n, seed, "cpu" if kind == "redfield" else "cuda").cuda()

        def f(r):
            T = torch.einsum("bkj,klj->bkl", r, Lam.conj())                           # sum_k |k><k| rho Lam_k^dag
            X = (1j * H + P) @ r
            return T + T.mH - X - X.mH
        pops, states = [], []

        def each(r):
            pops.append(torch.diagonal(r, dim1=-2, dim2=-1))
            states.append(r)
            if kind == "block":
                states[:-1] = []
        _rk4(f, rho, case["steps"], each)
        obs = torch.stack(pops, 1)
        if kind == "redfield":
            return dict(observables=obs[0].cpu().numpy(), states=torch.stack([s[0] for s in states]).cpu().numpy())
        return dict(observables=obs, states=V.mH @ states[-1] @ V)
    x = _correlations(case, seed)
    n = case["n"]
    k = torch.arange(n, device="cuda", dtype=torch.float64)
    f = torch.where(k < (n + 1) // 2, k, k - n) / (n * DT)
    freq = 2 * math.pi * torch.roll(f, n // 2)
    g = torch.roll(torch.fft.fft(x, dim=-1), n // 2, dims=-1) * (DT * torch.exp(torch.complex(torch.zeros_like(freq), -freq * DT)))
    return dict(spectrum=g, freq=freq)
