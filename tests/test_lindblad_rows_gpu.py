"""The FP64 propagator's generator forms and layouts against an eager
complex128 RK4 in PyTorch: full and sparse rows, real and complex, listed and
dense collapse operators, drives, at the edges of the items-a-thread,
cluster and shared-memory rules.

Tolerance: both sides round every operation to 2^-53; a few hundred
operations an element and stage bound the relative difference of states and
observables by 1e-12 over the steps taken here."""
import numpy as np
import pytest
import torch

from lime_gb300 import engine

pytestmark = pytest.mark.gpu
TOL = 1e-12
CDT = torch.complex128


@pytest.fixture(scope='module', autouse=True)
def _lib():
    from lime_gb300 import build, _native
    build.build()
    _native.require_device()


def _model(name, n, B, rng):
    """H (B, n, n), c_ops and (optional) SiteDephasing rates."""
    def cplx(*s):
        return rng.normal(size=s) + 1j * rng.normal(size=s)
    H = np.zeros((B, n, n), dtype=complex)
    i = np.arange(n)
    H[:, i, i] = rng.normal(0, 0.2, size=(B, n))
    k = np.arange(n - 1)
    hop = rng.normal(-0.1, 0.02, size=(B, n - 1)) + 0j
    if name == 'complex_chain':
        hop = hop * np.exp(1j * rng.uniform(0, 2, size=(B, n - 1)))
    H[:, k, k + 1] = hop
    H[:, k + 1, k] = hop.conj()
    if name == 'star' and n > 2:
        H[:, 0, 1:] = 0.05
        H[:, 1:, 0] = 0.05
    if name in ('dense_real', 'mixed', 'dense_ops'):
        X = rng.normal(0, 0.02, size=(B, n, n))
        H = H + X + X.transpose(0, 2, 1)
    if name == 'dense_complex':
        X = 0.02 * cplx(B, n, n)
        H = H + X + X.conj().transpose(0, 2, 1)
    ops = []
    if name in ('lowering', 'mixed') and n > 1:
        for q in range(min(n - 1, 40)):
            L = np.zeros((n, n), dtype=complex)
            L[q, q + 1] = 0.1 + 0.02j
            ops.append(L)
        L = np.zeros((n, n), dtype=complex)      # two entries in one row, off the diagonal and on it
        L[0, n - 1], L[0, 0] = 0.1j, 0.05
        ops.append(L)
    if name in ('mixed', 'dense_ops'):
        ops += [np.asarray(0.1 / np.sqrt(n) * cplx(B, n, n)) for _ in range(5 if n < 20 else 3)]
    rates = rng.uniform(0.01, 0.03, size=(B, n))
    return H, ops, rates


def _reference(H, ops, rates, rho, steps, drive=None, dt=0.05):
    H, rho = torch.as_tensor(H, device='cuda'), rho.clone()
    ops = [torch.as_tensor(L, device='cuda', dtype=CDT) for L in ops]
    g = torch.as_tensor(rates, device='cuda')
    out = []
    S = sum((L.mH @ L for L in ops), torch.zeros_like(H)) + torch.diag_embed(g).to(CDT)

    def f(r, Ht):
        heff = Ht - 0.5j * S
        y = -1j * (heff @ r - r @ heff.mH) + torch.diag_embed(g * torch.diagonal(r, dim1=-2, dim2=-1))
        for L in ops:
            y = y + L @ r @ L.mH
        return y
    for s in range(steps):
        Ht = H if drive is None else H - sum(c * D for c, D in zip(drive[1][s], drive[0]))
        k1 = f(rho, Ht)
        k2 = f(rho + k1 * (dt / 2), Ht)
        k3 = f(rho + k2 * (dt / 2), Ht)
        k4 = f(rho + k3 * dt, Ht)
        rho = rho + (k1 + 2 * k2 + 2 * k3 + k4) * (dt / 6)
        out.append(rho)
    return torch.stack(out, 1)


def _states(B, n, rng):
    a = rng.normal(size=(B, n, n)) + 1j * rng.normal(size=(B, n, n))
    r = torch.as_tensor(a @ a.conj().transpose(0, 2, 1), device='cuda')
    r = r / torch.diagonal(r, dim1=-2, dim2=-1).sum(-1).real[:, None, None]
    return (r + r.mH) / 2


def _close(a, b):
    assert float((a - b).abs().max()) <= TOL * float(b.abs().max())


CASES = [(1, 1, 'chain'), (2, 3, 'dense_complex'), (3, 1, 'mixed'), (4, 700, 'chain'), (16, 1, 'chain'),
         (16, 40, 'mixed'), (22, 2, 'lowering'), (23, 2, 'dense_real'), (31, 80, 'complex_chain'),
         (32, 76, 'chain'), (32, 77, 'star'), (33, 1, 'lowering'), (37, 36, 'mixed'), (45, 37, 'dense_real'),
         (46, 15, 'complex_chain'), (64, 16, 'chain'), (64, 1, 'dense_ops'), (64, 80, 'mixed'),
         (64, 77, 'dense_complex'), (65, 1, 'chain'), (65, 80, 'lowering'), (91, 1, 'dense_real'),
         (100, 40, 'mixed'), (129, 2, 'chain'), (129, 80, 'complex_chain'), (181, 1, 'dense_complex'),
         (200, 2, 'lowering')]


@pytest.mark.parametrize('n,B,name', CASES)
def test_generator_forms(n, B, name):
    rng = np.random.default_rng(n * 1000 + B)
    H, ops, rates = _model(name, n, B, rng)
    rho = _states(B, n, rng)
    steps = 4
    ref = _reference(H, ops, rates, rho, steps)
    gen = engine.LindbladGenerator.build(H, ops + [engine.SiteDephasing(rates)])
    # narrow and wide diagonal observables, then dense ones
    wide = [np.diag(rng.normal(size=n) + 1j * rng.normal(size=n)), np.diag(np.arange(n) == n - 1) + 0j]
    dense = [rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)), wide[1]]
    for E, every in ((wide, 1), (dense, 2)):
        Et = torch.as_tensor(np.stack(E), device='cuda')
        want = torch.einsum('oji,btij->bto', Et, ref)[:, every - 1::every]
        obs, states, end = engine.propagate(gen, rho, 0.05, steps, E, states_every=2, obs_every=every)
        _close(obs, want)
        _close(states, ref[:, 1::2])
        _close(end, ref[:, -1])


@pytest.mark.parametrize('n,name', [(5, 'chain'), (40, 'dense_real'), (70, 'complex_chain'), (64, 'lowering')])
def test_driven_forms(n, name):
    rng = np.random.default_rng(n)
    H, ops, rates = _model(name, n, 1, rng)
    rho = _states(1, n, rng)
    steps = 5
    D = np.zeros((2, n, n), dtype=complex)
    D[0, 0, n - 1] = D[0, n - 1, 0] = 0.3
    D[1, 1, 2], D[1, 2, 1] = 0.2j, -0.2j
    coef = rng.normal(size=(steps, 2))
    Dt, ct = torch.as_tensor(D, device='cuda'), torch.as_tensor(coef, device='cuda')
    ref = _reference(H, ops, rates, rho, steps, (Dt, ct))
    gen = engine.LindbladGenerator.build(H, ops + [engine.SiteDephasing(rates)])
    _, states, end = engine.propagate(gen, rho, 0.05, steps, None, states_every=1, drive=(Dt, ct))
    _close(states, ref)
    _close(end, ref[:, -1])


def test_continues_over_launches():
    """n = 110: launches of 25 steps."""
    rng = np.random.default_rng(4)
    H, ops, rates = _model('dense_real', 110, 1, rng)
    rho = _states(1, 110, rng)
    ref = _reference(H, ops, rates, rho, 30)
    gen = engine.LindbladGenerator.build(H, [engine.SiteDephasing(rates)])
    _, _, end = engine.propagate(gen, rho, 0.05, 30, None)
    _close(end, ref[:, -1])


@pytest.mark.parametrize('n,B,dense', [(64, 153, 0), (64, 228, 0), (37, 48, 2), (20, 170, 3), (24, 304, 0), (16, 151, 1)])
def test_batches_in_several_launches(n, B, dense):
    """A batch split over launches of different cluster sizes: every instance
    as it comes out alone, observables and states included."""
    from lime_gb300 import engine
    g = torch.Generator(device='cuda').manual_seed(n + B)

    def c(*s):
        return torch.complex(torch.randn(*s, generator=g, device='cuda', dtype=torch.float64),
                             torch.randn(*s, generator=g, device='cuda', dtype=torch.float64))
    H = c(B, n, n) / n
    H = H + H.mH
    ops = [0.2 * c(B, n, n) / n for _ in range(dense)]
    rho = c(B, n, n)
    rho = rho @ rho.mH
    rho = rho / torch.diagonal(rho, dim1=1, dim2=2).sum(1).real[:, None, None]
    rho = (rho + rho.mH) / 2
    args = dict(dt=0.05, n_steps=5, e_ops=engine.Populations(min(n, 7)), states_every=2)
    o, s, r = engine.propagate(engine.LindbladGenerator.build(H, ops), rho, **args)
    for b in (0, 1, B // 2, 151 % B, 152 % B, B - 2, B - 1):
        o1, s1, r1 = engine.propagate(engine.LindbladGenerator.build(H[b], [x[b] for x in ops]), rho[b], **args)
        # the same products in the same order, whatever the cluster
        assert (o[b] - o1[0]).abs().max().item() < 1e-14 and (s[b] - s1[0]).abs().max().item() < 1e-14
        assert (r[b] - r1[0]).abs().max().item() < 1e-14
