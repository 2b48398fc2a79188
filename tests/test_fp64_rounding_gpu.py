"""Rounding error of the FP64 propagator and of its gradient where a step is
large, beside the one of the same formulas in complex128 NumPy (products as
matrix products, gradient sums by rows at each stage), both against extended
precision.

Tolerance: the rms of thousands of independent roundings each, known to a few
per cent; one sum of all terms of a right-hand side, or one sum of all stages'
products an element, is 1.3 to 1.9 times off."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
LIM = 1.2


def _cplx(rng, *s):
    return rng.normal(size=s) + 1j * rng.normal(size=s)


def _model(kind, n, B, ops=3, strength=0.1):
    rng = np.random.default_rng(n)
    H = np.zeros((B, n, n), complex)
    H[:, range(n), range(n)] = 0.05 * rng.normal(size=(B, n))
    k = np.arange(n - 1)
    H[:, k, k + 1] = H[:, k + 1, k] = -0.1
    L = []
    if kind == 'full':
        X = 0.1 / np.sqrt(n) * _cplx(rng, B, n, n)
        H = H + X + X.conj().swapaxes(1, 2)
    else:
        L = [strength / (2 * np.sqrt(2 * n)) * _cplx(rng, B, n, n) for _ in range(ops)]
    psi = _cplx(rng, B, n)
    psi /= np.linalg.norm(psi, axis=1)[:, None]
    rho = psi[:, :, None] * psi[:, None, :].conj()
    return H, L, (rho + rho.conj().swapaxes(1, 2)) / 2


def _rk4(f, x, dt, steps):
    for _ in range(steps):
        k1 = f(x)
        k2 = f(x + dt / 2 * k1)
        k3 = f(x + dt / 2 * k2)
        k4 = f(x + dt * k3)
        x = x + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
    return x


def _rms(x, exact):
    return float(np.sqrt(np.mean(np.abs(x - exact) ** 2)))


@pytest.mark.parametrize('kind,n,B,dt,steps,more', [
    ('ops', 16, 16, 1.0, 10, {}), ('ops', 24, 4, 0.5, 2, dict(ops=6, strength=0.5)),
    ('ops', 12, 8, 0.4, 3, dict(ops=10, strength=0.5)), ('ops', 30, 3, 0.5, 2, dict(strength=1.0)),
    ('full', 12, 24, 0.5, 20, {}), ('full', 33, 6, 0.5, 16, {}), ('full', 70, 2, 0.5, 8, {})])
def test_states(kind, n, B, dt, steps, more):
    from lime_gb300 import engine
    H, ops, rho = _model(kind, n, B, **more)
    gen = engine.LindbladGenerator.build(H, ops)
    _, _, got = engine.propagate(gen, rho, dt, steps, [])
    heff = gen.heff.cpu().numpy()

    def run(c, r):
        h, L = heff.astype(c), [o.astype(c) for o in ops]

        def f(x):
            X = h @ x
            y = -1j * (X - X.conj().swapaxes(1, 2))
            return y + sum(o @ x @ o.conj().swapaxes(1, 2) for o in L) if L else y
        return _rk4(f, rho.astype(c), r(dt), steps)
    exact = run(np.clongdouble, np.longdouble)
    assert _rms(got.cpu().numpy(), exact) <= LIM * _rms(run(np.complex128, np.float64), exact)


def _gradient(n, B, steps, dt, par, rho, E, w, c, r):
    """The discrete adjoint by rows: gradients of Re sum conj(w) Tr(E rho)."""
    eps, bond, gam = par
    i, k = np.arange(n), np.arange(n - 1)
    H = np.zeros((B, n, n), c)
    H[:, i, i] = eps
    H[:, k, k + 1] = H[:, k + 1, k] = bond
    g = gam.astype(r)
    heff = H - r(0.5) * 1j * (g[:, :, None] * np.eye(n))
    hadj = -heff.conj().swapaxes(1, 2)

    def gen(h, x):
        X = h @ x
        y = -1j * (X - X.conj().swapaxes(1, 2))
        y[:, i, i] += g * x[:, i, i]
        return y
    d, f = r(dt), lambda x: gen(heff, x)
    states = [np.broadcast_to(rho, (B, n, n)).astype(c)]
    for _ in range(steps):
        states.append(_rk4(f, states[-1], d, 1))
    lam, E = np.zeros((B, n, n), c), E.astype(c)
    out = [np.zeros((B, n), r) for _ in range(3)]
    for s in range(steps - 1, -1, -1):
        ws = w[:, s].astype(c)[:, None, None]
        lam = lam + r(0.5) * (ws * E.conj().T + ws.conj() * E)
        y1 = states[s]
        y2 = y1 + d / 2 * f(y1)
        y3 = y1 + d / 2 * f(y2)
        y4 = y1 + d * f(y3)
        total = 0
        for y, a, cy, b in ((y4, d / 6, 0, None), (y3, d / 3, d, 1), (y2, d / 3, d / 2, 1), (y1, d / 6, d / 2, 1)):
            ab = a * lam if b is None else a * lam + cy * yb
            yb = gen(hadj, ab)
            total = total + yb
            im = ab.real * y.imag - ab.imag * y.real
            re = -(ab.real * y.real + ab.imag * y.imag)
            re[:, i, i] = 0
            bo = np.zeros((B, n, n), r)
            bo[:, :-1] = (ab[:, :-1].real * y[:, 1:].imag - ab[:, :-1].imag * y[:, 1:].real +
                          ab[:, 1:].real * y[:, :-1].imag - ab[:, 1:].imag * y[:, :-1].real)
            for o, v, m in zip(out, (im, bo, re), (2, 2, 1)):
                row = np.zeros((B, n), r)
                for q in range(n):
                    row += v[:, :, q]
                o += m * row
        lam = lam + total
    return out[0], out[1][:, :-1], out[2]


@pytest.mark.parametrize('n,B,steps', [(24, 12, 16), (16, 12, 30)])
def test_gradient(n, B, steps):
    from lime_gb300.adjoint import chain_observables
    rng = np.random.default_rng(n)
    par = [0.05 * rng.normal(size=(B, n)), -0.1 + 0.02 * rng.normal(size=(B, n - 1)), np.full((B, n), 0.01)]
    E, w = _cplx(rng, n, n), _cplx(rng, B, steps)
    psi = _cplx(rng, n)
    rho = np.outer(psi, psi.conj()) / np.vdot(psi, psi).real
    rho = (rho + rho.conj().T) / 2
    t = [torch.as_tensor(p, device='cuda').requires_grad_(True) for p in par]
    o = chain_observables(np.zeros((n, n)), *t, rho, [E], 0.05, steps, checkpoint=16)
    got = torch.autograd.grad(o, t, torch.as_tensor(w[:, :, None], device='cuda'))
    exact = _gradient(n, B, steps, 0.05, par, rho, E, w, np.clongdouble, np.longdouble)
    plain = _gradient(n, B, steps, 0.05, par, rho, E, w, np.complex128, np.float64)
    err = sum(_rms(a.cpu().numpy(), x) / _rms(p, x) for a, x, p in zip(got, exact, plain)) / 3
    assert err <= LIM
