"""Rounding error of the FP64 propagator where a step is large, beside the one
of the same formulas in complex128 NumPy (matrix products), both against
extended precision.

Tolerance: the rms of thousands of independent roundings each, known to a few
per cent; one sum of all terms of a right-hand side is 1.3 to 1.9 times off."""
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
