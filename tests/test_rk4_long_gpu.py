"""Rounding of the FP64 propagators over many steps.  A diagonal generator
leaves every element an oscillator of its own, whose RK4 result after N steps
is R(z)^N, R(z) = 1 + z + z^2/2 + z^3/6 + z^4/24, z = -i w dt, here in
extended precision.

Tolerance: a step rounds an element a few times, each by at most 2^-53 of it;
independent roundings add up to an rms of sqrt(N) 2^-53 at most.  A rounded
common factor (dt / 6) stretches every increment the same way instead and
leaves up to w dt N 2^-53."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
STEPS = 4000
LIM = np.sqrt(STEPS) * 2.0 ** -53


def _growth(w, dt):
    """R(-i w dt)^STEPS by repeated squaring."""
    x = -np.longdouble(w) * np.longdouble(dt)
    z = x.astype(np.clongdouble) * np.clongdouble(1j)
    r = 1 + z * (1 + z / 2 * (1 + z / 3 * (1 + z / 4)))
    out, k = np.ones_like(r), STEPS
    while k:
        if k & 1:
            out = out * r
        r, k = r * r, k >> 1
    return out


def _rms(got, start, growth):
    err = np.abs(got.astype(np.clongdouble) - start.astype(np.clongdouble) * growth) / np.abs(start)
    return float(np.sqrt(np.mean(err.astype(np.float64) ** 2)))


@pytest.mark.parametrize('dt', [0.05, 0.07, 0.1])
@pytest.mark.parametrize('n,B', [(8, 4), (24, 1), (66, 1)])
def test_lindblad(n, B, dt):
    from lime_gb300 import engine
    rng = np.random.default_rng(n)
    e = rng.integers(0, 2 ** 20, size=(B, n)) / 2.0 ** 19        # differences are exact
    X = rng.normal(size=(B, n, n)) + 1j * rng.normal(size=(B, n, n))
    rho = X + X.conj().swapaxes(-1, -2)
    H = np.zeros((B, n, n), complex)
    H[:, range(n), range(n)] = e
    gen = engine.LindbladGenerator.build(H, [])
    _, _, got = engine.propagate(gen, rho, dt, STEPS, [])
    w = e[:, :, None] - e[:, None, :]
    off = np.broadcast_to(~np.eye(n, dtype=bool), w.shape)
    assert _rms(got.cpu().numpy()[off], rho[off], _growth(w, dt)[off]) < LIM


@pytest.mark.parametrize('dt', [0.05, 0.07, 0.1])
@pytest.mark.parametrize('n', [3, 6, 14])       # one CTA, a cluster, the whole grid
def test_redfield(n, dt):
    from lime_gb300.redfield import propagate_vec
    rng = np.random.default_rng(n)
    D = n * n
    w = rng.integers(-2 ** 20, 2 ** 20, size=D) / 2.0 ** 19
    L = torch.diag(torch.as_tensor(-1j * w, device='cuda'))
    rho = rng.normal(size=(1, n, n)) + 1j * rng.normal(size=(1, n, n))
    _, _, got = propagate_vec((L, n), torch.as_tensor(rho, device='cuda'), dt, STEPS)
    assert _rms(got.cpu().numpy().reshape(D), rho.reshape(D), _growth(w, dt)) < LIM
