"""Host operators sorted and uploaded on the host give the generators and
observables that device operators give; a host batch whose rho(0) is not
Hermitian leaves the pipeline for the two-part run."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ops(n, kind, rng):
    D = [np.diag(rng.normal(size=n) + 1j * rng.normal(size=n)) for _ in range(2)]
    S = [np.zeros((n, n), complex) for _ in range(2)]
    for k, s in enumerate(S):
        s[k % n, k % n] = 0.3 + k
    L = [rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n)) for _ in range(2)]
    return {'none': [], 'diag': D, 'single': S, 'dense': L, 'mixed': [D[0], L[0], S[1], L[1]],
            'batched': [np.stack([L[0]] * 3), D[0], np.stack(D + D[:1])]}[kind]


@pytest.mark.parametrize('n', [1, 2, 5])
@pytest.mark.parametrize('kind', ['none', 'diag', 'single', 'dense', 'mixed', 'batched'])
def test_generator_of_host_operators(n, kind):
    from lime_gb300 import engine
    rng = np.random.default_rng(n)
    H = rng.normal(size=(n, n))
    H = H + H.T
    ops = _ops(n, kind, rng)
    a = engine.LindbladGenerator.build(H, ops)
    b = engine.LindbladGenerator.build(H, [torch.as_tensor(o, device='cuda') for o in ops])
    assert a.k_dense == b.k_dense and a.P == b.P and (a.m is None) == (b.m is None)
    assert torch.equal(a.heff, b.heff)
    if a.m is not None:
        assert torch.equal(a.m, b.m)
        assert engine.m_is_diagonal(a) == engine.is_diagonal(b.m)
    if a.l_dense is not None:
        assert torch.equal(a.l_dense, b.l_dense)


@pytest.mark.parametrize('kind', ['none', 'diag', 'single', 'dense', 'mixed'])
def test_observables_of_host_operators(kind):
    from lime_gb300 import engine
    n = 4
    ops = _ops(n, kind, np.random.default_rng(3))
    a = engine.prepare_obs(ops, n, 2, 'cuda')
    b = engine.prepare_obs([torch.as_tensor(o, device='cuda') for o in ops], n, 2, 'cuda')
    assert a[1:] == b[1:] and (a[0] is None) == (b[0] is None)
    if a[0] is not None:
        assert torch.equal(a[0], b[0])


def test_pipeline_returns_a_batch_that_is_not_hermitian():
    from lime_gb300 import engine
    P, n = 912, 24
    rng = np.random.default_rng(0)
    H = np.zeros((P, n, n), complex)
    H[:, range(n), range(n)] = rng.normal(size=(P, n))
    rho = np.zeros((P, n, n), complex)
    rho[:, 0, 0] = 1
    rates = np.full((P, n), 0.01)
    args = (H, rho, [engine.SiteDephasing(rates)], engine.Populations(n), 0.05, 2)
    assert engine.propagate_host_pipelined(*args) is not None
    rho[P - 1, 0, 1] = 0.5
    assert engine.propagate_host_pipelined(*args) is None
