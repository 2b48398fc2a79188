"""A host batch that is not Hermitian leaves the pipeline before anything is
launched, when its shared rho(0) shows it, or before it is propagated, when its
first one does; another one is found by the kernels."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _launches(where):
    from lime_gb300 import _native as nat
    from lime_gb300 import engine
    P, n = 1000, 12
    rng = np.random.default_rng(0)
    H = np.zeros((P, n, n), complex)
    H[:, range(n), range(n)] = rng.normal(size=(P, n))
    rho = np.zeros((P, n, n), complex)
    rho[:, 0, 0] = 1
    bad = np.zeros((n, n), complex)
    bad[1, 0] = 1
    rho = {'none': rho, 'shared': bad, 'shared3': bad[None], 'tensor': torch.as_tensor(bad)}.get(where, rho)
    if where == 'all':
        rho[:] = bad
    elif where in ('first', 'last'):
        rho[0 if where == 'first' else -1] = bad
    ops = [engine.SiteDephasing(np.full((P, n), 0.01))]
    nat.require_device()
    before = nat.launch_count()
    got = engine.propagate_host_pipelined(H, rho, ops, engine.Populations(n), 0.05, 3)
    return got is None, nat.launch_count() - before


@pytest.mark.parametrize('where', ['shared', 'shared3', 'all', 'first', 'last', 'tensor'])
def test_known_before_the_run(where):
    none, full = _launches('none')
    assert not none and full > 0
    none, launches = _launches(where)
    assert none
    if where == 'last':
        assert launches == full
    elif where in ('all', 'first'):
        assert launches < full          # the generators alone
    else:
        assert launches == 0
