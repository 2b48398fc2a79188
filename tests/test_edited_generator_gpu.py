"""A generator whose M is written to after it was built (one-entry collapse
operators give a diagonal M, the edit makes it dense): the tensor-core paths
take the M that is there."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('before', [False, True])       # a call before the edit
@pytest.mark.parametrize('n,replace', [(72, False), (72, True), (12, False), (12, True)])
def test_edited_m(n, replace, before):
    from lime_gb300 import engine
    rng = np.random.default_rng(n)
    H = np.diag(rng.normal(size=n)).astype(complex)
    H += np.diag(np.full(n - 1, -0.1), 1) + np.diag(np.full(n - 1, -0.1), -1)
    ops = []
    for k in range(n):
        L = np.zeros((n, n), complex)
        L[k, k] = 0.1
        ops.append(L)
    gen = engine.LindbladGenerator.build(H, ops)
    if n > 64 and before:
        engine.propagate(gen, np.eye(n) / n, 0.05, 2, [], precision='split')
    elif before:                                         # n <= 64 decides at its first call
        assert engine.m_is_diagonal(gen)
    l = rng.normal(size=n) * 0.05
    extra = torch.as_tensor(np.outer(l, l), device='cuda')
    if replace:
        gen.m = gen.m + extra
    else:
        gen.m += extra
    gen.heff -= 0.5j * torch.diag(torch.diagonal(extra))
    psi = rng.normal(size=n) + 1j * rng.normal(size=n)
    rho = np.outer(psi, psi.conj()) / np.vdot(psi, psi).real
    rho = (rho + rho.conj().T) / 2
    _, _, a = engine.propagate(gen, rho, 0.05, 20, [], precision='split')
    _, _, b = engine.propagate(gen, rho, 0.05, 20, [])
    assert (a - b).abs().max().item() < 1e-6 * b.abs().max().item()
