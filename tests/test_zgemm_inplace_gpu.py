"""A product written over one of its operands, or over a view of the same
storage: up to 64 x 64 the result is that of a separate output, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('conj', [False, True])
@pytest.mark.parametrize('where', ['A', 'B', 'At', 'scale'])
@pytest.mark.parametrize('n,Z', [(1, 3), (3, 500), (20, 100), (33, 40), (45, 300), (64, 10), (64, 200)])
def test_in_place(n, Z, where, conj):
    from lime_gb300 import zlinalg
    g = torch.Generator(device='cuda').manual_seed(n)
    A, B = (torch.randn(Z, n, n, generator=g, device='cuda', dtype=torch.complex128) for _ in range(2))
    scale = B[:, 0, :] if where == 'scale' else None
    X = A.transpose(1, 2) if where == 'At' else A
    want = zlinalg.bmm(X, B if where != 'scale' else A, conj_a=conj, scale=scale)
    for _ in range(3):
        a, b = A.clone(), B.clone()
        x = a.transpose(1, 2) if where == 'At' else a
        if where == 'scale':
            got = zlinalg.bmm(x, a, conj_a=conj, scale=b[:, 0, :], out=b)
        else:
            got = zlinalg.bmm(x, b, conj_a=conj, out=b if where == 'B' else a)
        assert torch.equal(got, want)
