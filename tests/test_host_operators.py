"""Host operators reach the generator through NumPy; every CPU tensor and
array that torch converts for the device is taken, and nothing else."""
import numpy as np
import pytest
import torch

from lime_gb300 import engine


def _tensors():
    g = torch.Generator().manual_seed(3)
    U = torch.randn(4, 4, dtype=torch.complex128, generator=g)
    R = torch.randn(4, 4, generator=g)
    return {'conj': U.conj(), 'neg': U.conj().imag, 'neg_complex': torch._neg_view(U), 'mH': U.mH,
            'bfloat16': R.to(torch.bfloat16), 'half': R.half(), 'complex32': U.to(torch.complex32),
            'int': torch.eye(4, dtype=torch.int32), 'bool': torch.eye(4, dtype=torch.bool),
            'grad': R.clone().requires_grad_(True), 'strided': torch.randn(8, 8, generator=g)[::2, ::2]}


@pytest.mark.filterwarnings('ignore:ComplexHalf')
@pytest.mark.parametrize('name', ['conj', 'neg', 'neg_complex', 'mH', 'bfloat16', 'half', 'complex32', 'int', 'bool',
                                  'grad', 'strided'])
def test_tensor(name):
    x = _tensors()[name]
    got = engine._host_or_device(x, 'cuda')
    want = x.detach().to(torch.complex128)
    assert got.dtype == np.complex128 and got.shape == (4, 4)
    assert torch.equal(torch.as_tensor(got.copy()), torch.complex(want.real + 0, want.imag + 0))


@pytest.mark.parametrize('order', ['C', 'F'])
@pytest.mark.parametrize('dtype', [np.complex128, np.complex64, np.float64, np.int64, bool])
def test_array(dtype, order):
    x = np.asarray(np.arange(16).reshape(4, 4) % 3, dtype=dtype, order=order)
    assert np.array_equal(engine._host_or_device(x, 'cuda'), x.astype(np.complex128))


def test_sparse_matrix():
    sparse = pytest.importorskip('scipy.sparse')
    x = sparse.csr_matrix(np.diag([1.0, 2j, 0.0]))
    assert np.array_equal(engine._host_or_device(x, 'cuda'), x.toarray())


@pytest.mark.parametrize('x', [np.array([['1', '2'], ['3', '4']]), np.array([[object()]], dtype=object),
                               np.eye(3)[::-1], torch.eye(3).to_sparse()])
def test_refused_as_by_torch(x):
    with pytest.raises(Exception):
        engine.as_device(x, 'cpu')
    with pytest.raises(Exception):
        engine._host_or_device(x, 'cuda')
