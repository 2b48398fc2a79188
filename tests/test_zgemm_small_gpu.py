"""lime_zgemm_strided_f64 on both sides of the element / tile rule: sizes
that waste a tile, few tiles and many, strides, conjugation and scale."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('Z,M,N,K', [(1, 1, 1, 1), (1, 20, 20, 20), (100, 20, 20, 20), (3, 33, 65, 17), (75, 64, 64, 5),
                                     (76, 64, 64, 5), (80, 46, 46, 9), (80, 45, 45, 9), (1, 640, 576, 40),
                                     (70000, 2, 1, 3)])
@pytest.mark.parametrize('variant', ['plain', 'strided'])
def test_against_torch(Z, M, N, K, variant):
    from lime_gb300 import zlinalg as zl
    g = torch.Generator(device='cuda').manual_seed(Z + M)

    def c(*s):
        return torch.complex(torch.randn(*s, generator=g, device='cuda', dtype=torch.float64),
                             torch.randn(*s, generator=g, device='cuda', dtype=torch.float64))
    if variant == 'plain':
        A, B = c(Z, M, K), c(Z, K, N)
        got, ref = zl.bmm(A, B), A @ B
    else:
        A, B, s = c(Z, K, M).transpose(1, 2), c(1, N, K).transpose(1, 2), c(Z, K)
        out = torch.empty((Z, N, M), dtype=torch.complex128, device='cuda').transpose(1, 2)
        zl.bmm(A, B, conj_a=True, conj_b=True, scale=s, out=out)
        got, ref = out, (A.conj() * s[:, None, :]) @ B.conj()
    # K products of unit normals, each with a few roundings of 2^-53
    assert (got - ref).abs().max().item() <= 2.2e-16 * 16 * K * max(1.0, ref.abs().max().item())
