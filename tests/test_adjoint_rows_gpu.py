"""The FP64 adjoint over the generators' nonzero entries against the tiled
GEMM kernel (which the same call takes with one zero dense operator): items
a thread from 1 to many, states in shared memory and in the workspace, sparse
and full generators, diagonal and dense observables."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
CDT = torch.complex128


def _segment(n, B, seg, step0, total, H, m, E, diag, ckpt, lam, g, obs_every, dense):
    from lime_gb300 import _native as nat
    lib = nat.require_device()
    d = nat.AdjointDesc()
    d.n, d.batch, d.param_batch, d.seg_steps = n, B, B, seg
    d.step0, d.total_steps, d.dt = step0, total, 0.05
    hadj = (-H.mH).contiguous()
    lam = lam.clone()
    gd, gb, gg = (torch.full((B, k), 0.5, dtype=torch.float64, device='cuda') for k in (n, max(n - 1, 1), n))
    d.ckpt, d.lam = ckpt.data_ptr(), lam.data_ptr()
    d.heff, d.heff_stride, d.heff_adj, d.heff_adj_stride = H.data_ptr(), n * n, hadj.data_ptr(), n * n
    if m is not None:
        mc = m.conj().resolve_conj().contiguous()
        d.m, d.m_stride, d.m_adj, d.m_adj_stride = m.data_ptr(), n * n, mc.data_ptr(), n * n
    zero = torch.zeros((1, n, n), dtype=CDT, device='cuda')
    if dense:
        d.k_dense, d.l_dense, d.l_dense_adj = 1, zero.data_ptr(), zero.data_ptr()
    d.n_obs, d.obs_diag, d.obs_every = E.shape[0], int(diag), obs_every
    d.obs_ops, d.obs_stride, d.obs_grad = E.data_ptr(), 0, g.data_ptr()
    d.grad_diag, d.grad_bond, d.grad_gamma = gd.data_ptr(), gb.data_ptr(), gg.data_ptr()
    wsb = lib.lime_lindblad_adjoint_f64_workspace(n, B, seg, int(dense))
    ws = torch.empty(wsb, dtype=torch.uint8, device='cuda')
    d.workspace, d.workspace_bytes = ws.data_ptr(), wsb
    nat.check(lib.lime_lindblad_adjoint_f64(d, torch.cuda.current_stream().cuda_stream), 'adjoint')
    torch.cuda.synchronize()
    return lam, gd, gb, gg


@pytest.mark.parametrize('n,B', [(1, 1), (2, 3), (5, 1), (16, 4), (22, 2), (23, 2), (32, 5), (33, 1), (40, 2), (41, 2),
                                 (45, 1), (46, 1), (64, 2), (70, 1)])
@pytest.mark.parametrize('full,with_m,diag', [(False, True, True), (True, False, False), (True, True, False)])
def test_against_the_gemm_kernel(n, B, full, with_m, diag):
    rng = np.random.default_rng(n + 7 * full)
    H = 0.1 * (rng.normal(size=(B, n, n)) + 1j * rng.normal(size=(B, n, n)))
    if not full:
        H = H.real * (np.abs(np.subtract.outer(np.arange(n), np.arange(n))) <= 1) + 0j
    H = H - 0.02j * np.eye(n)
    c = rng.normal(size=(B, n, n)) + 1j * rng.normal(size=(B, n, n))

    def herm(x):
        return torch.as_tensor((x + x.conj().swapaxes(1, 2)) / 2, device='cuda')
    ckpt, lam, m = herm(c), herm(rng.normal(size=(B, n, n)) + 0j), herm(0.05 * rng.normal(size=(B, n, n)) + 0j)
    E = rng.normal(size=(2, n) if diag else (2, n, n)) + 1j * rng.normal(size=(2, n) if diag else (2, n, n))
    E[0, 0] = 0
    seg, step0, total, every = 4, 3, 8, 2
    g = torch.as_tensor(rng.normal(size=(B, total // every, 2)) + 1j * rng.normal(size=(B, total // every, 2)),
                        device='cuda')
    args = (n, B, seg, step0, total, torch.as_tensor(H, device='cuda'), m if with_m else None,
            torch.as_tensor(E, device='cuda'), diag, ckpt, lam, g, every)
    for got, ref in zip(_segment(*args, dense=False), _segment(*args, dense=True)):
        # 16 generator applications of ~n terms and n-term sums in 64 bits
        assert (got - ref).abs().max().item() <= 2.2e-16 * 200 * (n + 8) * max(1.0, ref.abs().max().item())
