"""The batched split kernel for dimensions up to 32 gives the 64-wide
kernel's results bit for bit: the same system padded to 33 levels runs there
(the padding is zero), with the same scales."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
CDT = torch.complex128


def _run(n, B, H, rates, rho, E, mode, steps, obs_every, prepared, sb):
    from lime_gb300 import engine, _native as nat
    lib = nat.require_device()
    gen = engine.LindbladGenerator.build(H, [engine.SiteDephasing(rates)])
    d = nat.SplitDesc()
    n_obs = E.shape[0] if mode == 2 else 5
    obs = torch.zeros((B, steps // obs_every, max(n_obs, 1)), dtype=CDT, device='cuda')
    status = torch.zeros(1, dtype=torch.int32, device='cuda')
    out = torch.empty_like(rho)
    ops = engine.split_operands(gen)
    d.n, d.batch, d.param_batch, d.n_steps = n, B, B, steps
    d.obs_mode, d.n_obs, d.obs_every = mode, n_obs, obs_every
    d.scale_a_log2 = ops['scale_a']
    d.scale_b_log2 = sb
    if prepared:
        d.a_pieces, d.a_stride = ops['pieces'].data_ptr(), ops['stride']
    d.dt, d.trace_tol = 0.05, 1e-5
    d.rho, d.rho_out = rho.data_ptr(), out.data_ptr()
    d.heff, d.heff_stride = gen.heff.data_ptr(), (0 if gen.heff.shape[0] == 1 else n * n)
    d.m_diag, d.m_stride = ops['m_diag'].data_ptr(), (0 if ops['m_diag'].shape[0] == 1 else n)
    d.obs_ops, d.obs_stride = E.data_ptr(), 0
    d.obs_out, d.status = obs.data_ptr(), status.data_ptr()
    nat.check(lib.lime_lindblad_rk4_split(d, torch.cuda.current_stream().cuda_stream), 'split')
    assert int(status.item()) == 0
    return obs, out


@pytest.mark.parametrize('n,B', [(5, 1), (7, 3), (8, 2), (9, 700), (15, 2), (16, 1), (16, 610), (16, 1300), (17, 1),
                                 (24, 305), (31, 3), (32, 1), (32, 304), (32, 306), (32, 1300)])
@pytest.mark.parametrize('mode,obs_every,prepared', [(1, 1, True), (2, 2, False)])
def test_bitwise_equal_to_the_64_wide_kernel(n, B, mode, obs_every, prepared):
    rng = np.random.default_rng(n * 1000 + B)
    N, steps = 33, 6
    H = 0.1 * rng.normal(size=(B, n, n)) + 0.1j * rng.normal(size=(B, n, n))
    H = H + H.conj().swapaxes(1, 2)
    rates = 0.02 * rng.random((B, n))
    psi = rng.normal(size=(B, n)) + 1j * rng.normal(size=(B, n))
    psi /= np.linalg.norm(psi, axis=1, keepdims=True)
    rho = psi[:, :, None] * psi[:, None, :].conj()
    rho = (rho + rho.conj().swapaxes(1, 2)) / 2
    E = rng.normal(size=(2, n, n)) + 1j * rng.normal(size=(2, n, n))

    def pad(x, axes):
        w = [(0, 0)] * x.ndim
        for a in axes:
            w[a] = (0, N - n)
        return torch.as_tensor(np.pad(x, w), device='cuda').contiguous()

    def dev(x):
        return torch.as_tensor(np.ascontiguousarray(x), device='cuda')
    sb = 13 - int(np.ceil(np.log2(np.sqrt(32))))
    o, r = _run(n, B, dev(H), dev(rates), dev(rho), dev(E), mode, steps, obs_every, prepared, sb)
    O, R = _run(N, B, pad(H, (1, 2)), pad(rates, (1,)), pad(rho, (1, 2)), pad(E, (1, 2)), mode, steps, obs_every,
                prepared, sb)
    assert torch.equal(torch.view_as_real(r), torch.view_as_real(R[:, :n, :n].contiguous()))
    assert torch.equal(torch.view_as_real(o), torch.view_as_real(O))


@pytest.mark.parametrize('n', [1, 4, 16, 20, 32])
def test_against_fp64(n):
    from lime_gb300 import engine
    rng = np.random.default_rng(n)
    H = np.diag(0.05 * rng.normal(size=n)) - 0.1 * (np.eye(n, k=1) + np.eye(n, k=-1))
    gen = engine.LindbladGenerator.build(H.astype(complex), [engine.SiteDephasing(np.full(n, 0.01))])
    rho = np.full((n, n), 1.0 / n, complex)
    o, _, r = engine.propagate(gen, rho, 0.05, 200, engine.Populations(n), precision='split')
    o64, _, r64 = engine.propagate(gen, rho, 0.05, 200, engine.Populations(n))
    assert (o - o64).abs().max().item() < 1e-6 and (r - r64).abs().max().item() < 1e-6
    # a start that is not Hermitian is still recognised and run as two parts
    if n > 1:
        rho[0, 1] += 0.25
        _, _, r = engine.propagate(gen, rho, 0.05, 20, None, precision='split')
        _, _, r64 = engine.propagate(gen, rho, 0.05, 20, None)
        assert (r - r64).abs().max().item() < 1e-6
