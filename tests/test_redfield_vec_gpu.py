"""FP64 Redfield RK4 with few right-hand sides (one launch for the time
loop): every exchange mode, ragged output ranges, kept states and the
observables' chunks, against a torch FP64 restatement of lime/oqs.py:453-472."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DT = 0.05


def _system(n, R, n_obs, seed):
    g = torch.Generator(device='cuda').manual_seed(seed)

    def c(*s):
        return torch.complex(torch.randn(*s, generator=g, device='cuda', dtype=torch.float64),
                             torch.randn(*s, generator=g, device='cuda', dtype=torch.float64))
    D = n * n
    return c(D, D) / D, c(R, n, n), [c(n, n) for _ in range(n_obs)]


def _reference(L, rho, steps, E):
    x = rho.reshape(rho.shape[0], -1).T.contiguous()
    n = rho.shape[-1]
    obs, states = [], []
    for _ in range(steps):
        k1 = L @ x
        k2 = L @ (x + DT / 2 * k1)
        k3 = L @ (x + DT / 2 * k2)
        k4 = L @ (x + DT * k3)
        x = x + DT / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
        r = x.T.reshape(-1, n, n)
        states.append(r)
        obs.append(torch.stack([torch.einsum('ij,bji->b', e, r) for e in E], -1) if E else None)
    return obs, states


def _close(got, ref, steps, D):
    # each stage adds at most ~D roundings of terms bounded by the result; 4 stages a step
    scale = ref.abs().max().item()
    assert (got - ref).abs().max().item() <= 2.2e-16 * 8 * steps * np.sqrt(D) * scale


@pytest.mark.parametrize('n,R', [(1, 1), (2, 1), (3, 5), (6, 1), (8, 1), (8, 8), (9, 1), (11, 3), (13, 1), (16, 2),
                                 (20, 1), (22, 1), (23, 8), (12, 9), (38, 1), (40, 3)])
def test_against_torch(n, R):
    from lime_gb300.redfield import propagate_vec
    steps = 6
    L, rho, E = _system(n, R, 3, n * 100 + R)
    obs, states = _reference(L, rho, steps, E)
    o, st, fin = propagate_vec((L, n), rho, DT, steps, E, states_every=1)
    _close(fin, states[-1], steps, n * n)
    _close(st, torch.stack(states, 1), steps, n * n)
    _close(o, torch.stack(obs, 1), steps, n ** 3)


@pytest.mark.parametrize('n', [3, 7, 14])
@pytest.mark.parametrize('states_every,obs_every,steps', [(0, 1, 70), (2, 3, 103), (4, 4, 9), (0, 5, 3), (3, 1, 1)])
def test_strides_and_chunks(n, states_every, obs_every, steps):
    from lime_gb300.redfield import propagate_vec
    L, rho, E = _system(n, 2, 2, n + steps)
    obs, states = _reference(L, rho, steps, E)
    o, st, fin = propagate_vec((L, n), rho, DT, steps, E, states_every=states_every, obs_every=obs_every)
    _close(fin, states[-1], steps, n * n)
    assert o.shape[1] == steps // obs_every
    if steps // obs_every:
        _close(o, torch.stack(obs[obs_every - 1::obs_every], 1), steps, n ** 3)
    if states_every and steps // states_every:
        _close(st, torch.stack(states[states_every - 1::states_every], 1), steps, n * n)


def test_small_workspace_keeps_the_tiled_path():
    """A caller that gives only the tiled path's workspace is served as before."""
    from lime_gb300 import _native as nat
    lib = nat.require_device()
    n, steps = 7, 3
    L, rho, _ = _system(n, 1, 0, 5)
    out = []
    for small in (False, True):
        P = rho.reshape(n * n, 1).clone()
        size = 3 * n * n * 16 if small else lib.lime_redfield_rk4_f64_workspace(n, 1)
        ws = torch.empty(size, dtype=torch.uint8, device='cuda')
        d = nat.RedfieldRK4Desc()
        d.n, d.n_rhs, d.n_steps, d.dt = n, 1, steps, DT
        d.R, d.rho = L.data_ptr(), P.data_ptr()
        d.workspace, d.workspace_bytes = ws.data_ptr(), size
        nat.check(lib.lime_redfield_rk4_f64(d, torch.cuda.current_stream().cuda_stream), 'rk4')
        out.append(P.clone())
    _close(out[0], out[1], steps, n * n)
