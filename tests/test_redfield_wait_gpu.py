"""A wait of the FP64 Redfield loop that runs out (one CTA of the grid left
out): the status word says so, every state and observable from then on holds
NaN in each right-hand side that lacks a value, the Python call raises, and
the context stays usable."""
import pytest
import torch

from lime_gb300 import _native as nat

pytestmark = pytest.mark.gpu
POLLS = 256


@pytest.fixture(scope='module')
def lib():
    from lime_gb300 import build
    build.build()
    return nat.require_device()


def _inputs(n, R, n_obs=2):
    g = torch.Generator(device='cuda').manual_seed(n)

    def c(*s):
        return torch.randn(*s, generator=g, device='cuda', dtype=torch.complex128)
    D = n * n
    return c(D, D) / D, c(R, n, n), [c(n, n) for _ in range(n_obs)]


class _Withheld:
    """The library with the self-test in the place of the call."""

    def __init__(self, lib):
        self.lib = lib

    def __getattr__(self, name):
        return getattr(self.lib, name)

    def lime_redfield_rk4_f64_status(self, d, status, max_wait, stream):
        return self.lib.lime_redfield_wait_selftest(d, status, POLLS, stream)


# n_rhs 8 at D = 121: a CTA's outputs are fewer than a row's numbers; 80 steps are three launches
@pytest.mark.parametrize('n,R,steps,every', [(20, 1, 6, 1), (16, 3, 80, 1), (14, 1, 7, 3), (11, 8, 5, 2)])
def test_expired_wait_is_reported(lib, monkeypatch, n, R, steps, every):
    from lime_gb300 import redfield
    L, rho, E = _inputs(n, R)
    monkeypatch.setattr(nat, 'require_device', lambda: _Withheld(lib))
    with pytest.raises(nat.KernelFlagError) as err:
        redfield.propagate_vec((L, n), rho, 0.05, steps, E, obs_every=every)
    assert err.value.flags == nat.LIME_FLAG_TIMEOUT
    word = torch.zeros(1, dtype=torch.int32, device='cuda')
    o, st, fin = redfield.propagate_vec((L, n), rho, 0.05, steps, E, states_every=1, obs_every=every, status=word)
    assert int(word.item()) == nat.LIME_FLAG_TIMEOUT
    with pytest.raises(nat.KernelFlagError):
        redfield.check_status(word)
    assert o.shape[1] == steps // every and bool(torch.isnan(torch.view_as_real(o)).any(-1).all())
    for x in (st.reshape(R * steps, n * n), fin.reshape(R, n * n)):
        assert bool(torch.isnan(torch.view_as_real(x)).any(-1).any(-1).all())
    monkeypatch.undo()
    a = redfield.propagate_vec((L, n), rho, 0.05, 3, E)
    b = redfield.propagate_vec((L, n), torch.cat([rho] * 9), 0.05, 3, E)      # the tiled path
    assert (a[2] - b[2][:R]).abs().max().item() < 1e-13 * b[2].abs().max().item()


def test_arguments(lib):
    d = nat.RedfieldRK4Desc()
    word = torch.zeros(1, dtype=torch.int32, device='cuda')
    assert lib.lime_redfield_rk4_f64_status(None, word.data_ptr(), 0, None) == -1
    assert lib.lime_redfield_wait_selftest(d, None, POLLS, None) == -1
    assert lib.lime_redfield_wait_selftest(d, word.data_ptr(), 0, None) == -1


def test_no_waits_to_expire(lib):
    """Sizes of one CTA and of a cluster have no such waits."""
    for n in (2, 6):
        L, rho, _ = _inputs(n, 1)
        size = lib.lime_redfield_rk4_f64_workspace(n, 1)
        ws = torch.empty(size, dtype=torch.uint8, device='cuda')
        word = torch.zeros(1, dtype=torch.int32, device='cuda')
        d = nat.RedfieldRK4Desc()
        d.n, d.n_rhs, d.n_steps, d.dt = n, 1, 2, 0.05
        d.R, d.rho = L.data_ptr(), rho.data_ptr()
        d.workspace, d.workspace_bytes = ws.data_ptr(), size
        assert lib.lime_redfield_wait_selftest(d, word.data_ptr(), POLLS, None) == -2


@pytest.mark.parametrize('n,steps,fixed', [(2, 120000, 900), (6, 60000, 1700), (14, 30000, 3600)])
def test_launches_are_bounded(lib, n, steps, fixed):
    """A stage takes at least its mode's fixed clocks; 2e8 of them are a launch."""
    from lime_gb300 import redfield
    D = n * n
    L = torch.zeros(D, D, dtype=torch.complex128, device='cuda')
    rho = torch.ones(1, n, n, dtype=torch.complex128, device='cuda')
    before = nat.launch_count()
    _, _, fin = redfield.propagate_vec((L, n), rho, 0.05, steps)
    assert nat.launch_count() - before >= 4 * steps * fixed / 2e8
    assert torch.equal(fin, rho)


@pytest.mark.parametrize('n', [2, 6, 14])
def test_captured_call(lib, n):
    """A call recorded in a graph reads nothing back and replays."""
    from lime_gb300 import redfield
    L, rho, E = _inputs(n, 1)
    want = redfield.propagate_vec((L, n), rho, 0.05, 5, E)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = redfield.propagate_vec((L, n), rho, 0.05, 5, E)
    for _ in range(2):
        graph.replay()
        assert torch.equal(got[0], want[0]) and torch.equal(got[2], want[2])
