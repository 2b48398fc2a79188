"""lime_fft_f64 at every power of two it takes (each remainder of the
three-stage passes) and at chirp-z lengths on both sides of the powers of
two, against numpy in 64 bits: both signs, shifted and strided."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [1 << k for k in range(14)] + [3, 5, 7, 9, 15, 31, 33, 63, 65, 127, 129, 511, 999, 1023, 1025, 2047, 2049,
                                         4095]


@pytest.mark.parametrize('n', LENGTHS)
@pytest.mark.parametrize('inverse,shift,strided', [(0, 0, False), (1, 1, True)])
def test_against_numpy(n, inverse, shift, strided):
    from lime_gb300 import _native as nat
    lib = nat.require_device()
    B = 5
    rng = np.random.default_rng(n)
    x = rng.normal(size=(B, n)) + 1j * rng.normal(size=(B, n))
    post = np.exp(1j * rng.normal(size=n))
    ref = np.fft.ifft(x, axis=-1) * n if inverse else np.fft.fft(x, axis=-1)
    if shift:
        ref = np.roll(ref, n // 2, axis=-1) * post
    xt = torch.as_tensor(x, device='cuda')
    y = torch.empty((B, n), dtype=torch.complex128, device='cuda')
    if strided:
        xt = xt.t().contiguous().t()
        y = torch.empty((n, B), dtype=torch.complex128, device='cuda').t()
    pt = torch.as_tensor(post, device='cuda')
    wsb = int(lib.lime_fft_f64_workspace(n, B))
    ws = torch.empty(max(wsb, 16), dtype=torch.uint8, device='cuda')
    d = nat.FftDesc()
    d.n, d.batch, d.inverse, d.shift = n, B, inverse, shift
    d.x, d.x_s, d.x_bs = xt.data_ptr(), xt.stride(1), xt.stride(0)
    d.y, d.y_s, d.y_bs = y.data_ptr(), y.stride(1), y.stride(0)
    if shift:
        d.post = pt.data_ptr()
    d.workspace, d.workspace_bytes = ws.data_ptr(), wsb
    nat.check(lib.lime_fft_f64(d, torch.cuda.current_stream().cuda_stream), 'fft')
    got = y.cpu().numpy()
    # 2^-53 per stage and butterfly; the chirp-z form runs three transforms of up to 4 n
    err = np.linalg.norm(got - ref) / np.linalg.norm(ref)
    assert err < 4e-16 * (3 * np.log2(max(n, 2)) + 6)
