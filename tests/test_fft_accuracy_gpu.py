"""Rounding error of lime_fft_f64 at powers of two, beside the one of the
plain radix-2 transform (u + t, u - t with t = w v formed by a product and a
fused product, factors rounded to nearest) on the same inputs, both against
extended precision.

Tolerance: the two rms are sums over some 10^5 independent roundings, known to
about half a per cent; the bound leaves two."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _fma(a, b, c):
    return (np.longdouble(1) * a * b + c).astype(np.float64)


def _radix2(x):
    n = x.shape[-1]
    bits = n.bit_length() - 1
    order = [int(format(i, '0%db' % bits)[::-1], 2) for i in range(n)]
    re, im = x.real[:, order], x.imag[:, order]
    h = 1
    while h < n:
        a = -np.arange(h) * (np.arccos(np.longdouble(-1)) / h)
        wx, wy = np.cos(a).astype(np.float64), np.sin(a).astype(np.float64)
        if h > 1:
            wx[h // 2] = 0.0
        re, im = re.reshape(-1, n // (2 * h), 2, h), im.reshape(-1, n // (2 * h), 2, h)
        ur, vr, ui, vi = re[:, :, 0], re[:, :, 1], im[:, :, 0], im[:, :, 1]
        tr, ti = _fma(wx, vr, -(wy * vi)), _fma(wx, vi, wy * vr)
        re = np.stack([ur + tr, ur - tr], 2).reshape(-1, n)
        im = np.stack([ui + ti, ui - ti], 2).reshape(-1, n)
        h *= 2
    return re + 1j * im


@pytest.mark.parametrize('n', [64, 128, 256, 512, 1024, 2048, 4096])
def test_no_further_than_radix2(n):
    from lime_gb300.spectra import _dft_rows
    rng = np.random.default_rng(n)
    B = 2 ** 17 // n
    x = rng.normal(size=(B, n)) + 1j * rng.normal(size=(B, n))
    exact = np.fft.fft(x.astype(np.clongdouble), axis=-1)
    assert exact.dtype == np.clongdouble
    got = _dft_rows(torch.as_tensor(x, device='cuda'), False, False, None).cpu().numpy()

    def rms(y):
        return float(np.sqrt(np.mean(np.abs(y - exact) ** 2)))
    assert rms(got) <= 1.02 * rms(_radix2(x))
