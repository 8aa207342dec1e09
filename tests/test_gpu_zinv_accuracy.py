"""Rounding of the inverse's panel elimination, against the same elimination
in NumPy with every complex product formed (one rounding of it) before it is
subtracted. Adding the two real products to the element one after another
instead rounds at the size of the element twice: over these matrices its error
is 1.19 times as large, that of the product formed first 1.00. The mean over
1000 matrices scatters by 1.5 %, so the bound is 1.06."""

import ctypes

import numpy as np
import pytest
import torch

from quatrex_b200 import _native
from quatrex_b200._interop import mat

LD = np.longdouble


def _fma(a, b, c):
    return (a.astype(LD) * b.astype(LD) + c.astype(LD)).astype(float)


def _mul(a, b):
    return _fma(a[0], b[0], -(a[1] * b[1])), _fma(a[0], b[1], a[1] * b[0])


def _gauss_jordan(a, chained=False):
    """Inverses by Gauss-Jordan with the kernels' pivot rule, (B, n, n)."""
    batch, n, _ = a.shape
    x, every = [a.real.copy(), a.imag.copy()], np.arange(batch)
    order = np.tile(np.arange(n), (batch, 1))
    for k in range(n):
        p = k + np.argmax(np.abs(x[0][:, k:, k]) + np.abs(x[1][:, k:, k]), axis=1)
        for y in (*x, order):
            t = y[every, k].copy()
            y[every, k] = y[every, p]
            y[every, p] = t
        d = 1.0 / (x[0][:, k, k].astype(LD) + 1j * x[1][:, k, k].astype(LD))
        d = [d.real.astype(float)[:, None], d.imag.astype(float)[:, None]]
        row, m = _mul(d, [y[:, k, :] for y in x]), _mul([y[:, :, k] for y in x], d)
        mc, q = [y[:, :, None] for y in m], [y[:, None, k, :].copy() for y in x]
        if chained:
            x = [_fma(-mc[0], q[0], _fma(mc[1], q[1], x[0])), _fma(-mc[0], q[1], _fma(-mc[1], q[0], x[1]))]
        else:
            t = _mul(mc, q)
            x = [x[0] - t[0], x[1] - t[1]]
        for i in range(2):
            x[i][:, :, k] = -m[i]
            x[i][:, k, :] = row[i]
            x[i][:, k, k] = d[i][:, 0]
    out = np.empty_like(a)
    for b in range(batch):
        out[b][:, order[b]] = x[0][b] + 1j * x[1][b]
    return out


def _error(a, x):
    """Relative error, to first order from an 80-bit residual."""
    xl = x.astype(np.clongdouble)
    dx = (xl @ (np.eye(a.shape[1]) - a.astype(np.clongdouble) @ xl)).astype(complex)
    return np.linalg.norm(dx, axis=(1, 2)) / np.linalg.norm(x, axis=(1, 2))


def _matrices(n=16, batch=1000):
    """Energies minus a Hermitian block, as the decimation inverts them."""
    rng = np.random.default_rng(16)
    m = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    return (np.linspace(-1, 1, batch)[:, None, None] + 1e-3j) * np.eye(n) - (m + m.conj().swapaxes(1, 2)) / 16.0


def _ratio(a, x):
    return float(np.exp(np.mean(np.log(_error(a, x) / _error(a, _gauss_jordan(a))))))


def test_the_bound_tells_the_two_apart():
    a = _matrices()
    assert _ratio(a, _gauss_jordan(a, chained=True)) > 1.15


@pytest.mark.gpu
def test_panel_elimination_rounds_products_once(cuda_device):
    a = _matrices()
    t = torch.from_numpy(a).to(cuda_device)
    x = torch.empty_like(t)
    _native.check(_native.load().qtx_zinv_batched(a.shape[1], a.shape[0], mat(t), mat(x), None,
                                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    r = _ratio(a, x.cpu().numpy())
    assert r < 1.06, r
