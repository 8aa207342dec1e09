"""The per-entry reductions (a thread-block cluster of up to 8 CTAs an entry,
one CTA from about 600 entries on)."""

import ctypes

import numpy as np
import pytest
import torch

from quatrex_b200 import _native
from quatrex_b200._interop import mat

pytestmark = pytest.mark.gpu


def test_convergence_measure_of_an_overflown_step(cuda_device):
    """|x| of an entry with an infinite part is infinite even if its other part
    is NaN (C99 hypot), so an energy whose decimation overflows holds up the
    batch-wide stop: alpha^2 / eps = (1 - i)(1 + i) 1e308 here, with the finite
    products 1e308 and -1e308 behind its real part."""
    lib = _native.load()
    dev = lambda v: torch.tensor(v, dtype=torch.complex128, device=cuda_device).reshape(2, 1, 1)  # noqa: E731
    a_ii, a_ij, a_ji = dev([1j, 1.0]), dev([1e154 * (1 + 1j), 0.0]), dev([1e154 * (1 + 1j), 0.0])
    x = torch.empty_like(a_ii)
    delta = torch.zeros(2, dtype=torch.float64, device=cuda_device)
    ws = torch.empty(int(lib.qtx_sancho_rubio_workspace(1, 2)), dtype=torch.uint8, device=cuda_device)
    it, conv = ctypes.c_int(0), ctypes.c_int(0)
    _native.check(lib.qtx_sancho_rubio(1, 2, mat(a_ii), mat(a_ij), mat(a_ji), mat(x), 1, 1e-6, 0, ctypes.byref(it),
                                       ctypes.byref(conv), delta.data_ptr(), None, ws.data_ptr(), ws.numel(),
                                       ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    np.testing.assert_array_equal(delta.cpu().numpy(), [np.inf, 0.0])
    assert it.value == 1 and conv.value == 0
