"""The DMMA GEMM at the edges of its 32 x 32 tiles, 16 x 16 warp tiles, 16 x 8
fragments, 8-wide k-slices and 4-stage pipeline, against NumPy complex128.

Tolerance: a complex inner product of length k with three real products per
term errs by at most about (2 k + 6) u in units of |a||b| (u = 1.1e-16);
measured values grow like sqrt(k) u, the bound taken is 4 u sqrt(k + 4)
relative Frobenius."""

import ctypes

import numpy as np
import pytest
import torch

from quatrex_b200 import _native
from quatrex_b200._interop import mat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(16, 8, 4), (15, 9, 3), (17, 17, 8), (32, 31, 9), (33, 40, 12), (48, 24, 31),
                                   (31, 65, 32), (64, 33, 33), (100, 100, 40)])
@pytest.mark.parametrize("op_a,op_b", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_zgemm_tile_edges(cuda_device, m, n, k, op_a, op_b):
    rng = np.random.default_rng(m + 100 * n + 10000 * k)
    B, pad = 2, 3  # padded rows: leading dimensions larger than the width
    rand = lambda r, c: rng.standard_normal((B, r, c + pad)) + 1j * rng.standard_normal((B, r, c + pad))  # noqa: E731
    a, b, d = rand(*((k, m) if op_a else (m, k))), rand(*((n, k) if op_b else (k, n))), rand(m, n)
    A, Bt, D = (torch.from_numpy(x).to(cuda_device) for x in (a, b, d))
    h = lambda x, op: x.conj().swapaxes(-2, -1) if op else x  # noqa: E731
    ref = 2.0j * (h(a[..., :-pad], op_a) @ h(b[..., :-pad], op_b)) - d[..., :-pad]
    C = torch.full((B, m, n + pad), 7.0, dtype=torch.complex128, device=cuda_device)
    _native.check(_native.load().qtx_zgemm_batched(
        m, n, k, B, 0.0, 2.0, mat(A), op_a, mat(Bt), op_b, -1.0, 0.0, mat(D), 0, mat(C),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    got = C.cpu().numpy()
    assert (got[..., -pad:] == 7.0).all()
    err = np.linalg.norm(got[..., :-pad] - ref) / np.linalg.norm(ref)
    assert err < 4 * 1.1e-16 * np.sqrt(k + 4), err
