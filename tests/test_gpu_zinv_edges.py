"""The batched inverse at the edges of its paths: panels of 16 columns, the
shared-memory-resident limit (n = 103), the row and column splits, blocks of
257-512 columns (two CTAs at least from 433 on), and pivot ties.

Gauss-Jordan with partial pivoting leaves a residual of a few n u |A||X| for
well-conditioned blocks (u = 1.1e-16); the bound taken is 8 n u relative to
||A||_F ||X||_F (measured: below u)."""

import ctypes

import numpy as np
import pytest
import torch

from quatrex_b200 import _native
from quatrex_b200._interop import mat

pytestmark = pytest.mark.gpu


def _inv(a, path):
    lib = _native.load()
    B, n = a.shape[0], a.shape[-1]
    x = torch.full_like(a, float("nan"))
    info = torch.zeros(B, dtype=torch.int32, device=a.device)
    ws = torch.empty(max(int(lib.qtx_zinv_workspace(n, B)), 256), dtype=torch.uint8, device=a.device)
    _native.check(lib.qtx_set_inverse_path(path))
    try:
        _native.check(lib.qtx_zinv_batched_ws(n, B, mat(a), mat(x), info.data_ptr(), ws.data_ptr(), ws.numel(),
                                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    finally:
        _native.check(lib.qtx_set_inverse_path(0))
    return x, info.cpu().numpy()


def _residual(a, x):
    eye = torch.eye(a.shape[-1], dtype=a.dtype, device=a.device)
    return float((a @ x - eye).norm() / (a.norm() * x.norm()))


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 33, 64, 65, 96, 100, 101, 102, 103, 104, 128, 129, 200, 256,
                               257, 400, 416, 417, 432, 433, 512])
@pytest.mark.parametrize("batch", [2, 40])
def test_inverse_sizes_and_paths(cuda_device, n, batch):
    rng = np.random.default_rng(n)
    a = torch.from_numpy(rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))).to(cuda_device)
    x, info = _inv(a, 0)
    assert not info.any() and _residual(a, x) < 8 * n * 1.1e-16
    same = [_inv(a, p)[0] for p in ((1, 3, 4) if n <= 256 else (1, 4))]
    for y in same:
        assert torch.equal(y, x)
    y = a.clone()  # in place, padded rows
    pad = torch.zeros((batch, n, n + 3), dtype=a.dtype, device=a.device)
    pad[..., :n] = y
    _native.check(_native.load().qtx_zinv_batched(n, batch, mat(pad), mat(pad), None,
                                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert torch.equal(pad[..., :n].contiguous(), x) and not pad[..., n:].any()


@pytest.mark.parametrize("n", [20, 100, 130, 300])
@pytest.mark.parametrize("path", [1, 3, 4])
def test_pivot_ties_and_singular_blocks(cuda_device, n, path):
    """Entries from {+-1, +-i}: every column starts with n equal measures, so
    the lowest row has to win; block 1 has a zero column, block 2 is a
    permutation (exact result)."""
    if path == 3 and n > 256:
        pytest.skip("the distributed path takes n <= 256")
    rng = np.random.default_rng(n + path)
    a = np.array([1, -1, 1j, -1j])[rng.integers(0, 4, (3, n, n))].astype(np.complex128)
    a[1, :, n // 2] = 0.0
    perm = rng.permutation(n)
    a[2] = np.eye(n)[perm]
    t = torch.from_numpy(a).to(cuda_device)
    x, info = _inv(t, path)
    assert info[0] == 0 and info[1] == n // 2 + 1 and info[2] == 0
    assert _residual(t[:1], x[:1]) < 8 * n * 1.1e-16
    np.testing.assert_array_equal(x[2].cpu().numpy(), a[2].T)
    assert torch.equal(_inv(t, 4)[0][::2], x[::2])
