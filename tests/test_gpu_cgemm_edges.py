"""The split-TF32 complex64 GEMM at the edges of its 128 x 64 tiles and 32-wide
K blocks, with a plain and a conjugate-transposed addend, against complex128.

Each real product keeps a_hi b_hi + a_hi b_lo + a_lo b_hi of tf32 halves and is
accumulated in FP32: about 2^-21 per term and sqrt(k) 2^-24 of summation; the
bound taken is max(5e-6, 5e-7 sqrt(k)) relative Frobenius."""

import ctypes

import numpy as np
import pytest
import torch

from quatrex_b200 import _native
from quatrex_b200._interop import mat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(1, 1), (31, 33), (64, 32), (65, 31), (127, 64), (128, 65), (129, 96), (200, 40)])
@pytest.mark.parametrize("op_a,op_b,op_d", [(0, 0, 0), (0, 1, 1), (1, 0, 1), (1, 1, 0)])
def test_cgemm_tile_edges(cuda_device, n, k, op_a, op_b, op_d):
    rng = np.random.default_rng(1000 * n + k)
    rand = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)  # noqa: E731
    B = 3
    a, b, d = rand(B, *((k, n) if op_a else (n, k))), rand(B, *((n, k) if op_b else (k, n))), rand(B, n, n)
    h = lambda x, op: x.conj().swapaxes(-2, -1) if op else x  # noqa: E731
    ref = (0.5 - 1.0j) * (h(a, op_a).astype(complex) @ h(b, op_b)) + 2.0j * h(d, op_d)
    A, Bt, D = (torch.from_numpy(x).to(cuda_device) for x in (a, b, d))
    C = torch.full((B, n, n), float("nan"), dtype=torch.complex64, device=cuda_device)
    _native.check(_native.load().qtx_cgemm_batched(
        n, n, k, B, 0.5, -1.0, mat(A), op_a, mat(Bt), op_b, 0.0, 2.0, mat(D), op_d, mat(C), None,
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    err = np.linalg.norm(C.cpu().numpy() - ref) / np.linalg.norm(ref)
    assert err < max(5e-6, 5e-7 * np.sqrt(k)), err
