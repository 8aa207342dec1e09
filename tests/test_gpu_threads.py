"""Host threads that launch the same kernels at different sizes at the same time.

The shared-memory limit of a kernel is one attribute for all host threads: a
thread that sets it to the bytes of its own small call between another thread's
setting and launch makes that launch fail. Every call has to succeed and give
the bits of a call made alone."""

import ctypes
import threading

import numpy as np
import pytest
import torch

from quatrex_b200 import _native
from quatrex_b200._interop import mat

pytestmark = pytest.mark.gpu


# the distributed, the one-CTA (n <= 256, n <= 720, n <= 1024) and the multi-CTA inverses
@pytest.mark.parametrize("small,large,batch,ws,calls", [(33, 64, 4, False, 3000), (130, 256, 80, False, 200),
                                                        (520, 720, 1, False, 60), (730, 1024, 1, False, 30),
                                                        (520, 832, 1, True, 60)])
def test_inverses_of_two_sizes_from_two_threads(cuda_device, small, large, batch, ws, calls):
    lib = _native.load()
    work, failures = [], []
    for n in (small, large):
        rng = np.random.default_rng(n)
        a = torch.from_numpy(rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n)))
        a, stream = a.to(cuda_device), torch.cuda.Stream()
        nbytes = int(lib.qtx_zinv_workspace(n, batch)) if ws else 0
        scratch = torch.empty(max(nbytes, 256), dtype=torch.uint8, device=cuda_device)
        work.append((n, a, torch.empty_like(a), torch.empty_like(a), scratch, nbytes, stream))

    def call(n, a, x, scratch, nbytes, stream):
        _native.check(lib.qtx_zinv_batched_ws(n, batch, mat(a), mat(x), None, scratch.data_ptr() if nbytes else None,
                                              nbytes, ctypes.c_void_p(stream.cuda_stream)))

    for n, a, ref, _, scratch, nbytes, stream in work:
        call(n, a, ref, scratch, nbytes, stream)
    torch.cuda.synchronize()

    def loop(n, a, _, x, scratch, nbytes, stream):
        try:
            for _ in range(calls):
                call(n, a, x, scratch, nbytes, stream)
        except Exception as e:  # noqa: BLE001
            failures.append(e)

    threads = [threading.Thread(target=loop, args=w) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failures, failures[0]
    for _, _, ref, x, *_ in work:
        assert torch.equal(x, ref)
