"""Batches above the limits of one launch.

From 65536 entries on the products, the anti-Hermitian parts and the
conversions loop over their entries, in launches that hold several products
also from one product to the next; the reductions take one CTA per entry
instead of eight. An entry's result depends on neither, so every block and
current must have the bits of a batch of six."""

import numpy as np
import pytest
import scipy.sparse as sps
import torch

from quatrex_b200 import RGF, DSDBCOO, SanchoRubio, synthetic

pytestmark = pytest.mark.gpu

BATCH = 70000
SOME = [0, 1, 34999, 35000, 65536, BATCH - 1]


def _stack(dense, bs, factor):
    m = DSDBCOO.from_sparray(sps.coo_matrix(dense), bs, (1,))
    return DSDBCOO(m.data.to(factor.device) * factor[:, None], m.rows, m.cols, bs, (len(factor),))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_selected_solve(cuda_device, precision):
    bs = np.array([2, 3, 2])
    dense = synthetic.random_bt_dense(bs, seed=5)
    anti = [c * dense - np.conj(c) * dense.conj().T for c in (1.0, 1.0j)]
    factor = 1.0 + 0.2 * torch.rand(3, BATCH, dtype=torch.float64, device=cuda_device)
    solver = RGF(max_batch_size=BATCH, precision=precision)

    def solve(f):
        a, sl, sg = (_stack(d, bs, x) for d, x in zip((dense, *anti), f))
        xl, xg, xr, current = solver.selected_solve(a, sl, sg, return_retarded=True, return_current=True)
        return xl.data, xg.data, xr.data, current

    every, few = solve(factor), solve(factor[:, SOME])
    for x, y in zip(every, few):
        assert torch.equal(x[SOME], y)
        assert bool(torch.isfinite(torch.view_as_real(x)).all())


def test_decimation(cuda_device):
    rng = torch.Generator(device=cuda_device).manual_seed(7)
    r = lambda: torch.randn(BATCH, 3, 3, dtype=torch.complex128, device=cuda_device, generator=rng)  # noqa: E731
    system = (4.0 * torch.eye(3, dtype=torch.complex128, device=cuda_device) + 0.3 * r(), 0.4 * r(), 0.4 * r())
    sr = SanchoRubio(max_iterations=40, convergence_tol=1e-10, per_energy=True)
    x, _, converged = sr.solve_device(*system)
    y, _, _ = sr.solve_device(*(t[SOME].contiguous() for t in system))
    assert converged and torch.equal(x[SOME], y)
