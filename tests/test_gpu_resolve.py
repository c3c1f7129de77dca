"""Re-solves through the linear-solver seam on a pattern that is kept: the values that the device
gathers are those that a fresh solver builds, so solutions are the same bit for bit."""
import numpy as np
import pytest

from mguso import CsrMatrix, CudaLinearSolver, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", ["schwarz", "schwarz-ml", "block"])
@pytest.mark.parametrize("form", ["plain", "ragged", "twice", "unsorted"])
def test_resolve_matches_fresh(ctx, precond, form):
    nb, rp, col, val = scenes.grid_bsr(9, 4)
    n, crp, ci, cv = scenes.bsr_to_csr(nb, rp, col, val)
    crp, ci, cv = np.asarray(crp).astype(np.int64), np.asarray(ci), np.asarray(cv, np.float32)
    row = np.repeat(np.arange(n), np.diff(crp))
    if form == "ragged":  # blocks with entries left out (zeros of their block)
        keep = (row == ci) | ((row * 7 + ci * 7) % 5 != 0)
        row, ci, cv = row[keep], ci[keep], cv[keep]
    if form == "twice":  # every 11th entry as two halves
        d = np.arange(ci.size) % 11 == 0
        cv = np.where(d, cv * np.float32(0.5), cv)
        o = np.argsort(np.concatenate([np.arange(ci.size), np.flatnonzero(d)]), kind="stable")
        row, ci, cv = (np.concatenate([a, a[d]])[o] for a in (row, ci, cv))
    if form == "unsorted":
        o = np.lexsort((-ci.astype(np.int64), row))
        row, ci, cv = row[o], ci[o], cv[o]
    crp = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(row, minlength=n), out=crp[1:])
    b = np.random.default_rng(1).standard_normal(n).astype(np.float32)
    kept = CudaLinearSolver(ctx, precond=precond, domain=32)
    for scale in (1.0, 1.25, 0.75):  # exact in binary
        v = cv * np.float32(scale)
        v[v == 0] = -0.0
        a = CsrMatrix(n, crp.astype(np.uint32), ci.astype(np.uint32), v)
        x = kept.solve(a, b, 1e-6, 300)
        fresh = CudaLinearSolver(ctx, precond=precond, domain=32)
        assert np.array_equal(x, fresh.solve(a, b, 1e-6, 300))
        fresh.close()
    kept.close()
