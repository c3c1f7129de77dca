"""Which PCG a system is solved by, and that each solves it: the resident one up to where a CTA's rows
can be kept or staged, the fused kernels (scenes) and the per-kernel PCG (linear-solver seam)
beyond. mguso_scene_pcg_kernels tells them apart: it names no kernels before a fused solve."""
import numpy as np
import pytest

from mguso import CsrMatrix, CudaLinearSolver, ImplicitSolver, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precond", ["schwarz", "block"])
@pytest.mark.parametrize("n", [400, 470, 500])
def test_solver_around_the_limit(ctx, n, precond):
    """34, 47 and 53 domains a CTA: rows walked in the BSR, with Schwarz from 47 on the per-kernel PCG. The
    residual formed in float64 against ||b||, bounded as in the resident PCG's tests: 1e-6 by the solver's own FP32
    recurrence, which drifts by about iterations * 2^-24 (20 to 30 iterations)."""
    nb, rp, col, val = scenes.grid_bsr(n, seed=n)
    b = np.random.default_rng(n).standard_normal(3 * nb).astype(np.float32)
    a = CsrMatrix(*scenes.bsr_to_csr(nb, rp, col, val))
    for precision in ("mixed", "fp32"):
        s = CudaLinearSolver(ctx, precond=precond, domain=32, precision=precision)
        x = s.solve(a, b, 1e-6, 500)
        st = s.last_stats()
        assert st.status == 0 and 0 < st.iters < 500
        assert np.array_equal(x, s.solve(a, b, 1e-6, 500))
        s.close()
        r = b.astype(np.float64) - scenes.bsr_spmv_f64(rp, col, val, x)
        assert np.linalg.norm(r) / np.linalg.norm(b) <= 5e-6


@pytest.mark.parametrize("n,precond,domain,fused", [(300, 1, 32, False), (360, 1, 32, True), (330, 2, 32, False),
                                                    (400, 2, 32, True), (100, 2, 8, False), (150, 2, 8, True)])
def test_scenes_take_the_fused_kernels_where_rows_would_be_walked(ctx, n, precond, domain, fused):
    """20 and 28 runs a CTA (block Jacobi), 24 and 34 domains (Schwarz); of small domains 9 and 20."""
    sc = scenes.sheet_on_sphere(n, height=0.32)
    sc["params"] = dict(sc["params"], precond=precond, schwarz_domain=domain, newton_iters=2)
    g = ImplicitSolver(ctx, sc, "mixed")
    assert g.step(1)[0]["status"] == 0
    assert (g.pcg_kernels() != (-1, -1)) == fused
    g.close()


@pytest.mark.parametrize("n", [40, 130, 330, 400])
def test_mode_2_sums_over_fp16_tiles_in_fp64(ctx, n):
    """Mixed precision with FP16 tiles and pcg_mode 2: one, four and 24 (staged) domains a CTA and the fused
    kernels. Against the fused pair whose one-warp domain kernel sums in FP64 (pcg_variant 1), after
    four iterations from a rough right-hand side that moves vertices by a metre: FP64 sums in another
    order differ by 1e-13 or less of their terms, so a result rounds to another FP32 number for one entry in
    1e5 at most, where FP32 sums (1e-7) change every third to fiftieth."""
    sc = scenes.sheet_on_sphere(n, height=2.0)
    sc["velocities"] = (60 * np.random.default_rng(n).standard_normal(sc["positions"].shape)).astype(np.float32)
    out = []
    for kw in (dict(pcg_variant=1), dict(pcg_mode=2)):
        p = dict(sc["params"], self_collision=0, newton_iters=1, cg_max_iter=4, cg_tol=1e-9, **kw)
        g = ImplicitSolver(ctx, dict(sc, params=p), "mixed")
        assert g.step(1)[0]["status"] == 0
        out.append(g.positions.copy())
        g.close()
    assert np.abs(out[0] - sc["positions"]).max() > 0.5
    assert (out[0] == out[1]).mean() >= 0.999


@pytest.mark.parametrize("nv", [5000, 20000, 60000])
def test_random_patterns(ctx, nv):
    """Eight random neighbours a vertex: halos of up to ten thousand vertices a CTA, past the resident
    table's 1 536, and Schwarz domains of one to 32 vertices. Diagonally dominant, so 20 to 30 iterations;
    residual in float64 and its bound as above."""
    rng = np.random.default_rng(nv)
    e = rng.integers(0, nv, (4 * nv, 2))
    e = np.unique(np.sort(e[e[:, 0] != e[:, 1]], 1), axis=0)
    d = rng.standard_normal((len(e), 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    blk = d[:, :, None] * d[:, None, :]
    diag = np.tile(2.0 * np.eye(3), (nv, 1, 1))
    np.add.at(diag, e[:, 0], blk)
    np.add.at(diag, e[:, 1], blk)
    rows = np.concatenate([np.arange(nv), e[:, 0], e[:, 1]])
    cols = np.concatenate([np.arange(nv), e[:, 1], e[:, 0]])
    vals = np.concatenate([diag, -blk, -blk]).astype(np.float32)
    o = np.lexsort((cols, rows))
    rp = np.zeros(nv + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=nv), out=rp[1:])
    rp, cols, vals = rp.astype(np.uint32), cols[o].astype(np.uint32), vals[o]
    b = rng.standard_normal(3 * nv).astype(np.float32)
    a = CsrMatrix(*scenes.bsr_to_csr(nv, rp, cols, vals))
    for precond in ("schwarz", "block"):
        s = CudaLinearSolver(ctx, precond=precond, domain=32)
        x = s.solve(a, b, 1e-6, 500)
        st = s.last_stats()
        assert st.status == 0 and 0 < st.iters < 500
        s.close()
        r = b.astype(np.float64) - scenes.bsr_spmv_f64(rp, cols, vals, x)
        assert np.linalg.norm(r) / np.linalg.norm(b) <= 5e-6


@pytest.mark.parametrize("n,domain", [(40, 1), (40, 8), (40, 10), (100, 8), (120, 10)])
def test_one_tile_domains_sum_in_fp64(ctx, n, domain):
    """The default mode over domains of one tile: as pcg_mode 2 above, against the one-warp fused kernel."""
    sc = scenes.sheet_on_sphere(n, height=2.0)
    sc["velocities"] = (60 * np.random.default_rng(n).standard_normal(sc["positions"].shape)).astype(np.float32)
    out = []
    for kw in (dict(pcg_variant=1), {}):
        p = dict(sc["params"], self_collision=0, newton_iters=1, cg_max_iter=4, cg_tol=1e-9, schwarz_domain=domain, **kw)
        g = ImplicitSolver(ctx, dict(sc, params=p), "mixed")
        assert g.step(1)[0]["status"] == 0
        out.append(g.positions.copy())
        if not kw:
            assert g.pcg_kernels() == (-1, -1)  # resident
        g.close()
    assert (out[0] == out[1]).mean() >= 0.999


def test_solvers_on_threads_share_the_gpu():
    """Three threads, each with its own context and solver, solve at once: every launch wants all SMs, so
    they take turns, and each solution is the one a solver alone finds, bit for bit."""
    import threading

    from mguso import Context

    nb, rp, col, val = scenes.grid_bsr(100, seed=2)  # more domains than SMs
    a = CsrMatrix(*scenes.bsr_to_csr(nb, rp, col, val))
    b = np.random.default_rng(1).standard_normal(3 * nb).astype(np.float32)
    out = [[], [], []]

    def work(mine):
        ctx = Context(0)
        s = CudaLinearSolver(ctx, precond="schwarz", domain=32)
        for _ in range(20):
            mine.append(s.solve(a, b, 1e-6, 500))
        s.close()
        ctx.close()

    threads = [threading.Thread(target=work, args=(mine,)) for mine in out]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert [len(mine) for mine in out] == [20, 20, 20]
    assert all(np.array_equal(x, out[0][0]) for mine in out for x in mine)
