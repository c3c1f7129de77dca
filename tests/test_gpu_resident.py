"""The resident PCG (one cooperative launch per solve) through the linear-solver seam and the
step, at the sizes where its layout changes: fewer vertices than a domain, ragged domains,
rows that outgrow shared memory (staged), columns beyond the halo table (walked in the BSR),
isolated vertices with and without a load, and a system too large for it (per-kernel PCG).

Solves: the residual formed in float64 from the returned x. The solver stops at ||r|| <= 1e-6
||b|| by its own FP32 recurrence, whose residual drifts from the true one by at most about
iterations * 2^-24 (1e-6 for the 20 to 30 iterations of these matrices): bound 5e-6."""
import numpy as np
import pytest

from mguso import CsrMatrix, CudaLinearSolver, ImplicitSolver, scenes

pytestmark = pytest.mark.gpu


def solve_residual(ctx, nb, rp, col, val, precond, precision, b):
    a = CsrMatrix(*scenes.bsr_to_csr(nb, rp, col, val))
    s = CudaLinearSolver(ctx, precond=precond, domain=32, precision=precision)
    x = s.solve(a, b, 1e-6, 500)
    st = s.last_stats()
    assert st.status == 0 and 0 < st.iters < 500
    assert np.array_equal(x, s.solve(a, b, 1e-6, 500))  # reproducible
    s.close()
    r = b.astype(np.float64) - scenes.bsr_spmv_f64(rp, col, val, x)
    return np.linalg.norm(r) / np.linalg.norm(b)


@pytest.mark.parametrize("precond,precision", [("schwarz", "mixed"), ("schwarz", "fp32"), ("block", "mixed"),
                                               ("block", "fp32")])
@pytest.mark.parametrize("n", [1, 2, 5, 6, 37, 300, 620])
def test_grid_sizes(ctx, n, precond, precision):
    nb, rp, col, val = scenes.grid_bsr(n, seed=n)
    b = np.random.default_rng(n).standard_normal(3 * nb).astype(np.float32)
    assert solve_residual(ctx, nb, rp, col, val, precond, precision, b) <= 5e-6


def with_hubs(n, hubs, degree, seed=3):
    """A cloth-grid matrix whose first `hubs` vertices are also coupled to `degree` others each,
    kept symmetric and diagonally dominant."""
    nb, rp, col, val = scenes.grid_bsr(n, seed)
    rng = np.random.default_rng(seed)
    blocks = {}
    for v in range(nb):
        for k in range(rp[v], rp[v + 1]):
            blocks[(v, int(col[k]))] = val[k].astype(np.float64)
    for h in range(hubs):
        for w in rng.choice(np.arange(hubs, nb), degree, replace=False):
            m = 0.01 * rng.standard_normal((3, 3))
            blocks[(h, int(w))] = blocks.get((h, int(w)), 0) + m
            blocks[(int(w), h)] = blocks.get((int(w), h), 0) + m.T
            blocks[(h, h)] = blocks[(h, h)] + np.eye(3) * np.abs(m).sum()
            blocks[(int(w), int(w))] = blocks[(int(w), int(w))] + np.eye(3) * np.abs(m).sum()
    keys = sorted(blocks)
    rows = np.array([k[0] for k in keys])
    out_rp = np.zeros(nb + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=nb), out=out_rp[1:])
    return (nb, out_rp.astype(np.uint32), np.array([k[1] for k in keys], np.uint32),
            np.array([blocks[k] for k in keys], np.float32))


@pytest.mark.parametrize("hubs,degree", [(1, 300), (40, 60), (3, 3000)])
def test_long_rows_and_large_halos(ctx, hubs, degree):
    nb, rp, col, val = with_hubs(64, hubs, degree)
    b = np.random.default_rng(1).standard_normal(3 * nb).astype(np.float32)
    for precond in ("schwarz", "block"):
        assert solve_residual(ctx, nb, rp, col, val, precond, "mixed", b) <= 5e-6


def test_isolated_vertices(ctx):
    """Isolated vertices with b = 0 stay exactly 0; those with a load are solved."""
    nb0, rp0, col0, val0 = scenes.grid_bsr(20, 2)
    extra = 77
    nb = nb0 + extra
    rp = np.concatenate([rp0, rp0[-1] + 1 + np.arange(extra)]).astype(np.uint32)
    col = np.concatenate([col0, nb0 + np.arange(extra)]).astype(np.uint32)
    val = np.concatenate([val0, np.tile(2.0 * np.eye(3, dtype=np.float32), (extra, 1, 1))])
    b = np.random.default_rng(5).standard_normal((nb, 3)).astype(np.float32)
    b[nb0:nb0 + 40] = 0
    for precond in ("schwarz", "block"):
        assert solve_residual(ctx, nb, rp, col, val, precond, "mixed", b.reshape(-1)) <= 5e-6
        s = CudaLinearSolver(ctx, precond=precond)
        x = s.solve(CsrMatrix(*scenes.bsr_to_csr(nb, rp, col, val)), b.reshape(-1), 1e-6, 500).reshape(-1, 3)
        assert np.all(x[nb0:nb0 + 40] == 0)
        s.close()


def test_staged_fp16_domains_match_the_fused_kernels(ctx):
    """A 200 x 200 sheet in mixed precision: more domains per SM than shared memory holds, so
    rows and FP16 tiles are staged. Same step as the fused two-kernel PCG: the two solve to the
    same tolerance, positions within 1e-3 of the step's displacement as in the step tests."""
    sc = scenes.sheet_on_sphere(200, height=0.32)
    out = []
    for v in (0, 1):
        g = ImplicitSolver(ctx, dict(sc, params=dict(sc["params"], pcg_variant=v)), "mixed")
        st = g.step(1)[0]
        assert st["status"] == 0
        out.append((g.positions.astype(np.float64), st))
        g.close()
    disp = np.abs(out[0][0] - sc["positions"]).max()
    assert np.abs(out[0][0] - out[1][0]).max() <= 1e-3 * disp
    assert abs(out[0][1]["max_cg_iters"] - out[1][1]["max_cg_iters"]) <= 2


@pytest.mark.parametrize("precond", ["schwarz", "block"])
@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_non_finite_values_end_fp64_solves_as_fp32_ones(ctx, precond, bad):
    """FP64 sums take their FP32 operands' bits, which have no infinity or NaN: such rows go another
    way and the solve has to end where the FP32 one (plain conversions) does."""
    nb, rp, col, val = scenes.grid_bsr(12, 4)
    val = val.copy()
    v = 77  # an off-diagonal block, so that the diagonal stays what the preconditioner expects
    k = next(k for k in range(rp[v], rp[v + 1]) if col[k] != v)
    val[k, 1, 2] = bad
    a = CsrMatrix(*scenes.bsr_to_csr(nb, rp, col, val))
    b = np.random.default_rng(2).standard_normal(3 * nb).astype(np.float32)
    ends = []
    for precision in ("fp32", "mixed"):
        s = CudaLinearSolver(ctx, precond=precond, domain=32, precision=precision)
        try:
            x = s.solve(a, b, 1e-6, 500)
            ends.append((s.last_stats().status, s.last_stats().iters, np.isfinite(x).all()))
        except Exception as e:
            ends.append(type(e).__name__)
        s.close()
    assert ends[0] == ends[1]
