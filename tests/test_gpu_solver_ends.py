"""Solves at the ends of what their numbers can hold, through the linear-solver seam: where the sums
overflow or the matrix holds a NaN, the solve ends as the recurrences say it does."""
import os
import subprocess

import numpy as np
import pytest

from mguso import CsrMatrix, CudaLinearSolver, scenes

pytestmark = pytest.mark.gpu


def solve(ctx, nb, rp, col, val, b, precond, precision, max_iter=50):
    s = CudaLinearSolver(ctx, precond=precond, domain=32, precision=precision)
    x = s.solve(CsrMatrix(*scenes.bsr_to_csr(nb, rp, col, val)), b, 1e-6, max_iter)
    st = s.last_stats()
    s.close()
    return x, st


def test_overflowing_step_length(ctx):
    """Two coupled vertices whose r.z = 6 b^2 / d = 2.5e38 an FP32 sum holds and whose p.Ap = 1.9 r.z
    it does not: alpha = r.z / inf = 0, so x stays 0 up to the iteration limit. In mixed precision
    the sums fit and b, an eigenvector, is solved in one iteration."""
    d = np.float32(1e-10)
    eye = d * np.eye(3, dtype=np.float32)
    rp, col = np.array([0, 2, 4], np.uint32), np.array([0, 1, 0, 1], np.uint32)
    val = np.stack([eye, np.float32(0.9) * eye, np.float32(0.9) * eye, eye])
    b = np.full(6, 6.45e13, np.float32)
    x, st = solve(ctx, 2, rp, col, val, b, "block", "fp32")
    assert np.all(x == 0) and st.iters == 50 and st.status != 0 and st.residual == 1.0
    x, st = solve(ctx, 2, rp, col, val, b, "block", "mixed")
    assert st.status == 0 and st.iters == 1
    want = 6.45e13 / 1.9e-10
    assert np.abs(x - want).max() <= 1e-5 * want


@pytest.mark.parametrize("precond", ["schwarz", "block"])
@pytest.mark.parametrize("precision", ["fp32", "mixed"])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_isolated_vertex_with_a_non_finite_block(ctx, precond, precision, bad):
    """A vertex without neighbours and without a load whose block holds a NaN or an infinity: A p
    does too, p.Ap is not a number above zero and the solve breaks off before its first step."""
    nb0, rp0, col0, val0 = scenes.grid_bsr(12, 2)
    nb = nb0 + 3
    rp = np.concatenate([rp0, rp0[-1] + 1 + np.arange(3)]).astype(np.uint32)
    col = np.concatenate([col0, nb0 + np.arange(3)]).astype(np.uint32)
    val = np.concatenate([val0, np.tile(2 * np.eye(3, dtype=np.float32), (3, 1, 1))])
    val[-2, 0, 1] = bad
    b = np.random.default_rng(5).standard_normal((nb, 3)).astype(np.float32)
    b[nb0:] = 0
    x, st = solve(ctx, nb, rp, col, val, b.reshape(-1), precond, precision)
    assert st.iters == 0 and np.all(x == 0)


RECIP = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include "recip.cuh"
constexpr uint32_t N = 1u << 20;
__global__ void k(const double* v, double* r, double* q) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  r[i] = mg::recip(v[i]);
  q[i] = mg::quotient(3.0, v[i]);
}
int main() {
  double *v, *r, *q;
  if (cudaMallocManaged(&v, 8 * N) || cudaMallocManaged(&r, 8 * N) || cudaMallocManaged(&q, 8 * N)) return 2;
  uint64_t s = 1;
  for (uint32_t i = 0; i < N; ++i) {  // mantissas at random, exponents -1000 .. 999, both signs
    s = s * 6364136223846793005ull + 1442695040888963407ull;
    const uint64_t e = 23 + i % 2000, b = ((uint64_t)(i & 1) << 63) | (e << 52) | (s >> 12);
    memcpy(v + i, &b, 8);
  }
  const double ends[] = {INFINITY, -INFINITY, NAN};
  for (int i = 0; i < 3; ++i) v[N - 3 + i] = ends[i];
  k<<<N / 256, 256>>>(v, r, q);
  if (cudaDeviceSynchronize()) return 3;
  uint32_t bad = 0;
  for (uint32_t i = 0; i < N - 3; ++i) {
    const double w = 1.0 / v[i], u = nextafter(fabs(w), INFINITY) - fabs(w);
    if (!(fabs(r[i] - w) <= u)) ++bad;
    if (!(fabs(q[i] - 3.0 / v[i]) <= 4.45e-16 * fabs(3.0 / v[i]))) ++bad;
  }
  for (uint32_t i = N - 3; i < N; ++i) {
    const double w = 3.0 / v[i];
    if (std::isnan(w) ? !std::isnan(q[i]) : q[i] != w) ++bad;
  }
  printf("bad %u\n", bad);
  return bad != 0;
}
"""


def test_reciprocal_against_division(tmp_path):
    """The solver's reciprocal within a unit in the last place of the division over the range that it
    states, and its quotient (one rounding more: two units) also at the infinities."""
    src = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nguo-3d_b200", "csrc")
    (tmp_path / "r.cu").write_text(RECIP)
    exe = str(tmp_path / "r")
    subprocess.check_call(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", src, "-o", exe,
                           str(tmp_path / "r.cu")])
    assert subprocess.run([exe], capture_output=True, text=True).stdout.strip() == "bad 0"
