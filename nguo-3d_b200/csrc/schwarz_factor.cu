// Factorisation of the Schwarz domains (SchwarzTopology::factorize, linsolve.rs:177-240, and the
// coarse level of MultilevelSchwarz): per domain the dense block with the reference's diagonal
// floor 1e-6 (tr / m) + 1e-8, its Cholesky factor in FP64 (a pivot that is not above 1e-14
// falls back to the floored diagonal) and W = L^-1, stored as 32 x 32 tiles (tiles.cuh).
//
// One CTA of two warps per domain, the block in registers: thread (ti, tj) of an 8 x 8 grid holds
// the entries (ti + 8a, tj + 8b), b <= a, of the lower triangle. Factoring and inverting are one
// sweep of m steps over that triangle. Step k takes the pivot p = a_kk, and every row i > k
// loses (a_ik / p) times the vector v, where v_j is row k of the inverse so far for j < k, 1 for
// j = k and a_jk for j > k: to the right of column k that is the Schur complement, to its
// left the same elimination applied to the identity, so that after the last step row i holds
// sqrt(p_i) W_i. A step publishes v (the pivot's row and column) in shared memory, crosses
// one barrier and runs 78 (falling to 12) independent FP64 FMAs a thread.
//
// What bounds it: the m dependent steps (barrier, reciprocal, FMAs), with four domains sharing
// an SM. The kernel before this one (256 threads, 32-column panels in 75 KB of FP64 shared
// memory) waited at barriers while one warp factored the diagonal blocks and issued 13
// instructions per needed FMA. Before -> after: 32 768 domains of 96 rows 17.8 -> 2.58 ms, 4 100
// domains to FP16 tiles 2.30 -> 0.36 ms, 128 domains 147 -> 38 us, 2 500 domains of 48 rows
// 703 -> 45 us and their coarse level 214 -> 79 us. The block is cut over 64 threads and not
// more because a larger grid halves the FMAs per published value; 78 doubles a thread still fit
// its registers. Smaller domains use a smaller NB.
#include <algorithm>

#include "internal.cuh"
#include "recip.cuh"
#include "tiles.cuh"

namespace mg {

constexpr int FC_THREADS = 64;

template <class TS>
__device__ __forceinline__ TS to_tile(double v) {
  return (TS)v;
}
template <>
__device__ __forceinline__ __half to_tile<__half>(double v) {
  return __float2half_rn((float)v);
}

// leading dimension of the FP32 block in shared memory: 8 mod 32, so that the 4 x 8 entries a
// warp reads at once fall into distinct banks
template <int NB>
__host__ __device__ constexpr int fc_ld() {
  return (8 * NB + 23) / 32 * 32 + 8;
}
// shared memory: the block, reused for the finished tiles
template <int NB>
__host__ __device__ constexpr int fc_smem_bytes() {
  constexpr int T = (8 * NB + 31) / 32;
  constexpr int block = 8 * NB * fc_ld<NB>() * 4, tiles = T * (T + 1) / 2 * TILE_FLOATS * 4;
  return block > tiles ? block : tiles;
}

__device__ __forceinline__ double fc_block_sum(double v, double* s2) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) s2[threadIdx.x >> 5] = v;
  __syncthreads();
  v = s2[0] + s2[1];
  __syncthreads();
  return v;
}
__device__ __forceinline__ double fc_block_max(double v, double* s2) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) s2[threadIdx.x >> 5] = v;
  __syncthreads();
  v = fmax(s2[0], s2[1]);
  __syncthreads();
  return v;
}

// The m x m block in `sm` (FP32, leading dimension fc_ld<NB>(), lower triangle) factored, inverted
// and stored at `out` (FP16 tiles: W / scale with the domain's largest |W| in *scale_out).
template <int NB, class TS>
__device__ void fc_factor_store(float* sm, int m, TS* __restrict__ out, float* scale_out, uint32_t* status) {
  constexpr bool scaled = sizeof(TS) == 2;
  constexpr int LD = fc_ld<NB>(), M = 8 * NB;
  __shared__ double s_v[2][M], s_piv[M], s_two[2];
  const int tid = threadIdx.x, ti = tid >> 3, tj = tid & 7;
  double tr = 0.0;
  for (int k = tid; k < m; k += FC_THREADS) tr += (double)sm[k * LD + k];
  const double floor_ = 1e-6 * (fc_block_sum(tr, s_two) / (double)m) + 1e-8;

  double e[NB * (NB + 1) / 2];  // (a, b) at a (a + 1) / 2 + b
#pragma unroll
  for (int a = 0; a < NB; ++a)
#pragma unroll
    for (int b = 0; b <= a; ++b) {
      const int i = ti + 8 * a, j = tj + 8 * b;
      double v = (i < m && j <= i) ? (double)sm[i * LD + j] : 0.0;
      if (i == j && i < m) v += floor_;
      e[a * (a + 1) / 2 + b] = v;
    }

  bool fail = false;
#pragma unroll
  for (int kb = 0; kb < NB; ++kb) {
    for (int kk = 0; kk < 8; ++kk) {
      const int k = 8 * kb + kk;
      if (k >= m || fail) break;  // uniform
      double* v = s_v[k & 1];
      if (tj == kk) {
#pragma unroll
        for (int a = kb; a < NB; ++a)
          if (a > kb || ti >= kk) v[ti + 8 * a] = e[a * (a + 1) / 2 + kb];
      }
      if (ti == kk) {
#pragma unroll
        for (int b = 0; b <= kb; ++b)
          if (b < kb || tj < kk) v[tj + 8 * b] = e[kb * (kb + 1) / 2 + b];
      }
      __syncthreads();
      const double p = v[k];
      if (!(p > 1e-14)) {
        fail = true;
        break;
      }
      if (tid == 0) s_piv[k] = p;
      const double w = recip(p);  // p > 1e-14; an infinite one fails the next pivot's test
      double u[NB];
#pragma unroll
      for (int b = 0; b < NB; ++b) u[b] = v[tj + 8 * b];
      const bool own = tj == kk;
      if (own) u[kb] = 1.0;
#pragma unroll
      for (int a = kb; a < NB; ++a) {
        if (a > kb || ti > kk) {
          const double mi = -(v[ti + 8 * a] * w);
#pragma unroll
          for (int b = 0; b <= a; ++b) {
            double& x = e[a * (a + 1) / 2 + b];
            x = fma(mi, u[b], (b == kb && own) ? 0.0 : x);
          }
        }
      }
    }
  }
  __syncthreads();
  // row scales 1 / sqrt(p_i), or the reference's fallback L = diag(sqrt(ad_pp)) (1 where
  // ad_pp <= 1e-14)
  double mx = 0.0;
  for (int k = tid; k < M; k += FC_THREADS) {
    double s = 0.0;
    if (k < m) {
      if (!fail) {
        s = rsqrt(s_piv[k]);
      } else {
        const double d = (double)sm[k * LD + k] + floor_;
        s = d > 1e-14 ? 1.0 / sqrt(d) : 1.0;
      }
    }
    s_v[0][k] = s;
    mx = fmax(mx, s);
  }
  __syncthreads();
#pragma unroll
  for (int a = 0; a < NB; ++a) {
    const double s = s_v[0][ti + 8 * a];
#pragma unroll
    for (int b = 0; b <= a; ++b) {
      double& x = e[a * (a + 1) / 2 + b];
      const int i = ti + 8 * a, j = tj + 8 * b;
      x = i == j ? s : ((fail || j > i) ? 0.0 : x * s);
      if (scaled) mx = fmax(mx, fabs(x));
    }
  }
  double inv = 1.0;
  if (scaled) {
    mx = fc_block_max(mx, s_two);
    inv = 1.0 / (mx > 0.0 ? mx : 1.0);
    if (tid == 0) *scale_out = (float)(1.0 / inv);
  }
  if (fail && tid == 0) atomicOr(status, 1u << 8);
  // tiles in shared memory (the block's place), then out in whole 16-byte units
  const int T = (m + 31) >> 5, nt16 = T * (T + 1) / 2 * TILE_FLOATS * (int)sizeof(TS) / 16;
  uint4* t16 = reinterpret_cast<uint4*>(sm);
  __syncthreads();
  for (int i = tid; i < nt16; i += FC_THREADS) t16[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  TS* tiles = reinterpret_cast<TS*>(sm);
#pragma unroll
  for (int a = 0; a < NB; ++a)
#pragma unroll
    for (int b = 0; b <= a; ++b) {
      const int i = ti + 8 * a, j = tj + 8 * b;
      if (i < m && j <= i)
        tiles[tile_index(a >> 2, b >> 2) * TILE_FLOATS + tile_off<TS>(i & 31, j & 31)] =
            to_tile<TS>(e[a * (a + 1) / 2 + b] * inv);
    }
  __syncthreads();
  uint4* o16 = reinterpret_cast<uint4*>(out);
  for (int i = tid; i < nt16; i += FC_THREADS) o16[i] = t16[i];
}

// One vertex as its own domain (m = 3): the reference's floor 1e-6 (tr / 3) + 1e-8 on the
// diagonal, the row-by-row Cholesky with its pivot test (linsolve.rs:80-99; a failed pivot
// falls back to L = diag(sqrt(a_pp)), 1 where a_pp <= 1e-14), and W = L^-1 stored as its
// lower triangle (w00 w10 w11 w20 w21 w22).
__device__ void vertex_factor(double* a, float* __restrict__ w6, uint32_t* status) {
  const double fl = 1e-6 * ((a[0] + a[4] + a[8]) / 3.0) + 1e-8;
  a[0] += fl;
  a[4] += fl;
  a[8] += fl;
  double l[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  bool ok = true;
  for (int i = 0; i < 3 && ok; ++i)
    for (int j = 0; j <= i; ++j) {
      double sum = a[3 * i + j];
      for (int k = 0; k < j; ++k) sum -= l[3 * i + k] * l[3 * j + k];
      if (i == j) {
        if (!(sum > 1e-14)) {
          ok = false;
          break;
        }
        l[3 * i + i] = sqrt(sum);
      } else {
        l[3 * i + j] = sum / l[3 * j + j];
      }
    }
  if (!ok) {
    for (int e = 0; e < 9; ++e) l[e] = 0.0;
    for (int p = 0; p < 3; ++p) l[4 * p] = a[4 * p] > 1e-14 ? sqrt(a[4 * p]) : 1.0;
    atomicOr(status, 1u << 8);
  }
  const double w00 = 1.0 / l[0], w11 = 1.0 / l[4], w22 = 1.0 / l[8];
  const double w10 = -l[3] * w00 * w11;
  const double w21 = -l[7] * w11 * w22;
  const double w20 = -(l[6] * w00 + l[7] * w10) * w22;
  w6[0] = (float)w00;
  w6[1] = (float)w10;
  w6[2] = (float)w11;
  w6[3] = (float)w20;
  w6[4] = (float)w21;
  w6[5] = (float)w22;
}

struct FactorArgs {
  const uint32_t *row_ptr, *col;
  const float* val;
  const uint32_t *c_rp, *c_col;  // blocks outside the pattern (null: none)
  const float* c_val;
  const uint32_t *dom_start, *dom_verts, *vpos;
  const uint64_t* fac_off;
  void* fac;
  float* fac_scale;
  const uint8_t *dom_diag, *dom_inst;
  float* vfac;
  uint32_t active;
  uint32_t* status;
};

template <int NB, class TS>
__global__ void __launch_bounds__(FC_THREADS) k_schwarz_factor(const __grid_constant__ FactorArgs f) {
  extern __shared__ __align__(16) float fc_sm[];
  constexpr int LD = fc_ld<NB>();
  __shared__ uint32_t s_k0[32], s_nps[32], s_c0[32], s_pre[33];
  const uint32_t d = blockIdx.x;
  if (!((f.active >> f.dom_inst[d]) & 1u)) return;  // an instance the batch no longer iterates
  const uint32_t vs = f.dom_start[d], nvd = f.dom_start[d + 1] - vs;
  const int tid = threadIdx.x;
  if (f.dom_diag[d]) {
    for (uint32_t p = tid; p < nvd; p += FC_THREADS) {
      const uint32_t v = f.dom_verts[vs + p];
      double A9[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
      for (uint32_t k = f.row_ptr[v]; k < f.row_ptr[v + 1]; ++k)
        if (f.col[k] == v)
          for (int e = 0; e < 9; ++e) A9[e] = (double)f.val[9 * (size_t)k + e];
      vertex_factor(A9, f.vfac + 6 * (size_t)v, f.status);
    }
    return;
  }
  const int m = 3 * (int)nvd;
  for (int i = tid; i < m * LD; i += FC_THREADS) fc_sm[i] = 0.f;
  // the rows' blocks as one list (pattern, then contact blocks of each row), four at a time per
  // thread so that the chains column -> position -> values of several blocks overlap
  if (tid < 32) {
    uint32_t len = 0;
    if ((uint32_t)tid < nvd) {
      const uint32_t v = f.dom_verts[vs + tid];
      s_k0[tid] = f.row_ptr[v];
      s_nps[tid] = f.row_ptr[v + 1] - s_k0[tid];
      s_c0[tid] = f.c_rp ? f.c_rp[v] : 0u;
      len = s_nps[tid] + (f.c_rp ? f.c_rp[v + 1] - s_c0[tid] : 0u);
    }
    uint32_t incl = len;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (tid >= o) incl += t;
    }
    s_pre[tid + 1] = incl;
    if (tid == 0) s_pre[0] = 0;
  }
  __syncthreads();
  const uint32_t total = s_pre[32];
  for (uint32_t t0 = tid; t0 < total; t0 += 4 * FC_THREADS) {
    uint32_t row[4], pos[4];
    const float* src[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t t = t0 + u * FC_THREADS;
      row[u] = 0;
      pos[u] = 0xffffffffu;
      src[u] = nullptr;
      if (t < total) {
        uint32_t p = 0;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1)
          if (s_pre[p + s] <= t) p += s;
        const uint32_t sj = t - s_pre[p];
        const bool ps = sj < s_nps[p];
        const size_t k = ps ? s_k0[p] + sj : s_c0[p] + (sj - s_nps[p]);
        row[u] = p;
        pos[u] = f.vpos[ps ? f.col[k] : f.c_col[k]];
        src[u] = (ps ? f.val : f.c_val) + 9 * k;
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t q = pos[u] - vs;
      if (src[u] && q <= row[u]) {  // inside the domain, lower triangle
        float* o = fc_sm + 3 * row[u] * LD + 3 * q;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) o[i * LD + j] = src[u][3 * i + j];
      }
    }
  }
  __syncthreads();
  fc_factor_store<NB, TS>(fc_sm, m, (TS*)f.fac + f.fac_off[d], f.fac_scale ? f.fac_scale + d : nullptr, f.status);
}

struct CoarseArgs {
  const uint32_t *row_ptr, *col;
  const float* val;
  const uint32_t *c_rp, *c_col;
  const float* c_val;
  const uint32_t *dom_start, *dom_sorted, *cdom_start, *cdom_nodes;
  const uint2* cplace;
  const uint64_t* cfac_off;
  float* cfac;
  uint32_t* status;
};

// Coarse factorisation of the two-level form, one CTA per coarse domain: thread t owns
// row t = 3a + r of the domain's dense Galerkin block (coarse node a, component r) and adds,
// for every vertex i of node a in ascending order and every block (i, j) of the pattern and
// of the contact matrix in column order whose column vertex lies in this coarse domain, the
// block's row r. The sums run in FP32, entry by entry in the order of the fine values, as
// the reference's coarse_matrix does (linsolve.rs:618-630); rows without contact blocks read
// eight blocks at a time so that their look-ups overlap. What bounds the rows is the chain of
// loads per vertex: the next vertex's runs are read a vertex ahead, and a column's coarse place is
// one load (cplace) instead of three. 200 x 200 grid, 16-vertex domains: 81 -> 59 us. The block
// is then factored and stored like a level-0 domain.
template <int NB>
__global__ void __launch_bounds__(FC_THREADS) k_coarse_factor(const __grid_constant__ CoarseArgs f) {
  extern __shared__ __align__(16) float fc_sm[];
  constexpr int LD = fc_ld<NB>();
  const uint32_t d1 = blockIdx.x;
  const uint32_t n0 = f.cdom_start[d1], mn = f.cdom_start[d1 + 1] - n0;
  const int m = 3 * (int)mn, tid = threadIdx.x;
  for (int i = tid; i < m * LD; i += FC_THREADS) fc_sm[i] = 0.f;
  __syncthreads();
  for (int t = tid; t < m; t += FC_THREADS) {
    const int a = t / 3, r = t - 3 * a;
    const uint32_t g = f.cdom_nodes[n0 + a];
    float* row = fc_sm + (size_t)t * LD;
    const uint32_t p1 = f.dom_start[g + 1];
    uint32_t n1 = 0, ne1 = 0, n2 = 0, ne2 = 0;  // the next vertex's runs, read a vertex ahead
    auto runs = [&](uint32_t p) {
      if (p >= p1) return;
      const uint32_t i = f.dom_sorted[p];
      n1 = f.row_ptr[i];
      ne1 = f.row_ptr[i + 1];
      if (f.c_rp) {
        n2 = f.c_rp[i];
        ne2 = f.c_rp[i + 1];
      }
    };
    runs(f.dom_start[g]);
    for (uint32_t p = f.dom_start[g]; p < p1; ++p) {
      uint32_t k1 = n1, k2 = n2;
      const uint32_t e1 = ne1, e2 = ne2;
      runs(p + 1);
      if (k2 == e2) {
        for (; k1 < e1; k1 += 8) {
          int q[8];
          float b0[8], b1[8], b2[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            q[u] = -1;
            if (k1 + u < e1) {
              const uint2 at = f.cplace[f.col[k1 + u]];
              const float* b = f.val + 9 * (size_t)(k1 + u) + 3 * r;
              b0[u] = b[0];
              b1[u] = b[1];
              b2[u] = b[2];
              if (at.x == d1) q[u] = 3 * (int)at.y;
            }
          }
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (q[u] >= 0) {
              row[q[u]] += b0[u];
              row[q[u] + 1] += b1[u];
              row[q[u] + 2] += b2[u];
            }
        }
        continue;
      }
      while (k1 < e1 || k2 < e2) {
        const bool from_c = k1 >= e1 || (k2 < e2 && f.c_col[k2] < f.col[k1]);
        const uint32_t j = from_c ? f.c_col[k2] : f.col[k1];
        const float* b = from_c ? f.c_val + 9 * (size_t)k2++ : f.val + 9 * (size_t)k1++;
        const uint2 at = f.cplace[j];
        if (at.x != d1) continue;
        const int q = 3 * (int)at.y;
#pragma unroll
        for (int c = 0; c < 3; ++c) row[q + c] = row[q + c] + b[3 * r + c];
      }
    }
  }
  __syncthreads();
  fc_factor_store<NB, float>(fc_sm, m, f.cfac + f.cfac_off[d1], nullptr, f.status);
}

template <int NB>
static int launch_factor(const mguso_schwarz* s, const FactorArgs& f, cudaStream_t st) {
  if (s->half)
    k_schwarz_factor<NB, __half><<<s->ndom, FC_THREADS, fc_smem_bytes<NB>(), st>>>(f);
  else
    k_schwarz_factor<NB, float><<<s->ndom, FC_THREADS, fc_smem_bytes<NB>(), st>>>(f);
  MG_CUDA(cudaGetLastError());
  return MGUSO_OK;
}
template <int NB>
static int launch_coarse(const mguso_schwarz* s, const CoarseArgs& f, cudaStream_t st) {
  k_coarse_factor<NB><<<s->ncdom, FC_THREADS, fc_smem_bytes<NB>(), st>>>(f);
  MG_CUDA(cudaGetLastError());
  return MGUSO_OK;
}

int schwarz_factor_with(mguso_schwarz* s, const uint32_t* c_rp, const uint32_t* c_col, const float* c_val,
                        cudaStream_t st) {
  if (s->ndom == 0) return MGUSO_OK;
  mguso_bsr* a = s->a;
  FactorArgs f{};
  f.row_ptr = a->row_ptr.p;
  f.col = a->col.p;
  f.val = a->val.p;
  f.c_rp = c_col ? c_rp : nullptr;
  f.c_col = c_col;
  f.c_val = c_val;
  f.dom_start = s->dom_start.p;
  f.dom_verts = s->dom_verts.p;
  f.vpos = s->vpos.p;
  f.fac_off = s->fac_off.p;
  f.fac = s->half ? (void*)s->fac_h.p : (void*)s->fac.p;
  f.fac_scale = s->half ? s->fac_scale.p : nullptr;
  f.dom_diag = s->dom_diag.p;
  f.dom_inst = s->dom_inst.p;
  f.vfac = s->vfac.p;
  f.active = s->active;
  f.status = s->status.p;
  // the smallest register block that holds the largest domain (24, 48, 72 or 96 rows)
  const uint32_t m = s->max_m;
  MG_TRY(m <= 24 ? launch_factor<3>(s, f, st)
                 : m <= 48 ? launch_factor<6>(s, f, st) : m <= 72 ? launch_factor<9>(s, f, st) : launch_factor<12>(s, f, st));
  if (s->levels == 2 && s->ncdom) {
    CoarseArgs g{};
    g.row_ptr = f.row_ptr;
    g.col = f.col;
    g.val = f.val;
    g.c_rp = f.c_rp;
    g.c_col = f.c_col;
    g.c_val = f.c_val;
    g.dom_start = f.dom_start;
    g.dom_sorted = s->dom_sorted.p;
    g.cdom_start = s->cdom_start.p;
    g.cdom_nodes = s->cdom_nodes.p;
    g.cplace = s->cplace.p;
    g.cfac_off = s->cfac_off.p;
    g.cfac = s->cfac.p;
    g.status = s->status.p;
    const uint32_t m1 = s->max_m1;
    MG_TRY(m1 <= 24 ? launch_coarse<3>(s, g, st)
                    : m1 <= 48 ? launch_coarse<6>(s, g, st) : m1 <= 72 ? launch_coarse<9>(s, g, st) : launch_coarse<12>(s, g, st));
  }
  return MGUSO_OK;
}

int schwarz_factor(mguso_schwarz* s, cudaStream_t st) {
  return schwarz_factor_with(s, nullptr, nullptr, nullptr, st);
}

}  // namespace mg
