// One-level additive Schwarz preconditioner and 3x3 block Jacobi on the GPU.
//
// Reference: SchwarzTopology::{build, factorize, apply} (engine-core/src/linsolve.rs:
// 126-258): greedy BFS domains of <= D vertices over the block graph, per-domain dense
// block with the diagonal floor 1e-6*(tr/m) + 1e-8, Cholesky in f64 (fallback to the
// diagonal when a pivot is <= 1e-14), and z = (L L^T)^-1 r per domain.
//
// B200 layout: the factorisation (schwarz_factor.cu) stores W = L^-1 in FP32 as swizzled 32 x 32
// tiles of its lower block-triangle (4 KB aligned per tile), so that the FP32 preconditioner
// W~^T W~ is symmetric positive definite for any rounding of W. (An explicitly stored FP32
// inverse is not: with stiff seams a domain block reaches a condition number near 1e7 and
// rounding the inverse to FP32 can make it indefinite.) The apply is two dense triangular
// matvecs per domain, z = W^T (W r), with no sequential triangular sweeps: one warp per
// domain stages its tiles into shared memory with a single 1-D TMA bulk copy.
#include <algorithm>
#include <deque>

#include "reduce.cuh"
#include "tiles.cuh"

namespace mg {

int schwarz_configure();
int schwarz_build_coarse(mguso_schwarz* s);
// ---------------------------------------------------------------------------------------
// Host: BFS domains over the block pattern (linsolve.rs:152-173).
// ---------------------------------------------------------------------------------------
int schwarz_build(mguso_schwarz* s) {
  mguso_bsr* a = s->a;
  uint32_t nb = a->nb;
  const auto& rp = a->h_row_ptr;
  const auto& cl = a->h_col;
  std::vector<uint8_t> assigned(nb, 0);
  s->h_dom_start.assign(1, 0);
  s->h_dom_verts.clear();
  s->h_dom_verts.reserve(nb);
  s->h_dom_of.assign(nb, 0);
  uint32_t D = std::max<uint32_t>(s->domain, 1);
  uint32_t max_m = 0;
  // Vertices with no off-diagonal block (pinned collider vertices, unconnected points)
  // would each be a one-vertex domain; they are packed D at a time instead. Their blocks
  // do not couple, so the packed domain's factor is block diagonal and the preconditioner
  // is unchanged (only the diagonal floor averages over the packed vertices).
  std::vector<uint32_t> singles;
  for (uint32_t v = 0; v < nb && s->pack_singles; ++v) {
    bool iso = true;
    for (uint32_t k = rp[v]; k < rp[v + 1] && iso; ++k) iso = cl[k] == v;
    if (iso) {
      singles.push_back(v);
      assigned[v] = 1;
    }
  }
  s->h_dom_diag.clear();
  auto close_domain = [&](size_t base, bool diag = false) {
    uint32_t d = (uint32_t)s->h_dom_start.size() - 1;
    s->h_dom_diag.push_back(diag ? 1 : 0);
    for (size_t i = base; i < s->h_dom_verts.size(); ++i) s->h_dom_of[s->h_dom_verts[i]] = d;
    s->h_dom_start.push_back((uint32_t)s->h_dom_verts.size());
    max_m = std::max<uint32_t>(max_m, 3 * (uint32_t)(s->h_dom_verts.size() - base));
  };
  // instance by instance (vertex ranges; one range for a single scene), so that each
  // domain lies in one instance and the domains of an instance are contiguous
  std::vector<uint32_t> ranges = s->inst_vert;
  if (ranges.size() < 2) ranges = {0, nb};
  size_t si = 0;
  for (size_t r = 0; r + 1 < ranges.size(); ++r) {
  for (uint32_t seed = ranges[r]; seed < ranges[r + 1]; ++seed) {
    if (assigned[seed]) continue;
    size_t base = s->h_dom_verts.size();
    s->h_dom_verts.push_back(seed);
    assigned[seed] = 1;
    size_t fi = base;
    while (s->h_dom_verts.size() - base < D && fi < s->h_dom_verts.size()) {
      uint32_t v = s->h_dom_verts[fi++];
      // block columns are sorted and unique per row: the reference's sorted, deduped
      // adjacency minus the vertex itself.
      for (uint32_t k = rp[v]; k < rp[v + 1]; ++k) {
        uint32_t nbv = cl[k];
        if (nbv == v) continue;
        if (!assigned[nbv] && s->h_dom_verts.size() - base < D) {
          assigned[nbv] = 1;
          s->h_dom_verts.push_back(nbv);
        }
      }
    }
    close_domain(base);
  }
  // this instance's isolated vertices, D per domain
  size_t se = si;
  while (se < singles.size() && singles[se] < ranges[r + 1]) ++se;
  for (size_t i = si; i < se; i += D) {
    size_t base = s->h_dom_verts.size();
    for (size_t j = i; j < std::min(se, i + D); ++j) s->h_dom_verts.push_back(singles[j]);
    close_domain(base, true);
  }
  si = se;
  }
  s->ndom = (uint32_t)s->h_dom_start.size() - 1;
  s->max_m = max_m;
  std::vector<uint64_t> off(s->ndom + 1, 0);
  for (uint32_t d = 0; d < s->ndom; ++d) {
    uint64_t m = 3ull * (s->h_dom_start[d + 1] - s->h_dom_start[d]);
    uint64_t t = s->h_dom_diag[d] ? 0 : (m + 31) / 32;
    off[d + 1] = off[d] + t * (t + 1) / 2 * TILE_FLOATS;
  }
  s->fac_floats = off[s->ndom];
  MG_TRY(s->dom_diag.upload(s->h_dom_diag.data(), std::max<size_t>(s->h_dom_diag.size(), 1), a->ctx->stream));
  // each domain's instance (the range of its first vertex), for factorisations that skip
  // the instances a batch no longer iterates
  std::vector<uint8_t> dom_inst(std::max<uint32_t>(s->ndom, 1), 0);
  for (uint32_t d = 0; d < s->ndom; ++d) {
    const uint32_t v = s->h_dom_verts[s->h_dom_start[d]];
    dom_inst[d] = (uint8_t)(std::upper_bound(ranges.begin(), ranges.end(), v) - ranges.begin() - 1);
  }
  MG_TRY(s->dom_inst.upload(dom_inst.data(), dom_inst.size(), a->ctx->stream));
  MG_TRY(s->vfac.reserve(6 * (size_t)std::max<uint32_t>(nb, 1)));
  cudaStream_t st = a->ctx->stream;
  MG_TRY(s->dom_start.upload(s->h_dom_start.data(), s->h_dom_start.size(), st));
  MG_TRY(s->dom_verts.upload(s->h_dom_verts.data(), s->h_dom_verts.size(), st));
  MG_TRY(s->dom_of.upload(s->h_dom_of.data(), nb, st));
  std::vector<uint32_t> vpos(nb, 0);
  for (uint32_t i = 0; i < (uint32_t)s->h_dom_verts.size(); ++i) vpos[s->h_dom_verts[i]] = i;
  MG_TRY(s->vpos.upload(vpos.data(), nb, st));
  MG_TRY(s->fac_off.upload(off.data(), off.size(), st));
  if (s->half) {
    MG_TRY(s->fac_h.reserve(std::max<uint64_t>(s->fac_floats, 8)));
    MG_TRY(s->fac_scale.reserve(std::max<uint32_t>(s->ndom, 1)));
  } else {
    MG_TRY(s->fac.reserve(std::max<uint64_t>(s->fac_floats, 4)));
  }
  MG_TRY(s->status.reserve(4));
  MG_CUDA(cudaMemsetAsync(s->status.p, 0, 16, st));
  if (s->levels == 2) MG_TRY(schwarz_build_coarse(s));
  MG_CUDA(cudaStreamSynchronize(st));
  MG_TRY(schwarz_configure());
  return MGUSO_OK;
}

// Coarse level of the two-level form (MultilevelSchwarz::build, linsolve.rs:555-608): coarse
// node G = level-0 domain G; G and H are adjacent when some block (i, j) of the pattern has
// i in G and j in H; coarse domains are the reference's greedy BFS over that adjacency
// (seeds in node order, neighbours in ascending order, <= domain nodes each).
int schwarz_build_coarse(mguso_schwarz* s) {
  mguso_bsr* a = s->a;
  const uint32_t nb = a->nb, nd = s->ndom;
  const auto& rp = a->h_row_ptr;
  const auto& cl = a->h_col;
  std::vector<std::vector<uint32_t>> adj(nd);
  for (uint32_t v = 0; v < nb; ++v) {
    const uint32_t g = s->h_dom_of[v];
    for (uint32_t k = rp[v]; k < rp[v + 1]; ++k) {
      const uint32_t h = s->h_dom_of[cl[k]];
      if (h != g) adj[g].push_back(h);
    }
  }
  for (auto& x : adj) {
    std::sort(x.begin(), x.end());
    x.erase(std::unique(x.begin(), x.end()), x.end());
  }
  const uint32_t D = std::max<uint32_t>(s->domain, 1);
  std::vector<uint8_t> assigned(nd, 0);
  std::vector<uint32_t> cdom_of(nd, 0), cloc(nd, 0);
  s->h_cdom_start.assign(1, 0);
  s->h_cdom_nodes.clear();
  s->max_m1 = 0;
  for (uint32_t seed = 0; seed < nd; ++seed) {
    if (assigned[seed]) continue;
    const size_t base = s->h_cdom_nodes.size();
    s->h_cdom_nodes.push_back(seed);
    assigned[seed] = 1;
    size_t fi = base;
    while (s->h_cdom_nodes.size() - base < D && fi < s->h_cdom_nodes.size()) {
      const uint32_t g = s->h_cdom_nodes[fi++];
      for (uint32_t h : adj[g])
        if (!assigned[h] && s->h_cdom_nodes.size() - base < D) {
          assigned[h] = 1;
          s->h_cdom_nodes.push_back(h);
        }
    }
    const uint32_t d1 = (uint32_t)s->h_cdom_start.size() - 1;
    for (size_t i = base; i < s->h_cdom_nodes.size(); ++i) {
      cdom_of[s->h_cdom_nodes[i]] = d1;
      cloc[s->h_cdom_nodes[i]] = (uint32_t)(i - base);
    }
    s->h_cdom_start.push_back((uint32_t)s->h_cdom_nodes.size());
    s->max_m1 = std::max<uint32_t>(s->max_m1, 3 * (uint32_t)(s->h_cdom_nodes.size() - base));
  }
  s->ncdom = (uint32_t)s->h_cdom_start.size() - 1;
  std::vector<uint64_t> off(s->ncdom + 1, 0);
  for (uint32_t d = 0; d < s->ncdom; ++d) {
    const uint64_t m = 3ull * (s->h_cdom_start[d + 1] - s->h_cdom_start[d]);
    const uint64_t t = (m + 31) / 32;
    off[d + 1] = off[d] + t * (t + 1) / 2 * TILE_FLOATS;
  }
  std::vector<uint32_t> sorted(s->h_dom_verts);
  for (uint32_t d = 0; d < nd; ++d)
    std::sort(sorted.begin() + s->h_dom_start[d], sorted.begin() + s->h_dom_start[d + 1]);
  cudaStream_t st = a->ctx->stream;
  MG_TRY(s->cdom_start.upload(s->h_cdom_start.data(), s->h_cdom_start.size(), st));
  MG_TRY(s->cdom_nodes.upload(s->h_cdom_nodes.data(), std::max<size_t>(s->h_cdom_nodes.size(), 1), st));
  std::vector<uint2> place(std::max<uint32_t>(a->nb, 1));
  for (uint32_t v = 0; v < a->nb; ++v) place[v] = make_uint2(cdom_of[s->h_dom_of[v]], cloc[s->h_dom_of[v]]);
  MG_TRY(s->cplace.upload(place.data(), place.size(), st));
  MG_TRY(s->dom_sorted.upload(sorted.data(), std::max<size_t>(sorted.size(), 1), st));
  MG_TRY(s->cfac_off.upload(off.data(), off.size(), st));
  MG_TRY(s->cfac.reserve(std::max<uint64_t>(off[s->ncdom], 4)));
  MG_TRY(s->ec.reserve(std::max<uint64_t>(3ull * nd, 4)));
  MG_CUDA(cudaStreamSynchronize(st));
  return MGUSO_OK;
}

// ---------------------------------------------------------------------------------------
// Apply: one warp per domain (grid-stride over domains). The warp bulk-copies its domain's
// W tiles into its shared slice, gathers r, then
//   pass 1: y = W r    lane = row within a row tile, loop over columns c;
//   pass 2: z = W^T y  lane = column within a column tile, loop over rows r.
// The FP32 tile layout (c*32 + (r ^ c)) makes both passes free of bank conflicts. Every
// lane carries one accumulator per tile row/column (<= 3), so there are no long serial
// chains. Acc = double (mixed precision) accumulates in FP64.
// ---------------------------------------------------------------------------------------
constexpr int APPLY_WARPS = 4;

template <int WARPS, class Acc, class TS>
__global__ void __launch_bounds__(32 * WARPS) k_schwarz_apply(
    const uint32_t* __restrict__ dom_start, const uint32_t* __restrict__ dom_verts,
    const uint64_t* __restrict__ fac_off, const TS* __restrict__ fac, const float* __restrict__ fac_scale,
    const float* __restrict__ r, float* __restrict__ z, uint32_t ndom, uint32_t* status, DotSink dot, int with_dot,
    const uint8_t* __restrict__ dom_diag, const float* __restrict__ vfac) {
  extern __shared__ __align__(128) unsigned char smem[];
  if (with_dot && dot.sc->done) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint64_t* bar = (uint64_t*)(smem + 16 * w);
  TS* buf = (TS*)(smem + 128 + (size_t)w * apply_slice_bytes<TS>());
  float* rd = (float*)(buf + 6 * TILE_FLOATS);
  Acc* yd = (Acc*)(rd + 96);
  Acc acc = 0;
  if (lane == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  __syncwarp();
  uint32_t phase = 0;
  for (uint32_t d = blockIdx.x * WARPS + w; d < ndom; d += gridDim.x * WARPS) {
    const uint32_t vs = dom_start[d], nvd = dom_start[d + 1] - vs;
    const int m = 3 * (int)nvd;
    const uint64_t off = fac_off[d];
    const uint32_t bytes = (uint32_t)((fac_off[d + 1] - off) * sizeof(TS));
    const bool diag = dom_diag[d] != 0;
    if (lane == 0 && !diag) {
      fence_proxy_async();
      mbar_arrive_expect_tx(bar, bytes);
      bulk_g2s(buf, fac + off, bytes, bar);
    }
    for (int i = lane; i < 96; i += 32) {
      float v = 0.f;
      if (i < m) v = r[3 * dom_verts[vs + i / 3] + i % 3];
      rd[i] = v;
    }
    __syncwarp();
    if (diag) {
      if (lane < (int)nvd) {
        const uint32_t v = dom_verts[vs + lane];
        Acc zz[3];
        vertex_apply<Acc>(vfac + 6 * (size_t)v, rd + 3 * lane, zz);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float zi = (float)zz[c];
          z[3 * v + c] = zi;
          acc += (Acc)rd[3 * lane + c] * (Acc)zi;
        }
      }
      __syncwarp();
      continue;
    }
    if (!mbar_wait(bar, phase)) {
      if (lane == 0) atomicOr(status, ST_WAIT_TIMEOUT);
      mbar_wait(bar, phase);  // the copy may still land: bounded second wait, then stop
      break;
    }
    phase ^= 1;
    Acc zz[3];
    const int T = (m + 31) >> 5;
    if (T == 3)
      tiles_apply<3, Acc, TS>(buf, rd, yd, zz, lane);
    else if (T == 2)
      tiles_apply<2, Acc, TS>(buf, rd, yd, zz, lane);
    else
      tiles_apply<1, Acc, TS>(buf, rd, yd, zz, lane);
    const Acc sc = fac_scale ? (Acc)fac_scale[d] : (Acc)1;
#pragma unroll
    for (int J = 0; J < 3; ++J) {
      const int i = 32 * J + lane;
      if (i < m) {
        const float zi = (float)(zz[J] * sc * sc);
        z[3 * dom_verts[vs + i / 3] + i % 3] = zi;
        acc += (Acc)rd[i] * (Acc)zi;
      }
    }
    __syncwarp();  // every lane is done with buf before the next copy overwrites it
  }
  if (with_dot == 1) grid_dot_commit<Acc>(dot, acc);
}

// Coarse level of the two-level apply, one CTA per coarse domain: restriction
// rc = sum of r over each coarse node's vertices (linsolve.rs:648-655), the domain's
// z1 = W1^T (W1 rc) from its FP32 tiles, written as the coarse correction ec. A few hundred coarse
// domains do not fill the chip, so the chain in one of them is the time: a warp per coarse node
// (with one warp for all, its 16 to 32 nodes' gathers ran one after another) and a warp per
// tile in both products, whose partial sums are added in storage order. 200 x 200 grid,
// 16-vertex domains: 20.6 -> 6.2 us.
constexpr int CA_WARPS = 8;

__global__ void __launch_bounds__(32 * CA_WARPS) k_coarse_apply(
    const uint32_t* __restrict__ cdom_start, const uint32_t* __restrict__ cdom_nodes,
    const uint32_t* __restrict__ dom_start, const uint32_t* __restrict__ dom_verts,
    const uint64_t* __restrict__ cfac_off, const float* __restrict__ cfac, const float* __restrict__ r,
    float* __restrict__ ec, uint32_t ncdom, const PcgScalars* done) {
  __shared__ __align__(16) float buf[6 * TILE_FLOATS];
  __shared__ float rd[96];
  __shared__ double yd[96], part[6][32];
  if (done && done->done) return;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (uint32_t d1 = blockIdx.x; d1 < ncdom; d1 += gridDim.x) {
    const uint32_t n0 = cdom_start[d1], mn = cdom_start[d1 + 1] - n0;
    const int m = 3 * (int)mn, T = (m + 31) >> 5;
    const uint64_t off = cfac_off[d1];
    const int n4 = (int)(cfac_off[d1 + 1] - off) / 4;  // whole tiles
    for (int e = tid; e < n4; e += 32 * CA_WARPS)
      reinterpret_cast<float4*>(buf)[e] = __ldg(reinterpret_cast<const float4*>(cfac + off) + e);
#pragma unroll 4
    for (uint32_t a = w; a < mn; a += CA_WARPS) {
      const uint32_t g = cdom_nodes[n0 + a];
      double s0 = 0, s1 = 0, s2 = 0;
      for (uint32_t p = dom_start[g] + lane; p < dom_start[g + 1]; p += 32) {
        const uint32_t v = dom_verts[p];
        s0 += (double)r[3 * v];
        s1 += (double)r[3 * v + 1];
        s2 += (double)r[3 * v + 2];
      }
      s0 = warp_sum(s0);
      s1 = warp_sum(s1);
      s2 = warp_sum(s2);
      if (lane == 0) {
        rd[3 * a] = (float)s0;
        rd[3 * a + 1] = (float)s1;
        rd[3 * a + 2] = (float)s2;
      }
    }
    for (int i = m + tid; i < 96; i += 32 * CA_WARPS) rd[i] = 0.f;
    __syncthreads();
    const int I = w >= 3 ? 2 : (w >= 1 ? 1 : 0), J = w - I * (I + 1) / 2;  // this warp's tile
    const bool mine = w < T * (T + 1) / 2;
    const float* t = buf + w * TILE_FLOATS;
    if (mine) {
      double y = 0;
#pragma unroll 8
      for (int c = 0; c < 32; ++c) y += (double)tile_ld(t, tile_off<float>(lane, c)) * (double)rd[32 * J + c];
      part[w][lane] = y;
    }
    __syncthreads();
    if (w < T) {
      double y = part[w * (w + 1) / 2][lane];
      for (int k = 1; k <= w; ++k) y += part[w * (w + 1) / 2 + k][lane];
      yd[32 * w + lane] = y;
    }
    __syncthreads();
    if (mine) {
      double z = 0;
#pragma unroll 8
      for (int k = 0; k < 32; ++k) z += (double)tile_ld(t, tile_off<float>(k, lane)) * yd[32 * I + k];
      part[w][lane] = z;
    }
    __syncthreads();
    const int i = 32 * w + lane;
    if (w < T && i < m) {
      double z = part[w * (w + 1) / 2 + w][lane];
      for (int k = w + 1; k < T; ++k) z += part[k * (k + 1) / 2 + w][lane];
      ec[3 * cdom_nodes[n0 + i / 3] + i % 3] = (float)z;
    }
    __syncthreads();
  }
}

// z += w * ec[coarse node of the vertex] (the weighted prolongation, linsolve.rs:657-665),
// with the fused r.z of the PCG.
template <class Acc>
__global__ void k_prolong(const float* __restrict__ r, float* __restrict__ z, const float* __restrict__ ec,
                          const uint32_t* __restrict__ dom_of, uint32_t nb, float w, DotSink d, int with_dot) {
  if (with_dot && d.sc->done) return;
  Acc acc = 0;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nb; v += gridDim.x * blockDim.x) {
    const uint32_t g = dom_of[v];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float zc = fmaf(w, ec[3 * g + c], z[3 * v + c]);
      z[3 * v + c] = zc;
      acc += (Acc)r[3 * v + c] * (Acc)zc;
    }
  }
  if (with_dot) grid_dot_commit<Acc>(d, acc);
}

// Shared-memory opt-in for the largest domain (32 vertices, m = 96), set once outside any
// stream capture.
int schwarz_configure() {
  static bool done = false;
  if (done) return MGUSO_OK;
  const int asm32 = (int)(128 + (size_t)APPLY_WARPS * apply_slice_bytes<float>());
  const int asm16 = (int)(128 + (size_t)APPLY_WARPS * apply_slice_bytes<__half>());
  MG_CUDA(cudaFuncSetAttribute(k_schwarz_apply<APPLY_WARPS, double, float>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, asm32));
  MG_CUDA(cudaFuncSetAttribute(k_schwarz_apply<APPLY_WARPS, float, float>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, asm32));
  MG_CUDA(cudaFuncSetAttribute(k_schwarz_apply<APPLY_WARPS, double, __half>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, asm16));
  MG_CUDA(cudaFuncSetAttribute(k_schwarz_apply<APPLY_WARPS, float, __half>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, asm16));
  done = true;
  return MGUSO_OK;
}

int schwarz_apply(mguso_schwarz* s, const float* r, float* z, cudaStream_t st, const DotSink* dot) {
  DotSink d{};
  // two levels: the level-0 apply skips after convergence but leaves the r.z to the
  // prolongation, which completes z
  int with_dot = dot ? (s->levels == 2 ? 2 : 1) : 0;
  if (dot) d = *dot;
  bool mixed = dot && dot->mixed;
  if (s->max_m > 96) {
    set_error("Schwarz domain larger than 32 vertices");
    return MGUSO_ERR_UNSUPPORTED;
  }
  const bool h = s->half;
  size_t smem = 128 + (size_t)APPLY_WARPS * (h ? apply_slice_bytes<__half>() : apply_slice_bytes<float>());
  // resident CTAs per SM as shared memory allows (2 with FP32 tiles, 4 with FP16), grid-stride
  uint32_t grid = std::min<uint32_t>(ceil_div(s->ndom, APPLY_WARPS), (h ? 4u : 2u) * (uint32_t)s->a->ctx->sm_count);
  void* fn = h ? (mixed ? (void*)k_schwarz_apply<APPLY_WARPS, double, __half>
                        : (void*)k_schwarz_apply<APPLY_WARPS, float, __half>)
               : (mixed ? (void*)k_schwarz_apply<APPLY_WARPS, double, float>
                        : (void*)k_schwarz_apply<APPLY_WARPS, float, float>);
  const uint32_t* a0 = s->dom_start.p;
  const uint32_t* a1 = s->dom_verts.p;
  const uint64_t* a2 = s->fac_off.p;
  const void* a3 = h ? (const void*)s->fac_h.p : (const void*)s->fac.p;
  const float* a4 = h ? s->fac_scale.p : nullptr;
  uint32_t nd = s->ndom;
  uint32_t* stp = s->status.p;
  const uint8_t* a5 = s->dom_diag.p;
  const float* a6 = s->vfac.p;
  void* args[] = {(void*)&a0, (void*)&a1, (void*)&a2, (void*)&a3, (void*)&a4, (void*)&r, (void*)&z,
                  (void*)&nd, (void*)&stp, (void*)&d, (void*)&with_dot, (void*)&a5, (void*)&a6};
  if (grid == 0) return MGUSO_OK;
  MG_CUDA(cudaLaunchKernel(fn, dim3(grid), dim3(32 * APPLY_WARPS), args, smem, st));
  if (s->levels != 2 || s->ncdom == 0) return MGUSO_OK;
  const uint32_t cgrid = std::min<uint32_t>(s->ncdom, 8u * (uint32_t)s->a->ctx->sm_count);
  k_coarse_apply<<<cgrid, 32 * CA_WARPS, 0, st>>>(s->cdom_start.p, s->cdom_nodes.p, s->dom_start.p, s->dom_verts.p,
                                       s->cfac_off.p, s->cfac.p, r, s->ec.p, s->ncdom, dot ? dot->sc : nullptr);
  const uint32_t nb = s->a->nb;
  const uint32_t pgrid = std::max<uint32_t>(1, std::min<uint32_t>(ceil_div(nb, 256), 8u * (uint32_t)s->a->ctx->sm_count));
  const int wd = dot ? 1 : 0;
  if (mixed)
    k_prolong<double><<<pgrid, 256, 0, st>>>(r, z, s->ec.p, s->dom_of.p, nb, s->weight, d, wd);
  else
    k_prolong<float><<<pgrid, 256, 0, st>>>(r, z, s->ec.p, s->dom_of.p, nb, s->weight, d, wd);
  MG_CUDA(cudaGetLastError());
  return MGUSO_OK;
}

// ---------------------------------------------------------------------------------------
// Block Jacobi (linsolve.rs:294-315): per-vertex 3x3 inverse in f64, stored as 9 floats;
// a singular block (|det| < 1e-20) falls back to 1/diagonal (1 where the diagonal is 0).
// ---------------------------------------------------------------------------------------
__global__ void k_bj_factor(const uint32_t* __restrict__ row_ptr, const uint32_t* __restrict__ col,
                            const float* __restrict__ val, uint32_t nb, float* __restrict__ inv) {
  uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nb) return;
  double m[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (uint32_t k = row_ptr[v]; k < row_ptr[v + 1]; ++k)
    if (col[k] == v)
      for (int e = 0; e < 9; ++e) m[e] = (double)val[9 * (size_t)k + e];
  double det = m[0] * (m[4] * m[8] - m[5] * m[7]) - m[1] * (m[3] * m[8] - m[5] * m[6]) +
               m[2] * (m[3] * m[7] - m[4] * m[6]);
  double o[9];
  if (fabs(det) < 1e-20) {
    for (int e = 0; e < 9; ++e) o[e] = 0.0;
    for (int i = 0; i < 3; ++i) o[4 * i] = m[4 * i] != 0.0 ? 1.0 / m[4 * i] : 1.0;
  } else {
    double id = 1.0 / det;
    o[0] = (m[4] * m[8] - m[5] * m[7]) * id;
    o[1] = (m[2] * m[7] - m[1] * m[8]) * id;
    o[2] = (m[1] * m[5] - m[2] * m[4]) * id;
    o[3] = (m[5] * m[6] - m[3] * m[8]) * id;
    o[4] = (m[0] * m[8] - m[2] * m[6]) * id;
    o[5] = (m[2] * m[3] - m[0] * m[5]) * id;
    o[6] = (m[3] * m[7] - m[4] * m[6]) * id;
    o[7] = (m[1] * m[6] - m[0] * m[7]) * id;
    o[8] = (m[0] * m[4] - m[1] * m[3]) * id;
  }
  for (int e = 0; e < 9; ++e) inv[9 * (size_t)v + e] = (float)o[e];
}

int blockjacobi_factor(mguso_bsr* a, float* inv, cudaStream_t s) {
  if (a->nb == 0) return MGUSO_OK;
  k_bj_factor<<<ceil_div(a->nb, 128), 128, 0, s>>>(a->row_ptr.p, a->col.p, a->val.p, a->nb, inv);
  MG_CUDA(cudaGetLastError());
  return MGUSO_OK;
}

}  // namespace mg
