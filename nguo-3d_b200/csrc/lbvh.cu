// LBVH broad phase on sm_100a: Morton codes (30-bit u32 / 63-bit u64), a onesweep LSD
// radix sort of (key, payload) pairs, the Karras tree, a single-pass atomic-climb refit,
// and a traversal that emits every (query, triangle) pair whose boxes overlap.
//
// Reference pipeline (engine-gpu/src/{morton,radix,karras,bvh_aabb,bvh_traverse}.rs and
// the shaders of the same names): 30-bit codes only, an 8-bit LSD radix sort limited to
// 65 536 keys with a serial per-block scatter, level-by-level AABB passes, and one stack
// per thread. The results this file must reproduce bit-for-bit are the CPU oracles
// morton_codes_cpu (morton.rs:50-63; centroid = (a+b+c)/3, no FMA contraction), the
// stable sort permutation, karras_tree_cpu (karras.rs:24-88) and propagate_aabb_cpu
// (bvh_aabb.rs:28-56); the pair SET is `all(qlo <= bhi) && all(blo <= qhi)` against leaf
// boxes (bvh_traverse.wgsl:64-92).
#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>

#include "lbvh.cuh"

namespace mg {

// ---------------------------------------------------------------------------------------
// Morton codes
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t f2ord(float f) {
  uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b ^ 0x80000000u);
}
__device__ __forceinline__ float ord2f(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u ^ 0x80000000u) : ~u);
}

__device__ __forceinline__ float centroid_c(const float* __restrict__ pos, const uint32_t* t, int c) {
  float a = pos[3 * t[0] + c], b = pos[3 * t[1] + c], d = pos[3 * t[2] + c];
  return __fdiv_rn(__fadd_rn(__fadd_rn(a, b), d), 3.0f);
}

__global__ void k_centroid_bounds(const float* __restrict__ pos, const uint32_t* __restrict__ tris, uint32_t nt,
                                  uint32_t* __restrict__ ord /*6: lo.xyz as ord (min), hi.xyz (max)*/) {
  uint32_t lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0, 0, 0};
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < nt; t += gridDim.x * blockDim.x) {
    uint32_t tv[3] = {tris[3 * t], tris[3 * t + 1], tris[3 * t + 2]};
    for (int c = 0; c < 3; ++c) {
      uint32_t o = f2ord(centroid_c(pos, tv, c));
      lo[c] = min(lo[c], o);
      hi[c] = max(hi[c], o);
    }
  }
  for (int c = 0; c < 3; ++c) {
    for (int o = 16; o > 0; o >>= 1) {
      lo[c] = min(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
      hi[c] = max(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
    }
  }
  if ((threadIdx.x & 31) == 0) {
    for (int c = 0; c < 3; ++c) {
      atomicMin(&ord[c], lo[c]);
      atomicMax(&ord[3 + c], hi[c]);
    }
  }
}

// params: lo.xyz, inv.xyz (centroid_bounds, morton.rs:30-47)
__global__ void k_bounds_finish(const uint32_t* __restrict__ ord, float* __restrict__ params) {
  if (threadIdx.x == 0) {
    for (int c = 0; c < 3; ++c) {
      float lo = ord2f(ord[c]), hi = ord2f(ord[3 + c]);
      float ext = __fsub_rn(hi, lo);
      params[c] = lo;
      params[3 + c] = ext > 0.0f ? __fdiv_rn(1.0f, ext) : 0.0f;
    }
  }
}

__device__ __forceinline__ float clampf_nan(float v, float lo, float hi) { return v < lo ? lo : (v > hi ? hi : v); }

__device__ __forceinline__ uint32_t expand10(uint32_t v) {
  uint32_t x = v & 0x3ffu;
  x = (x | (x << 16)) & 0x030000ffu;
  x = (x | (x << 8)) & 0x0300f00fu;
  x = (x | (x << 4)) & 0x030c30c3u;
  x = (x | (x << 2)) & 0x09249249u;
  return x;
}
__device__ __forceinline__ uint64_t expand21(uint64_t v) {
  uint64_t x = v & 0x1fffffull;
  x = (x | (x << 32)) & 0x1f00000000ffffull;
  x = (x | (x << 16)) & 0x1f0000ff0000ffull;
  x = (x | (x << 8)) & 0x100f00f00f00f00full;
  x = (x | (x << 4)) & 0x10c30c30c30c30c3ull;
  x = (x | (x << 2)) & 0x1249249249249249ull;
  return x;
}

template <class K>
__device__ __forceinline__ K morton_of(float nx, float ny, float nz);
template <>
__device__ __forceinline__ uint32_t morton_of<uint32_t>(float nx, float ny, float nz) {
  auto q = [](float v) {
    return __float2uint_rz(clampf_nan(__fmul_rn(clampf_nan(v, 0.0f, 1.0f), 1023.0f), 0.0f, 1023.0f));
  };
  return expand10(q(nx)) * 4u + expand10(q(ny)) * 2u + expand10(q(nz));
}
template <>
__device__ __forceinline__ uint64_t morton_of<uint64_t>(float nx, float ny, float nz) {
  auto q = [](float v) {
    return (uint64_t)__float2uint_rz(clampf_nan(__fmul_rn(clampf_nan(v, 0.0f, 1.0f), 2097151.0f), 0.0f, 2097151.0f));
  };
  return expand21(q(nx)) * 4ull + expand21(q(ny)) * 2ull + expand21(q(nz));
}

template <class K>
__global__ void k_morton(const float* __restrict__ pos, const uint32_t* __restrict__ tris, uint32_t nt,
                         const float* __restrict__ params, K* __restrict__ keys, uint32_t* __restrict__ vals) {
  uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nt) return;
  uint32_t tv[3] = {tris[3 * t], tris[3 * t + 1], tris[3 * t + 2]};
  float n[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) n[c] = __fmul_rn(__fsub_rn(centroid_c(pos, tv, c), params[c]), params[3 + c]);
  keys[t] = morton_of<K>(n[0], n[1], n[2]);
  vals[t] = t;
}

// Morton codes of points (query ordering): same normalisation with the given params.
// Only their top bits order the queries (shift drops the rest).
__global__ void k_morton_points(const float* __restrict__ pts, uint32_t np, const float* __restrict__ params, int shift,
                                uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np) return;
  float n[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) n[c] = __fmul_rn(__fsub_rn(pts[3 * i + c], params[c]), params[3 + c]);
  keys[i] = morton_of<uint32_t>(n[0], n[1], n[2]) >> shift;
  vals[i] = i;
}

// ---------------------------------------------------------------------------------------
// Onesweep radix sort (stable LSD, 8-bit digits, decoupled look-back across tiles)
// ---------------------------------------------------------------------------------------
// Tiles: a pass is bound by latency when it has few tiles (ranking, then the look-back) and by the
// scatter's short runs and the look-back's chain when it has many. Small sorts take tiles of 2 048
// keys, so that 65 536 keys still spread over 32 SMs; from RS_LARGE keys on tiles of 6 144, whose
// runs per digit are three times as long. A pass over 65 536 u32 keys before -> after
// (look-back words read eight at a time, one memset for all passes, the digit scan in the pass
// itself): 9.8 -> 8.3 us, with half the launches between (whole sort 79 -> 53 us); a pass over
// 4 M keys and one over 12.6 M together 270 -> 199 us.
constexpr uint32_t RS_TILE_S = 256 * 8, RS_TILE_L = 384 * 16;
constexpr uint32_t RS_LARGE = 1u << 20;
constexpr uint32_t FLAG_AGG = 1u << 30, FLAG_PRE = 2u << 30, VAL_MASK = (1u << 30) - 1;
constexpr int RS_LOOK = 8;  // predecessors read at once by the look-back

template <class K>
__global__ void __launch_bounds__(256) k_rs_hist(const K* __restrict__ keys, uint32_t n, int passes,
                                                 uint32_t* __restrict__ hist) {
  __shared__ uint32_t sh[8 * 256];
  for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const uint32_t st = gridDim.x * blockDim.x;
  for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += 4 * st) {
    K k[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) k[u] = i0 + u * (uint64_t)st < n ? keys[i0 + u * st] : (K)0;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i0 + u * (uint64_t)st < n)
        for (int p = 0; p < passes; ++p) atomicAdd(&sh[p * 256 + (uint32_t)((k[u] >> (8 * p)) & 0xff)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * 256; i += blockDim.x)
    if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

// One pass: phist is its digit histogram, `skip` whether a pass whose keys all have one digit
// may only copy (the same decision in every CTA, so no look-back is started; the host never
// reads the histogram back).
template <class K, int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS) k_onesweep(const K* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                      K* __restrict__ kout, uint32_t* __restrict__ vout, uint32_t n,
                                                      int shift, const uint32_t* __restrict__ phist, int skip,
                                                      uint32_t* status, uint32_t* tile_counter, uint32_t* err) {
  constexpr uint32_t TILE = THREADS * ITEMS;
  constexpr int WARPS = THREADS / 32;
  extern __shared__ __align__(16) unsigned char rs_smem[];
  K* skeys = reinterpret_cast<K*>(rs_smem);
  uint32_t* svals = reinterpret_cast<uint32_t*>(skeys + TILE);
  __shared__ uint32_t whist[WARPS][256];
  __shared__ uint32_t tile_excl[256], g_pref[256];
  __shared__ uint32_t wsum[8], gsum[8];
  __shared__ uint32_t s_tile;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  if (skip && phist[(uint32_t)((kin[0] >> shift) & 0xff)] == n) {
    const uint32_t b0 = blockIdx.x * TILE, b1 = min(b0 + TILE, n);
    for (uint32_t j = b0 + tid; j < b1; j += THREADS) {
      kout[j] = kin[j];
      vout[j] = vin[j];
    }
    return;
  }
  if (tid == 0) s_tile = atomicAdd(tile_counter, 1u);
  for (int d = lane; d < 256; d += 32) whist[w][d] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint32_t base = tile * TILE;
  const uint32_t tile_n = min(TILE, n - base);
  K key[ITEMS];
  uint32_t val[ITEMS], rank[ITEMS];
  const uint32_t wbase = base + (uint32_t)w * ITEMS * 32;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const uint32_t idx = wbase + i * 32 + lane;
    key[i] = idx < n ? kin[idx] : (K)0;
    val[i] = idx < n ? vin[idx] : 0u;
  }
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const bool valid = wbase + i * 32 + lane < n;
    const uint32_t d = valid ? (uint32_t)((key[i] >> shift) & 0xff) : 0x100u + lane;
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    const int leader = __ffs(peers) - 1;
    const uint32_t before = __popc(peers & ((1u << lane) - 1u));
    uint32_t old = 0;
    if (valid && lane == leader) {
      old = whist[w][d];
      whist[w][d] = old + __popc(peers);
    }
    old = __shfl_sync(0xffffffffu, old, leader);
    rank[i] = old + before;
    __syncwarp();
  }
  __syncthreads();
  // per digit: offsets of each warp, the tile's count (published), and, while that travels, the
  // digit's start in the tile and in the whole output
  uint32_t run = 0, tincl = 0, gincl = 0, gcount = 0;
  if (tid < 256) {
    const int d = tid;
    for (int ww = 0; ww < WARPS; ++ww) {
      const uint32_t c = whist[ww][d];
      whist[ww][d] = run;
      run += c;
    }
    ((volatile uint32_t*)status)[(size_t)tile * 256 + d] = (tile ? FLAG_AGG : FLAG_PRE) | run;
    gcount = phist[d];
    tincl = run;
    gincl = gcount;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, tincl, o), g = __shfl_up_sync(0xffffffffu, gincl, o);
      if (lane >= o) {
        tincl += t;
        gincl += g;
      }
    }
    if (lane == 31) {
      wsum[w] = tincl;
      gsum[w] = gincl;
    }
  }
  __syncthreads();
  if (tid < 256) {
    const int d = tid;
    uint32_t tofs = 0, gofs = 0;
    for (int ww = 0; ww < w; ++ww) {
      tofs += wsum[ww];
      gofs += gsum[ww];
    }
    tile_excl[d] = tofs + tincl - run;
    // decoupled look-back, RS_LOOK predecessors in flight
    uint32_t excl = 0, spins = 0;
    int64_t j = (int64_t)tile - 1;
    bool more = tile > 0;
    while (more) {
      uint32_t v[RS_LOOK];
#pragma unroll
      for (int u = 0; u < RS_LOOK; ++u)
        v[u] = j - u >= 0 ? ((volatile uint32_t*)status)[(size_t)(j - u) * 256 + d] : FLAG_PRE + 0u;
      int used = 0;
#pragma unroll
      for (int u = 0; u < RS_LOOK; ++u) {
        if (!more || used < u) continue;  // stopped at an earlier one
        const uint32_t flag = v[u] & ~VAL_MASK;
        if (flag == 0) continue;
        used = u + 1;
        excl += v[u] & VAL_MASK;
        if (flag == FLAG_PRE) more = false;
      }
      j -= used;
      if (used == 0 && ++spins > (1u << 24)) {
        atomicOr(err, ST_WAIT_TIMEOUT);
        break;
      }
    }
    if (tile) ((volatile uint32_t*)status)[(size_t)tile * 256 + d] = FLAG_PRE | (excl + run);
    g_pref[d] = gofs + gincl - gcount + excl;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    if (wbase + i * 32 + lane < n) {
      const uint32_t d = (uint32_t)((key[i] >> shift) & 0xff);
      const uint32_t p = tile_excl[d] + whist[w][d] + rank[i];
      skeys[p] = key[i];
      svals[p] = val[i];
    }
  }
  __syncthreads();
  for (uint32_t j = tid; j < tile_n; j += THREADS) {
    const K k = skeys[j];
    const uint32_t d = (uint32_t)((k >> shift) & 0xff);
    const uint32_t o = g_pref[d] + (j - tile_excl[d]);
    kout[o] = k;
    vout[o] = svals[j];
  }
}

// ---------------------------------------------------------------------------------------
// Karras tree (karras.rs:24-88), with parent links for the refit
// ---------------------------------------------------------------------------------------
template <class K>
__device__ __forceinline__ int kdelta(const K* __restrict__ keys, int n, int i, int j) {
  if (j < 0 || j >= n) return -1;
  K x = keys[i] ^ keys[j];
  constexpr int W = 8 * sizeof(K);
  if (x == 0) return W + __clz((uint32_t)i ^ (uint32_t)j);
  if constexpr (sizeof(K) == 8)
    return __clzll((long long)x);
  else
    return __clz((int)x);
}

constexpr int RF_THREADS = 256;  // leaves of a subtree that the refit takes whole

template <class K>
__global__ void k_karras(const K* __restrict__ keys, uint32_t nn, uint32_t* __restrict__ parent_int,
                         uint32_t* __restrict__ parent_leaf, uint32_t* __restrict__ range_end,
                         uint32_t* __restrict__ flags, uint32_t* __restrict__ roots, uint32_t* __restrict__ nroots) {
  const int n = (int)nn;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  int d = (kdelta(keys, n, i, i + 1) - kdelta(keys, n, i, i - 1) < 0) ? -1 : 1;
  int dmin = kdelta(keys, n, i, i - d);
  int lmax = 2;
  while (kdelta(keys, n, i, i + lmax * d) > dmin) lmax *= 2;
  int l = 0;
  for (int t = lmax / 2; t >= 1; t /= 2)
    if (kdelta(keys, n, i, i + (l + t) * d) > dmin) l += t;
  int j = i + l * d;
  int first = min(i, j), last = max(i, j);
  int nd = kdelta(keys, n, first, last);
  int split = first, step = last - first;
  for (;;) {
    step = (step + 1) / 2;
    int ns = split + step;
    if (ns < last && kdelta(keys, n, first, ns) > nd) split = ns;
    if (step <= 1) break;
  }
  int g = split;
  range_end[i] = (uint32_t)j;
  flags[i] = 0;
  if (first == g)
    parent_leaf[g] = (uint32_t)i;
  else
    parent_int[g] = (uint32_t)i;
  if (last == g + 1)
    parent_leaf[g + 1] = (uint32_t)i | RIGHT_BIT;
  else
    parent_int[g + 1] = (uint32_t)i | RIGHT_BIT;
  if (i == 0) parent_int[0] = NO_PARENT;
  // the children that a refit's CTA can take whole
  if (last - first >= RF_THREADS) {
    const bool l = g - first < RF_THREADS, r = last - g <= RF_THREADS;
    if (l || r) {
      uint32_t at = atomicAdd(nroots, (uint32_t)l + (uint32_t)r);
      if (l) roots[at++] = (uint32_t)g | (first == g ? LEAF_BIT : 0u);
      if (r) roots[at] = (uint32_t)(g + 1) | (last == g + 1 ? LEAF_BIT : 0u);
    }
  }
}

// ---------------------------------------------------------------------------------------
// Boxes: one climb per leaf (in sorted order), which writes its box into its half of the parent's
// record; the second to arrive at a node goes on with the union of both halves. `v` is the
// positions, or the displacements for the CCD's records. What bounds a refit is the longest climb:
// a level across CTAs costs a fence, an atomic and a read of the sibling's half from L2, about 1 us.
// So CTAs take whole subtrees of up to 256 leaves (found with the tree: the largest such subtrees,
// listed in any order) and climb them in shared memory; only the tree above them is climbed
// through L2. Before -> after (leaf boxes in a kernel of their own, a memset of the flags,
// children's boxes and indices gathered again at every level), in brackets with CTAs of 256
// consecutive leaves, whose blocks cut subtrees at every level: 8 000 to 12 000 primitives
// 37 -> 15 (26) us, 41 401 50 -> 24 (36), 4.2 M 570 -> 340 (389; 640 MB are 100).
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void refit_climb(const float* __restrict__ v, const uint32_t* __restrict__ tris,
                                            const uint32_t* __restrict__ perm,
                                            const uint32_t* __restrict__ parent_leaf,
                                            const uint32_t* __restrict__ parent_int, float4* rec, uint32_t* flags,
                                            uint32_t nt, uint32_t b0, uint32_t top, const uint32_t* s_par,
                                            uint32_t* s_flag, float (*s_box)[6][RF_THREADS]) {
  const uint32_t i = b0 + threadIdx.x;
  const uint32_t t = perm[i];
  const uint32_t v0 = tris[3 * t], v1 = tris[3 * t + 1], v2 = tris[3 * t + 2];
  float lo[3], hi[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float a = v[3 * v0 + c], b = v[3 * v1 + c], d = v[3 * v2 + c];
    lo[c] = fminf(fminf(a, b), d);
    hi[c] = fmaxf(fmaxf(a, b), d);
  }
  if (nt == 1) {
    const float nan = __uint_as_float(0x7fffffffu);
    rec[0] = make_float4(lo[0], lo[1], lo[2], __uint_as_float(LEAF_BIT));
    rec[1] = make_float4(hi[0], hi[1], hi[2], 0.f);
    rec[2] = make_float4(nan, nan, nan, __uint_as_float(LEAF_BIT));
    rec[3] = make_float4(nan, nan, nan, 0.f);
    return;
  }
  uint32_t id = i | LEAF_BIT, up = parent_leaf[i];
  bool local = true;
  while (up != NO_PARENT) {
    local = local && up != top;
    const uint32_t p = up & ~RIGHT_BIT, side = up >> 31;
    float4* half = rec + 4 * (size_t)p + 2 * side;
    __stcg(half, make_float4(lo[0], lo[1], lo[2], __uint_as_float(id)));
    __stcg(half + 1, make_float4(hi[0], hi[1], hi[2], 0.f));
    if (local) {
      const uint32_t l = p - b0;
      if (l >= RF_THREADS) return;  // not of a tree: the sort gave up (its status says so)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        s_box[side][c][l] = lo[c];
        s_box[side][3 + c][l] = hi[c];
      }
      __threadfence_block();
      if (!(atomicAdd(&s_flag[l], 1u) & 1u)) return;
      __threadfence_block();
      volatile const float(*o)[RF_THREADS] = s_box[side ^ 1];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        lo[c] = fminf(lo[c], o[c][l]);
        hi[c] = fmaxf(hi[c], o[3 + c][l]);
      }
      up = s_par[l];
    } else {
      __threadfence();
      const uint32_t next = parent_int[p];
      if (!(atomicAdd(&flags[p], 1u) & 1u)) return;
      __threadfence();
      const float4* other = rec + 4 * (size_t)p + 2 * (side ^ 1u);
      const float4 olo = __ldcg(other), ohi = __ldcg(other + 1);
      lo[0] = fminf(lo[0], olo.x);
      lo[1] = fminf(lo[1], olo.y);
      lo[2] = fminf(lo[2], olo.z);
      hi[0] = fmaxf(hi[0], ohi.x);
      hi[1] = fmaxf(hi[1], ohi.y);
      hi[2] = fmaxf(hi[2], ohi.z);
      up = next;
    }
    id = p;
  }
}

__global__ void __launch_bounds__(RF_THREADS, 8) k_refit(const float* __restrict__ v, const uint32_t* __restrict__ tris,
                                                      const uint32_t* __restrict__ perm,
                                                      const uint32_t* __restrict__ parent_leaf,
                                                      const uint32_t* __restrict__ parent_int,
                                                      const uint32_t* __restrict__ range_end,
                                                      const uint32_t* __restrict__ roots,
                                                      const uint32_t* __restrict__ nroots, float4* rec,
                                                      uint32_t* flags, uint32_t nt) {
  __shared__ uint32_t s_par[RF_THREADS], s_flag[RF_THREADS];
  __shared__ float s_box[2][6][RF_THREADS];
  const uint32_t tid = threadIdx.x;
  const bool whole = nt <= RF_THREADS;
  const uint32_t nr = whole ? 1u : *nroots;
  for (uint32_t at = blockIdx.x; at < nr; at += gridDim.x) {
    // this subtree: leaves b0 .. b0 + count - 1, inner nodes within the same indices
    const uint32_t root = whole ? (nt == 1 ? LEAF_BIT : 0u) : roots[at], ri = root & ~LEAF_BIT;
    const uint32_t re = (root & LEAF_BIT) ? ri : range_end[ri], b0 = min(ri, re), count = max(ri, re) - b0 + 1;
    const uint32_t top = whole ? NO_PARENT : ((root & LEAF_BIT) ? parent_leaf[ri] : parent_int[ri]);
    __syncthreads();
    if (tid < count) {
      s_par[tid] = parent_int[b0 + tid];
      s_flag[tid] = 0;
    }
    __syncthreads();
    if (tid < count) refit_climb(v, tris, perm, parent_leaf, parent_int, rec, flags, nt, b0, top, s_par, s_flag, s_box);
  }
}

// ---------------------------------------------------------------------------------------
// Point queries: a warp takes 32 of them, neighbours in Morton order (qorder), down the tree
// together (warp_walk) and appends the pairs it finds 32 at a time, so that the pair counter takes
// one atomic per 32 pairs. 12.6 M points over 4.2 M triangles, before -> after (one stack per
// lane, boxes and child indices in separate arrays, one atomic per pair): 3.42 -> 2.13 ms, and 0.10
// ms for the query boxes, now made in registers. With all walks from the root 2.73. What bounds
// it is L1: 32 lanes on different nodes gather 64 bytes each. So the queues are short, which
// leaves L1 more of the SM's memory than the scenes' of 1 024 nodes would (2.50 ms; 256 nodes: no better).
// ---------------------------------------------------------------------------------------
constexpr int PT_CAP = 384;  // queued nodes per warp

__global__ void __launch_bounds__(WQ_WARPS * 32) k_traverse(BvhSet bv, const float* __restrict__ pts, float pad,
                                                            const uint32_t* __restrict__ qorder, uint32_t nq,
                                                            uint32_t per, uint32_t* __restrict__ pairs, uint64_t cap,
                                                            unsigned long long* __restrict__ count,
                                                            uint32_t* __restrict__ status) {
  __shared__ WalkMem<BoxQuery, PT_CAP> mem[WQ_WARPS];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, first = (blockIdx.x * WQ_WARPS + w) * per;
  const uint32_t k = first + lane;
  const bool valid = lane < per && k < nq;
  BoxQuery q;
  if (valid) {
    const uint32_t p = qorder ? qorder[k] : k;
    const float x = pts[3 * (size_t)p], y = pts[3 * (size_t)p + 1], z = pts[3 * (size_t)p + 2];
    q.lo = make_float4(__fsub_rn(x, pad), __fsub_rn(y, pad), __fsub_rn(z, pad), 0.f);
    q.hi = make_float4(__fadd_rn(x, pad), __fadd_rn(y, pad), __fadd_rn(z, pad), 0.f);
  }
  // the warp's common box goes down alone while it meets one child only
  float4 ulo = make_float4(INFINITY, INFINITY, INFINITY, 0.f), uhi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
  if (valid) {  // a NaN meets nothing and widens nothing
    ulo = make_float4(fminf(ulo.x, q.lo.x), fminf(ulo.y, q.lo.y), fminf(ulo.z, q.lo.z), 0.f);
    uhi = make_float4(fmaxf(uhi.x, q.hi.x), fmaxf(uhi.y, q.hi.y), fmaxf(uhi.z, q.hi.z), 0.f);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    ulo.x = fminf(ulo.x, __shfl_xor_sync(0xffffffffu, ulo.x, o));
    ulo.y = fminf(ulo.y, __shfl_xor_sync(0xffffffffu, ulo.y, o));
    ulo.z = fminf(ulo.z, __shfl_xor_sync(0xffffffffu, ulo.z, o));
    uhi.x = fmaxf(uhi.x, __shfl_xor_sync(0xffffffffu, uhi.x, o));
    uhi.y = fmaxf(uhi.y, __shfl_xor_sync(0xffffffffu, uhi.y, o));
    uhi.z = fmaxf(uhi.z, __shfl_xor_sync(0xffffffffu, uhi.z, o));
  }
  uint32_t start = 0;
  for (int level = 0; level < 128; ++level) {  // a tree is at most 64 key and 32 index bits deep
    const float4* r = bv.t[0].rec + 4 * (size_t)start;
    const float4 l0 = __ldg(r), h0 = __ldg(r + 1), l1 = __ldg(r + 2), h1 = __ldg(r + 3);
    const bool a = boxes_overlap(ulo, uhi, l0, h0), b = boxes_overlap(ulo, uhi, l1, h1);
    const uint32_t c = __float_as_uint(a ? l0.w : l1.w);
    if (a == b || (c & LEAF_BIT)) break;
    start = c;
  }
  const bool wide = ((uintptr_t)pairs & 7u) == 0;  // a caller's buffer may start on any 4 bytes
  const bool ok = warp_walk(mem[w], bv, first, valid, 0u, q, [](uint32_t, uint32_t) { return true; }, [&](uint2 e) {
    const unsigned m = __activemask();
    const int leader = __ffs(m) - 1;
    unsigned long long at = 0;
    if ((int)lane == leader) at = atomicAdd(count, (unsigned long long)__popc(m));
    at = __shfl_sync(m, at, leader) + __popc(m & ((1u << lane) - 1u));
    if (at < cap) {
      const uint32_t p = qorder ? qorder[e.x] : e.x;
      if (wide) {
        reinterpret_cast<uint2*>(pairs)[at] = make_uint2(p, e.y);
      } else {
        pairs[2 * at] = p;
        pairs[2 * at + 1] = e.y;
      }
    } else {
      atomicOr(status, ST_PAIR_OVERFLOW);
    }
  }, start);
  if (!ok) atomicOr(status, ST_STACK_OVERFLOW);
}

// ---------------------------------------------------------------------------------------
// Host orchestration
// ---------------------------------------------------------------------------------------
// The sort's device scratch: digit histograms of all passes, a tile counter per pass and the
// look-back words of all passes, laid out in that order so that one memset clears them.
struct SortScratch {
  uint32_t* words;
  unsigned char* tmpk;
  uint32_t *tmpv, *err;
};
static uint32_t rs_tile(uint32_t n) { return n >= RS_LARGE ? RS_TILE_L : RS_TILE_S; }
static size_t rs_words(uint32_t n, int passes) {
  return (size_t)passes * (256 + 1 + (size_t)ceil_div(n, rs_tile(n)) * 256);
}

template <class K, int THREADS, int ITEMS>
static int sort_pass(const K* kA, const uint32_t* vA, K* kB, uint32_t* vB, uint32_t n, int shift, const uint32_t* hist,
                     int skip, uint32_t* status, uint32_t* counter, uint32_t* err, cudaStream_t s) {
  constexpr uint32_t TILE = THREADS * ITEMS;
  constexpr int smem = (int)(TILE * (sizeof(K) + 4));
  auto fn = k_onesweep<K, THREADS, ITEMS>;
  if (smem > 32 * 1024) MG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  fn<<<ceil_div(n, TILE), THREADS, smem, s>>>(kA, vA, kB, vB, n, shift, hist, skip, status, counter, err);
  MG_CUDA(cudaGetLastError());
  return MGUSO_OK;
}

// Every pass is launched; with `skip`, a pass whose digit is the same for every key finds that
// out on the device and only copies, so the sort needs no readback.
template <class K>
static int sort_run(const SortScratch& sc, K* keys, uint32_t* vals, uint32_t n, int key_bits, int skip,
                    cudaStream_t s) {
  const int passes = (key_bits + 7) / 8;
  const uint32_t ntiles = ceil_div(n, rs_tile(n));
  uint32_t* hist = sc.words;
  uint32_t* counter = hist + 256 * passes;
  uint32_t* status = counter + passes;
  MG_CUDA(cudaMemsetAsync(sc.words, 0, 4 * rs_words(n, passes), s));
  const int sms = device_sm_count();
  k_rs_hist<K><<<std::min<uint32_t>(ceil_div(n, 1024), sms * 8), 256, 0, s>>>(keys, n, passes, hist);
  MG_CUDA(cudaGetLastError());
  K* kA = keys;
  uint32_t* vA = vals;
  K* kB = (K*)sc.tmpk;
  uint32_t* vB = sc.tmpv;
  for (int p = 0; p < passes; ++p) {
    const auto args = [&](auto fn) {
      return fn(kA, vA, kB, vB, n, 8 * p, hist + 256 * p, skip, status + (size_t)p * ntiles * 256, counter + p, sc.err,
                s);
    };
    if (n >= RS_LARGE)
      MG_TRY(args(sort_pass<K, 384, 16>));
    else
      MG_TRY(args(sort_pass<K, 256, 8>));
    std::swap(kA, kB);
    std::swap(vA, vB);
  }
  if (kA != keys) {
    MG_CUDA(cudaMemcpyAsync(keys, kA, sizeof(K) * (size_t)n, cudaMemcpyDeviceToDevice, s));
    MG_CUDA(cudaMemcpyAsync(vals, vA, 4 * (size_t)n, cudaMemcpyDeviceToDevice, s));
  }
  return MGUSO_OK;
}

template <class K>
static int sort_impl(Lbvh* b, K* keys, uint32_t* vals, uint32_t n, int key_bits, cudaStream_t s) {
  if (n <= 1) return MGUSO_OK;
  MG_TRY(b->rs_words.grow(rs_words(n, (key_bits + 7) / 8)));
  MG_TRY(b->rs_tmpk.grow((size_t)n * sizeof(K)));
  MG_TRY(b->rs_tmpv.grow(n));
  return sort_run<K>(SortScratch{b->rs_words.p, b->rs_tmpk.p, b->rs_tmpv.p, b->err_sink ? b->err_sink : b->status.p},
                     keys, vals, n, key_bits, 1, s);
}

int radix_sort_pairs(Lbvh* b, void* keys, uint32_t* vals, uint32_t n, int key_bits, cudaStream_t s) {
  if (key_bits <= 32) return sort_impl<uint32_t>(b, (uint32_t*)keys, vals, n, key_bits, s);
  return sort_impl<uint64_t>(b, (uint64_t*)keys, vals, n, key_bits, s);
}

// the centroid-bounds accumulator's start (ordered bits): the three minima at their highest
// value, the three maxima at their lowest; and the count of the refit's subtrees
__global__ void k_ord_init(uint32_t* __restrict__ ord, uint32_t* __restrict__ nroots) {
  if (threadIdx.x == 0) *nroots = 0;
  if (threadIdx.x < 6) ord[threadIdx.x] = threadIdx.x < 3 ? 0xffffffffu : 0u;
}

static int lbvh_reserve_nodes(Lbvh* b, uint32_t nt) {
  const size_t nn = std::max<uint32_t>(nt, 2);
  MG_TRY(b->shape.reserve(6 * nn + 1));
  b->parent_int = b->shape.p;
  b->parent_leaf = b->parent_int + nn;
  b->range_end = b->parent_leaf + nn;
  b->flags = b->range_end + nn;
  b->roots = b->flags + nn;  // at most nt of a tree; two per node whatever the keys
  b->nroots = b->roots + 2 * nn;
  return b->rec.reserve(4 * nn);
}

static int launch_refit(Lbvh* b, const float* v, const uint32_t* tris, float4* rec, cudaStream_t s) {
  // the subtrees' number is known on the device only: on average more than 64 leaves each. One per CTA,
  // so that the climbs above them overlap with the next (resident CTAs in a loop: 4.2 M 620 us).
  const uint32_t grid = b->nt <= RF_THREADS ? 1u : ceil_div(b->nt, 64);
  k_refit<<<grid, RF_THREADS, 0, s>>>(v, tris, b->perm.p, b->parent_leaf, b->parent_int, b->range_end, b->roots,
                                      b->nroots, rec, b->flags, b->nt);
  MG_CUDA(cudaGetLastError());
  return MGUSO_OK;
}

template <class K>
static int build_impl(Lbvh* b, const float* pos, const uint32_t* tris, uint32_t nt, int key_bits, cudaStream_t s) {
  b->shaped = false;
  b->nt = nt;
  b->key_bits = key_bits;
  MG_TRY(b->keys.reserve((size_t)std::max<uint32_t>(nt, 1) * sizeof(K)));
  MG_TRY(b->perm.reserve(std::max<uint32_t>(nt, 1)));
  MG_TRY(lbvh_reserve_nodes(b, nt));
  MG_TRY(b->params.reserve(8));
  MG_TRY(b->ord.reserve(8));
  MG_TRY(b->status.reserve(4));
  if (nt == 0) return MGUSO_OK;
  k_ord_init<<<1, 32, 0, s>>>(b->ord.p, b->nroots);
  int sms = device_sm_count();
  k_centroid_bounds<<<std::min<uint32_t>(ceil_div(nt, 256), sms * 8), 256, 0, s>>>(pos, tris, nt, b->ord.p);
  k_bounds_finish<<<1, 32, 0, s>>>(b->ord.p, b->params.p);
  K* keys = (K*)b->keys.p;
  k_morton<K><<<ceil_div(nt, 256), 256, 0, s>>>(pos, tris, nt, b->params.p, keys, b->perm.p);
  MG_CUDA(cudaGetLastError());
  if (b->ev_on) cudaEventRecord(b->ev[1], s);
  MG_TRY(sort_impl<K>(b, keys, b->perm.p, nt, key_bits, s));
  if (b->ev_on) cudaEventRecord(b->ev[2], s);
  if (nt > 1) {
    k_karras<K><<<ceil_div(nt - 1, 256), 256, 0, s>>>(keys, nt, b->parent_int, b->parent_leaf, b->range_end,
                                                     b->flags, b->roots, b->nroots);
  }
  if (b->ev_on) cudaEventRecord(b->ev[3], s);
  MG_TRY(launch_refit(b, pos, tris, b->rec.p, s));
  if (b->ev_on) cudaEventRecord(b->ev[4], s);
  b->shaped = true;
  return MGUSO_OK;
}

int lbvh_refit_disp(Lbvh* b, const float* dx, const uint32_t* tris, cudaStream_t s) {
  MG_TRY(b->drec.reserve(4 * (size_t)std::max<uint32_t>(b->nt, 2)));
  return b->nt ? launch_refit(b, dx, tris, b->drec.p, s) : MGUSO_OK;
}

int lbvh_refit_pos(Lbvh* b, const float* pos, const uint32_t* tris, cudaStream_t s) {
  MG_CHECK_ARG(b->shaped, "LBVH refit before a complete build");
  return b->nt ? launch_refit(b, pos, tris, b->rec.p, s) : MGUSO_OK;
}

// A node's children and its box, the union of its record's two halves (taken as the refit takes it).
__global__ void k_nodes(const float4* __restrict__ rec, uint32_t n, uint32_t* __restrict__ left,
                        uint32_t* __restrict__ right, float* __restrict__ boxes) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4* r = rec + 4 * (size_t)i;
  const float4 l0 = r[0], h0 = r[1], l1 = r[2], h1 = r[3];
  left[i] = __float_as_uint(l0.w);
  right[i] = __float_as_uint(l1.w);
  float* o = boxes + 6 * (size_t)i;
  o[0] = fminf(l0.x, l1.x);
  o[1] = fminf(l0.y, l1.y);
  o[2] = fminf(l0.z, l1.z);
  o[3] = fmaxf(h0.x, h1.x);
  o[4] = fmaxf(h0.y, h1.y);
  o[5] = fmaxf(h0.z, h1.z);
}

int lbvh_nodes(Lbvh* b, uint32_t* left, uint32_t* right, float* boxes) {
  const uint32_t n = b->nt - 1;
  cudaStream_t s = b->ctx->stream;
  MG_TRY(b->nodes.reserve(8 * (size_t)n));
  uint32_t *dl = b->nodes.p, *dr = dl + n;
  float* db = reinterpret_cast<float*>(dr + n);
  k_nodes<<<ceil_div(n, 256), 256, 0, s>>>(b->rec.p, n, dl, dr, db);
  MG_CUDA(cudaGetLastError());
  if (left) MG_CUDA(cudaMemcpyAsync(left, dl, 4 * (size_t)n, cudaMemcpyDeviceToHost, s));
  if (right) MG_CUDA(cudaMemcpyAsync(right, dr, 4 * (size_t)n, cudaMemcpyDeviceToHost, s));
  if (boxes) MG_CUDA(cudaMemcpyAsync(boxes, db, 24 * (size_t)n, cudaMemcpyDeviceToHost, s));
  MG_CUDA(cudaStreamSynchronize(s));
  return MGUSO_OK;
}

int lbvh_build(Lbvh* b, const float* pos, uint32_t nv, const uint32_t* tris, uint32_t nt, int key_bits,
               cudaStream_t s) {
  (void)nv;
  MG_CHECK_ARG(key_bits == 30 || key_bits == 63, "key_bits must be 30 or 63");
  MG_TRY(b->status.reserve(4));
  if (b->ev_on) cudaEventRecord(b->ev[0], s);
  if (key_bits == 30) return build_impl<uint32_t>(b, pos, tris, nt, key_bits, s);
  return build_impl<uint64_t>(b, pos, tris, nt, key_bits, s);
}

int lbvh_query_points(Lbvh* b, const float* pts, uint32_t np, float dhat, uint32_t* pairs, uint64_t cap,
                      unsigned long long* count, bool morton_order, cudaStream_t s) {
  MG_TRY(b->qkeys.reserve(std::max<uint32_t>(np, 1)));
  MG_TRY(b->qorder.reserve(std::max<uint32_t>(np, 1)));
  if (np == 0) return MGUSO_OK;
  const uint32_t* order = nullptr;
  if (morton_order && b->nt > 0) {
    // neighbours in a warp are enough: whole digits of the code's top bits, about two bits more
    // than the points have (12.6 M points: 24 of 30 bits)
    int bits = 8;
    while (bits < 24 && (1ull << bits) < 4ull * np) bits += 8;
    k_morton_points<<<ceil_div(np, 256), 256, 0, s>>>(pts, np, b->params.p, 30 - bits, b->qkeys.p, b->qorder.p);
    MG_TRY(sort_impl<uint32_t>(b, b->qkeys.p, b->qorder.p, np, bits, s));
    order = b->qorder.p;
  }
  MG_CUDA(cudaGetLastError());
  if (b->ev_on) cudaEventRecord(b->ev[5], s);
  if (b->nt > 0) {
    BvhSet set{};
    set.t[0] = lbvh_view(*b);
    uint32_t per = 32;
    while (per > 4 && (uint64_t)np < 16ull * (uint64_t)device_sm_count() * per) per /= 2;
    k_traverse<<<ceil_div(np, WQ_WARPS * per), WQ_WARPS * 32, 0, s>>>(set, pts, dhat, order, np, per, pairs, cap, count,
                                                                     b->status.p);
    MG_CUDA(cudaGetLastError());
  }
  if (b->ev_on) cudaEventRecord(b->ev[6], s);
  return MGUSO_OK;
}

// ---------------------------------------------------------------------------------------
// Allocation-free pair sort. Some callers may not allocate device memory after start-up:
// a host engine that hands all of the GPU's memory to its own pool when it starts, or a
// per-frame path where cudaMalloc's implicit device-wide synchronisation would stall the
// other streams. mguso_radix_sort_pairs_noalloc runs the same onesweep passes as
// radix_sort_pairs, with its temporaries in one fixed file-scope device array instead of
// buffers that grow on demand.
//
// Differences from radix_sort_pairs: every digit pass runs the full scatter (radix_sort_pairs
// turns a pass whose digit is the same for every key into a tile copy, found on the device;
// such a pass is the identity for a stable sort, so the output is the same), and the call
// waits for the sort to finish so it can report a look-back timeout from the scratch's
// error word.
// ---------------------------------------------------------------------------------------
constexpr uint32_t NOALLOC_MAX_PAIRS = 1u << 18;  // 262 144 pairs
constexpr size_t NA_TMPK = 0;                                         // u64 keys, ping-pong
constexpr size_t NA_TMPV = NA_TMPK + 8 * (size_t)NOALLOC_MAX_PAIRS;   // u32 payloads
constexpr size_t NA_WORDS = NA_TMPV + 4 * (size_t)NOALLOC_MAX_PAIRS;  // histograms, counters, look-back
constexpr size_t NA_ERR =
    NA_WORDS + (4 * 8 * (256 + 1 + 256 * (size_t)(NOALLOC_MAX_PAIRS / RS_TILE_S)) + 255) / 256 * 256;  // error word
constexpr size_t NA_BYTES = NA_ERR + 256;  // 4.1 MiB per device
static_assert(NOALLOC_MAX_PAIRS % RS_TILE_S == 0 && NOALLOC_MAX_PAIRS < RS_LARGE, "scratch holds whole small tiles");

// Every device that loads the library holds this array until the process exits. Host code
// must not pass the symbol itself to a kernel: its device address comes from
// cudaGetSymbolAddress, taken once per device below.
static __device__ __align__(256) unsigned char g_noalloc_sort_scratch[NA_BYTES];

constexpr int NA_MAX_DEVICES = 64;
static std::mutex g_noalloc_mu;
static unsigned char* g_noalloc_ptr[NA_MAX_DEVICES] = {};

// Device address of the scratch array on the current device (looked up on first use).
static int noalloc_scratch(unsigned char** out) {
  int dev = 0;
  MG_CUDA(cudaGetDevice(&dev));
  MG_CHECK_ARG(dev >= 0 && dev < NA_MAX_DEVICES, "device index beyond the allocation-free sort's table");
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_sort_scratch);
    if (e != cudaSuccess || !p) {
      set_error(std::string("cudaGetSymbolAddress(sort scratch): ") + cudaGetErrorString(e));
      return MGUSO_ERR_CUDA;
    }
    g_noalloc_ptr[dev] = (unsigned char*)p;
  }
  *out = g_noalloc_ptr[dev];
  return MGUSO_OK;
}

template <class K>
static int noalloc_sort(unsigned char* sc, K* keys, uint32_t* vals, uint32_t n, int key_bits, cudaStream_t s) {
  uint32_t* err = (uint32_t*)(sc + NA_ERR);
  // the array keeps the previous call's contents
  MG_CUDA(cudaMemsetAsync(err, 0, 4, s));
  MG_TRY(sort_run<K>(SortScratch{(uint32_t*)(sc + NA_WORDS), sc + NA_TMPK, (uint32_t*)(sc + NA_TMPV), err}, keys, vals,
                     n, key_bits, 0, s));
  uint32_t h_err = 0;
  MG_CUDA(cudaMemcpyAsync(&h_err, err, 4, cudaMemcpyDeviceToHost, s));
  MG_CUDA(cudaStreamSynchronize(s));
  if (h_err & ST_WAIT_TIMEOUT) {
    set_error("allocation-free sort: a decoupled look-back wait timed out");
    return MGUSO_ERR_TIMEOUT;
  }
  return MGUSO_OK;
}

}  // namespace mg

extern "C" int mguso_radix_sort_pairs_noalloc(void* keys, uint32_t* vals, uint32_t n, int key_bits, void* stream) {
  using namespace mg;
  MG_CHECK_ARG(key_bits >= 1 && key_bits <= 64, "key_bits must be in [1, 64]");
  if (n > NOALLOC_MAX_PAIRS) {
    set_error("mguso_radix_sort_pairs_noalloc: n = " + std::to_string(n) +
              " exceeds its fixed scratch limit of 262144 pairs; use mguso_radix_sort_pairs");
    return MGUSO_ERR_INVALID_ARG;
  }
  MG_CHECK_ARG(n == 0 || (keys && vals), "null argument");
  unsigned char* sc = nullptr;
  MG_TRY(noalloc_scratch(&sc));
  if (n <= 1) return MGUSO_OK;
  cudaStream_t s = (cudaStream_t)stream;
  if (key_bits <= 32) return noalloc_sort<uint32_t>(sc, (uint32_t*)keys, vals, n, key_bits, s);
  return noalloc_sort<uint64_t>(sc, (uint64_t*)keys, vals, n, key_bits, s);
}
