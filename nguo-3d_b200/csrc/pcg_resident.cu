// Resident PCG: one cooperative launch runs a whole solve (linsolve.rs:350-411: x0 = 0, r = b,
// z = M^-1 r, p = z; Ap, alpha = rz / pAp with a break on pAp <= 0 or NaN, x += alpha p,
// r -= alpha Ap, stop at ||r|| / ||b|| <= tol or max_iter, z = M^-1 r, beta = rz' / rz,
// p = z + beta p), with the matrix and the preconditioner kept in shared memory.
//
// What bounds a drape's PCG iteration is not its bytes but its chain of dependent steps: as two
// kernels per iteration it took 17 us for a 4 096-vertex sheet and 25 us for a 31 000-vertex
// garment, most of it launches, dependent loads from L2 and the last-CTA reductions (45 us for
// six garments, 137 MB an iteration). So here one CTA stays on each SM for the whole solve: 6.1,
// 9.5 and 33 us an iteration. What is left: two exchanges of 2.5 to 3 thousand cycles (1.3 thousand
// is what a store takes to be seen by another SM and read back), 1 to 1.5 thousand for the halo,
// and one warp's instruction chain in each phase.
//  - a CTA owns a run of Schwarz domains (block Jacobi: runs of 32 vertices), the domains'
//    vertices being also its matrix rows: r, p, z and Ap of its own rows never leave shared
//    memory, and x is touched by its owner only;
//  - at the start it packs its rows' blocks (pattern and contact blocks of a row in one list)
//    into shared memory, domain by domain: the domain's rows sorted by length, slot j holding
//    the j-th block of 32 rows as two float4 and a float2 per lane (three loads a block; slots
//    that fewer than 8 rows have are kept unpadded), with columns translated to places in
//    shared memory: its own vertices first, then the halo (distinct vertices of other CTAs,
//    found with a hash table). What does not fit (a batch of six garments needs 0.9 MB per SM)
//    is packed the same way into global scratch and streamed through a staging buffer per
//    team by bulk copies that run ahead of their use;
//  - the domains' W tiles follow in the rest of shared memory, FP16 ones else through the
//    staging buffers;
//  - an iteration exchanges one 32-byte record (z, p) per halo vertex and two scalars per CTA.
//    The CTAs of one instance synchronise twice per iteration by sending each other their partial
//    dot products, each in one 16-byte word with an epoch, and counting up; records carry the
//    epoch too, so what is read too early is seen to be and read again: no fence. Instances
//    of a batch never wait for another.
// Three warps (a team) take one domain at a time: for the rows each warp takes every third
// block of a row, for the preconditioner every third tile. Where a CTA has three domains or
// fewer, six warps do (36 warps in six such teams were no faster: 64 registers a thread spill).
//
// The CTAs are resident together (cooperative launch), so a solve takes the whole chip and starts
// once other kernels leave it to it (20 s of another stream's kernel delayed a solve by 20 s).
// Every poll is bounded: a CTA that gives up sets its instance's status and leaves, and the
// others follow. Dot products are summed in a
// fixed order that does not depend on timing (where a domain is kept changes no sum), so
// a solve is reproducible. Data written by other CTAs is read past L1 (relaxed loads of 16 bytes).
#include <algorithm>

#include "coop.cuh"
#include "recip.cuh"
#include "reduce.cuh"
#include "scene.cuh"
#include "tiles.cuh"

namespace mg {

constexpr int RS_WARPS = 18;          // six teams of three warps, or three of six
constexpr int RS_THREADS = 32 * RS_WARPS;
constexpr int RS_MAX_DOM = 64;       // domains (of <= 32 vertices) per CTA
constexpr uint32_t RS_HASH = 4096;   // halo hash table entries
constexpr uint32_t RS_PROBES = 64;   // a column not placed within these is read from global
constexpr uint32_t RS_MAX_HALO = 1536;
constexpr uint32_t RS_HASH_BYTES = RS_HASH * 6;
constexpr uint32_t RS_SCRATCH = 16128;    // the teams' scratch
constexpr uint32_t RS_CHUNK = 12288;      // a staging buffer (an FP16 domain's tiles); two per team
constexpr uint32_t RS_EMPTY = 0xffffffffu;
constexpr uint32_t RS_WIDE = 8;  // rows that make a slot worth padding to 32
constexpr uint32_t RS_ALWAYS = 0xffffffffu;  // epoch of a record that holds for the whole solve
constexpr int RS_MAX_G = 160;
// An exchange waits for the slowest CTA's phase: up to seconds. A record was stored before the exchange
// that its reader has passed, so only the store's way to L2 is waited for (a microsecond or two;
// 10 ms at most). That limit is each record's own, so a CTA that misses several (3 of a halo, or
// those of a row walked in the BSR) takes that many: a look at s_abort in the poll, inlined or
// not, cost the iterations registers (two steps of one garment 37.7 -> 38.3 to 39.5 ms).
constexpr uint32_t RS_EXCHANGE_POLLS = 1u << 22, RS_RECORD_POLLS = 1u << 14;

struct RsInst {
  uint32_t k, cta0, ncta;
  uint32_t dn0, dn1;  // its domains with tiles (block Jacobi: runs of 32 vertices from v0)
  uint32_t dd0, dd1;  // its block-diagonal domains (isolated vertices)
  uint32_t v0, v1;
};

struct RsArgs {
  uint32_t nrun;
  RsInst inst[PCG_MAX_INST];
  RsSystem sys;
  float* x;
  float4* rec;          // 2 per position: z, p
  float* jscr;          // packed rows that do not fit in shared memory
  uint32_t jcap;        // its capacity in 16-byte units
  uint32_t* jtop;       // units taken
  uint4* sums;          // published partial sums: p.Ap, r.r, r.z of each CTA
  uint32_t* count;      // per instance: CTAs that have published, 32 words apart
  uint32_t epoch;       // epochs of this solve are epoch + 1, + 2, ..
  FusedInst* out;
  float tol;
  uint32_t max_iter;
  uint32_t smem_bytes;
};

__device__ __forceinline__ float rs_fma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double rs_fma(double a, double b, double c) { return fma(a, b, c); }
// FP32 operands of FP64 sums. The conversion instruction runs at 16 lanes a cycle and SM, a quarter
// of the multiply-adds' rate, and took most of the row phase; a shift and a mask run at four times
// that. FP32 bits moved to where an FP64 number has them (exponent field unchanged) are
// the value times 2^-896, exactly, zeros and subnormals included; the other operand is converted
// and takes a factor 2^448, the sum another at its end. All three are exact and nothing in between
// leaves the normal range (a product of two FP32 numbers has an exponent of -298 to 256, here less
// 448), so sums are bit for bit those of converted operands. Infinities and NaN have no
// such image: matrix rows and tiles that hold one take the other paths (rs_finite).
// Time in the solves of one garment's two steps 26.2 -> 24.9 ms, of six garments' 84.8 -> 82.0.
__device__ __forceinline__ bool rs_finite(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }
// kept out of line: inlined into the set-up it costs the iterations registers (one 64 x 64 solve 1.18 ->
// 1.24 ms)
__device__ __noinline__ bool rs_block_finite(const float* m) {
  bool ok = true;
  for (int e = 0; e < 9; ++e) ok = ok && rs_finite(m[e]);
  return ok;
}
__device__ __forceinline__ float rs_widen(float v, float) { return v; }
__device__ __forceinline__ double rs_widen(float v, double) {
  const int b = __float_as_int(v);
  return __hiloint2double((b >> 3) & (int)0x8fffffffu, b << 29);
}
__device__ __forceinline__ float rs_lift(float v) { return v; }
__device__ __forceinline__ double rs_lift(double v) { return v * 0x1p448; }

template <int THREADS>
__device__ __forceinline__ void team_sync_of(int team) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(THREADS) : "memory");
}
// 16 bytes as one access: a record or a published sum and its epoch arrive together
__device__ __forceinline__ uint4 ld_rlx(const void* p) {
  unsigned long long lo, hi;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  return make_uint4((uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32));
}
__device__ __forceinline__ void st_rlx(void* p, uint4 v) {
  const unsigned long long lo = v.x | ((unsigned long long)v.y << 32), hi = v.z | ((unsigned long long)v.w << 32);
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p), "l"(lo),
               "l"(hi)
               : "memory");
}
__device__ __forceinline__ void st_rec(float4* p, float x, float y, float z, uint32_t epoch) {
  st_rlx(p, make_uint4(__float_as_uint(x), __float_as_uint(y), __float_as_uint(z), epoch));
}
// ---- a 32 x 32 tile held by a warp in registers -------------------------------------------
// Both passes of z = W^T (W r) run from one load of the tile: a warp reads it as whole 512-byte
// rows (no bank conflicts, full sectors from L2), every lane multiplies what it holds, and
// the lanes' partial sums are combined by halving exchanges (a lane keeps half of its sums and
// gets the partner's for them), 7 shuffles for 32 row sums instead of 32 element loads a lane.
// Summation type AA: the precision's, but FP32 over FP16 tiles (whose own rounding dwarfs FP32 sums
// of 32 terms), as the fused three-warp kernels sum, unless the caller asks for FP64 there
// (pcg_mode 2): two steps of one garment 30.4 -> 32.5 ms, of six 130 -> 147. Domains of one tile (10
// vertices or fewer), for which the one-warp kernel is the faster of the fused ones, take its FP64 sums.
template <class AA, class TS>
struct TileRegs;

// two FP32 multiply-adds in one instruction
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long x, y, z, d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(b.x), "f"(b.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(z) : "f"(c.x), "f"(c.y));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(x), "l"(y), "l"(z));
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(d));
  return r;
}

// FP16 tiles (tile_off<__half>): lane l holds rows 8k .. 8k + 7, k = ((l & 3) ^ (l >> 3)) & 3, of
// the four columns 8i + (l >> 2). The lanes that share k differ by the masks 4, 9 and 18.
template <class AA>
struct TileRegs<AA, __half> {
  uint4 u[4];
  __device__ __forceinline__ void load(const __half* t, int lane) {
    const uint4* s = reinterpret_cast<const uint4*>(t);
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i] = s[32 * i + lane];
  }
  __device__ __forceinline__ static void pairs(const uint4& v, float2 (&h)[4]) {
    h[0] = __half22float2(*reinterpret_cast<const __half2*>(&v.x));
    h[1] = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
    h[2] = __half22float2(*reinterpret_cast<const __half2*>(&v.z));
    h[3] = __half22float2(*reinterpret_cast<const __half2*>(&v.w));
  }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i] = make_uint4(0, 0, 0, 0);
  }
  // (W v)_row over the tile's columns; returns the lane's row and its sum
  __device__ __forceinline__ AA rows(const float* __restrict__ v, int lane, int& row) const {
    const int g = lane >> 2, k = ((lane & 3) ^ (lane >> 3)) & 3;
    float2 p[4] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float c = v[8 * i + g];
      float2 h[4];
      pairs(u[i], h);
#pragma unroll
      for (int t = 0; t < 4; ++t) p[t] = fma2(h[t], make_float2(c, c), p[t]);
    }
    AA s[8] = {p[0].x, p[0].y, p[1].x, p[1].y, p[2].x, p[2].y, p[3].x, p[3].y};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const AA send = (g & 4) ? s[t] : s[t + 4], keep = (g & 4) ? s[t + 4] : s[t];
      s[t] = keep + __shfl_xor_sync(0xffffffffu, send, 18);
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const AA send = (g & 2) ? s[t] : s[t + 2], keep = (g & 2) ? s[t + 2] : s[t];
      s[t] = keep + __shfl_xor_sync(0xffffffffu, send, 9);
    }
    const AA send = (g & 1) ? s[0] : s[1], keep = (g & 1) ? s[1] : s[0];
    row = 8 * k + g;
    return keep + __shfl_xor_sync(0xffffffffu, send, 4);
  }
  // (W^T y)_col over the tile's rows; returns the lane's column and its sum
  __device__ __forceinline__ AA cols(const AA* __restrict__ y, int lane, int& col) const {
    const int g = lane >> 2, k = ((lane & 3) ^ (lane >> 3)) & 3;
    const float4 ya = *reinterpret_cast<const float4*>(y + 8 * k), yb = *reinterpret_cast<const float4*>(y + 8 * k + 4);
    AA z[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 h[4], a = {0.f, 0.f};
      pairs(u[i], h);
      a = fma2(h[0], make_float2(ya.x, ya.y), a);
      a = fma2(h[1], make_float2(ya.z, ya.w), a);
      a = fma2(h[2], make_float2(yb.x, yb.y), a);
      a = fma2(h[3], make_float2(yb.z, yb.w), a);
      z[i] = a.x + a.y;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const AA send = (lane & 2) ? z[i] : z[i + 2], keep = (lane & 2) ? z[i + 2] : z[i];
      z[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
    }
    const AA send = (lane & 1) ? z[0] : z[1], keep = (lane & 1) ? z[1] : z[0];
    col = 8 * (lane & 3) + g;
    return keep + __shfl_xor_sync(0xffffffffu, send, 1);
  }
};

// FP16 tiles summed in FP64: as above, the FP16 bits moved to where an FP64 number has them (times
// 2^-1008, exactly, subnormals included; the vectors and the sums take 2^504 each).
template <>
struct TileRegs<double, __half> {
  uint4 u[4];
  __device__ __forceinline__ void load(const __half* t, int lane) {
    const uint4* s = reinterpret_cast<const uint4*>(t);
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i] = s[32 * i + lane];
  }
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 4; ++i) u[i] = make_uint4(0, 0, 0, 0);
  }
  __device__ __forceinline__ static double lift(double v) { return v * 0x1p504; }
  __device__ __forceinline__ static uint32_t word(const uint4& v, int t) {
    return t == 0 ? v.x : t == 1 ? v.y : t == 2 ? v.z : v.w;
  }
  __device__ __forceinline__ static double lo(uint32_t w) {
    return __hiloint2double(((int)(w << 16) >> 6) & (int)0x81fffc00u, 0);
  }
  __device__ __forceinline__ static double hi(uint32_t w) {
    return __hiloint2double(((int)w >> 6) & (int)0x81fffc00u, 0);
  }
  __device__ __forceinline__ double rows(const float* __restrict__ v, int lane, int& row) const {
    const int g = lane >> 2, k = ((lane & 3) ^ (lane >> 3)) & 3;
    double s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const double c = lift((double)v[8 * i + g]);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        s[2 * t] = fma(lo(word(u[i], t)), c, s[2 * t]);
        s[2 * t + 1] = fma(hi(word(u[i], t)), c, s[2 * t + 1]);
      }
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const double send = (g & 4) ? s[t] : s[t + 4], keep = (g & 4) ? s[t + 4] : s[t];
      s[t] = keep + __shfl_xor_sync(0xffffffffu, send, 18);
    }
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const double send = (g & 2) ? s[t] : s[t + 2], keep = (g & 2) ? s[t + 2] : s[t];
      s[t] = keep + __shfl_xor_sync(0xffffffffu, send, 9);
    }
    const double send = (g & 1) ? s[0] : s[1], keep = (g & 1) ? s[1] : s[0];
    row = 8 * k + g;
    return lift(keep + __shfl_xor_sync(0xffffffffu, send, 4));
  }
  __device__ __forceinline__ double cols(const double* __restrict__ y, int lane, int& col) const {
    const int g = lane >> 2, k = ((lane & 3) ^ (lane >> 3)) & 3;
    double z[4] = {0, 0, 0, 0};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const double2 yy = *reinterpret_cast<const double2*>(y + 8 * k + 2 * t);
      const double y0 = lift(yy.x), y1 = lift(yy.y);
#pragma unroll
      for (int i = 0; i < 4; ++i) z[i] = fma(hi(word(u[i], t)), y1, fma(lo(word(u[i], t)), y0, z[i]));
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const double send = (lane & 2) ? z[i] : z[i + 2], keep = (lane & 2) ? z[i + 2] : z[i];
      z[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
    }
    const double send = (lane & 1) ? z[0] : z[1], keep = (lane & 1) ? z[1] : z[0];
    col = 8 * (lane & 3) + g;
    return lift(keep + __shfl_xor_sync(0xffffffffu, send, 1));
  }
};

// FP32 tiles (element (r, c) at c * 32 + (r ^ c)): lane l holds rows 4w .. 4w + 3, w = l & 7, of
// the eight columns 4i + h, h = l >> 3; the value at place t of a group is row 4w + (t ^ h).
template <class AA>
struct TileRegs<AA, float> {
  float4 u[8];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 8; ++i) u[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __device__ __forceinline__ void load(const float* t, int lane) {
    const float4* s = reinterpret_cast<const float4*>(t);
    const int h = lane >> 3, w = lane & 7;
#pragma unroll
    for (int i = 0; i < 8; ++i) u[i] = s[8 * (4 * i + h) + (w ^ i)];
  }
  __device__ __forceinline__ AA rows(const float* __restrict__ v, int lane, int& row) const {
    const int h = lane >> 3, w = lane & 7;
    AA s[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const AA c = rs_lift((AA)v[4 * i + h]);
      s[0] += rs_widen(u[i].x, AA(0)) * c;
      s[1] += rs_widen(u[i].y, AA(0)) * c;
      s[2] += rs_widen(u[i].z, AA(0)) * c;
      s[3] += rs_widen(u[i].w, AA(0)) * c;
    }
    // into row order
    const AA a0 = (h & 1) ? s[1] : s[0], a1 = (h & 1) ? s[0] : s[1], a2 = (h & 1) ? s[3] : s[2],
             a3 = (h & 1) ? s[2] : s[3];
    // rows 0, 1 of the group are (a0, a1) without and (a2, a3) with h & 2
    const AA lo0 = (h & 2) ? a2 : a0, lo1 = (h & 2) ? a3 : a1, hi0 = (h & 2) ? a0 : a2, hi1 = (h & 2) ? a1 : a3;
    const AA k0 = ((h & 2) ? hi0 : lo0) + __shfl_xor_sync(0xffffffffu, (h & 2) ? lo0 : hi0, 16);
    const AA k1 = ((h & 2) ? hi1 : lo1) + __shfl_xor_sync(0xffffffffu, (h & 2) ? lo1 : hi1, 16);
    row = 4 * w + h;
    return rs_lift(((h & 1) ? k1 : k0) + __shfl_xor_sync(0xffffffffu, (h & 1) ? k0 : k1, 8));
  }
  __device__ __forceinline__ AA cols(const AA* __restrict__ y, int lane, int& col) const {
    const int h = lane >> 3, w = lane & 7;
    AA yy[4], z[8];
#pragma unroll
    for (int t = 0; t < 4; ++t) yy[t] = rs_lift(y[4 * w + (t ^ h)]);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      z[i] = rs_widen(u[i].x, AA(0)) * yy[0] + rs_widen(u[i].y, AA(0)) * yy[1] + rs_widen(u[i].z, AA(0)) * yy[2] + rs_widen(u[i].w, AA(0)) * yy[3];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const AA send = (w & 4) ? z[i] : z[i + 4], keep = (w & 4) ? z[i + 4] : z[i];
      z[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const AA send = (w & 2) ? z[i] : z[i + 2], keep = (w & 2) ? z[i + 2] : z[i];
      z[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
    }
    const AA send = (w & 1) ? z[0] : z[1], keep = (w & 1) ? z[1] : z[0];
    col = 4 * w + h;
    return rs_lift(keep + __shfl_xor_sync(0xffffffffu, send, 1));
  }
};

// row and column block of tile t (storage order)
__device__ __forceinline__ int rs_tile_i(int t) { return t >= 3 ? 2 : (t >= 1 ? 1 : 0); }
__device__ __forceinline__ int rs_tile_j(int t) { return t - rs_tile_i(t) * (rs_tile_i(t) + 1) / 2; }

// the next chunk a team stages: which domain's rows or tiles, and which part of them
struct StageNext {
  int di;
  uint32_t part, tiles, issued;
};

template <int PRE, class Acc, class TS, int TW, class AA>
__global__ void __launch_bounds__(RS_THREADS, 1) k_pcg_resident(const __grid_constant__ RsArgs a) {
  constexpr bool SCH = PRE == MGUSO_PRECOND_SCHWARZ;
  constexpr int TEAMS = RS_WARPS / TW, TEAM = 32 * TW;
  constexpr uint32_t TEAM_BYTES = RS_SCRATCH / TEAMS;  // per-team scratch
  constexpr uint32_t CHUNK_SLOTS = TW == 3 ? 9 : 6;    // whole slots of packed rows per chunk: a multiple of TW
  auto team_sync = [](int t) { team_sync_of<TEAM>(t); };
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint32_t s_dpos[RS_MAX_DOM + 1];  // first own vertex of each domain
  __shared__ uint32_t s_bytes[RS_MAX_DOM];  // of the packed rows
  __shared__ uint32_t s_jofs[RS_MAX_DOM], s_tofs[RS_MAX_DOM];
  __shared__ uint16_t s_wide[RS_MAX_DOM], s_tail[RS_MAX_DOM];  // whole slots; blocks past them
  __shared__ float s_scale[RS_MAX_DOM];
  __shared__ uint8_t s_jmode[RS_MAX_DOM];  // 0 shared memory, 1 staged from global scratch, 2 the BSR itself
  __shared__ uint8_t s_far[RS_MAX_DOM];
  __shared__ StageNext s_sg[TEAMS];
  __shared__ __align__(8) uint64_t s_bar[2 * TEAMS];
  __shared__ uint16_t s_len[RS_MAX_DOM * 32];
  __shared__ uint8_t s_row[RS_MAX_DOM * 32];
  __shared__ Acc s_red[2][RS_WARPS];
  __shared__ float s_alpha, s_beta;
  __shared__ double s_rr, s_rz, s_bnorm, s_lim2;  // warp 0's
  __shared__ uint32_t s_iters, s_status;
  __shared__ uint32_t s_nh, s_nlive, s_done, s_abort;
  __shared__ uint32_t s_stage;  // first byte of the staging buffers (0: none)
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int team = wid / TW, q = wid - TW * team, ti = 32 * q + lane;
  const RsSystem& S = a.sys;

  uint32_t ii = 0;
  while (ii + 1 < a.nrun && blockIdx.x >= a.inst[ii + 1].cta0) ++ii;
  const RsInst& I = a.inst[ii];
  const uint32_t G = I.ncta, j = blockIdx.x - I.cta0;
  auto share = [&](uint32_t n, uint32_t at) { return (uint32_t)((uint64_t)n * at / G); };
  auto dstart = [&](uint32_t d) -> uint32_t { return SCH ? S.dom_start[d] : min(I.v0 + 32 * (d - I.dn0), I.v1); };
  auto vert = [&](uint32_t pos) -> uint32_t { return SCH ? S.dom_verts[pos] : pos; };
  auto position = [&](uint32_t v) -> uint32_t { return SCH ? __ldg(S.vpos + v) : v; };
  const uint32_t d0 = I.dn0 + share(I.dn1 - I.dn0, j), d1 = I.dn0 + share(I.dn1 - I.dn0, j + 1);
  const int nD = (int)(d1 - d0);
  const uint32_t P0 = nD ? dstart(d0) : 0, own = nD ? dstart(d1) - P0 : 0;
  const uint32_t e0 = I.dd0 + share(I.dd1 - I.dd0, j), e1 = I.dd0 + share(I.dd1 - I.dd0, j + 1);
  const uint32_t Q0 = e1 > e0 ? S.dom_start[e0] : 0, nq = e1 > e0 ? S.dom_start[e1] - Q0 : 0;

  // ---- the halo: distinct columns of the CTA's rows that other CTAs own
  uint32_t* hkey = reinterpret_cast<uint32_t*>(smem + a.smem_bytes - RS_HASH_BYTES);
  uint16_t* hval = reinterpret_cast<uint16_t*>(hkey + RS_HASH);
  for (uint32_t h = tid; h < RS_HASH; h += RS_THREADS) {
    hkey[h] = RS_EMPTY;
    hval[h] = 0;
  }
  for (int di = tid; di <= nD; di += RS_THREADS) s_dpos[di] = nD ? dstart(d0 + di) - P0 : 0;
  for (int di = tid; di < nD; di += RS_THREADS) s_far[di] = 0;
  if (tid == 0) {
    s_nh = 0;
    s_done = 0;
    s_abort = 0;
    for (int t = 0; t < 2 * TEAMS; ++t) mbar_init(&s_bar[t], 1);
    for (int t = 0; t < TEAMS; ++t) s_sg[t] = StageNext{t, 0u, SCH ? 1u : 0u, 0u};
    fence_mbar_init();
    s_alpha = 0.f;
    s_beta = 0.f;
    s_status = 0;
  }
  __syncthreads();
  auto hash_of = [](uint32_t pos) { return (pos * 2654435761u) >> 20; };
  auto visit = [&](uint32_t c) {
    const uint32_t pos = position(c);
    if (pos - P0 < own) return;
    uint32_t h = hash_of(pos);
    for (uint32_t probe = 0; probe < RS_PROBES; ++probe, h = (h + 1) & (RS_HASH - 1)) {
      const uint32_t old = atomicCAS(hkey + h, RS_EMPTY, pos);
      if (old == pos) return;
      if (old == RS_EMPTY) {
        const uint32_t at = atomicAdd(&s_nh, 1u);
        if (at < RS_MAX_HALO) hval[h] = (uint16_t)(at + 1);
        return;
      }
    }
  };
  for (uint32_t i = wid; i < own; i += RS_WARPS) {
    const uint32_t v = vert(P0 + i);
    for (uint32_t k = S.rp[v] + lane; k < S.rp[v + 1]; k += 32) visit(S.col[k]);
    if (S.crp)
      for (uint32_t k = S.crp[v] + lane; k < S.crp[v + 1]; k += 32) visit(S.ccol[k]);
  }
  // rows of each domain by falling length (lane = row)
  for (int di = wid; di < nD; di += RS_WARPS) {
    const uint32_t nvd = s_dpos[di + 1] - s_dpos[di];
    uint32_t len = 0;
    if ((uint32_t)lane < nvd) {
      const uint32_t v = vert(P0 + s_dpos[di] + lane);
      len = S.rp[v + 1] - S.rp[v] + (S.crp ? S.crp[v + 1] - S.crp[v] : 0u);
    }
    uint32_t rank = 0, total = 0, wide = 0, in_wide = 0;
    for (int o = 0; o < 32; ++o) {
      const uint32_t l2 = __shfl_sync(0xffffffffu, len, o);
      rank += (l2 > len || (l2 == len && o < lane)) ? 1u : 0u;
      total += l2;
    }
    for (;; ++wide) {
      const uint32_t n = __popc(__ballot_sync(0xffffffffu, len > wide));
      if (n < RS_WIDE) break;
      in_wide += n;
    }
    s_len[32 * di + rank] = (uint16_t)min(len, 65535u);
    s_row[32 * di + rank] = (uint8_t)lane;
    if (lane == 0) {
      s_wide[di] = (uint16_t)min(wide, 65535u);
      s_tail[di] = (uint16_t)min(total - in_wide, 65535u);
      const uint64_t by = 1280ull * wide + ((40ull * (total - in_wide) + 15) & ~15ull);
      s_bytes[di] = total < 60000u ? (uint32_t)by : RS_EMPTY;  // longer: walked in the BSR
      s_scale[di] = SCH && S.fac_scale ? S.fac_scale[d0 + di] : 1.f;
    }
  }
  // isolated vertices: one without couplings, with b = 0 and a finite block keeps x = r = z = p = 0
  // exactly, so only the others ("live") are iterated; listed in order by one warp
  __syncthreads();
  const uint32_t H = min(s_nh, RS_MAX_HALO);
  float4* xs = reinterpret_cast<float4*>(smem + TEAMS * TEAM_BYTES);  // p of own vertices, then of the halo
  float* rv = reinterpret_cast<float*>(xs + own + H);
  float* az = rv + 3 * own;  // Ap after the rows, z after the preconditioner
  float* xv = az + 3 * own;  // the solution
  uint32_t* hpos = reinterpret_cast<uint32_t*>(xv + 3 * own);
  uint32_t* lv = hpos + H;
  for (uint32_t h = tid; h < RS_HASH; h += RS_THREADS)
    if (hval[h]) hpos[hval[h] - 1] = hkey[h];
  if (wid == 0) {
    uint32_t n = 0;
    for (uint32_t i0 = 0; i0 < nq; i0 += 32) {
      bool live = false;
      uint32_t v = 0;
      if (i0 + lane < nq) {
        v = S.dom_verts[Q0 + i0 + lane];
        const uint32_t k0 = S.rp[v], k1 = S.rp[v + 1];
        live = !(S.b[3 * v] == 0.f && S.b[3 * v + 1] == 0.f && S.b[3 * v + 2] == 0.f) || k1 - k0 > 1 ||
               (S.crp && S.crp[v + 1] > S.crp[v]);
        live = live || (k1 > k0 && !rs_block_finite(S.val + 9 * (size_t)k0));
        if (!live) {
          st_rec(a.rec + 2 * (size_t)(Q0 + i0 + lane), 0.f, 0.f, 0.f, RS_ALWAYS);
          st_rec(a.rec + 2 * (size_t)(Q0 + i0 + lane) + 1, 0.f, 0.f, 0.f, RS_ALWAYS);
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, live);
      if (live) lv[n + __popc(m & ((1u << lane) - 1u))] = i0 + lane;
      n += __popc(m);
    }
    if (lane == 0) s_nlive = n;
  }
  __syncthreads();
  const uint32_t nlive = s_nlive;
  float* lp = reinterpret_cast<float*>(lv + nlive);
  float* lr = lp + 3 * nlive;
  float* lz = lr + 3 * nlive;
  float* lx = lz + 3 * nlive;
  if (tid == 0) {
    // where the packed rows and the tiles are kept: all in shared memory if they fit there, else
    // with a staging buffer per team and as much of the rest as fits
    uint32_t cur = (uint32_t)((((unsigned char*)(lx + 3 * nlive) - smem) + 15u) & ~15u);
    uint64_t all = cur;
    for (int di = 0; di < nD; ++di) {
      all += s_bytes[di] == RS_EMPTY ? 0u : s_bytes[di];
      all += SCH ? (S.fac_off[d0 + di + 1] - S.fac_off[d0 + di]) * sizeof(TS) : (36u * (s_dpos[di + 1] - s_dpos[di]) + 15u) & ~15u;
    }
    uint32_t top = a.smem_bytes;
    if (all > a.smem_bytes && cur + 2 * TEAMS * RS_CHUNK <= a.smem_bytes)
      top -= 2 * TEAMS * RS_CHUNK;
    s_stage = top < a.smem_bytes ? top : 0u;
    const uint32_t lim = min(top, a.smem_bytes - RS_HASH_BYTES);
    for (int di = 0; di < nD; ++di) {
      const uint32_t bytes = s_bytes[di];
      s_jmode[di] = 2;
      if (bytes == RS_EMPTY) continue;
      if (cur + (uint64_t)bytes <= lim) {
        s_jmode[di] = 0;
        s_jofs[di] = cur;
        cur += bytes;
      } else if (s_stage && bytes - 1280u * s_wide[di] <= RS_CHUNK) {
        const uint32_t at = atomicAdd(a.jtop, bytes / 16);
        if (at <= a.jcap && bytes / 16 <= a.jcap - at) {
          s_jmode[di] = 1;
          s_jofs[di] = at;
        }
      }
    }
    s_nh = cur;  // where the tiles may begin
  }
  __syncthreads();
  auto jbase = [&](int di) -> float* {
    return s_jmode[di] ? a.jscr + 4 * (size_t)s_jofs[di] : reinterpret_cast<float*>(smem + s_jofs[di]);
  };
  for (int u = wid; u < TW * nD; u += RS_WARPS) {
    const int di = u / TW, uq = u - TW * di;
    if (s_jmode[di] == 2) continue;  // uniform
    const uint32_t len = s_len[32 * di + lane], maxlen = s_len[32 * di], wide = s_wide[di], nt = s_tail[di];
    const uint32_t row = s_row[32 * di + lane];
    float* jv = jbase(di);
    float* tv = jv + 320 * (size_t)wide;
    uint32_t k0 = 0, nps = 0, c0 = 0;
    if (len) {
      const uint32_t v = vert(P0 + s_dpos[di] + row);
      k0 = S.rp[v];
      nps = S.rp[v + 1] - k0;
      c0 = S.crp ? S.crp[v] : 0u;
    }
    bool far = false;
    auto fetch = [&](uint32_t sj, float (&m)[9]) -> uint32_t {  // the row's block sj and its column's slot
      const bool ps = sj < nps;
      const size_t k = ps ? k0 + sj : c0 + (sj - nps);
      const float* src = (ps ? S.val : S.cval) + 9 * k;
#pragma unroll
      for (int e = 0; e < 9; ++e) {
        m[e] = src[e];
        if (sizeof(Acc) == 8) far = far || !rs_finite(m[e]);
      }
      const uint32_t pos = position(ps ? S.col[k] : S.ccol[k]);
      if (pos - P0 < own) return 16 * (pos - P0);
      uint32_t h = hash_of(pos);
      for (uint32_t probe = 0; probe < RS_PROBES && hkey[h] != RS_EMPTY; ++probe, h = (h + 1) & (RS_HASH - 1))
        if (hkey[h] == pos) {
          if (hval[h]) return 16 * (own + hval[h] - 1);
          break;
        }
      far = true;
      return 0;
    };
    for (uint32_t sj = uq; sj < wide; sj += TW) {
      float m[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
      uint32_t code = 0;
      if (sj < len) code = fetch(sj, m);
      float4* s4 = reinterpret_cast<float4*>(jv) + 80 * (size_t)sj;
      s4[lane] = make_float4(m[0], m[1], m[2], m[3]);
      s4[32 + lane] = make_float4(m[4], m[5], m[6], m[7]);
      reinterpret_cast<float2*>(s4 + 64)[lane] = make_float2(m[8], __uint_as_float(code));
    }
    uint32_t o = 0;
    for (uint32_t sj = wide; sj < maxlen; ++sj) {
      const uint32_t cnt = __popc(__ballot_sync(0xffffffffu, len > sj));
      if (sj % TW == (uint32_t)uq && (uint32_t)lane < cnt) {
        float m[9];
        const uint32_t code = fetch(sj, m);
#pragma unroll
        for (int e = 0; e < 9; ++e) tv[9 * o + e * cnt + lane] = m[e];
        reinterpret_cast<uint32_t*>(tv + 9 * (size_t)nt)[o + lane] = code;
      }
      o += cnt;
    }
    // a column without a slot, or a value that rs_widen cannot take: the domain is walked in the BSR
    if (far) s_far[di] = 1;
  }
  // what follows reads the scratch and rewrites the hash table's place with bulk copies
  asm volatile("fence.proxy.async;" ::: "memory");
  __syncthreads();
  // the domains' tiles (block Jacobi: 3x3 inverses) into what is left of shared memory
  if (tid == 0) {
    uint32_t cur = s_nh;
    const uint32_t top = s_stage ? s_stage : a.smem_bytes;
    for (int di = 0; di < nD; ++di) {
      if (s_far[di]) s_jmode[di] = 2;
      const uint32_t nvd = s_dpos[di + 1] - s_dpos[di];
      const uint32_t bytes =
          SCH ? (uint32_t)((S.fac_off[d0 + di + 1] - S.fac_off[d0 + di]) * sizeof(TS)) : (36u * nvd + 15u) & ~15u;
      const bool in = cur + bytes <= top;
      s_tofs[di] = in ? cur : RS_EMPTY;
      if (in) cur += bytes;
    }
  }
  __syncthreads();
  for (int di = team; di < nD; di += TEAMS) {
    if (SCH && sizeof(AA) == 8) {
      // a tile that has no FP64 image by shifts: its domain's z is NaN, as its product would be
      const uint32_t n = (uint32_t)((S.fac_off[d0 + di + 1] - S.fac_off[d0 + di]) * sizeof(TS) / 4);
      const uint32_t* src = (const uint32_t*)((const TS*)S.fac + S.fac_off[d0 + di]);
      bool bad = false;
      for (uint32_t i = ti; i < n; i += TEAM) {
        const uint32_t w = __ldg(src + i);
        bad = bad || (sizeof(TS) == 4 ? (w & 0x7f800000u) == 0x7f800000u
                                      : (w & 0x7c00u) == 0x7c00u || (w & 0x7c000000u) == 0x7c000000u);
      }
      if (bad) s_scale[di] = __uint_as_float(0x7fffffffu);
    }
    if (s_tofs[di] == RS_EMPTY) continue;
    if (SCH) {
      const uint32_t n16 = (uint32_t)((S.fac_off[d0 + di + 1] - S.fac_off[d0 + di]) * sizeof(TS)) / 16;
      const uint4* src = reinterpret_cast<const uint4*>((const TS*)S.fac + S.fac_off[d0 + di]);
      uint4* dst = reinterpret_cast<uint4*>(smem + s_tofs[di]);
      for (uint32_t i = ti; i < n16; i += TEAM) dst[i] = __ldg(src + i);
    } else {
      const uint32_t nf = 9 * (s_dpos[di + 1] - s_dpos[di]);
      const float* src = S.bjinv + 9 * (size_t)(P0 + s_dpos[di]);
      float* dst = reinterpret_cast<float*>(smem + s_tofs[di]);
      for (uint32_t i = ti; i < nf; i += TEAM) dst[i] = __ldg(src + i);
    }
  }

  unsigned char* tscr = smem + team * TEAM_BYTES;
  uint4* sums = a.sums + I.cta0;
  uint32_t* count = a.count + 32 * ii;
  uint32_t target = 0;  // the counter once all have published

  // ---- staging: the rows and tiles of a team's domains that are not resident go round its two
  // buffers in chunks, in the order they are needed; a chunk's copy starts as soon as the team
  // has used the one two places before it, so copies run under the other phase and the exchanges
  const bool stage_tiles = SCH && sizeof(TS) == 2;  // FP32 tiles are read from L2 instead
  unsigned char* sbuf = smem + s_stage + 2 * team * RS_CHUNK;
  uint32_t taken = 0;  // chunks used; the same in all threads of a team
  auto staged_row = [&](int di) { return s_jmode[di] == 1; };
  auto staged_tile = [&](int di) { return stage_tiles && s_stage && s_tofs[di] == RS_EMPTY; };
  // rows' chunks: runs of whole slots, the blocks past them in the last run's chunk if they fit
  auto row_chunks = [&](int di, bool& joined) -> uint32_t {
    const uint32_t wide = s_wide[di], tail = s_bytes[di] - 1280u * wide;
    const uint32_t nw = (wide + CHUNK_SLOTS - 1) / CHUNK_SLOTS;
    joined = nw > 0 && 1280u * (wide - (nw - 1) * CHUNK_SLOTS) + tail <= RS_CHUNK;
    return nw + ((tail && !joined) ? 1u : 0u);
  };
  auto stage_issue = [&]() {  // the team's first thread
    if (ti != 0 || !s_stage) return;
    StageNext n = s_sg[team];
    for (int turn = 0; turn < 3; ++turn) {
      for (; n.di < nD; n.di += TEAMS) {
        if (!(n.tiles ? staged_tile(n.di) : staged_row(n.di))) continue;
        const unsigned char* src;
        uint32_t bytes;
        bool last = true;
        if (n.tiles) {
          const uint64_t f0 = S.fac_off[d0 + n.di];
          src = reinterpret_cast<const unsigned char*>((const TS*)S.fac + f0);
          bytes = (uint32_t)((S.fac_off[d0 + n.di + 1] - f0) * sizeof(TS));
        } else {
          bool joined;
          const uint32_t nc = row_chunks(n.di, joined);
          const uint32_t start = min(1280u * CHUNK_SLOTS * n.part, 1280u * s_wide[n.di]);
          last = n.part + 1 == nc;
          src = reinterpret_cast<const unsigned char*>(a.jscr + 4 * (size_t)s_jofs[n.di]) + start;
          bytes = last ? s_bytes[n.di] - start : min(1280u * CHUNK_SLOTS, 1280u * s_wide[n.di] - start);
        }
        uint64_t* bar = &s_bar[2 * team + (n.issued & 1u)];
        mbar_arrive_expect_tx(bar, bytes);
        bulk_g2s(sbuf + (n.issued & 1u) * RS_CHUNK, src, bytes, bar);
        ++n.issued;
        ++n.part;
        if (last) {
          n.di += TEAMS;
          n.part = 0;
        }
        s_sg[team] = n;
        return;
      }
      n.tiles = !n.tiles;
      n.di = team;
    }
  };
  // waits for the next chunk and returns its buffer
  auto stage_wait = [&]() -> const unsigned char* {
    uint64_t* bar = &s_bar[2 * team + (taken & 1u)];
    const uint32_t ph = (taken >> 1) & 1u;
    if (!mbar_wait(bar, ph)) {
      s_abort = 1;
      if (ti == 0) atomicOr(&a.out[I.k].status, ST_WAIT_TIMEOUT);
      mbar_wait(bar, ph);  // bounded again: the copy may still land
    }
    const unsigned char* b = sbuf + (taken & 1u) * RS_CHUNK;
    ++taken;
    return b;
  };

  // Sums v over the instance: block sum, publish it with its epoch, count up, wait until all CTAs
  // of the instance have, sum theirs in CTA order. Valid in warp 0. One lane per CTA polls one
  // counter (all lanes polling the sums themselves queue at the lines they share: 7.5 thousand
  // cycles for 148 CTAs against 2.4 thousand; a mailbox per CTA, written by all others, took 3
  // to 5 thousand). Nothing is fenced: a sum or record that is read too early has the wrong epoch
  // and is read again. fence: also orders the CTA's earlier stores before.
  auto exchange = [&](uint32_t epoch, Acc v0, Acc v1, bool two, bool fence, double& t0, double& t1) {
    v0 = warp_sum(v0);
    if (two) v1 = warp_sum(v1);
    if (lane == 0) {
      s_red[0][wid] = v0;
      s_red[1][wid] = v1;
    }
    __syncthreads();
    target += G;
    if (wid == 0) {
      const double b0 = (double)warp_sum(lane < RS_WARPS ? s_red[0][lane] : Acc(0));
      const double b1 = two ? (double)warp_sum(lane < RS_WARPS ? s_red[1][lane] : Acc(0)) : 0.0;
      uint4* at = sums + (two ? RS_MAX_G : 0);
      bool ok = true;
      if (lane == 0) {
        if (fence) __threadfence();
        st_rlx(at + j, make_uint4(__double2loint(b0), __double2hiint(b0), epoch, 0u));
        if (two) st_rlx(at + RS_MAX_G + j, make_uint4(__double2loint(b1), __double2hiint(b1), epoch, 0u));
        asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        uint32_t seen;
        for (uint32_t tries = 0;; ++tries) {
          asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
          if ((int)(seen - target) >= 0) break;
          if (tries > RS_EXCHANGE_POLLS) {
            ok = false;
            break;
          }
        }
      }
      __syncwarp();
      constexpr int PER = RS_MAX_G / 32;
      double p0[PER], p1[PER];
      for (uint32_t tries = 0;; ++tries) {
        bool here = true;
#pragma unroll
        for (int u = 0; u < PER; ++u) {
          const uint32_t c = lane + 32 * u;
          p0[u] = 0.0;
          p1[u] = 0.0;
          if (c < G) {
            const uint4 r0 = ld_rlx(at + c);
            here = here && r0.z == epoch;
            p0[u] = __hiloint2double((int)r0.y, (int)r0.x);
            if (two) {
              const uint4 r1 = ld_rlx(at + RS_MAX_G + c);
              here = here && r1.z == epoch;
              p1[u] = __hiloint2double((int)r1.y, (int)r1.x);
            }
          }
        }
        here = __all_sync(0xffffffffu, here);
        if (here) break;
        if (tries > (1u << 20)) {
          ok = false;
          break;
        }
      }
      if (fence) __threadfence();
      t0 = 0.0;
      t1 = 0.0;
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        t0 += p0[u];
        t1 += p1[u];
      }
      t0 = warp_sum(t0);
      if (two) t1 = warp_sum(t1);
      if (!__all_sync(0xffffffffu, ok) && lane == 0) {
        atomicOr(&a.out[I.k].status, ST_WAIT_TIMEOUT);
        s_abort = 1;
      }
    }
  };

  // p of a vertex from its record of this epoch (bounded wait for it)
  auto record = [&](size_t pos, uint32_t epoch, float be, float& x0, float& x1, float& x2) {
    uint4 z, p;
    for (uint32_t tries = 0;; ++tries) {
      z = ld_rlx(a.rec + 2 * pos);
      p = ld_rlx(a.rec + 2 * pos + 1);
      if ((z.w == epoch || z.w == RS_ALWAYS) && (p.w == epoch || p.w == RS_ALWAYS)) break;
      if (tries > RS_RECORD_POLLS) {
        atomicOr(&a.out[I.k].status, ST_WAIT_TIMEOUT);
        s_abort = 1;
        break;
      }
    }
    x0 = fmaf(be, __uint_as_float(p.x), __uint_as_float(z.x));
    x1 = fmaf(be, __uint_as_float(p.y), __uint_as_float(z.y));
    x2 = fmaf(be, __uint_as_float(p.z), __uint_as_float(z.z));
  };

  // one row's product with the matrix as it lies in the BSR (blocks from sj on, every step-th),
  // every x read as z + beta p from the records
  auto bsr_row = [&](uint32_t v, uint32_t sj, uint32_t step, uint32_t epoch, float be, Acc& y0, Acc& y1, Acc& y2) {
    const uint32_t k0 = S.rp[v], nps = S.rp[v + 1] - k0, c0 = S.crp ? S.crp[v] : 0u;
    const uint32_t len = nps + (S.crp ? S.crp[v + 1] - c0 : 0u);
    for (; sj < len; sj += step) {
      const bool ps = sj < nps;
      const size_t k = ps ? k0 + sj : c0 + (sj - nps);
      const float* m = (ps ? S.val : S.cval) + 9 * k;
      float f0, f1, f2;
      record(position(ps ? S.col[k] : S.ccol[k]), epoch, be, f0, f1, f2);
      const Acc x0 = (Acc)f0, x1 = (Acc)f1, x2 = (Acc)f2;
      y0 = rs_fma((Acc)m[0], x0, y0);
      y0 = rs_fma((Acc)m[1], x1, y0);
      y0 = rs_fma((Acc)m[2], x2, y0);
      y1 = rs_fma((Acc)m[3], x0, y1);
      y1 = rs_fma((Acc)m[4], x1, y1);
      y1 = rs_fma((Acc)m[5], x2, y1);
      y2 = rs_fma((Acc)m[6], x0, y2);
      y2 = rs_fma((Acc)m[7], x1, y2);
      y2 = rs_fma((Acc)m[8], x2, y2);
    }
  };

  // component e % 3 of own vertex e / 3's p
  auto xsc = [&](uint32_t e) -> float& { return reinterpret_cast<float*>(xs)[e + e / 3]; };

  // rows: Ap of the own domains into az, p.Ap
  auto rows_phase = [&](uint32_t epoch, float be) -> Acc {
    for (uint32_t h = tid; h < H; h += RS_THREADS) {
      float x0, x1, x2;
      record(hpos[h], epoch, be, x0, x1, x2);
      xs[own + h] = make_float4(x0, x1, x2, 0.f);
    }
    for (uint32_t v = tid; v < own; v += RS_THREADS) {
      const float4 p = xs[v];
      xs[v] = make_float4(fmaf(be, p.x, az[3 * v]), fmaf(be, p.y, az[3 * v + 1]), fmaf(be, p.z, az[3 * v + 2]), 0.f);
    }
    for (uint32_t e = tid; e < 3 * nlive; e += RS_THREADS) lp[e] = fmaf(be, lp[e], lz[e]);
    __syncthreads();
    Acc acc = 0;
    Acc* part = reinterpret_cast<Acc*>(tscr);  // [TW][96]
    for (int di = team; di < nD; di += TEAMS) {
      const uint32_t row = s_row[32 * di + lane], dp = s_dpos[di], dn = s_dpos[di + 1], wide = s_wide[di];
      const int mode = s_jmode[di];
      Acc y0 = 0, y1 = 0, y2 = 0;
      if (mode == 2) {
        if (dp + row < dn) bsr_row(vert(P0 + dp + row), q, TW, epoch, be, y0, y1, y2);
      } else {
        const unsigned char* xb = reinterpret_cast<const unsigned char*>(xs);
        // whole slots q, q + 3, .. below `n` of the run at `jv`
        auto whole = [&](const unsigned char* jv, uint32_t n) {
#pragma unroll 2
          for (uint32_t sj = q; sj < n; sj += TW) {
            const float4* s4 = reinterpret_cast<const float4*>(jv) + 80 * sj + lane;
            const float4 ma = s4[0], mb = s4[32];
            const float2 mc = *reinterpret_cast<const float2*>(jv + 1280 * sj + 1024 + 8 * lane);
            const float4 x = *reinterpret_cast<const float4*>(xb + __float_as_uint(mc.y));
            const Acc x0 = rs_lift((Acc)x.x), x1 = rs_lift((Acc)x.y), x2 = rs_lift((Acc)x.z);
            y0 = rs_fma(rs_widen(ma.x, Acc(0)), x0, y0);
            y1 = rs_fma(rs_widen(ma.w, Acc(0)), x0, y1);
            y2 = rs_fma(rs_widen(mb.z, Acc(0)), x0, y2);
            y0 = rs_fma(rs_widen(ma.y, Acc(0)), x1, y0);
            y1 = rs_fma(rs_widen(mb.x, Acc(0)), x1, y1);
            y2 = rs_fma(rs_widen(mb.w, Acc(0)), x1, y2);
            y0 = rs_fma(rs_widen(ma.z, Acc(0)), x2, y0);
            y1 = rs_fma(rs_widen(mb.y, Acc(0)), x2, y1);
            y2 = rs_fma(rs_widen(mc.x, Acc(0)), x2, y2);
          }
        };
        // the blocks of slots that few rows have
        auto rest = [&](const float* tv) {
          const uint32_t nt = s_tail[di], len = s_len[32 * di + lane], maxlen = s_len[32 * di];
          uint32_t o = 0;
          for (uint32_t sj = wide; sj < maxlen; ++sj) {
            const uint32_t cnt = __popc(__ballot_sync(0xffffffffu, len > sj));
            if (sj % TW == (uint32_t)q && (uint32_t)lane < cnt) {
              const float* m = tv + 9 * o + lane;
              const float4 x = *reinterpret_cast<const float4*>(
                  xb + reinterpret_cast<const uint32_t*>(tv + 9 * (size_t)nt)[o + lane]);
              const Acc x0 = rs_lift((Acc)x.x), x1 = rs_lift((Acc)x.y), x2 = rs_lift((Acc)x.z);
              y0 = rs_fma(rs_widen(m[0], Acc(0)), x0, y0);
              y1 = rs_fma(rs_widen(m[3 * cnt], Acc(0)), x0, y1);
              y2 = rs_fma(rs_widen(m[6 * cnt], Acc(0)), x0, y2);
              y0 = rs_fma(rs_widen(m[cnt], Acc(0)), x1, y0);
              y1 = rs_fma(rs_widen(m[4 * cnt], Acc(0)), x1, y1);
              y2 = rs_fma(rs_widen(m[7 * cnt], Acc(0)), x1, y2);
              y0 = rs_fma(rs_widen(m[2 * cnt], Acc(0)), x2, y0);
              y1 = rs_fma(rs_widen(m[5 * cnt], Acc(0)), x2, y1);
              y2 = rs_fma(rs_widen(m[8 * cnt], Acc(0)), x2, y2);
            }
            o += cnt;
          }
        };
        if (mode == 0) {
          const unsigned char* jv = smem + s_jofs[di];
          whole(jv, wide);
          if (s_tail[di]) rest(reinterpret_cast<const float*>(jv + 1280 * (size_t)wide));
        } else {
          bool joined;
          const uint32_t n = row_chunks(di, joined);
          for (uint32_t c = 0; c < n; ++c) {
            const unsigned char* b = stage_wait();
            const uint32_t first = min(CHUNK_SLOTS * c, wide), here = min(CHUNK_SLOTS, wide - first);
            whole(b, here);  // runs are a multiple of three slots: the same split between the warps
            if (c + 1 == n && s_tail[di]) rest(reinterpret_cast<const float*>(b + 1280 * (size_t)here));
            if (c + 1 < n) {
              team_sync(team);
              stage_issue();
            }
          }
        }
        y0 = rs_lift(y0);
        y1 = rs_lift(y1);
        y2 = rs_lift(y2);
      }
      Acc* mine = part + 96 * q + 3 * row;
      mine[0] = y0;
      mine[1] = y1;
      mine[2] = y2;
      team_sync(team);
      if (mode == 1) stage_issue();
      if (3 * dp + ti < 3 * dn) {
        Acc y = part[ti];
#pragma unroll
        for (int u = 1; u < TW; ++u) y += part[96 * u + ti];
        const float f = (float)y;
        az[3 * dp + ti] = f;
        acc += (Acc)xsc(3 * dp + ti) * (Acc)f;
      }
      if (di + TEAMS < nD) team_sync(team);
    }
    for (uint32_t l = tid; l < nlive; l += RS_THREADS) {
      Acc y0 = 0, y1 = 0, y2 = 0;
      bsr_row(S.dom_verts[Q0 + lv[l]], 0, 1, epoch, be, y0, y1, y2);
      const float f0 = (float)y0, f1 = (float)y1, f2 = (float)y2;
      lz[3 * l] = f0;
      lz[3 * l + 1] = f1;
      lz[3 * l + 2] = f2;
      acc += (Acc)lp[3 * l] * (Acc)f0 + (Acc)lp[3 * l + 1] * (Acc)f1 + (Acc)lp[3 * l + 2] * (Acc)f2;
    }
    return acc;
  };

  // preconditioner: x, r updated (init: r = b), z into az and the records, r.r and r.z
  auto precond_phase = [&](bool init, uint32_t epoch, Acc& rr, Acc& rz) {
    const float al = s_alpha;
    rr = 0;
    rz = 0;
    float* rd = reinterpret_cast<float*>(tscr);
    AA* part = reinterpret_cast<AA*>(tscr + 384);  // [6][32]
    AA* yd = part + 192;
    for (int di = team; di < nD; di += TEAMS) {
      const uint32_t dp = s_dpos[di], m = 3 * (s_dpos[di + 1] - dp), e = 3 * dp + ti;
      const int T = ((int)m + 31) >> 5;
      const TS* w = nullptr;
      const bool staged = staged_tile(di);
      if (SCH) {
        w = staged ? reinterpret_cast<const TS*>(stage_wait())
                   : (s_tofs[di] != RS_EMPTY ? reinterpret_cast<const TS*>(smem + s_tofs[di])
                                             : (const TS*)S.fac + S.fac_off[d0 + di]);
      }
      // warp q's tiles are tiles q and (teams of three) q + 3, zero past the domain's: one code path
      // for all
      TileRegs<AA, TS> ta, tb;
      auto load = [&](TileRegs<AA, TS>& t, int at) {
        if (at < T * (T + 1) / 2)
          t.load(w + at * TILE_FLOATS, lane);
        else
          t.zero();
      };
      constexpr bool KEEP = sizeof(TS) == 2 && sizeof(AA) == 4;  // in registers for both passes
      if (SCH && KEEP) {
        load(ta, q);
        if (TW == 3) load(tb, q + 3);
      }
      float r = 0.f, p = 0.f;
      if ((uint32_t)ti < m) {
        if (init) {
          r = S.b[3 * vert(P0 + dp + ti / 3) + ti % 3];
          xsc(e) = 0.f;
          xv[e] = 0.f;
        } else {
          p = xsc(e);
          xv[e] = fmaf(al, p, xv[e]);
          r = fmaf(-al, az[e], rv[e]);
        }
        rv[e] = r;
      }
      if (TW == 3 || ti < 96) rd[ti] = r;
      team_sync(team);
      if (KEEP && staged) stage_issue();  // the tiles are in registers
      float zi = 0.f;
      if (SCH) {
        int at;
        if (!KEEP) load(ta, q);
        AA v = ta.rows(rd + 32 * rs_tile_j(q), lane, at);
        AA v2 = 0;
        if (TW == 3) {
          if (!KEEP) load(tb, q + 3);
          v2 = tb.rows(rd + 32 * rs_tile_j(q + 3), lane, at);
        }
        part[32 * q + at] = v;
        if (TW == 3) part[32 * (q + 3) + at] = v2;
        team_sync(team);
        if (TW == 3 || q < 3) {  // y of tile row q: its tiles' partials in storage order
          const AA* pr = part + 32 * (q * (q + 1) / 2) + lane;
          AA y = pr[0];
          if (q > 0) y += pr[32];
          if (q > 1) y += pr[64];
          yd[ti] = y;
        }
        team_sync(team);
        if (!KEEP && (TW == 3 || sizeof(AA) == 8)) load(ta, q);
        v = ta.cols(yd + 32 * rs_tile_i(q), lane, at);
        if (TW == 3) {
          if (!KEEP) load(tb, q + 3);
          v2 = tb.cols(yd + 32 * rs_tile_i(q + 3), lane, at);
        }
        part[32 * q + at] = v;
        if (TW == 3) part[32 * (q + 3) + at] = v2;
        team_sync(team);
        if (!KEEP && staged) stage_issue();
        if (TW == 3 || q < 3) {  // z of tile column q
          AA z = part[32 * (q * (q + 1) / 2 + q) + lane];
          if (q < 2) z += part[32 * ((q + 1) * (q + 2) / 2 + q) + lane];
          if (q < 1) z += part[32 * 3 + lane];
          const AA sc = (AA)s_scale[di];
          zi = (float)(z * sc * sc);
        }
      } else if ((uint32_t)ti < m) {
        const uint32_t lvx = ti / 3, c = ti - 3 * lvx;
        const float* w9 = s_tofs[di] != RS_EMPTY ? reinterpret_cast<const float*>(smem + s_tofs[di]) + 9 * lvx
                                                 : S.bjinv + 9 * (size_t)(P0 + dp + lvx);
        zi = w9[3 * c] * rd[3 * lvx] + w9[3 * c + 1] * rd[3 * lvx + 1] + w9[3 * c + 2] * rd[3 * lvx + 2];
      }
      if ((uint32_t)ti < m) {
        az[e] = zi;
        rr += (Acc)r * (Acc)r;
        rz += (Acc)r * (Acc)zi;
      }
      team_sync(team);
      // records: z by one warp of the team, p by another
      if (q < 2 && 3 * (uint32_t)lane < m) {
        const uint32_t v = dp + lane;
        float4* rec = a.rec + 2 * (size_t)(P0 + v) + q;
        if (q == 0) {
          st_rec(rec, az[3 * v], az[3 * v + 1], az[3 * v + 2], epoch);
        } else {
          const float4 pv = xs[v];
          st_rec(rec, pv.x, pv.y, pv.z, epoch);
        }
      }
    }
    for (uint32_t l = tid; l < nlive; l += RS_THREADS) {
      const uint32_t pos = Q0 + lv[l], v = S.dom_verts[pos];
      float r3[3], z3[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (init) {
          r3[c] = S.b[3 * v + c];
          lp[3 * l + c] = 0.f;
          lx[3 * l + c] = 0.f;
        } else {
          lx[3 * l + c] = fmaf(al, lp[3 * l + c], lx[3 * l + c]);
          r3[c] = fmaf(-al, lz[3 * l + c], lr[3 * l + c]);
        }
        lr[3 * l + c] = r3[c];
      }
      Acc zz[3];
      vertex_apply<Acc>(S.vfac + 6 * (size_t)v, r3, zz);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        z3[c] = (float)zz[c];
        lz[3 * l + c] = z3[c];
        rr += (Acc)r3[c] * (Acc)r3[c];
        rz += (Acc)r3[c] * (Acc)z3[c];
      }
      st_rec(a.rec + 2 * (size_t)pos, z3[0], z3[1], z3[2], epoch);
      st_rec(a.rec + 2 * (size_t)pos + 1, lp[3 * l], lp[3 * l + 1], lp[3 * l + 2], epoch);
    }
  };

  __syncthreads();  // tiles in place
  stage_issue();
  stage_issue();
  // iteration 0 is the start: z = M^-1 b, ||b||, r.z
  for (uint32_t it = 0;; ++it) {
    Acc v0, v1;
    double t0, t1;
    if (it > 0) {
      v0 = rows_phase(a.epoch + it, s_beta);
      exchange(a.epoch + it, v0, Acc(0), false, false, t0, t1);
      if (tid == 0) {
        if (!(t0 > 0.0)) {  // the reference breaks out (linsolve.rs:386)
          s_done = 1;
          s_status = ST_PCG_BREAKDOWN;
        } else {
          s_alpha = (float)quotient(s_rz, t0);  // a p.Ap that overflowed takes no step
        }
      }
      __syncthreads();
      if (s_abort || s_done) break;
    }
    precond_phase(it == 0, a.epoch + it + 1, v0, v1);
    // the first exchange is fenced: it orders the records that hold for the whole solve
    exchange(a.epoch + it + 1, v0, v1, true, it == 0, t0, t1);
    if (tid == 0) {
      s_iters = it;
      s_rr = t0;
      if (it == 0) {
        const double bnorm = fmax(sqrt(t0), 1e-30), lim = (double)a.tol * bnorm;
        s_rz = t1;
        s_bnorm = bnorm;
        s_lim2 = lim * lim * (1.0 + 1e-12);
      } else if (it >= a.max_iter || (t0 <= s_lim2 && sqrt(t0) / s_bnorm <= (double)a.tol)) {
        s_done = 1;  // the residual itself is only formed where it can be within the tolerance
      } else {
        s_beta = (float)quotient(t1, s_rz);
        s_rz = t1;
      }
    }
    __syncthreads();
    if (s_abort || s_done) break;
  }
  while (s_stage && taken < s_sg[team].issued) stage_wait();  // no copy may outlive the CTA
  for (uint32_t e = tid; e < 3 * own; e += RS_THREADS) a.x[3 * vert(P0 + e / 3) + e % 3] = xv[e];
  for (uint32_t e = tid; e < 3 * nlive; e += RS_THREADS) a.x[3 * S.dom_verts[Q0 + lv[e / 3]] + e % 3] = lx[e];
  if (j == 0 && tid == 0) {
    FusedInst& o = a.out[I.k];
    o.rz = s_rz;
    o.bnorm = s_bnorm;
    o.residual = sqrt(s_rr) / s_bnorm;
    o.iters = s_iters;
    o.done = 1;
    atomicOr(&o.status, s_status);
  }
}

__global__ void k_rs_reset(uint32_t* __restrict__ count, FusedInst* __restrict__ out, uint32_t K, float* __restrict__ x,
                           uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, st = gridDim.x * blockDim.x;
  if (count && i <= 32 * PCG_MAX_INST) count[i] = 0;  // the counters and the scratch's top
  for (uint32_t e = i; e < n; e += st) x[e] = 0.f;
  if (i < K) out[i] = FusedInst{};
}

bool resident_domains(const mguso_schwarz& s, RsRun& run) {
  uint32_t d = 0;
  for (uint32_t k = 0; k < run.ninst; ++k) {
    run.dom[k] = d;
    auto inside = [&](uint32_t q) {
      const uint32_t v = s.h_dom_verts[s.h_dom_start[q]];
      return v >= run.vert[k] && v < run.vert[k + 1];
    };
    while (d < s.ndom && inside(d) && !s.h_dom_diag[d]) ++d;
    run.diag[k] = d;
    while (d < s.ndom && inside(d) && s.h_dom_diag[d]) ++d;
  }
  run.dom[run.ninst] = d;
  return d == s.ndom;
}

// The most blocks that one of instance k's CTAs would walk in the BSR, because their rows are neither
// resident nor staged or its halo outgrows the table; found as the kernel's set-up places rows
// (without contact blocks, which only the device knows, and isolated vertices, which bear no load in
// a scene). A walked block costs two polled records, 4 ns of its CTA's time, for which the others
// wait, so a chip full of them loses to the other PCGs. us an iteration, resident and the other
// (in brackets: thousands of blocks walked by the worst CTA):
//   scenes, Schwarz, mixed: 300 x 300 sheet (0) 24, 37; six garments (0) 31, 53; seven (11) 88, 60; eight 102, 73;
//   scenes, block Jacobi: 300 x 300 sheet (0) 20, 27; 360 x 360 (9) 39, 29; five garments 42, 29; 545 x
//     545 sheet 134, 53;
//   solver, Schwarz, mixed: 360 x 360 grid (7 blocks a row; 0) 51, 78; 400 x 400 (4.9) 81, 89; 440 (6.9) 102,
//     102; 480 (9.1) 121, 116; 330 x 330 with 13 blocks a row (0) 48, 76, 360 (8.9) 95, 88; 20 thousand
//     vertices with 8 random neighbours each (3.7, halo of 3 300) 44, 40, 40 thousand (7.5) 82, 52;
//   solver, block Jacobi, mixed: 400 (4.9) 26, 40; 480 (8.9) 38, 47; 520 (11) 46, 56; with 13 blocks a row
//     400 (12) 53, 54, 440 (15) 74, 65; 90 thousand vertices with random neighbours (5.5) 38, 44.
// So scenes, whose other PCG takes two launches an iteration, allow WALKED_SCENE blocks; the solver, whose
// other takes four over vectors in memory, walked_solver.
static uint32_t resident_walked(const mguso_bsr& a, const mguso_schwarz* sw, const RsRun& run, uint32_t k,
                                uint32_t ncta, uint32_t smem, uint32_t stage) {
  const uint32_t v0 = run.vert[k], nv = run.vert[k + 1] - v0;
  const uint32_t dn0 = sw ? run.dom[k] : 0, nd = sw ? run.diag[k] - dn0 : ceil_div(nv, 32);
  auto dstart = [&](uint32_t d) { return sw ? sw->h_dom_start[dn0 + d] : v0 + std::min(32 * d, nv); };
  auto vert = [&](uint32_t pos) { return sw ? sw->h_dom_verts[pos] : pos; };
  auto share = [&](uint32_t j) { return (uint32_t)((uint64_t)nd * j / ncta); };
  std::vector<uint32_t> owner(nv, ncta), seen(nv, ncta);
  for (uint32_t j = 0; j < ncta; ++j)
    for (uint32_t pos = dstart(share(j)); pos < dstart(share(j + 1)); ++pos) owner[vert(pos) - v0] = j;
  struct Dom {
    uint64_t bytes, tail;
    uint32_t blocks;
  };
  std::vector<Dom> doms;
  uint32_t worst = 0;
  for (uint32_t j = 0; j < ncta; ++j) {
    uint64_t own = 0, halo = 0, need = 0, blocks = 0, walked = 0;
    doms.clear();
    for (uint32_t d = share(j); d < share(j + 1); ++d) {
      uint32_t len[32] = {}, n = 0;
      Dom m{0, 0, 0};
      for (uint32_t pos = dstart(d); pos < dstart(d + 1); ++pos) {
        const uint32_t v = vert(pos);
        m.blocks += len[n++] = a.h_row_ptr[v + 1] - a.h_row_ptr[v];
        for (uint32_t e = a.h_row_ptr[v]; e < a.h_row_ptr[v + 1]; ++e) {
          const uint32_t c = a.h_col[e] - v0;
          if (c >= nv || owner[c] == j || seen[c] == j) continue;
          seen[c] = j;
          ++halo;
        }
      }
      std::sort(len, len + n, [](uint32_t x, uint32_t y) { return x > y; });
      const uint32_t wide = len[RS_WIDE - 1];
      for (uint32_t i = 0; i < n; ++i) m.tail += len[i] - std::min(len[i], wide);
      m.tail = (40 * m.tail + 15) & ~15ull;
      m.bytes = 1280ull * wide + m.tail;
      const uint32_t T = (3 * n + 31) / 32;
      need += m.bytes + (sw ? (uint64_t)T * (T + 1) / 2 * TILE_FLOATS * (run.half ? 2 : 4) : (36ull * n + 15) & ~15ull);
      own += n;
      blocks += m.blocks;
      doms.push_back(m);
    }
    uint64_t cur = RS_SCRATCH + 52 * own + 20 * std::min<uint64_t>(halo, RS_MAX_HALO) + 16;
    const bool staged = cur + need > smem && cur + stage <= smem;
    const uint64_t lim = std::min(smem - (staged ? stage : 0u), smem - RS_HASH_BYTES);
    for (const Dom& m : doms) {
      if (m.blocks < 60000u && cur + m.bytes <= lim)
        cur += m.bytes;
      else if (!(m.blocks < 60000u && staged && m.tail <= RS_CHUNK))
        walked += m.blocks;
    }
    worst = std::max(worst, (uint32_t)(halo > RS_MAX_HALO ? blocks : walked));
  }
  return worst;
}

template <class Acc, class TS, int TW, class AA = Acc>
static void* schwarz_kernel() {
  return (void*)k_pcg_resident<MGUSO_PRECOND_SCHWARZ, Acc, TS, TW, AA>;
}

template <int TW>
static void* resident_kernel(const RsRun& run) {
  if (!run.half) return run.mixed ? schwarz_kernel<double, float, TW>() : schwarz_kernel<float, float, TW>();
  if (!run.mixed) return schwarz_kernel<float, __half, TW>();
  return run.fp64_tiles ? schwarz_kernel<double, __half, TW>() : schwarz_kernel<double, __half, TW, float>();
}

int pcg_resident(const RsSystem& sys, const mguso_bsr& bsr, const mguso_schwarz* sw, RsWork& w, const RsRun& run,
                 float* x, uint32_t active, float tol, uint32_t max_iter, FusedInst* out, cudaStream_t st) {
  const uint32_t K = run.ninst;
  MG_CHECK_ARG(K >= 1 && K <= PCG_MAX_INST, "resident PCG: 1..8 instances");
  // CTAs per active instance: one each, then one at a time to the instance with the most domains
  // per CTA, until the SMs or the domains run out
  RsArgs a{};
  uint32_t nd[PCG_MAX_INST], used = 0;
  for (uint32_t k = 0; k < K; ++k) {
    if (!((active >> k) & 1u)) continue;
    RsInst& I = a.inst[a.nrun];
    I.k = k;
    I.dn0 = run.dom[k];
    I.dn1 = run.diag[k];
    I.dd0 = run.diag[k];
    I.dd1 = run.dom[k + 1];
    I.v0 = run.vert[k];
    I.v1 = run.vert[k + 1];
    if (run.precond == MGUSO_PRECOND_BLOCK_JACOBI) {
      I.dn0 = 0;
      I.dn1 = ceil_div(I.v1 - I.v0, 32);
      I.dd0 = I.dd1 = 0;
    }
    nd[a.nrun] = I.dn1 - I.dn0;
    I.ncta = 1;
    ++a.nrun;
    ++used;
  }
  if (a.nrun == 0) {
    k_rs_reset<<<64, 256, 0, st>>>(nullptr, out, K, x, 3 * run.nv);
    MG_CUDA(cudaGetLastError());
    return MGUSO_OK;
  }
  const uint32_t sms = std::min<uint32_t>((uint32_t)run.sms, RS_MAX_G);
  if (used > sms) return MGUSO_ERR_UNSUPPORTED;
  while (used < sms) {
    int best = -1;
    for (uint32_t i = 0; i < a.nrun; ++i)
      if (a.inst[i].ncta < nd[i] &&
          (best < 0 || (uint64_t)nd[i] * a.inst[best].ncta > (uint64_t)nd[best] * a.inst[i].ncta))
        best = (int)i;
    if (best < 0) break;
    a.inst[best].ncta++;
    ++used;
  }
  uint32_t grid = 0, most = 0;  // most: domains of a CTA
  for (uint32_t i = 0; i < a.nrun; ++i) {
    a.inst[i].cta0 = grid;
    grid += a.inst[i].ncta;
    most = std::max(most, ceil_div(nd[i], a.inst[i].ncta));
  }
  // Schwarz: teams of six warps, a domain each, where three teams are enough. Time in the solves, three
  // -> six warps: 64 x 64 grid (one domain per CTA) 1.13 -> 0.97 ms, 100 x 100 (two or three) 2.05 ->
  // 1.89, a 64 x 64 sheet's step 3.89 -> 3.45; with four domains per CTA three teams take two
  // turns. Block Jacobi has no tiles to share and loses (100 x 100: 2.70 -> 2.76).
  const int wide = run.precond == MGUSO_PRECOND_SCHWARZ && most <= 3 ? 1 : 0;
  void* fn = run.precond == MGUSO_PRECOND_BLOCK_JACOBI
                 ? (run.mixed ? (void*)k_pcg_resident<MGUSO_PRECOND_BLOCK_JACOBI, double, float, 3, double>
                              : (void*)k_pcg_resident<MGUSO_PRECOND_BLOCK_JACOBI, float, float, 3, float>)
             : wide ? resident_kernel<6>(run)
                    : resident_kernel<3>(run);
  if (w.fn[wide] != fn) {
    w.fn[wide] = nullptr;
    w.smem[wide] = 0;
    int dev = 0, optin = 0, per_sm = 0;
    cudaFuncAttributes fa;
    MG_CUDA(cudaGetDevice(&dev));
    MG_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    MG_CUDA(cudaFuncGetAttributes(&fa, fn));
    const int dyn = (optin - (int)fa.sharedSizeBytes) / 128 * 128;
    if (dyn > 0 && cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, RS_THREADS, dyn) == cudaSuccess && per_sm >= 1)
      w.smem[wide] = (uint32_t)dyn;
    cudaGetLastError();
    w.fn[wide] = fn;
  }
  const uint32_t smem = w.smem[wide];
  if (!smem) return MGUSO_ERR_UNSUPPORTED;
  for (uint32_t i = 0; i < a.nrun; ++i) {
    const RsInst& I = a.inst[i];
    const uint32_t dom = ceil_div(nd[i], I.ncta), dia = 32 * ceil_div(I.dd1 - I.dd0, I.ncta);
    // the vectors of a CTA's vertices, the halo and the hash table have to fit
    const uint64_t need = RS_SCRATCH + 52ull * 32 * dom + 20ull * RS_MAX_HALO + 52ull * dia + 64 + RS_HASH_BYTES;
    if (dom > (uint32_t)RS_MAX_DOM || need > smem || (sw && dom > run.dom_max)) return MGUSO_ERR_UNSUPPORTED;
    // looked at row by row, once: more CTAs fit at least as well
    const uint32_t stage = 2 * (RS_WARPS / (wide ? 6 : 3)) * RS_CHUNK;
    if (w.good[I.k] && I.ncta >= w.good[I.k]) continue;
    if (I.ncta > w.poor[I.k]) {
      if (resident_walked(bsr, sw, run, I.k, I.ncta, smem, stage) <= run.walked_max) {
        w.good[I.k] = I.ncta;
        continue;
      }
      w.poor[I.k] = I.ncta;
    }
    return MGUSO_ERR_UNSUPPORTED;
  }
  // records and published sums carry epochs: cleared when allocated and when the epochs run out
  const size_t nrec = 2 * (size_t)std::max<uint32_t>(run.nv, 1), nsum = 3 * (size_t)RS_MAX_G;
  const uint32_t span = max_iter < (1u << 30) ? max_iter + 2 : (1u << 30);
  max_iter = std::min(max_iter, 1u << 30);
  const bool fresh = !w.rec.p || w.rec.cap < nrec || !w.sums.p || w.epoch + span >= 0x80000000u;
  MG_TRY(w.rec.reserve(nrec));
  MG_TRY(w.sums.reserve(nsum));
  MG_TRY(w.count.reserve(32 * PCG_MAX_INST + 1));
  if (fresh) {
    MG_CUDA(cudaMemsetAsync(w.rec.p, 0, 16 * w.rec.cap, st));
    MG_CUDA(cudaMemsetAsync(w.sums.p, 0, 16 * w.sums.cap, st));
    w.epoch = 0;
  }
  // rows padded to whole slots: by a third on the meshes measured, half as much again allowed for
  const size_t j16 = std::min<size_t>((size_t)run.nnz * 15 / 4 + 1024, 0x7fffffffu);
  MG_TRY(w.jscr.reserve(4 * j16));
  a.sys = sys;
  a.x = x;
  a.rec = w.rec.p;
  a.jscr = w.jscr.p;
  a.jcap = (uint32_t)j16;
  a.sums = w.sums.p;
  a.count = w.count.p;
  a.jtop = w.count.p + 32 * PCG_MAX_INST;
  a.epoch = w.epoch;
  a.out = out;
  a.tol = tol;
  a.max_iter = max_iter;
  a.smem_bytes = smem;
  w.epoch += span;
  k_rs_reset<<<64, 256, 0, st>>>(a.count, out, K, x, 3 * run.nv);
  MG_CUDA(cudaGetLastError());
  void* args[] = {(void*)&a};
  const cudaError_t e = cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(RS_THREADS), args, smem, st);
  if (coop_refused(e)) {
    cudaGetLastError();
    w.smem[wide] = 0;  // nor will it be the next time
    return MGUSO_ERR_UNSUPPORTED;
  }
  MG_CUDA(e);
  return MGUSO_OK;
}

int pcg_resident_scene(Scene& s, uint32_t active) {
  const uint32_t K = s.ninst;
  mguso_schwarz* sw = s.schwarz.get();
  RsRun& r = s.rs_run;
  if (!s.rs_ready) {
    r.precond = sw ? MGUSO_PRECOND_SCHWARZ : MGUSO_PRECOND_BLOCK_JACOBI;
    r.mixed = s.mixed;
    r.half = sw && sw->half;
    r.fp64_tiles = s.p.pcg_mode == 2 || (sw && sw->max_m <= 32);
    r.sms = s.ctx->sm_count;
    r.nv = s.nv;
    r.ninst = K;
    r.nnz = s.Ps.nnz;
    r.walked_max = WALKED_SCENE;
    r.dom_max = dom_max_scene(s.nv);
    for (uint32_t k = 0; k <= K; ++k) r.vert[k] = s.inst_vert[k];
    MG_CHECK_ARG(!sw || resident_domains(*sw, r), "resident PCG: Schwarz domains are not grouped by instance");
    s.rs_ready = true;
  }
  RsSystem y{};
  y.rp = s.Ps.row_ptr.p;
  y.col = s.Ps.col.p;
  y.val = s.A->val.p;
  y.crp = s.c_row_ptr.p;
  y.ccol = s.c_col.p ? s.c_col.p : s.c_row_ptr.p;
  y.cval = s.c_val.p;
  y.bjinv = s.bjinv.p;
  y.b = s.work.b.p;
  if (sw) {
    y.dom_start = sw->dom_start.p;
    y.dom_verts = sw->dom_verts.p;
    y.vpos = sw->vpos.p;
    y.fac_off = sw->fac_off.p;
    y.fac = sw->half ? (const void*)sw->fac_h.p : (const void*)sw->fac.p;
    y.fac_scale = sw->half ? sw->fac_scale.p : nullptr;
    y.vfac = sw->vfac.p;
  }
  MG_TRY(s.fr_inst.reserve(PCG_MAX_INST));
  MG_TRY(s.fr_out.reserve(PCG_MAX_INST));
  // at least one iteration, as the fused kernels run
  MG_TRY(pcg_resident(y, *s.A, sw, s.rs, r, s.work.x.p, active, s.p.cg_tol, std::max<uint32_t>(s.p.cg_max_iter, 1), s.fr_inst.p,
                      s.st));
  MG_CUDA(cudaMemcpyAsync(s.fr_out.p, s.fr_inst.p, sizeof(FusedInst) * K, cudaMemcpyDeviceToHost, s.st));
  return MGUSO_OK;
}

}  // namespace mg
