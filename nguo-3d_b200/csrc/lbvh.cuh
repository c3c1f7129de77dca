// LBVH state behind the mguso_lbvh handle.
#pragma once
#include "internal.cuh"

namespace mg {

constexpr uint32_t LEAF_BIT = 0x80000000u;  // karras.rs:14
constexpr uint32_t RIGHT_BIT = 0x80000000u;  // of a parent link: the child is the right one
constexpr uint32_t NO_PARENT = 0xffffffffu;

struct Lbvh {
  mguso_ctx* ctx = nullptr;
  uint32_t nt = 0;
  int key_bits = 30;
  bool shaped = false;              // the last build enqueued its whole shape (refits may follow)
  DevBuf<unsigned char> keys;       // nt keys (u32 or u64), sorted after build
  DevBuf<uint32_t> perm;            // sorted leaf -> triangle
  // the shape, in one allocation: per inner node, its parent (the top bit says that it is the right
  // child), its range's other end (its own index is one end) and the arrivals at it (0 after a build's
  // shape, even after each refit); per leaf, its parent; the refit's subtrees: their roots
  // (LEAF_BIT for a leaf) and number
  DevBuf<uint32_t> shape;
  uint32_t *parent_int = nullptr, *parent_leaf = nullptr, *range_end = nullptr, *flags = nullptr, *roots = nullptr,
           *nroots = nullptr;
  // Per inner node, one 64-byte record of its two children: (lo, id), (hi, -), of the left, then of
  // the right one, id the child's index with LEAF_BIT for a leaf (as float bits), so that a walk
  // reads a node's children and their boxes in one round of loads. A one-primitive tree has one
  // record, its right child empty (NaN: never entered). drec: the same of the displacement boxes
  // (CCD pruning).
  DevBuf<float4> rec, drec;
  DevBuf<float> params;             // centroid lo.xyz, inv.xyz
  DevBuf<uint32_t> ord;
  DevBuf<uint32_t> status;
  uint32_t* err_sink = nullptr;     // when set, the sort's wait-timeout bit goes here instead of status
  // radix-sort scratch
  DevBuf<uint32_t> rs_words, rs_tmpv;
  DevBuf<unsigned char> rs_tmpk;
  // query scratch
  DevBuf<uint32_t> qkeys, qorder;
  DevBuf<uint32_t> nodes;  // of lbvh_nodes: 8 words per inner node
  // optional per-stage timing events: 0 start, 1 morton, 2 sort, 3 karras, 4 refit,
  // 5 query prep, 6 traversal
  bool ev_on = false;
  cudaEvent_t ev[7] = {};
};

int radix_sort_pairs(Lbvh* b, void* keys, uint32_t* vals, uint32_t n, int key_bits, cudaStream_t s);
int lbvh_build(Lbvh* b, const float* pos, uint32_t nv, const uint32_t* tris, uint32_t nt, int key_bits,
               cudaStream_t s);
// The records at pos over the tree's existing shape (keys, permutation and parents from the last
// lbvh_build, which must have had the same primitives; MGUSO_ERR_INVALID_ARG when that build
// did not complete): the boxes are exact unions again, so every overlap query returns the same
// leaves as after a rebuild at pos, only the shape fits pos less tightly.
int lbvh_refit_pos(Lbvh* b, const float* pos, const uint32_t* tris, cudaStream_t s);
// The displacement records (AABB of dx over each primitive's vertices, refitted up the tree), for
// the CCD's pruning test.
int lbvh_refit_disp(Lbvh* b, const float* dx, const uint32_t* tris, cudaStream_t s);
// The nodes as the caller of a build sees them: children and boxes (lo, hi) of each, to host memory
// (null: not wanted), once every stream has passed the build.
int lbvh_nodes(Lbvh* b, uint32_t* left, uint32_t* right, float* boxes);
int lbvh_query_points(Lbvh* b, const float* pts, uint32_t np, float dhat, uint32_t* pairs, uint64_t cap,
                      unsigned long long* count, bool morton_order, cudaStream_t s);

}  // namespace mg

struct mguso_lbvh {
  mg::Lbvh b;
  mg::DevBuf<unsigned long long> count;
  mg::DevBuf<float> hpos;
  mg::DevBuf<uint32_t> htris, hpairs;
};

namespace mg {

__device__ __forceinline__ bool boxes_overlap(const float4& qlo, const float4& qhi, const float4& lo, const float4& hi) {
  return qlo.x <= hi.x && qlo.y <= hi.y && qlo.z <= hi.z && lo.x <= qhi.x && lo.y <= qhi.y && lo.z <= qhi.z;
}

// CCD traversal test (ccd_max_step's broad phase, implicit.rs:1690-1947, with exact pruning).
// A subtree is entered when the search box overlaps its position box [lo, hi] and its
// pairs with the query are not all settled by accd_toi's first test (contact.rs:378-437),
// which returns max_t = 1.25 whenever 1.25 u_max < 0.98 d0 (u_max: the largest relative
// displacement of the pair's four points; d0: their distance). Over a subtree, with the
// query's displacements inside the ball (cq, rq) and the subtree's inside its displacement
// box D (db, read only when needed), the pairs' relative displacements are bounded by 2 rq
// (within the query), the diagonal of D (within a primitive) and rq + farthest(cq, D)
// (across), so u_max <= max(2 rq, diag D, rq + farthest(cq, D)); and d0 >= the distance
// between the query's box (qlo, qhi) and the subtree's position box. The subtree is skipped
// when 1.3 u_bound < 0.98 distance (4% margin over 1.25 for rounding).
struct CcdQuery {
  float4 slo, shi, qlo, qhi;
  float4 c;  // cq, rq
  __device__ __forceinline__ bool enter(const float4 lo, const float4 hi, const float4* db) const {
    if (!boxes_overlap(slo, shi, lo, hi)) return false;
    const float gx = fmaxf(fmaxf(qlo.x - hi.x, lo.x - qhi.x), 0.f);
    const float gy = fmaxf(fmaxf(qlo.y - hi.y, lo.y - qhi.y), 0.f);
    const float gz = fmaxf(fmaxf(qlo.z - hi.z, lo.z - qhi.z), 0.f);
    const float gap2 = gx * gx + gy * gy + gz * gz;
    if (gap2 == 0.f) return true;
    const float4 dlo = __ldg(db), dhi = __ldg(db + 1);
    const float rq = c.w;
    const float fx = fmaxf(fabsf(c.x - dlo.x), fabsf(c.x - dhi.x));
    const float fy = fmaxf(fabsf(c.y - dlo.y), fabsf(c.y - dhi.y));
    const float fz = fmaxf(fabsf(c.z - dlo.z), fabsf(c.z - dhi.z));
    const float ex = dhi.x - dlo.x, ey = dhi.y - dlo.y, ez = dhi.z - dlo.z;
    const float u = fmaxf(fmaxf(2.f * rq, sqrtf(ex * ex + ey * ey + ez * ez)), rq + sqrtf(fx * fx + fy * fy + fz * fz));
    return !(1.3f * u < 0.98f * sqrtf(gap2));
  }
};
struct BoxQuery {
  float4 lo, hi;
  __device__ __forceinline__ bool enter(const float4 blo, const float4 bhi, const float4*) const {
    return boxes_overlap(lo, hi, blo, bhi);
  }
};

// One tree as the walks read it, and one per instance over that instance's primitives (a query only
// meets its own instance); base[k] turns a tree's local primitive index into the scene's.
struct BvhView {
  const uint32_t* prim;
  const float4 *rec, *drec;
  uint32_t n;
};
struct BvhSet {
  BvhView t[PCG_MAX_INST];
  uint32_t base[PCG_MAX_INST];
};
inline BvhView lbvh_view(const Lbvh& b) { return BvhView{b.perm.p, b.rec.p, b.drec.p, b.nt}; }

// ---- warp walks -------------------------------------------------------------------------------
// A warp takes `per` consecutive queries (up to 32) down their trees together: its queue holds
// (query, node) pairs, each round takes up to 32 of them, newest first, one per lane, tests the
// node's two children against the query and queues those entered; leaves go, as (query,
// primitive) pairs, to a second queue, from which the whole warp takes 32 at a time through the
// remaining filters and the narrow phase (distances, accd_toi). What bounds a walk is its chain
// of dependent rounds: with a stack per lane, a warp ran as many rounds as its longest query
// has nodes (some hundreds, about half of the lanes idle), while a shared queue keeps all
// lanes on nodes of any query and needs little more than their number over 32, so that few
// queries per warp (small scenes) spread over more warps. 64 x 64 sheet, before -> after: edge-edge
// CCD 219 -> 87 us, vertex-triangle CCD 150 -> 30, stencils 140 -> 40 and 97 -> 22; one garment:
// 160 -> 129, 176 -> 98, 145 -> 94 and 140 -> 49; six garments: 522 -> 421, 320 -> 243,
// 408 -> 302 and 205 -> 122.
// Results are order-free: stencils are sorted by their pair key afterwards, CCD results are
// minima and sums, and the leaves reached do not depend on the order of the tests.
constexpr int WQ_WARPS = 4;   // 128-thread blocks
constexpr int WQ_QCAP = 96;   // < 32 left over + 2 leaves per lane and round
// queued nodes per warp: a round adds at most 32; with FW_SPARE places left one node is taken at a
// time, which goes down depth first and adds at most one per level
constexpr int FW_CAP = 1024, FW_SPARE = 128;

template <class Q, int CAP = FW_CAP>
struct WalkMem {  // shared memory of one warp
  Q query[32];
  uint32_t node[CAP];
  uint2 pair[WQ_QCAP];
  uint8_t slot[CAP];
  uint8_t inst[32];
};

__device__ __forceinline__ void wq_push(uint2* q, int& n, bool has, uint2 e) {
  const unsigned m = __ballot_sync(0xffffffffu, has);
  if (has) q[n + __popc(m & ((1u << (threadIdx.x & 31)) - 1u))] = e;
  n += __popc(m);
}

// Takes batches of up to 32 queued pairs while at least min_n are queued (n is warp-uniform).
template <class F>
__device__ __forceinline__ void wq_take(uint2* q, int& n, int min_n, F&& solve) {
  const int lane = (int)(threadIdx.x & 31);
  __syncwarp();
  while (n >= min_n && n > 0) {
    const int take = n < 32 ? n : 32;
    const bool has = lane < take;
    const uint2 e = has ? q[n - take + lane] : make_uint2(0u, 0u);
    __syncwarp();
    n -= take;
    if (has) solve(e);
  }
}

// Walks the trees of the warp's queries: lane l holds query l (valid or not) of instance k,
// numbered first + l. keep(slot, primitive) says whether a leaf reached is to be solved. The walks
// begin at node `start` (0, the root, or one that covers all that the queries can meet).
// Returns false when the node queue overflowed.
template <class Q, int CAP, class KEEP, class SOLVE>
__device__ __forceinline__ bool warp_walk(WalkMem<Q, CAP>& m, const BvhSet& bs, uint32_t first, bool valid, uint32_t k,
                                          const Q& mine, KEEP&& keep, SOLVE&& solve, uint32_t start = 0) {
  const int lane = (int)(threadIdx.x & 31);
  const unsigned below = (1u << lane) - 1u;
  int n = 0, np = 0;
  bool ok = true;
  const bool root = valid && bs.t[k].n > 0;
  if (root) {
    m.query[lane] = mine;
    m.inst[lane] = (uint8_t)k;
  }
  {
    const unsigned r = __ballot_sync(0xffffffffu, root);
    if (root) {
      const int at = __popc(r & below);
      m.node[at] = start;
      m.slot[at] = (uint8_t)lane;
    }
    n = __popc(r);
  }
  __syncwarp();
  while (n > 0) {
    const int take = n <= CAP - FW_SPARE ? min(n, 32) : 1;
    if (n + take > CAP) {
      ok = false;
      break;
    }
    const bool has = lane < take;
    uint32_t ch[2] = {0, 0}, slot = 0, base = 0;
    const uint32_t* prims = nullptr;
    bool in[2] = {false, false};
    if (has) {
      const uint32_t cur = m.node[n - take + lane];
      slot = m.slot[n - take + lane];
      const BvhView& t = bs.t[m.inst[slot]];
      base = bs.base[m.inst[slot]];
      prims = t.prim;
      const float4* cb = t.rec + 4 * (size_t)cur;
      const float4* db = t.drec + 4 * (size_t)cur;
      const float4 l0 = __ldg(cb), h0 = __ldg(cb + 1), l1 = __ldg(cb + 2), h1 = __ldg(cb + 3);
      ch[0] = __float_as_uint(l0.w);
      ch[1] = __float_as_uint(l1.w);
      const Q& q = m.query[slot];
      in[0] = q.enter(l0, h0, db);
      in[1] = q.enter(l1, h1, db + 2);
    }
    n -= take;
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const bool inner = in[c] && !(ch[c] & LEAF_BIT);
      const unsigned b = __ballot_sync(0xffffffffu, inner);
      if (inner) {
        const int at = n + __popc(b & below);
        m.node[at] = ch[c];
        m.slot[at] = (uint8_t)slot;
      }
      n += __popc(b);
      bool leaf = in[c] && (ch[c] & LEAF_BIT);
      uint32_t prim = 0;
      if (leaf) {
        prim = base + __ldg(prims + (ch[c] & ~LEAF_BIT));
        leaf = keep(slot, prim);
      }
      wq_push(m.pair, np, leaf, make_uint2(first + slot, prim));
    }
    wq_take(m.pair, np, 32, solve);
    __syncwarp();
  }
  wq_take(m.pair, np, 1, solve);
  return ok;
}

}  // namespace mg
