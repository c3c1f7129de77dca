// LBVH state behind the mguso_lbvh handle.
#pragma once
#include "internal.cuh"

namespace mg {

constexpr uint32_t LEAF_BIT = 0x80000000u;  // karras.rs:14
constexpr uint32_t NO_PARENT = 0xffffffffu;

struct Lbvh {
  mguso_ctx* ctx = nullptr;
  uint32_t nt = 0;
  int key_bits = 30;
  bool shaped = false;              // the last build enqueued its whole shape (refits may follow)
  DevBuf<unsigned char> keys;       // nt keys (u32 or u64), sorted after build
  DevBuf<uint32_t> perm;            // sorted leaf -> triangle
  DevBuf<uint32_t> left, right;     // nt - 1 internal nodes
  DevBuf<uint32_t> parent_int, parent_leaf;
  DevBuf<float4> leaf, node;        // 2 float4 per box (lo, hi)
  DevBuf<float4> dleaf, dnode;      // displacement boxes of the same tree (CCD pruning)
  // per internal node, its two children's boxes side by side (left lo, hi, right lo, hi), so
  // that a walk reads a node's child indices and their boxes in one round of loads; kept only
  // when child_boxes is set (the scene's trees, whose walks read them)
  DevBuf<float4> cbox, dcbox;
  bool child_boxes = true;
  DevBuf<uint32_t> flags;
  DevBuf<float> params;             // centroid lo.xyz, inv.xyz
  DevBuf<uint32_t> ord;
  DevBuf<uint32_t> status;
  uint32_t* err_sink = nullptr;     // when set, the sort's wait-timeout bit goes here instead of status
  // radix-sort scratch
  DevBuf<uint32_t> rs_words, rs_tmpv;
  DevBuf<unsigned char> rs_tmpk;
  // query scratch
  DevBuf<float4> qbox;
  DevBuf<uint32_t> qkeys, qorder;
  // optional per-stage timing events: 0 start, 1 morton, 2 sort, 3 karras, 4 refit,
  // 5 query prep, 6 traversal
  bool ev_on = false;
  cudaEvent_t ev[7] = {};
};

int radix_sort_pairs(Lbvh* b, void* keys, uint32_t* vals, uint32_t n, int key_bits, cudaStream_t s);
int lbvh_build(Lbvh* b, const float* pos, uint32_t nv, const uint32_t* tris, uint32_t nt, int key_bits,
               cudaStream_t s);
// Leaf and node boxes at pos over the tree's existing shape (keys, permutation and children
// from the last lbvh_build, which must have had the same primitives; MGUSO_ERR_INVALID_ARG
// when that build did not complete): the boxes are exact
// unions again, so every overlap query returns the same leaves as after a rebuild at pos,
// only the shape fits pos less tightly.
int lbvh_refit_pos(Lbvh* b, const float* pos, const uint32_t* tris, cudaStream_t s);
// Displacement boxes (AABB of dx over each primitive's vertices, refitted up the tree) into
// dleaf/dnode, for the CCD's pruning test.
int lbvh_refit_disp(Lbvh* b, const float* dx, const uint32_t* tris, cudaStream_t s);
int lbvh_query_boxes(Lbvh* b, const float4* qbox, const uint32_t* qorder, uint32_t nq, uint32_t* pairs, uint64_t cap,
                     unsigned long long* count, cudaStream_t s);
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

}  // namespace mg
