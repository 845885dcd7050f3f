// query.cu -- fixed-radius / bounded-KNN / KNN rows and the directed
// nearest-distance (Hausdorff) reduction over a built scene.
//
// Semantics (rubaolee/rtdl src/rtdsl/reference.py:349-434, 882-890): a search
// point is a fixed-radius neighbor when the FP64 value ((dx*dx + dy*dy) +
// dz*dz), dx = search - query, is <= radius*radius; neighbors of one query are
// ordered by (sqrt(d2), neighbor_id, search input index) and the first k_max
// (or k) are kept; rows are grouped by query_id in query input order.
//
// How the device reaches that exactly:
//   * Traversal and candidate tests run in FP32.  A candidate is accepted
//     without further work when its FP32 d2 is below lo2, dropped above hi2, and
//     re-decided in FP64 in between.  lo2/hi2 bracket r^2 by a relative band
//     (1e-5) plus, for inputs that are not FP32-exact, an absolute band of
//     8 * 2^-24 * max|coordinate| (the FP32 rounding of the inputs); see
//     k_bands.
//   * A warp walks the wide tree for a packet of 32 neighbouring queries and
//     keeps every query's candidates (collect); eight lanes or more per query
//     then sort them by FP32 keys, re-decide near ties exactly (FP64 sqrt(d2),
//     then neighbor id, then search input index) and write the rows (emit).  The distance is
//     computed in FP64 without fused multiply-adds, so it is bit-identical to
//     the reference.
//   * k nearest (k <= 64) is the same with a radius per query that holds its k
//     nearest.
//   * Queries with more candidates than a slab row are collected again at a
//     smaller radius; what that does not resolve, and k or k_max above 64 with
//     more than 256 candidates, goes to a generic block-per-query path (gather,
//     bitonic sort in global memory, emit).
#include <cstdlib>
#include <cstring>
#include <functional>
#include <mutex>

#include "internal.cuh"
#include "walk.cuh"

namespace rtdl_b200 {

namespace {

constexpr int kExpandThreads = 256;
constexpr int kHeavyThreads = 256;

struct DevBands {
  float hi2, lo2, box_hi2;
  float top, width;  // the bucket test's form of [lo2, hi2], see set_band_top
  float rho, e_abs, floor2;
  double r2;
  unsigned int ids_sorted;
};

// The bucket test's form of [lo2, hi2].  It computes d2 - top as one fma chain
// and looks at the sign, so top lies above hi2 and top - width below lo2 by
// more than the chain's rounding near the boundary (a few units of hi2; eight
// are added on either side): a point with a positive difference is outside,
// one with a difference below -width inside, and FP64 decides the rest.
__device__ __forceinline__ void set_band_top(DevBands& b) {
  const double u = 5.9604644775390625e-08;  // 2^-24
  const double lo = fminf(b.lo2, FLT_MAX), hi = fminf(b.hi2, FLT_MAX);
  b.top = fminf(__double2float_ru(hi * (1.0 + 8.0 * u)), FLT_MAX);
  b.width = __double2float_ru((double)b.top - lo * (1.0 - 8.0 * u));
}

// Band constants from the statistics of both point sets.  Error model (FP32
// d2 from FP32-rounded coordinates vs the exact distance d):
//   |d_fp32 - d| <= 3u*d + 3.5u*M (u = 2^-24, M = max |coordinate|; the M
//   term is absent when every coordinate is FP32-exact).
// The bands below are wider: relative 1e-5 and absolute 8u*M.
__device__ DevBands make_bands(const PointStats* scene, const PointStats* queries, double radius, int has_radius) {
  const double M = fmax(__longlong_as_double((long long)scene->max_abs_bits),
                        __longlong_as_double((long long)queries->max_abs_bits));
  const bool inexact = scene->inexact || queries->inexact;
  const double u = 5.9604644775390625e-08;
  const double e_abs = inexact ? 8.0 * u * M : 0.0;
  const double rho = 1.0e-5;
  DevBands b;
  b.rho = (float)rho;
  b.e_abs = __double2float_ru(e_abs);
  b.floor2 = 1.0e-30f;
  b.ids_sorted = queries->ids_unsorted ? 0u : 1u;
  if (has_radius) {
    const double r_hi = radius * (1.0 + rho) + e_abs + 1.0e-18;
    const double r_lo = radius * (1.0 - rho) - e_abs;
    float hi2 = __double2float_ru(r_hi * r_hi);
    if (hi2 < b.floor2) hi2 = b.floor2;
    b.hi2 = hi2;
    b.lo2 = r_lo > 0.0 ? __double2float_rd(r_lo * r_lo) : 0.0f;
    b.box_hi2 = __double2float_ru((double)hi2 * (1.0 + 1.0e-6));
    b.r2 = radius * radius;
  } else {
    b.hi2 = INFINITY;
    b.lo2 = INFINITY;
    b.box_hi2 = INFINITY;
    b.r2 = INFINITY;
  }
  set_band_top(b);
  return b;
}

__global__ void k_bands(const PointStats* scene, const PointStats* queries, double radius, int has_radius,
                        DevBands* out) {
  if (threadIdx.x == 0) *out = make_bands(scene, queries, radius, has_radius);
}

// Problem batch: bands per problem (the statistics are the whole batch's, which
// only widens the bands); ids_sorted from the batch's per-problem check.
__global__ void k_bands_batch(const PointStats* scene, const PointStats* queries, const double* radius, uint32_t m,
                              const unsigned int* ids_sorted, DevBands* out) {
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < m; p += gridDim.x * blockDim.x) {
    DevBands b = make_bands(scene, queries, radius[p], 1);
    b.ids_sorted = *ids_sorted;
    out[p] = b;
  }
}

struct Ctx {
  float qx, qy, qz;
  double ex, ey, ez;  // exact query coordinates
  const float4* pts;
  const double* pts64;
  const uint32_t* perm;
  int scene_inexact;
  float rho, e_abs, floor2;
};

__device__ __forceinline__ double exact_d2(const Ctx& c, uint32_t i) {
  double sx, sy, sz;
  if (c.scene_inexact) {
    const double* p = c.pts64 + 3ull * i;
    sx = p[0];
    sy = p[1];
    sz = p[2];
  } else {
    const float4 p = __ldg(&c.pts[i]);
    sx = p.x;
    sy = p.y;
    sz = p.z;
  }
  const double dx = __dsub_rn(sx, c.ex), dy = __dsub_rn(sy, c.ey), dz = __dsub_rn(sz, c.ez);
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

__device__ __forceinline__ float key_tol(const Ctx& c, float m) {
  float t = c.rho * m + c.floor2;
  if (c.e_abs > 0.f) t += 2.f * sqrtf(m) * c.e_abs + c.e_abs * c.e_abs;
  return t;
}

__device__ __forceinline__ double exact_d2_at(double ex, double ey, double ez, const float4* pts, const double* pts64,
                                              int inexact, uint32_t i) {
  double sx, sy, sz;
  if (inexact) {
    const double* p = pts64 + 3ull * i;
    sx = p[0];
    sy = p[1];
    sz = p[2];
  } else {
    const float4 p = __ldg(&pts[i]);
    sx = p.x;
    sy = p.y;
    sz = p.z;
  }
  const double dx = __dsub_rn(sx, ex), dy = __dsub_rn(sy, ey), dz = __dsub_rn(sz, ez);
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

// Exact comparison of two candidates by the reference's sort key.  Out of
// line and with scalar arguments, so the caller's query context stays in
// registers.
__device__ __noinline__ bool exact_before(double ex, double ey, double ez, const float4* pts, const double* pts64,
                                          const uint32_t* perm, int inexact, uint32_t ia, uint32_t ib) {
  const double da = __dsqrt_rn(exact_d2_at(ex, ey, ez, pts, pts64, inexact, ia));
  const double db = __dsqrt_rn(exact_d2_at(ex, ey, ez, pts, pts64, inexact, ib));
  if (da != db) return da < db;
  const uint32_t na = __float_as_uint(__ldg(&pts[ia].w)), nb = __float_as_uint(__ldg(&pts[ib].w));
  if (na != nb) return na < nb;
  return __ldg(&perm[ia]) < __ldg(&perm[ib]);
}

// Counters of RTDL_B200_STATS, by their place in rtdl_b200_get_last_query_stats
// (the walks gather neither nodes, leaf points, inserts, shifts, band checks nor
// leaf pairs: those read 0).
enum Stat { kStatNodes, kStatLeafPoints, kStatInRadius, kStatInserts, kStatShifts, kStatBand, kStatMaxLeafPoints,
            kStatGenericQueries, kStatLargeQueries, kStatLeafPairs, kStatEmitFixups, kStatRefined, kStatCount };

// ---- fixed-radius collect pass ----------------------------------------------
// Queries in curve order, a packet of 32 per warp.  A query's in-radius points
// go to its row of the candidate slab; the exact in-radius count is kept, so
// the overflow flag and the row offsets are exact without any per-query list.
constexpr int kSlab = 256;  // candidates kept per query
constexpr unsigned int kStrideBlocks = kSmCount * 8;  // grid of the kernels that stride over device counts

// Candidate slab: kSlab sorted point indices per processing rank, so a warp
// reads a query's candidates with contiguous loads.
__host__ __device__ __forceinline__ size_t slab_base(uint32_t t) { return (size_t)t * kSlab; }

// Per-query record written by the collect pass at the query's processing rank
// and read by the emit kernels, so they find the query's exact coordinates,
// id and candidate count with one load.
struct __align__(16) QueryInfo {
  double ex, ey, ez;  // exact query coordinates (z = 0 in 2D)
  uint32_t qid;
  uint32_t meta;      // candidates (9 bits), the kQuery* bits, kmax (9 bits); 0: nothing to emit
};
constexpr uint32_t kQueryCountMask = 511u;
constexpr uint32_t kQueryGeneric = 1u << 18;  // candidates not kept: generic path
constexpr uint32_t kQueryBig = 1u << 19;      // 65..kSlab candidates: k_emit_mid, k_emit_big
constexpr int kQueryKmaxShift = 20;           // kmax, at most kSlab
__device__ __forceinline__ int query_kmax(uint32_t meta) { return (int)((meta >> kQueryKmaxShift) & 511u); }

struct CollectParams {
  SceneView S;
  const float4* qpts;
  const double* qraw;
  int qstride;
  const uint32_t* qorder;    // processing rank -> query input index (kNone: padding of a problem batch)
  uint32_t nq;               // processing ranks (a batch pads every problem to whole warps)
  uint32_t width;            // queries per packet, at most 32 (see launch_collect)
  uint32_t kmax;
  double radius;             // of a single problem
  const DevBands* bands;     // one per problem (one in all for a single problem)
  const uint32_t* warp_prob; // problem batch: the problem of each warp of processing ranks (nullptr: single)
  const uint32_t* prob_kmax; // problem batch: kmax per problem
  const double* prob_radius; // problem batch: radius per problem
  const double* rank_radius; // KNN: the radius of each processing rank (holds its kmax nearest); else nullptr
  uint32_t* slab;            // slab_base(nq) entries
  uint32_t* counts;          // min(in-radius count, kmax), query input order
  QueryInfo* qinfo;          // by processing rank
  uint8_t* flags;            // bit0: count > kmax, bit1: generic path (query input order)
  uint32_t* heavy_list;      // generic path: query input index,
  uint32_t* heavy_m;         // in-radius count at heavy_rad,
  double* heavy_rad;         // a radius that holds the query's kmax nearest,
  uint32_t* heavy_t;         // and processing rank
  uint32_t* mid_list;        // processing ranks of the queries with 65..128 candidates
  uint32_t* big_list;        // processing ranks of the queries with 129..kSlab candidates
  uint32_t* single_list;     // processing ranks the packets leave to k_collect_single
  unsigned int* small;       // [0] generic-path query count, [1] the generic path's error bits, [2] mid_list length,
                             // [3] big_list length, [4] emit fixup queue length, [6] single_list length
  uint8_t* overflow_out;     // optional: 1 per query (input order) when count > kmax
  unsigned long long* stats;
};

// The bands of DevBands recomputed for another radius (same formulas; the
// FP32 e_abs is rounded up, which only widens them).
__device__ __forceinline__ DevBands bands_at_radius(const DevBands& base, double radius) {
  DevBands b = base;
  const double rho = (double)base.rho, e_abs = (double)base.e_abs;
  const double r_hi = radius * (1.0 + rho) + e_abs + 1.0e-18;
  const double r_lo = radius * (1.0 - rho) - e_abs;
  float hi2 = __double2float_ru(r_hi * r_hi);
  if (hi2 < b.floor2) hi2 = b.floor2;
  b.hi2 = hi2;
  b.lo2 = r_lo > 0.0 ? __double2float_rd(r_lo * r_lo) : 0.0f;
  b.box_hi2 = __double2float_ru((double)hi2 * (1.0 + 1.0e-6));
  b.r2 = radius * radius;
  set_band_top(b);
  return b;
}

// Which of the hits among four buckets' points are within the query's radius:
// those whose FP32 distance is not below the band, in FP64 (a lane calls it
// when a hit lies inside the band; `lo` is the band's lower edge in the bucket
// test's form).  On a lattice whose spacing divides the radius most packets
// come here: counts of 60k queries over 1M points 932 us with all 32 points
// decided in FP64, 696 with the hits taken one by one, 556 so.
template <int DIM>
__device__ __noinline__ uint32_t exact_buckets_mask(const SceneView& S, int inexact, const double* rq, float4 q,
                                                    float lo, double r2, uint4 four, uint32_t hits) {
  BucketQuery bq;
  bq.set(q.x, q.y, q.z, lo);
  for (uint32_t m = hits & ~buckets_mask<DIM, false>(S.bucket_pts, four, bq, nullptr); m; m &= m - 1u) {
    const int j = __ffs((int)m) - 1;
    const uint32_t b = j < 8 ? four.x : j < 16 ? four.y : j < 24 ? four.z : four.w;
    if (!(exact_d2_at(rq[1], rq[2], DIM == 3 ? rq[3] : 0.0, S.pts, S.pts64, inexact, b * kBucketPoints + (j & 7)) <= r2))
      hits &= ~(1u << j);
  }
  return hits;
}

// One warp walks a tree for one query and its lanes test the reached buckets'
// points together, four buckets at a time: point(i, p, has) runs on every lane
// with its point and returns true, on all of them, to end the walk.  has is
// false where there is no bucket and for the points at infinity that fill one
// up, which a radius whose square overflows would hold.
template <typename Point>
__device__ __forceinline__ void walk_single(const SceneView& S, const TreeShape* T, const float4& q,
                                            const float& reach2, WalkStack& stack, int lane, Point&& point) {
  const PacketBox box{q.x, q.y, q.z, q.x, q.y, q.z};
  const uint32_t bucket0 = __ldg(&T->base[0]);
  walk_wide(S, T, box, nullptr, reach2, stack, lane, [&](uint32_t first, uint32_t mask) {
    while (mask) {
      // lane group g (eight lanes) takes the g-th set bucket
      uint32_t m = mask;
      for (int g = 0; g < (lane >> 3); ++g) m &= m - 1u;
      const uint32_t i = (bucket0 + first + (m ? (uint32_t)(__ffs((int)m) - 1) : 0u)) * kBucketPoints + (lane & 7);
      const float4 p = __ldg(&S.pts[i]);
      if (point(i, p, m != 0u && p.x < INFINITY)) return true;
#pragma unroll
      for (int g = 0; g < 4; ++g) mask &= mask - 1u;
    }
    return false;
  });
}

// A warp's queue of buckets that hold in-radius points, one column per lane:
// (bucket << 8) | the points' bits, the bucket counted within the tree.  A
// store per bucket, kept or overwritten, instead of an append per point keeps
// the walk free of divergent steps (on the clustered sets a query gets 32
// points from 10 buckets); the lanes expand their words together when the queue
// is flushed, four indices to a 16-byte store.
constexpr int kQueueWords = 25;  // the last row only takes stores of lanes without a hit
struct CollectWarp {
  uint32_t queue[kQueueWords][32];
  __align__(16) uint32_t list[kBucketList];
  WalkStack stack;
};

// A packet's walk: every lane with `active` collects its points within band B
// (their number in *count); the others keep what they have.  BAND: the radius
// decides the rows, so points inside the band are decided in FP64.  A KNN radius
// only has to hold the k nearest: what lies just outside it may come along (it
// is widened from the distance of a point, which would always lie in the band).
template <int DIM, bool BAND>
__device__ __forceinline__ void collect_walk(const CollectParams& P, const TreeShape* T, const DevBands& B,
                                             int scene_inexact, const float4& q, uint32_t qin, uint32_t t,
                                             bool active, CollectWarp& W, int lane, const PacketBox& box,
                                             const PacketBox* limit, float reach2, uint32_t* count) {
  const SceneView& S = P.S;
  const uint32_t bucket0 = __ldg(&T->base[0]);
  BucketQuery bq;
  bq.set(q.x, q.y, q.z, B.top);
  // near < band: in the band; never for a lane that collects nothing
  const int band = active ? (int)(0x80000001u + __float_as_uint(B.width)) : (int)0x80000000;
  const uint32_t keep = active ? 0xffffffffu : 0u;
  uint32_t found = 0;      // points
  int words = 0;           // words in the queue
  uint32_t pending = 0;    // points in the queue
  uint32_t stored = 0;     // indices stored, a multiple of four until the last flush
  // Stores the queued points in fours; a rest of at most three stays queued
  // unless `last` (whose last store may hold up to three stray indices).
  auto flush = [&](bool last) {
    __syncwarp();
    uint32_t fours = last ? (pending + 3) / 4 : pending / 4;
    const uint32_t room = ((uint32_t)kSlab - stored) / 4;  // beyond kSlab they are only counted
    const bool full = fours > room;
    if (full) fours = room;
    const uint32_t most = __reduce_max_sync(0xffffffffu, fours);
    uint32_t bits = 0, word = 0, first = 0;
    int w = 0;
    uint32_t* out = P.slab + slab_base(t) + stored;
    for (uint32_t k = 0; k < most; ++k) {
      if (k < fours) {
        uint32_t i[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (bits == 0 && w < words) {
            word = W.queue[w++][lane];
            bits = word & 255u;
            first = (bucket0 + (word >> 8)) * kBucketPoints;
          }
          i[u] = first + (bits ? (uint32_t)(__ffs((int)bits) - 1) : 0u);
          bits &= bits - 1u;
        }
        *reinterpret_cast<uint4*>(out + 4 * k) = make_uint4(i[0], i[1], i[2], i[3]);
      }
    }
    stored += 4 * fours;
    int rest = 0;
    if (!full && !last) {
      if (bits) W.queue[rest++][lane] = (word & ~255u) | bits;
      while (w < words) W.queue[rest++][lane] = W.queue[w++][lane];
      pending -= 4 * fours;
    } else {
      pending = 0;
    }
    words = rest;
    __syncwarp();
  };
  walk_fours(S, T, box, limit, reach2, W.stack, W.list, lane, 32u, [&](const uint4& four) {
    int near;
    uint32_t hits = buckets_mask<DIM, BAND>(S.bucket_pts, four, bq, &near);
    if (BAND && near < band)
      hits = exact_buckets_mask<DIM>(S, scene_inexact, P.qraw + (size_t)qin * P.qstride, q,
                                     __fsub_rd(B.top, B.width), B.r2, four, hits);
    hits &= keep;
    found += __popc(hits);
    pending += __popc(hits);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t bucket = u == 0 ? four.x : u == 1 ? four.y : u == 2 ? four.z : four.w;
      const uint32_t byte = (hits >> (8 * u)) & 255u;
      W.queue[words][lane] = ((bucket - bucket0) << 8) | byte;  // kept when it has a hit
      words += byte != 0u;
    }
    if (__any_sync(0xffffffffu, words > kQueueWords - 5)) flush(false);
    return false;
  });
  flush(true);
  if (active) *count = found;
}

// What a packet walk that keeps no candidates needs of shared memory.
struct PacketWarp {
  __align__(16) uint32_t list[kBucketList];
  WalkStack stack;
};

// The same for one query by the whole warp (all arguments warp-uniform).
__device__ __noinline__ uint32_t collect_alone(const CollectParams& P, const TreeShape* T, const DevBands& B,
                                               int scene_inexact, uint32_t qin, uint32_t t, WalkStack& stack) {
  const SceneView& S = P.S;
  const int lane = threadIdx.x & 31;
  const float4 q = P.qpts[qin];
  const double* rq = P.qraw + (size_t)qin * P.qstride;
  uint32_t* out = P.slab + slab_base(t);
  uint32_t count = 0;
  walk_single(S, T, q, B.box_hi2, stack, lane, [&](uint32_t i, const float4& p, bool has) {
    const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
    const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    bool hit = has && d2 <= B.hi2;
    if (hit && d2 >= B.lo2)
      hit = exact_d2_at(rq[1], rq[2], P.qstride == 4 ? rq[3] : 0.0, S.pts, S.pts64, scene_inexact, i) <= B.r2;
    const uint32_t hits = __ballot_sync(0xffffffffu, hit);
    const uint32_t at = count + __popc(hits & ((1u << lane) - 1u));
    if (hit && at < (uint32_t)kSlab) out[at] = i;
    count += __popc(hits);
    return false;
  });
  return count;
}

// A query whose radius holds more than kSlab points needs only its kmax (<= 64)
// nearest.  If at least kmax points lie within a smaller radius r', those kmax
// nearest are all among them, so the query is collected again at r' (its rows
// and counts still refer to the original radius).  r' is chosen from the
// in-radius count (cube-root scaling towards ~2 kmax points) inside a bracket
// [lo, hi] that every pass narrows; a query still unresolved after the passes
// (many points at one distance) takes the generic path, which gathers within
// the smallest tested radius that holds its rows.  The passes run inside the
// collect, by the packet that holds the query: the lanes are neighbours, the
// nodes are in the caches, and nothing is listed or read back.
constexpr int kRefinePasses = 6;

struct RefineState {
  float rad, lo, hi, frad;  // frad < 0: the original radius
  uint32_t total, full;     // in-radius counts at the original radius and at frad
  bool active, generic;
};

// After pass `pass` found c points: done, or the next radius in st.rad.
__device__ __forceinline__ void refine_step(RefineState& st, int pass, uint32_t c, uint32_t kmax, double radius) {
  if (pass == 0) {
    st.total = st.full = c;
    st.frad = -1.f;
    st.lo = 0.f;
    st.hi = __double2float_ru(radius);
    st.rad = st.hi;
  }
  if (c <= (uint32_t)kSlab && (pass == 0 || c >= kmax)) {
    st.active = false;
    return;
  }
  if (pass > 0) {
    if (c > (uint32_t)kSlab && c < st.full) {
      st.full = c;
      st.frad = st.rad;
    }
    if (c < kmax) st.lo = st.rad;
    else st.hi = st.rad;
  }
  if (kmax > (uint32_t)kMaxList || pass == kRefinePasses) {
    st.active = false;
    st.generic = true;
    return;
  }
  float est = st.rad * cbrtf(2.0f * (float)kmax / (float)(c > 0u ? c : 1u));
  if (!(est > st.lo && est < st.hi)) est = 0.5f * (st.lo + st.hi);
  st.rad = est;
}

__device__ __forceinline__ void collect_finish(const CollectParams& P, uint32_t t, uint32_t qin,
                                               const RefineState& st, uint32_t points, uint32_t kmax,
                                               double radius) {
  if (P.stats) {
    atomicAdd(&P.stats[kStatInRadius], (unsigned long long)st.total);
    atomicMax(&P.stats[kStatMaxLeafPoints], (unsigned long long)st.total);
    if (st.total > (uint32_t)kSlab && !st.generic) atomicAdd(&P.stats[kStatRefined], 1ull);
    if (points > 64u && !st.generic) atomicAdd(&P.stats[kStatLargeQueries], 1ull);
  }
  P.counts[qin] = st.total < kmax ? st.total : kmax;
  const bool over = st.total > kmax;
  uint32_t meta = ((kmax < (uint32_t)kSlab ? kmax : (uint32_t)kSlab) << kQueryKmaxShift);
  if (st.generic) {
    meta |= kQueryGeneric;
    const unsigned int h = atomicAdd(&P.small[0], 1u);
    P.heavy_list[h] = qin;
    P.heavy_m[h] = st.full;
    P.heavy_rad[h] = st.frad < 0.f ? radius : (double)st.frad;
    P.heavy_t[h] = t;
  } else {
    meta |= points;
    if (points > 128u) {
      meta |= kQueryBig;
      P.big_list[atomicAdd(&P.small[3], 1u)] = t;
    } else if (points > 64u) {
      meta |= kQueryBig;
      P.mid_list[atomicAdd(&P.small[2], 1u)] = t;
    }
  }
  const double* r = P.qraw + (size_t)qin * P.qstride;
  QueryInfo qi;
  qi.ex = r[1];
  qi.ey = r[2];
  qi.ez = P.qstride == 4 ? r[3] : 0.0;
  qi.qid = __float_as_uint(P.qpts[qin].w);
  qi.meta = meta;
  P.qinfo[t] = qi;
  P.flags[qin] = (over ? 1 : 0) | (st.generic ? 2 : 0);
  if (P.overflow_out) P.overflow_out[qin] = over ? 1 : 0;
}

// The record of a KNN query (no points: k_knn_single writes its rows).
__device__ __forceinline__ void collect_finish_knn(const CollectParams& P, uint32_t t, uint32_t qin,
                                                   uint32_t points, uint32_t kmax) {
  if (P.stats && points) {  // (k_knn_single counts its own)
    atomicAdd(&P.stats[kStatInRadius], (unsigned long long)points);
    atomicMax(&P.stats[kStatMaxLeafPoints], (unsigned long long)points);
    if (points > 64u) atomicAdd(&P.stats[kStatLargeQueries], 1ull);
  }
  uint32_t meta = points ? kmax << kQueryKmaxShift | points : 0u;
  if (points > 128u) {
    meta |= kQueryBig;
    P.big_list[atomicAdd(&P.small[3], 1u)] = t;
  } else if (points > 64u) {
    meta |= kQueryBig;
    P.mid_list[atomicAdd(&P.small[2], 1u)] = t;
  }
  const double* r = P.qraw + (size_t)qin * P.qstride;
  P.qinfo[t] = QueryInfo{r[1], r[2], P.qstride == 4 ? r[3] : 0.0, __float_as_uint(P.qpts[qin].w), meta};
}

// One warp per 32 curve-consecutive queries (a packet): the warp walks the
// wide tree once for the box around them (or around each run of them that is
// worth it, see cut_packet), then tests every reached bucket's eight points
// with each lane's query.  Node, bucket and control flow are warp-uniform.
// BATCH: several problems (a problem batch, or several requests on one scene):
// each warp has one problem, its tree, its bands and its kmax.  OWN: every
// query has a radius of its own (KNN).
// A packet of the clustered 1M x 1M sets takes 18 node steps and 87 buckets of
// about 45 instructions each; what bounds it is the bucket loads (load/store pipe
// 63% busy, issue 49%, 20 warps per SM to wait on them).
template <int DIM, bool BATCH, bool OWN>
__device__ __forceinline__ void collect_packet_body(const CollectParams& P, uint32_t t, CollectWarp& W) {
  const int lane = threadIdx.x & 31;
  // a problem batch pads every problem to whole warps, so a warp has one problem
  // (lanes past the packet's width hold no rank: the problem is lane 0's)
  const uint32_t prob = BATCH ? P.warp_prob[(t - (uint32_t)lane) >> 5] : 0u;
  const bool rank = (uint32_t)lane < P.width && t < P.nq;
  const uint32_t qin = rank ? P.qorder[t] : kNone;
  const bool valid = qin != kNone;
  if (BATCH && !valid && rank) P.qinfo[t] = QueryInfo{0.0, 0.0, 0.0, 0u, 0u};  // padding: nothing to emit
  const uint32_t kmax = BATCH ? P.prob_kmax[prob] : P.kmax;
  const double radius = OWN ? (valid ? P.rank_radius[t] : 0.0) : BATCH ? P.prob_radius[prob] : P.radius;
  const TreeShape* T = P.S.trees + (BATCH ? prob * P.S.tree_stride : 0u);
  const int scene_inexact = *P.S.inexact;
  const float4 q = valid ? P.qpts[qin] : make_float4(0.f, 0.f, 0.f, 0.f);
  DevBands B = P.bands[prob];
  if (OWN) B = bands_at_radius(B, radius);
  RefineState st{};
  st.active = valid;
  bool left = false;  // to k_collect_single
  uint32_t count = 0;
  for (int pass = 0;; ++pass) {
    cut_packet(
        P.S, T, q, B.box_hi2, OWN || pass > 0, st.active, W.stack, lane,
        [&](bool mine, const PacketBox& box, const PacketBox* limit, float reach2) {
          collect_walk<DIM, !OWN>(P, T, B, scene_inexact, q, qin, t, mine, W, lane, box, limit, reach2, &count);
        },
        [&](uint32_t run) {
          if (OWN || pass == 0) {  // a warp of its own for each of them
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&P.small[6], (unsigned int)__popc(run));
            at = __shfl_sync(0xffffffffu, at, 0);
            if ((run >> lane) & 1u) {
              P.single_list[at + __popc(run & ((1u << lane) - 1u))] = t;
              left = true;
            }
          } else {
            for (; run; run &= run - 1u) {
              const int from = __ffs((int)run) - 1;
              const DevBands one = bands_at_radius(P.bands[prob], (double)__shfl_sync(0xffffffffu, st.rad, from));
              const uint32_t c = collect_alone(P, T, one, scene_inexact, __shfl_sync(0xffffffffu, qin, from),
                                               __shfl_sync(0xffffffffu, t, from), W.stack);
              if (lane == from) count = c;
            }
          }
        });
    if (left) st.active = false;
    if (OWN) break;
    if (st.active) refine_step(st, pass, count, kmax, radius);
    if (!__any_sync(0xffffffffu, st.active)) break;
    B = bands_at_radius(P.bands[prob], (double)st.rad);
  }
  if (OWN) {
    // a radius that holds too many points (it only bounds the k-th distance):
    // k_knn_single finds the k nearest with a shrinking one
    const bool heavy = valid && !left && count > (uint32_t)kSlab;
    const uint32_t m = __ballot_sync(0xffffffffu, heavy);
    if (m) {
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(&P.small[6], (unsigned int)__popc(m));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (heavy) P.single_list[at + __popc(m & ((1u << lane) - 1u))] = t;
    }
    if (valid) collect_finish_knn(P, t, qin, left || heavy ? 0u : count, kmax);
    return;
  }
  if (valid && !left) collect_finish(P, t, qin, st, count, kmax, radius);
}

constexpr int kCollectThreads = 128;

template <int DIM, bool BATCH, bool OWN>
__global__ void __launch_bounds__(kCollectThreads, OWN ? 6 : 7) k_collect_packet(const __grid_constant__ CollectParams P) {
  __shared__ CollectWarp warps[kCollectThreads / 32];
  const uint32_t t = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * P.width + (threadIdx.x & 31);
  if (!__any_sync(0xffffffffu, t < P.nq)) return;  // whole warp past the end
  collect_packet_body<DIM, BATCH, OWN>(P, t, warps[threadIdx.x >> 5]);
}

// One warp per query: every query of a call too small to fill the GPU with
// packets (`listed` false), where the walk's latency is what counts, or those
// the packets left.
__global__ void __launch_bounds__(128) k_collect_single(const __grid_constant__ CollectParams P, bool listed) {
  __shared__ WalkStack stacks[128 / 32];
  const int lane = threadIdx.x & 31;
  const uint32_t n = listed ? P.small[6] : P.nq;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; j < n; j += warps) {
    const uint32_t t = listed ? P.single_list[j] : j;
    const uint32_t qin = P.qorder[t];
    if (qin == kNone) {
      if (lane == 0) P.qinfo[t] = QueryInfo{0.0, 0.0, 0.0, 0u, 0u};
      continue;
    }
    const uint32_t prob = P.warp_prob ? P.warp_prob[t >> 5] : 0u;
    const uint32_t kmax = P.warp_prob ? P.prob_kmax[prob] : P.kmax;
    const double radius = P.warp_prob ? P.prob_radius[prob] : P.radius;
    DevBands B = P.bands[prob];
    RefineState st{};
    st.active = true;
    uint32_t count;
    for (int pass = 0;; ++pass) {
      count = collect_alone(P, P.S.trees + prob * P.S.tree_stride, B, *P.S.inexact, qin, t, stacks[threadIdx.x >> 5]);
      refine_step(st, pass, count, kmax, radius);
      if (!st.active) break;
      B = bands_at_radius(P.bands[prob], (double)st.rad);
    }
    if (lane == 0) collect_finish(P, t, qin, st, count, kmax, radius);
  }
}

// ---- emit ---------------------------------------------------------------------
// Emitted row writer.
struct RowSink {
  void* rows;
  unsigned long long capacity;
  int ranked;
  __device__ __forceinline__ void put(unsigned long long row, uint32_t qid, uint32_t nid, double dist,
                                      uint32_t rank) const {
    if (row >= capacity) return;
    const unsigned long long db = (unsigned long long)__double_as_longlong(dist);
    if (!ranked) {
      reinterpret_cast<uint4*>(rows)[row] = make_uint4(qid, nid, (uint32_t)db, (uint32_t)(db >> 32));
    } else {
      uint2* out = reinterpret_cast<uint2*>(static_cast<char*>(rows) + row * 24);
      out[0] = make_uint2(qid, nid);
      out[1] = make_uint2((uint32_t)db, (uint32_t)(db >> 32));
      out[2] = make_uint2(rank, 0u);
    }
  }
};

struct EmitParams {
  SceneView S;
  uint32_t nq;
  const uint32_t* slab;
  const QueryInfo* qinfo;     // by processing rank
  const unsigned long long* poff;  // first row of each query, by processing rank
  RowSink sink;
  uint32_t* fix_list;         // processing ranks queued for k_emit_fixup
  unsigned int* fix_count;
  // Emission of one range [out_lo, out_hi) of output ranks (rows copied to the
  // host range by range): k_emit takes the range's queries through `order`
  // (output rank -> processing rank), k_emit_mid and k_emit_big the range's part
  // [list_start[range], list_start[range + 1]) of its list partitioned by
  // range, and the fix-up the queue from `*fix_begin`.  All null: every
  // query at once.
  const uint32_t* order = nullptr;
  const unsigned int* list_start = nullptr;
  const unsigned int* fix_begin = nullptr;
  uint32_t out_lo = 0, out_hi = 0;
  int range = 0;
};

// Packed sort element: the exact FP64 d2 rounded to FP32 with its low SHIFT
// mantissa bits replaced by the candidate's slot.  Valid keys are below
// 0x80000000, so the padding value 0xFFFFFFFF sorts last.  Two elements whose
// truncated keys differ by two units or more are in exact order; closer pairs
// are re-decided exactly.
template <int SHIFT>
__device__ __forceinline__ uint32_t pack_key(uint32_t key_bits, uint32_t slot) {
  return (key_bits & ~((1u << SHIFT) - 1u)) | slot;
}

// Bitonic sort across the warp of 32 * E packed elements in a striped layout
// (element i = r * 32 + lane): exchanges at distance >= 32 stay in a lane's
// registers, shorter ones take one shuffle per register.  Ascending.
template <int E>
__device__ __forceinline__ void warp_bitonic_striped(uint32_t (&v)[E], int lane) {
#pragma unroll
  for (int k = 2; k <= 32 * E; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
        const int rj = j >> 5;
#pragma unroll
        for (int r = 0; r < E; ++r) {
          const int pr = r ^ rj;
          if (pr > r) {
            const bool up = (((r << 5) | lane) & k) == 0;
            const uint32_t a = v[r], b = v[pr];
            v[r] = up ? min(a, b) : max(a, b);
            v[pr] = up ? max(a, b) : min(a, b);
          }
        }
      } else {
        const bool lower = (lane & j) == 0;
#pragma unroll
        for (int r = 0; r < E; ++r) {
          const bool up = (((r << 5) | lane) & k) == 0;
          const uint32_t other = __shfl_xor_sync(0xffffffffu, v[r], j);
          v[r] = (lower == up) ? min(v[r], other) : max(v[r], other);
        }
      }
    }
  }
}

// Odd-even transposition over a warp's sorted buffer (the pairs of one parity
// are disjoint, so the lanes take them in parallel), restricted to neighbours
// whose truncated keys differ by at most one unit, until no swap happens
// (bounded by n passes).  Runs only when such a pair exists.  The exact distances
// and ids are the slots' in shared memory: on a lattice nearly every query comes
// here, and computing both distances anew for each comparison took k_emit_fixup
// 873 us for KNN k = 4 of 300k queries over 1M points, 397 so.
__device__ __noinline__ void exact_fixup_sorted(uint32_t* buf, int n, int shift, const double* dist,
                                                const uint32_t* nid, const uint32_t* cand, const uint32_t* perm,
                                                int lane) {
  const uint32_t mask = (1u << shift) - 1u;
  for (int pass = 0; pass < n; ++pass) {
    bool changed = false;
    for (int parity = 0; parity < 2; ++parity) {
      for (int i = parity + 2 * lane; i + 1 < n; i += 64) {
        const uint32_t a = buf[i], b = buf[i + 1];
        if ((b >> shift) - (a >> shift) > 1u) continue;
        const uint32_t sa = a & mask, sb = b & mask;
        bool swap = dist[sb] < dist[sa];
        if (dist[sb] == dist[sa])
          swap = nid[sb] != nid[sa] ? nid[sb] < nid[sa] : __ldg(&perm[cand[sb]]) < __ldg(&perm[cand[sa]]);
        if (swap) {
          buf[i] = b;
          buf[i + 1] = a;
          changed = true;
        }
      }
      __syncwarp();
    }
    if (!__any_sync(0xffffffffu, changed)) break;
  }
}

// Only the first kk of a query's n sorted candidates become rows.  An element
// whose truncated key is two units or more above that of element kk - 1
// orders after every element up to kk - 1 exactly as well, so the exact
// re-decision of near ties only has to cover the first m elements: those
// within one unit of element kk - 1 or below it (m = n when kk = n).  `v`
// holds the warp-sorted packed keys in the striped layout (padding
// 0xFFFFFFFF); every lane returns the same m.
template <int E, int SHIFT>
__device__ __forceinline__ int exact_window(const uint32_t (&v)[E], int n, int kk, int lane) {
  if (kk >= n) return n;
  const int c = kk - 1;
  uint32_t vc = v[0];
#pragma unroll
  for (int r = 1; r < E; ++r)
    if ((c >> 5) == r) vc = v[r];
  const uint32_t limit = (__shfl_sync(0xffffffffu, vc, c & 31) >> SHIFT) + 1u;
  int m = 0;
#pragma unroll
  for (int r = 0; r < E; ++r) m += __popc(__ballot_sync(0xffffffffu, v[r] != 0xFFFFFFFFu && (v[r] >> SHIFT) <= limit));
  return m;
}

// What a warp needs of one query before it sorts: three independent loads (the
// query's record, its first row and candidate `lane`), so a query costs one
// memory round trip before the point gather.
struct EmitQuery {
  QueryInfo qi;
  unsigned long long base;  // first row of the query
  uint32_t i0;              // candidate `lane` (read before the count is known; unused beyond it)
};

__device__ __forceinline__ void emit_load(const EmitParams& P, uint32_t t, int lane, EmitQuery& q) {
  q.qi = P.qinfo[t];
  q.base = P.poff[t];
  q.i0 = P.slab[slab_base(t) + lane];  // inside the query's kSlab entries whatever its count
}

// Per-warp shared memory of an emit: distance and id of each candidate, for the
// lane that writes its row.
template <int E>
struct EmitWarp {
  double dist[32 * E];
  uint32_t nid[32 * E];
};

// Sorts the query's n <= 32 * E candidates by the reference's key and writes
// its first min(n, kmax) rows; lane l writes rows l, l + 32, ... so each store
// instruction covers 32 consecutive rows.  The points are gathered once: the
// exact distance gives the sort key, and waits in shared memory for the lane
// that writes the row.  Neighbours that need the exact comparison are re-decided
// through `wbuf` and `cand` (shared memory, 32 * E words each).
template <int E>
__device__ __forceinline__ void emit_query(const EmitParams& P, uint32_t t, const EmitQuery& q, int n, int lane,
                                           EmitWarp<E>& W, uint32_t* cand, uint32_t* wbuf) {
  constexpr int SHIFT = E == 4 ? 7 : 8;
  constexpr uint32_t kMask = (1u << SHIFT) - 1u;
  const double ex = q.qi.ex, ey = q.qi.ey, ez = q.qi.ez;
  const int inexact = *P.S.inexact;
  uint32_t v[E];
#pragma unroll
  for (int r = 0; r < E; ++r) {
    const int s = (r << 5) | lane;
    v[r] = 0xFFFFFFFFu;
    if (s < n) {
      const uint32_t i = r == 0 ? q.i0 : P.slab[slab_base(t) + s];
      const float4 p = __ldg(&P.S.pts[i]);
      double sx = p.x, sy = p.y, sz = p.z;
      if (inexact) {
        const double* pp = P.S.pts64 + 3ull * i;
        sx = pp[0];
        sy = pp[1];
        sz = pp[2];
      }
      const double dx = __dsub_rn(sx, ex), dy = __dsub_rn(sy, ey), dz = __dsub_rn(sz, ez);
      const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
      v[r] = pack_key<SHIFT>(__float_as_uint(__double2float_rn(d2)), (uint32_t)s);
      W.dist[s] = __dsqrt_rn(d2);
      W.nid[s] = __float_as_uint(p.w);
      cand[s] = i;
    }
  }
  warp_bitonic_striped<E>(v, lane);
  const int kmax = query_kmax(q.qi.meta);
  const int kk = n < kmax ? n : kmax;
  const int m = exact_window<E, SHIFT>(v, n, kk, lane);
  // ambiguous neighbours inside the window: element i and i + 1 within one truncated unit
  bool amb = false;
#pragma unroll
  for (int r = 0; r < E; ++r) {
    uint32_t nx = __shfl_down_sync(0xffffffffu, v[r], 1);
    const uint32_t wrap = __shfl_sync(0xffffffffu, v[r + 1 < E ? r + 1 : r], 0);
    if (lane == 31) nx = r + 1 < E ? wrap : 0xFFFFFFFFu;
    amb |= ((r << 5) | lane) + 1 < m && (nx >> SHIFT) - (v[r] >> SHIFT) <= 1u;
  }
  if (__any_sync(0xffffffffu, amb)) {
#pragma unroll
    for (int r = 0; r < E; ++r) wbuf[(r << 5) | lane] = v[r];
    __syncwarp();
    exact_fixup_sorted(wbuf, m, SHIFT, W.dist, W.nid, cand, P.S.perm, lane);
#pragma unroll
    for (int r = 0; r < E; ++r) v[r] = wbuf[(r << 5) | lane];
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < E; ++r) {
    const int i = (r << 5) | lane;
    if (i < kk) {
      const uint32_t slot = v[r] & kMask;
      P.sink.put(q.base + i, q.qi.qid, W.nid[slot], W.dist[slot], (uint32_t)i + 1);
    }
  }
  __syncwarp();  // the shared memory is free again
}

// ---- emit: a group of lanes per query ---------------------------------------
// Sorted keys of a group of GL lanes, R per lane: element lane * R + r.  Each
// merge starts by comparing element e of a block with its mirror image, so all
// later steps ascend: the steps inside a lane are plain min/max pairs, and only
// a stride of R elements or more takes a shuffle.  64 keys cost 6 shuffles a
// register over 8 lanes (12 per query), where a warp with two keys a lane
// needs 40 per query.
template <int GL, int R>
__device__ __forceinline__ void group_sort(uint32_t (&v)[R], int gl) {
#pragma unroll
  for (int k = 2; k <= GL * R; k <<= 1) {
    if (k <= R) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int o = r ^ (k - 1);
        if (o > r) {
          const uint32_t a = v[r], b = v[o];
          v[r] = min(a, b);
          v[o] = max(a, b);
        }
      }
    } else {
      const bool lower = (gl & (k / R / 2)) == 0;
      uint32_t w[R];
#pragma unroll
      for (int r = 0; r < R; ++r) w[r] = __shfl_xor_sync(0xffffffffu, v[R - 1 - r], k / R - 1);
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = lower ? min(v[r], w[r]) : max(v[r], w[r]);
    }
#pragma unroll
    for (int j = k >> 2; j > 0; j >>= 1) {
      if (j >= R) {
        const bool lower = (gl & (j / R)) == 0;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint32_t w = __shfl_xor_sync(0xffffffffu, v[r], j / R);
          v[r] = lower ? min(v[r], w) : max(v[r], w);
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int o = r ^ j;
          if (o > r) {
            const uint32_t a = v[r], b = v[o];
            v[r] = min(a, b);
            v[o] = max(a, b);
          }
        }
      }
    }
  }
}

// Shared memory of a warp whose groups of GL lanes hold up to 8 * GL candidates
// each: exact squared distance and id by slot, and the slots in sorted order.
// The rows are padded so that the groups of a warp use different banks.
template <int GL>
struct EmitGroups {
  static constexpr int kGroups = 32 / GL, kCap = 8 * GL;
  double d2[kGroups][kCap + 8];
  uint32_t nid[kGroups][kCap + 8];
  uint8_t slot[kGroups][kCap + 8];
};

// Sorts a group's n <= GL * R candidates by the reference's key and writes its
// first min(n, kmax) rows (n == 0: the group has nothing to do).  The points are
// gathered once, four loads of a lane in flight; the square root is taken only
// for the rows that are written.  A query whose near ties need the exact
// comparison is queued for k_emit_fixup.  All lanes of the warp call this.
template <int GL, int R>
__device__ __forceinline__ void emit_group(const EmitParams& P, uint32_t t, const QueryInfo& qi,
                                           unsigned long long base, const uint32_t (&first)[4], int n, int nmax,
                                           int lane, EmitGroups<GL>& W) {
  constexpr int SHIFT = GL * R == 16 ? 4 : GL * R == 32 ? 5 : GL * R == 64 ? 6 : 7;
  static_assert(GL * R == 1 << SHIFT, "a slot fills the key's low bits");
  constexpr uint32_t kMask = (1u << SHIFT) - 1u;
  constexpr int H = R < 4 ? R : 4;
  const int gl = lane & (GL - 1), g = lane / GL;
  const int inexact = *P.S.inexact;
  uint32_t v[R];
#pragma unroll
  for (int h = 0; h < R; h += H) {
#pragma unroll
    for (int r = h; r < h + H; ++r) v[r] = 0xFFFFFFFFu;
    if (h * GL >= nmax) continue;  // nothing here in any group
    uint32_t id[H];
    float4 p[H];
#pragma unroll
    for (int r = 0; r < H; ++r) {
      const int s = (h + r) * GL + gl;
      id[r] = 0;
      if (s < n) id[r] = h == 0 ? first[r] : P.slab[slab_base(t) + s];
    }
#pragma unroll
    for (int r = 0; r < H; ++r) p[r] = __ldg(&P.S.pts[id[r]]);
#pragma unroll
    for (int r = 0; r < H; ++r) {
      const int s = (h + r) * GL + gl;
      if (s < n) {
        double sx = p[r].x, sy = p[r].y, sz = p[r].z;
        if (inexact) {
          const double* pp = P.S.pts64 + 3ull * id[r];
          sx = pp[0];
          sy = pp[1];
          sz = pp[2];
        }
        const double dx = __dsub_rn(sx, qi.ex), dy = __dsub_rn(sy, qi.ey), dz = __dsub_rn(sz, qi.ez);
        const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
        v[h + r] = pack_key<SHIFT>(__float_as_uint(__double2float_rn(d2)), (uint32_t)s);
        W.d2[g][s] = d2;
        W.nid[g][s] = __float_as_uint(p[r].w);
      }
    }
  }
  group_sort<GL, R>(v, gl);
  const int kmax = query_kmax(qi.meta);
  const int kk = n < kmax ? n : kmax;
  // Near ties matter among the elements that can become rows: up to one unit
  // above element kk - 1 (all of them when every candidate is a row).
  uint32_t limit = 0x7FFFFFFFu >> SHIFT;
  {
    const int c = kk > 0 ? kk - 1 : 0;
    uint32_t vc = v[0];
#pragma unroll
    for (int r = 1; r < R; ++r)
      if ((c & (R - 1)) == r) vc = v[r];
    vc = __shfl_sync(0xffffffffu, vc, c / R, GL);
    if (kk < n) limit = (vc >> SHIFT) + 1u;
  }
  uint32_t next = __shfl_down_sync(0xffffffffu, v[0], 1, GL);
  if (gl == GL - 1) next = 0xFFFFFFFFu;
  bool amb = false;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t nx = (r + 1 < R ? v[r + 1 < R ? r + 1 : r] : next) >> SHIFT;
    amb |= nx <= limit && nx - (v[r] >> SHIFT) <= 1u;
  }
  const unsigned int any = __ballot_sync(0xffffffffu, amb) >> (lane & ~(GL - 1));
  const bool defer = (any & (GL == 32 ? 0xFFFFFFFFu : (1u << (GL & 31)) - 1u)) != 0;
  if (defer && gl == 0) P.fix_list[atomicAdd(P.fix_count, 1u)] = t;
  if (R == 2) {
    *reinterpret_cast<uint16_t*>(&W.slot[g][gl * R]) = (uint16_t)((v[0] & kMask) | (v[1] & kMask) << 8);
  } else {
#pragma unroll
    for (int r = 0; r < R; r += 4)
      *reinterpret_cast<uint32_t*>(&W.slot[g][gl * R + r]) =
          (v[r] & kMask) | (v[r + 1 < R ? r + 1 : r] & kMask) << 8 | (v[r + 2 < R ? r + 2 : r] & kMask) << 16 |
          (v[r + 3 < R ? r + 3 : r] & kMask) << 24;
  }
  __syncwarp();
  const int rows = defer ? 0 : kk;
  for (int i = gl; i < rows; i += GL) {
    const uint32_t slot = W.slot[g][i];
    P.sink.put(base + i, qi.qid, W.nid[g][slot], __dsqrt_rn(W.d2[g][slot]), (uint32_t)i + 1);
  }
  __syncwarp();  // the shared memory is free again
}

// A warp's 32 / GL queries (t of this lane's group; live: the group has one that
// is this kernel's): the records, first rows and first candidates in one round
// trip, then the network for the largest count in the warp.
template <int GL>
__device__ __forceinline__ void emit_groups(const EmitParams& P, uint32_t t, bool live, uint32_t skip, int lane,
                                            EmitGroups<GL>& W) {
  const QueryInfo qi = P.qinfo[t];
  const unsigned long long base = P.poff[t];
  uint32_t first[4];  // read before the count is known; inside the query's kSlab entries whatever it is
#pragma unroll
  for (int r = 0; r < 4; ++r) first[r] = P.slab[slab_base(t) + r * GL + (lane & (GL - 1))];
  const int n = live && !(qi.meta & skip) ? (int)(qi.meta & kQueryCountMask) : 0;
  const int nmax = (int)__reduce_max_sync(0xffffffffu, (unsigned int)n);
  if (nmax == 0) return;
  if (nmax <= 2 * GL) emit_group<GL, 2>(P, t, qi, base, first, n, nmax, lane, W);
  else if (nmax <= 4 * GL) emit_group<GL, 4>(P, t, qi, base, first, n, nmax, lane, W);
  else emit_group<GL, 8>(P, t, qi, base, first, n, nmax, lane, W);
}

// Queries with at most 64 candidates in processing (curve) order, eight lanes
// each (1M clustered queries: 253 us; a warp each took 325, with the load/store
// pipe 71% busy, half of it shuffles).  Bound by the latency of the point
// gathers.  Queries with 65..kSlab candidates are k_emit_mid's and k_emit_big's, those on the
// generic path get their rows from k_expand.
constexpr int kEmitThreads = 256;
constexpr int kEmitLanes = 8;

// The grid fills the GPU once (emit_grid) and each warp strides over the
// queries: a warp takes its next four as soon as it is done with some, instead
// of short blocks retiring and launching.  Four blocks: 64 registers without
// spills (three blocks 2460, five 2361 and four 2264 us for a batch's emit phase).
constexpr int kEmitBlocksPerSm = 4;

__global__ void __launch_bounds__(kEmitThreads, kEmitBlocksPerSm) k_emit(const __grid_constant__ EmitParams P) {
  __shared__ EmitGroups<kEmitLanes> shared[kEmitThreads / 32];
  constexpr uint32_t kQueries = 32 / kEmitLanes;
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (kEmitThreads / 32);
  const uint32_t total = P.order ? P.out_hi - P.out_lo : P.nq;  // P.order: one range of output ranks
  for (uint32_t w = blockIdx.x * (kEmitThreads / 32) + (threadIdx.x >> 5); (uint64_t)w * kQueries < total; w += warps) {
    const uint32_t j = w * kQueries + lane / kEmitLanes;
    const bool live = j < total;
    const uint32_t o = live ? j : total - 1;
    emit_groups<kEmitLanes>(P, P.order ? P.order[P.out_lo + o] : o, live, kQueryGeneric | kQueryBig, lane,
                            shared[threadIdx.x >> 5]);
  }
}

// Blocks of k_emit for `queries` queries: one resident wave at most.
inline unsigned int emit_grid(uint64_t queries) {
  const uint64_t blocks = div_up(queries * kEmitLanes, (uint64_t)kEmitThreads);
  const uint64_t cap = (uint64_t)kSmCount * kEmitBlocksPerSm;
  return (unsigned int)(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

// The queries the emit kernels queued (at most 128 candidates), one warp per
// query, near ties decided in place.  The queue length is read on the device,
// so no host round trip is needed.
constexpr int kFixupThreads = 128;

__global__ void __launch_bounds__(kFixupThreads) k_emit_fixup(const __grid_constant__ EmitParams P) {
  __shared__ EmitWarp<4> shared[kFixupThreads / 32];
  __shared__ uint32_t cands[kFixupThreads / 32][128], keys[kFixupThreads / 32][128];
  const unsigned int m = *P.fix_count;
  const unsigned int first = P.fix_begin ? *P.fix_begin : 0u;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t j = first + (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); j < m; j += warps) {
    const uint32_t t = P.fix_list[j];
    EmitQuery q;
    emit_load(P, t, lane, q);
    emit_query<4>(P, t, q, (int)(q.qi.meta & kQueryCountMask), lane, shared[warp], cands[warp], keys[warp]);
  }
}

// ---- k nearest ---------------------------------------------------------------
// k <= 64 goes through the fixed-radius machinery: a radius that holds every
// query's k nearest is read off the points around its place on the curve,
// the collect gathers what lies within it, and the emit sorts and keeps k.

// First sorted point whose curve code is not below `code`.
__device__ __forceinline__ uint32_t curve_position(const uint32_t* __restrict__ codes, uint32_t n, uint32_t code) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(&codes[mid]) < code) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Ascending bitonic steps over a thread's registers: a full sort, or (MERGE)
// only the last merge of a bitonic sequence.
template <int N, bool MERGE>
__device__ __forceinline__ void thread_bitonic(float (&v)[N]) {
#pragma unroll
  for (int k = MERGE ? N : 2; k <= N; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const int o = i ^ j;
        if (o > i) {
          const bool up = (i & k) == 0 || k == N;
          const float a = v[i], b = v[o];
          v[i] = up ? fminf(a, b) : fmaxf(a, b);
          v[o] = up ? fmaxf(a, b) : fminf(a, b);
        }
      }
    }
  }
}

// A radius that holds each query's k nearest (k <= KP): the k-th smallest FP32
// distance among the 4 KP points around the query's place on the curve, widened
// by the FP32 error.  One thread per query keeps the KP smallest in registers:
// each further KP distances are sorted by a bitonic network and merged, about
// 20 instructions per point and lane and no shared memory.  On the clustered
// 1M x 1M sets 4 KP points bound k = 16 by 46 points on average (2 KP: 71,
// 8 KP: 37, at twice this kernel's cost).
template <int DIM, int KP>
__global__ void __launch_bounds__(128) k_knn_radius(SceneView S, const uint32_t* __restrict__ scodes,
                                                   const float4* __restrict__ qpts,
                                                   const uint32_t* __restrict__ qorder,
                                                   const uint32_t* __restrict__ qcodes, uint32_t nq, uint32_t k,
                                                   const DevBands* bands, double* __restrict__ radius) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nq) return;
  const float4 q = qpts[qorder[t]];
  const uint32_t buckets = (S.n + kBucketPoints - 1) / kBucketPoints;
  constexpr uint32_t kWindow = KP / 2;  // buckets
  const uint32_t at = curve_position(scodes, S.n, qcodes[t]) / kBucketPoints;
  uint32_t b0 = at > kWindow / 2 ? at - kWindow / 2 : 0u;
  if (b0 + kWindow > buckets) b0 = buckets > kWindow ? buckets - kWindow : 0u;
  BucketQuery bq;
  bq.set(q.x, q.y, q.z, 0.f);
  float best[KP];
#pragma unroll
  for (int i = 0; i < KP; ++i) best[i] = INFINITY;
  for (uint32_t w = 0; w < kWindow; w += KP / 8) {
    float v[KP];
#pragma unroll
    for (int g = 0; g < KP / 8; ++g) {
      const uint32_t b = b0 + w + g;
      float d2[8];
      bucket_d2<DIM>(S.bucket_pts, b < buckets ? b : buckets - 1, bq, d2);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[8 * g + j] = b < buckets ? d2[j] : INFINITY;
    }
    thread_bitonic<KP, false>(v);
#pragma unroll
    for (int i = 0; i < KP; ++i) best[i] = fminf(best[i], v[KP - 1 - i]);
    thread_bitonic<KP, true>(best);
  }
  const uint32_t kk = k < S.n ? k : S.n;
  float r2 = best[KP - 1];
#pragma unroll
  for (int i = 0; i < KP - 1; ++i)
    if ((uint32_t)i + 1 == kk) r2 = best[i];
  // 1e-22 covers squares that underflow
  radius[t] = sqrt((double)r2) * (1.0 + (double)bands->rho) + (double)bands->e_abs + 1.0e-22;
}

// k nearest of single queries, a warp per query: the sorted list of the k best
// lies in registers (entry l and l + 32 in lane l) under the exact order
// (FP64 distance, id, search input index), and the walk's reach shrinks with its
// last entry.  For the few queries whose radius holds more points than a slab
// row (duplicates, mixed densities), and for callers without scratch.  Where
// many points tie at the k-th distance the time is the points', so 32 of them are
// compared with the last entry at once and only what orders before it is
// inserted, a warp step each: k = 16 of 100k queries over 200 sites of 1,000
// points 7.45 -> 1.86 ms (every point inserted or refused by itself before).
struct SingleParams {
  SceneView S;
  const float4* qpts;
  const double* qraw;
  int qstride;
  const DevBands* bands;
  uint32_t k;
  const uint32_t* work;           // processing ranks (nullptr: every rank)
  const unsigned int* nwork_dev;  // their number (nullptr: nwork)
  uint32_t nwork;
  const uint32_t* qorder;         // processing rank -> query input index
  const double* rank_radius;      // a radius that holds the k nearest, by processing rank
  const uint32_t* qcodes;         // without rank_radius: curve codes by processing rank
  const uint32_t* scodes;
  const unsigned long long* poff; // rows: first row by processing rank
  RowSink sink;
  uint32_t* nearest;              // instead of rows: the nearest point by query input index
  unsigned long long* stats;      // STATS
};

struct SingleEntry {
  double d;
  uint32_t i;
};
__device__ __forceinline__ bool entry_before(const SceneView& S, const SingleEntry& a, const SingleEntry& b) {
  if (a.d != b.d) return a.d < b.d;
  if (a.i == kNone || b.i == kNone) return b.i == kNone && a.i != kNone;
  const uint32_t na = __float_as_uint(__ldg(&S.pts[a.i].w)), nb = __float_as_uint(__ldg(&S.pts[b.i].w));
  if (na != nb) return na < nb;
  return __ldg(&S.perm[a.i]) < __ldg(&S.perm[b.i]);
}

// STATS: counts the points within reach (a counter in the plain form cost 6% of
// a served k = 32 call).
template <bool STATS>
__global__ void __launch_bounds__(256) k_knn_single(SingleParams P) {
  __shared__ WalkStack stacks[256 / 32];
  const int lane = threadIdx.x & 31;
  const SceneView& S = P.S;
  const uint32_t n = P.nwork_dev ? *P.nwork_dev : P.nwork;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  const DevBands B = *P.bands;
  const int scene_inexact = *S.inexact;
  for (uint32_t j = (uint32_t)(((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); j < n; j += warps) {
    const uint32_t t = P.work ? P.work[j] : j;
    const uint32_t qin = P.qorder ? P.qorder[t] : t;
    const float4 q = P.qpts[qin];
    const double* rq = P.qraw + (size_t)qin * P.qstride;
    const double ex = rq[1], ey = rq[2], ez = P.qstride == 4 ? rq[3] : 0.0;
    double r;
    if (P.rank_radius) {
      r = P.rank_radius[t];
    } else {  // k = 1: the nearest of the 32 points around the query's place on the curve
      const uint32_t at = curve_position(P.scodes, S.n, P.qcodes[t]);
      uint32_t a = at > 16u ? at - 16u : 0u;
      if (a + 32u > S.n) a = S.n > 32u ? S.n - 32u : 0u;
      const float4 p = __ldg(&S.pts[a + (uint32_t)lane < S.n ? a + lane : a]);
      const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
      const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
      r = sqrt((double)__uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(d2)))) *
              (1.0 + (double)B.rho) + (double)B.e_abs + 1.0e-22;
    }
    float hi2, reach2;
    auto set_reach = [&](double radius) {
      const double w = radius * (1.0 + (double)B.rho) + (double)B.e_abs + 1.0e-18;
      hi2 = fmaxf(__double2float_ru(w * w), B.floor2);
      reach2 = __fmul_ru(hi2, 1.000001f);
    };
    set_reach(r);
    SingleEntry e0{INFINITY, kNone}, e1{INFINITY, kNone}, kth{INFINITY, kNone};
    const int last = (int)(P.k < S.n ? P.k : S.n) - 1;
    uint32_t found = 0;
    walk_single(S, S.trees, q, reach2, stacks[threadIdx.x >> 5], lane, [&](uint32_t i, const float4& p, bool has) {
      const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
      const bool pass = has && fmaf(dz, dz, fmaf(dy, dy, dx * dx)) <= hi2;
      if (!__any_sync(0xffffffffu, pass)) return false;
      if (STATS) found += __popc(__ballot_sync(0xffffffffu, pass));
      SingleEntry mine{INFINITY, kNone};
      if (pass) mine = SingleEntry{__dsqrt_rn(exact_d2_at(ex, ey, ez, S.pts, S.pts64, scene_inexact, i)), i};
      // only what orders before the list's last entry is inserted, one at a time
      unsigned int m = __ballot_sync(0xffffffffu, pass && entry_before(S, mine, kth));
      bool changed = false;
      while (m) {
        const int from = __ffs((int)m) - 1;
        m &= m - 1u;
        const SingleEntry c{__shfl_sync(0xffffffffu, mine.d, from), __shfl_sync(0xffffffffu, mine.i, from)};
        const int pos = __popc(__ballot_sync(0xffffffffu, entry_before(S, e0, c))) +
                        __popc(__ballot_sync(0xffffffffu, entry_before(S, e1, c)));
        if (pos > last) continue;
        changed = true;
        SingleEntry u0{__shfl_up_sync(0xffffffffu, e0.d, 1), __shfl_up_sync(0xffffffffu, e0.i, 1)};
        SingleEntry u1{__shfl_up_sync(0xffffffffu, e1.d, 1), __shfl_up_sync(0xffffffffu, e1.i, 1)};
        const SingleEntry top{__shfl_sync(0xffffffffu, e0.d, 31), __shfl_sync(0xffffffffu, e0.i, 31)};
        if (lane == 0) u1 = top;
        if (lane >= pos) e0 = lane == pos ? c : u0;
        if (lane + 32 >= pos) e1 = lane + 32 == pos ? c : u1;
      }
      if (changed) {
        kth.d = __shfl_sync(0xffffffffu, last < 32 ? e0.d : e1.d, last & 31);
        kth.i = __shfl_sync(0xffffffffu, last < 32 ? e0.i : e1.i, last & 31);
        if (kth.d < r) {
          r = kth.d;
          set_reach(r);
        }
      }
      return false;
    });
    if (STATS && lane == 0) {
      atomicAdd(&P.stats[kStatInRadius], (unsigned long long)found);
      atomicMax(&P.stats[kStatMaxLeafPoints], (unsigned long long)found);
    }
    if (P.nearest) {
      if (lane == 0) P.nearest[qin] = e0.i == kNone ? 0u : e0.i;
      continue;
    }
    const unsigned long long base = P.poff[t];
    const uint32_t qid = __float_as_uint(q.w);
    if (lane <= last && e0.i != kNone)
      P.sink.put(base + lane, qid, __float_as_uint(__ldg(&S.pts[e0.i].w)), e0.d, (uint32_t)lane + 1);
    if (lane + 32 <= last && e1.i != kNone)
      P.sink.put(base + 32 + lane, qid, __float_as_uint(__ldg(&S.pts[e1.i].w)), e1.d, (uint32_t)lane + 33);
  }
}

// ---- nearest point and the Hausdorff witness ------------------------------------
struct Witness {
  unsigned long long dist;  // FP64 bits
  uint32_t qid, nid;
};
// max by (distance, -query_id, -neighbor_id)
__device__ __forceinline__ bool witness_better(const Witness& a, const Witness& b) {
  if (a.dist != b.dist) return a.dist > b.dist;
  if (a.qid != b.qid) return a.qid < b.qid;
  return a.nid < b.nid;
}

// The best witness of a warp, in every lane.
__device__ __forceinline__ Witness warp_witness(Witness best) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Witness other;
    other.dist = __shfl_xor_sync(0xffffffffu, best.dist, o);
    other.qid = __shfl_xor_sync(0xffffffffu, best.qid, o);
    other.nid = __shfl_xor_sync(0xffffffffu, best.nid, o);
    if (witness_better(other, best)) best = other;
  }
  return best;
}

// The nearest point of every query (directed Hausdorff), a packet of 32
// queries per warp.  The smallest distance among 32 points around a query's
// place on the curve bounds its search; the warp walks what that bound reaches
// and shrinks its reach as the lanes' bounds fall.  Points whose FP32 distances
// are closer than the error band are ordered exactly (FP64 distance, id,
// search input index).
struct NearestParams {
  SceneView S;
  const float4* qpts;
  const double* qraw;
  int qstride;
  const uint32_t* qorder;
  const uint32_t* qcodes;
  const uint32_t* scodes;
  uint32_t nq;
  const DevBands* bands;
  uint32_t* nearest;  // by query input index
};

// Whether point i at FP32 squared distance d2 orders before the best so far.
__device__ __forceinline__ bool nearer(const NearestParams& P, const Ctx& c, uint32_t qin, float d2, uint32_t i,
                                       float best, uint32_t besti) {
  if (besti == kNone) return true;
  const float tol = key_tol(c, fmaxf(d2, best));
  if (best - d2 > tol) return true;
  if (d2 - best > tol) return false;
  const double* rq = P.qraw + (size_t)qin * P.qstride;
  return exact_before(rq[1], rq[2], P.qstride == 4 ? rq[3] : 0.0, P.S.pts, P.S.pts64, P.S.perm, c.scene_inexact, i,
                      besti);
}

// The nearest point of one query by the whole warp (packets whose queries lie
// far apart); everything below `bound` may order first.
__device__ __noinline__ uint32_t nearest_alone(const NearestParams& P, const Ctx& c, uint32_t qin, float bound,
                                               WalkStack& stack) {
  const float4 q = P.qpts[qin];
  float best = INFINITY, reach2 = __fmul_ru(bound, 1.000001f);
  uint32_t besti = kNone;
  walk_single(P.S, P.S.trees, q, reach2, stack, (int)(threadIdx.x & 31),
              [&](uint32_t i, const float4& p, bool has) {
                const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
                const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                for (uint32_t m = __ballot_sync(0xffffffffu, has && d2 < bound); m; m &= m - 1u) {
                  const int from = __ffs((int)m) - 1;
                  const float cd = __shfl_sync(0xffffffffu, d2, from);
                  const uint32_t ci = __shfl_sync(0xffffffffu, i, from);
                  if (!nearer(P, c, qin, cd, ci, best, besti)) continue;
                  best = cd;
                  besti = ci;
                  bound = fminf(bound, best + key_tol(c, best));
                  reach2 = __fmul_ru(bound, 1.000001f);
                }
                return false;
              });
  return besti;
}

// 64 registers, eight blocks per SM: the walk waits on its bucket loads, and 80
// registers left 22 warps to hide them (4M 2D queries, whole call: 1534 us at 80,
// 1439 at 72, 1424 at 64).
template <int DIM>
__global__ void __launch_bounds__(128, 8) k_nearest(const __grid_constant__ NearestParams P) {
  __shared__ PacketWarp warps[128 / 32];
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (!__any_sync(0xffffffffu, t < P.nq)) return;  // whole warp past the end
  const bool valid = t < P.nq;
  const int lane = threadIdx.x & 31;
  const SceneView& S = P.S;
  const uint32_t tq = valid ? t : P.nq - 1;
  const uint32_t qin = P.qorder[tq];
  const float4 q = P.qpts[qin];
  const DevBands B = *P.bands;
  Ctx c;
  c.scene_inexact = *S.inexact;
  c.rho = B.rho;
  c.e_abs = B.e_abs;
  c.floor2 = B.floor2;
  BucketQuery bq;
  bq.set(q.x, q.y, q.z, 0.f);
  const uint32_t buckets = (S.n + kBucketPoints - 1) / kBucketPoints;
  const uint32_t at = curve_position(P.scodes, S.n, P.qcodes[tq]) / kBucketPoints;
  uint32_t b0 = at > 2u ? at - 2u : 0u;
  if (b0 + 4u > buckets) b0 = buckets > 4u ? buckets - 4u : 0u;
  float best = INFINITY;
  for (uint32_t w = b0; w < b0 + 4u && w < buckets; ++w) {
    float d2[8];
    bucket_d2<DIM>(S.bucket_pts, w, bq, d2);
#pragma unroll
    for (int j = 0; j < 8; ++j) best = fminf(best, d2[j]);
  }
  uint32_t besti = kNone;
  float bound = best + key_tol(c, best);  // what may still order first lies below it
  bq.nd = pack2(-bound);
  WalkStack& stack = warps[threadIdx.x >> 5].stack;
  cut_packet(
      S, S.trees, q, __fmul_ru(bound, 1.000001f), true, valid, stack, lane,
      [&](bool mine, const PacketBox& box, const PacketBox* limit, float reach2) {
        bq.nd = pack2(mine ? -bound : INFINITY);  // no candidates for the other lanes
        walk_fours(S, S.trees, box, limit, reach2, stack, warps[threadIdx.x >> 5].list, lane, 4u,
                   [&](const uint4& four) {
                     uint32_t hits = buckets_mask<DIM, false>(S.bucket_pts, four, bq, nullptr);
                     for (; hits; hits &= hits - 1u) {
                       const int j = __ffs((int)hits) - 1;
                       const uint32_t b = j < 8 ? four.x : j < 16 ? four.y : j < 24 ? four.z : four.w;
                       const uint32_t i = b * kBucketPoints + (j & 7);
                       const float4 p = __ldg(&S.pts[i]);
                       const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
                       const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                       if (nearer(P, c, qin, d2, i, best, besti)) {
                         best = d2;
                         besti = i;
                         bound = fminf(bound, best + key_tol(c, best));
                         bq.nd = pack2(-bound);
                       }
                     }
                     reach2 = __uint_as_float(__reduce_max_sync(
                         0xffffffffu, __float_as_uint(mine ? __fmul_ru(bound, 1.000001f) : 0.f)));
                     return false;
                   });
      },
      [&](uint32_t run) {
        for (; run; run &= run - 1u) {
          const int from = __ffs((int)run) - 1;
          const uint32_t i = nearest_alone(P, c, __shfl_sync(0xffffffffu, qin, from),
                                           __shfl_sync(0xffffffffu, bound, from), stack);
          if (lane == from) besti = i;
        }
      });
  if (valid) P.nearest[qin] = besti == kNone ? 0u : besti;
}

// ---- nearest in-radius witness (k_max 1, one row per query) -------------------
// offsets[o] = input index of output rank o, offsets[nq] = nq: the emit then
// writes a query's first row at its input position.
__global__ void k_witness_offsets(const uint32_t* oorder, const unsigned int* identity, uint32_t nq,
                                  unsigned long long* offsets) {
  const bool ident = *identity != 0;
  for (uint64_t o = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; o <= nq; o += (uint64_t)gridDim.x * blockDim.x)
    offsets[o] = o == nq ? nq : (ident ? o : oorder[o]);
}

// The row of a query without a neighbour in radius (rtdl_optix_core.cpp:6043-6090:
// neighbor id 0xFFFFFFFF, distance FLT_MAX).
__global__ void k_witness_fill(const float4* qpts, uint32_t nq, RtdlFixedRadiusNeighborRow* rows,
                               unsigned long long capacity) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nq && i < capacity;
       i += (uint64_t)gridDim.x * blockDim.x)
    rows[i] = RtdlFixedRadiusNeighborRow{__float_as_uint(qpts[i].w), 0xFFFFFFFFu, 3.4028234663852886e38};
}

// ---- fixed-radius count with a threshold --------------------------------------
// The reference's generic count (generic_primitives.py:198-227): a query's
// in-radius points are counted (radius inclusive, FP64 distances) until the
// threshold is reached; threshold 0 counts them all.  Here the count uses the
// collect's accept rule (FP32 outside the band, FP64 inside) on a packet walk,
// and a lane stops testing once its query reaches the threshold; the walk ends
// when every lane of the warp has.
struct CountParams {
  SceneView S;
  const float4* qpts;
  const double* qraw;
  int qstride;
  const uint32_t* qorder;       // processing rank -> input index
  uint32_t nq;
  const DevBands* bands;
  uint32_t threshold;
  uint32_t* ids_out;            // per query, input order (each optional)
  uint32_t* counts_out;
  uint32_t* flags_out;
  RtdlFixedRadiusCountRow* rows_out;
  unsigned long long* reached;  // optional: queries that reached the threshold
  // point groups (optional): a candidate also needs its group's box within radius
  const uint32_t* group_of;     // group of each scene point (scene input order)
  const double* group_boxes;    // min_x, min_y, max_x, max_y per group
};

// The reference's group test (rtdl_optix_core.cpp:6143-6147) in FP64: the
// squared distance from the query to the group's box, within radius.
__device__ __forceinline__ bool group_box_ok(const CountParams& P, const SceneView& S, uint32_t qin, uint32_t i,
                                             double r2) {
  const double* rq = P.qraw + (size_t)qin * P.qstride;
  const double qx = rq[1], qy = rq[2];
  const double* g = P.group_boxes + 4ull * P.group_of[S.perm[i]];
  const double dx = qx < g[0] ? __dsub_rn(g[0], qx) : (qx > g[2] ? __dsub_rn(qx, g[2]) : 0.0);
  const double dy = qy < g[1] ? __dsub_rn(g[1], qy) : (qy > g[3] ? __dsub_rn(qy, g[3]) : 0.0);
  return __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)) <= r2;
}

// The count of one query by the whole warp (packets whose queries lie far apart).
__device__ __noinline__ uint32_t count_alone(const CountParams& P, const DevBands& B, int scene_inexact, uint32_t qin,
                                             WalkStack& stack) {
  const SceneView& S = P.S;
  const float4 q = P.qpts[qin];
  const double* rq = P.qraw + (size_t)qin * P.qstride;
  uint32_t count = 0;
  walk_single(S, S.trees, q, B.box_hi2, stack, (int)(threadIdx.x & 31), [&](uint32_t i, const float4& p, bool has) {
    const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
    const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    bool hit = has && d2 <= B.hi2;
    if (hit && d2 >= B.lo2)
      hit = exact_d2_at(rq[1], rq[2], P.qstride == 4 ? rq[3] : 0.0, S.pts, S.pts64, scene_inexact, i) <= B.r2;
    if (hit && P.group_of) hit = group_box_ok(P, S, qin, i, B.r2);
    count += __popc(__ballot_sync(0xffffffffu, hit));
    return P.threshold != 0u && count >= P.threshold;
  });
  return P.threshold != 0u && count > P.threshold ? P.threshold : count;
}

template <int DIM>
__global__ void __launch_bounds__(128) k_count_packet(const __grid_constant__ CountParams P) {
  __shared__ PacketWarp warps[128 / 32];
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (!__any_sync(0xffffffffu, t < P.nq)) return;  // whole warp past the end
  const bool valid = t < P.nq;
  const DevBands B = *P.bands;
  const SceneView& S = P.S;
  const int scene_inexact = *S.inexact;
  uint32_t qin = 0;
  float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
  if (valid) {
    qin = P.qorder[t];
    q = P.qpts[qin];
  }
  const uint32_t thr = P.threshold;
  uint32_t count = 0;
  bool active = valid;
  const int lane = threadIdx.x & 31;
  const TreeShape* T = S.trees;
  BucketQuery bq;
  bq.set(q.x, q.y, q.z, B.top);
  const int band = valid ? (int)(0x80000001u + __float_as_uint(B.width)) : (int)0x80000000;
  const float reach2 = B.box_hi2;
  WalkStack& stack = warps[threadIdx.x >> 5].stack;
  cut_packet(
      S, T, q, reach2, false, valid, stack, lane,
      [&](bool mine, const PacketBox& box, const PacketBox*, float reach) {
        walk_fours(S, T, box, nullptr, reach, stack, warps[threadIdx.x >> 5].list, lane, 32u, [&](const uint4& four) {
          int near;
          uint32_t hits = buckets_mask<DIM, true>(S.bucket_pts, four, bq, &near);
          if (near < band)
            hits = exact_buckets_mask<DIM>(S, scene_inexact, P.qraw + (size_t)qin * P.qstride, q,
                                           __fsub_rd(B.top, B.width), B.r2, four, hits);
          if (!mine || !active) hits = 0;
          if (P.group_of) {
            for (uint32_t h = hits; h; h &= h - 1u) {
              const int i = __ffs((int)h) - 1;
              const uint32_t b = i < 8 ? four.x : i < 16 ? four.y : i < 24 ? four.z : four.w;
              if (!group_box_ok(P, S, qin, b * kBucketPoints + (i & 7), B.r2)) hits &= ~(1u << i);
            }
          }
          count += __popc(hits);
          if (thr == 0u) return false;
          if (count >= thr) {  // the count stops at the threshold
            count = thr;
            active = false;
          }
          return !__any_sync(0xffffffffu, mine && active);  // every query of the run reached its threshold
        });
      },
      [&](uint32_t run) {
        for (; run; run &= run - 1u) {
          const int from = __ffs((int)run) - 1;
          const uint32_t c = count_alone(P, B, scene_inexact, __shfl_sync(0xffffffffu, qin, from), stack);
          if (lane == from) count = c;
        }
      });
  const bool reached = valid && thr != 0u && count >= thr;
  if (valid) {
    const uint32_t id = __float_as_uint(q.w);
    if (P.ids_out) P.ids_out[qin] = id;
    if (P.counts_out) P.counts_out[qin] = count;
    if (P.flags_out) P.flags_out[qin] = reached ? 1u : 0u;
    if (P.rows_out) P.rows_out[qin] = RtdlFixedRadiusCountRow{id, count, reached ? 1u : 0u};
  }
  if (P.reached) {
    const unsigned int m = __ballot_sync(0xffffffffu, reached);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(P.reached, (unsigned long long)__popc(m));
  }
}

// Point groups: the nearest point within radius whose group box is also within
// radius, by exact FP64 distance then smaller id (rtdl_optix_core.cpp:6215-6306);
// one row per query at its input index, 0xFFFFFFFF / FLT_MAX when none.
__global__ void __launch_bounds__(128) k_group_nearest_packet(const __grid_constant__ CountParams P, RtdlFixedRadiusNeighborRow* rows) {
  __shared__ PacketWarp warps[128 / 32];
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (!__any_sync(0xffffffffu, t < P.nq)) return;  // whole warp past the end
  const bool valid = t < P.nq;
  const DevBands B = *P.bands;
  const SceneView& S = P.S;
  const int scene_inexact = *S.inexact;
  uint32_t qin = 0;
  float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
  if (valid) {
    qin = P.qorder[t];
    q = P.qpts[qin];
  }
  double best = 0.0;
  uint32_t best_id = 0xFFFFFFFFu;
  bool found = false;
  const int lane = threadIdx.x & 31;
  const TreeShape* T = S.trees;
  BucketQuery bq;
  bq.set(q.x, q.y, q.z, B.top);  // every point that may be within radius, decided below
  const float reach2 = B.box_hi2;
  WalkStack& stack = warps[threadIdx.x >> 5].stack;
  cut_packet(
      S, T, q, reach2, false, valid, stack, lane,
      [&](bool mine, const PacketBox& box, const PacketBox*, float reach) {
        walk_fours(S, T, box, nullptr, reach, stack, warps[threadIdx.x >> 5].list, lane, 32u, [&](const uint4& four) {
          uint32_t hits = buckets_mask<2, false>(S.bucket_pts, four, bq, nullptr);
          if (!mine) hits = 0;
          for (; hits; hits &= hits - 1u) {
            const int j = __ffs((int)hits) - 1;
            const uint32_t b = j < 8 ? four.x : j < 16 ? four.y : j < 24 ? four.z : four.w;
            const uint32_t i = b * kBucketPoints + (j & 7);
            const double* rq = P.qraw + (size_t)qin * P.qstride;
            const double e2 = exact_d2_at(rq[1], rq[2], 0.0, S.pts, S.pts64, scene_inexact, i);
            if (e2 > B.r2) continue;
            if (P.group_of && !group_box_ok(P, S, qin, i, B.r2)) continue;
            const uint32_t id = __float_as_uint(__ldg(&S.pts[i].w));
            if (!found || e2 < best || (e2 == best && id < best_id)) {
              best = e2;
              best_id = id;
              found = true;
            }
          }
          return false;
        });
      },
      [&](uint32_t run) {  // one query at a time, the lanes over its points
        for (; run; run &= run - 1u) {
          const int from = __ffs((int)run) - 1;
          const uint32_t one = __shfl_sync(0xffffffffu, qin, from);
          const float4 q1 = P.qpts[one];
          const double* rq = P.qraw + (size_t)one * P.qstride;
          double d = INFINITY;
          uint32_t id = 0xFFFFFFFFu;
          walk_single(S, T, q1, reach2, stack, lane, [&](uint32_t i, const float4& p, bool has) {
            const float dx = p.x - q1.x, dy = p.y - q1.y;
            if (has && fmaf(dy, dy, dx * dx) <= B.hi2) {
              const double e2 = exact_d2_at(rq[1], rq[2], 0.0, S.pts, S.pts64, scene_inexact, i);
              const uint32_t pid = __float_as_uint(p.w);
              if (e2 <= B.r2 && (!P.group_of || group_box_ok(P, S, one, i, B.r2)) &&
                  (e2 < d || (e2 == d && pid < id))) {
                d = e2;
                id = pid;
              }
            }
            return false;
          });
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const double od = __shfl_xor_sync(0xffffffffu, d, o);
            const uint32_t oid = __shfl_xor_sync(0xffffffffu, id, o);
            if (od < d || (od == d && oid < id)) {
              d = od;
              id = oid;
            }
          }
          if (lane == from && d < INFINITY) {
            best = d;
            best_id = id;
            found = true;
          }
        }
      });
  if (valid)
    rows[qin] = RtdlFixedRadiusNeighborRow{__float_as_uint(q.w), found ? best_id : 0xFFFFFFFFu,
                                           found ? __dsqrt_rn(best) : 3.4028234663852886e38};
}

// The witness row of largest distance, ties to the smaller query id then
// neighbour id; a query without a witness counts as infinitely far
// (rtdl_optix_core.cpp:6310-6358).  One block.
__device__ __forceinline__ bool witness_after(const RtdlFixedRadiusNeighborRow& c, const RtdlFixedRadiusNeighborRow& b) {
  if (c.distance != b.distance) return c.distance > b.distance;
  if (c.query_id != b.query_id) return c.query_id < b.query_id;
  return c.neighbor_id < b.neighbor_id;
}

__global__ void __launch_bounds__(1024) k_witness_max(const RtdlFixedRadiusNeighborRow* rows, uint32_t n,
                                                      RtdlFixedRadiusNeighborRow* out) {
  __shared__ RtdlFixedRadiusNeighborRow sb[1024];
  RtdlFixedRadiusNeighborRow best{0xFFFFFFFFu, 0xFFFFFFFFu, -1.0};
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
    RtdlFixedRadiusNeighborRow r = rows[i];
    if (r.neighbor_id == 0xFFFFFFFFu || !isfinite(r.distance)) r.distance = INFINITY;
    if (witness_after(r, best)) best = r;
  }
  sb[threadIdx.x] = best;
  __syncthreads();
  for (unsigned int stride = blockDim.x >> 1; stride > 0; stride >>= 1) {
    if (threadIdx.x < stride && witness_after(sb[threadIdx.x + stride], sb[threadIdx.x]))
      sb[threadIdx.x] = sb[threadIdx.x + stride];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = sb[0];
}

// The 3-D device-output contract with threshold 0 (rtdl_optix_core.cpp:4189-4201):
// every query reaches it with a count of 0, and no walk is needed.
__global__ void k_count_trivial(const float4* qpts, uint32_t nq, uint32_t* ids_out, uint32_t* counts_out,
                                uint32_t* flags_out) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nq; i += (uint64_t)gridDim.x * blockDim.x) {
    ids_out[i] = __float_as_uint(qpts[i].w);
    counts_out[i] = 0u;
    flags_out[i] = 1u;
  }
}

// ---- ranked summaries ----------------------------------------------------------
// A query's rows (contiguous, in output order) are reduced to the reference's
// ranked summary: count, first and last row, and the distances added one by one
// in row order (so the sum is the one a sequential loop over the rows gives).
// Every eight consecutive queries also give a partial aggregate, added in query
// order, which k_summary_final reduces in a fixed order: the aggregate is the
// same on every run.
struct SummaryPartial {
  unsigned long long count, nearest, kth;
  double sum;
};

struct SummarySpec {
  RtdlFixedRadiusRankedNeighborSummary* summaries_dev;  // per query, input order (optional)
  RtdlFixedRadiusRankedNeighborAggregate* aggregate_host;
};

constexpr int kSummaryThreads = 128;
constexpr int kSummaryGroup = 8;  // queries per partial aggregate

// A thread per query.  The sum of a query's distances is a chain of FP64 adds;
// with a warp per query every add cost the warp two shuffles for one query, here
// 32 chains share a warp, and a thread keeps eight distance loads in flight.  262k
// queries with 50 rows each: 58 us, a warp per query 190.
__global__ void __launch_bounds__(kSummaryThreads)
    k_summarize(const RtdlFixedRadiusNeighborRow* __restrict__ rows, const unsigned long long* __restrict__ offsets,
                const uint32_t* __restrict__ oorder, const unsigned int* __restrict__ identity,
                const float4* __restrict__ qpts, uint32_t nq, RtdlFixedRadiusRankedNeighborSummary* summaries,
                SummaryPartial* partial) {
  __shared__ SummaryPartial per_query[kSummaryThreads];
  const uint64_t j = (uint64_t)blockIdx.x * kSummaryThreads + threadIdx.x;
  SummaryPartial mine{0ull, 0ull, 0ull, 0.0};
  if (j < nq) {
    const uint32_t qin = *identity ? (uint32_t)j : oorder[j];
    const unsigned long long a = offsets[j], b = offsets[j + 1];
    const uint32_t cnt = (uint32_t)(b - a);
    double sum = 0.0;
    for (uint32_t i = 0; i < cnt; i += 8) {
      double d[8];
#pragma unroll
      for (uint32_t u = 0; u < 8; ++u) d[u] = i + u < cnt ? rows[a + i + u].distance : 0.0;
#pragma unroll
      for (uint32_t u = 0; u < 8; ++u)
        if (i + u < cnt) sum += d[u];
    }
    RtdlFixedRadiusRankedNeighborSummary sm;
    sm.query_id = __float_as_uint(qpts[qin].w);
    sm.neighbor_count = cnt;
    sm.nearest_neighbor_id = cnt ? rows[a].neighbor_id : 0xFFFFFFFFu;
    sm.kth_neighbor_id = cnt ? rows[b - 1].neighbor_id : 0xFFFFFFFFu;
    sm.nearest_distance = cnt ? rows[a].distance : 0.0;
    sm.kth_distance = cnt ? rows[b - 1].distance : 0.0;
    sm.sum_distance = sum;
    if (summaries) summaries[qin] = sm;
    mine = SummaryPartial{(unsigned long long)cnt, sm.nearest_neighbor_id, sm.kth_neighbor_id, sum};
  }
  per_query[threadIdx.x] = mine;
  __syncthreads();
  const uint32_t g = threadIdx.x;
  const uint64_t out = (uint64_t)blockIdx.x * (kSummaryThreads / kSummaryGroup) + g;
  if (g < kSummaryThreads / kSummaryGroup && out * kSummaryGroup < nq) {
    SummaryPartial acc{0ull, 0ull, 0ull, 0.0};
    for (int w = 0; w < kSummaryGroup; ++w) {
      const SummaryPartial& q = per_query[g * kSummaryGroup + w];
      acc.count += q.count;
      acc.nearest += q.nearest;
      acc.kth += q.kth;
      acc.sum += q.sum;
    }
    partial[out] = acc;
  }
}

// One block: thread t adds partials t, t + blockDim, ... in order, then a
// fixed tree over the threads.
__global__ void __launch_bounds__(1024) k_summary_final(const SummaryPartial* partial, uint32_t m, uint32_t nq,
                                                        RtdlFixedRadiusRankedNeighborAggregate* out) {
  __shared__ SummaryPartial sp[1024];
  SummaryPartial acc{0ull, 0ull, 0ull, 0.0};
  for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
    acc.count += partial[i].count;
    acc.nearest += partial[i].nearest;
    acc.kth += partial[i].kth;
    acc.sum += partial[i].sum;
  }
  sp[threadIdx.x] = acc;
  __syncthreads();
  for (unsigned int stride = blockDim.x >> 1; stride > 0; stride >>= 1) {
    if (threadIdx.x < stride) {
      sp[threadIdx.x].count += sp[threadIdx.x + stride].count;
      sp[threadIdx.x].nearest += sp[threadIdx.x + stride].nearest;
      sp[threadIdx.x].kth += sp[threadIdx.x + stride].kth;
      sp[threadIdx.x].sum += sp[threadIdx.x + stride].sum;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out->query_count = nq;
    out->bounded_neighbor_count = sp[0].count;
    out->nearest_id_checksum = sp[0].nearest;
    out->kth_id_checksum = sp[0].kth;
    out->sum_distance = sp[0].sum;
  }
}

// Row offsets in processing order: poff[t] = offsets[qrank[qorder[t]]].
__global__ void k_proc_offsets(const uint32_t* qorder, const uint32_t* qrank, const unsigned long long* offsets,
                               uint32_t nq, unsigned long long* poff) {
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nq; t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t qin = qorder[t];
    poff[t] = qin == kNone ? 0ull : offsets[qrank[qin]];
  }
}

constexpr int kEmitListThreads = 128;

// The part of a work list (processing ranks) a list kernel takes: the list's
// length is read on the device, or one range of output ranks.
__device__ __forceinline__ void list_part(const EmitParams& P, const unsigned int* nwork_dev, uint32_t& begin,
                                          uint32_t& end) {
  begin = 0;
  if (nwork_dev) end = *nwork_dev;
  if (P.list_start) {
    begin = P.list_start[P.range];
    end = P.list_start[P.range + 1];
  }
}

// 65..128 candidates: 16 lanes per query (exact fixups deferred to k_emit_fixup);
// 99 us for the 13% of 1M clustered queries, 141 with a warp per query.
__global__ void __launch_bounds__(kEmitListThreads)
    k_emit_mid(const __grid_constant__ EmitParams P, const uint32_t* work, uint32_t nwork, const unsigned int* nwork_dev) {
  __shared__ EmitGroups<16> shared[kEmitListThreads / 32];
  const int lane = threadIdx.x & 31;
  uint32_t begin, end = nwork;
  list_part(P, nwork_dev, begin, end);
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t w = begin + 2 * ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); w < end; w += 2 * warps) {
    const uint32_t j = w + lane / 16;
    emit_groups<16>(P, work[j < end ? j : w], j < end, 0u, lane, shared[threadIdx.x >> 5]);
  }
}

// 129..kSlab candidates: a warp per query, fixups in place through shared memory.
__global__ void __launch_bounds__(kEmitListThreads)
    k_emit_big(const __grid_constant__ EmitParams P, const uint32_t* work, uint32_t nwork, const unsigned int* nwork_dev) {
  __shared__ EmitWarp<8> shared[kEmitListThreads / 32];
  __shared__ uint32_t cands[kEmitListThreads / 32][256], wbuf[kEmitListThreads / 32][256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t begin, end = nwork;
  list_part(P, nwork_dev, begin, end);
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t j = begin + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); j < end; j += warps) {  // whole warps
    const uint32_t t = work[j];
    EmitQuery q;
    emit_load(P, t, lane, q);
    emit_query<8>(P, t, q, (int)(q.qi.meta & kQueryCountMask), lane, shared[warp], cands[warp], wbuf[warp]);
  }
}

// Output rank -> processing rank map for emission range by range (padding
// ranks hold no query).
__global__ void k_emit_order(const uint32_t* qorder, const uint32_t* qrank, uint32_t np, uint32_t* order) {
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < np; t += gridDim.x * blockDim.x) {
    const uint32_t qin = qorder[t];
    if (qin != kNone) order[qrank[qin]] = t;
  }
}

// The download range of output rank r: the c with nq*c/C <= r < nq*(c+1)/C
// (integer division, as the range bounds are cut).
__device__ __forceinline__ uint32_t download_range(uint32_t r, uint32_t nq, uint32_t chunks) {
  return (uint32_t)((((uint64_t)r + 1) * chunks - 1) / nq);
}

// A work list of processing ranks partitioned by download range (a counting
// sort; the order inside a range is arbitrary, which the per-query emit does
// not see).  part[0..C) counts, part[C..2C] the range starts, part[2C+1..3C]
// the scatter cursors.
__global__ void k_range_count(const uint32_t* list, const unsigned int* n_dev, const uint32_t* qorder,
                              const uint32_t* qrank, uint32_t nq, uint32_t chunks, unsigned int* part) {
  const unsigned int n = *n_dev;
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
    atomicAdd(&part[download_range(qrank[qorder[list[j]]], nq, chunks)], 1u);
}

__global__ void k_range_starts(uint32_t chunks, unsigned int* part) {
  unsigned int sum = 0;
  for (uint32_t c = 0; c < chunks; ++c) {
    part[chunks + c] = sum;
    part[2 * chunks + 1 + c] = sum;
    sum += part[c];
  }
  part[2 * chunks] = sum;
}

__global__ void k_range_scatter(const uint32_t* list, const unsigned int* n_dev, const uint32_t* qorder,
                                const uint32_t* qrank, uint32_t nq, uint32_t chunks, unsigned int* part,
                                uint32_t* out) {
  const unsigned int n = *n_dev;
  for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const uint32_t t = list[j];
    const uint32_t c = download_range(qrank[qorder[t]], nq, chunks);
    out[atomicAdd(&part[2 * chunks + 1 + c], 1u)] = t;
  }
}

// First row of each range of output ranks [c * nq / chunks, ...), and the total.
__global__ void k_chunk_rows(const unsigned long long* offsets, uint32_t nq, int chunks, unsigned long long* out) {
  const int c = threadIdx.x;
  if (c <= chunks) out[c] = offsets[(uint64_t)nq * (uint32_t)c / (uint32_t)chunks];
}

// The next range's fix-ups start after this range's.
__global__ void k_fix_advance(unsigned int* fix_begin, const unsigned int* fix_count) { *fix_begin = *fix_count; }

// Problem batch: *flag stays nonzero while every problem's query ids ascend.
__global__ void k_batch_ids_sorted(const float4* qpts, const uint32_t* qprob, uint32_t n, unsigned int* flag) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x + 1; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    if (qprob[i] == qprob[i - 1] && __float_as_uint(qpts[i].w) < __float_as_uint(qpts[i - 1].w)) *flag = 0u;
}

// Problem batch: the sorted queries into the padded processing order (kNone
// fills a problem's last warp) and each warp's problem.  A thread per rank
// finds its problem by bisection (the same one for a whole warp); a block per
// problem left one block copying the largest problem alone (0.51 ms for the 128
// problems of 6M queries).
__global__ void k_batch_pad(const unsigned long long* qoff, const unsigned long long* pstart, uint32_t problems,
                            uint32_t np, const uint32_t* sorted, uint32_t* qorder, uint32_t* warp_prob) {
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < np; t += gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = problems;  // first problem that starts after t
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (__ldg(&pstart[mid]) <= t) lo = mid + 1;
      else hi = mid;
    }
    const uint32_t p = lo - 1;
    const unsigned long long j = qoff[p] + (t - pstart[p]);
    qorder[t] = j < qoff[p + 1] ? sorted[j] : kNone;
    if ((t & 31u) == 0) warp_prob[t >> 5] = p;
  }
}

// keys[j] = src[order[j]] (skipped when *skip is nonzero).
__global__ void k_gather_u32(const uint32_t* src, const uint32_t* order, uint32_t n, const unsigned int* skip,
                             uint32_t* keys) {
  if (*skip) return;
  for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x)
    keys[j] = src[order[j]];
}

// out[p] = offsets[qoff[p]]: the first row of each problem (and the total).
__global__ void k_problem_rows(const unsigned long long* offsets, const unsigned long long* qoff, uint32_t m,
                               unsigned long long* out) {
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p <= m; p += gridDim.x * blockDim.x) out[p] = offsets[qoff[p]];
}

__global__ void k_invert(const uint32_t* order, uint32_t n, const unsigned int* identity_flag, uint32_t* inv) {
  const bool ident = *identity_flag != 0;
  for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (uint64_t)gridDim.x * blockDim.x)
    inv[ident ? j : order[j]] = (uint32_t)j;
}

// k > 64 KNN: every query takes the generic path.
__global__ void k_mark_all_heavy(const uint32_t* qorder, uint32_t nq, uint32_t n, uint32_t k, uint32_t* counts,
                                 uint8_t* flags, uint32_t* temp, uint32_t* heavy_list, uint32_t* heavy_m) {
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nq; t += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t qin = qorder[t];
    heavy_list[t] = qin;
    heavy_m[t] = n;
    counts[qin] = k < n ? k : n;
    flags[qin] = 2;
    temp[qin] = (uint32_t)t;
  }
}

__global__ void k_extract_ids(const float4* qpts, uint32_t n, const unsigned int* skip, uint32_t* ids) {
  if (*skip) return;  // the ids ascend: nothing is sorted
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    ids[i] = __float_as_uint(qpts[i].w);
}

struct HeavyEntry {
  unsigned long long key;  // bits of the FP64 distance (non-negative: bit order == value order)
  uint32_t nid;
  uint32_t sidx;
};

__device__ __forceinline__ Ctx make_ctx(const SceneView& S, const float4* qpts, const double* qraw, int qstride,
                                        uint32_t qin, const DevBands& B) {
  Ctx c;
  const float4 q = qpts[qin];
  c.qx = q.x;
  c.qy = q.y;
  c.qz = q.z;
  const double* r = qraw + (size_t)qin * qstride;
  c.ex = r[1];
  c.ey = r[2];
  c.ez = qstride == 4 ? r[3] : 0.0;
  c.pts = S.pts;
  c.pts64 = S.pts64;
  c.perm = S.perm;
  c.scene_inexact = *S.inexact;
  c.rho = B.rho;
  c.e_abs = B.e_abs;
  c.floor2 = B.floor2;
  return c;
}

__global__ void __launch_bounds__(kHeavyThreads)
    k_heavy_gather(SceneView S, const float4* qpts, const double* qraw, int qstride, const uint32_t* heavy_list,
                   const unsigned long long* seg_off, const uint32_t* seg_size, const DevBands* bands,
                   HeavyEntry* scratch, unsigned int* error) {
  __shared__ unsigned int cnt;
  if (threadIdx.x == 0) cnt = 0;
  __syncthreads();
  const uint32_t h = blockIdx.x;
  const uint32_t qin = heavy_list[h];
  const DevBands B = *bands;
  const Ctx c = make_ctx(S, qpts, qraw, qstride, qin, B);
  HeavyEntry* seg = scratch + seg_off[h];
  const uint32_t P2 = seg_size[h];
  for (uint32_t i = threadIdx.x; i < S.n; i += blockDim.x) {
    const double dist = __dsqrt_rn(exact_d2(c, i));
    const unsigned int pos = atomicAdd(&cnt, 1u);
    if (pos < P2) {
      HeavyEntry e;
      e.key = (unsigned long long)__double_as_longlong(dist);
      e.nid = __float_as_uint(__ldg(&S.pts[i].w));
      e.sidx = i;
      seg[pos] = e;
    } else {
      atomicOr(error, 2u);
    }
  }
  __syncthreads();
  for (uint32_t i = cnt + threadIdx.x; i < P2; i += blockDim.x) {
    HeavyEntry e;
    e.key = ~0ull;
    e.nid = kNone;
    e.sidx = kNone;
    seg[i] = e;
  }
}

// Generic-path gather for a radius query with more than kSlab candidates: one
// warp per query walks the tree; the lanes test the reached
// bucket's points together and append in-radius candidates with a ballot
// prefix (no atomics).
__global__ void __launch_bounds__(32)
    k_heavy_gather_bvh(SceneView S, const float4* qpts, const double* qraw, int qstride, const uint32_t* heavy_list,
                       const unsigned long long* seg_off, const uint32_t* seg_size, const DevBands* bands,
                       const uint32_t* qprob, const double* item_rad, HeavyEntry* scratch, unsigned int* error) {
  __shared__ WalkStack stack;
  const int lane = threadIdx.x;
  const uint32_t h = blockIdx.x;
  const uint32_t qin = heavy_list[h];
  const uint32_t prob = qprob ? qprob[qin] : 0u;
  // item_rad: the radius this query gathers within (a tested radius that holds its rows)
  const DevBands B = item_rad ? bands_at_radius(bands[prob], item_rad[h]) : bands[prob];
  const Ctx c = make_ctx(S, qpts, qraw, qstride, qin, B);
  HeavyEntry* seg = scratch + seg_off[h];
  const uint32_t P2 = seg_size[h];
  const unsigned int lt_mask = (1u << lane) - 1u;
  uint32_t cnt = 0;
  const float4 q = make_float4(c.qx, c.qy, c.qz, 0.f);
  walk_single(S, S.trees + prob * S.tree_stride, q, B.box_hi2, stack, lane,
              [&](uint32_t i, const float4& p, bool has) {
                const float dx = p.x - c.qx, dy = p.y - c.qy, dz = p.z - c.qz;
                const float d2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
                const bool acc = has && d2 <= B.hi2 && (d2 < B.lo2 || exact_d2(c, i) <= B.r2);
                const unsigned int m = __ballot_sync(0xffffffffu, acc);
                if (acc) {
                  const uint32_t pos = cnt + __popc(m & lt_mask);
                  if (pos < P2) {
                    HeavyEntry en;
                    en.key = (unsigned long long)__double_as_longlong(__dsqrt_rn(exact_d2(c, i)));
                    en.nid = __float_as_uint(p.w);
                    en.sidx = i;
                    seg[pos] = en;
                  } else {
                    atomicOr(error, 2u);
                  }
                }
                cnt += __popc(m);
                return false;
              });
  for (uint32_t i = cnt + lane; i < P2; i += 32) {
    HeavyEntry en;
    en.key = ~0ull;
    en.nid = kNone;
    en.sidx = kNone;
    seg[i] = en;
  }
}

__device__ __forceinline__ bool heavy_greater(const HeavyEntry& a, const HeavyEntry& b, const uint32_t* perm) {
  if (a.key != b.key) return a.key > b.key;
  if (a.nid != b.nid) return a.nid > b.nid;
  if (a.sidx == kNone || b.sidx == kNone) return a.sidx == kNone && b.sidx != kNone;
  return perm[a.sidx] > perm[b.sidx];
}

constexpr uint32_t kHeavySmemEntries = 2048;  // 32 KiB of 16-B entries per block

template <typename Ptr>
__device__ __forceinline__ void bitonic_block(Ptr e, uint32_t P2, const uint32_t* perm) {
  for (uint32_t k = 2; k <= P2; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      for (uint32_t i = threadIdx.x; i < P2; i += blockDim.x) {
        const uint32_t ixj = i ^ j;
        if (ixj > i) {
          const HeavyEntry a = e[i], b = e[ixj];
          const bool up = (i & k) == 0;
          if (heavy_greater(a, b, perm) == up) {
            e[i] = b;
            e[ixj] = a;
          }
        }
      }
      __syncthreads();
    }
  }
}

// Block-per-query bitonic sort of a segment by (distance, neighbor id, search
// input index); in shared memory up to 2,048 entries, in global memory above.
__global__ void __launch_bounds__(kHeavyThreads)
    k_heavy_sort(const unsigned long long* seg_off, const uint32_t* seg_size, HeavyEntry* scratch,
                 const uint32_t* perm) {
  extern __shared__ HeavyEntry heavy_smem[];
  HeavyEntry* e = scratch + seg_off[blockIdx.x];
  const uint32_t P2 = seg_size[blockIdx.x];
  if (P2 <= kHeavySmemEntries) {
    for (uint32_t i = threadIdx.x; i < P2; i += blockDim.x) heavy_smem[i] = e[i];
    __syncthreads();
    bitonic_block(heavy_smem, P2, perm);
    for (uint32_t i = threadIdx.x; i < P2; i += blockDim.x) e[i] = heavy_smem[i];
  } else {
    bitonic_block(e, P2, perm);
  }
}

__global__ void k_heavy_emit(const unsigned long long* seg_off, const unsigned long long* out_off,
                             const uint32_t* out_count, const HeavyEntry* scratch, uint32_t* heavy_out) {
  const HeavyEntry* e = scratch + seg_off[blockIdx.x];
  uint32_t* dst = heavy_out + out_off[blockIdx.x];
  const uint32_t k = out_count[blockIdx.x];
  for (uint32_t j = threadIdx.x; j < k; j += blockDim.x) dst[j] = e[j].sidx;
}

struct ExpandParams {
  SceneView S;
  const float4* qpts;
  const double* qraw;
  int qstride;
  const uint32_t* oorder;
  const DevBands* bands;
  uint32_t nq;
  int L;
  const uint32_t* counts;
  const uint8_t* flags;
  const uint32_t* temp;
  const uint32_t* heavy_out;
  const unsigned long long* heavy_out_off;
  const unsigned long long* offsets;
  void* rows;
  unsigned long long capacity;
  int ranked;
  uint8_t* overflow_out;
  unsigned int* error;
  const uint32_t* work_list;  // optional: process only these queries (input indices)
  const uint32_t* qrank;      // with work_list: input index -> output rank
};

// A warp per query writes its rows with the exact FP64 distance: all queries
// in output order, or the queries of `work_list` (generic path).
__global__ void __launch_bounds__(kExpandThreads) k_expand(ExpandParams P) {
  constexpr int G = 32;
  const int lane = threadIdx.x & (G - 1);
  const uint64_t groups = ((uint64_t)gridDim.x * blockDim.x) / G;
  const bool ids_sorted = P.bands->ids_sorted != 0;
  const bool scene_inexact = *P.S.inexact != 0;
  for (uint64_t j = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / G; j < P.nq; j += groups) {
    const uint32_t qin = P.work_list ? P.work_list[j] : (ids_sorted ? (uint32_t)j : P.oorder[j]);
    const uint32_t cnt = P.counts[qin];
    const uint8_t fl = P.flags[qin];
    if (P.overflow_out != nullptr && lane == 0) P.overflow_out[qin] = fl & 1;
    if (cnt == 0 || P.rows == nullptr) continue;
    const unsigned long long base = P.offsets[P.work_list ? P.qrank[qin] : (uint32_t)j];
    const uint32_t qid = __float_as_uint(P.qpts[qin].w);
    const double* r = P.qraw + (size_t)qin * P.qstride;
    const double ex = r[1], ey = r[2], ez = P.qstride == 4 ? r[3] : 0.0;
    const uint32_t* src = P.work_list ? P.heavy_out + P.heavy_out_off[j]
                          : (fl & 2) ? P.heavy_out + P.heavy_out_off[P.temp[(size_t)qin * P.L]]
                                     : P.temp + (size_t)qin * P.L;
    for (uint32_t s = lane; s < cnt; s += G) {
      const uint32_t sidx = src[s];
      if (sidx >= P.S.slots) {  // never expected: a generic-path slot without a candidate
        atomicOr(P.error, 4u);
        continue;
      }
      const float4 p = __ldg(&P.S.pts[sidx]);
      double sx, sy, sz;
      if (scene_inexact) {
        const double* pp = P.S.pts64 + 3ull * sidx;
        sx = pp[0];
        sy = pp[1];
        sz = pp[2];
      } else {
        sx = p.x;
        sy = p.y;
        sz = p.z;
      }
      const double dx = __dsub_rn(sx, ex), dy = __dsub_rn(sy, ey), dz = __dsub_rn(sz, ez);
      const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
      const double dist = __dsqrt_rn(d2);
      const unsigned long long row = base + s;
      if (row >= P.capacity) continue;
      const uint32_t nid = __float_as_uint(p.w);
      const unsigned long long db = (unsigned long long)__double_as_longlong(dist);
      if (!P.ranked) {
        reinterpret_cast<uint4*>(P.rows)[row] = make_uint4(qid, nid, (uint32_t)db, (uint32_t)(db >> 32));
      } else {
        uint2* out = reinterpret_cast<uint2*>(static_cast<char*>(P.rows) + row * 24);
        out[0] = make_uint2(qid, nid);
        out[1] = make_uint2((uint32_t)db, (uint32_t)(db >> 32));
        out[2] = make_uint2(s + 1, 0u);
      }
    }
  }
}

// ---- directed Hausdorff: FP64 max over per-query nearest distances ---------
// Exact distances of the nearest points in input order, and a witness per block.
// A chain of two dependent loads per query, the second scattered: with two
// blocks per SM and one thread over the partial results 172 us for 4M queries,
// with eight and k_witness_best 104.
__global__ void __launch_bounds__(256)
    k_nearest_reduce(SceneView S, const float4* qpts, const double* qraw, int qstride, uint32_t nq,
                     const uint32_t* temp, double* nearest_dist, uint32_t* nearest_id, Witness* partial) {
  __shared__ Witness warp_best[8];
  Witness best{0ull, kNone, kNone};
  bool have = false;
  const bool scene_inexact = *S.inexact != 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nq; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t sidx = temp[i];
    const float4 p = __ldg(&S.pts[sidx]);
    const double* r = qraw + i * qstride;
    double sx, sy, sz;
    if (scene_inexact) {
      const double* pp = S.pts64 + 3ull * sidx;
      sx = pp[0];
      sy = pp[1];
      sz = pp[2];
    } else {
      sx = p.x;
      sy = p.y;
      sz = p.z;
    }
    const double dx = __dsub_rn(sx, r[1]), dy = __dsub_rn(sy, r[2]), dz = __dsub_rn(sz, qstride == 4 ? r[3] : 0.0);
    const double dist = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
    const Witness w{(unsigned long long)__double_as_longlong(dist), __float_as_uint(qpts[i].w), __float_as_uint(p.w)};
    if (nearest_dist) nearest_dist[i] = dist;
    if (nearest_id) nearest_id[i] = w.nid;
    if (!have || witness_better(w, best)) {
      best = w;
      have = true;
    }
  }
  if (!have) best = Witness{0ull, kNone, kNone};
  best = warp_witness(best);
  if ((threadIdx.x & 31) == 0) warp_best[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    Witness b = warp_best[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
      if (witness_better(warp_best[w], b)) b = warp_best[w];
    partial[blockIdx.x] = b;
  }
}

// The best of n witnesses; one block.
__global__ void __launch_bounds__(256) k_witness_best(const Witness* __restrict__ in, uint32_t n, Witness* out) {
  __shared__ Witness warp_best[8];
  Witness best{0ull, kNone, kNone};
  for (uint32_t i = threadIdx.x; i < n; i += 256) {
    const Witness w = in[i];
    if (witness_better(w, best)) best = w;
  }
  best = warp_witness(best);
  if ((threadIdx.x & 31) == 0) warp_best[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x < 32) {
    best = warp_witness(threadIdx.x < 8 ? warp_best[threadIdx.x] : Witness{0ull, kNone, kNone});
    if (threadIdx.x == 0) *out = best;
  }
}

bool stats_enabled() {
  static const bool on = std::getenv("RTDL_B200_STATS") != nullptr;
  return on;
}



}  // namespace

std::vector<unsigned long long>& last_stats() {
  thread_local std::vector<unsigned long long> v(kStatCount, 0ull);
  return v;
}

namespace {

// Ranges of output ranks whose rows are copied to the host as each completes.
constexpr int kDownloadChunks = 8;

struct Readback {
  unsigned long long rows;
  unsigned int heavy;  // these four are copied together from the `small` device counters
  unsigned int error;
  unsigned int mid;
  unsigned int big;
  unsigned int scene_bad;
  unsigned int query_bad;
  unsigned int fixups;
  unsigned long long chunk_rows[kDownloadChunks + 1];  // first row of each download range
};

// Pinned and mapped into the device address space, so small reads of device
// counters can be written into it by a kernel (SmallReads) instead of being
// copied by the copy engine.
Readback* pinned_readback() {
  thread_local Readback* rb = nullptr;
  if (rb == nullptr)
    RTDL_CUDA_CHECK(cudaHostAlloc(reinterpret_cast<void**>(&rb), sizeof(Readback),
                                  cudaHostAllocMapped | cudaHostAllocPortable));
  return rb;
}

// Small reads of device counters into the thread's Readback, written by one
// kernel of one warp.  Kernel stores do not queue behind copies: a call whose
// rows are being copied to the host (the copy engine busy for milliseconds)
// reads its counts at once instead of after those copies.  Sources and
// fields are 4-byte words; the host reads the fields after the stream has
// been synchronized.
struct SmallRead {
  static constexpr int kMax = 6;
  const uint32_t* src[kMax];
  uint32_t* dst[kMax];
  uint32_t words[kMax];
  int n;
};

__global__ void k_read_small(SmallRead r) {
  for (int k = 0; k < r.n; ++k)
    for (uint32_t i = threadIdx.x; i < r.words[k]; i += blockDim.x) r.dst[k][i] = r.src[k][i];
}

class SmallReads {
 public:
  explicit SmallReads(Readback* rb) : rb_(rb) {
    void* alias = nullptr;
    RTDL_CUDA_CHECK(cudaHostGetDevicePointer(&alias, rb, 0));
    alias_ = static_cast<char*>(alias);
    r_.n = 0;
  }
  // `field` is a member of the Readback given at construction.
  void add(void* field, const void* dev, size_t bytes) {
    if (r_.n == SmallRead::kMax) throw std::runtime_error("too many small reads in one launch");
    r_.src[r_.n] = static_cast<const uint32_t*>(dev);
    r_.dst[r_.n] = reinterpret_cast<uint32_t*>(alias_ + (static_cast<char*>(field) - reinterpret_cast<char*>(rb_)));
    r_.words[r_.n] = (uint32_t)(bytes / 4);
    ++r_.n;
  }
  void launch(cudaStream_t s) {
    k_read_small<<<1, 32, 0, s>>>(r_);
    RTDL_LAUNCHED(1);
    r_.n = 0;
  }

 private:
  Readback* rb_;
  char* alias_;
  SmallRead r_;
};

inline unsigned int grid_for(uint64_t n, int threads) {
  uint64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  const uint64_t cap = (uint64_t)kSmCount * 32;
  return (unsigned int)(b < cap ? b : cap);
}

inline uint32_t next_pow2(uint32_t v) {
  uint32_t p = 1;
  while (p < v) p <<= 1;
  return p;
}

struct QueryPrep {
  PointStats* qst = nullptr;
  float4* qpts = nullptr;
  DevBands* bands = nullptr;   // one, or one per problem of a batch
  uint32_t* qorder = nullptr;  // processing rank -> input index (a batch pads problems to whole warps: kNone)
  uint32_t* qcodes = nullptr;  // curve codes in processing order (qcodes[t] belongs to qorder[t]); single only
  uint32_t* oorder = nullptr;
  uint32_t nproc = 0;          // processing ranks
  const unsigned int* order_identity = nullptr;  // device flag: output order == input order
  // problem batch only
  uint32_t* qprob = nullptr;      // problem of each query (input order)
  uint32_t* warp_prob = nullptr;  // problem of each warp of processing ranks
  uint32_t* prob_kmax = nullptr;
  unsigned int* sorted_flag = nullptr;
  unsigned long long* qoff = nullptr;  // device copy of the query offsets
  double* prob_radius = nullptr;       // radius of each problem
  SceneView view{};                    // the scene as the traversal kernels see it
  const PreparedQueries* borrowed = nullptr;  // set: the query-side buffers belong to a prepared query set
};

// The call-side view of a prepared query set: its buffers are borrowed, only
// the bands (scene and query statistics, this radius) are computed.
QueryPrep borrow_prepared(Scene* sc, const PreparedQueries* pq, double radius, cudaStream_t s) {
  QueryPrep qp;
  qp.borrowed = pq;
  qp.qst = pq->qst;
  qp.qpts = pq->qpts;
  qp.qorder = pq->qorder;
  qp.oorder = pq->oorder;
  qp.nproc = pq->n;
  qp.order_identity = pq->identity;
  qp.view = sc->view();
  qp.bands = static_cast<DevBands*>(dev_alloc(sizeof(DevBands), s));
  k_bands<<<1, 32, 0, s>>>(sc->stats, pq->qst, radius, 1, qp.bands);
  RTDL_LAUNCHED(1);
  return qp;
}



QueryPrep prepare_queries(Scene* sc, const void* queries_dev, uint32_t nq, bool has_radius, double radius,
                          bool want_output_order, cudaStream_t s) {
  QueryPrep qp;
  qp.qst = static_cast<PointStats*>(dev_alloc(sizeof(PointStats), s));
  qp.qpts = static_cast<float4*>(dev_alloc(sizeof(float4) * nq, s));
  qp.bands = static_cast<DevBands*>(dev_alloc(sizeof(DevBands), s));
  qp.qorder = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * nq, s));
  reset_stats(qp.qst, s);
  prep_points(queries_dev, nq, sc->dim, qp.qpts, qp.qst, s);
  k_bands<<<1, 32, 0, s>>>(sc->stats, qp.qst, radius, has_radius ? 1 : 0, qp.bands);
  RTDL_LAUNCHED(1);
  qp.nproc = nq;
  qp.order_identity = &qp.bands->ids_sorted;
  qp.view = sc->view();
  qp.qcodes = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * nq, s));
  SortWork sort;
  uint32_t* digits = radix_sort_counts(nq, 0, curve_bits(sc->dim), sort, s);
  curve_codes(qp.qpts, nq, sc->dim, sc->stats, qp.qcodes, digits, s);
  radix_sort_counted(qp.qcodes, qp.qorder, nq, true, sort, nullptr, &qp.qst->bad, s);
  if (want_output_order) {
    qp.oorder = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * nq, s));
    uint32_t* ids = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * nq, s));
    k_extract_ids<<<grid_for(nq, 256), 256, 0, s>>>(qp.qpts, nq, &qp.bands->ids_sorted, ids);
    RTDL_LAUNCHED(1);
    radix_sort_pairs(ids, qp.oorder, nq, 0, 32, true, &qp.bands->ids_sorted, &qp.qst->bad, s);
    dev_free(ids, s);
  }
  return qp;
}

// A problem batch's query preparation: per-query problem ids, per-problem
// bands and kmax, composite (problem, curve) sort, processing order padded
// so each warp holds queries of one problem, and the output order (problem,
// then query id, stable).
QueryPrep prepare_queries_batch(Scene* sc, const void* queries_dev, uint32_t nq, const BatchSpec& bs,
                                cudaStream_t s) {
  const uint32_t P = bs.problems;
  QueryPrep qp;
  const bool shared = sc->problems == 0;  // several requests against one plain scene
  qp.view = sc->view();
  std::vector<unsigned long long> pstart(P + 1, 0);
  for (uint32_t p = 0; p < P; ++p) pstart[p + 1] = pstart[p] + (bs.qoff[p + 1] - bs.qoff[p] + 31) / 32 * 32;
  if (pstart[P] > 0xFFFFFFFFull - 32) throw std::runtime_error("problem batch has too many queries");
  qp.nproc = (uint32_t)pstart[P];
  qp.qst = static_cast<PointStats*>(dev_alloc(sizeof(PointStats), s));
  qp.qpts = static_cast<float4*>(dev_alloc(sizeof(float4) * (nq ? nq : 1), s));
  qp.bands = static_cast<DevBands*>(dev_alloc(sizeof(DevBands) * P, s));
  qp.qorder = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * (qp.nproc ? qp.nproc : 1), s));
  qp.qprob = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * (nq ? nq : 1), s));
  qp.warp_prob = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * (qp.nproc / 32 + 1), s));
  qp.prob_kmax = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * P, s));
  qp.sorted_flag = static_cast<unsigned int*>(dev_alloc(sizeof(unsigned int), s));
  qp.qoff = static_cast<unsigned long long*>(dev_alloc(sizeof(unsigned long long) * (P + 1), s));
  qp.order_identity = qp.sorted_flag;
  unsigned long long* d_pstart = static_cast<unsigned long long*>(dev_alloc(sizeof(unsigned long long) * (P + 1), s));
  qp.prob_radius = static_cast<double*>(dev_alloc(sizeof(double) * P, s));
  double* d_radius = qp.prob_radius;
  RTDL_CUDA_CHECK(cudaMemcpyAsync(qp.qoff, bs.qoff, sizeof(unsigned long long) * (P + 1), cudaMemcpyHostToDevice, s));
  RTDL_CUDA_CHECK(cudaMemcpyAsync(d_pstart, pstart.data(), sizeof(unsigned long long) * (P + 1),
                                  cudaMemcpyHostToDevice, s));
  RTDL_CUDA_CHECK(cudaMemcpyAsync(d_radius, bs.radius, sizeof(double) * P, cudaMemcpyHostToDevice, s));
  RTDL_CUDA_CHECK(cudaMemcpyAsync(qp.prob_kmax, bs.kmax, sizeof(uint32_t) * P, cudaMemcpyHostToDevice, s));
  RTDL_CUDA_CHECK(cudaMemsetAsync(qp.sorted_flag, 0xFF, sizeof(unsigned int), s));  // nonzero: sorted
  reset_stats(qp.qst, s);
  prep_points(queries_dev, nq, sc->dim, qp.qpts, qp.qst, s);
  batch_problem_ids(qp.qoff, P, nq, qp.qprob, s);
  if (nq > 1) {
    k_batch_ids_sorted<<<grid_for(nq, 256), 256, 0, s>>>(qp.qpts, qp.qprob, nq, qp.sorted_flag);
    RTDL_LAUNCHED(1);
  }
  k_bands_batch<<<div_up(P, 128), 128, 0, s>>>(sc->stats, qp.qst, d_radius, P, qp.sorted_flag, qp.bands);
  RTDL_LAUNCHED(1);
  // processing order: composite (problem, curve in the problem's box) sort, padded per problem
  uint32_t* codes = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * (nq ? nq : 1), s));
  uint32_t* sorted = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * (nq ? nq : 1), s));
  SortWork sort;
  uint32_t* digits = radix_sort_counts(nq, 0, 32, sort, s);
  if (shared)
    batch_codes(qp.qpts, qp.qprob, nq, sc->dim, sc->stats, 0, batch_code_bits(P, sc->dim), codes, digits, s);
  else
    batch_codes(qp.qpts, qp.qprob, nq, sc->dim, sc->prob_stats, 1, sc->code_bits, codes, digits, s);
  radix_sort_counted(codes, sorted, nq, true, sort, nullptr, &qp.qst->bad, s);
  k_batch_pad<<<grid_for(qp.nproc, 256), 256, 0, s>>>(qp.qoff, d_pstart, P, qp.nproc, sorted, qp.qorder, qp.warp_prob);
  RTDL_LAUNCHED(1);
  // output order: by query id, then (stable) by problem; skipped when every
  // problem's ids are already ascending
  qp.oorder = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * (nq ? nq : 1), s));
  k_extract_ids<<<grid_for(nq, 256), 256, 0, s>>>(qp.qpts, nq, qp.sorted_flag, codes);
  RTDL_LAUNCHED(1);
  radix_sort_pairs(codes, qp.oorder, nq, 0, 32, true, qp.sorted_flag, &qp.qst->bad, s);
  k_gather_u32<<<grid_for(nq, 256), 256, 0, s>>>(qp.qprob, qp.oorder, nq, qp.sorted_flag, codes);
  RTDL_LAUNCHED(1);
  radix_sort_pairs(codes, qp.oorder, nq, 0, batch_problem_bits(P), false, qp.sorted_flag, &qp.qst->bad, s);
  dev_free(codes, s);
  dev_free(sorted, s);
  dev_free(d_pstart, s);
  return qp;
}

void free_prep(QueryPrep& qp, cudaStream_t s) {
  if (qp.borrowed) {
    dev_free(qp.bands, s);
    return;
  }
  dev_free(qp.qst, s);
  dev_free(qp.qpts, s);
  dev_free(qp.bands, s);
  dev_free(qp.qorder, s);
  dev_free(qp.qcodes, s);
  dev_free(qp.oorder, s);
  dev_free(qp.qprob, s);
  dev_free(qp.warp_prob, s);
  dev_free(qp.prob_kmax, s);
  dev_free(qp.sorted_flag, s);
  dev_free(qp.qoff, s);
  dev_free(qp.prob_radius, s);
}

}  // namespace

namespace {

// Output of the generic (block/warp-per-query) path: sorted candidate indices
// per query, located through heavy_out_off[h] (h = the query's generic slot).
struct GenericOut {
  uint32_t* heavy_out = nullptr;
  unsigned long long* heavy_out_off = nullptr;
  void release(cudaStream_t s) {
    dev_free(heavy_out, s);
    dev_free(heavy_out_off, s);
    heavy_out = nullptr;
    heavy_out_off = nullptr;
  }
};

// Runs the generic path for H queries listed in heavy_list with candidate
// counts heavy_m (read back here).  knn: gather every scene point (brute
// force); otherwise gather in-radius candidates through the BVH.
GenericOut run_generic_path(Scene* sc, const QueryPrep& qp, const void* queries_dev, int qstride, uint32_t H,
                            const uint32_t* heavy_list, const uint32_t* heavy_m, uint32_t limit, bool knn,
                            unsigned int* error, cudaStream_t s, const double* item_rad = nullptr) {
  GenericOut g;
  std::vector<uint32_t> hm(H);
  RTDL_CUDA_CHECK(cudaMemcpyAsync(hm.data(), heavy_m, sizeof(uint32_t) * H, cudaMemcpyDeviceToHost, s));
  RTDL_CUDA_CHECK(cudaStreamSynchronize(s));
  std::vector<unsigned long long> seg_off(H), out_off(H);
  std::vector<uint32_t> seg_size(H), out_cnt(H);
  unsigned long long seg_total = 0, out_total = 0;
  for (uint32_t h = 0; h < H; ++h) {
    seg_size[h] = next_pow2(hm[h] ? hm[h] : 1);
    seg_off[h] = seg_total;
    seg_total += seg_size[h];
    out_cnt[h] = hm[h] < limit ? hm[h] : limit;
    out_off[h] = out_total;
    out_total += out_cnt[h];
  }
  const unsigned long long kScratchLimit = 1ull << 28;  // entries (4 GiB of 16-B sort entries)
  if (seg_total > kScratchLimit)
    throw std::runtime_error(
        "b200 backend: the generic path for limits above 64 needs more than 4 GiB of sort scratch; "
        "reduce k/k_max or split the query set");
  unsigned long long* d_seg_off = static_cast<unsigned long long*>(dev_alloc(sizeof(unsigned long long) * H, s));
  uint32_t* d_seg_size = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * H, s));
  g.heavy_out_off = static_cast<unsigned long long*>(dev_alloc(sizeof(unsigned long long) * H, s));
  uint32_t* d_out_cnt = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * H, s));
  HeavyEntry* scratch = static_cast<HeavyEntry*>(dev_alloc(sizeof(HeavyEntry) * seg_total, s));
  g.heavy_out = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * (out_total ? out_total : 1), s));
  RTDL_CUDA_CHECK(cudaMemcpyAsync(d_seg_off, seg_off.data(), sizeof(unsigned long long) * H, cudaMemcpyHostToDevice, s));
  RTDL_CUDA_CHECK(cudaMemcpyAsync(d_seg_size, seg_size.data(), sizeof(uint32_t) * H, cudaMemcpyHostToDevice, s));
  RTDL_CUDA_CHECK(cudaMemcpyAsync(g.heavy_out_off, out_off.data(), sizeof(unsigned long long) * H,
                                  cudaMemcpyHostToDevice, s));
  RTDL_CUDA_CHECK(cudaMemcpyAsync(d_out_cnt, out_cnt.data(), sizeof(uint32_t) * H, cudaMemcpyHostToDevice, s));
  if (knn)
    k_heavy_gather<<<H, kHeavyThreads, 0, s>>>(sc->view(), qp.qpts, static_cast<const double*>(queries_dev), qstride,
                                               heavy_list, d_seg_off, d_seg_size, qp.bands, scratch, error);
  else
    k_heavy_gather_bvh<<<H, 32, 0, s>>>(qp.view, qp.qpts, static_cast<const double*>(queries_dev), qstride,
                                        heavy_list, d_seg_off, d_seg_size, qp.bands, qp.qprob, item_rad, scratch,
                                        error);
  k_heavy_sort<<<H, kHeavyThreads, sizeof(HeavyEntry) * kHeavySmemEntries, s>>>(d_seg_off, d_seg_size, scratch,
                                                                                sc->perm);
  k_heavy_emit<<<H, kHeavyThreads, 0, s>>>(d_seg_off, g.heavy_out_off, d_out_cnt, scratch, g.heavy_out);
  RTDL_LAUNCHED(3);
  RTDL_CUDA_CHECK(cudaStreamSynchronize(s));  // the host vectors above are read by the copies
  dev_free(d_seg_off, s);
  dev_free(d_seg_size, s);
  dev_free(d_out_cnt, s);
  dev_free(scratch, s);
  return g;
}

// Calls of at most this many queries collect a warp per query (32 warps on
// every SM); above it packets fill the GPU.
constexpr uint32_t kSingleQueries = kSmCount * 32;

// Whether the queries of a call on one scene walk alone, a warp each, because
// they are few or lie far apart among its points: the box around a packet then
// holds little that its queries share.  Time of walking alone over the packets'
// (fixed radius with 0.5, 32 and 130 in radius; KNN k = 1, 8, 32; uniform and
// clustered points): 3D, 10k queries 0.70 to 0.95 at any number of points, 80k
// over 1M points 0.68 to 1.05, 120k 0.77 to 0.97, 160k 0.93 to 1.16, over 2M
// points 160k 0.67 to 0.91, 240k 0.86 to 1.18; 2D, 20k over 1M points 0.63 to
// 0.96, 40k 0.72 to 1.19.  With 11,000 in radius 3D packets share more: 40k over
// 1M points 0.80, 80k 1.35.
inline bool queries_alone(uint64_t queries, uint64_t points, int dim) {
  return dim == 3 ? queries <= 3 * kSingleQueries || 10 * queries <= points
                  : queries <= kSingleQueries || 50 * queries <= points;
}
// Nearest points bound their packets better: 3D, 40k queries over 1M points 0.57
// (uniform), 0.60 (clustered) and 0.86 (a lattice) of the packets' time, 80k 0.86,
// 0.81 and 1.39.
inline bool nearest_alone(uint64_t queries, uint64_t points, int dim) {
  return queries_alone(dim == 3 && queries > 3 * kSingleQueries ? 2 * queries : queries, points, dim);
}

// The queries the packets left (their number is on the device).
void launch_collect_left(const CollectParams& C, uint32_t np, cudaStream_t s) {
  const unsigned int blocks = div_up(np, 128 / 32), cap = kSmCount * 8;
  k_collect_single<<<blocks < cap ? blocks : cap, 128, 0, s>>>(C, true);
  RTDL_LAUNCHED(1);
}

// Queries per packet: full packets once they give every SM `warps` of them, fewer
// below that, where the longest packet sets the time (a packet of eight meets
// half the buckets of one of 32).  A plain call's packets are alike: 24 warps are
// what an SM holds, and asking for 96 took a 262k-query summary from 1550 to
// 1835 us.  The problems of a batch are not, and short packets fill its last
// wave: with 96 instead of 24 (32 always, in a batch graph) six served requests
// went from 1190 to 1060 us, batches of 6 and 31 small problems from 725 and 770
// to 660 and 675, a graph of 8 problems from 785 to 650; 192 gave the same.
uint32_t packet_width(uint32_t np, bool batch) {
  const uint64_t warps = batch ? 96 : 24;
  return np >= 32u * warps * kSmCount ? 32u : np >= 16u * warps * kSmCount ? 16u : 8u;
}

// The collect pass over np processing ranks.
void launch_collect(CollectParams& C, uint32_t np, bool batch, cudaStream_t s) {
  if (!C.rank_radius && (batch ? np <= kSingleQueries : queries_alone(np, C.S.n, C.qstride - 1))) {
    k_collect_single<<<div_up(np, 128 / 32), 128, 0, s>>>(C, false);
    RTDL_LAUNCHED(1);
    return;
  }
  C.width = packet_width(np, batch);
  const unsigned int grid = div_up((uint64_t)div_up(np, C.width) * 32, kCollectThreads);
  const bool flat = C.qstride == 3;
  if (batch)
    flat ? k_collect_packet<2, true, false><<<grid, kCollectThreads, 0, s>>>(C)
         : k_collect_packet<3, true, false><<<grid, kCollectThreads, 0, s>>>(C);
  else if (C.rank_radius)
    flat ? k_collect_packet<2, false, true><<<grid, kCollectThreads, 0, s>>>(C)
         : k_collect_packet<3, false, true><<<grid, kCollectThreads, 0, s>>>(C);
  else
    flat ? k_collect_packet<2, false, false><<<grid, kCollectThreads, 0, s>>>(C)
         : k_collect_packet<3, false, false><<<grid, kCollectThreads, 0, s>>>(C);
  RTDL_LAUNCHED(1);
  if (!C.rank_radius) launch_collect_left(C, np, s);
}

void launch_emit(const EmitParams& E, uint32_t queries, cudaStream_t s) {
  k_emit<<<emit_grid(queries), kEmitThreads, 0, s>>>(E);
  RTDL_LAUNCHED(1);
}

// Blocks of the kernels that stride over a device list of at most np queries.
inline unsigned int list_grid(uint32_t np) {
  const unsigned int blocks = div_up(np, kEmitListThreads / 32);
  return blocks < kStrideBlocks ? blocks : kStrideBlocks;
}
static_assert(kEmitListThreads == kFixupThreads, "list_grid serves both");

// The list kernels over the collect's lists (lengths in small[2], small[3]).
void launch_emit_lists(const EmitParams& E, const CollectParams& C, uint32_t np, cudaStream_t s) {
  k_emit_mid<<<list_grid(np), kEmitListThreads, 0, s>>>(E, C.mid_list, 0, C.small + 2);
  k_emit_big<<<list_grid(np), kEmitListThreads, 0, s>>>(E, C.big_list, 0, C.small + 3);
  RTDL_LAUNCHED(2);
}

// fixed_radius_neighbors / bounded_knn_rows: collect, scan, emit.
QueryResult run_radius_query(Scene* sc, const void* queries_dev, uint32_t nq, int predicate, double radius,
                             uint32_t kmax, void* rows_dev, size_t rows_capacity, void** rows_alloc,
                             uint8_t* overflow_dev, cudaStream_t s, PhaseTimer* timer, const BatchSpec* bs = nullptr,
                             const SummarySpec* ss = nullptr, const PreparedQueries* pq = nullptr,
                             bool witness = false, RowDownload* dl = nullptr) {
  // witness (k_max 1): one row per query at its input position, pre-filled
  // with the no-witness row; the nearest in-radius neighbour overwrites it.
  QueryResult res;
  void* summary_rows = nullptr;  // ranked summaries: the rows stay internal
  if (ss) rows_alloc = &summary_rows;
  if (pq) queries_dev = pq->raw;
  const int qstride = sc->dim == 3 ? 4 : 3;
  if (bs) {  // the largest kmax bounds the generic path's output
    kmax = 1;
    for (uint32_t p = 0; p < bs->problems; ++p) kmax = bs->kmax[p] > kmax ? bs->kmax[p] : kmax;
  }
  QueryPrep qp = pq   ? borrow_prepared(sc, pq, radius, s)
                 : bs ? prepare_queries_batch(sc, queries_dev, nq, *bs, s)
                      : prepare_queries(sc, queries_dev, nq, true, radius, true, s);
  const uint32_t np = qp.nproc;  // processing ranks
  const size_t nq1 = nq ? nq : 1, np1 = np ? np : 1;
  uint32_t* qrank = pq ? pq->qrank : static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * nq1, s));
  if (!pq) {
    k_invert<<<grid_for(nq, 256), 256, 0, s>>>(qp.oorder, nq, qp.order_identity, qrank);
    RTDL_LAUNCHED(1);
  }
  if (timer) timer->mark("query_prep");
  std::vector<void*> bufs;
  auto alloc = [&](size_t bytes) {
    void* p = dev_alloc(bytes ? bytes : 1, s);
    bufs.push_back(p);
    return p;
  };
  uint32_t* counts = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * nq1));
  unsigned int* small = static_cast<unsigned int*>(alloc(sizeof(unsigned int) * 8));
  unsigned long long* offsets = static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * ((size_t)nq + 1)));
  unsigned long long* poff = static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * np1));
  unsigned long long* prob_rows =
      bs ? static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * (bs->problems + 1))) : nullptr;
  RTDL_CUDA_CHECK(cudaMemsetAsync(small, 0, sizeof(unsigned int) * 8, s));
  GenericOut g;
  auto cleanup = [&]() {
    g.release(s);
    if (!pq) dev_free(qrank, s);
    for (void* p : bufs) dev_free(p, s);
    free_prep(qp, s);
  };
  try {
    CollectParams C;
    C.S = qp.view;
    C.qpts = qp.qpts;
    C.qraw = static_cast<const double*>(queries_dev);
    C.qstride = qstride;
    C.qorder = qp.qorder;
    C.nq = np;
    C.kmax = kmax;
    C.radius = radius;
    C.bands = qp.bands;
    C.warp_prob = qp.warp_prob;
    C.prob_kmax = qp.prob_kmax;
    C.prob_radius = qp.prob_radius;
    C.rank_radius = nullptr;
    C.slab = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * slab_base((uint32_t)np1)));
    C.counts = counts;
    C.qinfo = static_cast<QueryInfo*>(alloc(sizeof(QueryInfo) * np1));
    C.flags = static_cast<uint8_t*>(alloc(nq1));
    C.heavy_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * nq1));
    C.heavy_m = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * nq1));
    C.heavy_rad = static_cast<double*>(alloc(sizeof(double) * nq1));
    C.heavy_t = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * nq1));
    C.mid_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * np1));
    C.big_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * np1));
    C.single_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * np1));
    C.small = small;
    C.overflow_out = overflow_dev;
    C.stats = nullptr;
    const bool stats = stats_enabled();
    if (stats) {
      C.stats = static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * kStatCount));
      RTDL_CUDA_CHECK(cudaMemsetAsync(C.stats, 0, sizeof(unsigned long long) * kStatCount, s));
    }
    if (timer) timer->mark("setup");
    launch_collect(C, np, bs != nullptr, s);
    if (stats)
      RTDL_CUDA_CHECK(cudaMemcpyAsync(last_stats().data(), C.stats, sizeof(unsigned long long) * kStatCount,
                                      cudaMemcpyDeviceToHost, s));
    if (timer) timer->mark("traverse");
    if (witness) {
      k_witness_offsets<<<grid_for(nq + 1, 256), 256, 0, s>>>(qp.oorder, qp.order_identity, nq, offsets);
      RTDL_LAUNCHED(1);
    } else {
      scan_counts_u64(counts, qp.oorder, qp.order_identity, nq, offsets, s);
    }
    if (bs) {
      k_problem_rows<<<div_up(bs->problems + 1, 256), 256, 0, s>>>(offsets, qp.qoff, bs->problems, prob_rows);
      RTDL_LAUNCHED(1);
      RTDL_CUDA_CHECK(cudaMemcpyAsync(bs->row_offsets, prob_rows, sizeof(unsigned long long) * (bs->problems + 1),
                                      cudaMemcpyDeviceToHost, s));
    }
    if (timer) timer->mark("scan");
    Readback* rb = pinned_readback();
    SmallReads reads(rb);
    // the row count, the list lengths and the input checks; waits
    auto read_counts = [&]() {
      reads.add(&rb->rows, offsets + nq, sizeof(unsigned long long));
      reads.add(&rb->heavy, small, sizeof(unsigned int) * 4);
      reads.add(&rb->fixups, small + 4, sizeof(unsigned int));
      reads.add(&rb->scene_bad, &sc->stats->bad, sizeof(unsigned int));
      reads.add(&rb->query_bad, &qp.qst->bad, sizeof(unsigned int));
      reads.launch(s);
      RTDL_CUDA_CHECK(cudaStreamSynchronize(s));
      throw_if_bad(rb->scene_bad | rb->query_bad);
      res.rows = rb->rows;
      res.heavy = rb->heavy;
      return *rb;
    };
    // queries whose candidates were not kept: gathered within the smallest
    // tested radius that holds their rows, sorted and written
    auto generic_path = [&](uint32_t n) {
      g = run_generic_path(sc, qp, queries_dev, qstride, n, C.heavy_list, C.heavy_m, kmax, false, small + 1, s,
                           C.heavy_rad);
      ExpandParams X;
      X.S = sc->view();
      X.qpts = qp.qpts;
      X.qraw = static_cast<const double*>(queries_dev);
      X.qstride = qstride;
      X.oorder = qp.oorder;
      X.bands = qp.bands;
      X.nq = n;
      X.L = kSlab;
      X.counts = counts;
      X.flags = C.flags;
      X.temp = nullptr;  // unused with a work list
      X.heavy_out = g.heavy_out;
      X.heavy_out_off = g.heavy_out_off;
      X.offsets = offsets;
      X.rows = rows_dev;
      X.capacity = rows_dev ? rows_capacity : 0;
      X.ranked = predicate == kFrn ? 0 : 1;
      X.overflow_out = nullptr;
      X.error = small + 1;
      X.work_list = C.heavy_list;
      X.qrank = qrank;
      k_expand<<<grid_for((uint64_t)n * 32, kExpandThreads), kExpandThreads, 0, s>>>(X);
      RTDL_LAUNCHED(1);
      if (stats) last_stats()[kStatGenericQueries] = n;
    };
    // Rows only counted: the total is known after the scan (no emit).
    const bool count_only = rows_alloc == nullptr && rows_dev == nullptr && !bs && !ss && !witness;
    if (count_only) {
      read_counts();
    } else {
      // rows copied to the host range by range as they are emitted
      bool chunked = dl != nullptr && (dl->alloc != nullptr || dl->host_fixed != nullptr) && rows_alloc != nullptr &&
                     !bs && !ss && !witness &&
                     nq >= (uint32_t)kDownloadChunks * 1024u;
      const size_t row_size = predicate == kFrn ? 16 : 24;
      Readback r{};
      if (rows_alloc != nullptr) {  // the row buffer is sized from the count
        if (chunked) {
          unsigned long long* chunk_dev =
              static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * (kDownloadChunks + 1)));
          k_chunk_rows<<<1, 32, 0, s>>>(offsets, nq, kDownloadChunks, chunk_dev);
          RTDL_LAUNCHED(1);
          reads.add(rb->chunk_rows, chunk_dev, sizeof(unsigned long long) * (kDownloadChunks + 1));
        }
        r = read_counts();
        if (res.rows == 0) chunked = false;
        rows_dev = res.rows ? dev_alloc(row_size * res.rows, s) : nullptr;
        rows_capacity = res.rows;
        *rows_alloc = rows_dev;
      }
      if (witness && rows_dev) {
        k_witness_fill<<<grid_for(nq, 256), 256, 0, s>>>(qp.qpts, nq, static_cast<RtdlFixedRadiusNeighborRow*>(rows_dev),
                                                         rows_capacity);
        RTDL_LAUNCHED(1);
      }
      k_proc_offsets<<<grid_for(np, 256), 256, 0, s>>>(qp.qorder, qrank, offsets, np, poff);
      RTDL_LAUNCHED(1);
      EmitParams E;
      E.S = sc->view();
      E.nq = np;
      E.slab = C.slab;
      E.qinfo = C.qinfo;
      E.poff = poff;
      E.sink.rows = rows_dev;
      E.sink.capacity = rows_dev ? rows_capacity : 0;
      E.sink.ranked = predicate == kFrn ? 0 : 1;
      E.fix_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * np1));
      E.fix_count = small + 4;
      if (chunked) {
        if (dl->host_fixed) {
          dl->host = dl->host_fixed;
          dl->pinned = true;
        } else {
          dl->host = dl->alloc(row_size * res.rows, &dl->pinned);
        }
        // Range by range in output order: each range's queries are emitted
        // (the list kernels and k_emit skip queries outside it), its deferred
        // queries fixed up, and the copy of its rows queued on the copy
        // stream, which overlaps the emission of the ranges after it.  The
        // generic queries' rows are written first.
        const uint32_t mid = r.mid, big = r.big;
        if (r.heavy > 0) generic_path(r.heavy);
        uint32_t* eorder = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * nq1));
        k_emit_order<<<grid_for(np, 256), 256, 0, s>>>(qp.qorder, qrank, np, eorder);
        RTDL_LAUNCHED(1);
        // the two list kernels' work, partitioned by range (list lengths in small[2], small[3])
        constexpr uint32_t C8 = kDownloadChunks, kPart = 3 * C8 + 1;
        unsigned int* part = static_cast<unsigned int*>(alloc(sizeof(unsigned int) * 2 * kPart));
        RTDL_CUDA_CHECK(cudaMemsetAsync(part, 0, sizeof(unsigned int) * 2 * kPart, s));
        uint32_t* lists_by_range[2] = {nullptr, nullptr};
        const uint32_t list_len[2] = {mid, big};
        uint32_t* lists[2] = {C.mid_list, C.big_list};
        for (int l = 0; l < 2; ++l) {
          if (list_len[l] == 0) continue;
          lists_by_range[l] = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * list_len[l]));
          const unsigned int grid = grid_for(list_len[l], 256);
          k_range_count<<<grid, 256, 0, s>>>(lists[l], small + 2 + l, qp.qorder, qrank, nq, C8, part + l * kPart);
          k_range_starts<<<1, 1, 0, s>>>(C8, part + l * kPart);
          k_range_scatter<<<grid, 256, 0, s>>>(lists[l], small + 2 + l, qp.qorder, qrank, nq, C8, part + l * kPart,
                                               lists_by_range[l]);
          RTDL_LAUNCHED(3);
        }
        E.order = eorder;
        E.fix_begin = small + 5;
        unsigned long long first[kDownloadChunks + 1];
        for (int c = 0; c <= kDownloadChunks; ++c) first[c] = r.chunk_rows[c];
        if (first[kDownloadChunks] != res.rows) throw std::runtime_error("row ranges disagree with the row count");
        for (int c = 0; c < (int)C8; ++c) {
          if (first[c + 1] == first[c]) continue;  // no rows in this range
          E.out_lo = (uint32_t)((uint64_t)nq * (uint32_t)c / C8);
          E.out_hi = (uint32_t)((uint64_t)nq * (uint32_t)(c + 1) / C8);
          E.range = c;
          // the list kernels stride over the range's part: grids sized for an even split
          if (mid > 0) {
            E.list_start = part + C8;
            k_emit_mid<<<div_up((uint64_t)div_up(mid, C8) * 32, kEmitListThreads), kEmitListThreads, 0, s>>>(
                E, lists_by_range[0], 0, nullptr);
          }
          if (big > 0) {
            E.list_start = part + kPart + C8;
            k_emit_big<<<div_up((uint64_t)div_up(big, C8) * 32, kEmitListThreads), kEmitListThreads, 0,
                                    s>>>(E, lists_by_range[1], 0, nullptr);
          }
          E.list_start = nullptr;
          launch_emit(E, E.out_hi - E.out_lo, s);
          k_emit_fixup<<<kSmCount * 4, kFixupThreads, 0, s>>>(E);
          k_fix_advance<<<1, 1, 0, s>>>(small + 5, small + 4);
          RTDL_LAUNCHED(4);
          const cudaEvent_t ev_range = aux_event(kEventRange);
          RTDL_CUDA_CHECK(cudaEventRecord(ev_range, s));
          RTDL_CUDA_CHECK(cudaStreamWaitEvent(dl->copy, ev_range, 0));
          RTDL_CUDA_CHECK(cudaMemcpyAsync(static_cast<char*>(dl->host) + first[c] * row_size,
                                          static_cast<const char*>(rows_dev) + first[c] * row_size,
                                          (first[c + 1] - first[c]) * row_size, cudaMemcpyDeviceToHost, dl->copy));
          ++dl->copies;
        }
      } else {
        // The list kernels (queries with 65..kSlab candidates: few warps, long
        // sorts) read their lengths on the device, so nothing waits for the
        // host between the collect and the rows.  In calls that fill the GPU
        // they run on the second stream beside k_emit, so each fills the
        // other's partial waves; they write disjoint rows, and the fix-up waits
        // for both.
        const bool side = np > kSingleQueries;
        cudaStream_t ls = s;
        if (side) {
          const cudaEvent_t ev_fork = aux_event(kEventFork);
          ls = aux_stream();
          RTDL_CUDA_CHECK(cudaEventRecord(ev_fork, s));
          RTDL_CUDA_CHECK(cudaStreamWaitEvent(ls, ev_fork, 0));
        }
        launch_emit_lists(E, C, np, ls);
        launch_emit(E, np, s);
        if (side) {
          const cudaEvent_t ev_join = aux_event(kEventJoin);
          RTDL_CUDA_CHECK(cudaEventRecord(ev_join, ls));
          RTDL_CUDA_CHECK(cudaStreamWaitEvent(s, ev_join, 0));
        }
        k_emit_fixup<<<list_grid(np), kFixupThreads, 0, s>>>(E);
        RTDL_LAUNCHED(1);
        r = read_counts();
        if (r.heavy > 0) generic_path(r.heavy);
      }
      if (timer) timer->mark("emit");
      if (chunked || r.heavy > 0) {
        reads.add(&rb->error, small + 1, sizeof(unsigned int));
        reads.add(&rb->fixups, small + 4, sizeof(unsigned int));
        reads.launch(s);
        RTDL_CUDA_CHECK(cudaStreamSynchronize(s));
        if (rb->error & 6u) throw std::runtime_error("generic neighbor path produced an inconsistent candidate count");
      }
      if (stats) last_stats()[kStatEmitFixups] = rb->fixups;
      if (chunked) {
        cleanup();
        return res;
      }
    }
    if (ss) {
      const uint32_t parts = div_up(nq, kSummaryGroup);
      SummaryPartial* partial = static_cast<SummaryPartial*>(dev_alloc(sizeof(SummaryPartial) * parts, s));
      RtdlFixedRadiusRankedNeighborAggregate* agg = static_cast<RtdlFixedRadiusRankedNeighborAggregate*>(
          dev_alloc(sizeof(RtdlFixedRadiusRankedNeighborAggregate), s));
      k_summarize<<<div_up(nq, kSummaryThreads), kSummaryThreads, 0, s>>>(static_cast<const RtdlFixedRadiusNeighborRow*>(summary_rows),
                                                    offsets, qp.oorder, qp.order_identity, qp.qpts, nq,
                                                    ss->summaries_dev, partial);
      k_summary_final<<<1, 1024, 0, s>>>(partial, parts, nq, agg);
      RTDL_LAUNCHED(2);
      RTDL_CUDA_CHECK(cudaMemcpyAsync(ss->aggregate_host, agg, sizeof(*agg), cudaMemcpyDeviceToHost, s));
      RTDL_CUDA_CHECK(cudaStreamSynchronize(s));
      dev_free(partial, s);
      dev_free(agg, s);
      if (timer) timer->mark("summarize");
    }
  } catch (...) {
    sync_quietly(s);
    sync_quietly(aux_stream(0));  // the list kernels may run there
    dev_free(summary_rows, s);
    cleanup();
    throw;
  }
  dev_free(summary_rows, s);
  cleanup();
  return res;
}

}  // namespace

QueryResult run_ranked_summaries(Scene* sc, const void* queries_dev, uint32_t nq, double radius, uint32_t kmax,
                                 RtdlFixedRadiusRankedNeighborSummary* summaries_dev,
                                 RtdlFixedRadiusRankedNeighborAggregate* aggregate_host, cudaStream_t s,
                                 PhaseTimer* timer, const PreparedQueries* pq) {
  if (pq) {
    if (pq->dim != sc->dim) throw std::runtime_error("prepared queries and scene differ in dimension");
    nq = pq->n;
  }
  if (sc->problems) throw std::runtime_error("a problem batch is queried with the batch entry points");
  if (kmax < 1 || kmax > 64)
    throw std::runtime_error("prepared ranked fixed_radius_neighbors_3d aggregate currently supports k_max <= 64");
  *aggregate_host = RtdlFixedRadiusRankedNeighborAggregate{nq, 0u, 0u, 0u, 0.0};
  if (nq == 0) return QueryResult{};
  // an empty search set gives no summaries and a zero aggregate, as the
  // reference's wrappers do (optix_runtime.py:2555-2572, 2644-2651)
  if (sc->n == 0) return QueryResult{};
  if (timer) timer->mark("start");
  SummarySpec ss{summaries_dev, aggregate_host};
  return run_radius_query(sc, queries_dev, nq, kFrn, radius, kmax, nullptr, 0, nullptr, nullptr, s, timer, nullptr,
                          &ss, pq);
}

QueryResult run_query_prepared(Scene* sc, const PreparedQueries* pq, double radius, uint32_t kmax, void* rows_dev,
                               size_t rows_capacity, uint8_t* overflow_dev, cudaStream_t s, PhaseTimer* timer) {
  if (sc->problems) throw std::runtime_error("a problem batch is queried with the batch entry points");
  if (pq->dim != sc->dim) throw std::runtime_error("prepared queries and scene differ in dimension");
  if (kmax < 1 || kmax > (uint32_t)kMaxList) throw std::runtime_error("prepared queries take k_max in [1, 64]");
  if (pq->n == 0) return QueryResult{};
  if (sc->n == 0) {
    if (overflow_dev) RTDL_CUDA_CHECK(cudaMemsetAsync(overflow_dev, 0, pq->n, s));
    return QueryResult{};
  }
  if (timer) timer->mark("start");
  return run_radius_query(sc, pq->raw, pq->n, kFrn, radius, kmax, rows_dev, rows_capacity, nullptr, overflow_dev, s,
                          timer, nullptr, nullptr, pq);
}

namespace {
// SoA point columns (partner-owned device buffers) -> RtdlPoint records.
__global__ void k_columns_to_records_2d(const uint32_t* ids, const double* x, const double* y, uint32_t n,
                                        RtdlPoint* out) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = RtdlPoint{ids[i], x[i], y[i]};
}
}  // namespace

void columns_to_records_2d(const uint32_t* ids, const double* x, const double* y, uint32_t n, void* out,
                           cudaStream_t s) {
  if (n == 0) return;
  k_columns_to_records_2d<<<grid_for(n, 256), 256, 0, s>>>(ids, x, y, n, static_cast<RtdlPoint*>(out));
  RTDL_LAUNCHED(1);
}

// ---- count with threshold, nearest witness --------------------------------------
namespace {
// The count (or, with nearest_rows, the point-group witness) walk over a scene;
// group_of / group_boxes restrict candidates to groups whose box is in radius.
void count_walk(Scene* sc, const void* queries_dev, uint32_t nq, double radius, uint32_t threshold,
                const CountOutputs& out, const uint32_t* group_of, const double* group_boxes,
                RtdlFixedRadiusNeighborRow* nearest_rows, cudaStream_t s) {
  if (nq == 0) return;
  if (sc->problems) throw std::runtime_error("a problem batch is queried with the batch entry points");
  QueryPrep qp = prepare_queries(sc, queries_dev, nq, true, radius, false, s);
  unsigned long long* reached = nullptr;
  try {
    if (out.reached_host) {
      reached = static_cast<unsigned long long*>(dev_alloc(sizeof(unsigned long long), s));
      RTDL_CUDA_CHECK(cudaMemsetAsync(reached, 0, sizeof(unsigned long long), s));
    }
    CountParams P;
    P.S = sc->view();
    P.qpts = qp.qpts;
    P.qraw = static_cast<const double*>(queries_dev);
    P.qstride = sc->dim == 3 ? 4 : 3;
    P.qorder = qp.qorder;
    P.nq = nq;
    P.bands = qp.bands;
    P.threshold = threshold;
    P.ids_out = out.ids;
    P.counts_out = out.counts;
    P.flags_out = out.flags;
    P.rows_out = out.rows;
    P.reached = reached;
    P.group_of = group_of;
    P.group_boxes = group_boxes;
    if (nearest_rows)
      k_group_nearest_packet<<<div_up(nq, 128), 128, 0, s>>>(P, nearest_rows);
    else if (sc->dim == 3)
      k_count_packet<3><<<div_up(nq, 128), 128, 0, s>>>(P);
    else
      k_count_packet<2><<<div_up(nq, 128), 128, 0, s>>>(P);
    RTDL_LAUNCHED(1);
    Readback* rb = pinned_readback();
    RTDL_CUDA_CHECK(cudaMemcpyAsync(&rb->scene_bad, &sc->stats->bad, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
    RTDL_CUDA_CHECK(cudaMemcpyAsync(&rb->query_bad, &qp.qst->bad, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
    if (reached)
      RTDL_CUDA_CHECK(cudaMemcpyAsync(&rb->rows, reached, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    RTDL_CUDA_CHECK(cudaStreamSynchronize(s));
    throw_if_bad(rb->scene_bad | rb->query_bad);
    if (out.reached_host) *out.reached_host = rb->rows;
  } catch (...) {
    sync_quietly(s);
    dev_free(reached, s);
    free_prep(qp, s);
    throw;
  }
  dev_free(reached, s);
  free_prep(qp, s);
}
}  // namespace

void run_count_threshold(Scene* sc, const void* queries_dev, uint32_t nq, double radius, uint32_t threshold,
                         const CountOutputs& out, cudaStream_t s) {
  count_walk(sc, queries_dev, nq, radius, threshold, out, nullptr, nullptr, nullptr, s);
}

PointGroupScene* point_group_create(const RtdlPoint* points, size_t count, const RtdlPointGroupBounds2D* groups,
                                    size_t group_count, double max_radius, cudaStream_t s) {
  size_t total = 0;
  for (size_t g = 0; g < group_count; ++g) {
    const RtdlPointGroupBounds2D& G = groups[g];
    if ((size_t)G.point_offset > count || (size_t)G.point_count > count - (size_t)G.point_offset)
      throw std::runtime_error("point_group_nearest_witness group span exceeds search point count");
    if (G.max_x < G.min_x || G.max_y < G.min_y)
      throw std::runtime_error("point_group_nearest_witness group bounds must be ordered");
    total += G.point_count;
  }
  if (total > (size_t)kMaxScenePoints) throw std::runtime_error("point groups reference more than 67,108,864 points");
  // the scene holds every group's points (a point in two groups twice), each tagged with its group
  std::vector<RtdlPoint> expanded(total);
  std::vector<uint32_t> group_of(total);
  std::vector<double> boxes(4 * group_count);
  size_t k = 0;
  for (size_t g = 0; g < group_count; ++g) {
    const RtdlPointGroupBounds2D& G = groups[g];
    for (uint32_t i = 0; i < G.point_count; ++i, ++k) {
      expanded[k] = points[G.point_offset + i];
      group_of[k] = (uint32_t)g;
    }
    boxes[4 * g] = G.min_x;
    boxes[4 * g + 1] = G.min_y;
    boxes[4 * g + 2] = G.max_x;
    boxes[4 * g + 3] = G.max_y;
  }
  PointGroupScene* pg = new PointGroupScene();
  pg->groups = (uint32_t)group_count;
  pg->points = (uint32_t)total;
  pg->max_radius = max_radius;
  void* d_pts = nullptr;
  try {
    d_pts = dev_alloc(sizeof(RtdlPoint) * (total ? total : 1), s);
    pg->group_of = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * (total ? total : 1), s));
    pg->boxes = static_cast<double*>(dev_alloc(sizeof(double) * (boxes.empty() ? 4 : boxes.size()), s));
    if (total) {
      RTDL_CUDA_CHECK(cudaMemcpyAsync(d_pts, expanded.data(), sizeof(RtdlPoint) * total, cudaMemcpyHostToDevice, s));
      RTDL_CUDA_CHECK(cudaMemcpyAsync(pg->group_of, group_of.data(), sizeof(uint32_t) * total, cudaMemcpyHostToDevice,
                                      s));
    }
    if (!boxes.empty())
      RTDL_CUDA_CHECK(cudaMemcpyAsync(pg->boxes, boxes.data(), sizeof(double) * boxes.size(), cudaMemcpyHostToDevice, s));
    pg->sc = build_scene(d_pts, (uint32_t)total, 2, s);
    unsigned int bad = 0;
    RTDL_CUDA_CHECK(cudaMemcpyAsync(&bad, &pg->sc->stats->bad, sizeof(bad), cudaMemcpyDeviceToHost, s));
    RTDL_CUDA_CHECK(cudaStreamSynchronize(s));  // the host vectors stay alive until the copies are done
    throw_if_bad(bad);
  } catch (...) {
    sync_quietly(s);
    dev_free(d_pts, s);
    point_group_destroy(pg);
    throw;
  }
  dev_free(d_pts, s);
  return pg;
}

void point_group_destroy(PointGroupScene* pg) {
  if (!pg) return;
  cudaStream_t s = pg->sc ? pg->sc->stream : nullptr;
  dev_free(pg->group_of, s);
  dev_free(pg->boxes, s);
  destroy_scene(pg->sc);
  if (s) cudaStreamSynchronize(s);
  delete pg;
}

void point_group_count(PointGroupScene* pg, const void* queries_dev, uint32_t nq, double radius, uint32_t threshold,
                       const CountOutputs& out, cudaStream_t s) {
  count_walk(pg->sc, queries_dev, nq, radius, threshold, out, pg->group_of, pg->boxes, nullptr, s);
}

void point_group_nearest(PointGroupScene* pg, const void* queries_dev, uint32_t nq, double radius,
                         RtdlFixedRadiusNeighborRow* rows_dev, RtdlFixedRadiusNeighborRow* max_row_host,
                         cudaStream_t s) {
  count_walk(pg->sc, queries_dev, nq, radius, 0, CountOutputs{}, pg->group_of, pg->boxes, rows_dev, s);
  if (max_row_host) {
    RtdlFixedRadiusNeighborRow* d_max =
        static_cast<RtdlFixedRadiusNeighborRow*>(dev_alloc(sizeof(RtdlFixedRadiusNeighborRow), s));
    k_witness_max<<<1, 1024, 0, s>>>(rows_dev, nq, d_max);
    RTDL_LAUNCHED(1);
    RTDL_CUDA_CHECK(cudaMemcpyAsync(max_row_host, d_max, sizeof(RtdlFixedRadiusNeighborRow), cudaMemcpyDeviceToHost, s));
    dev_free(d_max, s);
    RTDL_CUDA_CHECK(cudaStreamSynchronize(s));
  }
}

void run_count_trivial(const void* queries_dev, uint32_t nq, int dim, const CountOutputs& out, cudaStream_t s) {
  if (nq == 0) return;
  float4* qpts = static_cast<float4*>(dev_alloc(sizeof(float4) * nq, s));
  PointStats* st = static_cast<PointStats*>(dev_alloc(sizeof(PointStats), s));
  reset_stats(st, s);
  prep_points(queries_dev, nq, dim, qpts, st, s);
  k_count_trivial<<<grid_for(nq, 256), 256, 0, s>>>(qpts, nq, out.ids, out.counts, out.flags);
  RTDL_LAUNCHED(1);
  dev_free(qpts, s);
  dev_free(st, s);
}

QueryResult run_nearest_witness(Scene* sc, const void* queries_dev, uint32_t nq, double radius, void** rows_alloc,
                                cudaStream_t s, PhaseTimer* timer) {
  if (rows_alloc) *rows_alloc = nullptr;
  if (nq == 0 || sc->n == 0) return QueryResult{};
  if (sc->problems) throw std::runtime_error("a problem batch is queried with the batch entry points");
  return run_radius_query(sc, queries_dev, nq, kFrn, radius, 1, nullptr, 0, rows_alloc, nullptr, s, timer, nullptr,
                          nullptr, nullptr, true);
}

// ---- the plain per-call form: build and query in one call ---------------------
QueryResult run_build_and_query(const BuildQueryInputs& in, int predicate, double radius, uint32_t limit,
                                void* rows_dev, size_t rows_capacity, void** rows_alloc, uint8_t* overflow_dev,
                                cudaStream_t s, cudaStream_t aux, PhaseTimer* timer, Scene** scene_out,
                                void** query_owned, RowDownload* download) {
  *scene_out = nullptr;
  *query_owned = nullptr;
  const size_t qbytes = (in.dim == 3 ? sizeof(RtdlPoint3D) : sizeof(RtdlPoint)) * (size_t)in.nq;
  const bool overlap = predicate != kKnn && limit <= (uint32_t)kMaxList && in.nq > 0 && in.ns > 0 && aux != nullptr;
  if (!overlap) {
    const void* q = in.query_dev;
    if (in.query_host && in.nq) {
      *query_owned = dev_alloc(qbytes, s);
      RTDL_CUDA_CHECK(cudaMemcpyAsync(*query_owned, in.query_host, qbytes, cudaMemcpyHostToDevice, s));
      q = *query_owned;
    }
    Scene* sc = build_scene(in.search_dev, in.ns, in.dim, s);
    *scene_out = sc;
    if (timer) timer->mark("build");
    return run_query(sc, q, in.nq, predicate, radius, limit, rows_dev, rows_capacity, rows_alloc, overflow_dev, s,
                     timer);
  }
  // the query side does not need the scene until its bands: it is prepared on
  // `aux` (own-box curve order) while the scene builds on `s`
  const cudaEvent_t ev_start = aux_event(kEventStart), ev_ready = aux_event(kEventReady);
  RTDL_CUDA_CHECK(cudaEventRecord(ev_start, s));
  RTDL_CUDA_CHECK(cudaStreamWaitEvent(aux, ev_start, 0));  // whatever the caller queued on s comes first
  Scene* sc = build_scene(in.search_dev, in.ns, in.dim, s);
  *scene_out = sc;
  const void* q = in.query_dev;
  if (in.query_host) {  // a pageable copy holds the host; the build is already queued
    *query_owned = dev_alloc(qbytes, aux);
    RTDL_CUDA_CHECK(cudaMemcpyAsync(*query_owned, in.query_host, qbytes, cudaMemcpyHostToDevice, aux));
    q = *query_owned;
  }
  PreparedQueries* pq = nullptr;
  try {
    pq = prepare_query_set(q, in.nq, in.dim, aux);
  } catch (...) {
    sync_quietly(aux);
    throw;
  }
  RTDL_CUDA_CHECK(cudaEventRecord(ev_ready, aux));
  RTDL_CUDA_CHECK(cudaStreamWaitEvent(s, ev_ready, 0));
  pq->stream = s;  // from here the set is used and released on s
  if (timer) timer->mark("build");
  QueryResult r;
  try {
    r = run_radius_query(sc, q, in.nq, predicate, radius, limit, rows_dev, rows_capacity, rows_alloc, overflow_dev, s,
                         timer, nullptr, nullptr, pq, false, download);
  } catch (...) {
    pq->raw = nullptr;
    destroy_query_set(pq);
    throw;
  }
  pq->raw = nullptr;  // the caller's records (or *query_owned)
  destroy_query_set(pq);
  return r;
}

// Rows to host memory with the query set cut into `chunks` ranges of its input
// order, answered one after another against one scene: each range's rows are
// copied to their place in `host_rows` (the ranges' rows follow one another
// in input order, as one call's would) range by range on `copy` while the
// next range is collected and emitted on `s`.  The transfer of the rows,
// which bounds such a call, so starts after the first range's query instead
// of after the whole set's.  Each range is an ordinary query: its rows are
// the rows a call with only those queries gives.
QueryResult run_build_and_query_chunked(const BuildQueryInputs& in, int predicate, double radius, uint32_t limit,
                                        cudaStream_t s, cudaStream_t copy, PhaseTimer* timer, Scene** scene_out,
                                        void* host_rows, unsigned long long host_capacity_rows, int chunks) {
  *scene_out = nullptr;
  const size_t rec = in.dim == 3 ? sizeof(RtdlPoint3D) : sizeof(RtdlPoint);
  const size_t row_size = predicate == kFrn ? sizeof(RtdlFixedRadiusNeighborRow) : sizeof(RtdlKnnNeighborRow);
  // Each range's query set is uploaded and prepared (curve order, its own
  // statistics) on a third stream one range ahead: the first range's beside
  // the scene build, every later one beside the query of the range before it.
  cudaStream_t ps = aux_stream(1);
  std::vector<PreparedQueries*> sets(chunks, nullptr);
  std::vector<cudaEvent_t> ready(chunks, nullptr);
  auto range_of = [&](int c, uint32_t& q0, uint32_t& n) {
    q0 = (uint32_t)((uint64_t)in.nq * (uint32_t)c / (uint32_t)chunks);
    n = (uint32_t)((uint64_t)in.nq * (uint32_t)(c + 1) / (uint32_t)chunks) - q0;
  };
  auto prepare_range = [&](int c) {
    uint32_t q0, n;
    range_of(c, q0, n);
    void* d_q = dev_alloc(rec * n, ps);
    RTDL_CUDA_CHECK(cudaMemcpyAsync(d_q, static_cast<const char*>(in.query_host) + rec * q0, rec * n,
                                    cudaMemcpyHostToDevice, ps));
    PreparedQueries* pq = nullptr;
    try {
      pq = prepare_query_set(d_q, n, in.dim, ps);  // owns d_q from here
    } catch (...) {
      dev_free(d_q, ps);
      throw;
    }
    sets[c] = pq;
    RTDL_CUDA_CHECK(cudaEventCreateWithFlags(&ready[c], cudaEventDisableTiming));
    RTDL_CUDA_CHECK(cudaEventRecord(ready[c], ps));
  };
  // Every range keeps its device rows until all copies are done: a buffer
  // released behind its copies would make the pool order the next range's
  // allocation, and so its emission, after them.
  std::vector<void*> range_rows;
  auto release = [&]() {
    sync_quietly(ps);
    for (int c = 0; c < chunks; ++c) {
      if (sets[c]) {
        sets[c]->stream = s;
        destroy_query_set(sets[c]);
        sets[c] = nullptr;
      }
      if (ready[c]) {
        note_cleanup_error(cudaEventDestroy(ready[c]), "cudaEventDestroy");
        ready[c] = nullptr;
      }
    }
    for (void* p : range_rows) dev_free(p, s);
    range_rows.clear();
  };
  QueryResult total;
  try {
    // the query side waits for what the caller queued on s (the search set's upload)
    const cudaEvent_t ev_start = aux_event(kEventStart);
    RTDL_CUDA_CHECK(cudaEventRecord(ev_start, s));
    RTDL_CUDA_CHECK(cudaStreamWaitEvent(ps, ev_start, 0));
    prepare_range(0);
    Scene* sc = build_scene(in.search_dev, in.ns, in.dim, s);
    *scene_out = sc;
    if (timer) timer->mark("build");
    for (int c = 0; c < chunks; ++c) {
      uint32_t q0, nqc;
      range_of(c, q0, nqc);
      if (total.rows + (unsigned long long)nqc * limit > host_capacity_rows)
        throw std::runtime_error("host row buffer too small for the query ranges");
      RTDL_CUDA_CHECK(cudaStreamWaitEvent(s, ready[c], 0));
      PreparedQueries* pq = sets[c];
      pq->stream = s;  // from here the set is used and released on s
      if (c + 1 < chunks) prepare_range(c + 1);
      void* d_rows = nullptr;
      RowDownload dl;
      dl.host_fixed = static_cast<char*>(host_rows) + total.rows * row_size;
      dl.copy = copy;
      QueryResult r;
      try {
        r = run_radius_query(sc, nullptr, nqc, predicate, radius, limit, nullptr, 0, &d_rows, nullptr, s, nullptr,
                             nullptr, nullptr, pq, false, &dl);
        if (r.rows && dl.copies == 0)  // a range too small to be copied piecewise: one copy after its emit
          RTDL_CUDA_CHECK(cudaMemcpyAsync(dl.host_fixed, d_rows, r.rows * row_size, cudaMemcpyDeviceToHost, s));
      } catch (...) {
        if (d_rows) range_rows.push_back(d_rows);
        throw;
      }
      range_rows.push_back(d_rows);
      destroy_query_set(pq);
      sets[c] = nullptr;
      total.rows += r.rows;
      total.heavy += r.heavy;
    }
    if (timer) timer->mark("queries");
    // the rows are released on `s` once it has waited for the copies
    const cudaEvent_t ev_copied = aux_event(kEventCopied);
    RTDL_CUDA_CHECK(cudaEventRecord(ev_copied, copy));
    RTDL_CUDA_CHECK(cudaStreamWaitEvent(s, ev_copied, 0));
    release();
  } catch (...) {
    sync_quietly(copy);
    sync_quietly(s);
    release();
    throw;
  }
  return total;
}

// ---- captured summary graphs ------------------------------------------------
namespace {

constexpr unsigned int kGraphStatusGeneric = 2u;   // heavy queries left for the generic path
constexpr unsigned int kBatchGraphStatusRows = 4u;  // a batch graph's rows exceed the caller's row buffer

__global__ void k_graph_status(const unsigned int* small, uint32_t requests, unsigned int* status) {
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < requests; r += gridDim.x * blockDim.x)
    status[r] = small[8 * (size_t)r] ? kGraphStatusGeneric : 0u;
}

}  // namespace

struct SummaryGraph {
  Scene* sc = nullptr;
  const PreparedQueries* pq = nullptr;
  cudaStream_t stream = nullptr;
  uint32_t R = 0, nq = 0, kcap = 0;  // requests, queries, row capacity per query
  std::vector<double> radius;
  std::vector<uint32_t> kmax;
  std::vector<void*> buffers;  // device, released at destroy
  DevBands* bands = nullptr;   // one per request
  uint32_t* slab = nullptr;
  uint32_t* counts = nullptr;
  QueryInfo* qinfo = nullptr;
  uint8_t* flags = nullptr;
  uint32_t *heavy_list = nullptr, *heavy_m = nullptr, *heavy_t = nullptr;
  double* heavy_rad = nullptr;
  uint32_t* single_list = nullptr;
  uint32_t *mid_list = nullptr, *big_list = nullptr, *fix_list = nullptr;
  unsigned int* small = nullptr;       // 8 counters per request (CollectParams::small)
  unsigned long long *offsets = nullptr, *poff = nullptr;
  void* scan_ws = nullptr;
  void* rows = nullptr;  // nq * kcap rows
  SummaryPartial* partial = nullptr;
  uint32_t summary_parts = 0;
  RtdlFixedRadiusRankedNeighborAggregate* agg = nullptr;  // one per request
  unsigned int* status = nullptr;                         // one per request
  RtdlFixedRadiusRankedNeighborAggregate* agg_host = nullptr;  // pinned
  unsigned int* status_host = nullptr;                          // pinned
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int kernels = 0;  // kernel nodes per replay
  uint64_t fallbacks = 0;
};

namespace {

void graph_check_requests(const Scene* sc, const double* radii, const uint32_t* kmax, uint32_t requests) {
  if (requests == 0) throw std::runtime_error("fixed_radius_neighbors_3d graph request_count must be positive");
  if (!radii || !kmax) throw std::runtime_error("radii and k_values must not be null");
  for (uint32_t r = 0; r < requests; ++r) {
    if (!(radii[r] >= 0.0)) throw std::runtime_error("fixed_radius_neighbors_3d radius must be non-negative");
    if (radii[r] > sc->max_radius + 1.0e-7)
      throw std::runtime_error("fixed_radius_neighbors_3d radius exceeds prepared max_radius");
    if (kmax[r] == 0) throw std::runtime_error("fixed_radius_neighbors_3d k_max must be positive");
    if (kmax[r] > 64)
      throw std::runtime_error("prepared ranked fixed_radius_neighbors_3d aggregate currently supports k_max <= 64");
  }
}

// One request's kernels, device-driven (no host reads, no allocation).
void graph_enqueue_request(SummaryGraph* g, uint32_t r, cudaStream_t s) {
  Scene* sc = g->sc;
  const PreparedQueries* pq = g->pq;
  const uint32_t nq = g->nq, np = nq;
  const double radius = g->radius[r];
  const uint32_t kmax = g->kmax[r];
  unsigned int* small = g->small + 8 * (size_t)r;
  k_bands<<<1, 32, 0, s>>>(sc->stats, pq->qst, radius, 1, g->bands + r);
  RTDL_LAUNCHED(1);
  CollectParams C;
  C.S = sc->view();
  C.qpts = pq->qpts;
  C.qraw = static_cast<const double*>(pq->raw);
  C.qstride = sc->dim == 3 ? 4 : 3;
  C.qorder = pq->qorder;
  C.nq = np;
  C.kmax = kmax;
  C.radius = radius;
  C.bands = g->bands + r;
  C.warp_prob = nullptr;
  C.prob_kmax = nullptr;
  C.prob_radius = nullptr;
  C.slab = g->slab;
  C.counts = g->counts;
  C.qinfo = g->qinfo;
  C.flags = g->flags;
  C.heavy_list = g->heavy_list;
  C.heavy_m = g->heavy_m;
  C.heavy_rad = g->heavy_rad;
  C.heavy_t = g->heavy_t;
  C.mid_list = g->mid_list;
  C.big_list = g->big_list;
  C.single_list = g->single_list;
  C.small = small;
  C.overflow_out = nullptr;
  C.rank_radius = nullptr;
  C.stats = nullptr;
  launch_collect(C, np, false, s);
  scan_counts_u64_ws(g->counts, pq->oorder, pq->identity, nq, g->offsets, g->scan_ws, s);
  k_proc_offsets<<<grid_for(np, 256), 256, 0, s>>>(pq->qorder, pq->qrank, g->offsets, np, g->poff);
  RTDL_LAUNCHED(1);
  EmitParams E;
  E.S = sc->view();
  E.nq = np;
  E.slab = g->slab;
  E.qinfo = g->qinfo;
  E.poff = g->poff;
  E.sink.rows = g->rows;
  E.sink.capacity = (unsigned long long)nq * g->kcap;
  E.sink.ranked = 0;
  E.fix_list = g->fix_list;
  E.fix_count = small + 4;
  launch_emit(E, np, s);
  launch_emit_lists(E, C, np, s);
  k_emit_fixup<<<list_grid(np), kFixupThreads, 0, s>>>(E);
  k_summarize<<<div_up(nq, kSummaryThreads), kSummaryThreads, 0, s>>>(static_cast<const RtdlFixedRadiusNeighborRow*>(g->rows),
                                                            g->offsets, pq->oorder, pq->identity, pq->qpts, nq,
                                                            nullptr, g->partial);
  k_summary_final<<<1, 1024, 0, s>>>(g->partial, g->summary_parts, nq, g->agg + r);
  RTDL_LAUNCHED(3);
}

void graph_release(SummaryGraph* g) {
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  g->exec = nullptr;
  g->graph = nullptr;
}

void graph_capture(SummaryGraph* g) {
  graph_release(g);
  cudaStream_t s = g->stream;
  const unsigned long long before = launches_counted();
  RTDL_CUDA_CHECK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  try {
    RTDL_CUDA_CHECK(cudaMemsetAsync(g->small, 0, sizeof(unsigned int) * 8 * (size_t)g->R, s));
    for (uint32_t r = 0; r < g->R; ++r) graph_enqueue_request(g, r, s);
    k_graph_status<<<div_up(g->R, 256), 256, 0, s>>>(g->small, g->R, g->status);
    RTDL_LAUNCHED(1);
  } catch (...) {
    cudaGraph_t partial = nullptr;
    cudaStreamEndCapture(s, &partial);
    if (partial) cudaGraphDestroy(partial);
    cudaGetLastError();
    count_launches(-(int)(launches_counted() - before));
    throw;
  }
  // captured kernels are counted when a replay launches them
  count_launches(-(int)(launches_counted() - before));
  RTDL_CUDA_CHECK(cudaStreamEndCapture(s, &g->graph));
  RTDL_CUDA_CHECK(cudaGraphInstantiate(&g->exec, g->graph, 0));
  size_t n = 0;
  RTDL_CUDA_CHECK(cudaGraphGetNodes(g->graph, nullptr, &n));
  std::vector<cudaGraphNode_t> nodes(n);
  RTDL_CUDA_CHECK(cudaGraphGetNodes(g->graph, nodes.data(), &n));
  g->kernels = 0;
  for (size_t i = 0; i < n; ++i) {
    cudaGraphNodeType t;
    RTDL_CUDA_CHECK(cudaGraphNodeGetType(nodes[i], &t));
    if (t == cudaGraphNodeTypeKernel) ++g->kernels;
  }
}

void graph_set_requests(SummaryGraph* g, const double* radii, const uint32_t* kmax, uint32_t requests) {
  g->radius.assign(radii, radii + requests);
  g->kmax.assign(kmax, kmax + requests);
}

// Row buffer for the largest k_max of the requests (grown by an update, never shrunk).
void graph_size_rows(SummaryGraph* g) {
  uint32_t k = 1;
  for (uint32_t v : g->kmax) k = v > k ? v : k;
  if (g->rows && k <= g->kcap) return;
  dev_free(g->rows, g->stream);
  g->rows = nullptr;
  g->kcap = 0;
  g->rows = dev_alloc(sizeof(RtdlFixedRadiusNeighborRow) * (size_t)g->nq * k, g->stream);
  g->kcap = k;
}

}  // namespace

SummaryGraph* summary_graph_create(Scene* sc, const PreparedQueries* pq, const double* radii, const uint32_t* kmax,
                                   uint32_t requests) {
  if (!sc) throw std::runtime_error("prepared OptiX fixed-radius-neighbor 3D handle must not be null");
  if (!pq) throw std::runtime_error("prepared fixed-radius query handle must not be null");
  if (sc->problems) throw std::runtime_error("a problem batch is queried with the batch entry points");
  if (pq->dim != sc->dim) throw std::runtime_error("prepared queries and scene differ in dimension");
  graph_check_requests(sc, radii, kmax, requests);
  if (pq->n == 0 || sc->n == 0)
    throw std::runtime_error("fixed_radius_neighbors_3d graph requires non-empty prepared search and query handles");
  SummaryGraph* g = new SummaryGraph();
  g->sc = sc;
  g->pq = pq;
  g->R = requests;
  g->nq = pq->n;
  graph_set_requests(g, radii, kmax, requests);
  try {
    RTDL_CUDA_CHECK(cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking));
    cudaStream_t s = g->stream;
    // the scene and the prepared queries were built on their own streams
    RTDL_CUDA_CHECK(cudaStreamSynchronize(sc->stream));
    RTDL_CUDA_CHECK(cudaStreamSynchronize(pq->stream));
    unsigned int bad[2] = {0, 0};
    RTDL_CUDA_CHECK(cudaMemcpy(&bad[0], &sc->stats->bad, sizeof(unsigned int), cudaMemcpyDeviceToHost));
    RTDL_CUDA_CHECK(cudaMemcpy(&bad[1], &pq->qst->bad, sizeof(unsigned int), cudaMemcpyDeviceToHost));
    throw_if_bad(bad[0] | bad[1]);
    auto alloc = [&](size_t bytes) {
      void* p = dev_alloc(bytes ? bytes : 1, s);
      g->buffers.push_back(p);
      return p;
    };
    const size_t n = g->nq, R = g->R;
    g->bands = static_cast<DevBands*>(alloc(sizeof(DevBands) * R));
    g->slab = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * slab_base(g->nq)));
    g->counts = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * n));
    g->qinfo = static_cast<QueryInfo*>(alloc(sizeof(QueryInfo) * n));
    g->flags = static_cast<uint8_t*>(alloc(n));
    g->heavy_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * n));
    g->heavy_m = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * n));
    g->heavy_t = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * n));
    g->mid_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * n));
    g->big_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * n));
    g->fix_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * n));
    g->small = static_cast<unsigned int*>(alloc(sizeof(unsigned int) * 8 * R));
    g->offsets = static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * (n + 1)));
    g->poff = static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * n));
    g->scan_ws = alloc(scan_workspace_bytes(g->nq));
    graph_size_rows(g);
    g->heavy_rad = static_cast<double*>(alloc(sizeof(double) * n));
    g->single_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * n));
    g->summary_parts = div_up(n, kSummaryGroup);
    g->partial = static_cast<SummaryPartial*>(alloc(sizeof(SummaryPartial) * g->summary_parts));
    g->agg = static_cast<RtdlFixedRadiusRankedNeighborAggregate*>(
        alloc(sizeof(RtdlFixedRadiusRankedNeighborAggregate) * R));
    g->status = static_cast<unsigned int*>(alloc(sizeof(unsigned int) * R));
    RTDL_CUDA_CHECK(cudaMallocHost(&g->agg_host, sizeof(RtdlFixedRadiusRankedNeighborAggregate) * R));
    RTDL_CUDA_CHECK(cudaMallocHost(&g->status_host, sizeof(unsigned int) * R));
    RTDL_CUDA_CHECK(cudaStreamSynchronize(s));  // allocations ready before capture
    graph_capture(g);
  } catch (...) {
    summary_graph_destroy(g);
    throw;
  }
  return g;
}

void summary_graph_update(SummaryGraph* g, const double* radii, const uint32_t* kmax, uint32_t requests) {
  if (!g) throw std::runtime_error("prepared fixed_radius_neighbors_3d graph handle must not be null");
  if (requests != g->R)
    throw std::runtime_error("fixed_radius_neighbors_3d graph request update requires unchanged request_count");
  graph_check_requests(g->sc, radii, kmax, requests);
  RTDL_CUDA_CHECK(cudaStreamSynchronize(g->stream));  // no replay in flight while the graph is replaced
  graph_set_requests(g, radii, kmax, requests);
  graph_size_rows(g);
  RTDL_CUDA_CHECK(cudaStreamSynchronize(g->stream));
  graph_capture(g);
}

void summary_graph_launch(SummaryGraph* g) {
  if (!g || !g->exec) throw std::runtime_error("prepared fixed_radius_neighbors_3d graph handle must not be null");
  RTDL_CUDA_CHECK(cudaGraphLaunch(g->exec, g->stream));
  count_launches(g->kernels);
}

void summary_graph_replay(SummaryGraph* g, RtdlFixedRadiusRankedNeighborAggregate* out) {
  if (!out) throw std::runtime_error("aggregates_out must not be null");
  summary_graph_launch(g);
  cudaStream_t s = g->stream;
  RTDL_CUDA_CHECK(cudaMemcpyAsync(g->agg_host, g->agg, sizeof(RtdlFixedRadiusRankedNeighborAggregate) * g->R,
                                  cudaMemcpyDeviceToHost, s));
  RTDL_CUDA_CHECK(cudaMemcpyAsync(g->status_host, g->status, sizeof(unsigned int) * g->R, cudaMemcpyDeviceToHost, s));
  RTDL_CUDA_CHECK(cudaStreamSynchronize(s));
  for (uint32_t r = 0; r < g->R; ++r) {
    if (g->status_host[r] & kGraphStatusGeneric) {
      // the plain call, with its generic path for the queries refinement left
      run_ranked_summaries(g->sc, nullptr, g->nq, g->radius[r], g->kmax[r], nullptr, &out[r], s, nullptr, g->pq);
      ++g->fallbacks;
    } else {
      out[r] = g->agg_host[r];
    }
  }
}

const RtdlFixedRadiusRankedNeighborAggregate* summary_graph_device_aggregates(const SummaryGraph* g) { return g->agg; }
const unsigned int* summary_graph_device_status(const SummaryGraph* g) { return g->status; }
cudaStream_t summary_graph_stream(const SummaryGraph* g) { return g->stream; }
uint32_t summary_graph_requests(const SummaryGraph* g) { return g->R; }
uint64_t summary_graph_fallbacks(const SummaryGraph* g) { return g->fallbacks; }

void summary_graph_destroy(SummaryGraph* g) {
  if (!g) return;
  if (g->stream) cudaStreamSynchronize(g->stream);
  graph_release(g);
  for (void* p : g->buffers) dev_free(p, g->stream);
  dev_free(g->rows, g->stream);
  if (g->stream) {
    sync_quietly(g->stream);
    note_cleanup_error(cudaStreamDestroy(g->stream), "cudaStreamDestroy");
  }
  if (g->agg_host) cudaFreeHost(g->agg_host);
  if (g->status_host) cudaFreeHost(g->status_host);
  delete g;
}

namespace {
__global__ void k_identity_flag(const PointStats* qst, unsigned int* identity) {
  if (threadIdx.x == 0) *identity = qst->ids_unsorted ? 0u : 1u;
}
}  // namespace

PreparedQueries* prepare_query_set(const void* records_dev, uint32_t n, int dim, cudaStream_t s) {
  PreparedQueries* pq = new PreparedQueries();
  pq->dim = dim;
  pq->n = n;
  pq->stream = s;
  RTDL_CUDA_CHECK(cudaGetDevice(&pq->device));
  const size_t n1 = n ? n : 1;
  try {
    pq->raw = const_cast<void*>(records_dev);
    pq->qst = static_cast<PointStats*>(dev_alloc(sizeof(PointStats), s));
    pq->qpts = static_cast<float4*>(dev_alloc(sizeof(float4) * n1, s));
    pq->qorder = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * n1, s));
    pq->oorder = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * n1, s));
    pq->qrank = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * n1, s));
    pq->identity = static_cast<unsigned int*>(dev_alloc(sizeof(unsigned int), s));
    reset_stats(pq->qst, s);
    prep_points(records_dev, n, dim, pq->qpts, pq->qst, s);
    k_identity_flag<<<1, 32, 0, s>>>(pq->qst, pq->identity);
    RTDL_LAUNCHED(1);
    uint32_t* codes = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * n1, s));
    SortWork sort;
    uint32_t* digits = radix_sort_counts(n, 0, curve_bits(dim), sort, s);
    curve_codes(pq->qpts, n, dim, pq->qst, codes, digits, s);  // the set's own box: the order only groups neighbours
    radix_sort_counted(codes, pq->qorder, n, true, sort, nullptr, &pq->qst->bad, s);
    k_extract_ids<<<grid_for(n, 256), 256, 0, s>>>(pq->qpts, n, pq->identity, codes);
    RTDL_LAUNCHED(1);
    radix_sort_pairs(codes, pq->oorder, n, 0, 32, true, pq->identity, &pq->qst->bad, s);
    k_invert<<<grid_for(n, 256), 256, 0, s>>>(pq->oorder, n, pq->identity, pq->qrank);
    RTDL_LAUNCHED(1);
    dev_free(codes, s);
  } catch (...) {
    pq->raw = nullptr;
    destroy_query_set(pq);
    throw;
  }
  return pq;
}

void destroy_query_set(PreparedQueries* pq) {
  if (!pq) return;
  cudaStream_t s = pq->stream;
  dev_free(pq->raw, s);
  dev_free(pq->qst, s);
  dev_free(pq->qpts, s);
  dev_free(pq->qorder, s);
  dev_free(pq->oorder, s);
  dev_free(pq->qrank, s);
  dev_free(pq->identity, s);
  delete pq;
}

QueryResult run_query_batch(Scene* sc, const void* queries_dev, const BatchSpec& bs, void* rows_dev,
                            size_t rows_capacity, void** rows_alloc, uint8_t* overflow_dev, cudaStream_t s,
                            PhaseTimer* timer) {
  if (rows_alloc) *rows_alloc = nullptr;
  if (sc->problems != 0 && sc->problems != bs.problems)
    throw std::runtime_error("query batch and scene batch differ in problem count");
  if (bs.qoff[0] != 0) throw std::runtime_error("query offsets must start at 0");
  for (uint32_t p = 0; p < bs.problems; ++p) {
    if (bs.qoff[p + 1] < bs.qoff[p]) throw std::runtime_error("query offsets must be non-decreasing");
    if (!(bs.radius[p] >= 0.0)) throw std::runtime_error("radius must be non-negative");
    if (bs.kmax[p] < 1 || bs.kmax[p] > 64) throw std::runtime_error("a problem batch takes k_max in [1, 64]");
  }
  const unsigned long long nq = bs.qoff[bs.problems];
  if (nq > 0xFFFFFFFFull) throw std::runtime_error("query_count exceeds uint32 limit");
  if (nq == 0 || sc->n == 0) {
    for (uint32_t p = 0; p <= bs.problems; ++p) bs.row_offsets[p] = 0;
    return QueryResult{};
  }
  return run_radius_query(sc, queries_dev, (uint32_t)nq, kFrn, 0.0, 0, rows_dev, rows_capacity, rows_alloc,
                          overflow_dev, s, timer, &bs);
}

namespace {

// Row offsets by processing rank when every query has `rows` rows.
__global__ void k_uniform_offsets(const uint32_t* qorder, const uint32_t* qrank, uint32_t nq, uint32_t rows,
                                  unsigned long long* poff) {
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < nq; t += (uint64_t)gridDim.x * blockDim.x)
    poff[t] = (unsigned long long)qrank[qorder[t]] * rows;
}

template <int KP>
void launch_knn_radius(const Scene* sc, const QueryPrep& qp, uint32_t nq, uint32_t k, double* radius, cudaStream_t s) {
  if (sc->dim == 3)
    k_knn_radius<3, KP><<<div_up(nq, 128), 128, 0, s>>>(sc->view(), sc->codes, qp.qpts, qp.qorder, qp.qcodes, nq, k,
                                                       qp.bands, radius);
  else
    k_knn_radius<2, KP><<<div_up(nq, 128), 128, 0, s>>>(sc->view(), sc->codes, qp.qpts, qp.qorder, qp.qcodes, nq, k,
                                                       qp.bands, radius);
  RTDL_LAUNCHED(1);
}

// Processing ranks answered at a time by run_knn: bounds the slab (4 GiB).
constexpr uint32_t kKnnRanks = 1u << 22;

// knn_rows with k <= 64: every query has min(k, n) rows, so nothing is scanned
// and the host reads nothing back before the rows are written.
QueryResult run_knn(Scene* sc, const void* queries_dev, uint32_t nq, uint32_t k, void* rows_dev, size_t rows_capacity,
                    void** rows_alloc, uint8_t* overflow_dev, cudaStream_t s, PhaseTimer* timer) {
  QueryResult res;
  const int qstride = sc->dim == 3 ? 4 : 3;
  const uint32_t kk = k < sc->n ? k : sc->n;
  std::vector<void*> bufs;
  QueryPrep qp = prepare_queries(sc, queries_dev, nq, false, 0.0, true, s);
  auto alloc = [&](size_t bytes) {
    void* p = dev_alloc(bytes ? bytes : 1, s);
    bufs.push_back(p);
    return p;
  };
  auto cleanup = [&]() {
    for (void* p : bufs) dev_free(p, s);
    free_prep(qp, s);
  };
  try {
    uint32_t* qrank = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * nq));
    k_invert<<<grid_for(nq, 256), 256, 0, s>>>(qp.oorder, nq, qp.order_identity, qrank);
    RTDL_LAUNCHED(1);
    if (timer) timer->mark("query_prep");
    res.rows = (unsigned long long)nq * kk;
    if (rows_alloc != nullptr) {
      rows_dev = dev_alloc(sizeof(RtdlKnnNeighborRow) * res.rows, s);
      rows_capacity = res.rows;
      *rows_alloc = rows_dev;
    }
    if (overflow_dev) RTDL_CUDA_CHECK(cudaMemsetAsync(overflow_dev, 0, nq, s));
    const bool stats = stats_enabled();
    if (rows_dev) {
      const uint32_t most = nq < kKnnRanks ? nq : kKnnRanks;
      double* radius = static_cast<double*>(alloc(sizeof(double) * nq));
      unsigned long long* poff = static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * nq));
      k_uniform_offsets<<<grid_for(nq, 256), 256, 0, s>>>(qp.qorder, qrank, nq, kk, poff);
      RTDL_LAUNCHED(1);
      if (kk <= 8) launch_knn_radius<8>(sc, qp, nq, k, radius, s);
      else if (kk <= 16) launch_knn_radius<16>(sc, qp, nq, k, radius, s);
      else if (kk <= 32) launch_knn_radius<32>(sc, qp, nq, k, radius, s);
      else launch_knn_radius<64>(sc, qp, nq, k, radius, s);
      unsigned int* small = static_cast<unsigned int*>(alloc(sizeof(unsigned int) * 8));
      CollectParams C;
      C.S = qp.view;
      C.qpts = qp.qpts;
      C.qraw = static_cast<const double*>(queries_dev);
      C.qstride = qstride;
      C.kmax = kk;
      C.radius = 0.0;
      C.bands = qp.bands;
      C.warp_prob = nullptr;
      C.prob_kmax = nullptr;
      C.prob_radius = nullptr;
      C.slab = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * slab_base(most)));
      C.counts = nullptr;
      C.qinfo = static_cast<QueryInfo*>(alloc(sizeof(QueryInfo) * most));
      C.flags = nullptr;
      C.heavy_list = C.heavy_m = C.heavy_t = nullptr;
      C.heavy_rad = nullptr;
      C.mid_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * most));
      C.big_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * most));
      C.single_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * most));
      C.small = small;
      C.overflow_out = nullptr;
      C.stats = nullptr;
      if (stats) {
        C.stats = static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * kStatCount));
        RTDL_CUDA_CHECK(cudaMemsetAsync(C.stats, 0, sizeof(unsigned long long) * kStatCount, s));
      }
      EmitParams E;
      E.S = sc->view();
      E.slab = C.slab;
      E.qinfo = C.qinfo;
      E.sink.rows = rows_dev;
      E.sink.capacity = rows_capacity;
      E.sink.ranked = 1;
      E.fix_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * most));
      E.fix_count = small + 4;
      for (uint32_t t0 = 0; t0 < nq; t0 += most) {  // kernels see one range of ranks at a time
        const uint32_t np = nq - t0 < most ? nq - t0 : most;
        RTDL_CUDA_CHECK(cudaMemsetAsync(small, 0, sizeof(unsigned int) * 8, s));
        C.qorder = qp.qorder + t0;
        C.nq = np;
        C.rank_radius = radius + t0;
        E.nq = np;
        E.poff = poff + t0;
        SingleParams H{};
        H.S = sc->view();
        H.qpts = qp.qpts;
        H.qraw = C.qraw;
        H.qstride = qstride;
        H.bands = qp.bands;
        H.k = kk;
        H.qorder = C.qorder;
        H.rank_radius = C.rank_radius;
        H.poff = E.poff;
        H.sink = E.sink;
        H.stats = C.stats;
        if (queries_alone(np, sc->n, sc->dim)) {
          H.nwork = np;
          stats ? k_knn_single<true><<<div_up(np, 256 / 32), 256, 0, s>>>(H)
                : k_knn_single<false><<<div_up(np, 256 / 32), 256, 0, s>>>(H);
          RTDL_LAUNCHED(1);
          continue;
        }
        launch_collect(C, np, false, s);
        // the queries the packets left, beside the emit kernels (disjoint rows)
        const cudaEvent_t ev_fork = aux_event(kEventFork), ev_join = aux_event(kEventJoin);
        cudaStream_t ls = aux_stream();
        RTDL_CUDA_CHECK(cudaEventRecord(ev_fork, s));
        RTDL_CUDA_CHECK(cudaStreamWaitEvent(ls, ev_fork, 0));
        H.work = C.single_list;
        H.nwork_dev = small + 6;
        stats ? k_knn_single<true><<<kSmCount * 4, 256, 0, ls>>>(H)
              : k_knn_single<false><<<kSmCount * 4, 256, 0, ls>>>(H);
        launch_emit_lists(E, C, np, ls);
        RTDL_CUDA_CHECK(cudaEventRecord(ev_join, ls));
        launch_emit(E, np, s);
        RTDL_CUDA_CHECK(cudaStreamWaitEvent(s, ev_join, 0));
        k_emit_fixup<<<list_grid(np), kFixupThreads, 0, s>>>(E);
        RTDL_LAUNCHED(2);
      }
      if (stats)
        RTDL_CUDA_CHECK(cudaMemcpyAsync(last_stats().data(), C.stats, sizeof(unsigned long long) * kStatCount,
                                        cudaMemcpyDeviceToHost, s));
    }
    if (timer) timer->mark("traverse");
    Readback* rb = pinned_readback();
    SmallReads reads(rb);
    reads.add(&rb->scene_bad, &sc->stats->bad, sizeof(unsigned int));
    reads.add(&rb->query_bad, &qp.qst->bad, sizeof(unsigned int));
    reads.launch(s);
    RTDL_CUDA_CHECK(cudaStreamSynchronize(s));
    throw_if_bad(rb->scene_bad | rb->query_bad);
  } catch (...) {
    sync_quietly(s);
    sync_quietly(aux_stream());  // the list kernels may run there
    if (rows_alloc && *rows_alloc) {
      dev_free(*rows_alloc, s);
      *rows_alloc = nullptr;
    }
    cleanup();
    throw;
  }
  cleanup();
  return res;
}

}  // namespace

QueryResult run_query(Scene* sc, const void* queries_dev, uint32_t nq, int predicate, double radius, uint32_t limit,
                      void* rows_dev, size_t rows_capacity, void** rows_alloc, uint8_t* overflow_dev, cudaStream_t s,
                      PhaseTimer* timer) {
  QueryResult res;
  if (rows_alloc) *rows_alloc = nullptr;
  if (sc->problems) throw std::runtime_error("a problem batch is queried with the batch entry points");
  const int qstride = sc->dim == 3 ? 4 : 3;
  if (nq == 0) return res;
  if (sc->n == 0) {
    if (overflow_dev) RTDL_CUDA_CHECK(cudaMemsetAsync(overflow_dev, 0, nq, s));
    return res;
  }
  if (timer) timer->mark("start");
  if (predicate != kKnn)
    return run_radius_query(sc, queries_dev, nq, predicate, radius, limit, rows_dev, rows_capacity, rows_alloc,
                            overflow_dev, s, timer);
  if (limit <= (uint32_t)kMaxList)
    return run_knn(sc, queries_dev, nq, limit, rows_dev, rows_capacity, rows_alloc, overflow_dev, s, timer);
  // k > 64: every query takes the generic path over the whole scene
  QueryPrep qp = prepare_queries(sc, queries_dev, nq, false, radius, true, s);
  if (timer) timer->mark("query_prep");
  uint32_t* counts = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * nq, s));
  uint8_t* flags = static_cast<uint8_t*>(dev_alloc(nq, s));
  uint32_t* temp = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * (size_t)nq, s));
  uint32_t* heavy_list = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * nq, s));
  uint32_t* heavy_m = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * nq, s));
  unsigned int* small = static_cast<unsigned int*>(dev_alloc(sizeof(unsigned int) * 4, s));  // heavy count, error
  unsigned long long* offsets = static_cast<unsigned long long*>(dev_alloc(sizeof(unsigned long long) * (nq + 1), s));
  RTDL_CUDA_CHECK(cudaMemsetAsync(small, 0, sizeof(unsigned int) * 4, s));
  GenericOut g;
  auto cleanup = [&]() {
    g.release(s);
    dev_free(counts, s);
    dev_free(flags, s);
    dev_free(temp, s);
    dev_free(heavy_list, s);
    dev_free(heavy_m, s);
    dev_free(small, s);
    dev_free(offsets, s);
    free_prep(qp, s);
  };
  try {
    k_mark_all_heavy<<<grid_for(nq, 256), 256, 0, s>>>(qp.qorder, nq, sc->n, limit, counts, flags, temp, heavy_list,
                                                       heavy_m);
    RTDL_LAUNCHED(1);
    if (timer) timer->mark("traverse");
    scan_counts_u64(counts, qp.oorder, &qp.bands->ids_sorted, nq, offsets, s);
    if (timer) timer->mark("scan");

    Readback* rb = pinned_readback();
    SmallReads reads(rb);
    reads.add(&rb->rows, offsets + nq, sizeof(unsigned long long));
    reads.add(&rb->scene_bad, &sc->stats->bad, sizeof(unsigned int));
    reads.add(&rb->query_bad, &qp.qst->bad, sizeof(unsigned int));
    reads.launch(s);
    RTDL_CUDA_CHECK(cudaStreamSynchronize(s));
    throw_if_bad(rb->scene_bad | rb->query_bad);
    res.rows = rb->rows;
    res.heavy = nq;
    g = run_generic_path(sc, qp, queries_dev, qstride, nq, heavy_list, heavy_m, limit, true, small + 1, s);
    if (timer) timer->mark("generic_path");
    if (rows_alloc != nullptr) {
      rows_dev = res.rows ? dev_alloc(sizeof(RtdlKnnNeighborRow) * res.rows, s) : nullptr;
      rows_capacity = res.rows;
      *rows_alloc = rows_dev;
    }
    if (res.rows > 0 || overflow_dev != nullptr) {
      ExpandParams E;
      E.S = sc->view();
      E.qpts = qp.qpts;
      E.qraw = static_cast<const double*>(queries_dev);
      E.qstride = qstride;
      E.oorder = qp.oorder;
      E.bands = qp.bands;
      E.nq = nq;
      E.L = 1;
      E.counts = counts;
      E.flags = flags;
      E.temp = temp;
      E.heavy_out = g.heavy_out;
      E.heavy_out_off = g.heavy_out_off;
      E.offsets = offsets;
      E.rows = rows_dev;
      E.capacity = rows_dev ? rows_capacity : 0;
      E.ranked = 1;
      E.overflow_out = overflow_dev;
      E.error = small + 1;
      E.work_list = nullptr;
      E.qrank = nullptr;
      k_expand<<<grid_for((uint64_t)nq * 32, kExpandThreads), kExpandThreads, 0, s>>>(E);
      RTDL_LAUNCHED(1);
    }
    if (timer) timer->mark("emit");
    RTDL_CUDA_CHECK(cudaMemcpyAsync(&rb->error, small + 1, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
    RTDL_CUDA_CHECK(cudaStreamSynchronize(s));
    if (rb->error & 6u) throw std::runtime_error("generic neighbor path produced an inconsistent candidate count");
  } catch (...) {
    sync_quietly(s);
    cleanup();
    throw;
  }
  cleanup();
  return res;
}

HausdorffResult run_directed_hausdorff(Scene* sc, const void* queries_dev, uint32_t nq, double* nearest_dist_dev,
                                       uint32_t* nearest_id_dev, cudaStream_t s, PhaseTimer* timer) {
  if (sc->problems) throw std::runtime_error("a problem batch is queried with the batch entry points");
  if (nq == 0 || sc->n == 0) throw std::runtime_error("Hausdorff distance requires non-empty point sets");
  const int qstride = sc->dim == 3 ? 4 : 3;
  if (timer) timer->mark("start");
  QueryPrep qp = prepare_queries(sc, queries_dev, nq, false, 0.0, false, s);
  if (timer) timer->mark("query_prep");
  uint32_t* temp = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * nq, s));
  const unsigned int blocks = grid_for(nq, 256) < 8 * kSmCount ? grid_for(nq, 256) : 8 * kSmCount;
  Witness* partial = static_cast<Witness*>(dev_alloc(sizeof(Witness) * blocks, s));
  Witness* best = static_cast<Witness*>(dev_alloc(sizeof(Witness), s));
  NearestParams P;
  P.S = sc->view();
  P.qpts = qp.qpts;
  P.qraw = static_cast<const double*>(queries_dev);
  P.qstride = qstride;
  P.qorder = qp.qorder;
  P.qcodes = qp.qcodes;
  P.scodes = sc->codes;
  P.nq = nq;
  P.bands = qp.bands;
  P.nearest = temp;
  if (nearest_alone(nq, sc->n, sc->dim)) {
    SingleParams H{};
    H.S = P.S;
    H.qpts = P.qpts;
    H.qraw = P.qraw;
    H.qstride = qstride;
    H.bands = P.bands;
    H.k = 1;
    H.nwork = nq;
    H.qorder = P.qorder;
    H.qcodes = P.qcodes;
    H.scodes = P.scodes;
    H.nearest = temp;
    k_knn_single<false><<<div_up(nq, 256 / 32), 256, 0, s>>>(H);
  } else if (sc->dim == 3)
    k_nearest<3><<<div_up(nq, 128), 128, 0, s>>>(P);
  else
    k_nearest<2><<<div_up(nq, 128), 128, 0, s>>>(P);
  RTDL_LAUNCHED(1);
  if (timer) timer->mark("traverse");
  k_nearest_reduce<<<blocks, 256, 0, s>>>(sc->view(), qp.qpts, static_cast<const double*>(queries_dev), qstride, nq,
                                          temp, nearest_dist_dev, nearest_id_dev, partial);
  k_witness_best<<<1, 256, 0, s>>>(partial, blocks, best);
  RTDL_LAUNCHED(2);
  // one read of the witness (into the record's row-range words) and the error words
  Readback* rb = pinned_readback();
  static_assert(sizeof(Witness) <= sizeof(rb->chunk_rows), "readback record too small for the witness");
  SmallReads reads(rb);
  reads.add(rb->chunk_rows, best, sizeof(Witness));
  reads.add(&rb->scene_bad, &sc->stats->bad, sizeof(unsigned int));
  reads.add(&rb->query_bad, &qp.qst->bad, sizeof(unsigned int));
  reads.launch(s);
  RTDL_CUDA_CHECK(cudaStreamSynchronize(s));
  Witness w;
  memcpy(&w, rb->chunk_rows, sizeof(Witness));
  const unsigned int bad = rb->scene_bad | rb->query_bad;
  if (timer) timer->mark("reduce");
  dev_free(temp, s);
  dev_free(partial, s);
  dev_free(best, s);
  free_prep(qp, s);
  throw_if_bad(bad);
  HausdorffResult out;
  unsigned long long db = w.dist;
  memcpy(&out.distance, &db, sizeof(double));
  out.source_id = w.qid;
  out.target_id = w.nid;
  return out;
}


// ---- allocation-free directed Hausdorff ------------------------------------
// Some callers cannot allocate device memory while they run this query: an
// application that hands the whole device heap to its own allocator, code
// running between the capture points of a larger CUDA graph it does not own,
// or a real-time loop where an allocation could stall.  For them
// rtdl_b200_scene_directed_hausdorff_noalloc takes every scratch buffer of
// the nearest pass and of the max-witness reduction from this file-scope
// device array instead of the stream-ordered allocator.  Every GPU that loads
// the library holds the array until the process exits.
namespace {

constexpr uint32_t kNoAllocMaxQueries = 1u << 18;  // 262,144 queries per call
constexpr unsigned int kNoAllocReduceBlocks = 2 * kSmCount;

constexpr size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

struct NoAllocLayout {  // byte offsets into the scratch array, 256-B aligned
  static constexpr size_t kStats = 0;
  static constexpr size_t kBands = align256(kStats + sizeof(PointStats));
  static constexpr size_t kBest = align256(kBands + sizeof(DevBands));
  static constexpr size_t kPartial = align256(kBest + sizeof(Witness));
  static constexpr size_t kQpts = align256(kPartial + kNoAllocReduceBlocks * sizeof(Witness));
  static constexpr size_t kTemp = align256(kQpts + (size_t)kNoAllocMaxQueries * sizeof(float4));
  static constexpr size_t kCodes = align256(kTemp + (size_t)kNoAllocMaxQueries * sizeof(uint32_t));
  static constexpr size_t kTotal = align256(kCodes + (size_t)kNoAllocMaxQueries * sizeof(uint32_t));
};

// 9.75 MiB: scratch for up to kNoAllocMaxQueries queries.
static __device__ __align__(256) unsigned char g_noalloc_scratch[NoAllocLayout::kTotal];

// Converts the reduced witness into the public record and folds in the
// input checks, so the call never needs a host round trip.
__global__ void k_noalloc_finish(const Witness* best, const PointStats* scene_stats, const PointStats* query_stats,
                                 RtdlB200Witness* out) {
  if (threadIdx.x != 0) return;
  RtdlB200Witness w;
  unsigned long long db = best->dist;
  w.distance = __longlong_as_double((long long)db);
  w.source_id = best->qid;
  w.target_id = best->nid;
  const unsigned int bad = scene_stats->bad | query_stats->bad;
  w.status = (bad & kBadSortWait) ? 3u : bad ? 1u : 0u;
  w.reserved = 0u;
  *out = w;
}

unsigned char* noalloc_scratch_for_current_device() {
  static std::mutex m;
  static std::vector<unsigned char*> ptrs;
  int dev = 0;
  RTDL_CUDA_CHECK(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> g(m);
  if ((int)ptrs.size() <= dev) ptrs.resize(dev + 1, nullptr);
  if (ptrs[dev] == nullptr) {
    // The symbol name is a host-side stand-in; the device address comes from
    // the runtime, per device, with that device current.
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess)
      throw std::runtime_error(std::string("cudaGetSymbolAddress of the scratch array failed: ") +
                               cudaGetErrorString(e));
    ptrs[dev] = static_cast<unsigned char*>(p);
  }
  return ptrs[dev];
}

}  // namespace

void run_directed_hausdorff_noalloc(Scene* sc, const void* queries_dev, uint32_t nq, double* nearest_dist_dev,
                                    uint32_t* nearest_id_dev, RtdlB200Witness* witness_dev, cudaStream_t s) {
  if (sc->problems) throw std::runtime_error("a problem batch is queried with the batch entry points");
  if (nq == 0 || sc->n == 0) throw std::runtime_error("Hausdorff distance requires non-empty point sets");
  if (nq > kNoAllocMaxQueries)
    throw std::runtime_error("rtdl_b200_scene_directed_hausdorff_noalloc: query_count exceeds the limit of 262144 "
                             "queries set by its fixed scratch array");
  unsigned char* base = noalloc_scratch_for_current_device();
  PointStats* qst = reinterpret_cast<PointStats*>(base + NoAllocLayout::kStats);
  DevBands* bands = reinterpret_cast<DevBands*>(base + NoAllocLayout::kBands);
  Witness* best = reinterpret_cast<Witness*>(base + NoAllocLayout::kBest);
  Witness* partial = reinterpret_cast<Witness*>(base + NoAllocLayout::kPartial);
  float4* qpts = reinterpret_cast<float4*>(base + NoAllocLayout::kQpts);
  uint32_t* temp = reinterpret_cast<uint32_t*>(base + NoAllocLayout::kTemp);
  uint32_t* codes = reinterpret_cast<uint32_t*>(base + NoAllocLayout::kCodes);
  // The array keeps the previous call's contents: reset what must start at zero.
  reset_stats(qst, s);
  prep_points(queries_dev, nq, sc->dim, qpts, qst, s);
  k_bands<<<1, 32, 0, s>>>(sc->stats, qst, 0.0, 0, bands);
  RTDL_LAUNCHED(1);
  curve_codes(qpts, nq, sc->dim, sc->stats, codes, nullptr, s);  // input order (no sort, hence no sort scratch)
  SingleParams P{};
  P.S = sc->view();
  P.qpts = qpts;
  P.qraw = static_cast<const double*>(queries_dev);
  P.qstride = sc->dim == 3 ? 4 : 3;
  P.bands = bands;
  P.k = 1;
  P.nwork = nq;
  P.qcodes = codes;
  P.scodes = sc->codes;
  P.nearest = temp;
  k_knn_single<false><<<grid_for((uint64_t)nq * 32, 256), 256, 0, s>>>(P);
  RTDL_LAUNCHED(1);
  const unsigned int blocks = grid_for(nq, 256) < kNoAllocReduceBlocks ? grid_for(nq, 256) : kNoAllocReduceBlocks;
  k_nearest_reduce<<<blocks, 256, 0, s>>>(sc->view(), qpts, static_cast<const double*>(queries_dev), P.qstride, nq,
                                          temp, nearest_dist_dev, nearest_id_dev, partial);
  k_witness_best<<<1, 256, 0, s>>>(partial, blocks, best);
  k_noalloc_finish<<<1, 32, 0, s>>>(best, sc->stats, qst, witness_dev);
  RTDL_LAUNCHED(3);
}


// ---- captured graphs over prepared problem batches --------------------------
// Many uneven fixed-radius problems, already built into problem batches
// (build_scene_batch: each problem a tree of its own), answered
// by one CUDA graph replay with no host read-back inside.  Per batch the graph
// holds ONE persistent collect launch -- a grid that fills the GPU once, whose
// warps take packets of 32, 16 or 8 queries (one problem each) from a device
// work queue until the batch's packets are gone, so small and large problems
// share the SMs -- then the queries the packets left, the scan (rows of this
// batch start where the previous batch's end) and the emit kernels striding over
// device list lengths.  Batches run one after another in the graph and share
// one set of scratch buffers sized for the largest.  A batch whose heavy
// queries the narrowing inside the collect does not resolve is flagged in its
// status word and recomputed by the plain batch call at replay, so rows always
// equal it.
namespace {

__global__ void k_add_row_base(unsigned long long* offsets, uint32_t n, const unsigned long long* base,
                               unsigned long long* next_base) {
  const unsigned long long b = *base;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= n; i += gridDim.x * blockDim.x) {
    const unsigned long long v = offsets[i] + b;
    offsets[i] = v;
    if (i == n) *next_base = v;
  }
}

__global__ void k_empty_batch_rows(const unsigned long long* base, uint32_t problems, unsigned long long* prob_rows,
                                   unsigned long long* next_base) {
  const unsigned long long b = *base;
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p <= problems; p += gridDim.x * blockDim.x) prob_rows[p] = b;
  if (blockIdx.x == 0 && threadIdx.x == 0) *next_base = b;
}

// Persistent collect over one batch: packets from a work queue.
template <int DIM>
__global__ void __launch_bounds__(kCollectThreads, 6) k_collect_persistent(const __grid_constant__ CollectParams P, unsigned int* queue) {
  __shared__ CollectWarp warps[kCollectThreads / 32];
  const uint32_t packets = (P.nq + P.width - 1u) / P.width;
  const uint32_t lane = threadIdx.x & 31u;
  for (;;) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(queue, 1u);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= packets) return;
    collect_packet_body<DIM, true, false>(P, item * P.width + lane, warps[threadIdx.x >> 5]);
  }
}

__global__ void k_batch_graph_status(const unsigned int* small, uint32_t batches, const unsigned long long* total, unsigned long long capacity,
                                     unsigned int* status) {
  for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < batches; b += gridDim.x * blockDim.x)
    status[b] = (small[8 * (size_t)b] ? kGraphStatusGeneric : 0u) |
                (*total > capacity ? kBatchGraphStatusRows : 0u);
}

}  // namespace

struct BatchGraphPart {  // one prepared problem batch
  Scene* sc = nullptr;                        // borrowed
  const void* queries = nullptr;              // the caller's records of this batch's problems
  uint32_t p0 = 0, problems = 0;              // global problem range
  uint32_t nq = 0;
  std::vector<unsigned long long> qoff;       // problems + 1, local
  std::vector<double> radius;
  std::vector<uint32_t> kmax;
  QueryPrep qp;
  uint32_t* qrank = nullptr;
  unsigned long long* offsets = nullptr;      // nq + 1, global row offsets once the base is added
};

struct BatchGraph {
  std::vector<BatchGraphPart> parts;
  int device = 0;
  cudaStream_t stream = nullptr;
  uint32_t problems = 0;
  void* rows = nullptr;                       // the caller's
  unsigned long long capacity = 0;
  std::vector<void*> buffers;
  // scratch shared by the batches (sized for the largest)
  uint32_t* slab = nullptr;
  uint32_t* counts = nullptr;
  QueryInfo* qinfo = nullptr;
  uint8_t* flags = nullptr;
  uint32_t *heavy_list = nullptr, *heavy_m = nullptr, *heavy_t = nullptr;
  double* heavy_rad = nullptr;
  uint32_t* single_list = nullptr;
  uint32_t *mid_list = nullptr, *big_list = nullptr, *fix_list = nullptr;
  unsigned long long* poff = nullptr;
  void* scan_ws = nullptr;
  // per batch
  unsigned int* small = nullptr;        // 8 counters per batch
  unsigned int* queue = nullptr;        // work-queue counter per batch
  unsigned long long* base = nullptr;   // batches + 1: first row of each batch, then the total
  unsigned long long* prob_rows = nullptr;  // problems + 1: first row of each problem, then the total
  unsigned int* status = nullptr;
  unsigned int* status_host = nullptr;      // pinned
  unsigned long long* rows_host = nullptr;  // pinned, problems + 1
  unsigned int persistent_grid = 0;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int kernels = 0;
  uint64_t fallbacks = 0;
};

namespace {

void batch_graph_enqueue(BatchGraph* g, uint32_t i, cudaStream_t s) {
  BatchGraphPart& b = g->parts[i];
  unsigned int* small = g->small + 8 * (size_t)i;
  if (b.nq == 0) {  // no queries in this batch: its problems get no rows
    k_empty_batch_rows<<<div_up(b.problems + 1, 256), 256, 0, s>>>(g->base + i, b.problems, g->prob_rows + b.p0,
                                                                  g->base + i + 1);
    RTDL_LAUNCHED(1);
    return;
  }
  uint32_t kmax = 1;
  for (uint32_t k : b.kmax) kmax = k > kmax ? k : kmax;
  CollectParams C;
  C.S = b.qp.view;
  C.qpts = b.qp.qpts;
  C.qraw = static_cast<const double*>(b.queries);
  C.qstride = b.sc->dim == 3 ? 4 : 3;
  C.qorder = b.qp.qorder;
  C.nq = b.qp.nproc;
  C.kmax = kmax;
  C.width = packet_width(b.qp.nproc, true);
  C.radius = 0.0;
  C.bands = b.qp.bands;
  C.warp_prob = b.qp.warp_prob;
  C.prob_kmax = b.qp.prob_kmax;
  C.prob_radius = b.qp.prob_radius;
  C.slab = g->slab;
  C.counts = g->counts;
  C.qinfo = g->qinfo;
  C.flags = g->flags;
  C.heavy_list = g->heavy_list;
  C.heavy_m = g->heavy_m;
  C.heavy_rad = g->heavy_rad;
  C.heavy_t = g->heavy_t;
  C.mid_list = g->mid_list;
  C.big_list = g->big_list;
  C.single_list = g->single_list;
  C.small = small;
  C.overflow_out = nullptr;
  C.rank_radius = nullptr;
  C.stats = nullptr;
  const uint32_t np = b.qp.nproc;
  if (b.sc->dim == 3)
    k_collect_persistent<3><<<g->persistent_grid, kCollectThreads, 0, s>>>(C, g->queue + i);
  else
    k_collect_persistent<2><<<g->persistent_grid, kCollectThreads, 0, s>>>(C, g->queue + i);
  launch_collect_left(C, b.qp.nproc, s);
  RTDL_LAUNCHED(1);
  scan_counts_u64_ws(g->counts, b.qp.oorder, b.qp.order_identity, b.nq, b.offsets, g->scan_ws, s);
  k_add_row_base<<<grid_for(b.nq + 1, 256), 256, 0, s>>>(b.offsets, b.nq, g->base + i, g->base + i + 1);
  k_problem_rows<<<div_up(b.problems + 1, 256), 256, 0, s>>>(b.offsets, b.qp.qoff, b.problems, g->prob_rows + b.p0);
  RTDL_LAUNCHED(2);
  k_proc_offsets<<<grid_for(np, 256), 256, 0, s>>>(b.qp.qorder, b.qrank, b.offsets, np, g->poff);
  RTDL_LAUNCHED(1);
  EmitParams E;
  E.S = b.sc->view();
  E.nq = np;
  E.slab = g->slab;
  E.qinfo = g->qinfo;
  E.poff = g->poff;
  E.sink.rows = g->rows;
  E.sink.capacity = g->rows ? g->capacity : 0;
  E.sink.ranked = 0;
  E.fix_list = g->fix_list;
  E.fix_count = small + 4;
  launch_emit(E, np, s);
  launch_emit_lists(E, C, np, s);
  k_emit_fixup<<<list_grid(np), kFixupThreads, 0, s>>>(E);
  RTDL_LAUNCHED(1);
}

void batch_graph_release(BatchGraph* g) {
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  g->exec = nullptr;
  g->graph = nullptr;
}

void batch_graph_capture(BatchGraph* g) {
  batch_graph_release(g);
  cudaStream_t s = g->stream;
  const uint32_t B = (uint32_t)g->parts.size();
  const unsigned long long before = launches_counted();
  RTDL_CUDA_CHECK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  try {
    RTDL_CUDA_CHECK(cudaMemsetAsync(g->small, 0, sizeof(unsigned int) * 8 * (size_t)B, s));
    RTDL_CUDA_CHECK(cudaMemsetAsync(g->queue, 0, sizeof(unsigned int) * B, s));
    RTDL_CUDA_CHECK(cudaMemsetAsync(g->base, 0, sizeof(unsigned long long), s));
    for (uint32_t i = 0; i < B; ++i) batch_graph_enqueue(g, i, s);
    k_batch_graph_status<<<div_up(B, 256), 256, 0, s>>>(g->small, B, g->base + B, g->capacity,
                                                        g->status);
    RTDL_LAUNCHED(1);
  } catch (...) {
    cudaGraph_t partial = nullptr;
    cudaStreamEndCapture(s, &partial);
    if (partial) cudaGraphDestroy(partial);
    cudaGetLastError();
    count_launches(-(int)(launches_counted() - before));
    throw;
  }
  count_launches(-(int)(launches_counted() - before));  // counted when a replay launches them
  RTDL_CUDA_CHECK(cudaStreamEndCapture(s, &g->graph));
  RTDL_CUDA_CHECK(cudaGraphInstantiate(&g->exec, g->graph, 0));
  size_t n = 0;
  RTDL_CUDA_CHECK(cudaGraphGetNodes(g->graph, nullptr, &n));
  std::vector<cudaGraphNode_t> nodes(n);
  RTDL_CUDA_CHECK(cudaGraphGetNodes(g->graph, nodes.data(), &n));
  g->kernels = 0;
  for (size_t i = 0; i < n; ++i) {
    cudaGraphNodeType t;
    RTDL_CUDA_CHECK(cudaGraphNodeGetType(nodes[i], &t));
    if (t == cudaGraphNodeTypeKernel) ++g->kernels;
  }
}

}  // namespace

BatchGraph* batch_graph_create(Scene* const* batches, uint32_t batch_count, const void* queries_dev,
                               const unsigned long long* query_offsets, const double* radius, const uint32_t* kmax,
                               void* rows_dev, unsigned long long rows_capacity) {
  if (batch_count == 0) throw std::runtime_error("a batch graph needs at least one problem batch");
  if (!batches || !query_offsets || !radius || !kmax)
    throw std::runtime_error("batches, query_offsets, radius and k_max must not be null");
  for (uint32_t i = 0; i < batch_count; ++i) {
    if (!batches[i] || batches[i]->problems == 0)
      throw std::runtime_error("batch graph inputs must be problem batch handles");
    if (batches[i]->dim != batches[0]->dim) throw std::runtime_error("problem batches of a graph must share a dimension");
  }
  BatchGraph* g = new BatchGraph();
  try {
    RTDL_CUDA_CHECK(cudaGetDevice(&g->device));
    RTDL_CUDA_CHECK(cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking));
    cudaStream_t s = g->stream;
    g->rows = rows_dev;
    g->capacity = rows_dev ? rows_capacity : 0;
    uint32_t p0 = 0, most_np = 0, most_nq = 0;
    const size_t rec = batches[0]->dim == 2 ? sizeof(RtdlPoint) : sizeof(RtdlPoint3D);
    g->parts.reserve(batch_count);
    for (uint32_t i = 0; i < batch_count; ++i) {
      Scene* sc = batches[i];
      RTDL_CUDA_CHECK(cudaStreamSynchronize(sc->stream));  // built on its own stream
      g->parts.emplace_back();
      BatchGraphPart& b = g->parts.back();
      b.sc = sc;
      b.p0 = p0;
      b.problems = sc->problems;
      const unsigned long long q0 = query_offsets[p0], q1 = query_offsets[p0 + sc->problems];
      if (q1 < q0 || q1 - q0 > 0xFFFFFFFFull - 32) throw std::runtime_error("query offsets must be non-decreasing");
      b.nq = (uint32_t)(q1 - q0);
      if (b.nq > 0 && !queries_dev) throw std::runtime_error("query_points_dev must not be null when queries exist");
      b.queries = static_cast<const char*>(queries_dev) + q0 * rec;
      b.qoff.resize(sc->problems + 1);
      for (uint32_t p = 0; p <= sc->problems; ++p) b.qoff[p] = query_offsets[p0 + p] - q0;
      b.radius.assign(radius + p0, radius + p0 + sc->problems);
      b.kmax.assign(kmax + p0, kmax + p0 + sc->problems);
      for (uint32_t p = 0; p < sc->problems; ++p) {
        if (b.qoff[p + 1] < b.qoff[p]) throw std::runtime_error("query offsets must be non-decreasing");
        if (!(b.radius[p] >= 0.0)) throw std::runtime_error("radius must be non-negative");
        if (b.kmax[p] < 1 || b.kmax[p] > 64) throw std::runtime_error("a problem batch takes k_max in [1, 64]");
      }
      if (b.nq > 0) {
        BatchSpec bs;
        bs.problems = sc->problems;
        bs.qoff = b.qoff.data();
        bs.radius = b.radius.data();
        bs.kmax = b.kmax.data();
        b.qp = prepare_queries_batch(sc, b.queries, b.nq, bs, s);
        b.qrank = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * b.nq, s));
        k_invert<<<grid_for(b.nq, 256), 256, 0, s>>>(b.qp.oorder, b.nq, b.qp.order_identity, b.qrank);
        RTDL_LAUNCHED(1);
      }
      b.offsets = static_cast<unsigned long long*>(dev_alloc(sizeof(unsigned long long) * ((size_t)b.nq + 1), s));
      RTDL_CUDA_CHECK(cudaMemsetAsync(b.offsets, 0, sizeof(unsigned long long) * ((size_t)b.nq + 1), s));
      most_np = b.qp.nproc > most_np ? b.qp.nproc : most_np;
      most_nq = b.nq > most_nq ? b.nq : most_nq;
      p0 += sc->problems;
    }
    g->problems = p0;
    const size_t n = most_np ? most_np : 1, nqm = most_nq ? most_nq : 1, B = batch_count;
    auto alloc = [&](size_t bytes) {
      void* p = dev_alloc(bytes ? bytes : 1, s);
      g->buffers.push_back(p);
      return p;
    };
    g->slab = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * slab_base((uint32_t)n)));
    g->counts = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * nqm));
    g->qinfo = static_cast<QueryInfo*>(alloc(sizeof(QueryInfo) * n));
    g->flags = static_cast<uint8_t*>(alloc(nqm));
    g->heavy_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * nqm));
    g->heavy_m = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * nqm));
    g->heavy_t = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * nqm));
    g->mid_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * n));
    g->big_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * n));
    g->fix_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * n));
    g->poff = static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * n));
    g->scan_ws = alloc(scan_workspace_bytes((uint32_t)nqm));
    g->heavy_rad = static_cast<double*>(alloc(sizeof(double) * nqm));
    g->single_list = static_cast<uint32_t*>(alloc(sizeof(uint32_t) * n));
    g->small = static_cast<unsigned int*>(alloc(sizeof(unsigned int) * 8 * B));
    g->queue = static_cast<unsigned int*>(alloc(sizeof(unsigned int) * B));
    g->base = static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * (B + 1)));
    g->prob_rows = static_cast<unsigned long long*>(alloc(sizeof(unsigned long long) * ((size_t)g->problems + 1)));
    g->status = static_cast<unsigned int*>(alloc(sizeof(unsigned int) * B));
    RTDL_CUDA_CHECK(cudaMemsetAsync(g->prob_rows, 0, sizeof(unsigned long long) * ((size_t)g->problems + 1), s));
    RTDL_CUDA_CHECK(cudaMallocHost(&g->status_host, sizeof(unsigned int) * B));
    RTDL_CUDA_CHECK(cudaMallocHost(&g->rows_host, sizeof(unsigned long long) * ((size_t)g->problems + 1)));
    int per_sm = 0;
    if (batches[0]->dim == 3)
      RTDL_CUDA_CHECK(
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_collect_persistent<3>, kCollectThreads, 0));
    else
      RTDL_CUDA_CHECK(
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_collect_persistent<2>, kCollectThreads, 0));
    int sms = kSmCount;
    RTDL_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device));
    g->persistent_grid = (unsigned int)(sms * (per_sm > 0 ? per_sm : 1));
    // bad coordinates or a failed sort wait in a batch or its queries fail creation
    Readback* rb = pinned_readback();
    for (auto& b : g->parts) {
      RTDL_CUDA_CHECK(cudaMemcpyAsync(&rb->scene_bad, &b.sc->stats->bad, sizeof(unsigned int), cudaMemcpyDeviceToHost,
                                      s));
      rb->query_bad = 0;
      if (b.qp.qst)
        RTDL_CUDA_CHECK(cudaMemcpyAsync(&rb->query_bad, &b.qp.qst->bad, sizeof(unsigned int), cudaMemcpyDeviceToHost,
                                        s));
      RTDL_CUDA_CHECK(cudaStreamSynchronize(s));
      throw_if_bad(rb->query_bad | rb->scene_bad);
    }
    RTDL_CUDA_CHECK(cudaStreamSynchronize(s));  // everything allocated and prepared before capture
    batch_graph_capture(g);
  } catch (...) {
    batch_graph_destroy(g);
    throw;
  }
  return g;
}

void batch_graph_launch(BatchGraph* g, cudaStream_t s) {
  count_launches(g->kernels);
  if (s && s != g->stream) {
    cudaEvent_t e;
    RTDL_CUDA_CHECK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    RTDL_CUDA_CHECK(cudaEventRecord(e, s));
    RTDL_CUDA_CHECK(cudaStreamWaitEvent(g->stream, e, 0));
    RTDL_CUDA_CHECK(cudaGraphLaunch(g->exec, g->stream));
    RTDL_CUDA_CHECK(cudaEventRecord(e, g->stream));
    RTDL_CUDA_CHECK(cudaStreamWaitEvent(s, e, 0));
    note_cleanup_error(cudaEventDestroy(e), "cudaEventDestroy");
  } else {
    RTDL_CUDA_CHECK(cudaGraphLaunch(g->exec, g->stream));
  }
}

void batch_graph_replay(BatchGraph* g, unsigned long long* row_offsets_out, unsigned int* status_out) {
  batch_graph_launch(g, nullptr);
  cudaStream_t s = g->stream;
  const uint32_t B = (uint32_t)g->parts.size();
  RTDL_CUDA_CHECK(cudaMemcpyAsync(g->status_host, g->status, sizeof(unsigned int) * B, cudaMemcpyDeviceToHost, s));
  RTDL_CUDA_CHECK(cudaMemcpyAsync(g->rows_host, g->prob_rows, sizeof(unsigned long long) * ((size_t)g->problems + 1),
                                  cudaMemcpyDeviceToHost, s));
  RTDL_CUDA_CHECK(cudaStreamSynchronize(s));
  unsigned int all = 0;
  for (uint32_t i = 0; i < B; ++i) {
    const unsigned int st = g->status_host[i];
    all |= st;
    if ((st & kGraphStatusGeneric) && g->rows && !(st & kBatchGraphStatusRows)) {
      // heavy queries the refinement did not resolve: this batch's rows by the plain batch call
      BatchGraphPart& b = g->parts[i];
      const unsigned long long first = g->rows_host[b.p0];
      std::vector<unsigned long long> local(b.problems + 1);
      BatchSpec bs;
      bs.problems = b.problems;
      bs.qoff = b.qoff.data();
      bs.radius = b.radius.data();
      bs.kmax = b.kmax.data();
      bs.row_offsets = local.data();
      run_query_batch(b.sc, b.queries, bs, static_cast<char*>(g->rows) + first * sizeof(RtdlFixedRadiusNeighborRow),
                      g->capacity - first, nullptr, nullptr, s, nullptr);
      RTDL_CUDA_CHECK(cudaStreamSynchronize(s));
      ++g->fallbacks;
    }
  }
  if (status_out) *status_out = all;
  if (row_offsets_out)
    std::memcpy(row_offsets_out, g->rows_host, sizeof(unsigned long long) * ((size_t)g->problems + 1));
}

uint32_t batch_graph_problems(const BatchGraph* g) { return g->problems; }
int batch_graph_kernels(const BatchGraph* g) { return g->kernels; }
uint64_t batch_graph_fallbacks(const BatchGraph* g) { return g->fallbacks; }

void batch_graph_destroy(BatchGraph* g) {
  if (!g) return;
  if (g->stream) sync_quietly(g->stream);
  batch_graph_release(g);
  cudaStream_t s = g->stream;
  for (auto& b : g->parts) {
    if (b.nq > 0) free_prep(b.qp, s);
    dev_free(b.qrank, s);
    dev_free(b.offsets, s);
  }
  for (void* p : g->buffers) dev_free(p, s);
  if (g->status_host) note_cleanup_error(cudaFreeHost(g->status_host), "cudaFreeHost");
  if (g->rows_host) note_cleanup_error(cudaFreeHost(g->rows_host), "cudaFreeHost");
  if (s) {
    sync_quietly(s);
    note_cleanup_error(cudaStreamDestroy(s), "cudaStreamDestroy");
  }
  delete g;
}

}  // namespace rtdl_b200
