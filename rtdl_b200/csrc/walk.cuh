// walk.cuh -- the warp walk of the wide tree and the bucket test.
#pragma once

#include <cfloat>

#include "internal.cuh"

namespace rtdl_b200 {
namespace {

// Two FP32 values in one 64-bit register pair: Blackwell's packed add and fma
// take half the instructions of the scalar forms.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float v) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// A lane's side of the bucket test: minus its query's coordinates and minus
// the squared distance the points are compared with, each twice.
struct BucketQuery {
  f32x2 nx, ny, nz, nd;
  __device__ __forceinline__ void set(float x, float y, float z, float d2) {
    nx = pack2(-x);
    ny = pack2(-y);
    nz = pack2(-z);
    nd = pack2(-d2);
  }
};

// Four buckets against the lane's query: bit 8 u + j of the result is set when
// point j of bucket u has an FP32 squared distance below the compared value
// (the signs of d2 - value, shifted in).  BAND: *near receives the smallest of
// the differences' bits as signed integers, which is 0x80000000 + the smallest
// magnitude among the negative ones: one three-way minimum per two points tells
// the caller when a point lies just below the value.  The point loads are
// warp-uniform 16-byte loads, six (four in 2D) for eight points.
template <int DIM, bool BAND>
__device__ __forceinline__ uint32_t buckets_mask(const float4* __restrict__ bucket_pts, const uint4& four,
                                                 const BucketQuery& q, int* near) {
  uint32_t mask = 0;
  int least = 0x7fffffff;
#pragma unroll
  for (int u = 3; u >= 0; --u) {
    const uint32_t bucket = u == 0 ? four.x : u == 1 ? four.y : u == 2 ? four.z : four.w;
    const ulonglong2* c = reinterpret_cast<const ulonglong2*>(bucket_pts) + (size_t)bucket * (2 * DIM);
    f32x2 t[4];
#pragma unroll
    for (int a = 0; a < DIM; ++a) {
      const ulonglong2 lo = __ldg(c + 2 * a), hi = __ldg(c + 2 * a + 1);
      const f32x2 v[4] = {lo.x, lo.y, hi.x, hi.y};
      const f32x2 n = a == 0 ? q.nx : a == 1 ? q.ny : q.nz;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const f32x2 d = add2(v[k], n);
        t[k] = fma2(d, d, a == 0 ? q.nd : t[k]);
      }
    }
#pragma unroll
    for (int k = 3; k >= 0; --k) {
      float lo, hi;
      unpack2(t[k], lo, hi);
      mask = __funnelshift_l(__float_as_uint(hi), mask, 1);
      mask = __funnelshift_l(__float_as_uint(lo), mask, 1);
      if (BAND) least = __vimin3_s32(least, __float_as_int(lo), __float_as_int(hi));
    }
  }
  if (BAND) *near = least;
  return mask;
}

// The FP32 squared distances of a bucket's points to the lane's query (its
// compared value is not used); +inf for the points that fill a bucket up.
template <int DIM>
__device__ __forceinline__ void bucket_d2(const float4* __restrict__ bucket_pts, uint32_t bucket,
                                          const BucketQuery& q, float (&d2)[8]) {
  const ulonglong2* c = reinterpret_cast<const ulonglong2*>(bucket_pts) + (size_t)bucket * (2 * DIM);
  f32x2 t[4];
#pragma unroll
  for (int a = 0; a < DIM; ++a) {
    const ulonglong2 u = __ldg(c + 2 * a), w = __ldg(c + 2 * a + 1);
    const f32x2 v[4] = {u.x, u.y, w.x, w.y};
    const f32x2 n = a == 0 ? q.nx : a == 1 ? q.ny : q.nz;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const f32x2 d = add2(v[k], n);
      t[k] = a == 0 ? fma2(d, d, 0ull) : fma2(d, d, t[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) unpack2(t[k], d2[2 * k], d2[2 * k + 1]);
}

// Axis-aligned box of a warp's queries (lanes without a query take no part).
struct PacketBox {
  float lx, ly, lz, hx, hy, hz;
};
__device__ __forceinline__ PacketBox packet_box(const float4& q, bool valid) {
  const float inf = INFINITY;
  PacketBox b;
  b.lx = ordered_to_float(__reduce_min_sync(0xffffffffu, float_to_ordered(valid ? q.x : inf)));
  b.ly = ordered_to_float(__reduce_min_sync(0xffffffffu, float_to_ordered(valid ? q.y : inf)));
  b.lz = ordered_to_float(__reduce_min_sync(0xffffffffu, float_to_ordered(valid ? q.z : inf)));
  b.hx = ordered_to_float(__reduce_max_sync(0xffffffffu, float_to_ordered(valid ? q.x : -inf)));
  b.hy = ordered_to_float(__reduce_max_sync(0xffffffffu, float_to_ordered(valid ? q.y : -inf)));
  b.hz = ordered_to_float(__reduce_max_sync(0xffffffffu, float_to_ordered(valid ? q.z : -inf)));
  return b;
}

// The box around the lanes' spheres: each lane's cube of half-width h, rounded
// outward.
__device__ __forceinline__ PacketBox packet_reach_box(const float4& q, float h, bool valid) {
  const float inf = INFINITY;
  PacketBox b;
  b.lx = ordered_to_float(__reduce_min_sync(0xffffffffu, float_to_ordered(valid ? __fsub_rd(q.x, h) : inf)));
  b.ly = ordered_to_float(__reduce_min_sync(0xffffffffu, float_to_ordered(valid ? __fsub_rd(q.y, h) : inf)));
  b.lz = ordered_to_float(__reduce_min_sync(0xffffffffu, float_to_ordered(valid ? __fsub_rd(q.z, h) : inf)));
  b.hx = ordered_to_float(__reduce_max_sync(0xffffffffu, float_to_ordered(valid ? __fadd_ru(q.x, h) : -inf)));
  b.hy = ordered_to_float(__reduce_max_sync(0xffffffffu, float_to_ordered(valid ? __fadd_ru(q.y, h) : -inf)));
  b.hz = ordered_to_float(__reduce_max_sync(0xffffffffu, float_to_ordered(valid ? __fadd_ru(q.z, h) : -inf)));
  return b;
}

// Half-width of the cube around a sphere of squared radius r2, rounded up.
__device__ __forceinline__ float reach_half_width(float r2) { return __fmul_ru(__fsqrt_ru(r2), 1.000001f); }

__device__ __forceinline__ bool boxes_meet(const PacketBox& w, const float4& lo, const float4& hi) {
  return lo.x <= w.hx && hi.x >= w.lx && lo.y <= w.hy && hi.y >= w.ly && lo.z <= w.hz && hi.z >= w.lz;
}

// Squared distance of two boxes.
__device__ __forceinline__ float boxes_d2(const PacketBox& w, const float4& lo, const float4& hi) {
  const float dx = fmaxf(fmaxf(lo.x - w.hx, w.lx - hi.x), 0.f);
  const float dy = fmaxf(fmaxf(lo.y - w.hy, w.ly - hi.y), 0.f);
  const float dz = fmaxf(fmaxf(lo.z - w.hz, w.lz - hi.z), 0.f);
  return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
}

struct __align__(16) WalkStack {
  uint2 level[kTreeLevels];  // first node (within the level) and the children still to visit
};

// Depth-first walk of a wide tree by one warp: a node's children are tested
// in one step (a lane each) and entered in order.  visit(first, mask) gets
// the buckets [first, first + 32) of the tree whose bits are set in mask, all
// within sqrt(reach2) of the box; it returns true to end the walk.  `reach2` is
// read before every step, so a visitor may shrink it (warp-uniform).  With
// `limit` (lanes whose radii differ) a node must also meet that box: at KNN
// radii of k = 16 a packet then tests 167 buckets instead of 233.
// LEAF 1: the walk ends at the level-1 nodes, which visit() gets instead.
template <int LEAF = 0, typename Visit>
__device__ __forceinline__ void walk_wide(const SceneView& S, const TreeShape* __restrict__ T, const PacketBox& w,
                                          const PacketBox* limit, const float& reach2, WalkStack& stack, int lane,
                                          Visit&& visit) {
  const uint32_t buckets = __ldg(&T->buckets);
  if (buckets == 0) return;
  const uint32_t top = __ldg(&T->top);
  uint32_t l = top, first = 0;
  if (LEAF == 1 && top == 0) return;  // at most 32 buckets
  for (;;) {
    const uint32_t count = tree_level_nodes(buckets, l) - first;
    bool over = false;
    if ((uint32_t)lane < count) {
      const float4* node = S.wide + 2 * (size_t)(__ldg(&T->base[l]) + first + lane);
      const float4 lo = __ldg(node), hi = __ldg(node + 1);
      over = boxes_d2(w, lo, hi) <= reach2 && (limit == nullptr || boxes_meet(*limit, lo, hi));
    }
    const uint32_t mask = __ballot_sync(0xffffffffu, over);
    if (l == LEAF) {
      if (mask && visit(first, mask)) return;
    } else {
      if (lane == 0) stack.level[l] = make_uint2(first, mask);
      --l;  // so that the search for the next child starts at this level
    }
    // the next unvisited child on the way up
    uint2 e;
    __syncwarp();
    do {
      if (++l > top) return;
      e = stack.level[l];
    } while (e.y == 0u);
    __syncwarp();
    if (lane == 0) stack.level[l].y = e.y & (e.y - 1u);
    first = (e.x + (uint32_t)(__ffs((int)e.y) - 1)) * kFan;
    --l;
  }
}

// The walk for packets: the buckets are listed (a lane per child, no loop over
// the bits) and handed on in fours, four(ids) returning true to end the walk.
// The list is filled up at the end with the scene's empty bucket, which no
// query reaches.  Ids count from the first bucket of the scene.  `start` buckets
// are listed before any is handed on.
constexpr int kBucketList = 72;
template <typename Four>
__device__ __forceinline__ void walk_fours(const SceneView& S, const TreeShape* __restrict__ T, const PacketBox& w,
                                           const PacketBox* limit, const float& reach2, WalkStack& stack,
                                           uint32_t* list, int lane, uint32_t start, Four&& four) {
  const uint32_t bucket0 = __ldg(&T->base[0]);
  const uint32_t below = (1u << lane) - 1u;
  uint32_t n = 0;
  bool done = false;
  walk_wide(S, T, w, limit, reach2, stack, lane, [&](uint32_t first, uint32_t mask) {
    if ((mask >> lane) & 1u) list[n + __popc(mask & below)] = bucket0 + first + lane;
    n += __popc(mask);
    if (n < start) return false;
    __syncwarp();
    uint32_t i = 0;
    for (; i + 4 <= n; i += 4)
      if (four(*reinterpret_cast<const uint4*>(list + i))) {
        done = true;
        return true;
      }
    const uint32_t rest = n - i, v = list[i + (lane & 3)];
    __syncwarp();
    if ((uint32_t)lane < rest) list[lane] = v;
    n = rest;
    return false;
  });
  if (done || n == 0) return;
  if (lane < 4) list[n + lane] = S.slots / kBucketPoints;
  __syncwarp();
  for (uint32_t i = 0; i < n; i += 4)
    if (four(*reinterpret_cast<const uint4*>(list + i))) return;
  __syncwarp();
}

// How many nodes of level LEAF the box meets; the count may stop once it is
// above `most`.
template <int LEAF>
__device__ __forceinline__ uint32_t nodes_met(const SceneView& S, const TreeShape* __restrict__ T, const PacketBox& box,
                                              const PacketBox* limit, float reach2, WalkStack& stack, int lane,
                                              uint32_t most) {
  uint32_t nodes = 0;
  walk_wide<LEAF>(S, T, box, limit, reach2, stack, lane, [&](uint32_t, uint32_t mask) {
    nodes += __popc(mask);
    return nodes > most;
  });
  return nodes;
}

// Cuts a packet into runs of neighbouring queries that are worth walking
// together.  The box around a run may meet far more of the scene than its
// queries reach: at the edge of a cluster, between clusters, or in a call of
// few queries over many points.  A walk costs about 45 instructions per bucket
// its box meets; a query alone costs 400 and 18 per bucket its own cube meets,
// which are the cube's share of the run's buckets by volume.  So a run of s
// queries is walked together when its box meets at most 400 s / (45 - 18 s
// share) buckets (9 to 20 s), else its halves are tried, and runs of four that
// still do not fit go to single().  With 10 s whatever the share, rows of 32 in
// radius for 160k queries over 1M points took 651 us (566), six served requests
// 1009 (984), a batch of 128 problems 6035 (5918); with 16 and 24 s, 0.5 in radius of
// 240k queries over 1M clustered points 555 and 636 us (521).  With radii of their
// own 10 s holds (6 and 16 s: KNN k = 32 of 100k queries 1.26 and 1.12 ms against
// 1.08).  The buckets are only counted (a step per level-1 node) when the number
// of level-1 nodes, which hold 32 buckets and of which a box meets about 6 each,
// does not decide (a count of about five steps over the upper levels): up to s / 2 + 4
// fit, more than 2 s do not.  Counting the buckets of every hopeless run kept
// the last packets of a 65k-query shell 25 us longer; with s in place of 2 s too
// many queries went alone (six served requests 1.03 -> 2.2 ms).  Neither is
// counted when the box is at most 8 times one query's cube and all radii are
// equal (on the clustered 1M x 1M sets it is 5.8 times, 14 nodes and 87
// buckets).  Judged by the nodes alone a packet could still meet 1,000 buckets,
// and a few such packets kept the kernel running 0.2 ms after the rest had
// ended.
// walk(mine, box, limit, reach2) gets the lanes of a run, single(mask) the
// lanes that go alone.
template <typename Walk, typename Single>
__device__ __forceinline__ void cut_packet(const SceneView& S, const TreeShape* __restrict__ T, const float4& q,
                                           float lane_reach2, bool own_radii, bool active, WalkStack& stack, int lane,
                                           Walk&& walk, Single&& single) {
  const uint32_t act = __ballot_sync(0xffffffffu, active);
  const float half = own_radii ? reach_half_width(lane_reach2) : 0.f;
  int s = 32;
  // A narrow packet starts at its own width, so the limits fit its queries (a
  // 65k-query shell 360 -> 310 us, a 20k-query summary 336 -> 261).  With radii of
  // their own the queries left over cost too much (KNN k = 32 1.06 -> 1.26 ms).
  while (!own_radii && s > 4 && (act >> (s / 2)) == 0) s >>= 1;
  for (int at = 0; at < 32 && (act >> at) != 0;) {
    const uint32_t run = act & ((0xffffffffu >> (32 - s)) << at);
    if (run) {
      const bool mine = (run >> lane) & 1u;
      const PacketBox box = packet_box(q, mine);
      PacketBox limit;
      float reach2 = lane_reach2;  // equal in every lane unless own_radii
      uint32_t most = 10u * (uint32_t)s;  // buckets the run may meet
      bool fits = false;
      if (own_radii) {
        limit = packet_reach_box(q, half, mine);
        reach2 = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mine ? lane_reach2 : 0.f)));
      } else {
        const float w = 2.f * sqrtf(reach2), cube = w * w * w;
        const float all = (box.hx - box.lx + w) * (box.hy - box.ly + w) * (box.hz - box.lz + w);
        fits = all <= 8.f * cube;
        most = (uint32_t)((float)s * fminf(400.f / fmaxf(45.f - 18.f * (float)s * (cube / all), 1.f), 20.f));
      }
      const PacketBox* lim = own_radii ? &limit : nullptr;
      if (!fits) {
        const uint32_t w = (uint32_t)s, met = nodes_met<1>(S, T, box, lim, reach2, stack, lane, 2 * w);
        fits = met <= w / 2 + 4 ||
               (met <= 2 * w && nodes_met<0>(S, T, box, lim, reach2, stack, lane, most) <= most);
      }
      if (!fits && s > 4) {
        s >>= 1;
        continue;
      }
      if (fits) walk(mine, box, lim, reach2);
      else single(run);
    }
    at += s;
    // the next run: the largest aligned one (`at` is a multiple of s)
    while (s < 32 && (at & s) == 0 && at < 32) s <<= 1;
  }
}

}  // namespace
}  // namespace rtdl_b200
