// lbvh.cu -- on-device linear BVH over the search points.
//
// Build steps, all on one stream with no host round trip:
//   1. prep:    AoS FP64 records (RtdlPoint / RtdlPoint3D) -> float4 {x, y, z, id}
//               plus set statistics (box, largest |coordinate|, FP32
//               exactness, finiteness, id order);
//   2. codes:   30-bit (3D, 10 bits per axis) or 32-bit (2D, 16 bits per
//               axis) Hilbert codes relative to the set's box;
//   3. sort:    stable radix sort of (code, input index) pairs (sort_scan.cu);
//   4. buckets: points into code order, eight to a bucket, with the boxes of
//               the buckets and of the nodes of 32 buckets; exact FP64
//               coordinates alongside when the set is not FP32-exact;
//   5. levels:  the boxes of the upper levels, 32 children per node, until a
//               level has at most 32 nodes.
// The tree's shape follows from the number of points, so there are no splits,
// links or counts to compute: 1M points build in 0.17 ms, of which the sort's
// passes take 0.07 (the binary radix tree over the same codes, with its collapse,
// refit and pre-order records, took 0.38 ms).
#include "internal.cuh"

namespace rtdl_b200 {

namespace {

constexpr int kThreads = 256;

inline unsigned int grid_for(uint64_t n, int threads = kThreads) {
  uint64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  const uint64_t cap = (uint64_t)kSmCount * 16;
  return (unsigned int)(b < cap ? b : cap);
}

constexpr int kPrepThreads = 256;

// k_prep's grid: enough blocks to fill the SMs a few times over, few enough
// that the per-block atomics stay cheap.
inline unsigned int prep_grid(uint64_t n) {
  uint64_t b = (n + kPrepThreads - 1) / kPrepThreads;
  if (b < 1) b = 1;
  const uint64_t cap = (uint64_t)kSmCount * 4;
  return (unsigned int)(b < cap ? b : cap);
}

template <int DIM>
__global__ void __launch_bounds__(kPrepThreads) k_prep(const double* __restrict__ raw, uint32_t n, float4* __restrict__ out,
                       PointStats* __restrict__ st) {
  constexpr int kStride = DIM == 3 ? 4 : 3;  // record size in doubles (id occupies the first slot)
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  double max_abs = 0.0;
  unsigned int inexact = 0, bad = 0, unsorted = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const double* r = raw + i * kStride;
    const uint32_t id = *reinterpret_cast<const uint32_t*>(r);
    double c[3] = {r[1], r[2], DIM == 3 ? r[3] : 0.0};
    float f[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double v = c[a];
      const double av = fabs(v);
      if (!(av <= kMaxCoordinate)) bad = 1;  // also catches NaN
      f[a] = __double2float_rn(v);
      if ((double)f[a] != v) inexact = 1;
      lo[a] = fminf(lo[a], f[a]);
      hi[a] = fmaxf(hi[a], f[a]);
      max_abs = fmax(max_abs, av);
    }
    if (i > 0) {
      const uint32_t prev = *reinterpret_cast<const uint32_t*>(raw + (i - 1) * kStride);
      if (id < prev) unsorted = 1;
    }
    out[i] = make_float4(f[0], f[1], f[2], __uint_as_float(id));
  }
  // warp reduction, then a block reduction through shared memory, then one set
  // of atomics per block (same-address atomics from every warp would
  // serialise in L2)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
      hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
    }
    max_abs = fmax(max_abs, __shfl_xor_sync(0xffffffffu, max_abs, o));
    inexact |= __shfl_xor_sync(0xffffffffu, inexact, o);
    bad |= __shfl_xor_sync(0xffffffffu, bad, o);
    unsorted |= __shfl_xor_sync(0xffffffffu, unsorted, o);
  }
  __shared__ float s_lo[3][kPrepThreads / 32], s_hi[3][kPrepThreads / 32];
  __shared__ double s_abs[kPrepThreads / 32];
  __shared__ unsigned int s_flags[kPrepThreads / 32];
  const int warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      s_lo[a][warp] = lo[a];
      s_hi[a][warp] = hi[a];
    }
    s_abs[warp] = max_abs;
    s_flags[warp] = inexact | (bad << 1) | (unsorted << 2);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned int fl = 0;
    for (int w = 0; w < nwarps; ++w) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        lo[a] = fminf(lo[a], s_lo[a][w]);
        hi[a] = fmaxf(hi[a], s_hi[a][w]);
      }
      max_abs = fmax(max_abs, s_abs[w]);
      fl |= s_flags[w];
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      if (lo[a] <= hi[a]) {
        atomicMin(&st->lo[a], float_to_ordered(lo[a]));
        atomicMax(&st->hi[a], float_to_ordered(hi[a]));
      }
    }
    atomicMax(&st->max_abs_bits, (unsigned long long)__double_as_longlong(max_abs));
    if (fl & 1u) atomicOr(&st->inexact, 1u);
    if (fl & 2u) atomicOr(&st->bad, kBadCoordinates);
    if (fl & 4u) atomicOr(&st->ids_unsorted, 1u);
  }
}

__global__ void k_reset_stats(PointStats* st) {
  if (threadIdx.x == 0) {
    for (int a = 0; a < 3; ++a) {
      st->lo[a] = 0xFFFFFFFFu;
      st->hi[a] = 0u;
    }
    st->max_abs_bits = 0ull;
    st->inexact = 0u;
    st->bad = 0u;
    st->ids_unsorted = 0u;
    st->pad = 0u;
  }
}

__device__ __forceinline__ uint32_t spread10(uint32_t v) {  // 10 bits -> every third bit
  v &= 0x3FFu;
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}
__device__ __forceinline__ uint32_t spread16(uint32_t v) {  // 16 bits -> every other bit
  v &= 0xFFFFu;
  v = (v | (v << 8)) & 0x00FF00FFu;
  v = (v | (v << 4)) & 0x0F0F0F0Fu;
  v = (v | (v << 2)) & 0x33333333u;
  v = (v | (v << 1)) & 0x55555555u;
  return v;
}

// Hilbert index of a cell with `bits` bits per axis, by Skilling's transform
// ("Programming the Hilbert curve", AIP Conf. Proc. 707, 2004): the axes are
// turned into the transposed index in place, then interleaved, axis 0 first.
// Neighbours on the curve are neighbours in space, which the Morton curve's
// jumps are not: on the clustered 1M x 1M sets a packet of 32 consecutive
// queries reaches 28.9 leaf buckets along it instead of 31.6, and the boxes
// that only its bounding box meets fall from 21 to 9.
template <int DIM, int BITS>
__device__ __forceinline__ uint32_t hilbert_code(uint32_t x, uint32_t y, uint32_t z, int bits) {
#pragma unroll
  for (int b = BITS - 1; b > 0; --b) {
    if (b >= bits) continue;  // fewer bits than BITS (problem batches)
    const uint32_t q = 1u << b, p = q - 1u;
    uint32_t t;
    if (x & q) x ^= p;
    t = (y & q) ? 0u : (x ^ y) & p;
    x ^= (y & q) ? p : t;
    y ^= t;
    if (DIM == 3) {
      t = (z & q) ? 0u : (x ^ z) & p;
      x ^= (z & q) ? p : t;
      z ^= t;
    }
  }
  y ^= x;
  if (DIM == 3) z ^= y;
  const uint32_t last = DIM == 3 ? z : y;
  uint32_t t = last >> 1;  // bit i: the parity of the bits above i
  t ^= t >> 1;
  t ^= t >> 2;
  t ^= t >> 4;
  t ^= t >> 8;
  x ^= t;
  y ^= t;
  z ^= t;
  return DIM == 3 ? (spread10(x) << 2) | (spread10(y) << 1) | spread10(z) : (spread16(x) << 1) | spread16(y);
}

constexpr uint32_t kNoProblem = 0xFFFFFFFFu;

// Digit counts of a block's codes for the sort's four passes: each warp keeps
// its own histograms in shared memory, summed into `counts` at the end.
struct DigitCounts {
  unsigned int h[kThreads / 32][4][256];
};
__device__ __forceinline__ void digits_clear(DigitCounts& D) {
  for (int i = threadIdx.x; i < (kThreads / 32) * 4 * 256; i += kThreads) (&D.h[0][0][0])[i] = 0;
  __syncthreads();
}
// All lanes of the warp call this.  The top digit of neighbouring inputs is often
// one and the same (a batch's problem number), so it is counted once then.
__device__ __forceinline__ void digits_add(DigitCounts& D, uint32_t code, bool valid) {
  const unsigned int mask = __ballot_sync(0xffffffffu, valid);
  const uint32_t top = code >> 24, top0 = __shfl_sync(0xffffffffu, top, 0);
  const bool one = __all_sync(0xffffffffu, top == top0 || !valid);
  if (!valid) return;
  unsigned int (&h)[4][256] = D.h[threadIdx.x >> 5];
#pragma unroll
  for (int p = 0; p < 3; ++p) atomicAdd(&h[p][(code >> (8 * p)) & 255u], 1u);
  if (!one) atomicAdd(&h[3][top], 1u);
  else if ((threadIdx.x & 31) == 0) atomicAdd(&h[3][top], (unsigned int)__popc(mask));
}
__device__ __forceinline__ void digits_sum(DigitCounts& D, uint32_t* counts) {
  __syncthreads();
  for (int i = threadIdx.x; i < 4 * 256; i += kThreads) {
    unsigned int c = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) c += (&D.h[w][0][0])[i];
    if (c) atomicAdd(&counts[i], c);
  }
}
// Blocks of a kernel that counts digits: the histograms' 32 KB bound them.
inline unsigned int digits_grid(uint64_t n) {
  const uint64_t b = (n + kThreads - 1) / kThreads, cap = (uint64_t)kSmCount * 6;
  return (unsigned int)(b < cap ? b : cap);
}

// counts non-null: the sort's digit counts as well, without another read of the
// codes: 18 us at 1M points, where the codes alone took 19.5 us while the parity
// step went bit by bit.
template <int DIM>
__global__ void __launch_bounds__(kThreads) k_curve_codes(const float4* __restrict__ pts, uint32_t n,
                                                         const PointStats* __restrict__ box,
                                                         uint32_t* __restrict__ codes, uint32_t* counts) {
  constexpr int kBits = DIM == 3 ? 10 : 16;
  __shared__ DigitCounts digits;
  if (counts) digits_clear(digits);
  float lo[3], scale[3];
  const float cells = (float)((1u << kBits) - 1u);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const unsigned int ol = box->lo[a], oh = box->hi[a];
    const bool empty = ol == 0xFFFFFFFFu;
    const float l = empty ? 0.f : ordered_to_float(ol);
    const float h = empty ? 0.f : ordered_to_float(oh);
    lo[a] = l;
    const float ext = h - l;
    scale[a] = (ext > 0.f && isfinite(ext)) ? cells / ext : 0.f;
  }
  const int lane = threadIdx.x & 31;
  for (uint64_t i0 = ((uint64_t)blockIdx.x * kThreads + threadIdx.x) - lane; i0 < n;
       i0 += (uint64_t)gridDim.x * kThreads) {
    const uint64_t i = i0 + lane;
    const bool valid = i < n;
    uint32_t code = 0;
    if (valid) {
      const float4 p = pts[i];
      const float c[3] = {p.x, p.y, p.z};
      uint32_t q[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        float t = (c[a] - lo[a]) * scale[a];
        t = fminf(fmaxf(t, 0.f), cells);
        q[a] = (uint32_t)t;
      }
      code = hilbert_code<DIM, kBits>(q[0], q[1], q[2], kBits);
      codes[i] = code;
    }
    if (counts) digits_add(digits, code, valid);
  }
  if (counts) digits_sum(digits, counts);
}

// The problem whose level-`level` nodes include node g (trees are laid out
// problem after problem in every level, problems without nodes take no room).
__device__ __forceinline__ uint32_t problem_of_node(const TreeShape* __restrict__ trees, uint32_t problems,
                                                    int level, uint32_t g) {
  uint32_t lo = 0, hi = problems;  // first problem whose nodes start after g
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (trees[mid].base[level] <= g) lo = mid + 1;
    else hi = mid;
  }
  return lo - 1;
}

struct BucketBuild {
  const float4* in;        // prepared points, input order
  const double* raw;       // their records
  const uint32_t* order;   // curve order -> input index
  const unsigned long long* first;  // batch: first point of each problem; nullptr: one problem
  const PointStats* st;
  const TreeShape* trees;  // batch: per problem
  uint32_t problems;
  TreeShape plain;         // one problem: its tree, written to trees_out
  TreeShape* trees_out;
  uint32_t slots;
  float4* pts;
  uint32_t* perm;
  double* pts64;
  float4* bucket_pts;
  float4* wide;
};

// Points into curve order, and the two lowest levels of the wide tree: one
// block per level-1 node takes its 256 points, eight lanes per bucket reduce
// the bucket's box, the block the node's.  A thread reads its point once and
// writes it to both layouts; the rest of the build reads 1/256 of the points'
// bytes.  Bound by the gather's DRAM traffic.
template <int DIM>
__global__ void __launch_bounds__(256) k_buckets(BucketBuild B) {
  constexpr int kStride = DIM == 3 ? 4 : 3;
  __shared__ uint32_t s_prob;
  __shared__ float4 s_lo[8], s_hi[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  TreeShape T = B.plain;
  unsigned long long first = 0;
  uint32_t node = blockIdx.x;  // level-1 node within its problem
  if (B.first) {
    const uint32_t g = B.trees[0].base[1] + blockIdx.x;
    if (tid == 0) s_prob = problem_of_node(B.trees, B.problems, 1, g);
    __syncthreads();
    const uint32_t p = s_prob;
    T = B.trees[p];
    first = B.first[p];
    node = g - T.base[1];
  } else if (blockIdx.x == 0 && tid == 0) {
    *B.trees_out = T;
  }
  if (blockIdx.x == 0 && tid < DIM * kBucketPoints)  // the empty bucket after the last
    reinterpret_cast<float*>(B.bucket_pts)[(uint64_t)B.slots * DIM + tid] = INFINITY;
  const uint32_t j = node * 256u + tid;     // point within the problem
  const uint32_t bucket = node * 32u + (tid >> 3);
  const bool slot = bucket < T.buckets, has = j < T.points;
  float4 p = make_float4(INFINITY, INFINITY, DIM == 3 ? INFINITY : 0.f, 0.f);
  const uint64_t i = (uint64_t)T.base[0] * kBucketPoints + j;
  if (has) {
    const uint32_t src = B.order[first + j];
    p = B.in[src];
    B.perm[i] = src;
    if (B.st->inexact != 0) {
      const double* r = B.raw + (uint64_t)src * kStride;
      B.pts64[3 * i + 0] = r[1];
      B.pts64[3 * i + 1] = r[2];
      B.pts64[3 * i + 2] = DIM == 3 ? r[3] : 0.0;
    }
  } else if (slot) {
    B.perm[i] = kNone;
    if (B.st->inexact != 0)
      for (int a = 0; a < 3; ++a) B.pts64[3 * i + a] = INFINITY;
  }
  if (slot) {
    B.pts[i] = p;
    float* soa = reinterpret_cast<float*>(B.bucket_pts) + ((uint64_t)T.base[0] + bucket) * (DIM * kBucketPoints);
    soa[tid & 7] = p.x;
    soa[8 + (tid & 7)] = p.y;
    if (DIM == 3) soa[16 + (tid & 7)] = p.z;
  }
  float4 lo = has ? p : make_float4(INFINITY, INFINITY, INFINITY, 0.f);
  float4 hi = has ? p : make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    if (o == 8 && (tid & 7) == 0 && slot) {
      float4* w = B.wide + 2 * ((uint64_t)T.base[0] + bucket);
      w[0] = make_float4(lo.x, lo.y, lo.z, 0.f);
      w[1] = make_float4(hi.x, hi.y, hi.z, 0.f);
    }
    lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o));
    lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
    lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o));
    hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
    hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
    hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
  }
  if (lane == 0) {
    s_lo[warp] = lo;
    s_hi[warp] = hi;
  }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < 8; ++w) {
      lo = make_float4(fminf(lo.x, s_lo[w].x), fminf(lo.y, s_lo[w].y), fminf(lo.z, s_lo[w].z), 0.f);
      hi = make_float4(fmaxf(hi.x, s_hi[w].x), fmaxf(hi.y, s_hi[w].y), fmaxf(hi.z, s_hi[w].z), 0.f);
    }
    float4* w = B.wide + 2 * ((uint64_t)T.base[1] + node);
    w[0] = make_float4(lo.x, lo.y, lo.z, 0.f);
    w[1] = make_float4(hi.x, hi.y, hi.z, 0.f);
  }
}

// Level `level` (2 and up) of the wide tree: a warp per node, a lane per child.
__global__ void __launch_bounds__(256) k_wide_level(const TreeShape* __restrict__ trees, uint32_t problems, int level,
                                                    uint32_t first, uint32_t count, float4* wide) {
  const int lane = threadIdx.x & 31;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < count; k += warps) {
    const uint32_t g = first + k;
    const TreeShape& T = trees[problems > 1 ? problem_of_node(trees, problems, level, g) : 0];
    const uint32_t child = (g - T.base[level]) * kFan + lane;
    float4 lo = make_float4(INFINITY, INFINITY, INFINITY, 0.f);
    float4 hi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
    if (child < tree_level_nodes(T.buckets, level - 1)) {
      const float4* c = wide + 2 * ((uint64_t)T.base[level - 1] + child);
      lo = c[0];
      hi = c[1];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo.x = fminf(lo.x, __shfl_xor_sync(0xffffffffu, lo.x, o));
      lo.y = fminf(lo.y, __shfl_xor_sync(0xffffffffu, lo.y, o));
      lo.z = fminf(lo.z, __shfl_xor_sync(0xffffffffu, lo.z, o));
      hi.x = fmaxf(hi.x, __shfl_xor_sync(0xffffffffu, hi.x, o));
      hi.y = fmaxf(hi.y, __shfl_xor_sync(0xffffffffu, hi.y, o));
      hi.z = fmaxf(hi.z, __shfl_xor_sync(0xffffffffu, hi.z, o));
    }
    if (lane == 0) {
      wide[2 * (uint64_t)g] = lo;
      wide[2 * (uint64_t)g + 1] = hi;
    }
  }
}

// Problem id of every point, by bisection over the offsets.
__global__ void k_batch_ids(const unsigned long long* __restrict__ offsets, uint32_t problems, uint32_t n,
                            uint32_t* __restrict__ pid) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = problems;  // first problem that starts after i
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (__ldg(&offsets[mid]) <= i) lo = mid + 1;
      else hi = mid;
    }
    pid[i] = lo - 1;
  }
}

// The points a warp takes when the whole grid shares n points in input order:
// one contiguous span (whole rounds of 32), so it meets few problems and keeps
// what belongs to one in registers.
__device__ __forceinline__ void warp_span(uint32_t n, uint64_t& begin, uint64_t& end) {
  const uint64_t warps = (uint64_t)gridDim.x * (kThreads / 32);
  const uint64_t span = ((n + warps - 1) / warps + 31) & ~31ull;
  begin = ((uint64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5)) * span;
  end = begin + span < n ? begin + span : n;
}

// Per-problem boxes: each lane keeps the running box of the problem the warp's
// rounds lie in; a change of problem (or the span's end) reduces it over the
// warp and issues one set of atomics.  Rounds that hold several problems use
// per-lane atomics.  6M points of 128 problems: 30 us; a reduction per round of
// 32 took 160 us.
__global__ void __launch_bounds__(kThreads) k_batch_boxes(const float4* __restrict__ pts,
                                                         const uint32_t* __restrict__ pid, uint32_t n,
                                                         PointStats* __restrict__ st) {
  const int lane = threadIdx.x & 31;
  uint64_t begin, end;
  warp_span(n, begin, end);
  uint32_t cur = kNoProblem;
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  auto flush = [&]() {
    if (cur == kNoProblem) return;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      float l = lo[a], h = hi[a];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        l = fminf(l, __shfl_xor_sync(0xffffffffu, l, o));
        h = fmaxf(h, __shfl_xor_sync(0xffffffffu, h, o));
      }
      if (lane == 0) {
        atomicMin(&st[cur].lo[a], float_to_ordered(l));
        atomicMax(&st[cur].hi[a], float_to_ordered(h));
      }
      lo[a] = INFINITY;
      hi[a] = -INFINITY;
    }
  };
  constexpr int kAhead = 4;  // rounds loaded together
  for (uint64_t i0 = begin; i0 < end; i0 += 32 * kAhead) {
    uint32_t p[kAhead];
    float4 q[kAhead];
#pragma unroll
    for (int r = 0; r < kAhead; ++r) {
      const uint64_t i = i0 + 32 * r + lane;
      p[r] = i < end ? pid[i] : kNoProblem;
      q[r] = i < end ? pts[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int r = 0; r < kAhead; ++r) {
      const bool valid = p[r] != kNoProblem;
      const uint32_t p0 = __shfl_sync(0xffffffffu, p[r], 0);
      if (p0 == kNoProblem) continue;  // past the end
      const float c[3] = {q[r].x, q[r].y, q[r].z};
      if (__all_sync(0xffffffffu, p[r] == p0 || !valid)) {
        if (p0 != cur) {
          flush();
          cur = p0;
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          lo[a] = valid ? fminf(lo[a], c[a]) : lo[a];
          hi[a] = valid ? fmaxf(hi[a], c[a]) : hi[a];
        }
      } else {
        flush();
        cur = kNoProblem;
        if (valid) {
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            atomicMin(&st[p[r]].lo[a], float_to_ordered(c[a]));
            atomicMax(&st[p[r]].hi[a], float_to_ordered(c[a]));
          }
        }
      }
    }
  }
  flush();
}

__global__ void k_reset_stats_n(PointStats* st, uint32_t m) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    for (int a = 0; a < 3; ++a) {
      st[i].lo[a] = 0xFFFFFFFFu;
      st[i].hi[a] = 0u;
    }
    st[i].max_abs_bits = 0ull;
    st[i].inexact = 0u;
    st[i].bad = 0u;
    st[i].ids_unsorted = 0u;
    st[i].pad = 0u;
  }
}

// Composite sort keys (problem << code_bits) | curve code of the point in its
// problem's box, code_bits / dim bits per axis.
template <int DIM>
__global__ void __launch_bounds__(kThreads) k_batch_codes(const float4* __restrict__ pts,
                                                         const uint32_t* __restrict__ pid, uint32_t n,
                                                         const PointStats* __restrict__ st, int stats_stride,
                                                         int code_bits, uint32_t* __restrict__ codes,
                                                         uint32_t* counts) {
  constexpr int kBits = DIM == 3 ? 10 : 16;
  __shared__ DigitCounts digits;
  if (counts) digits_clear(digits);
  const int bpa = code_bits / DIM;
  const float cells = (float)((1u << bpa) - 1u);
  uint64_t begin, end;
  warp_span(n, begin, end);
  uint32_t cur = kNoProblem;  // the problem lo and scale belong to
  float lo[3] = {0.f, 0.f, 0.f}, scale[3] = {0.f, 0.f, 0.f};
  for (uint64_t i0 = begin; i0 < end; i0 += 32) {
    const uint64_t i = i0 + (threadIdx.x & 31);
    const bool valid = i < end;
    uint32_t code = 0;
    if (valid) {
      const uint32_t p = pid[i];
      const float4 q = pts[i];
      if (p != cur) {
        const PointStats& box = st[(size_t)p * stats_stride];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const unsigned int ol = box.lo[a], oh = box.hi[a];
          lo[a] = ol == 0xFFFFFFFFu ? 0.f : ordered_to_float(ol);
          const float ext = (ol == 0xFFFFFFFFu ? 0.f : ordered_to_float(oh)) - lo[a];
          scale[a] = (ext > 0.f && isfinite(ext)) ? cells / ext : 0.f;
        }
        cur = p;
      }
      const float c[3] = {q.x, q.y, q.z};
      uint32_t m[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        float t = (c[a] - lo[a]) * scale[a];
        t = fminf(fmaxf(t, 0.f), cells);
        m[a] = (uint32_t)t;
      }
      code = (code_bits < 32 ? (p << code_bits) : 0u) | hilbert_code<DIM, kBits>(m[0], m[1], m[2], bpa);
      codes[i] = code;
    }
    if (counts) digits_add(digits, code, valid);
  }
  if (counts) digits_sum(digits, counts);
}

}  // namespace

void reset_stats(PointStats* stats, cudaStream_t s) {
  k_reset_stats<<<1, 32, 0, s>>>(stats);
  RTDL_LAUNCHED(1);
}

void prep_points(const void* points_dev, uint32_t n, int dim, float4* out, PointStats* stats, cudaStream_t s) {
  if (n == 0) return;
  const double* raw = static_cast<const double*>(points_dev);
  if (dim == 3)
    k_prep<3><<<prep_grid(n), kPrepThreads, 0, s>>>(raw, n, out, stats);
  else
    k_prep<2><<<prep_grid(n), kPrepThreads, 0, s>>>(raw, n, out, stats);
  RTDL_LAUNCHED(1);
}

void curve_codes(const float4* pts, uint32_t n, int dim, const PointStats* box_stats, uint32_t* codes,
                 uint32_t* digit_counts, cudaStream_t s) {
  if (n == 0) return;
  if (dim == 3)
    k_curve_codes<3><<<digits_grid(n), kThreads, 0, s>>>(pts, n, box_stats, codes, digit_counts);
  else
    k_curve_codes<2><<<digits_grid(n), kThreads, 0, s>>>(pts, n, box_stats, codes, digit_counts);
  RTDL_LAUNCHED(1);
}

int batch_problem_bits(uint32_t problems) {
  int b = 0;
  while (b < 32 && (1ull << b) < (unsigned long long)problems) ++b;
  return b;
}

int batch_code_bits(uint32_t problems, int dim) {
  int bits = 32 - batch_problem_bits(problems);
  if (bits > (dim == 3 ? 30 : 32)) bits = dim == 3 ? 30 : 32;
  return bits - bits % dim;
}

void batch_problem_ids(const unsigned long long* offsets_dev, uint32_t problems, uint32_t n, uint32_t* pid,
                       cudaStream_t s) {
  if (n == 0 || problems == 0) return;
  k_batch_ids<<<grid_for(n), kThreads, 0, s>>>(offsets_dev, problems, n, pid);
  RTDL_LAUNCHED(1);
}

void batch_boxes(const float4* pts, const uint32_t* pid, uint32_t n, PointStats* prob_stats, uint32_t problems,
                 cudaStream_t s) {
  k_reset_stats_n<<<div_up(problems, 256), 256, 0, s>>>(prob_stats, problems);
  RTDL_LAUNCHED(1);
  if (n == 0) return;
  k_batch_boxes<<<digits_grid(n), kThreads, 0, s>>>(pts, pid, n, prob_stats);
  RTDL_LAUNCHED(1);
}

void batch_codes(const float4* pts, const uint32_t* pid, uint32_t n, int dim, const PointStats* prob_stats,
                 int stats_stride, int code_bits, uint32_t* codes, uint32_t* digit_counts, cudaStream_t s) {
  if (n == 0) return;
  if (dim == 3)
    k_batch_codes<3><<<digits_grid(n), kThreads, 0, s>>>(pts, pid, n, prob_stats, stats_stride, code_bits, codes,
                                                        digit_counts);
  else
    k_batch_codes<2><<<digits_grid(n), kThreads, 0, s>>>(pts, pid, n, prob_stats, stats_stride, code_bits, codes,
                                                        digit_counts);
  RTDL_LAUNCHED(1);
}

namespace {

Scene* build_scene_impl(const void* points_dev, uint32_t n, int dim, cudaStream_t s,
                        const unsigned long long* offsets, uint32_t problems) {
  if (dim != 2 && dim != 3) throw std::runtime_error("dimension must be 2 or 3");
  if (n > (uint32_t)kMaxScenePoints)
    throw std::runtime_error("search_count exceeds the scene limit of 67,108,864 points");
  const bool batch = offsets != nullptr;
  Scene* sc = new Scene();
  sc->dim = dim;
  sc->n = n;
  sc->stream = s;
  RTDL_CUDA_CHECK(cudaGetDevice(&sc->device));
  sc->stats = static_cast<PointStats*>(dev_alloc(sizeof(PointStats), s));
  reset_stats(sc->stats, s);
  if (batch) {
    sc->problems = problems;
    sc->code_bits = batch_code_bits(problems, dim);
    sc->prob_offsets.assign(offsets, offsets + problems + 1);
    sc->prob_stats = static_cast<PointStats*>(dev_alloc(sizeof(PointStats) * problems, s));
  }
  if (n == 0) {
    // trees of no buckets, where every walk ends at once
    const size_t bytes = sizeof(TreeShape) * (batch ? problems : 1);
    sc->trees = static_cast<TreeShape*>(dev_alloc(bytes, s));
    RTDL_CUDA_CHECK(cudaMemsetAsync(sc->trees, 0, bytes, s));
    if (batch) batch_boxes(nullptr, nullptr, 0, sc->prob_stats, problems, s);
    return sc;
  }
  // The wide tree's shape follows from the point counts alone; a batch's is
  // copied before any kernel is queued (a pageable copy waits for the stream).
  std::vector<TreeShape> shapes(batch ? problems : 1);
  uint32_t level_first[kTreeLevels + 1], level_nodes[kTreeLevels] = {0};
  for (uint32_t p = 0; p < shapes.size(); ++p) {
    TreeShape& T = shapes[p];
    T.points = batch ? (uint32_t)(offsets[p + 1] - offsets[p]) : n;
    T.buckets = div_up(T.points, kBucketPoints);
    T.top = 0;
    while (tree_level_nodes(T.buckets, T.top) > (uint32_t)kFan) ++T.top;
    for (int l = 0; l < kTreeLevels; ++l) {
      T.base[l] = level_nodes[l];  // within the level until the level sizes are known
      // level 1 exists for every problem with points (a build block writes it)
      if (T.points && ((uint32_t)l <= T.top || l == 1)) level_nodes[l] += tree_level_nodes(T.buckets, l);
    }
  }
  level_first[0] = 0;
  for (int l = 0; l < kTreeLevels; ++l) level_first[l + 1] = level_first[l] + level_nodes[l];
  for (TreeShape& T : shapes)
    for (int l = 0; l < kTreeLevels; ++l) T.base[l] += level_first[l];
  sc->slots = level_nodes[0] * kBucketPoints;
  sc->trees = static_cast<TreeShape*>(dev_alloc(sizeof(TreeShape) * shapes.size(), s));
  if (batch)
    RTDL_CUDA_CHECK(cudaMemcpyAsync(sc->trees, shapes.data(), sizeof(TreeShape) * shapes.size(),
                                    cudaMemcpyHostToDevice, s));
  const double* raw = static_cast<const double*>(points_dev);
  float4* pts_in = static_cast<float4*>(dev_alloc(sizeof(float4) * n, s));
  prep_points(points_dev, n, dim, pts_in, sc->stats, s);
  uint32_t* codes = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * n, s));
  unsigned long long* d_off = nullptr;
  SortWork sort;
  uint32_t* digits = radix_sort_counts(n, 0, batch ? 32 : curve_bits(dim), sort, s);
  if (batch) {
    d_off = static_cast<unsigned long long*>(dev_alloc(sizeof(unsigned long long) * (problems + 1), s));
    RTDL_CUDA_CHECK(cudaMemcpyAsync(d_off, sc->prob_offsets.data(), sizeof(unsigned long long) * (problems + 1),
                                    cudaMemcpyHostToDevice, s));
    uint32_t* pid = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * n, s));
    batch_problem_ids(d_off, problems, n, pid, s);
    batch_boxes(pts_in, pid, n, sc->prob_stats, problems, s);
    batch_codes(pts_in, pid, n, dim, sc->prob_stats, 1, sc->code_bits, codes, digits, s);
    dev_free(pid, s);
  } else {
    curve_codes(pts_in, n, dim, sc->stats, codes, digits, s);
  }
  uint32_t* order = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * n, s));
  radix_sort_counted(codes, order, n, true, sort, nullptr, &sc->stats->bad, s);
  sc->perm = static_cast<uint32_t*>(dev_alloc(sizeof(uint32_t) * sc->slots, s));
  sc->pts = static_cast<float4*>(dev_alloc(sizeof(float4) * sc->slots, s));
  sc->pts64 = static_cast<double*>(dev_alloc(sizeof(double) * 3 * (size_t)sc->slots, s));
  sc->bucket_pts = static_cast<float4*>(dev_alloc(sizeof(float) * dim * ((size_t)sc->slots + kBucketPoints), s));
  sc->wide = static_cast<float4*>(dev_alloc(sizeof(float4) * 2 * (size_t)level_first[kTreeLevels], s));
  BucketBuild BB;
  BB.in = pts_in;
  BB.raw = raw;
  BB.order = order;
  BB.first = d_off;
  BB.st = sc->stats;
  BB.trees = sc->trees;
  BB.problems = (uint32_t)shapes.size();
  BB.plain = shapes[0];
  BB.trees_out = sc->trees;
  BB.slots = sc->slots;
  BB.pts = sc->pts;
  BB.perm = sc->perm;
  BB.pts64 = sc->pts64;
  BB.bucket_pts = sc->bucket_pts;
  BB.wide = sc->wide;
  if (dim == 3)
    k_buckets<3><<<level_nodes[1], 256, 0, s>>>(BB);
  else
    k_buckets<2><<<level_nodes[1], 256, 0, s>>>(BB);
  RTDL_LAUNCHED(1);
  for (int l = 2; l < kTreeLevels && level_nodes[l] > 0; ++l) {
    k_wide_level<<<grid_for((uint64_t)level_nodes[l] * 32), kThreads, 0, s>>>(sc->trees, BB.problems, l,
                                                                             level_first[l], level_nodes[l],
                                                                             sc->wide);
    RTDL_LAUNCHED(1);
  }
  dev_free(order, s);
  dev_free(d_off, s);
  dev_free(pts_in, s);
  if (batch) {
    dev_free(codes, s);
    return sc;
  }
  sc->codes = codes;  // kept: nearest searches seed from a window around the query's code
  return sc;
}

}  // namespace

Scene* build_scene(const void* points_dev, uint32_t n, int dim, cudaStream_t s) {
  return build_scene_impl(points_dev, n, dim, s, nullptr, 0);
}

Scene* build_scene_batch(const void* points_dev, const unsigned long long* offsets, uint32_t problems, int dim,
                         cudaStream_t s) {
  if (problems == 0) throw std::runtime_error("a problem batch needs at least one problem");
  for (uint32_t p = 0; p < problems; ++p)
    if (offsets[p + 1] < offsets[p]) throw std::runtime_error("problem offsets must be non-decreasing");
  if (offsets[0] != 0) throw std::runtime_error("problem offsets must start at 0");
  if (offsets[problems] > (unsigned long long)kMaxScenePoints)
    throw std::runtime_error("a problem batch holds at most 67,108,864 search points");
  if (batch_problem_bits(problems) > 26)
    throw std::runtime_error("a problem batch holds at most 67,108,864 problems");
  return build_scene_impl(points_dev, (uint32_t)offsets[problems], dim, s, offsets, problems);
}

void destroy_scene(Scene* sc) {
  if (!sc) return;
  cudaStream_t s = sc->stream;
  dev_free(sc->pts, s);
  dev_free(sc->perm, s);
  dev_free(sc->pts64, s);
  dev_free(sc->codes, s);
  dev_free(sc->stats, s);
  dev_free(sc->prob_stats, s);
  dev_free(sc->bucket_pts, s);
  dev_free(sc->wide, s);
  dev_free(sc->trees, s);
  if (sc->own_stream && s) {
    sync_quietly(s);
    note_cleanup_error(cudaStreamDestroy(s), "cudaStreamDestroy");
  }
  delete sc;
}

}  // namespace rtdl_b200
