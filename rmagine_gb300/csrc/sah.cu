// Top-down binned-SAH build of a binary BVH with one triangle per leaf, on the
// GPU: the binned surface area heuristic of Wald ("On fast construction of
// SAH-based bounding volume hierarchies", IEEE RT 2007).
//
// An internal node's task is a contiguous range of the triangle permutation.
// Its triangles fall into kNB bins per axis over the bounds of their box
// centres; the split is the plane between bins of least A_L * N_L + A_R * N_R
// over the three axes, or a halving by position where the centres coincide or
// a side would let the tree grow deeper than kMaxDepth; a stable partition
// puts the left side's triangles first.  The leaf of position k holds the k-th
// triangle of the final permutation.  A subtree over m triangles has m - 1
// internal nodes, so nodes are numbered in preorder without counting them: the
// left child of node i is i + 1 and the right child i + (triangles on the
// left).  Nothing depends on thread timing: minima, maxima and counts are
// exact, and lists filled through atomics only order independent work.
//
// Tasks are handled by their size:
//   large (more than kSmall triangles), one level at a time over chunks of
//     kChunk positions of one task: k_bin (bins in shared memory, flushed to
//     the task's), k_split (one warp per task), k_partition (records moved to
//     the other buffer; a chunk's first rank comes from the chunks' bin counts);
//   small: k_small, one CTA per task, builds the whole subtree in shared
//     memory: warps bin and partition tasks of more than 32 triangles, and
//     finish those of up to 32 with one lane per triangle, where every lane
//     evaluates the planes after its own triangle's centre (no bins).
// A triangle travels as its box and id (32 B).  Every task writes its own box
// into its parent's record when it is split, so no refit follows.
//
// What bounds the build is the many levels over the same triangles: with one
// global pass per level (bins of 13 words updated by up to 39 global atomics a
// triangle in the lower levels, a device-wide scan per level, two host
// synchronisations per level) a 537,000-triangle terrain took 6.3 ms of kernels
// in 329 launches.
#include <algorithm>

#include "internal.h"

namespace rmg {
namespace {

#ifndef RMG_SAH_BINS
#define RMG_SAH_BINS 16
#endif
constexpr int kNB = RMG_SAH_BINS;     // bins per axis
static_assert(kNB >= 2 && kNB <= 16, "a half warp scans one axis");
constexpr int kBins = 3 * kNB;
constexpr int kBinWords = 7;          // count, box lo, box hi; odd, so that bins lie in different banks
constexpr uint32_t kMaxDepth = 32;    // leaves at most this many edges below the root
constexpr uint32_t kChunk = 1024;     // positions of a large task handled by one CTA
constexpr uint32_t kSmall = 512;      // largest task built in shared memory
constexpr int kBlk = 256;             // threads of the large-task kernels
constexpr int kSmallBlk = 128;        // threads of k_small
constexpr int kSmallWarps = kSmallBlk / 32;

// A triangle: box lo and id, box hi.
struct __align__(16) Rec {
  float4 a, b;
};

struct Task {
  uint32_t first, count;
  int node;        // internal node id
  int parent;      // the node whose child this is (-1: the root), and on which side
  uint32_t side, depth;
  uint32_t chunk0;   // large: first entry of the task's chunks
  uint32_t buf;      // small: which record buffer holds its range
  int clo[3], chi[3];  // large: bounds of the box centres (order-preserving ints)
};

struct Split {
  int axis;          // -1: halved by position
  int bin;           // bins 0..bin go left
  uint32_t left;     // triangles going left
  int big[2];        // large-task slot of each side in the next level, -1 if it is not large
};

// Counters of one build, in device memory.
struct Build {
  uint32_t n_big[2];     // large tasks of the even / odd levels
  uint32_t n_chunks[2];  // their chunks
  uint32_t n_small;
  uint32_t next_small;   // k_small's work counter
  uint32_t depth;        // deepest leaf (edges)
  uint32_t bad;          // partition disagreed with the bins, or a list was full: never
  uint32_t bad_face;     // a face names a vertex that is not there
  int root[6];           // bounds of all box centres
};

__device__ __forceinline__ int f2o(float f) {
  const int b = __float_as_int(f);
  return b >= 0 ? b : b ^ 0x7fffffff;
}
__device__ __forceinline__ float o2f(int o) { return __int_as_float(o >= 0 ? o : o ^ 0x7fffffff); }

constexpr int kEmptyLo = 0x7f800000;        // f2o(+inf)
constexpr int kEmptyHi = (int)0x807fffff;   // f2o(-inf)

__device__ __forceinline__ int ceil_log2(uint32_t x) { return x <= 1 ? 0 : 32 - __clz(x - 1); }

__device__ __forceinline__ float3 tri_v(const float* v, uint32_t i) {
  return make_float3(v[3 * (size_t)i], v[3 * (size_t)i + 1], v[3 * (size_t)i + 2]);
}

// The centre of the triangle's box (not the vertex mean: on a box room the
// vertex mean of a large wall triangle sits a third of the way across the
// wall, and the tree costs 13% more node visits per ray).
__device__ __forceinline__ float3 centre(const float4& a, const float4& b) {
  return make_float3(__fmul_rn(__fadd_rn(a.x, b.x), 0.5f), __fmul_rn(__fadd_rn(a.y, b.y), 0.5f),
                     __fmul_rn(__fadd_rn(a.z, b.z), 0.5f));
}

// Bin of centre coordinate c in bounds [lo, hi] (the same float operations
// wherever a bin is computed).
__device__ __forceinline__ int bin_of(float c, float lo, float hi) {
  const float ext = __fsub_rn(hi, lo);
  if (!(ext > 0.f)) return 0;
  const float s = __fdiv_rn((float)kNB, ext);
  const int b = (int)__fmul_rn(__fsub_rn(c, lo), s);
  return min(max(b, 0), kNB - 1);
}

__device__ __forceinline__ float half_area(const float lo[3], const float hi[3]) {
  const float ex = fmaxf(hi[0] - lo[0], 0.f), ey = fmaxf(hi[1] - lo[1], 0.f), ez = fmaxf(hi[2] - lo[2], 0.f);
  return ex * ey + ey * ez + ez * ex;
}

__device__ __forceinline__ bool too_deep(uint32_t depth, uint32_t l, uint32_t r) {
  return depth + 1 + ceil_log2(l) > kMaxDepth || depth + 1 + ceil_log2(r) > kMaxDepth;
}

// A child's box in its parent's record.  A coordinate that is NaN in every
// vertex below the child has an empty interval here (see k_prep) and is NaN in
// the record, as a refit leaves it.
__device__ __forceinline__ void write_box(Node* nodes, int parent, uint32_t side, const float lo[3], const float hi[3]) {
  Node* p = nodes + parent;
  const float nan = __int_as_float(0x7fffffff);
  float l[3], h[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const bool empty = lo[k] > hi[k];
    l[k] = empty ? nan : lo[k];
    h[k] = empty ? nan : hi[k];
  }
  const float4 xy = make_float4(l[0], h[0], l[1], h[1]);
  if (side == 0) p->a = xy; else p->b = xy;
  reinterpret_cast<float2*>(&p->c)[side] = make_float2(l[2], h[2]);
}

// Links of one node whose task covers `count` triangles from position `first`,
// `left` of them on the left.
__device__ __forceinline__ void write_links(Node* nodes, int node, int parent, uint32_t first, uint32_t count,
                                            uint32_t left) {
  const int l = left == 1 ? ~(int)first : node + 1;
  const int r = count - left == 1 ? ~(int)(first + left) : node + (int)left;
  nodes[node].d = make_int4(l, r, parent, 0);
}

// Adds a triangle to the bins of its three axes.  Minima and maxima first look
// at the bins: after a few triangles most would not change them.  A single warp
// (AHEAD) reads all eighteen words at once; where many warps share the bins a
// look just before the update saves more updates (k_bin 197 against 228 us).
template <bool AHEAD>
__device__ __forceinline__ void bin_add(int* bins, const Rec& r, const float3& c, const float clo[3], const float chi[3]) {
  const int lo[3] = {f2o(r.a.x), f2o(r.a.y), f2o(r.a.z)}, hi[3] = {f2o(r.b.x), f2o(r.b.y), f2o(r.b.z)};
  const float cc[3] = {c.x, c.y, c.z};
  int* B[3];
  int now[3][6];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    B[a] = bins + kBinWords * (a * kNB + bin_of(cc[a], clo[a], chi[a]));
    if (AHEAD) {
#pragma unroll
      for (int k = 0; k < 6; ++k) now[a][k] = B[a][1 + k];
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    atomicAdd(B[a], 1);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (lo[k] < (AHEAD ? now[a][k] : *(volatile int*)(B[a] + 1 + k))) atomicMin(B[a] + 1 + k, lo[k]);
      if (hi[k] > (AHEAD ? now[a][3 + k] : *(volatile int*)(B[a] + 4 + k))) atomicMax(B[a] + 4 + k, hi[k]);
    }
  }
}

__device__ __forceinline__ int empty_word(int i) {
  const int k = i % kBinWords;
  return k == 0 ? 0 : (k < 4 ? kEmptyLo : kEmptyHi);
}

// The split of a task from its bins, by one whole warp: lane k of the lower
// half warp holds bin k of one axis at a time; prefix and suffix boxes and
// counts by shuffles.  Every lane returns the same answer; box is the task's.
struct Choice {
  int axis, bin;
  uint32_t left;
  float lo[3], hi[3];
};

__device__ __forceinline__ Choice warp_split(const int* bins, uint32_t count, uint32_t depth) {
  const uint32_t lane = threadIdx.x & 31;
  Choice ch;
  ch.axis = -1;
  ch.bin = -1;
  ch.left = count / 2;
  float best = INFINITY;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    uint32_t pc = 0, sc = 0;
    float pl[3] = {INFINITY, INFINITY, INFINITY}, ph[3] = {-INFINITY, -INFINITY, -INFINITY}, sl[3], sh[3];
    if (lane < kNB) {
      const int* B = bins + kBinWords * (a * kNB + (int)lane);
      pc = (uint32_t)B[0];
#pragma unroll
      for (int k = 0; k < 3; ++k) { pl[k] = o2f(B[1 + k]); ph[k] = o2f(B[4 + k]); }
    }
    sc = pc;
#pragma unroll
    for (int k = 0; k < 3; ++k) { sl[k] = pl[k]; sh[k] = ph[k]; }
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const uint32_t uc = __shfl_up_sync(0xffffffffu, pc, o), dc = __shfl_down_sync(0xffffffffu, sc, o);
      if (lane >= (uint32_t)o) pc += uc;
      sc += lane + o < 32 ? dc : 0u;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float ul = __shfl_up_sync(0xffffffffu, pl[k], o), uh = __shfl_up_sync(0xffffffffu, ph[k], o);
        const float dl = __shfl_down_sync(0xffffffffu, sl[k], o), dh = __shfl_down_sync(0xffffffffu, sh[k], o);
        if (lane >= (uint32_t)o) { pl[k] = fminf(pl[k], ul); ph[k] = fmaxf(ph[k], uh); }
        if (lane + o < 32) { sl[k] = fminf(sl[k], dl); sh[k] = fmaxf(sh[k], dh); }
      }
    }
    if (a == 0) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        ch.lo[k] = __shfl_sync(0xffffffffu, sl[k], 0);
        ch.hi[k] = __shfl_sync(0xffffffffu, sh[k], 0);
      }
    }
    // plane after bin `lane`: left = bins 0..lane, right = the next lane's suffix
    const float sarea = half_area(sl, sh);
    const float rarea = __shfl_down_sync(0xffffffffu, sarea, 1);
    const uint32_t rcnt = __shfl_down_sync(0xffffffffu, sc, 1);
    float cost = INFINITY;
    if (lane < kNB - 1 && pc > 0 && rcnt > 0 && !too_deep(depth, pc, rcnt))
      cost = half_area(pl, ph) * (float)pc + rarea * (float)rcnt;
    if (!(cost < INFINITY)) cost = INFINITY;  // NaN
    float m = cost;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fminf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (m < best) {
      const int k = __ffs((int)__ballot_sync(0xffffffffu, cost == m)) - 1;
      best = m;
      ch.axis = a;
      ch.bin = k;
      ch.left = __shfl_sync(0xffffffffu, pc, k);
    }
  }
  return ch;
}

// ---- large tasks ---------------------------------------------------------------------

// Boxes and ids of all triangles; bounds of their box centres.  A coordinate that
// is NaN in all three vertices gets the empty interval (+inf, -inf): the bins'
// order-preserving integers would take a NaN for the largest of numbers, while
// every minimum and maximum passes over an empty interval, as fminf and fmaxf
// pass over a NaN.  (Its centre is NaN still, and falls into bin 0.)
__global__ void __launch_bounds__(kBlk) k_prep(const float* v, uint32_t n_vertices, const uint32_t* f, uint32_t n, Rec* rec,
                                               Build* B) {
  __shared__ int sb[6];
  if (threadIdx.x < 6) sb[threadIdx.x] = threadIdx.x < 3 ? kEmptyLo : kEmptyHi;
  __syncthreads();
  float cl[3] = {INFINITY, INFINITY, INFINITY}, chh[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (uint32_t i = blockIdx.x * kBlk + threadIdx.x; i < n; i += gridDim.x * kBlk) {
    uint32_t q[3] = {f[3 * (size_t)i], f[3 * (size_t)i + 1], f[3 * (size_t)i + 2]};
#pragma unroll
    for (int k = 0; k < 3; ++k)
      if (q[k] >= n_vertices) { B->bad_face = 1; q[k] = 0; }
    const float3 a = tri_v(v, q[0]), b = tri_v(v, q[1]), d = tri_v(v, q[2]);
    Rec r;
    r.a = make_float4(fminf(fminf(a.x, b.x), d.x), fminf(fminf(a.y, b.y), d.y), fminf(fminf(a.z, b.z), d.z),
                      __uint_as_float(i));
    r.b = make_float4(fmaxf(fmaxf(a.x, b.x), d.x), fmaxf(fmaxf(a.y, b.y), d.y), fmaxf(fmaxf(a.z, b.z), d.z), 0.f);
    if (isnan(r.a.x)) { r.a.x = INFINITY; r.b.x = -INFINITY; }
    if (isnan(r.a.y)) { r.a.y = INFINITY; r.b.y = -INFINITY; }
    if (isnan(r.a.z)) { r.a.z = INFINITY; r.b.z = -INFINITY; }
    rec[i] = r;
    const float3 c = centre(r.a, r.b);
    cl[0] = fminf(cl[0], c.x); cl[1] = fminf(cl[1], c.y); cl[2] = fminf(cl[2], c.z);
    chh[0] = fmaxf(chh[0], c.x); chh[1] = fmaxf(chh[1], c.y); chh[2] = fmaxf(chh[2], c.z);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int l = __reduce_min_sync(0xffffffffu, f2o(cl[k])), h = __reduce_max_sync(0xffffffffu, f2o(chh[k]));
    if ((threadIdx.x & 31) == 0) { atomicMin(&sb[k], l); atomicMax(&sb[3 + k], h); }
  }
  __syncthreads();
  if (threadIdx.x < 3) atomicMin(&B->root[threadIdx.x], sb[threadIdx.x]);
  else if (threadIdx.x < 6) atomicMax(&B->root[threadIdx.x], sb[threadIdx.x]);
}

// The root's task: one large task with its chunks and cleared bins, or the one
// small task.  One CTA.
__global__ void k_root(uint32_t n, Build* B, Task* big, uint2* chunks, int* bins, Task* small) {
  const uint32_t nc = (n + kChunk - 1) / kChunk;
  Task t;
  t.first = 0;
  t.count = n;
  t.node = 0;
  t.parent = -1;
  t.side = 0;
  t.depth = 0;
  t.chunk0 = 0;
  t.buf = 0;
  for (int k = 0; k < 3; ++k) { t.clo[k] = B->root[k]; t.chi[k] = B->root[3 + k]; }
  if (n <= kSmall) {
    if (threadIdx.x == 0) { small[0] = t; B->n_small = 1; }
    return;
  }
  if (threadIdx.x == 0) { big[0] = t; B->n_big[0] = 1; B->n_chunks[0] = nc; }
  for (uint32_t c = threadIdx.x; c < nc; c += blockDim.x) chunks[c] = make_uint2(0u, c);
  for (int i = threadIdx.x; i < kBins * kBinWords; i += blockDim.x) bins[i] = empty_word(i);
}

// Bins of one chunk, added to its task's; the chunk's prefix counts per axis
// for k_partition.  A lane's triangles lie kChunk / 32 positions from its
// neighbour's, so that the lanes of a warp, whose records are sectors of their
// own anyway, seldom meet in one bin of a mesh that is stored in space order.
__global__ void __launch_bounds__(kBlk) k_bin(Build* B, uint32_t par, const Task* tasks, const uint2* chunks,
                                              const Rec* rec, int* bins, uint32_t* hist) {
  if (blockIdx.x == 0 && threadIdx.x == 0) { B->n_big[par ^ 1u] = 0; B->n_chunks[par ^ 1u] = 0; }  // k_split fills them
  if (blockIdx.x >= B->n_chunks[par]) return;
  __shared__ int sb[kBins * kBinWords];
  const uint2 ck = chunks[blockIdx.x];
  const Task& T = tasks[ck.x];
  float clo[3], chi[3];
  for (int k = 0; k < 3; ++k) { clo[k] = o2f(T.clo[k]); chi[k] = o2f(T.chi[k]); }
  for (int i = threadIdx.x; i < kBins * kBinWords; i += kBlk) sb[i] = empty_word(i);
  __syncthreads();
  const uint32_t off = ck.y * kChunk, len = min(kChunk, T.count - off);
  const Rec* r0 = rec + T.first + off;
  for (uint32_t k = threadIdx.x >> 5; k < kChunk / 32; k += kBlk / 32) {
    const uint32_t i = (threadIdx.x & 31) * (kChunk / 32) + k;
    if (i < len) {
      const Rec r = r0[i];
      bin_add<false>(sb, r, centre(r.a, r.b), clo, chi);
    }
  }
  __syncthreads();
  int* g = bins + (size_t)ck.x * kBins * kBinWords;
  for (int i = threadIdx.x; i < kBins * kBinWords; i += kBlk) {
    if (sb[i / kBinWords * kBinWords] == 0) continue;
    const int k = i % kBinWords;
    if (k == 0) atomicAdd(g + i, sb[i]);
    else if (k < 4) atomicMin(g + i, sb[i]);
    else atomicMax(g + i, sb[i]);
  }
  if (threadIdx.x < kBins) {
    const int a = threadIdx.x / kNB, b = threadIdx.x % kNB;
    uint32_t c = 0;
    for (int k = 0; k <= b; ++k) c += (uint32_t)sb[kBinWords * (a * kNB + k)];
    hist[(size_t)blockIdx.x * kBins + threadIdx.x] = c;
  }
}

// One warp per large task: its split, its node, its children's tasks.
__global__ void __launch_bounds__(128) k_split(Build* B, uint32_t par, const Task* tasks, const int* bins, Split* splits,
                                               Task* next, uint2* next_chunks, int* next_bins, Task* small,
                                               uint32_t max_big, uint32_t max_chunks, uint32_t max_small, Node* nodes,
                                               int* leaf_parent) {
  const uint32_t j = (blockIdx.x * 128 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (j >= B->n_big[par]) return;
  const Task T = tasks[j];
  const Choice ch = warp_split(bins + (size_t)j * kBins * kBinWords, T.count, T.depth);
  Split s;
  s.axis = ch.axis;
  s.bin = ch.bin;
  s.left = ch.left;
  const uint32_t first[2] = {T.first, T.first + ch.left}, count[2] = {ch.left, T.count - ch.left};
  for (int side = 0; side < 2; ++side) {
    s.big[side] = -1;
    if (count[side] == 1) {
      if (lane == 0) {
        leaf_parent[first[side]] = T.node;
        atomicMax(&B->depth, T.depth + 1);
      }
      continue;
    }
    Task c;
    c.first = first[side];
    c.count = count[side];
    c.node = side == 0 ? T.node + 1 : T.node + (int)ch.left;
    c.parent = T.node;
    c.side = (uint32_t)side;
    c.depth = T.depth + 1;
    c.chunk0 = 0;
    c.buf = par ^ 1u;
    for (int k = 0; k < 3; ++k) { c.clo[k] = kEmptyLo; c.chi[k] = kEmptyHi; }
    uint32_t slot = 0;
    if (count[side] <= kSmall) {
      if (lane == 0) {
        slot = atomicAdd(&B->n_small, 1u);
        if (slot < max_small) small[slot] = c; else B->bad = 1;
      }
      continue;
    }
    const uint32_t nc = (count[side] + kChunk - 1) / kChunk;
    if (lane == 0) {
      slot = atomicAdd(&B->n_big[par ^ 1u], 1u);
      c.chunk0 = atomicAdd(&B->n_chunks[par ^ 1u], nc);
    }
    slot = __shfl_sync(0xffffffffu, slot, 0);
    c.chunk0 = __shfl_sync(0xffffffffu, c.chunk0, 0);
    if (slot >= max_big || c.chunk0 + nc > max_chunks) {  // disjoint ranges: never
      if (lane == 0) B->bad = 1;
      continue;
    }
    if (lane == 0) next[slot] = c;
    for (uint32_t k = lane; k < nc; k += 32) next_chunks[c.chunk0 + k] = make_uint2(slot, k);
    int* nb = next_bins + (size_t)slot * kBins * kBinWords;
    for (int i = (int)lane; i < kBins * kBinWords; i += 32) nb[i] = empty_word(i);
    s.big[side] = (int)slot;
  }
  if (lane == 0) {
    splits[j] = s;
    write_links(nodes, T.node, T.parent, T.first, T.count, ch.left);
    if (T.parent >= 0) write_box(nodes, T.parent, T.side, ch.lo, ch.hi);
  }
}

// Stable partition of one chunk into the other record buffer, the centre bounds
// of large children, and leaf children.
__global__ void __launch_bounds__(kBlk) k_partition(Build* B, uint32_t par, const Task* tasks, const uint2* chunks,
                                                    const Split* splits, const uint32_t* hist, const Rec* src, Rec* dst,
                                                    Task* next, Node* nodes, uint32_t* order) {
  if (blockIdx.x >= B->n_chunks[par]) return;
  __shared__ uint32_t s_base, s_warp[kBlk / 32];
  __shared__ int s_b[12];
  const uint2 ck = chunks[blockIdx.x];
  const Task& T = tasks[ck.x];
  const Split S = splits[ck.x];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float clo[3], chi[3];
  for (int k = 0; k < 3; ++k) { clo[k] = o2f(T.clo[k]); chi[k] = o2f(T.chi[k]); }
  if (threadIdx.x < 12) s_b[threadIdx.x] = threadIdx.x % 6 < 3 ? kEmptyLo : kEmptyHi;
  if (threadIdx.x == 0) s_base = 0;
  __syncthreads();
  const uint32_t off = ck.y * kChunk, len = min(kChunk, T.count - off);
  if (S.axis >= 0) {  // left triangles of the task's earlier chunks
    uint32_t c = 0;
    for (uint32_t j = threadIdx.x; j < ck.y; j += kBlk)
      c += hist[(size_t)(T.chunk0 + j) * kBins + S.axis * kNB + S.bin];
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0 && c) atomicAdd(&s_base, c);
  } else if (threadIdx.x == 0) {
    s_base = min(off, S.left);
  }
  float bl[2][3], bh[2][3];
  for (int q = 0; q < 2; ++q)
    for (int k = 0; k < 3; ++k) { bl[q][k] = INFINITY; bh[q][k] = -INFINITY; }
  for (uint32_t r = 0; r < len; r += kBlk) {
    const uint32_t i = r + threadIdx.x;
    const bool in = i < len;
    Rec x;
    bool left = false;
    float3 c = make_float3(0.f, 0.f, 0.f);
    if (in) {
      x = src[T.first + off + i];
      c = centre(x.a, x.b);
      if (S.axis < 0) left = off + i < S.left;
      else {
        const float cc = S.axis == 0 ? c.x : (S.axis == 1 ? c.y : c.z);
        const float l = S.axis == 0 ? clo[0] : (S.axis == 1 ? clo[1] : clo[2]);
        const float h = S.axis == 0 ? chi[0] : (S.axis == 1 ? chi[1] : chi[2]);
        left = bin_of(cc, l, h) <= S.bin;
      }
    }
    const unsigned bal = __ballot_sync(0xffffffffu, left);
    if (lane == 0) s_warp[warp] = (uint32_t)__popc(bal);
    __syncthreads();
    uint32_t before = s_base, total = 0;
    for (uint32_t w = 0; w < kBlk / 32; ++w) { if (w < warp) before += s_warp[w]; total += s_warp[w]; }
    const uint32_t rank = before + (uint32_t)__popc(bal & ((1u << lane) - 1u));
    if (in) {
      const uint32_t side = left ? 0u : 1u;
      const uint32_t p = left ? rank : S.left + (off + i - rank);
      if (p >= T.count) {
        B->bad = 1;
      } else {
        dst[T.first + p] = x;
        const uint32_t cnt = left ? S.left : T.count - S.left;
        if (cnt == 1) {  // a leaf
          const float lo[3] = {x.a.x, x.a.y, x.a.z}, hi[3] = {x.b.x, x.b.y, x.b.z};
          write_box(nodes, T.node, side, lo, hi);
          order[T.first + p] = __float_as_uint(x.a.w);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (left != (q == 0)) continue;
          bl[q][0] = fminf(bl[q][0], c.x); bl[q][1] = fminf(bl[q][1], c.y); bl[q][2] = fminf(bl[q][2], c.z);
          bh[q][0] = fmaxf(bh[q][0], c.x); bh[q][1] = fmaxf(bh[q][1], c.y); bh[q][2] = fmaxf(bh[q][2], c.z);
        }
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) s_base += total;
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    if (S.big[q] < 0) continue;  // uniform
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int l = __reduce_min_sync(0xffffffffu, f2o(bl[q][k])), h = __reduce_max_sync(0xffffffffu, f2o(bh[q][k]));
      if (lane == 0) { atomicMin(&s_b[6 * q + k], l); atomicMax(&s_b[6 * q + 3 + k], h); }
    }
  }
  __syncthreads();
  if (threadIdx.x < 12) {
    const int q = threadIdx.x / 6, k = threadIdx.x % 6;
    if (S.big[q] >= 0) {
      Task* c = next + S.big[q];
      if (k < 3) atomicMin(&c->clo[k], s_b[threadIdx.x]); else atomicMax(&c->chi[k - 3], s_b[threadIdx.x]);
    }
  }
}

// ---- small tasks ---------------------------------------------------------------------

struct Sub {  // a task inside k_small's range
  uint16_t first, count;
  int node, parent;
  uint32_t side_depth;  // side << 8 | depth
};

struct SmallShared {
  Rec rec[kSmall];
  uint16_t perm[2][kSmall];
  __align__(16) int bins[kSmallWarps][kBins * kBinWords];
  Sub mid[2][kSmall / 33 + 1];  // tasks of more than 32 triangles, by level
  Sub tiny[kSmall / 2];
  uint32_t n_mid[2], n_tiny, task;
};

struct SmallOut {
  Node* nodes;
  int* leaf_parent;
  uint32_t* order;
};

// A task of up to 32 triangles, one lane each: all its subtasks, level by
// level.  No bins here: every lane evaluates, on each axis, the plane just after
// its own box centre (centres up to it go left) by walking over its subtask's
// triangles -- the full sweep over all planes -- and the least (cost, axis,
// lane) wins.  The lanes' records live in `slot` (32 of them).
__device__ void build_tiny(Rec* slot, const uint16_t* perm, const Rec* rec, const Sub& t, uint32_t first,
                           const SmallOut& out, uint32_t& max_depth) {
  const uint32_t lane = threadIdx.x & 31, m = t.count;
  const bool live = lane < m;
  __syncwarp();
  if (live) slot[lane] = rec[perm[t.first + lane]];
  __syncwarp();
  uint32_t s = live ? 0 : lane, e = live ? m : lane;   // this lane's subtask, as lanes [s, e)
  int node = t.node, parent = t.parent;
  uint32_t side = t.side_depth >> 8, depth = t.side_depth & 255u;
  while (__any_sync(0xffffffffu, e - s > 1)) {
    const bool on = e - s > 1;
    Rec me;
    float3 c;
    float cost = INFINITY;
    uint32_t key = 0;
    float lo[3], hi[3];
    if (on) {
      me = slot[lane];
      c = centre(me.a, me.b);
      float ll[3][3], lh[3][3], rl[3][3], rh[3][3];
      uint32_t lc = 0;  // left counts, one byte per axis
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int k = 0; k < 3; ++k) { ll[a][k] = rl[a][k] = INFINITY; lh[a][k] = rh[a][k] = -INFINITY; }
#pragma unroll 2
      for (uint32_t j = s; j < e; ++j) {
        const float4 ja = slot[j].a, jb = slot[j].b;
        const float3 jc = centre(ja, jb);
        const bool left[3] = {jc.x <= c.x, jc.y <= c.y, jc.z <= c.z};
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          if (left[a]) {
            lc += 1u << (8 * a);
            ll[a][0] = fminf(ll[a][0], ja.x); ll[a][1] = fminf(ll[a][1], ja.y); ll[a][2] = fminf(ll[a][2], ja.z);
            lh[a][0] = fmaxf(lh[a][0], jb.x); lh[a][1] = fmaxf(lh[a][1], jb.y); lh[a][2] = fmaxf(lh[a][2], jb.z);
          } else {
            rl[a][0] = fminf(rl[a][0], ja.x); rl[a][1] = fminf(rl[a][1], ja.y); rl[a][2] = fminf(rl[a][2], ja.z);
            rh[a][0] = fmaxf(rh[a][0], jb.x); rh[a][1] = fmaxf(rh[a][1], jb.y); rh[a][2] = fmaxf(rh[a][2], jb.z);
          }
        }
      }
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const uint32_t l = (lc >> (8 * a)) & 255u, r = e - s - l;
        if (l == 0 || r == 0 || too_deep(depth, l, r)) continue;
        const float x = half_area(ll[a], lh[a]) * (float)l + half_area(rl[a], rh[a]) * (float)r;
        if (x < cost) { cost = x; key = (uint32_t)a << 8 | lane; }
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) { lo[k] = fminf(ll[0][k], rl[0][k]); hi[k] = fmaxf(lh[0][k], rh[0][k]); }
    }
    // least (cost, axis, lane) of the subtask (the spare words of the slots carry
    // them; the id stays in the lane's register)
    __syncwarp();
    if (on) { slot[lane].a.w = cost; slot[lane].b.w = __uint_as_float(key); }
    __syncwarp();
    bool left = false;
    if (on) {
#pragma unroll 4
      for (uint32_t j = s; j < e; ++j) {
        const float x = slot[j].a.w;
        const uint32_t k = __float_as_uint(slot[j].b.w);
        if (x < cost || (x == cost && k < key)) { cost = x; key = k; }
      }
      if (!(cost < INFINITY)) {
        left = lane - s < (e - s) / 2;  // halved by position
      } else {
        const Rec& w = slot[key & 255u];
        const float3 wc = centre(w.a, w.b);
        const uint32_t axis = key >> 8;
        left = axis == 0 ? c.x <= wc.x : (axis == 1 ? c.y <= wc.y : c.z <= wc.z);
      }
    }
    const unsigned bal = __ballot_sync(0xffffffffu, left);
    uint32_t p = lane, L = 0;
    if (on) {
      const unsigned seg = (e == 32 ? 0u : 1u << e) - (1u << s);  // lanes [s, e)
      L = (uint32_t)__popc(bal & seg);
      const uint32_t rank = (uint32_t)__popc(bal & seg & ((1u << lane) - 1u));
      p = left ? s + rank : s + L + (lane - s - rank);
      if (lane == s) {
        write_links(out.nodes, node, parent, first + t.first + s, e - s, L);
        if (parent >= 0) write_box(out.nodes, parent, side, lo, hi);
      }
    }
    __syncwarp();
    if (on) slot[p] = me;
    __syncwarp();
    if (on) {
      parent = node;
      ++depth;
      if (lane < s + L) { node = node + 1; side = 0; e = s + L; }
      else { node = node + (int)L; side = 1; s = s + L; }
      if (e - s == 1) {
        const Rec x = slot[lane];
        const float xl[3] = {x.a.x, x.a.y, x.a.z}, xh[3] = {x.b.x, x.b.y, x.b.z};
        write_box(out.nodes, parent, side, xl, xh);
        out.leaf_parent[first + t.first + lane] = parent;
        out.order[first + t.first + lane] = __float_as_uint(x.a.w);
        max_depth = max(max_depth, depth);
      }
    }
  }
}

// One CTA builds the subtree of one small task at a time.
__global__ void __launch_bounds__(kSmallBlk) k_small(Build* B, uint32_t p, const Task* small, const Rec* rec0,
                                                     const Rec* rec1, SmallOut out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SmallShared& S = *reinterpret_cast<SmallShared*>(smem_raw);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t n_small = B->n_small;
  uint32_t max_depth = 0;
  // large tasks are left (of level parity p), or the build has failed
  if (threadIdx.x == 0) S.task = B->n_big[p] | B->bad | B->bad_face;
  __syncthreads();
  if (S.task != 0) return;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) S.task = atomicAdd(&B->next_small, 1u);
    __syncthreads();
    if (S.task >= n_small) break;
    const Task T = small[S.task];
    const Rec* src = (T.buf ? rec1 : rec0) + T.first;
    for (uint32_t i = threadIdx.x; i < T.count; i += kSmallBlk) {
      S.rec[i] = src[i];
      S.perm[0][i] = (uint16_t)i;
    }
    if (threadIdx.x == 0) {
      const Sub root{0, (uint16_t)T.count, T.node, T.parent, T.side << 8 | T.depth};
      S.n_mid[0] = S.n_mid[1] = S.n_tiny = 0;
      if (T.count > 32) { S.mid[0][0] = root; S.n_mid[0] = 1; }
      else { S.tiny[0] = root; S.n_tiny = 1; }
    }
    __syncthreads();
    uint32_t par = 0;
    while (S.n_mid[par] > 0) {
      const uint32_t nm = S.n_mid[par];
      for (uint32_t q = warp; q < nm; q += kSmallWarps) {
        const Sub t = S.mid[par][q];
        const uint32_t depth = t.side_depth & 255u;
        int* bins = S.bins[warp];
        uint16_t* perm = S.perm[0] + t.first;
        uint16_t* perm2 = S.perm[1] + t.first;
        for (int i = (int)lane; i < kBins * kBinWords; i += 32) bins[i] = empty_word(i);
        float clo[3] = {INFINITY, INFINITY, INFINITY}, chi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (uint32_t i = lane; i < t.count; i += 32) {
          const Rec& r = S.rec[perm[i]];
          const float3 c = centre(r.a, r.b);
          clo[0] = fminf(clo[0], c.x); clo[1] = fminf(clo[1], c.y); clo[2] = fminf(clo[2], c.z);
          chi[0] = fmaxf(chi[0], c.x); chi[1] = fmaxf(chi[1], c.y); chi[2] = fmaxf(chi[2], c.z);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          clo[k] = o2f(__reduce_min_sync(0xffffffffu, f2o(clo[k])));
          chi[k] = o2f(__reduce_max_sync(0xffffffffu, f2o(chi[k])));
        }
        __syncwarp();
        for (uint32_t i = lane; i < t.count; i += 32) {
          const Rec r = S.rec[perm[i]];
          bin_add<true>(bins, r, centre(r.a, r.b), clo, chi);
        }
        __syncwarp();
        const Choice ch = warp_split(bins, t.count, depth);
        uint32_t base = 0;
        for (uint32_t r = 0; r < t.count; r += 32) {
          const uint32_t i = r + lane;
          bool left = false;
          uint16_t id = 0;
          if (i < t.count) {
            id = perm[i];
            if (ch.axis < 0) left = i < ch.left;
            else {
              const float3 c = centre(S.rec[id].a, S.rec[id].b);
              const float cc = ch.axis == 0 ? c.x : (ch.axis == 1 ? c.y : c.z);
              const float l = ch.axis == 0 ? clo[0] : (ch.axis == 1 ? clo[1] : clo[2]);
              const float h = ch.axis == 0 ? chi[0] : (ch.axis == 1 ? chi[1] : chi[2]);
              left = bin_of(cc, l, h) <= ch.bin;
            }
          }
          const unsigned bal = __ballot_sync(0xffffffffu, left);
          const uint32_t rank = base + (uint32_t)__popc(bal & ((1u << lane) - 1u));
          if (i < t.count) {
            const uint32_t p = left ? rank : ch.left + (i - rank);
            if (p < t.count) perm2[p] = id; else B->bad = 1;
          }
          base += (uint32_t)__popc(bal);
        }
        __syncwarp();
        for (uint32_t i = lane; i < t.count; i += 32) perm[i] = perm2[i];
        __syncwarp();
        if (lane == 0) {
          write_links(out.nodes, t.node, t.parent, T.first + t.first, t.count, ch.left);
          if (t.parent >= 0) write_box(out.nodes, t.parent, t.side_depth >> 8, ch.lo, ch.hi);
        }
        if (lane < 2) {  // the two children
          const uint32_t left = ch.left;
          Sub c;
          c.first = (uint16_t)(lane == 0 ? t.first : t.first + left);
          c.count = (uint16_t)(lane == 0 ? left : t.count - left);
          c.node = lane == 0 ? t.node + 1 : t.node + (int)left;
          c.parent = t.node;
          c.side_depth = lane << 8 | (depth + 1);
          if (c.count > 32) {
            S.mid[par ^ 1][atomicAdd(&S.n_mid[par ^ 1], 1u)] = c;
          } else if (c.count > 1) {
            S.tiny[atomicAdd(&S.n_tiny, 1u)] = c;
          } else {
            const Rec& x = S.rec[perm[c.first - t.first]];
            const float xl[3] = {x.a.x, x.a.y, x.a.z}, xh[3] = {x.b.x, x.b.y, x.b.z};
            write_box(out.nodes, t.node, lane, xl, xh);
            out.leaf_parent[T.first + c.first] = t.node;
            out.order[T.first + c.first] = __float_as_uint(x.a.w);
            max_depth = max(max_depth, depth + 1);
          }
        }
      }
      __syncthreads();
      if (threadIdx.x == 0) S.n_mid[par] = 0;
      par ^= 1;
      __syncthreads();
    }
    // the warps' bins are free now: 32 records of build_tiny each
    Rec* slot = reinterpret_cast<Rec*>(S.bins[warp]);
    static_assert(sizeof(Rec) * 32 <= sizeof(int) * kBins * kBinWords, "tiny tasks live in the bins' memory");
    const uint32_t n_tiny = S.n_tiny;
    for (uint32_t q = warp; q < n_tiny; q += kSmallWarps)
      build_tiny(slot, S.perm[0], S.rec, S.tiny[q], T.first, out, max_depth);
  }
  max_depth = __reduce_max_sync(0xffffffffu, max_depth);
  if (lane == 0 && max_depth > 0) atomicMax(&B->depth, max_depth);
}

inline unsigned blocks(size_t n, unsigned per) { return (unsigned)((n + per - 1) / per); }

}  // namespace

// A one-triangle-per-leaf SAH tree over the map's n >= 2 faces: links, parents
// and boxes in m->d_nodes, m->d_leaf_parent, the face of every leaf in d_order,
// m->depth.  Face indices are checked here.  Synchronises.
int sah_build(rmg_map* m, cudaStream_t st, uint32_t* d_order) {
  const uint32_t n = m->n_faces;
  if (n < 2) return fail(RMG_ERR_INVALID_ARG, "SAH build needs two or more faces");
  // large tasks of a level are disjoint ranges of more than kSmall triangles
  const uint32_t max_big = n / kSmall + 1, max_chunks = n / kChunk + max_big + 1;
  const uint32_t max_small = std::min<uint64_t>(n / 2 + 1, 2ull * (kMaxDepth + 1) * max_big + 1);
  const size_t bin_bytes = sizeof(int) * kBins * kBinWords;
  // one scratch allocation, carved
  size_t off = 0;
  auto carve = [&](size_t bytes) { const size_t at = off; off = (off + bytes + 255) & ~size_t(255); return at; };
  const size_t o_rec0 = carve(sizeof(Rec) * (size_t)n), o_rec1 = carve(sizeof(Rec) * (size_t)n);
  const size_t o_big0 = carve(sizeof(Task) * max_big), o_big1 = carve(sizeof(Task) * max_big);
  const size_t o_ck0 = carve(sizeof(uint2) * max_chunks), o_ck1 = carve(sizeof(uint2) * max_chunks);
  const size_t o_bin0 = carve(bin_bytes * max_big), o_bin1 = carve(bin_bytes * max_big);
  const size_t o_hist = carve(sizeof(uint32_t) * kBins * max_chunks);
  const size_t o_split = carve(sizeof(Split) * max_big);
  const size_t o_small = carve(sizeof(Task) * max_small);
  const size_t o_build = carve(sizeof(Build));
  unsigned char* base = nullptr;
  int s = pool_alloc(&base, off, st, "SAH build");
  if (s != RMG_OK) return s;
  Rec* rec[2] = {reinterpret_cast<Rec*>(base + o_rec0), reinterpret_cast<Rec*>(base + o_rec1)};
  Task* big[2] = {reinterpret_cast<Task*>(base + o_big0), reinterpret_cast<Task*>(base + o_big1)};
  uint2* chunks[2] = {reinterpret_cast<uint2*>(base + o_ck0), reinterpret_cast<uint2*>(base + o_ck1)};
  int* bins[2] = {reinterpret_cast<int*>(base + o_bin0), reinterpret_cast<int*>(base + o_bin1)};
  uint32_t* hist = reinterpret_cast<uint32_t*>(base + o_hist);
  Split* splits = reinterpret_cast<Split*>(base + o_split);
  Task* small = reinterpret_cast<Task*>(base + o_small);
  Build* B = reinterpret_cast<Build*>(base + o_build);
  Build h{};
  for (int k = 0; k < 3; ++k) { h.root[k] = kEmptyLo; h.root[3 + k] = kEmptyHi; }
  auto chk = [&](cudaError_t e, const char* what) { if (s == RMG_OK) s = cuda_status(e, what); };
  chk(cudaMemcpyAsync(B, &h, sizeof h, cudaMemcpyHostToDevice, st), "sah init");
  if (s == RMG_OK) {
    k_prep<<<std::min(blocks(n, kBlk), 8u * (unsigned)device_sm_count()), kBlk, 0, st>>>(m->d_vertices, m->n_vertices,
                                                                                         m->d_faces, n, rec[0], B);
    k_root<<<1, 1024, 0, st>>>(n, B, big[0], chunks[0], bins[0], small);
    chk(cudaGetLastError(), "sah prep");
  }
  // Levels of large tasks: as many as a balanced tree has and one more, then the
  // small tasks; where large ones are left after all, k_small does nothing and the
  // host, which looks once at the end, adds levels.  (A look before k_small as well
  // was 15 us of an idle GPU.)
  const int smem = (int)sizeof(SmallShared);
  int per_sm = 0;
  chk(cudaFuncSetAttribute(k_small, cudaFuncAttributeMaxDynamicSharedMemorySize, smem), "k_small shared memory");
  chk(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_small, kSmallBlk, smem), "k_small occupancy");
  const unsigned most = (unsigned)(std::max(per_sm, 1) * device_sm_count());
  uint32_t level = 0, upto = 0;
  if (n > kSmall) {
    while ((uint64_t)kSmall << upto < n) ++upto;
    upto += 1;
  }
  while (s == RMG_OK) {
    for (; level < upto; ++level) {
      const uint32_t p = level & 1u;
      // a level's chunks: at most one per kChunk positions and one more per task
      const uint32_t tasks = std::min<uint64_t>(max_big, 1ull << std::min(level, 31u));
      const uint32_t grid = std::min<uint64_t>(max_chunks, (uint64_t)n / kChunk + tasks + 1);
      k_bin<<<grid, kBlk, 0, st>>>(B, p, big[p], chunks[p], rec[p], bins[p], hist);
      k_split<<<blocks(tasks, 4), 128, 0, st>>>(B, p, big[p], bins[p], splits, big[p ^ 1], chunks[p ^ 1], bins[p ^ 1],
                                                small, max_big, max_chunks, max_small, m->d_nodes, m->d_leaf_parent);
      k_partition<<<grid, kBlk, 0, st>>>(B, p, big[p], chunks[p], splits, hist, rec[p], rec[p ^ 1], big[p ^ 1],
                                         m->d_nodes, d_order);
    }
    k_small<<<std::min(most, max_small), kSmallBlk, smem, st>>>(B, level & 1u, small, rec[0], rec[1],
                                                                SmallOut{m->d_nodes, m->d_leaf_parent, d_order});
    chk(cudaGetLastError(), "sah levels");
    chk(cudaMemcpyAsync(&h, B, sizeof h, cudaMemcpyDeviceToHost, st), "sah counters");
    chk(cudaStreamSynchronize(st), "sah sync");
    if (s != RMG_OK || h.bad || h.bad_face || h.n_big[level & 1u] == 0) break;
    if (level > kMaxDepth) { s = fail(RMG_ERR_CUDA, "SAH build: too many levels"); break; }
    upto = level + 3;
  }
  if (s == RMG_OK && h.bad_face) s = fail(RMG_ERR_INVALID_ARG, "rmg_map_build: face index out of range");
  if (s == RMG_OK && h.bad) s = fail(RMG_ERR_CUDA, "SAH build: partition disagrees with the split counts");
  m->depth = h.depth;
  pool_free(base, st);
  return s;
}

}  // namespace rmg
