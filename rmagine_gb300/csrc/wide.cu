// 4-wide tree collapsed from the binary LBVH.
//
// Same leaves (one packed triangle each) and the same boxes as the binary
// tree; a 4-wide node holds up to four children, chosen top-down: start from a
// binary node's two children and repeatedly open the internal child of
// largest surface area until four children are collected or only leaves
// remain (the greedy collapse of Wald, Benthin and Boulos, "Getting rid of
// packets", RT 2008, and of most wide-BVH builders since).  Every slot keeps
// the binary record its box came from (parent node and side), so after a
// binary refit the wide boxes are refreshed by one copy kernel.  Node indices
// are allocated level by level with an atomic counter, a node's internal
// children as one block; their order does not affect any result (the traversal's closest hit is order-independent).
#include <algorithm>
#include <vector>

#include "internal.h"

namespace rmg {
namespace {

constexpr int kBlock4 = 256;
constexpr int kMaxLevels4 = 192;  // a binary tree's depth at most (128 for the trail walks) and some more

struct Cand {
  int id;        // binary child link: >= 0 internal node, < 0 leaf ~k
  int src;       // 2 * binary parent + side
  float lo[3], hi[3];
};

__device__ __forceinline__ Cand cand_of(const Node& n, int parent, int side) {
  Cand c;
  c.src = 2 * parent + side;
  if (side == 0) {
    c.id = n.d.x;
    c.lo[0] = n.a.x; c.hi[0] = n.a.y; c.lo[1] = n.a.z; c.hi[1] = n.a.w; c.lo[2] = n.c.x; c.hi[2] = n.c.y;
  } else {
    c.id = n.d.y;
    c.lo[0] = n.b.x; c.hi[0] = n.b.y; c.lo[1] = n.b.z; c.hi[1] = n.b.w; c.lo[2] = n.c.z; c.hi[2] = n.c.w;
  }
  return c;
}

__device__ __forceinline__ float half_area(const Cand& c) {
  const float ex = fmaxf(c.hi[0] - c.lo[0], 0.f), ey = fmaxf(c.hi[1] - c.lo[1], 0.f),
              ez = fmaxf(c.hi[2] - c.lo[2], 0.f);
  return ex * ey + ey * ez + ez * ex;
}

__host__ __device__ __forceinline__ void set_slot(Node4& w, int k, const float lo[3], const float hi[3]) {
  float* lox = &w.lox.x; float* hix = &w.hix.x; float* loy = &w.loy.x;
  float* hiy = &w.hiy.x; float* loz = &w.loz.x; float* hiz = &w.hiz.x;
  lox[k] = lo[0]; hix[k] = hi[0]; loy[k] = lo[1]; hiy[k] = hi[1]; loz[k] = lo[2]; hiz[k] = hi[2];
}

// The collapse's counters in device memory.
struct WideBuild {
  unsigned int count;            // wide nodes allocated
  unsigned int levels;           // levels that held nodes
  unsigned int end[kMaxLevels4 + 2];   // level l: nodes [end[l], end[l + 1])
  unsigned int done[kMaxLevels4];      // CTAs of the level's launch that have finished
};

__device__ __forceinline__ void swap_cand(Cand& x, Cand& y, bool yes) {
  if (!yes) return;
  const Cand t = x;
  x = y;
  y = t;
}

// Level `level` of the collapse: its wide nodes, whose binary roots are
// bin_of[j], get their children; internal children receive new wide indices, a
// CTA's with one addition to the counter.  The last CTA to finish closes the
// next level, so the launches follow one another without the host.  537,000
// triangles, 13 levels: 188 us with all allocations made, where a host
// synchronisation per level and an atomic per node took 330; 130 us of kernels
// since fewer empty levels are launched.
__global__ void __launch_bounds__(kBlock4) k_collapse(const Node* __restrict__ bn, int* bin_of, WideBuild* B, int level,
                                                      uint32_t cap, Node4* w4, int* src4) {
  const uint32_t lo4 = B->end[level], hi4 = min(B->end[level + 1], cap);
  if (lo4 >= hi4 && blockIdx.x != 0) return;
  __shared__ uint32_t s_sum[kBlock4 / 32], s_base;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t j0 = lo4 + blockIdx.x * kBlock4; j0 < hi4; j0 += gridDim.x * kBlock4) {
    const uint32_t j = j0 + threadIdx.x;
    Cand c[4];
    int n = 0, ni = 0;
    if (j < hi4) {
      const int b = bin_of[j];
      const Node root = bn[b];
      c[0] = cand_of(root, b, 0);
      c[1] = cand_of(root, b, 1);
      n = root.d.x == root.d.y ? 1 : 2;  // the one-triangle tree: both links name leaf 0
#pragma unroll
      for (int open = 0; open < 2; ++open) {  // the internal child of largest area gives way to its two
        int best = -1;
        float ba = -1.f;
#pragma unroll
        for (int k = 0; k < 2 + open; ++k) {
          if (k < n && c[k].id >= 0) {
            const float a = half_area(c[k]);
            if (a > ba) { ba = a; best = k; }
          }
        }
        if (best >= 0) {
          int id = 0;
#pragma unroll
          for (int k = 0; k < 2 + open; ++k)
            if (k == best) id = c[k].id;
          const Node nb = bn[id];
          const Cand l = cand_of(nb, id, 0);
#pragma unroll
          for (int k = 0; k < 2 + open; ++k)
            if (k == best) c[k] = l;
          // n == 2 + open here: the earlier opening succeeded too, or this is the first
          c[2 + open] = cand_of(nb, id, 1);
          ++n;
        } else {
          break;
        }
      }
      // internal children take the first slots and get consecutive wide indices, so
      // a walk finds child `slot` at base + slot without reading the links
#pragma unroll
      for (int pass = 0; pass < 3; ++pass)
#pragma unroll
        for (int k = 0; k < 3 - pass; ++k) swap_cand(c[k], c[k + 1], k + 1 < n && c[k].id < 0 && c[k + 1].id >= 0);
#pragma unroll
      for (int k = 0; k < 4; ++k) ni += k < n && c[k].id >= 0 ? 1 : 0;
    }
    uint32_t at = (uint32_t)ni;  // inclusive prefix over the CTA
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, at, o);
      if (lane >= (uint32_t)o) at += u;
    }
    if (lane == 31) s_sum[warp] = at;
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (uint32_t w = 0; w < kBlock4 / 32; ++w) { if (w < warp) before += s_sum[w]; total += s_sum[w]; }
    if (threadIdx.x == 0) s_base = total ? atomicAdd(&B->count, total) : 0;
    __syncthreads();
    const int base = ni > 0 ? (int)(s_base + before + at - (uint32_t)ni) : 0;
    __syncthreads();
    if (j >= hi4 || (uint32_t)(base + ni) > cap) continue;  // more nodes than the binary tree has: never
    Node4 w;
    const float far[3] = {1e30f, 1e30f, 1e30f};
    int child[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k < n) {
        set_slot(w, k, c[k].lo, c[k].hi);
        if (c[k].id < 0) {
          child[k] = c[k].id;
        } else {
          bin_of[base + k] = c[k].id;
          child[k] = base + k;
        }
      } else {
        set_slot(w, k, far, far);
        child[k] = kEmpty4;
        c[k].src = -1;
      }
    }
    reinterpret_cast<int4*>(src4)[j] = make_int4(c[0].src, c[1].src, c[2].src, c[3].src);
    w.child = make_int4(child[0], child[1], child[2], child[3]);
    w.meta = make_int4(base, (((1 << n) - 1) ^ ((1 << ni) - 1)) | (((1 << ni) - 1) << 4), 0, 0);
    w4[j] = w;
  }
  __threadfence();
  __syncthreads();
  const uint32_t ctas = lo4 >= hi4 ? 1u : gridDim.x;
  if (threadIdx.x == 0 && atomicAdd(&B->done[level], 1u) == ctas - 1) {
    B->end[level + 2] = atomicAdd(&B->count, 0u);
    if (lo4 < hi4) B->levels = (unsigned int)level + 1u;
  }
}

// Boxes of every slot from the (refitted) binary records, one thread per slot.
__global__ void k_wide_refit(const Node* __restrict__ bn, const int* __restrict__ src4, uint32_t n4, Node4* w4) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 4ull * n4) return;
  const int s = src4[i];
  if (s < 0) return;
  const Node* b = bn + (s >> 1);
  const int side = s & 1;
  const float4 xy = __ldg(side ? &b->b : &b->a);
  const float2 z = __ldg(reinterpret_cast<const float2*>(&b->c) + side);
  float* w = reinterpret_cast<float*>(w4 + (i >> 2)) + (i & 3);
  w[0] = xy.x; w[4] = xy.y; w[8] = xy.z; w[12] = xy.w; w[16] = z.x; w[20] = z.y;
}

}  // namespace

void wide_free(rmg_map* m) {
  wide8_free(m);
  pool_release(m->d_nodes4);  // the caller has waited for the device
  m->d_nodes4 = nullptr;
  m->d_src4 = nullptr;
  m->n_nodes4 = 0;
  m->depth4 = 0;
}

// Builds the 4-wide tree of a map whose binary tree is complete (its depth
// known).  Synchronises once, or twice for a tree whose wide levels descend less
// than two binary ones each.
int wide_build(rmg_map* m, cudaStream_t st) {
  wide_free(m);
  if (m->n_faces == 0) return RMG_OK;
  const uint32_t cap = std::max<uint32_t>(m->n_nodes, 1u);
  int* bin_of = nullptr;
  WideBuild* B = nullptr;
  // all nodes, then the four sources of each
  unsigned char* base = nullptr;
  int s = pool_alloc(&base, (sizeof(Node4) + 4 * sizeof(int)) * (size_t)cap, st, "wide nodes");
  if (s == RMG_OK) {
    m->d_nodes4 = reinterpret_cast<Node4*>(base);
    m->d_src4 = reinterpret_cast<int*>(base + sizeof(Node4) * (size_t)cap);
  }
  if (s == RMG_OK) s = pool_alloc(&bin_of, cap, st, "wide roots");
  if (s == RMG_OK) s = pool_alloc(&B, 1, st, "wide counters");
  WideBuild h{};
  h.count = 1;
  h.end[1] = 1;
  if (s == RMG_OK) s = cuda_status(cudaMemsetAsync(bin_of, 0, 4, st), "wide init");
  if (s == RMG_OK) s = cuda_status(cudaMemcpyAsync(B, &h, sizeof h, cudaMemcpyHostToDevice, st), "wide init");
  // Every wide level descends at least one binary level, most descend two: half the
  // depth and two more are launched before the host looks whether nodes are left
  // (a launch that finds none takes 4 us, an early look 10).
  const int levels = (int)std::min<unsigned>(std::max(m->depth, 1u), (unsigned)kMaxLevels4);
  for (int l = 0, upto = std::min(levels, levels / 2 + 2); s == RMG_OK && l < levels; upto = levels) {
    for (; s == RMG_OK && l < upto; ++l) {
      const uint64_t most = std::min<uint64_t>(cap, 1ull << std::min(2 * l, 62));
      const unsigned grid = (unsigned)std::min<uint64_t>((most + kBlock4 - 1) / kBlock4, 4ull * device_sm_count());
      k_collapse<<<grid, kBlock4, 0, st>>>(m->d_nodes, bin_of, B, l, cap, m->d_nodes4, m->d_src4);
      s = cuda_status(cudaGetLastError(), "k_collapse");
    }
    if (s == RMG_OK) s = cuda_status(cudaMemcpyAsync(&h, B, sizeof h, cudaMemcpyDeviceToHost, st), "wide count");
    if (s == RMG_OK) s = cuda_status(cudaStreamSynchronize(st), "wide sync");
    if (h.end[l + 1] == h.end[l]) break;
  }
  if (s == RMG_OK && h.count > cap) s = fail(RMG_ERR_CUDA, "wide build: node count exceeds the binary tree");
  pool_free(bin_of, st);
  pool_free(B, st);
  if (s != RMG_OK) {
    cudaStreamSynchronize(st);
    wide_free(m);
    return s;
  }
  // a tree deeper than kMaxLevels4 keeps no 4-wide form (its walk takes at most
  // 21 levels anyway, see have_wide4)
  if (h.end[h.levels + 1] != h.end[h.levels]) { wide_free(m); return RMG_OK; }
  m->n_nodes4 = h.count;
  m->depth4 = h.levels;
  return RMG_OK;
}

// Test hook: slot `slot` of wide node `node` gets the link `child` (range-checked
// by the caller).  The walk takes internal children as consecutive nodes, so the
// node's slots are put in order again (internal ones first) and its internal
// children are copied to a new block behind the last node.  Synchronises.
int wide_set_child(rmg_map* m, uint32_t node, uint32_t slot, int child) {
  const uint32_t n4 = m->n_nodes4;
  std::vector<Node4> w(n4);
  std::vector<int> src(4 * (size_t)n4);
  RMG_CUDA_TRY(cudaMemcpy(w.data(), m->d_nodes4, sizeof(Node4) * n4, cudaMemcpyDeviceToHost));
  RMG_CUDA_TRY(cudaMemcpy(src.data(), m->d_src4, sizeof(int) * src.size(), cudaMemcpyDeviceToHost));
  const Node4 old = w[node];
  const int old_src[4] = {src[4 * node], src[4 * node + 1], src[4 * node + 2], src[4 * node + 3]};
  int link[4] = {old.child.x, old.child.y, old.child.z, old.child.w};
  link[slot] = child;
  int order[4], n = 0, ni = 0;
  for (int pass = 0; pass < 3; ++pass)  // internal, leaf, empty
    for (int k = 0; k < 4; ++k)
      if ((link[k] >= 0 ? 0 : (link[k] == kEmpty4 ? 2 : 1)) == pass) {
        order[n++] = k;
        if (pass == 0) ++ni;
      }
  if ((uint64_t)n4 + ni > std::max<uint32_t>(m->n_nodes, 1u))
    return fail(RMG_ERR_INVALID_ARG, "rmg_map_debug_set_child: no room for the changed node's children");
  Node4 nw = old;
  uint32_t leaves = 0;
  for (int j = 0; j < 4; ++j) {
    const int k = order[j];
    const float lo[3] = {(&old.lox.x)[k], (&old.loy.x)[k], (&old.loz.x)[k]};
    const float hi[3] = {(&old.hix.x)[k], (&old.hiy.x)[k], (&old.hiz.x)[k]};
    set_slot(nw, j, lo, hi);
    (&nw.child.x)[j] = j < ni ? (int)n4 + j : link[k];
    if (link[k] < 0 && link[k] != kEmpty4) leaves |= 1u << j;
    src[4 * node + j] = old_src[k];
  }
  nw.meta = make_int4((int)n4, (int)leaves | (((1 << ni) - 1) << 4), 0, 0);
  w[node] = nw;
  for (int j = 0; j < ni; ++j) {
    const int from = link[order[j]];
    w.push_back(Node4(w[from]));
    for (int k = 0; k < 4; ++k) src.push_back(int(src[4 * from + k]));
  }
  RMG_CUDA_TRY(cudaMemcpy(m->d_nodes4, w.data(), sizeof(Node4) * w.size(), cudaMemcpyHostToDevice));
  RMG_CUDA_TRY(cudaMemcpy(m->d_src4, src.data(), sizeof(int) * src.size(), cudaMemcpyHostToDevice));
  m->n_nodes4 = (uint32_t)w.size();
  return RMG_OK;
}

// Refreshes the wide boxes after the binary tree was refitted (asynchronous).
int wide_refit(rmg_map* m, cudaStream_t st) {
  if (!m->d_nodes4 || m->n_nodes4 == 0) return RMG_OK;
  k_wide_refit<<<(unsigned)((4ull * m->n_nodes4 + kBlock4 - 1) / kBlock4), kBlock4, 0, st>>>(m->d_nodes, m->d_src4,
                                                                                          m->n_nodes4, m->d_nodes4);
  const int s = cuda_status(cudaGetLastError(), "k_wide_refit");
  return s == RMG_OK ? wide8_refit(m, st) : s;
}

}  // namespace rmg
