// Fused simulate -> statistics: one launch casts the model scan at each
// estimated pose and reduces the ray-index correspondences with a dataset scan
// straight into CrossStatistics (and, optionally, the Umeyama transform).
//
// It replaces, per pose, the inner step of rmagine's RCC / MICP-L correction
// loop (tests/embree/correction_rcc.cpp:139-160):
//     sim.simulate(Tbm_est, model)                         // points, normals, hits
//     stats = statistics_p2l(Tpre, dataset, model, params) // statistics.cpp:84-126
//     T = umeyama_transform(stats)                         // optimization.cpp:12-49
// with the model bundle never written to memory.  Ray i of pose p pairs the
// dataset point i of the pose's scan (pre-transformed) with the model hit of
// ray i; the model side is valid when the ray hits with range >= range.min (the
// Hits attribute, the model mask of the RCC loop); the model point / normal are
// the Points / Normals attributes of the plain simulator bit for bit
// (hit_point / hit_normal in trace.cuh), and the pairing / filter arithmetic is
// that of the statistics kernels (stats.cuh).  Rays whose dataset point is
// masked out (mask == 0 or id != dataset_id) are not cast at all.
//
// Reduction: a warp casts one 32-ray tile at a time; the tile's correspondences
// are summed around the tile's first valid correspondence in binary32, then 16
// lanes turn the 16 sums into raw moments about the sensor origin in binary64
// (one moment per lane) and accumulate them over the warp's tiles.  A CTA adds its warps in a fixed order into one partial
// record; k_fused_final adds a pose's partials in a fixed order, forms the
// means and the covariance E[m d^T] - E[m] E[d]^T and runs Umeyama in binary64.
// Deterministic; the result differs from simulate + statistics only by the
// order of the binary32/binary64 additions (n_meas is exact).
#include "internal.h"
#include "linalg4.cuh"
#include "stats.cuh"
#include "trace.cuh"

namespace rmg {
namespace {

// Tiles (32 rays) that a warp reduces before its CTA writes one partial record.
// Fewer make more CTAs, of which the last, partly idle wave is a smaller part;
// more make fewer records and less final work.  8 / 4 / 2 / 1 tiles, us: 256 poses
// x 180 tiles 201 / 178 / 167 / 169, 1 pose 90 / 59 / 45 / 39, 48 x 656 416 / 291 /
// 230 / 212, 4,000 x 180 1,953 / 1,960 / 2,000 / 2,094, 300 x 4,096 3,993 / 3,998 /
// 4,093 / 4,322.  The number depends on the sensor alone, so that a pose's sums
// do not depend on how many poses a launch holds.
constexpr uint32_t tiles_per_warp(uint32_t tiles_per_pose) { return tiles_per_pose >= 1024 ? 4 : 2; }

struct FusedParams {
  TraceParams T;
  const float* dp;        // dataset points (float3), [n_scans][width*height]
  const uint8_t* dmask;   // may be NULL
  const uint32_t* dids;   // may be NULL
  uint64_t d_stride;      // rays per scan when every pose has its own scan, else 0
  const rmg_transform* pre;
  uint32_t pre_stride;    // 1: one pre-transform per pose, 0: one for every pose
  float max_dist;
  uint32_t dataset_id;
  uint32_t ctas_per_pose;
  uint32_t tiles_per_cta;
  double* partial;        // [n_poses * ctas_per_pose][16]
};

// Adds a tile's sums to the moments about the origin in binary64.  Lane 2 k (and
// its neighbour) holds moment k and x, the tile's (n, sum d', sum m', sum m' d'^T
// row-major) around the shift (sd, sm):
//   n, sum d = sum d' + n sd, sum m = sum m' + n sm,
//   sum m d^T = sum m' d'^T + (sum m') sd^T + sm (sum d)^T.
// A binary64 instruction takes 64 cycles for a warp, however many of its lanes
// are on, so every lane does the same three, on its own operands.  With branches
// on k there were some 15, and the 16 sums took 80 shuffles: 256 poses of 16 x 360
// rays 240 -> 235 us a call.
__device__ __forceinline__ double add_moment(double acc, float x, float n, const V& sd, const V& sm) {
  const uint32_t k = (threadIdx.x & 31) >> 1;
  const uint32_t e = k < 7 ? 0 : k - 7, i = e / 3, j = e - 3 * i;
  const float sum_mi = __shfl_sync(0xffffffffu, x, 2 * (4 + i));
  const float smi = i == 0 ? sm.x : (i == 1 ? sm.y : sm.z);
  const uint32_t c = k < 4 ? k - 1 : k < 7 ? k - 4 : j;
  const float b0 = k < 4 || k >= 7 ? sd.x : sm.x, b1 = k < 4 || k >= 7 ? sd.y : sm.y, b2 = k < 4 || k >= 7 ? sd.z : sm.z;
  const float b = k == 0 ? 0.f : c == 0 ? b0 : (c == 1 ? b1 : b2);
  const double y = fma((double)(k < 7 ? n : sum_mi), (double)b, (double)x);
  const double sum_dj = __shfl_sync(0xffffffffu, y, 2 * (1 + j));
  return acc + fma(k < 7 ? 0.0 : (double)smi, k < 7 ? 0.0 : sum_dj, y);
}

template <bool P2L, int OK, int SS, int TB>
__global__ void __maxnreg__((trace_regs<TB>())) k_trace_stats(const FusedParams F) {
  const TraceParams& P = F.T;
  const uint32_t pose = blockIdx.x / F.ctas_per_pose;
  const uint32_t cta = blockIdx.x - pose * F.ctas_per_pose;
  const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t W = P.sen.width, H = P.sen.height;
  // the pose's transforms wait in shared memory, not in registers, while rays walk
  __shared__ Tf s_tsm, s_pre;
  if (threadIdx.x == 0) s_tsm = tmul(load_tf(P.Tbm[pose]), P.Tsb);
  if (threadIdx.x == 32 % blockDim.x && F.pre) s_pre = load_tf(F.pre[F.pre_stride ? pose : 0]);
  __syncthreads();
  const uint64_t dbase = (uint64_t)pose * F.d_stride;
  const uint32_t tile_w = 1u << P.tile_w_log2;
  double acc = 0.0;
  const uint32_t t0 = cta * F.tiles_per_cta;
  const uint32_t t1 = min(P.tiles_per_pose, t0 + F.tiles_per_cta);
  for (uint32_t tile = t0 + wib; tile < t1; tile += nw) {  // warp-uniform
    const uint32_t ty = P.by_tiles_x(tile), tx = tile - ty * P.tiles_x;
    const uint32_t vid = ty * P.tile_h + (lane >> P.tile_w_log2);
    const uint32_t hid = tx * tile_w + (lane & (tile_w - 1));
    bool ok = false;
    V D{0.f, 0.f, 0.f}, M{0.f, 0.f, 0.f};
    if (vid < H && hid < W) {
      const uint32_t loc = visit_loc(P.sen, vid * W + hid);
      const uint64_t di = dbase + loc;
      if ((!F.dmask || F.dmask[di] != 0) && (!F.dids || F.dids[di] == F.dataset_id)) {
        Hit h;
        bool over = false;
        {
          V dir_s, orig_s, o, d;
          setup_ray<OK>(P.sen, reread(&s_tsm), loc, dir_s, orig_s, o, d);
          trace_ray<SS, TB>(P.map, o, d, P.sen.range_max, P.budget, h, over);
        }
        if (over) atomicExch(P.map.status, (unsigned)RMG_ERR_TRAVERSAL_BUDGET);
        if (h.tri >= 0 && h.t >= P.sen.range_min) {
          V dir_s, orig_s;
          reread_ray<OK>(P.sen, loc, dir_s, orig_s);
          const V mpt = hit_point<OK>(dir_s, orig_s, h.t);
          const V npt = P2L ? hit_normal(P.map, h, dir_s, reread(&s_tsm)) : V{0.f, 0.f, 0.f};
          const V dpt{__ldg(F.dp + 3 * di), __ldg(F.dp + 3 * di + 1), __ldg(F.dp + 3 * di + 2)};
          D = F.pre ? tf_point(reread(&s_pre), dpt) : dpt;
          ok = match<P2L>(D, mpt, npt, F.max_dist, M);
        }
      }
    }
    const unsigned bal = __ballot_sync(0xffffffffu, ok);
    if (bal == 0u) continue;
    const int src = __ffs(bal) - 1;
    const V sd{__shfl_sync(0xffffffffu, D.x, src), __shfl_sync(0xffffffffu, D.y, src),
               __shfl_sync(0xffffffffu, D.z, src)};
    const V sm{__shfl_sync(0xffffffffu, M.x, src), __shfl_sync(0xffffffffu, M.y, src),
               __shfl_sync(0xffffffffu, M.z, src)};
    float v[16];
    {
      const float dx = ok ? D.x - sd.x : 0.f, dy = ok ? D.y - sd.y : 0.f, dz = ok ? D.z - sd.z : 0.f;
      const float mx = ok ? M.x - sm.x : 0.f, my = ok ? M.y - sm.y : 0.f, mz = ok ? M.z - sm.z : 0.f;
      v[0] = ok ? 1.f : 0.f;
      v[1] = dx; v[2] = dy; v[3] = dz;
      v[4] = mx; v[5] = my; v[6] = mz;
      v[7] = mx * dx; v[8] = mx * dy; v[9] = mx * dz;
      v[10] = my * dx; v[11] = my * dy; v[12] = my * dz;
      v[13] = mz * dx; v[14] = mz * dy; v[15] = mz * dz;
    }
    const float x = warp_sums(v);
    acc = add_moment(acc, x, (float)__popc(bal), sd, sm);
  }
  __shared__ double red[16][8];
  if (!(lane & 1)) red[lane >> 1][wib] = acc;
  __syncthreads();
  if (threadIdx.x < 16) {
    double s = 0.0;
    for (uint32_t w = 0; w < nw; ++w) s += red[threadIdx.x][w];
    F.partial[16ull * blockIdx.x + threadIdx.x] = s;
  }
}

// One warp, one CTA per pose: each half warp adds moment k over every other
// partial record of the pose, in order; lane k forms mean or covariance element k,
// and the lanes, in groups of four, all solve the same problem.  The time is that
// of the chain: 256 poses 36 us with one lane doing the divisions and the solve, now 15.
__global__ void __launch_bounds__(32) k_fused_final(const double* partial, uint32_t ctas, rmg_cross_stats* stats,
                                                    rmg_transform* transforms) {
  const uint32_t pose = blockIdx.x, lane = threadIdx.x;
  double s = 0.0;
  const double* p = partial + 16ull * pose * ctas + (lane & 15u);
#pragma unroll 4
  for (uint32_t c = lane >> 4; c < ctas; c += 2) s += __ldg(p + 16ull * c);
  s += __shfl_xor_sync(0xffffffffu, s, 16);
  const double n = __shfl_sync(0xffffffffu, s, 0);
  const double x = n > 0.0 ? s / n : 0.0;  // lanes 1-6: the means, 7-15: E[m d^T]
  const uint32_t k = lane & 15u, e = k < 7 ? 0 : k - 7;
  const double mi = __shfl_sync(0xffffffffu, x, 4 + e / 3), dj = __shfl_sync(0xffffffffu, x, 1 + e % 3);
  const double cov = x - mi * dj;
  double dm[3], mm[3];
  M3d C;
#pragma unroll
  for (int i = 0; i < 3; ++i) { dm[i] = __shfl_sync(0xffffffffu, x, 1 + i); mm[i] = __shfl_sync(0xffffffffu, x, 4 + i); }
#pragma unroll
  for (int i = 0; i < 9; ++i) C.a[i / 3][i % 3] = __shfl_sync(0xffffffffu, cov, 7 + i);
  if (stats && lane == 0) store_cross_stats(n, dm, mm, &C.a[0][0], stats + pose);
  if (transforms) {
    double q[4], t[3];
    umeyama_lanes(C, dm, mm, (unsigned int)n, q, t);
    if (lane == 0) store_tf(transforms + pose, q, t);
  }
}

// out[i] = a[i or 0] * b[i or 0] (Transform::mult, Transform.tcc:34-42), exact order.
__global__ void k_compose(const rmg_transform* a, uint32_t a_stride, const rmg_transform* b, uint32_t b_stride,
                          rmg_transform* out, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Tf r = tmul(load_tf(a[a_stride ? i : 0]), load_tf(b[b_stride ? i : 0]));
  rmg_transform T;
  T.R = rmg_quat{r.R.x, r.R.y, r.R.z, r.R.w};
  T.t = rmg_vec3{r.t.x, r.t.y, r.t.z};
  T.stamp = 0;
  out[i] = T;
}

template <bool P2L, int OK>
cudaError_t launch_fused_ok(const FusedParams& F, unsigned grid, unsigned block, cudaStream_t st) {
  if (F.T.wide) {
    k_trace_stats<P2L, OK, 0, kWideTB><<<grid, block, 0, st>>>(F);
    return cudaGetLastError();
  }
  if (F.T.full_stack) {
    k_trace_stats<P2L, OK, kFullStack, 0><<<grid, block, 0, st>>>(F);
    return cudaGetLastError();
  }
  switch (F.T.trail_bits) {
    case 32: k_trace_stats<P2L, OK, 16, 32><<<grid, block, 0, st>>>(F); break;
    case 64: k_trace_stats<P2L, OK, 16, 64><<<grid, block, 0, st>>>(F); break;
    default: k_trace_stats<P2L, OK, 16, 128><<<grid, block, 0, st>>>(F); break;
  }
  return cudaGetLastError();
}

template <bool P2L>
cudaError_t launch_fused(const FusedParams& F, int kind, unsigned grid, unsigned block, cudaStream_t st) {
  switch (kind) {
    case RMG_MODEL_SPHERICAL:
    case RMG_MODEL_PINHOLE: return launch_fused_ok<P2L, ORIGIN_POSE>(F, grid, block, st);
    case RMG_MODEL_O1DN: return launch_fused_ok<P2L, ORIGIN_SINGLE>(F, grid, block, st);
    default: return launch_fused_ok<P2L, ORIGIN_TABLE>(F, grid, block, st);
  }
}

}  // namespace

int default_config(const rmg_sensor* s, rmg_launch_config* cfg);
int make_trace_params(const rmg_map* map, const rmg_sensor* sensor, const rmg_transform* Tsb,
                      const rmg_transform* Tbm, uint32_t n_poses, const rmg_outputs* out,
                      const rmg_launch_config& cfg, TraceParams& P, bool any_tile);

}  // namespace rmg

using namespace rmg;

extern "C" int rmg_simulate_statistics(const rmg_map* map, const rmg_sensor* sensor, const rmg_transform* Tsb,
                                       const rmg_transform* Tbm, uint32_t n_poses, const rmg_scan* dataset,
                                       const rmg_transform* pre_transforms, uint32_t pre_transform_stride,
                                       const rmg_umeyama_constraints* params, int point_to_plane,
                                       rmg_cross_stats* stats, rmg_transform* transforms, void* stream) {
  return guarded("rmg_simulate_statistics", [&]() -> int {
    if (!map || !sensor || !Tsb || !dataset || !params)
      return fail(RMG_ERR_INVALID_ARG, "rmg_simulate_statistics: NULL map, sensor, Tsb, dataset or params");
    if (n_poses == 0) return RMG_OK;
    if (!Tbm || !dataset->points) return fail(RMG_ERR_INVALID_ARG, "rmg_simulate_statistics: NULL Tbm or dataset points");
    if (!stats && !transforms) return fail(RMG_ERR_INVALID_ARG, "rmg_simulate_statistics: no output requested");
    rmg_launch_config cfg;
    default_config(sensor, &cfg);
    rmg_outputs out{};
    FusedParams F;
    make_trace_params(map, sensor, Tsb, Tbm, n_poses, &out, cfg, F.T, false);
    F.dp = reinterpret_cast<const float*>(dataset->points);
    F.dmask = dataset->mask;
    F.dids = dataset->ids;
    F.d_stride = dataset->per_pose ? (uint64_t)sensor->width * sensor->height : 0ull;
    F.pre = pre_transforms;
    F.pre_stride = pre_transform_stride ? 1u : 0u;
    F.max_dist = params->max_dist;
    F.dataset_id = params->dataset_id;
    F.tiles_per_cta = cfg.block_warps * tiles_per_warp(F.T.tiles_per_pose);
    F.ctas_per_pose = (F.T.tiles_per_pose + F.tiles_per_cta - 1) / F.tiles_per_cta;
    const uint64_t grid = (uint64_t)F.ctas_per_pose * n_poses;
    if (grid > 0x7fffffffull) return fail(RMG_ERR_INVALID_ARG, "rmg_simulate_statistics: too many rays for one launch");
    cudaStream_t st = as_stream(stream);
    double* partial = nullptr;
    int s = pool_alloc(&partial, 16 * (size_t)grid, st, "fused partials");
    if (s != RMG_OK) return s;
    F.partial = partial;
    const unsigned block = 32u * cfg.block_warps;
    const cudaError_t e = point_to_plane ? launch_fused<true>(F, sensor->model.kind, (unsigned)grid, block, st)
                                         : launch_fused<false>(F, sensor->model.kind, (unsigned)grid, block, st);
    s = cuda_status(e, "k_trace_stats");
    if (s == RMG_OK) {
      k_fused_final<<<n_poses, 32, 0, st>>>(partial, F.ctas_per_pose, stats, transforms);
      s = cuda_status(cudaGetLastError(), "k_fused_final");
    }
    pool_free(partial, st);
    return s;
  });
}

extern "C" int rmg_transforms_compose(const rmg_transform* a, uint32_t a_stride, const rmg_transform* b,
                                      uint32_t b_stride, rmg_transform* out, uint32_t n, void* stream) {
  return guarded("rmg_transforms_compose", [&]() -> int {
    if (n == 0) return RMG_OK;
    if (!a || !b || !out) return fail(RMG_ERR_INVALID_ARG, "rmg_transforms_compose: NULL argument");
    k_compose<<<(n + 255) / 256, 256, 0, as_stream(stream)>>>(a, a_stride, b, b_stride, out, n);
    return cuda_status(cudaGetLastError(), "k_compose");
  });
}
