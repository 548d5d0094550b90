// Per-camera summary of a finished sparse reconstruction, the part of
// cameras.json computed from the bundle-adjusted problem (sparse.rs:470-483
// and 515-533), and the f32 point copy stored in sparse.ply (mod.rs:31-35):
//
//  * neighbours: the cameras sharing the most points with each camera, best
//    first (the reference sorts a HashMap's entries by count, so the order
//    of equal counts is unspecified there; here it is ascending camera
//    index), at most `max_nb` of them (8 in sparse.rs:532);
//  * depth range: camera-frame depths z of the camera's observed points,
//    sorted by total order, (d[n/20] * 0.8, d[19n/20] * 1.25) when n >= 10,
//    else (0.3 agl, 3 agl) (sparse.rs:519-525);
//  * points as f32, rounded to nearest.
//
// Observations are grouped by camera with one stable radix sort; a CTA per
// camera walks its observations' points, counts co-observing cameras in a
// shared-memory histogram (global scratch when the camera count does not
// fit), picks the top entries by CTA-wide argmax, and selects the two depths.
#include <algorithm>
#include <cmath>
#include <vector>

#include "ba_gb300.h"
#include "context.cuh"
#include "primitives.cuh"
#include "select.cuh"

namespace ba {
namespace {

constexpr int kNbThreads = 512;
constexpr int kMaxNeighbours = 64;
constexpr int64_t kSmemHistCams = 24576;  // 96 KB of u32 counts

__global__ void check_obs_kernel(int64_t no, int64_t nc, int64_t np, const uint32_t* obs_cam,
                                 const uint32_t* obs_pt, uint32_t* err) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= no) return;
  if (obs_cam[i] >= (uint64_t)nc || obs_pt[i] >= (uint64_t)np) atomicOr(err, ERR_BAD_INDEX);
  if (i > 0 && obs_pt[i - 1] > obs_pt[i]) atomicOr(err, ERR_UNSORTED);
}

__global__ void cam_keys_kernel(int64_t no, const uint32_t* obs_cam, uint64_t* key,
                                uint32_t* idx) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= no) return;
  key[i] = obs_cam[i];
  idx[i] = (uint32_t)i;
}

__device__ __forceinline__ uint64_t block_max_u64(uint64_t v, uint64_t* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, (uint64_t)__shfl_xor_sync(kFull, v, o));
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    v = lane < kNbThreads / 32 ? red[lane] : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, (uint64_t)__shfl_xor_sync(kFull, v, o));
    if (lane == 0) red[kNbThreads / 32] = v;
  }
  __syncthreads();
  const uint64_t r = red[kNbThreads / 32];
  __syncthreads();
  return r;
}

struct CamArgs {
  int64_t nc;
  const uint32_t* cam_ptr;  // [nc + 1] into cam_obs
  const uint32_t* cam_obs;  // observation indices grouped by camera
  const uint32_t* pt_ptr;   // [np + 1] into the (point-sorted) observations
  const uint32_t* obs_cam;
  const uint32_t* obs_pt;
  const double* rot;
  const double* center;
  const double* points;
  double agl;
  int max_nb;
  uint32_t* hist_global;  // gridDim.x * nc counts when not in shared memory
  uint32_t keys;          // depth keys of a camera in shared memory
  uint64_t* key_global;   // [n_obs] depth keys of cameras beyond `keys`
  uint32_t* nb;           // [nc * max_nb], UINT32_MAX padded
  uint32_t* shared;       // [nc * max_nb], 0 padded
  int32_t* n_nb;          // [nc]
  double* range;          // [nc * 2]
};

// Depth keys of a camera in shared memory: where they and the counts leave room
// for one CTA an SM only (above some 12,000 cameras), the fewer (13,000 cameras
// of 60 observations: 1.91 -> 1.42 ms, of 2000: 10.2 -> 8.9 although their keys
// are then in global memory; 24,576 of 30: 3.79 -> 3.18).
constexpr uint32_t kDepthKeys = 8192, kDepthKeysFew = 1024;

// Camera-frame depth of a point, (R (X - C)).z with the products summed left
// to right and no fused multiply-add (Pose::to_cam, geometry.rs:57-59, as
// sparse.rs:476 uses it).  R: the third row.
__device__ __forceinline__ double depth_of(const double* R, const double* C, const double* X) {
  const double d0 = __dsub_rn(X[0], C[0]), d1 = __dsub_rn(X[1], C[1]),
               d2 = __dsub_rn(X[2], C[2]);
  return __dadd_rn(__dadd_rn(__dmul_rn(R[0], d0), __dmul_rn(R[1], d1)), __dmul_rn(R[2], d2));
}

// Persistent CTAs, one camera at a time, a thread per observation of the
// camera: the point's depth, and a count for every other camera of the point
// (sparse.rs:477-481: every ordered pair of distinct cameras of a point);
// then the largest counts by CTA-wide argmax, and the two depths of the range
// by selection (sparse.rs:519-525).
//
// Bound by the latency of the gathers (observation, point, track).  A warp
// per observation, its lanes over the six or seven cameras of the point, left
// 25 of 32 lanes idle (1.34 ms for 3.0 million observations of 500 cameras);
// the depths were sorted over all cameras, by value and then by camera, in
// nine passes (0.75 ms).  The whole summary of that survey: 2.68 -> 0.88 ms.
template <bool kSmem>
__global__ void __launch_bounds__(kNbThreads) camera_summary_kernel(CamArgs A) {
  extern __shared__ __align__(8) unsigned char smem_raw[];
  __shared__ uint64_t red[kNbThreads / 32 + 1];
  __shared__ uint32_t bytes[256], found[3];
  uint64_t* skey = reinterpret_cast<uint64_t*>(smem_raw);
  uint32_t* hist = kSmem ? reinterpret_cast<uint32_t*>(skey + A.keys)
                         : A.hist_global + (size_t)blockIdx.x * A.nc;
  for (int64_t c = threadIdx.x; c < A.nc; c += kNbThreads) hist[c] = 0;
  __syncthreads();
  for (int64_t a = blockIdx.x; a < A.nc; a += gridDim.x) {
    const uint32_t b = A.cam_ptr[a], n = A.cam_ptr[a + 1] - b;
    uint64_t* key = n <= A.keys ? skey : A.key_global + b;
    const double R[3] = {A.rot[9 * a + 6], A.rot[9 * a + 7], A.rot[9 * a + 8]};
    const double C[3] = {A.center[3 * a], A.center[3 * a + 1], A.center[3 * a + 2]};
    for (uint32_t i = threadIdx.x; i < n; i += kNbThreads) {
      const uint32_t p = A.obs_pt[A.cam_obs[b + i]];
      key[i] = total_order_key(depth_of(R, C, A.points + 3 * (size_t)p));
      const uint32_t e = A.pt_ptr[p + 1];
#pragma unroll 4
      for (uint32_t j = A.pt_ptr[p]; j < e; ++j) {
        const uint32_t o = A.obs_cam[j];
        if (o != (uint32_t)a) atomicAdd(&hist[o], 1u);
      }
    }
    __syncthreads();
    if (n >= 10) {
      const uint64_t lo = select_key<kNbThreads>(key, n, n / 20, bytes, found);
      const uint64_t hi =
          select_key<kNbThreads>(key, n, (uint32_t)((uint64_t)n * 19 / 20), bytes, found);
      if (threadIdx.x == 0) {
        A.range[2 * a] = from_total_order_key(lo) * 0.8;
        A.range[2 * a + 1] = from_total_order_key(hi) * 1.25;
      }
    } else if (threadIdx.x == 0) {
      A.range[2 * a] = A.agl * 0.3;
      A.range[2 * a + 1] = A.agl * 3.0;
    }
    int r = 0;
    for (; r < A.max_nb; ++r) {
      uint64_t best = 0;
      for (int64_t c = threadIdx.x; c < A.nc; c += kNbThreads) {
        const uint32_t h = hist[c];
        if (h) best = max(best, ((uint64_t)h << 32) | (uint32_t)(0xffffffffu - (uint32_t)c));
      }
      best = block_max_u64(best, red);
      if (best == 0) break;
      const uint32_t o = 0xffffffffu - (uint32_t)best;
      if (threadIdx.x == 0) {
        A.nb[a * A.max_nb + r] = o;
        A.shared[a * A.max_nb + r] = (uint32_t)(best >> 32);
        hist[o] = 0;
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      A.n_nb[a] = r;
      for (int q = r; q < A.max_nb; ++q) A.nb[a * A.max_nb + q] = 0xffffffffu, A.shared[a * A.max_nb + q] = 0;
    }
    for (int64_t c = threadIdx.x; c < A.nc; c += kNbThreads) hist[c] = 0;
    __syncthreads();
  }
}

__global__ void points_f32_kernel(int64_t n, const double* p, float* q) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) q[i] = __double2float_rn(p[i]);
}

int bit_width(uint64_t v) {
  int b = 0;
  while (v) ++b, v >>= 1;
  return b;
}

// Device outputs of one summary.
struct SummaryRun {
  DevBuf<uint32_t> err, pt_ptr, cam_ptr, cam_obs, nb, shared, hist;
  DevBuf<int32_t> n_nb;
  DevBuf<double> range;
  DevBuf<float> pts32;

  // All pointers are device pointers.
  void run(int64_t nc, int64_t np, int64_t no, const uint32_t* obs_cam, const uint32_t* obs_pt,
           const double* rot, const double* center, const double* points, int max_nb,
           double agl, int n_sm, cudaStream_t s) {
    if (max_nb < 1 || max_nb > kMaxNeighbours) throw BadInput("max_neighbours must be in 1..64");
    if (!std::isfinite(agl)) throw BadInput("agl must be finite");
    if (no > 0xfffffff0LL || np > 0xfffffff0LL || nc > 0xfffffff0LL)
      throw BadInput("too many cameras, points or observations for 32-bit indexing");
    auto A = [&](auto& d, int64_t n) { d.alloc(std::max<int64_t>(n, 1), s); };
    A(err, 1), A(pt_ptr, np + 1), A(cam_ptr, nc + 1), A(cam_obs, no);
    A(nb, nc * max_nb), A(shared, nc * max_nb), A(n_nb, nc), A(range, 2 * nc), A(pts32, 3 * np);
    err.zero();
    if (no > 0)
      BA_LAUNCH(check_obs_kernel<<<grid_for(no, 256), 256, 0, s>>>(no, nc, np, obs_cam, obs_pt, err));
    uint32_t e = 0;
    check(cudaMemcpyAsync(&e, err.p, 4, cudaMemcpyDeviceToHost, s), "d2h");
    check(cudaStreamSynchronize(s), "summary check");
    if (e & ERR_BAD_INDEX) throw BadInput("obs_cam or obs_pt out of range");
    if (e & ERR_UNSORTED) throw BadInput("observations must be sorted by point");
    if (np > 0) lower_bounds_u32(obs_pt, no, pt_ptr, np, s);
    {
      // Observations grouped by camera (stable: index order within a camera).
      DevBuf<uint64_t> key(std::max<int64_t>(no, 1), s), ktmp(std::max<int64_t>(no, 1), s);
      DevBuf<uint32_t> vtmp(std::max<int64_t>(no, 1), s);
      if (no > 0) {
        BA_LAUNCH(cam_keys_kernel<<<grid_for(no, 256), 256, 0, s>>>(no, obs_cam, key, cam_obs));
        radix_sort_u64_u32(key, cam_obs, ktmp, vtmp, no, bit_width(nc), s);
      }
      if (nc > 0) lower_bounds_u64(key, no, cam_ptr, nc, 1, s);
    }
    if (nc > 0) {
      const bool in_smem = nc <= kSmemHistCams;
      uint32_t keys = kDepthKeys;
      size_t smem = keys * 8 + (in_smem ? (size_t)nc * 4 : 0);
      auto kernel = in_smem ? camera_summary_kernel<true> : camera_summary_kernel<false>;
      // The limit belongs to the process: the same value from every call, so that
      // none lowers it between another thread's setting and its launch.
      check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(kDepthKeys * 8 + (in_smem ? kSmemHistCams * 4 : 0))),
            "summary smem");
      int occ = 0;
      check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, kNbThreads, smem),
            "occupancy");
      if (occ < 2) {
        keys = kDepthKeysFew, smem -= (kDepthKeys - kDepthKeysFew) * 8;
        check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, kNbThreads, smem),
              "occupancy");
      }
      const unsigned grid =
          (unsigned)std::min<int64_t>(nc, (int64_t)std::max(occ, 1) * std::max(n_sm, 1));
      if (!in_smem) A(hist, (int64_t)grid * nc);
      DevBuf<uint64_t> key(no > (int64_t)keys ? no : 1, s);
      CamArgs ca{nc,     cam_ptr, cam_obs, pt_ptr, obs_cam, obs_pt, rot,  center, points,
                 agl,    max_nb,  hist,    keys,   key,     nb,     shared, n_nb, range};
      BA_LAUNCH(kernel<<<grid, kNbThreads, smem, s>>>(ca));
    }
    if (np > 0) BA_LAUNCH(points_f32_kernel<<<grid_for(3 * np, 256), 256, 0, s>>>(3 * np, points, pts32));
  }

  void copy_out(int64_t nc, int64_t np, int max_nb, uint32_t* o_nb, uint32_t* o_shared,
                int32_t* o_n_nb, double* o_range, float* o_pts, cudaStream_t s) const {
    auto down = [&](auto* h, const auto& d, int64_t n) {
      if (h && n > 0) check(cudaMemcpyAsync(h, d.p, n * sizeof(*h), cudaMemcpyDefault, s), "copy out");
    };
    down(o_nb, nb, nc * max_nb), down(o_shared, shared, nc * max_nb), down(o_n_nb, n_nb, nc);
    down(o_range, range, 2 * nc), down(o_pts, pts32, 3 * np);
    check(cudaStreamSynchronize(s), "summary");
  }
};

int sm_count() {
  int dev = 0, n = 0;
  check(cudaGetDevice(&dev), "cudaGetDevice");
  check(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev), "attribute");
  return n;
}

}  // namespace
}  // namespace ba

using namespace ba;

extern "C" ba_status ba_sparse_summary(const ba_problem* problem, const ba_state* state,
                                       int32_t max_neighbours, double agl, void* stream,
                                       uint32_t* neighbours, uint32_t* shared,
                                       int32_t* n_neighbours, double* depth_range,
                                       float* points_f32) {
  return guarded([&] {
    if (!problem || !state) throw BadInput("null problem or state");
    const int64_t nc = problem->n_cams, np = problem->n_points, no = problem->n_obs;
    if (nc < 0 || np < 0 || no < 0) throw BadInput("negative size");
    if ((no > 0 && (!problem->obs_cam || !problem->obs_pt)) ||
        (nc > 0 && (!state->rot || !state->center)) || (np > 0 && !state->points))
      throw BadInput("null array");
    cudaStream_t s = (cudaStream_t)stream;
    auto A = [&](auto& d, int64_t n) { d.alloc(std::max<int64_t>(n, 1), s); };
    DevBuf<uint32_t> cam, pt;
    DevBuf<double> rot, center, points;
    A(cam, no), A(pt, no), A(rot, 9 * nc), A(center, 3 * nc), A(points, 3 * np);
    auto up = [&](auto& d, const auto* h, int64_t n) {
      if (n > 0) check(cudaMemcpyAsync(d.p, h, n * sizeof(*h), cudaMemcpyDefault, s), "copy in");
    };
    up(cam, problem->obs_cam, no), up(pt, problem->obs_pt, no);
    up(rot, state->rot, 9 * nc), up(center, state->center, 3 * nc), up(points, state->points, 3 * np);
    SummaryRun R;
    R.run(nc, np, no, cam, pt, rot, center, points, max_neighbours, agl, sm_count(), s);
    R.copy_out(nc, np, max_neighbours, neighbours, shared, n_neighbours, depth_range, points_f32, s);
  });
}

extern "C" ba_status ba_context_sparse_summary(ba_context* ctx, int32_t max_neighbours, double agl,
                                               uint32_t* neighbours, uint32_t* shared,
                                               int32_t* n_neighbours, double* depth_range,
                                               float* points_f32) {
  return guarded([&] {
    if (!ctx) throw BadInput("null context");
    if (!ctx->uploaded) throw BadInput("no problem uploaded");
    if (ctx->nm != 1) throw BadInput("the context must hold one model");
    check(cudaSetDevice(ctx->device), "cudaSetDevice");
    cudaStream_t s = ctx->stream;
    SummaryRun R;
    R.run(ctx->nc, ctx->np, ctx->no, ctx->obs_cam, ctx->obs_pt, ctx->rot, ctx->center,
          ctx->points, max_neighbours, agl, ctx->n_sm, s);
    R.copy_out(ctx->nc, ctx->np, max_neighbours, neighbours, shared, n_neighbours, depth_range,
               points_f32, s);
  });
}
