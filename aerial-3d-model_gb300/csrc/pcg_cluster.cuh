// Block-Jacobi PCG of the reduced camera system (ba.rs:155-196) with one
// thread-block cluster per model and the whole solve in the cluster's
// distributed shared memory: mixed form only (FP32 matrix and vectors,
// double-float inner products).
//
// A model's block rows are split over the CTAs of its cluster (balanced by
// blocks); each CTA keeps its rows' state (x, r, z, two buffers of p, q and
// the block-Jacobi inverse) and its rows' S blocks in shared memory for the
// whole solve.  Every value another CTA needs is pushed to it: a CTA keeps a
// cache of the neighbour rows its blocks multiply (z_j and p_j), and each
// row's owner stores the row's new z into the caches of the CTAs that read it
// (a host-built subscriber list) before the cluster barrier after which they
// are read; every CTA then forms p_j = z_j + β p_j of its cached rows itself,
// once an iteration.  Remote loads would be round trips a
// warp waits on (~4.5k cycles when its lanes read from 16 CTAs); remote
// stores complete behind the barrier's release.  The two reductions of an
// iteration meet at hardware cluster barriers: no global memory traffic and
// no software spin inside the iteration.
//
// Two-level form (coarse correction z = B^-1 r + W E^-1 W^T r): the coarse
// vector of the next residual, w = W^T r_{k+1}, is formed as W^T r_k −
// α W^T q_k from group sums every CTA publishes before the iteration's first
// barrier (α is known right after it), so an iteration still needs only two
// cluster reductions: p·q (then α, the coarse gather and c = E^-1 w), and
// r·r with r·z (then β).  The coarse step runs on the warps beside warp 0
// after the p·q barrier, when every warp has formed α.
//
// S blocks beyond the shared memory are read every iteration: of 1200
// cameras 58 %, 220 KB a CTA, for which the loads of 16 bytes a lane at 144
// bytes' distance (a cache line a lane, and a small L1 beside 227 KB of shared
// memory) took half of the iteration.  They are turned once per solve into
// runs that a warp loads in whole lines: 29.2 -> 22.3 us per iteration (1200
// cameras, two levels, 16 CTAs).  A batch with more models than clusters of one CTA an SM
// runs two CTAs an SM on half the shared memory, the large models first: an
// iteration waits for its barriers most of the time, and a second cluster
// fills the wait.  32 models of 20 to 400 cameras, 12 CTAs each: 31.5 -> 20.7 ms
// of a solve's PCG.
//
// What is left is latency: three or four rows a warp, one after the other, and
// two exchanges.  A row of S p is a warp's work, a lane a block; what is six
// values a row (p.q, the update of x, r and z, their pushes) is done for five
// rows at a time, and p is formed per cached row instead of pushed and formed
// per block.  Two rows of S p at once in a warp's registers were slower (the
// longer code: 7.1 -> 7.6 ms).  Together 22.3 -> 15.8 us per iteration (1200
// cameras), 11.0 -> 9.0 us (500), 20.7 -> 18.8 ms (the batch).
//
// Every CTA of a cluster executes the same sequence of cluster barriers:
// loop exits depend only on reduced scalars, which every CTA computes from
// the same partials in the same order (bit-identical), and the kernel has no
// early return after its first barrier.
#pragma once

#include <cooperative_groups.h>

#include "coarse.cuh"
#include "pcg.cuh"

namespace ba {

namespace cgx = cooperative_groups;

// Threads per CTA: 512, or 1024 for a warp per block row where a CTA holds
// about 32 rows (the autotuner picks per problem shape).  The row loops take
// rows warp, warp + warps, ...; the reductions sum the warps' partials in a
// fixed order for either size.
constexpr int kCgThreads = 512;
constexpr int kCgThreadsWide = 1024;
constexpr int kCgMaxCluster = 16;
// Row state in floats: x r z p0 p1 q (6 each) | M (36) | the row's first and
// end block, its lens block, its coarse group slot and number of subscribers,
// its first subscriber (int bits).  Accessed one component per lane, or one
// row per lane (the pitch is odd: 32 rows in 32 banks).
constexpr int kCgX = 0, kCgR = 6, kCgZ = 12, kCgP = 18, kCgQ = 30, kCgM = 36, kCgIdx = 72;
constexpr int kCgPitch = 77;
// Floats of shared memory per row.
constexpr int kCgRow = 80;
// A block's column is one of the CTA's own rows when its slot carries this
// bit (the low bits are the local row), else a slot of the neighbour cache.
constexpr uint32_t kCgOwnRow = 0x80000000u;
// Neighbour cache in floats per slot: z, and in an array behind all slots' z
// the slot's p (6 each; read in pairs, 16 consecutive slots in 32 banks).
constexpr int kCgCache = 12;
// Rows that a warp takes at once where a row is six lanes' work.
constexpr int kCgLaneRows = 5;
// Which models a cluster serves (LmEngine::try_cluster) is a rule of their own
// sizes, not of what this kernel happens to need: 24 floats a neighbour slot, 4
// bytes a block's slot and a static part of 1616 + threads / 2 bytes beside the
// row state.  The kernel gets by with less, so that every model it serves fits;
// but with the kernel a model would change the layout of its sums, and the
// mixed form's end game, which depends on their rounding, its result.
constexpr int kCgCacheAsk = 24;
constexpr size_t cg_static_ask(int threads) { return 1616 + (size_t)threads / 2; }

struct CgJob {
  int32_t model;
  uint32_t row0, row1;  // this CTA's block rows
};

struct CgArgs {
  const CgJob* jobs;        // [grid]
  const uint32_t* row_loc;  // [nb]: owner rank << 16 | local row index
  const uint32_t* row_ptr;
  const uint32_t* col_idx;
  const float* S;
  const float* pre;
  const float* b;
  float* x;
  const int32_t* lens_row;  // [nm]
  const int32_t* lens_pos;  // [nb]
  const uint32_t* diag_pos; // [nb]
  uint32_t cap_rows;        // row-state capacity (same in every CTA)
  uint32_t cap_blocks;      // cached S blocks per CTA (the rest read from global)
  uint32_t cap_slots;       // blocks per CTA whose cache slot is in shared memory
  uint32_t cap_subs;        // subscriber entries per CTA in shared memory (0: read from global)
  const int32_t* active;
  int32_t* iters;
  int32_t max_iter;
  double tol;
  // Two-level (coarse) form only: see coarse.cuh.
  const float* W;            // [nb * 42]
  const float* Einv;         // per model, D x D
  const int64_t* model_eoff; // [nm]
  const int32_t* model_g0;   // [nm + 1]
  const int32_t* grp_row0;   // [groups]
  const int32_t* grp_row1;   // [groups]
  const int32_t* job_g0;     // [grid]: this CTA's groups [job_g0, job_g1)
  const int32_t* job_g1;
  const uint32_t* grp_loc;   // [groups]: owner rank << 16 | local group slot
  uint32_t cap_groups;       // group slots per CTA
  uint32_t cap_dim;          // largest model coarse dimension
  // Neighbour caches: the cache slot of every block's column in its row's
  // CTA, and per row the (CTA rank << 16 | slot) entries of the caches that
  // hold it.
  const uint32_t* blk_slot;  // [nz]
  const uint32_t* sub_ptr;   // [nb + 1]
  const uint32_t* sub_ent;
  uint32_t cap_cache;        // cache slots per CTA
  const int32_t* cap = nullptr;  // [nm] or null: per-model iteration cap (below max_iter)
  float* turned = nullptr;   // [nz * 36]: where the blocks that are not cached are turned
  const int32_t* order = nullptr;  // [grid / cluster]: the cluster's model, largest first
  unsigned* err = nullptr;   // device error bits (a staging wait that gave up)
  long long spin = 0;        // limit of that wait, in SM clock cycles
};

// The CTA's S blocks are one contiguous run of global memory (rows are
// consecutive, blocks row-major): one bulk asynchronous copy (the TMA engine,
// cp.async.bulk) brings them to shared memory while the threads stage the
// rest, completing on an mbarrier.  Both addresses are 16-byte aligned (a
// block is 144 bytes; the run and the shared row state before it are
// multiples of 16 bytes) and the size is a multiple of 16.
__device__ __forceinline__ void cg_bulk_stage(uint64_t* bar, float* dst, const float* src,
                                              uint32_t bytes) {
  const uint32_t b = (uint32_t)__cvta_generic_to_shared(bar);
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(d), "l"(src), "r"(bytes), "r"(b)
      : "memory");
}
// Wait for phase 0 of the staging mbarrier, at most `spin` cycles (<= 0: the
// default 4e9); false if it gave up.
__device__ __forceinline__ bool cg_bulk_wait(uint64_t* bar, long long spin) {
  const uint32_t b = (uint32_t)__cvta_generic_to_shared(bar);
  const long long limit = spin > 0 ? spin : 4000000000LL;
  const long long t0 = clock64();
  for (;;) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(b)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > limit) return false;
  }
}

// A block's cache slot as kept in shared memory: the CTA's own row in the low
// 15 bits under bit 15, else the slot (a slot takes 48 bytes and a row 320 of
// the same shared memory, so both numbers stay far below 2^15).
constexpr uint32_t kCgOwnSlot = 0x8000u;
__device__ __forceinline__ uint32_t cg_slot16(uint32_t e) {
  return ((e & kCgOwnRow) ? kCgOwnSlot : 0u) | (e & 0x7fffu);
}
// Slots in shared memory, in whole 16-byte words.
inline size_t cg_slot_bytes(uint32_t cap_slots) { return ((size_t)cap_slots * 2 + 15) / 16 * 16; }
inline size_t cg_smem_bytes(uint32_t cap_rows, uint32_t cap_blocks, uint32_t cap_cache,
                            uint32_t cap_slots, uint32_t cap_subs) {
  return (size_t)cap_rows * kCgRow * 4 + (size_t)cap_blocks * (36 * 4) +
         (size_t)cap_cache * kCgCache * 4 + cg_slot_bytes(cap_slots) + (size_t)cap_subs * 4;
}

// Extra shared memory of the two-level form, in floats: per row W (42); per
// own group its rows of E^-1 (7 x D) and c (7); the model's group sums of
// W^T r (two buffers by iteration parity: owners push the next one while the
// current one is read) and of W^T q (D each), pushed by every group's owner.
constexpr int kCgCoarseRowF = 42;
__host__ __device__ constexpr size_t cg_coarse_fixed_floats(uint32_t cap_groups,
                                                            uint32_t cap_dim) {
  return (size_t)cap_groups * (kCoarseModes * cap_dim + kCoarseModes) + 3 * (size_t)cap_dim;
}
inline size_t cg_coarse_smem_bytes(uint32_t cap_rows, uint32_t cap_groups, uint32_t cap_dim) {
  return ((size_t)cap_rows * kCgCoarseRowF + cg_coarse_fixed_floats(cap_groups, cap_dim)) * 4;
}

// Sum over lanes 0..7 (lanes >= 8 hold 0); lanes 0..7 receive it.
__device__ __forceinline__ float cg_sum8f(float v) {
  v += __shfl_xor_sync(kFull, v, 1);
  v += __shfl_xor_sync(kFull, v, 2);
  v += __shfl_xor_sync(kFull, v, 4);
  return v;
}

// Double-float numbers: hi + lo with |lo| <= ulp(hi) / 2, about 48 bits from
// FP32 instructions (on this GPU an FP64 warp instruction occupies its SM
// sub-partition for ~64 cycles).
struct DFloat {
  float hi, lo;
};
// Sum of two double-floats (Knuth's two-sum of the high parts, the low parts
// added to the error, renormalised).
__device__ __forceinline__ DFloat df_sum(DFloat a, DFloat b) {
  const float s = a.hi + b.hi;
  const float bb = s - a.hi;
  const float e = ((a.hi - (s - bb)) + (b.hi - bb)) + (a.lo + b.lo);
  const float hi = s + e;
  return DFloat{hi, e - (hi - s)};
}
// x y for FP32 x and a double-float y: the exact product x y.hi (split by an
// FMA) plus x y.lo.
__device__ __forceinline__ DFloat df_scale(float x, DFloat y) {
  const float p = x * y.hi;
  const float e = fmaf(x, y.hi, -p) + x * y.lo;
  const float hi = p + e;
  return DFloat{hi, e - (hi - p)};
}
__device__ __forceinline__ DFloat df_shfl_xor(DFloat v, int o) {
  return DFloat{__shfl_xor_sync(kFull, v.hi, o), __shfl_xor_sync(kFull, v.lo, o)};
}

// The cluster's totals from an inbox: lane r < cluster size (<= 16) of a
// half-warp holds CTA r's values, the others zeros, and a butterfly within
// each half-warp leaves totals in it: values 0 .. kIn - 1 in lanes 0..15, the
// rest in lanes 16..31 (one value: in both).  The loop is rolled: this runs on
// one warp between two barriers, where the fetch of straight-line code would
// take longer than the sums.
template <int N>
struct CgInbox {
  static constexpr int kIn = (N + 1) / 2;  // values per half-warp
  DFloat v[kIn];
  __device__ __forceinline__ CgInbox(const DFloat (*inbox)[4], int csize, int lane) {
    const int r = lane & 15, first = N > 1 ? kIn * (lane >> 4) : 0;
#pragma unroll
    for (int i = 0; i < kIn; ++i) v[i] = r < csize ? inbox[r][first + i] : DFloat{0.0f, 0.0f};
#pragma unroll 1
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < kIn; ++i) v[i] = df_sum(v[i], df_shfl_xor(v[i], o));
  }
  // Total i, in every lane.
  __device__ __forceinline__ DFloat total(int i) const {
    const int src = N > 1 && i >= kIn ? 16 : 0;
    const DFloat t = v[i % kIn];
    return DFloat{__shfl_sync(kFull, t.hi, src), __shfl_sync(kFull, t.lo, src)};
  }
};

// The totals of an inbox, in every thread.  Of
// 512 threads every warp sums the inbox: that saves the CTA barrier after it,
// and the 16 warps fetch the same instructions at the same time.  32 warps
// issue their sums for longer than the barrier takes: there warp 0 sums for
// all, and lane 0 runs post(v) before that barrier (77 cameras, four steps of
// 400 iterations without the coarse correction: every warp 11.95 ms, warp 0
// 10.6; 250 cameras 16.3 and 14.9).
template <int kThreads, int N, typename Post>
__device__ __forceinline__ void cg_totals(const DFloat (*inbox)[4], int csize, int lane,
                                          DFloat* tot, DFloat (&v)[N], Post&& post) {
  if constexpr (kThreads == kCgThreads) {
    const CgInbox<N> in(inbox, csize, lane);
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = in.total(i);
  } else {
    if (threadIdx.x < 32) {
      const CgInbox<N> in(inbox, csize, lane);
#pragma unroll
      for (int i = 0; i < N; ++i) {
        v[i] = in.total(i);
        if (lane == 0) tot[i] = v[i];
      }
      if (lane == 0) post(v);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = tot[i];
  }
}

// Inner products: a warp sums its rows' products in FP32 (a few rows of six
// components); the warps' partials are summed as double-floats over the CTA
// by warp 0, which pushes them to every CTA of the cluster, and after the
// cluster barrier the CTA's inbox is summed (cg_totals): the same partials
// in the same order everywhere, so every thread of the cluster holds
// bit-identical totals.  wv: N (<= 4) values held by lane 0 of every warp.
// While warp 0 sums and pushes, warps 1.. run side(w) with w = warp - 1 (the
// coarse group sums, which read the same row state after the same CTA
// barrier).
//
// Exchange by push: before the cluster barrier, lane r of warp 0 stores the
// CTA's partials into CTA r's inbox (inbox[source rank][value]); after it,
// every CTA reads its own inbox.  A warp that loads from many CTAs waits on
// each remote round trip (measured: ~4.5k cycles for one load per CTA of a
// 16-CTA cluster), while remote stores complete behind the barrier's
// release.  Consecutive exchanges use different inboxes: a CTA can only
// write inbox n + 2 after the barrier of exchange n + 1, which every reader
// of inbox n has passed.
template <int kWarps, int N, typename Side>
__device__ __forceinline__ void cg_exchange(cgx::cluster_group& cl, const float (&wv)[N],
                                            float* wsm, DFloat (*inbox)[4], Side&& side) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < 4; ++i) wsm[warp * 4 + i] = i < N ? wv[i < N ? i : 0] : 0.0f;
  __syncthreads();
  if (warp == 0) {
    // lane = 4 w + i: warps w, w + 8, ... (value i) in order, then over w in
    // a fixed tree
    static_assert(kWarps % 8 == 0 && kWarps >= 16 && kWarps <= 32, "2-4 warp partials per lane");
    DFloat c = df_sum(DFloat{wsm[lane], 0.0f}, DFloat{wsm[32 + lane], 0.0f});
#pragma unroll
    for (int h = 2; h < kWarps / 8; ++h) c = df_sum(c, DFloat{wsm[32 * h + lane], 0.0f});
#pragma unroll 1
    for (int o = 4; o < 32; o *= 2) c = df_sum(c, df_shfl_xor(c, o));
    DFloat v[N];
#pragma unroll
    for (int i = 0; i < N; ++i)
      v[i] = DFloat{__shfl_sync(kFull, c.hi, i), __shfl_sync(kFull, c.lo, i)};
    if (lane < (int)cl.num_blocks()) {
      DFloat* dst = cl.map_shared_rank(&inbox[0][0], (unsigned)lane) + 4 * cl.block_rank();
#pragma unroll
      for (int i = 0; i < N; ++i) dst[i] = v[i];
    }
  } else {
    side(warp - 1);
  }
  cl.sync();
}

// One output of the coarse step: sc[o] = (E^-1 w)_o for this CTA's (group,
// mode) output o, with the model's w = W^T r − α W^T q (wq null at the
// start: w = W^T b); a warp, then a fixed butterfly.
__device__ __forceinline__ void cg_coarse_dot(const float* sEi, uint32_t cap_dim, int D, int o,
                                              const float* wr, const float* wq, float alpha,
                                              float* sc) {
  const int lane = threadIdx.x & 31;
  const float* er = sEi + (size_t)o * cap_dim;
  float v = 0.0f;
  if (wq)
    for (int t = lane; t < D; t += 32) v += er[t] * (wr[t] - alpha * wq[t]);
  else
    for (int t = lane; t < D; t += 32) v += er[t] * wr[t];
#pragma unroll
  for (int q = 16; q > 0; q >>= 1) v += __shfl_xor_sync(kFull, v, q);
  if (lane == 0) sc[o] = v;
}

// A row's coarse share of z, (W c)_i for lane i < 6 (rows outside every
// group, such as the lens row, add nothing).
__device__ __forceinline__ float cg_row_wc(const float* sWrow, int32_t lg, const float* sc,
                                           int ci) {
  if (lg < 0) return 0.0f;
  const float* w = sWrow + kCoarseModes * ci;
  const float* c = sc + kCoarseModes * lg;
  float add = 0.0f;
#pragma unroll
  for (int j = 0; j < kCoarseModes; ++j) add += w[j] * c[j];
  return add;
}

// Per own group: the sum over its rows of W^T x, x the row-state vector at
// float offset `xoff`, pushed into the model-wide array `dst` (D floats, at
// this CTA's groups' offset) of every CTA.  A warp per (group, mode), warp
// `w` of kWorkers taking (group, mode) w, w + kWorkers, ...: lane l takes the
// group's rows (local rows grp[2 g] .. grp[2 g + 1]) l, l + 32, ... (each row's six products in component order), then a
// fixed butterfly.
__device__ __forceinline__ void cg_group_sum_push(cgx::cluster_group& cl, int o, const int* grp,
                                                  int32_t goff, const float* sW,
                                                  const float* rs, int xoff, float* dst) {
  const int lane = threadIdx.x & 31;
  const int csize = (int)cl.num_blocks();
  const int l = o / kCoarseModes, j = o % kCoarseModes;
  float v = 0.0f;
  for (int r = grp[2 * l] + lane; r < grp[2 * l + 1]; r += 32) {
    const float* w = sW + (size_t)r * 42 + j;
    const float* x = rs + (size_t)r * kCgPitch + xoff;
#pragma unroll
    for (int i = 0; i < 6; ++i) v += w[kCoarseModes * i] * x[i];
  }
#pragma unroll
  for (int q = 16; q > 0; q >>= 1) v += __shfl_xor_sync(kFull, v, q);
  if (lane < csize) cl.map_shared_rank(dst, (unsigned)lane)[goff + o] = v;
}
template <int kWorkers>
__device__ __forceinline__ void cg_group_sums_push(cgx::cluster_group& cl, int w, int32_t ngr,
                                                   const int* grp, int32_t goff, const float* sW,
                                                   const float* rs, int xoff, float* dst) {
  for (int o = w; o < ngr * kCoarseModes; o += kWorkers)
    cg_group_sum_push(cl, o, grp, goff, sW, rs, xoff, dst);
}

// Push a value x of a row, its component c, into z of the neighbour cache of
// every CTA that reads the row: its n subscribers.
__device__ __forceinline__ void cg_push_z(cgx::cluster_group& cl, float* cz, const uint32_t* sub,
                                          int n, float x, int c) {
#pragma unroll 4
  for (int t = 0; t < n; ++t) {
    const uint32_t e = sub[t];
    cl.map_shared_rank(cz, e >> 16)[(size_t)(e & 0xffffu) * 6 + c] = x;
  }
}
// A row's coarse group slot (-1: none), number of subscribers, and the first
// of them.
__device__ __forceinline__ int32_t cg_row_group(const float* st) {
  return (__float_as_int(st[kCgIdx + 3]) & 7) - 1;
}
__device__ __forceinline__ int cg_row_nsub(const float* st) {
  return __float_as_int(st[kCgIdx + 3]) >> 3;
}
__device__ __forceinline__ uint32_t cg_row_sub(const float* st) {
  return (uint32_t)__float_as_int(st[kCgIdx + 4]);
}

// A block's 36 values from a turned run of up to 32 blocks that starts at
// block c0 of a row that ends at block b1: this CTA's warps wrote them before
// the cluster barrier after the staging.
__device__ __forceinline__ void cg_load_turned(const float* turned, uint32_t c0, uint32_t b1,
                                               int i, float (&m)[36]) {
  const uint32_t n = b1 - c0 < 32u ? b1 - c0 : 32u;
  const float4* v = reinterpret_cast<const float4*>(turned) + (size_t)c0 * 9 + i;
#pragma unroll
  for (int t = 0; t < 9; ++t) {
    const float4 w = v[t * n];
    m[4 * t] = w.x, m[4 * t + 1] = w.y, m[4 * t + 2] = w.z, m[4 * t + 3] = w.w;
  }
}

template <bool kCoarse, int kThreads, int kCtas>
static __global__ void __launch_bounds__(kThreads, kCtas) pcg_cluster_kernel(CgArgs A) {
  constexpr int kCgWarps = kThreads / 32;
  __shared__ float wsm[kCgWarps * 4];
  __shared__ DFloat inbox[3][kCgMaxCluster][4];  // reduction inboxes (push)
  __shared__ DFloat tot[4];    // an exchange's totals (1024 threads)
  __shared__ float lens_p[4];  // the lens row's p, pushed by its owner
  __shared__ uint64_t stage_bar;  // completion of the S blocks' bulk copy
  extern __shared__ __align__(16) unsigned char cg_smem[];
  cgx::cluster_group cl = cgx::this_cluster();
  // clusters are 1-D: the cluster's CTAs are consecutive blocks
  const uint32_t csz = (uint32_t)cl.num_blocks();
  const uint32_t job = (uint32_t)A.order[blockIdx.x / csz] * csz + blockIdx.x % csz;
  const CgJob J = A.jobs[job];
  if (!A.active[J.model]) return;  // uniform over the cluster
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t nrows = J.row1 - J.row0;
  const uint32_t B0 = A.row_ptr[J.row0];
  const uint32_t nblk = A.row_ptr[J.row1] - B0;
  const uint32_t ncached = nblk < A.cap_blocks ? nblk : A.cap_blocks;
  const uint32_t sub0 = A.sub_ptr[J.row0], nsub = A.sub_ptr[J.row1] - sub0;
  const uint32_t nslots = nblk < A.cap_slots ? nblk : A.cap_slots;
  // Shared memory: row state | cached S blocks | neighbour cache | the
  // blocks' cache slots | the rows' subscribers | two-level form: W per row, E^-1 rows and c per own
  // group, the model's group sums of W^T r (two buffers) and W^T q.
  float* rs = reinterpret_cast<float*>(cg_smem);
  // behind the rows, in what their pitch leaves of kCgRow: the groups' first
  // and end local rows
  int* sGrp = reinterpret_cast<int*>(rs + (size_t)A.cap_rows * kCgPitch);
  float* sS = rs + (size_t)A.cap_rows * kCgRow;
  float* cz = sS + (size_t)A.cap_blocks * 36;
  float* cp = cz + (size_t)A.cap_cache * 6;
  uint16_t* sL = reinterpret_cast<uint16_t*>(cp + (size_t)A.cap_cache * 6);
  uint32_t* sSub = reinterpret_cast<uint32_t*>(sL + ((size_t)A.cap_slots + 7) / 8 * 8);
  float* sW = reinterpret_cast<float*>(sSub + A.cap_subs);
  float* sEi = sW + (size_t)A.cap_rows * 42;
  const size_t gsz = (size_t)A.cap_groups * kCoarseModes;
  float* scf = sEi + gsz * A.cap_dim;        // c, own outputs
  float* wall_r = scf + gsz;                  // [2][D]
  float* wall_q = wall_r + 2 * (size_t)A.cap_dim;  // [D]
  const int32_t cg0 = kCoarse ? A.job_g0[job] : 0;
  const int32_t ngr = kCoarse ? A.job_g1[job] - cg0 : 0;
  const int32_t goff = kCoarse ? kCoarseModes * (cg0 - A.model_g0[J.model]) : 0;
  const int32_t lens = A.lens_row[J.model];
  // the model's coarse dimension and this CTA's coarse outputs (two-level form)
  const int cD = kCoarse ? kCoarseModes * (A.model_g0[J.model + 1] - A.model_g0[J.model]) : 0;
  const int nco = kCoarseModes * ngr;
  {
    if (threadIdx.x == 0 && ncached > 0)
      cg_bulk_stage(&stage_bar, sS, A.S + (size_t)B0 * 36, ncached * 36u * 4u);
    for (uint32_t t = threadIdx.x; t < nslots; t += blockDim.x)
      sL[t] = (uint16_t)cg_slot16(A.blk_slot[B0 + t]);
    // p of the iteration before the first is 0 in every cached row; the z
    // values arrive by push after the first cluster barrier.
    if (A.cap_subs > 0)
      for (uint32_t t = threadIdx.x; t < nsub; t += blockDim.x) sSub[t] = A.sub_ent[sub0 + t];
    for (uint32_t t = threadIdx.x; t < A.cap_cache * kCgCache; t += blockDim.x) cz[t] = 0.0f;
    for (uint32_t t = threadIdx.x; t < nrows * 36; t += blockDim.x)
      rs[(size_t)(t / 36) * kCgPitch + kCgM + (t % 36)] = A.pre[36 * (size_t)J.row0 + t];
    // Per row: its block range (the lens row: its diagonal block only; its
    // camera columns arrive through the camera rows' transposed terms) and
    // the position of its lens block.
    for (uint32_t lr = threadIdx.x; lr < nrows; lr += blockDim.x) {
      const uint32_t row = J.row0 + lr;
      float* st = rs + (size_t)lr * kCgPitch;
      uint32_t b0 = A.row_ptr[row], b1 = A.row_ptr[row + 1];
      if ((int32_t)row == lens) b0 = A.diag_pos[row], b1 = b0 + 1;
      st[kCgIdx] = __int_as_float((int)b0);
      st[kCgIdx + 1] = __int_as_float((int)b1);
      st[kCgIdx + 2] = __int_as_float((int32_t)row == lens ? -1 : A.lens_pos[row]);
      int32_t lg = -1;  // local group slot (two-level form)
      if constexpr (kCoarse)
        for (int32_t l = 0; l < ngr; ++l)
          if ((int32_t)row >= A.grp_row0[cg0 + l] && (int32_t)row < A.grp_row1[cg0 + l]) lg = l;
      const uint32_t s0 = A.sub_ptr[row];
      st[kCgIdx + 3] = __int_as_float((int)(A.sub_ptr[row + 1] - s0) * 8 + lg + 1);
      st[kCgIdx + 4] = __int_as_float((int)(s0 - sub0));
    }
    if constexpr (kCoarse) {
      if ((int)threadIdx.x < 2 * ngr)
        sGrp[threadIdx.x] =
            ((threadIdx.x & 1) ? A.grp_row1 : A.grp_row0)[cg0 + threadIdx.x / 2] - (int)J.row0;
      for (uint32_t t = threadIdx.x; t < nrows * 42; t += blockDim.x)
        sW[t] = A.W[42 * (size_t)J.row0 + t];
      const int32_t gm0 = A.model_g0[J.model];
      const int D = kCoarseModes * (A.model_g0[J.model + 1] - gm0);
      const float* Ei = A.Einv + A.model_eoff[J.model];
      for (int t = threadIdx.x; t < ngr * kCoarseModes * D; t += blockDim.x) {
        const int o = t / D, col = t % D;
        sEi[(size_t)o * A.cap_dim + col] =
            Ei[(size_t)(kCoarseModes * (cg0 - gm0) + o) * D + col];
      }
    }
  }
  // The blocks that shared memory has no room for, turned once per solve: the
  // 32 blocks that a warp multiplies at a time lie block by block, and lanes
  // that each load one block's pieces touch 32 cache lines a load; turned,
  // piece t of the blocks side by side, a load is 512 bytes in a row.
  if (ncached < nblk) {
    __syncthreads();
    for (uint32_t lr = warp; lr < nrows; lr += kCgWarps) {
      const float* st = rs + (size_t)lr * kCgPitch;
      const uint32_t b0 = (uint32_t)__float_as_int(st[kCgIdx]);
      const uint32_t b1 = (uint32_t)__float_as_int(st[kCgIdx + 1]);
      for (uint32_t c0 = b0; c0 < b1; c0 += 32) {
        const uint32_t n = b1 - c0 < 32u ? b1 - c0 : 32u;
        if (c0 + n - B0 <= ncached) continue;
        const float4* src = reinterpret_cast<const float4*>(A.S) + (size_t)c0 * 9;
        float4* dst = reinterpret_cast<float4*>(A.turned) + (size_t)c0 * 9;
#pragma unroll
        for (int u = 0; u < 9; ++u) {
          const uint32_t e = 32 * u + lane;
          if (e < 9 * n) dst[(e % 9) * n + e / 9] = __ldg(src + e);
        }
      }
    }
  }
  // The S blocks' copy has landed: thread 0 waits on the mbarrier (the
  // cluster barrier below then orders the copy before every thread's reads).
  // A wait that gives up records the error; the kernel still runs its
  // barriers to the end, and the call fails.
  if (threadIdx.x == 0 && ncached > 0 && !cg_bulk_wait(&stage_bar, A.spin) && A.err)
    atomicOr(A.err, ERR_BARRIER_TIMEOUT);
  // Every CTA of the cluster has started (its shared memory is live for the
  // pushes below) and its staging is done.
  cl.sync();
  const bool lens_here = lens >= 0 && (uint32_t)lens >= J.row0 && (uint32_t)lens < J.row1;
  const bool vl = lane < 6;
  const int ci = vl ? lane : 0;
  // lane 6 g + c: row g and component c of kCgLaneRows rows at a time (lanes
  // 30 and 31 repeat row 0's first components and write nothing)
  const int gi = lane / 6, gb = gi < kCgLaneRows ? gi : 0, gc = lane - 6 * gi;
  const uint32_t* subs = A.cap_subs > 0 ? sSub : A.sub_ent + sub0;
#define CGROW(lr) (rs + (size_t)(lr) * kCgPitch)
  // x = 0, r = b, z = M r, p(prev) = 0 (ba.rs:164-168).  Inner products:
  // each lane accumulates its component's FP32 products over the warp's rows;
  // the lanes are summed once per phase.
  float drz = 0.0f, dbb = 0.0f;
  for (uint32_t lr = warp; lr < nrows; lr += kCgWarps) {
    float* st = CGROW(lr);
    const float ri = vl ? A.b[6 * (size_t)(J.row0 + lr) + ci] : 0.0f;
    float zi = 0.0f;
#pragma unroll
    for (int j = 0; j < 6; ++j) zi += st[kCgM + 6 * ci + j] * __shfl_sync(kFull, ri, j);
    if (vl) {
      st[kCgX + ci] = 0.0f;
      st[kCgR + ci] = ri;
      st[kCgZ + ci] = zi;
      st[kCgP + 6 + ci] = 0.0f;  // p buffer 1 = p(prev) of iteration 0
      drz += ri * zi;
      dbb += ri * ri;
    }
  }
  const float w2[2] = {cg_sum8f(drz), cg_sum8f(dbb)};
  // The iteration's scalars, in every thread: r.z, b.b and β in FP32 (the
  // precision of the vectors they scale).
  float rz, b2, bf = 0.0f;
  // r.z and b.b; the two-level form pushes the group sums of W^T b beside it
  // and forms c = E^-1 W^T b after the barrier (z = B^-1 b + W c below)
  cg_exchange<kCgWarps, 2>(cl, w2, wsm, inbox[1], [&](int w) {
    if constexpr (kCoarse)
      cg_group_sums_push<kCgWarps - 1>(cl, w, ngr, sGrp, goff, sW, rs, kCgR, wall_r);
  });
  {
    DFloat v[2];
    cg_totals<kThreads>(inbox[1], (int)csz, lane, tot, v, [](auto&) {});
    rz = v[0].hi, b2 = v[1].hi;
  }
  if constexpr (kCoarse) {
    for (int o = warp - 1; o >= 0 && o < nco; o += kCgWarps - 1)
      cg_coarse_dot(sEi, A.cap_dim, cD, o, wall_r, nullptr, 0.0f, scf);
    __syncthreads();
  }
  if constexpr (kCoarse) {
    // z = B^-1 b + W E^-1 W^T b, and r . z with it.
    float drz0 = 0.0f;
    for (uint32_t lr = warp; lr < nrows; lr += kCgWarps) {
      float* st = CGROW(lr);
      const int32_t lg = cg_row_group(st);
      const float add = cg_row_wc(sW + (size_t)lr * 42, lg, scf, ci);
      float zi = 0.0f;
      if (vl) {
        zi = st[kCgZ + ci] + add;
        st[kCgZ + ci] = zi;
        drz0 += st[kCgR + ci] * zi;
      }
      if (vl) cg_push_z(cl, cz, subs + cg_row_sub(st), cg_row_nsub(st), zi, ci);
    }
    const float w1[1] = {cg_sum8f(drz0)};
    cg_exchange<kCgWarps, 1>(cl, w1, wsm, inbox[2], [](int) {});
    DFloat v[1];
    cg_totals<kThreads>(inbox[2], (int)csz, lane, tot, v, [](auto&) {});
    rz = v[0].hi;
  } else {
    for (uint32_t lr = warp; lr < nrows; lr += kCgWarps) {
      const float* st = CGROW(lr);
      if (vl) cg_push_z(cl, cz, subs + cg_row_sub(st), cg_row_nsub(st), st[kCgZ + ci], ci);
    }
    cl.sync();  // z of iteration 0 in every cache
  }
  int32_t spmv = 0;
  const int32_t max_it = A.cap ? min(A.max_iter, A.cap[J.model]) : A.max_iter;
  for (int32_t it = 0; it < max_it; ++it) {
    const int cur = it & 1, prv = cur ^ 1;
    // p = z + β p of every cached row, once: the rows' owners push z only.
    if (A.cap_cache > 0) {
      for (uint32_t t = threadIdx.x; t < A.cap_cache * 6; t += kThreads) cp[t] = cz[t] + cp[t] * bf;
      __syncthreads();
    }
    // q = S p: a lane per block of a row.
    for (uint32_t lr = warp; lr < nrows; lr += kCgWarps) {
      float* st = CGROW(lr);
      const uint32_t b0 = (uint32_t)__float_as_int(st[kCgIdx]);
      const uint32_t b1 = (uint32_t)__float_as_int(st[kCgIdx + 1]);
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      for (uint32_t k = b0 + lane; k < b1; k += 32) {
        const uint32_t kk = k - B0;
        const uint32_t slot = kk < nslots ? sL[kk] : cg_slot16(__ldg(A.blk_slot + k));
        float m[36], pp[6];
        if (kk < ncached)
          load_block(sS + (size_t)kk * 36, m);
        else
          cg_load_turned(A.turned, k - lane, b1, lane, m);
        if (slot & kCgOwnSlot) {  // one of this CTA's rows: its row state
          const float* o = CGROW(slot & ~kCgOwnSlot);
#pragma unroll
          for (int j = 0; j < 6; ++j) pp[j] = o[kCgZ + j] + o[kCgP + 6 * prv + j] * bf;
        } else {
          const float2* pv = reinterpret_cast<const float2*>(cp + (size_t)slot * 6);
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            const float2 v = pv[j];
            pp[2 * j] = v.x, pp[2 * j + 1] = v.y;
          }
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) {
          float v = acc[i];
#pragma unroll
          for (int j = 0; j < 6; ++j) v += m[6 * i + j] * pp[j];
          acc[i] = v;
        }
      }
      warp_sum8(acc);  // lane 4i holds q_i
      if ((lane & 3) == 0 && lane < 24) st[kCgQ + (lane >> 2)] = acc[0];
    }
    __syncwarp();
    // p.q and the lens column's S_cg^T p_c, kCgLaneRows of the warp's rows at a
    // time: lane 6 g + c has component c of row g, and lanes 0..5 add the
    // rows' products in the rows' order.
    float dpq = 0.0f, dlens = 0.0f;
    for (uint32_t l0 = warp; l0 < nrows; l0 += kCgLaneRows * kCgWarps) {
      const uint32_t lr = l0 + gi * kCgWarps;
      const bool on = gi < kCgLaneRows && lr < nrows;
      float* st = CGROW(on ? lr : l0);
      const float qi = st[kCgQ + gc];
      const float pi = st[kCgZ + gc] + st[kCgP + 6 * prv + gc] * bf;
      if (on) st[kCgP + 6 * cur + gc] = pi;
      const int32_t lp = on ? __float_as_int(st[kCgIdx + 2]) : -1;
      float pt[6];
#pragma unroll
      for (int t = 0; t < 6; ++t) pt[t] = __shfl_sync(kFull, pi, 6 * gb + t);
      if (lens_here) {
        const unsigned at = __ballot_sync(kFull, on && (int32_t)(J.row0 + lr) == lens);
        if (at) {  // every CTA needs the lens row's p (its share of p.q): push it
          const int src = __ffs(at) - 1;
          const float p0 = __shfl_sync(kFull, pi, src), p1 = __shfl_sync(kFull, pi, src + 1),
                      p2 = __shfl_sync(kFull, pi, src + 2);
          if (lane < (int)csz) {
            float* dst = cl.map_shared_rank(lens_p, (unsigned)lane);
            dst[0] = p0, dst[1] = p1, dst[2] = p2;
          }
        }
      }
      float v = 0.0f;
      if (lp >= 0 && gc < 3) {  // S_cg^T p_c for the lens column
        const uint32_t kk = (uint32_t)lp - B0;
        const float* blk = (kk < ncached ? sS + (size_t)kk * 36 : A.S + (size_t)lp * 36) + gc;
        float w[6];
#pragma unroll
        for (int t = 0; t < 6; ++t) w[t] = __fmul_rn(blk[6 * t], pt[t]);
        v = (__fadd_rn(w[0], w[1]) + __fadd_rn(w[2], w[3])) + __fadd_rn(w[4], w[5]);
      }
#pragma unroll
      for (int g = 0; g < kCgLaneRows; ++g) {
        // (uniform; 512 threads have three or four rows a warp, and the test
        // there takes longer than it saves)
        if (kThreads == kCgThreadsWide && l0 + g * kCgWarps >= nrows) break;
        const float pg = __shfl_sync(kFull, pi, 6 * g + ci), qg = __shfl_sync(kFull, qi, 6 * g + ci);
        const float vg = __shfl_sync(kFull, v, 6 * g + ci);
        const int32_t lg = __shfl_sync(kFull, lp, 6 * g);
        if (l0 + g * kCgWarps < nrows) {
          if (vl) dpq += pg * qg;
          if (lg >= 0 && lane < 3) dlens += vg;  // lanes 0, 1, 2: components 0, 1, 2
        }
      }
    }
    const float w4[4] = {cg_sum8f(dpq), __shfl_sync(kFull, dlens, 0), __shfl_sync(kFull, dlens, 1),
                         __shfl_sync(kFull, dlens, 2)};
    // p.q; the two-level form pushes the group sums of W^T q beside it and,
    // after the barrier, forms c = E^-1 (W^T r − α W^T q) of the next
    // residual beside warp 0
    const float* wr_cur = wall_r + (size_t)cur * A.cap_dim;
    cg_exchange<kCgWarps, 4>(cl, w4, wsm, inbox[0], [&](int w) {
      if constexpr (kCoarse)
        cg_group_sums_push<kCgWarps - 1>(cl, w, ngr, sGrp, goff, sW, rs, kCgQ, wall_q);
    });
    float af;
    bool stop;
    {
      // The lens row's q gets the transposed camera terms; its share of p.q is
      // p_g . (sum S_cg^T p_c), with p_g pushed by its owner before the barrier.
      DFloat pq;
      auto lens_q = [&](int c, DFloat t) {
        float* q = CGROW((uint32_t)lens - J.row0) + kCgQ;
        q[c] = df_sum(DFloat{q[c], 0.0f}, t).hi;
      };
      if constexpr (kThreads == kCgThreads) {
        const CgInbox<4> in(inbox[0], (int)csz, lane);
        pq = in.total(0);
        if (lens >= 0) {
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const DFloat t = in.total(1 + c);
            pq = df_sum(pq, df_scale(lens_p[c], t));
            if (lens_here && threadIdx.x == 0) lens_q(c, t);
          }
        }
      } else {
        DFloat v[4];
        cg_totals<kThreads>(inbox[0], (int)csz, lane, tot, v, [&](auto& t) {
          if (lens_here)
            for (int c = 0; c < 3; ++c) lens_q(c, t[1 + c]);
        });
        pq = v[0];
        if (lens >= 0)
#pragma unroll
          for (int c = 0; c < 3; ++c) pq = df_sum(pq, df_scale(lens_p[c], v[1 + c]));
      }
      // ba.rs:174 breaks on a vanishing p.q; an FP32 quotient needs it normal
      stop = fabsf(pq.hi) < 1.17549435e-38f;
      af = stop ? 0.0f : rz / pq.hi;
    }
    if constexpr (kCoarse)
      for (int o = warp - 1; o >= 0 && o < nco; o += kCgWarps - 1)
        cg_coarse_dot(sEi, A.cap_dim, cD, o, wr_cur, wall_q, af, scf);
    ++spmv;
    if (stop) break;
    // c, and the lens row's q
    if (kCoarse || (kThreads == kCgThreads && lens_here)) __syncthreads();
    float drr = 0.0f, drz2 = 0.0f;
    for (uint32_t l0 = warp; l0 < nrows; l0 += kCgLaneRows * kCgWarps) {
      const uint32_t lr = l0 + gi * kCgWarps;
      const bool on = gi < kCgLaneRows && lr < nrows;
      float* st = CGROW(on ? lr : l0);
      const float xi = st[kCgX + gc] + st[kCgP + 6 * cur + gc] * af;
      const float ri = st[kCgR + gc] - st[kCgQ + gc] * af;
      float zi = 0.0f;
#pragma unroll
      for (int j = 0; j < 6; ++j) zi += st[kCgM + 6 * gc + j] * __shfl_sync(kFull, ri, 6 * gb + j);
      if constexpr (kCoarse) {
        // z = B^-1 r + W c
        zi += cg_row_wc(sW + (size_t)(on ? lr : l0) * 42, cg_row_group(st), scf, gc);
      }
      if (on) {
        st[kCgX + gc] = xi;
        st[kCgR + gc] = ri;
        st[kCgZ + gc] = zi;
        cg_push_z(cl, cz, subs + cg_row_sub(st), cg_row_nsub(st), zi, gc);
      }
#pragma unroll
      for (int g = 0; g < kCgLaneRows; ++g) {
        if (kThreads == kCgThreadsWide && l0 + g * kCgWarps >= nrows) break;
        const float rg = __shfl_sync(kFull, ri, 6 * g + ci), zg = __shfl_sync(kFull, zi, 6 * g + ci);
        if (vl && l0 + g * kCgWarps < nrows) {
          drr += rg * rg;
          drz2 += rg * zg;
        }
      }
    }
    const float w2b[2] = {cg_sum8f(drr), cg_sum8f(drz2)};
    // r.r and r.z; the two-level form pushes the group sums of the next
    // W^T r beside them
    cg_exchange<kCgWarps, 2>(cl, w2b, wsm, inbox[1], [&](int w) {
      if constexpr (kCoarse)
        cg_group_sums_push<kCgWarps - 1>(cl, w, ngr, sGrp, goff, sW, rs, kCgR,
                                         wall_r + (size_t)prv * A.cap_dim);
    });
    {
      DFloat v[2];
      cg_totals<kThreads>(inbox[1], (int)csz, lane, tot, v, [](auto&) {});
      const float rr = v[0].hi, rz1 = v[1].hi;
      bf = rz1 / rz;  // ba.rs:189-190
      rz = rz1;
      if (rr < (float)A.tol * b2) break;  // ba.rs:182
    }
  }
  for (uint32_t lr = warp; lr < nrows; lr += kCgWarps)
    if (vl) A.x[6 * (size_t)(J.row0 + lr) + ci] = CGROW(lr)[kCgX + ci];
#undef CGROW
  if (cl.block_rank() == 0 && threadIdx.x == 0) A.iters[J.model] = spmv;
  cl.sync();  // no CTA leaves while another may still read its shared memory
}

}  // namespace ba
