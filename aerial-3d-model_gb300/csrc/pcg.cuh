// Block-Jacobi preconditioned conjugate gradients on the reduced camera
// system (ba.rs:155-196), as one persistent cooperative kernel.
//
// Each model's block rows are split over a group of CTAs and, inside a CTA,
// over its warps: a warp owns whole block rows.  The reference's iteration
//     q = S p;  a = rz / p·q;  x += a p;  r -= a q;  stop if r·r < tol b·b;
//     z = M r;  β = r·z / rz;  p = z + β p
// needs three group-wide exchanges (p, p·q, r·r and r·z).  Here p is never
// exchanged: every lane keeps the previous p of the columns its blocks
// multiply (in shared memory beside the blocks) and forms p_j = z_j + β
// p_j(prev) on the fly, so an iteration exchanges z and the two reductions.
//
// Everything that crosses CTAs travels as 16-byte words that hold their own
// sequence number (one single-copy-atomic 128-bit access each): a reader
// polls the word itself until the number is the one it waits for.  An
// exchange is then one store and one load through L2 with no fence, no
// arrival counter and no second round trip for the values behind it, and the
// neighbours' z are gathered while the reductions are still on their way.
// Measured (FP64, per iteration; with a counter barrier and separate partials
// -> now): 500 cameras, 126 CTAs, 13.5 -> 11.5 µs; 77 cameras, 20 CTAs,
// 11.7 -> 9.0 µs; 12 cameras, 4 CTAs, 9.9 -> 7.0 µs (and 6.0 in halves, below).
//
// A CTA keeps its rows' state (x, r, z, p, q and the 6x6 block-Jacobi
// inverse) in shared memory for the whole solve, and its S blocks too when
// they fit; only the gathered neighbour z come from L2 each iteration.
//
// The lens block row of a model couples to every camera, so it is not
// multiplied by one warp: every camera row c adds S_cg^T p_c to a lens
// partial that travels with the p·q partial sums (S is symmetric).
//
// FP64 instructions on this GPU cost ~64 cycles per SM sub-partition whatever
// the number of active lanes, so the iteration is a chain of them: row vectors
// live one component per lane, reductions pack several values per
// instruction (p·q and the three lens components in the four groups of eight
// lanes), the totals are summed by one warp per value on different
// sub-partitions, and x, which nothing waits for, is updated while the last
// reduction is on its way.
//
// Inner products are FP64 and summed in a fixed order (fixed lane trees, CTA
// partials in rank order), so every CTA of a group sees bit-identical scalars
// and results do not depend on timing.  Models never wait on each other.
#pragma once

#include "lm_kernels.cuh"

namespace ba {

constexpr int kPcgThreads = 256;
constexpr int kPcgWarps = kPcgThreads / 32;

struct PcgJob {
  int32_t model, rank, gsize, base;  // base: first CTA of the group
  uint32_t row0, row1;               // this CTA's block rows
};

// A 16-byte word of an exchange: 8 bytes of value and a sequence number (R =
// float: three values and a 32-bit number).
struct __align__(16) PcgWord {
  unsigned long long v, tag;
};

// Words from one CTA's partials (one row's z) to the next's: a line that
// many CTAs write while many poll it is slow.  Measured, every CTA polling
// every other's partial (20 / 56 / 126 CTAs, two values, cycles per
// exchange): partials side by side 1710 / 2790 / 6570, 64 bytes apart
// 1770 / 1810 / 2290; pushed into an inbox per reader 2260 / 2660 / 4170.
constexpr int kPartPitch = 4;
// (a row's z: 96 of 128 bytes in FP64, 32 of 64 in FP32, whose rows 128 bytes
// apart took the same time: 250 cameras 21.7 ms, now 21.0)
template <typename R>
constexpr int kZRowWords = sizeof(R) == 8 ? 8 : 4;
constexpr int kSaidPitch = 8;

// Groups of up to this many CTAs: every CTA collects every partial and forms
// the totals itself (one hop).  Larger groups: the last CTA (it owns the lens
// row: the plan gives every CTA of a group rows) collects them, and the others
// wait for its result (two hops, but no polling of everything by everyone).  Measured with 2 / 4 values per
// exchange, cycles: 4 CTAs 970 / 1260 against 1920 / 1960; 126 CTAs 2100 /
// 3620 against 2740 / 2950, and CTAs that arrive early no longer slow the
// loads of those that are late (126 CTAs inside the solver: 7500 cycles from
// the last partial of p·q to its arrival everywhere).
constexpr int kDirectCtas = 32;

template <typename R>
struct PcgArgs {
  const PcgJob* jobs;
  const int32_t* cta_job0;  // [ncta+1]
  unsigned long long* epoch;  // [nm] last sequence number of each model's earlier launches
  PcgWord* part;              // [3][ncta][kPartPitch] partial sums of the three exchanges
  PcgWord* said;              // [nm][3][kSaidPitch] the leader's result of each exchange
  PcgWord* zx;                // [nb][kZRowWords<R>] z = M r, gathered by neighbours
  int32_t ncta;
  const uint32_t* row_ptr;
  const uint32_t* col_idx;
  const R* S;
  const R* pre;  // block-Jacobi inverses, computed in FP64, stored in R
  const R* b;
  R* x;
  R* pblk;  // [nz][6] p(prev) of blocks that shared memory does not hold (no memory of
            // its own: the sub-segments' sums, dead between assembly and the next Schur pass)
  const int32_t* lens_row;  // [nm]: the model's single lens block row, or -1
  const int32_t* lens_pos;  // [nb]: block index of (row, lens row), or -1
  const uint32_t* diag_pos; // [nb]: block index of the diagonal block
  uint32_t smem_rows;       // row-state capacity of the dynamic shared memory
  uint32_t smem_blocks;     // S blocks cached per CTA (the rest read from global)
  const int32_t* active;
  int32_t* iters;
  int32_t max_iter;
  double tol;
  unsigned* err;
  long long spin;    // spin limit of a group wait, in SM clock cycles
  int32_t hold_cta;  // fault injection: CTA hold_cta - 1 leaves before its first exchange (0: off)
  const int32_t* cap = nullptr;  // [nm] or null: per-model iteration cap (below max_iter)
};

// Partial-sum slots of the matrix-free kernel: 0,1 init (rz, bb) | 2..5 (pq,
// lens q 0..2) | 6,7 (rr, rz) | 8 (barrier) | 9..11 (lens terms).  Consecutive
// exchanges must use disjoint slots: a CTA may still be reading one
// exchange's partials while a faster one writes the next.
constexpr int kParts = 12;
// A reader lane loads up to kReadUnroll members' partials at once.
constexpr int kReadUnroll = 4;
constexpr int kMaxGroupCtas = 32 * kReadUnroll * 4;

// Row state per local row in shared memory: x, r, z, p, q (6 each), M (36),
// padded to a multiple of 16 bytes in both precisions.
constexpr int kRowState = 68;

// Dynamic shared memory: row state, cached S blocks with their columns'
// previous p and their column indices, and per row its block range and lens
// block (3 words).
template <typename R>
constexpr size_t pcg_block_bytes() {
  return 42 * sizeof(R) + 4;
}
template <typename R>
constexpr size_t pcg_smem_bytes(uint32_t rows, uint32_t blocks) {
  return (size_t)rows * kRowState * sizeof(R) + (size_t)blocks * pcg_block_bytes<R>() +
         (size_t)rows * 12;
}

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_add_release_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Warp sum of 8 values per lane by recursive halving: afterwards lane 4k
// (k < 8) holds the full sum of value k.  9 adds instead of 8 x 5.
template <typename T>
__device__ __forceinline__ void warp_sum8(T (&v)[8]) {
  const int lane = threadIdx.x & 31;
  {
    const bool up = lane & 16;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const T send = up ? v[i] : v[4 + i];
      const T recv = __shfl_xor_sync(kFull, send, 16);
      v[i] = (up ? v[4 + i] : v[i]) + recv;
    }
  }
  {
    const bool up = lane & 8;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const T send = up ? v[i] : v[2 + i];
      const T recv = __shfl_xor_sync(kFull, send, 8);
      v[i] = (up ? v[2 + i] : v[i]) + recv;
    }
  }
  {
    const bool up = lane & 4;
    const T send = up ? v[0] : v[1];
    const T recv = __shfl_xor_sync(kFull, send, 4);
    v[0] = (up ? v[1] : v[0]) + recv;
  }
  v[0] += __shfl_xor_sync(kFull, v[0], 2);
  v[0] += __shfl_xor_sync(kFull, v[0], 1);
}

// The same within every group of eight lanes, rolled.
__device__ __forceinline__ double sum8_rolled(double v) {
#pragma unroll 1
  for (int o = 1; o < 8; o *= 2) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// Sum over lanes 0..7 (lanes >= 8 must hold 0): result in lanes 0..7.
__device__ __forceinline__ double sum8(double v) {
  v += __shfl_xor_sync(kFull, v, 1);
  v += __shfl_xor_sync(kFull, v, 2);
  v += __shfl_xor_sync(kFull, v, 4);
  return v;
}

// N (<= 4) values per warp (held by lane 0) summed over the CTA's warps with
// one shuffle tree, then over the group's CTAs in rank order; every thread
// receives the totals in tot[].
//
// Group barrier: every member adds 1 to the group's monotonic 64-bit counter
// (release) after publishing its partials, and waits (acquire) until the
// counter reaches `target`, which grows by the group size per exchange from
// the launch's base value.  Only warp 0 of a CTA takes part; the partials are
// then read with all loads in flight at once.  Bounded: after A.spin cycles
// the waiter sets ERR_BARRIER_TIMEOUT; every CTA leaves at its next exchange.
// Args: any type with part, ncta, bar, err and spin as in PcgArgs.
template <int N, typename Args, typename Post>
__device__ __forceinline__ bool group_reduce(const double (&wv)[N], double* wsm, double* tot,
                                             const Args& A, const PcgJob& J, int slot,
                                             unsigned long long& target, Post&& post) {
  __shared__ int ok_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < 4; ++i) wsm[warp * 4 + i] = i < N ? wv[i < N ? i : 0] : 0.0;
  __syncthreads();
  if (warp == 0) {
    // lane = 4 w + i: warp w, value i; sum over w in a fixed tree.
    double c = wsm[lane];
    c += __shfl_xor_sync(kFull, c, 4);
    c += __shfl_xor_sync(kFull, c, 8);
    c += __shfl_xor_sync(kFull, c, 16);
    if (J.gsize == 1) {
      if (lane < N) tot[lane] = c;
      __syncwarp();
      if (lane == 0) {
        ok_s = 1;
        post();  // the iteration's scalars, once per CTA
      }
    } else {
      if (lane < N) A.part[(size_t)(slot + lane) * A.ncta + J.base + J.rank] = c;
      __threadfence();
      __syncwarp();
      int ok = 1;
      if (lane == 0) {
        target += (unsigned long long)J.gsize;
        unsigned long long* ctr = A.bar + J.model;
        red_add_release_u64(ctr, 1ULL);
        const long long t0 = clock64();
        while (ld_acquire_u64(ctr) < target) {
          if ((*(volatile unsigned*)A.err) & ERR_BARRIER_TIMEOUT) {
            ok = 0;
            break;
          }
          if (clock64() - t0 > A.spin) {
            atomicOr(A.err, ERR_BARRIER_TIMEOUT);
            ok = 0;
            break;
          }
        }
        ok_s = ok;
      }
      __syncwarp();
      double v[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      for (int k0 = 0; k0 < J.gsize; k0 += 32 * kReadUnroll) {
        double t[4][kReadUnroll];
#pragma unroll
        for (int u = 0; u < kReadUnroll; ++u) {
          const int k = k0 + lane + 32 * u;
#pragma unroll
          for (int i = 0; i < 4; ++i)
            t[i][u] = (i < N && k < J.gsize)
                          ? __ldcg(A.part + (size_t)(slot + i) * A.ncta + J.base + k)
                          : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kReadUnroll; ++u)
#pragma unroll
          for (int i = 0; i < 4; ++i) v[i] += t[i][u];
      }
      warp_sum8(v);  // lane 4i holds value i
      if ((lane & 3) == 0 && (lane >> 2) < N) tot[lane >> 2] = v[0];
      __syncwarp();
      if (lane == 0) post();  // the iteration's scalars, once per CTA
    }
  }
  __syncthreads();
  return ok_s != 0;
}

// Scalars of an iteration, computed once per CTA by thread 0 (FP64 division
// and conversions would otherwise run on every warp's FP64 pipe).
template <typename R>
struct PcgScalars {
  double rz, b2, beta, a;
  R beta_r, a_r;  // beta and a in storage precision
  int stop;
};

// A 6x6 block into registers with 16-byte loads (global or shared).
template <typename A>
__device__ __forceinline__ void load_block(const double* blk, A* m) {
  const double2* v = reinterpret_cast<const double2*>(blk);
#pragma unroll
  for (int i = 0; i < 18; ++i) {
    const double2 t = v[i];
    m[2 * i] = (A)t.x, m[2 * i + 1] = (A)t.y;
  }
}
template <typename A>
__device__ __forceinline__ void load_block(const float* blk, A* m) {
  const float4* v = reinterpret_cast<const float4*>(blk);
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    const float4 t = v[i];
    m[4 * i] = (A)t.x, m[4 * i + 1] = (A)t.y, m[4 * i + 2] = (A)t.z, m[4 * i + 3] = (A)t.w;
  }
}

// A row of such a block.
__device__ __forceinline__ void load_row6(const double* r, double (&m)[6]) {
  const double2* v = reinterpret_cast<const double2*>(r);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double2 t = v[i];
    m[2 * i] = t.x, m[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ void load_row6(const float* r, float (&m)[6]) {
  const float2* v = reinterpret_cast<const float2*>(r);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float2 t = v[i];
    m[2 * i] = t.x, m[2 * i + 1] = t.y;
  }
}

// p_j = z_j + β p_j(prev), the reference's update (ba.rs:192), in storage
// precision; the same expression for own rows and for gathered columns.
template <typename R>
__device__ __forceinline__ R p_of(R zj, R pj, R beta_r) {
  return (R)(zj + pj * beta_r);
}

// ---- exchange words -----------------------------------------------------------

__device__ __forceinline__ PcgWord ld_word(const PcgWord* p) {
  PcgWord w;
  asm volatile(
      "{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
      : "=l"(w.v), "=l"(w.tag)
      : "l"(p)
      : "memory");
  return w;
}
__device__ __forceinline__ void st_word(PcgWord* p, unsigned long long v,
                                        unsigned long long tag) {
  asm volatile(
      "{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(
          p),
      "l"(v), "l"(tag)
      : "memory");
}

// A waiter's limit: false once `spin` cycles have passed since `t0` (the
// error bit is set) or another waiter has given up.
__device__ __forceinline__ bool pcg_keep_waiting(unsigned* err, long long spin, long long t0) {
  if ((*(volatile unsigned*)err) & ERR_BARRIER_TIMEOUT) return false;
  if (clock64() - t0 > spin) {
    atomicOr(err, ERR_BARRIER_TIMEOUT);
    return false;
  }
  return true;
}

// A row's z in exchange words: FP64 one value a word, FP32 three.
__device__ __forceinline__ bool zx_load(const PcgWord* w, unsigned long long tag,
                                        double (&z)[6]) {
  bool ok = true;
  PcgWord t[6];
#pragma unroll
  for (int j = 0; j < 6; ++j) t[j] = ld_word(w + j);
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    ok &= t[j].tag == tag;
    z[j] = __longlong_as_double((long long)t[j].v);
  }
  return ok;
}
__device__ __forceinline__ bool zx_load(const PcgWord* w, unsigned long long tag, float (&z)[6]) {
  const PcgWord a = ld_word(w), b = ld_word(w + 1);
  z[0] = __uint_as_float((uint32_t)a.v), z[1] = __uint_as_float((uint32_t)(a.v >> 32));
  z[2] = __uint_as_float((uint32_t)a.tag);
  z[3] = __uint_as_float((uint32_t)b.v), z[4] = __uint_as_float((uint32_t)(b.v >> 32));
  z[5] = __uint_as_float((uint32_t)b.tag);
  return (uint32_t)(a.tag >> 32) == (uint32_t)tag && (uint32_t)(b.tag >> 32) == (uint32_t)tag;
}
// Store a row's z, component `c` of lane c < 6 (the whole warp calls).
__device__ __forceinline__ void zx_store(PcgWord* w, unsigned long long tag, double zi, int lane) {
  if (lane < 6) st_word(w + lane, (unsigned long long)__double_as_longlong(zi), tag);
}
__device__ __forceinline__ void zx_store(PcgWord* w, unsigned long long tag, float zi, int lane) {
  const int s = lane < 2 ? 3 * lane : 0;
  const uint32_t a = __float_as_uint(__shfl_sync(kFull, zi, s));
  const uint32_t b = __float_as_uint(__shfl_sync(kFull, zi, s + 1));
  const uint32_t c = __float_as_uint(__shfl_sync(kFull, zi, s + 2));
  if (lane < 2)
    st_word(w + lane, a | ((unsigned long long)b << 32),
            c | ((unsigned long long)(uint32_t)tag << 32));
}

// One value of an exchange, by one warp: the CTA's partial (its warps' values
// wsm[4 w + i], by a fixed tree), published, and, if `collect`, the total
// over the group's CTAs in rank order (lane l adds members l, l + 32, ...,
// then a fixed butterfly) in lane 0.  Clears *ok_s if a wait gives up.  Not inlined, and
// its loops rolled: see pcg_job on code size.
static __device__ __noinline__ double pcg_total(const double* wsm, int i, PcgWord* part, int rank,
                                                int gsize, bool collect, unsigned long long tag,
                                                unsigned* err, long long spin, int* ok_s) {
  const int lane = threadIdx.x & 31;
  // lane = 4 w + i: warp w, value i
  double v = wsm[lane];
#pragma unroll 1
  for (int o = 4; o <= 16; o *= 2) v += __shfl_xor_sync(kFull, v, o);
  v = __shfl_sync(kFull, v, i);
  if (gsize == 1) return v;
  if (lane == 0) st_word(part + rank * kPartPitch, (unsigned long long)__double_as_longlong(v), tag);
  if (!collect) return v;
  bool ok = true;
#pragma unroll 1
  for (int k0 = 0; k0 < gsize; k0 += 32 * kReadUnroll) {
    double t[kReadUnroll];
    unsigned need = 0;
#pragma unroll
    for (int u = 0; u < kReadUnroll; ++u) {
      t[u] = 0.0;
      if (k0 + lane + 32 * u < gsize) need |= 1u << u;
    }
    const long long t0 = clock64();
    int tries = 0;
    while (need) {
      PcgWord w[kReadUnroll];
#pragma unroll
      for (int u = 0; u < kReadUnroll; ++u)
        if ((need >> u) & 1u) w[u] = ld_word(part + (k0 + lane + 32 * u) * kPartPitch);
#pragma unroll
      for (int u = 0; u < kReadUnroll; ++u)
        if (((need >> u) & 1u) && w[u].tag == tag) {
          t[u] = __longlong_as_double((long long)w[u].v);
          need &= ~(1u << u);
        }
      if (need && (++tries & 31) == 0 && !pcg_keep_waiting(err, spin, t0)) {
        ok = false;
        break;
      }
    }
    __syncwarp();
    if (k0 == 0)
      v = t[0];
    else
      v += t[0];
#pragma unroll
    for (int u = 1; u < kReadUnroll; ++u)
      if (k0 + 32 * u < gsize) v += t[u];  // uniform over the warp
  }
  // The butterfly's upper levels would add zeros where the group is smaller.
#pragma unroll 1
  for (int o = 16; o > 0; o >>= 1)
    if (gsize > o) v += __shfl_xor_sync(kFull, v, o);
  if (!ok) *(volatile int*)ok_s = 0;
  return v;
}

static __device__ __noinline__ double pcg_quotient(double a, double b) { return a / b; }

// N (<= 4) values per warp, in wsm[4 warp + i], summed over the group into
// tot[] of the CTAs that decide (all of a small group's, else the last).
// Warp kPcgWarps - 1 - i takes value i (pcg_total): the values' warps sit on
// different SM sub-partitions, and the rows (warps 0, 1, ...) are not theirs
// unless a CTA holds more rows than it has other warps.  Warp kPcgWarps - 1
// then runs post(), which sets *out and *stop; where the last CTA decides,
// it publishes them and the others take them from there.  The other warps
// run idle() meanwhile.  False once a wait gave up.
constexpr unsigned long long kSaidStop = 1ULL << 63;  // the word's sequence number, or with this

template <typename R, typename Idle, typename Post>
__device__ __forceinline__ bool pcg_exchange(const PcgArgs<R>& A, const PcgJob& J, int n,
                                             double* wsm, double* tot, int* ok_s, R* out,
                                             int* stop, int slot, unsigned long long tag,
                                             Idle&& idle, Post&& post) {
  const int lane = threadIdx.x & 31, i = kPcgWarps - 1 - (int)(threadIdx.x >> 5);
  const bool direct = J.gsize <= kDirectCtas, leads = J.rank == J.gsize - 1;
  __syncthreads();
  if (i < n) {
    const double v = pcg_total(wsm, i, A.part + ((size_t)slot * A.ncta + J.base) * kPartPitch + i,
                               J.rank, J.gsize, direct || leads, tag, A.err, A.spin, ok_s);
    PcgWord* said = A.said + ((size_t)J.model * 3 + slot) * kSaidPitch;
    if (direct || leads) {
      if (lane == 0) tot[i] = v;
      asm volatile("bar.sync 1, %0;" ::"r"(32 * n) : "memory");
      if (i == 0) {
        post();
        if (!direct && lane == 0 && *(volatile int*)ok_s)
          st_word(said, (unsigned long long)__double_as_longlong((double)*out),
                  *stop ? tag | kSaidStop : tag);
      }
    } else if (i == 0 && lane == 0) {
      PcgWord w = ld_word(said);
      const long long t0 = clock64();
      for (int tries = 0; (w.tag & ~kSaidStop) != tag; w = ld_word(said))
        if ((++tries & 31) == 0 && !pcg_keep_waiting(A.err, A.spin, t0)) {
          *(volatile int*)ok_s = 0;
          break;
        }
      *out = (R)__longlong_as_double((long long)w.v);
      *stop = (w.tag & kSaidStop) != 0;
    }
  } else {
    idle();
  }
  __syncthreads();
  return *(volatile int*)ok_s != 0;
}

// Sum over the warp of six values per lane (as warp_sum8's tree: offsets 16,
// 8, 4, 2, 1): afterwards lane sum6_lane(k) holds the sum of value k.  Eight
// adds; six -> three -> two (one) -> one value per lane.
__host__ __device__ constexpr int sum6_lane(int k) { return k < 3 ? 4 * k : 4 * k + 4; }
// From the second step: lanes 0 .. 15 hold values 0, 1, 2 in a, the others 3, 4, 5.
template <typename T>
__device__ __forceinline__ T warp_sum3(const T (&a)[3]) {
  const int lane = threadIdx.x & 31;
  const bool u8 = lane & 8, u4 = lane & 4;
  // lower: values 0, 1 of the three; upper: value 2
  const T r0 = __shfl_xor_sync(kFull, u8 ? a[0] : a[2], 8);
  const T r1 = __shfl_xor_sync(kFull, a[1], 8);
  const T b0 = (u8 ? a[2] : a[0]) + r0, b1 = a[1] + r1;
  const T r2 = __shfl_xor_sync(kFull, u8 ? b0 : (u4 ? b0 : b1), 4);
  T c = (u8 ? b0 : (u4 ? b1 : b0)) + r2;
  c += __shfl_xor_sync(kFull, c, 2);
  c += __shfl_xor_sync(kFull, c, 1);
  return c;
}
template <typename T>
__device__ __forceinline__ T warp_sum6(const T (&v)[6]) {
  const bool u16 = threadIdx.x & 16;
  T a[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const T recv = __shfl_xor_sync(kFull, u16 ? v[i] : v[3 + i], 16);
    a[i] = (u16 ? v[3 + i] : v[i]) + recv;
  }
  return warp_sum3(a);
}

// Blocks that a CTA's rows multiply: all of theirs, but only the diagonal one
// of the model's single lens row (the last of its rows, -1: none).
__host__ __device__ inline uint32_t pcg_blocks(const uint32_t* row_ptr, const PcgJob& J,
                                               int32_t lens) {
  if (lens >= (int32_t)J.row0 && lens < (int32_t)J.row1)
    return row_ptr[lens] - row_ptr[J.row0] + 1;
  return row_ptr[J.row1] - row_ptr[J.row0];
}

// kAll: shared memory holds every S block of the CTA's rows.
//
// Code size: an iteration is one pass over code that each warp runs once, so
// straight-line code waits for its instruction fetches.  The FP64 form keeps
// its longest loop rolled (its overhead hides behind the FP64 operations) and
// shares the exchange and the division as functions: 3.6 µs of a 9.6 µs
// iteration went into two inlined exchanges before.
//
// kHalves (FP64, kAll; every row has up to 16 blocks): a block is in lanes l
// and l + 16, which take three of its rows each: half the operations of the
// product and one step less of the sum, whose first step would have added the
// zeros of lanes without a block.  12 cameras: 7.0 -> 6.0 µs an iteration.  A
// kernel of its own: in one with the other forms it cost those registers and
// instruction fetches (77 cameras: 9.0 -> 9.7 µs).
template <typename R, bool kAll, bool kHalves>
__device__ bool pcg_job(const PcgArgs<R>& A, const PcgJob& J, double* wsm, double* tot,
                        PcgScalars<R>& sc, int* ok_s, R* rs) {
  constexpr bool kWide = sizeof(R) == 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t nrows = J.row1 - J.row0;
  const uint32_t B0 = A.row_ptr[J.row0];
  const int32_t lens = A.lens_row[J.model];  // -1: no transposed lens row
  const bool lens_here = lens >= 0 && (uint32_t)lens >= J.row0 && (uint32_t)lens < J.row1;
  // The blocks that the CTA multiplies, numbered 0..nblk: its rows' blocks in
  // order; the lens row, last, uses only its diagonal block.  The first
  // ncached live in shared memory.
  const uint32_t nblk = pcg_blocks(A.row_ptr, J, lens);
  const uint32_t ncached = nblk < A.smem_blocks ? nblk : A.smem_blocks;
  const uint32_t lens_diag = lens_here ? A.diag_pos[lens] : 0u;
  auto blk = [&](uint32_t kk) {  // position in the matrix of block kk
    return lens_here && kk == nblk - 1 ? lens_diag : B0 + kk;
  };
  // Sequence numbers of this launch follow the earlier launches' (written by
  // rank 0 at their end).  Initial exchange: base + 1; iteration it: z and
  // p·q base + 2 + 2 it, r·r and r·z base + 3 + 2 it.
  const unsigned long long base = A.epoch[J.model];
  // Shared-memory carve-up: row state, then cached S blocks, their columns'
  // previous p and their columns.
  R* sS = rs + (size_t)A.smem_rows * kRowState;
  R* sP = sS + (size_t)A.smem_blocks * 36;
  uint32_t* sC = reinterpret_cast<uint32_t*>(sP + (size_t)A.smem_blocks * 6);
  int32_t* sM = reinterpret_cast<int32_t*>(sC + A.smem_blocks);
  {
    constexpr uint32_t kChunks = (uint32_t)(36 * sizeof(R) / 16);
    const float4* src = reinterpret_cast<const float4*>(A.S);
    float4* dst = reinterpret_cast<float4*>(sS);
    for (uint32_t c = threadIdx.x; c < ncached * kChunks; c += blockDim.x)
      dst[c] = src[(size_t)blk(c / kChunks) * kChunks + c % kChunks];
    for (uint32_t t = threadIdx.x; t < ncached; t += blockDim.x) sC[t] = A.col_idx[blk(t)];
    for (uint32_t t = threadIdx.x; t < ncached * 6; t += blockDim.x) sP[t] = (R)0;
    if constexpr (!kAll)
      for (uint32_t t = threadIdx.x; t < (nblk - ncached) * 6; t += blockDim.x)
        A.pblk[6 * (size_t)blk(ncached + t / 6) + t % 6] = (R)0;
    // Per row: its range of the CTA's blocks and its lens block (the lens
    // row's camera columns arrive through the camera rows' transposed terms).
    for (uint32_t lr = threadIdx.x; lr < nrows; lr += blockDim.x) {
      const uint32_t row = J.row0 + lr;
      const bool is_lens = (int32_t)row == lens;
      sM[3 * lr] = (int32_t)(A.row_ptr[row] - B0);
      sM[3 * lr + 1] = (int32_t)(is_lens ? nblk : A.row_ptr[row + 1] - B0);
      const int32_t lp = A.lens_pos[row];
      sM[3 * lr + 2] = is_lens || lp < 0 ? -1 : lp - (int32_t)B0;
    }
  }
  for (uint32_t t = threadIdx.x; t < nrows * 36; t += blockDim.x)
    rs[(t / 36) * kRowState + 30 + (t % 36)] = A.pre[36 * (size_t)J.row0 + t];
  if (threadIdx.x == 0) *ok_s = 1;
  __syncthreads();
  const bool vl = lane < 6;
  const int ci = vl ? lane : 0;
  // FP64: component ct of group g, so that one operation works on up to four
  // vectors of six.
  const int g = lane >> 3, t8 = lane & 7;
  const bool vt = t8 < 6;
  const int ct = vt ? t8 : 0;
  // row state: x 0..5 | r 6..11 | z 12..17 | p 18..23 | q 24..29 | M 30..65
#define ROW(lr) (rs + (size_t)(lr) * kRowState)
  auto col_of = [&](uint32_t k) { return kAll || k < ncached ? sC[k] : A.col_idx[blk(k)]; };
  auto p_at = [&](uint32_t k) {
    return kAll || k < ncached ? sP + 6 * (size_t)k : A.pblk + 6 * (size_t)blk(k);
  };
  auto s_at = [&](uint32_t k) {
    return kAll || k < ncached ? sS + 36 * (size_t)k : A.S + 36 * (size_t)blk(k);
  };

  // z of block column `col`: this CTA's rows from the row state (a CTA
  // barrier ago), others' from their exchange words.
  auto z_of = [&](uint32_t col, unsigned long long tag, R (&z)[6]) {
    const uint32_t l = col - J.row0;
    if (l < nrows) {
      const R* st = ROW(l);
#pragma unroll
      for (int j = 0; j < 6; ++j) z[j] = st[12 + j];
      return;
    }
    const PcgWord* w = A.zx + (size_t)col * kZRowWords<R>;
    if (zx_load(w, tag, z)) return;
    const long long t0 = clock64();
    int tries = 0;
    while (!zx_load(w, tag, z))
      if ((++tries & 31) == 0 && !pcg_keep_waiting(A.err, A.spin, t0)) {
        *(volatile int*)ok_s = 0;
        return;
      }
  };
  // The z of the warp's first 32 blocks are gathered while the reductions
  // before the product are on their way.
  R za[6];
  bool ahead = false;
  const int bl = kHalves ? lane & 15 : lane;  // the lane's block of a row's first
  auto gather_ahead = [&](unsigned long long tag) {
    if (warp >= (int)nrows) return;
    const uint32_t b0 = (uint32_t)sM[3 * warp], b1 = (uint32_t)sM[3 * warp + 1];
    const uint32_t k = b0 + bl;
    if (k < b1) z_of(col_of(k), tag, za);
    ahead = true;
  };

  // x = 0, r = b, z = M r, p(prev) = 0 (ba.rs:164-168; β = 0 gives p = z)
  double w2[2] = {0.0, 0.0};
  for (uint32_t lr = warp; lr < nrows; lr += kPcgWarps) {
    const uint32_t row = J.row0 + lr;
    R* st = ROW(lr);
    const R ri = vl ? A.b[6 * (size_t)row + ci] : (R)0;
    R zi = (R)0;
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      const R rj = __shfl_sync(kFull, ri, j);
      zi += st[30 + 6 * ci + j] * rj;
    }
    double a = 0.0, bb = 0.0;
    zx_store(A.zx + (size_t)row * kZRowWords<R>, base + 2, zi, lane);
    if (vl) {
      st[ci] = (R)0;
      st[6 + ci] = ri;
      st[12 + ci] = zi;
      st[18 + ci] = (R)0;
      a = (double)ri * (double)zi;
      bb = (double)ri * (double)ri;
    }
    w2[0] += sum8(a);
    w2[1] += sum8(bb);
  }
  if (lane == 0) wsm[4 * warp] = w2[0], wsm[4 * warp + 1] = w2[1];
  if (!pcg_exchange(
          A, J, 2, wsm, tot, ok_s, &sc.beta_r, &sc.stop, 0, base + 1,
          [&] { gather_ahead(base + 2); },
          [&] {
            if (lane == 0) {
              sc.rz = tot[0];
              sc.b2 = fmax(tot[1], 1e-300);
              sc.beta = 0.0;
              sc.beta_r = (R)0;
              sc.stop = 0;
            }
          }))
    return false;
  int32_t spmv = 0;
  const bool decides = J.gsize <= kDirectCtas || J.rank == J.gsize - 1;
  R plens = (R)0;  // last warp: component lane < 3 of the lens row's p
  const int32_t max_it = A.cap ? min(A.max_iter, A.cap[J.model]) : A.max_iter;
  for (int32_t it = 0; it < max_it; ++it) {
    const unsigned long long tag = base + 2 + 2 * (unsigned long long)it;
    const R beta = sc.beta_r;
    // q = S p (ba.rs:144-152) for the warp's rows.
    double wp = 0.0;                      // FP64: lanes 0, 8, 16, 24
    double w4[4] = {0.0, 0.0, 0.0, 0.0};  // FP32
    for (uint32_t lr = warp; lr < nrows; lr += kPcgWarps) {
      R* st = ROW(lr);
      const uint32_t b0 = (uint32_t)sM[3 * lr], b1 = (uint32_t)sM[3 * lr + 1];
      R q6;
      if constexpr (kHalves) {
        const uint32_t k = b0 + bl;
        R a3[3] = {0, 0, 0}, pp[6];
        if (k < b1) {
          if (ahead && lr == (uint32_t)warp) {
#pragma unroll
            for (int j = 0; j < 6; ++j) pp[j] = za[j];
          } else {
            z_of(col_of(k), tag, pp);
          }
          const R* pv = p_at(k);
#pragma unroll
          for (int j = 0; j < 6; ++j) pp[j] = p_of<R>(pp[j], pv[j], beta);
          const R* sb = s_at(k) + (lane >= 16 ? 18 : 0);
#pragma unroll 1
          for (int i = 0; i < 3; ++i) {
            R m[6];
            load_row6(sb + 6 * i, m);
            R s = (R)0;
#pragma unroll
            for (int j = 0; j < 6; ++j) s += m[j] * pp[j];
            a3[0] = a3[1], a3[1] = a3[2], a3[2] = s;
          }
        }
        __syncwarp();
        if (lane < 16 && k < b1) {  // both of its lanes have read the block's p
          R* pv = p_at(k);
#pragma unroll
          for (int j = 0; j < 6; ++j) pv[j] = pp[j];
        }
        q6 = warp_sum3(a3);
      } else {
        R acc[6] = {0, 0, 0, 0, 0, 0};
        for (uint32_t k = b0 + lane; k < b1; k += 32) {
          R pp[6];
          if (ahead && lr == (uint32_t)warp && k == b0 + lane) {
#pragma unroll
            for (int j = 0; j < 6; ++j) pp[j] = za[j];
          } else {
            z_of(col_of(k), tag, pp);
          }
          R* pv = p_at(k);
#pragma unroll
          for (int j = 0; j < 6; ++j) {
            pp[j] = p_of<R>(pp[j], pv[j], beta);
            pv[j] = pp[j];
          }
          const R* sb = s_at(k);
          // acc[i] of the rolled form is always the front of a queue
          constexpr int kUnroll = kWide ? 1 : 6;
#pragma unroll(kUnroll)
          for (int i = 0; i < 6; ++i) {
            R m[6];
            load_row6(sb + 6 * i, m);
            R s = acc[0];
#pragma unroll
            for (int j = 0; j < 6; ++j) s += m[j] * pp[j];
#pragma unroll
            for (int j = 0; j < 5; ++j) acc[j] = acc[j + 1];
            acc[5] = s;
          }
        }
        __syncwarp();
        q6 = warp_sum6(acc);
      }
      // own p = z + β p(prev); S_cg^T p_c of the row's lens block
      const int32_t lp = sM[3 * lr + 2];
      if constexpr (kWide) {
        const double qi = __shfl_sync(kFull, q6, sum6_lane(ct));
        const double pi = p_of<double>(st[12 + ct], st[18 + ct], beta);
        double v = 0.0;
        if (vt) {
          if (g == 0)
            v = qi;
          else if (lp >= 0)
            v = s_at((uint32_t)lp)[6 * ct + g - 1];
        }
        __syncwarp();
        if (vt && g == 0) {
          st[24 + ct] = qi;
          st[18 + ct] = pi;
        }
        v = sum8_rolled(__dmul_rn(v, pi));
        wp = lr < kPcgWarps ? v : wp + v;
      } else {
        const R qi = __shfl_sync(kFull, q6, sum6_lane(ci));
        const R pi = p_of<R>(st[12 + ci], st[18 + ci], beta);
        __syncwarp();
        if (vl) {
          st[24 + ci] = qi;
          st[18 + ci] = pi;
        }
        w4[0] += sum8(vl ? (double)pi * (double)qi : 0.0);
        // S_cg^T p_c for the lens column: lane 3t + j multiplies S_cg[t][j] p_t
        if (lp >= 0) {
          const int t = lane / 3, j = lane - 3 * (lane / 3);
          const R pt = __shfl_sync(kFull, pi, t < 6 ? t : 0);
          R v = (R)0;
          if (lane < 18) v = s_at((uint32_t)lp)[6 * t + j] * pt;
          v += __shfl_down_sync(kFull, v, 3);
          v += __shfl_down_sync(kFull, v, 6);
          v += __shfl_down_sync(kFull, v, 12);
          // lanes 0, 1, 2 hold the three components; every lane adds the same
          w4[1] += (double)__shfl_sync(kFull, v, 0);
          w4[2] += (double)__shfl_sync(kFull, v, 1);
          w4[3] += (double)__shfl_sync(kFull, v, 2);
        }
      }
    }
    if constexpr (kWide) {
      if (t8 == 0) wsm[4 * warp + g] = wp;
    } else if (lane == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) wsm[4 * warp + i] = w4[i];
    }
    ahead = false;
    if (lens >= 0 && warp == kPcgWarps - 1 && decides) {  // its share of p·q needs the lens row's p
      R zl[6];
      z_of((uint32_t)lens, tag, zl);
      __syncwarp();
      plens = p_of<R>(lane == 1 ? zl[1] : lane == 2 ? zl[2] : zl[0], plens, beta);
    }
    if (!pcg_exchange(A, J, 4, wsm, tot, ok_s, &sc.a_r, &sc.stop, 1, tag, [] {}, [&] {
          const R p0 = __shfl_sync(kFull, plens, 0), p1 = __shfl_sync(kFull, plens, 1),
                  p2 = __shfl_sync(kFull, plens, 2);
          if (lane != 0) return;
          double pq = tot[0];
          if (lens >= 0) {
            // The lens row's q: its diagonal product plus the transposed
            // partials; its share of p·q: p_g · (Σ S_cg^T p_c).
            pq += (double)p0 * tot[1] + (double)p1 * tot[2] + (double)p2 * tot[3];
            if (lens_here) {
              R* q = ROW((uint32_t)lens - J.row0) + 24;
              for (int c = 0; c < 3; ++c) q[c] = (R)((double)q[c] + tot[1 + c]);
            }
          }
          sc.stop = fabs(pq) < 1e-300 ? 1 : 0;  // ba.rs:174
          sc.a = sc.stop ? 0.0 : pcg_quotient(sc.rz, pq);
          sc.a_r = (R)sc.a;
        }))
      return false;
    ++spmv;
    if (sc.stop) break;
    const R a = sc.a_r;
    // x += a p, r -= a q, z = M r (ba.rs:178-188), one component per lane;
    // x waits for the exchange except on the warps that poll it.
    auto add_x = [&](uint32_t lr) {
      R* st = ROW(lr);
      if (vl) st[ci] = st[ci] + st[18 + ci] * a;
    };
    double w2b[2] = {0.0, 0.0};  // FP32
    double wr = 0.0;             // FP64: lane 0 r·r, lane 8 r·z
    for (uint32_t lr = warp; lr < nrows; lr += kPcgWarps) {
      const uint32_t row = J.row0 + lr;
      R* st = ROW(lr);
      if (warp >= kPcgWarps - 2) add_x(lr);
      const int c = kWide ? ct : ci;
      R ri = (R)0;
      if (kWide ? vt : vl) ri = st[6 + c] - st[24 + c] * a;
      R zi = (R)0;
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        const R rj = __shfl_sync(kFull, ri, j);
        zi += st[30 + 6 * c + j] * rj;
      }
      zx_store(A.zx + (size_t)row * kZRowWords<R>, tag + 2, zi, lane);
      if (vl) {
        st[6 + ci] = ri;
        st[12 + ci] = zi;
      }
      if constexpr (kWide) {
        const double v = sum8_rolled(vt ? __dmul_rn(ri, g == 0 ? ri : zi) : 0.0);
        wr = lr < kPcgWarps ? v : wr + v;
      } else {
        double rr = 0.0, rzl = 0.0;
        if (vl) {
          rr = (double)ri * (double)ri;
          rzl = (double)ri * (double)zi;
        }
        w2b[0] += sum8(rr);
        w2b[1] += sum8(rzl);
      }
    }
    if constexpr (kWide) {
      if (t8 == 0) wsm[4 * warp + g] = wr;
    } else if (lane == 0) {
      wsm[4 * warp] = w2b[0], wsm[4 * warp + 1] = w2b[1];
    }
    if (!pcg_exchange(
            A, J, 2, wsm, tot, ok_s, &sc.beta_r, &sc.stop, 2, tag + 1,
            [&] {
              gather_ahead(tag + 2);
              for (uint32_t lr = warp; lr < nrows; lr += kPcgWarps) add_x(lr);
            },
            [&] {
              if (lane != 0) return;
              sc.stop = tot[0] < A.tol * sc.b2 ? 1 : 0;  // ba.rs:182
              sc.beta = pcg_quotient(tot[1], sc.rz);       // ba.rs:189-190
              sc.beta_r = (R)sc.beta;
              sc.rz = tot[1];
            }))
      return false;
    if (sc.stop) break;
  }
  for (uint32_t lr = warp; lr < nrows; lr += kPcgWarps)
    if (vl) A.x[6 * (size_t)(J.row0 + lr) + ci] = ROW(lr)[ci];
#undef ROW
  if (J.rank == 0 && threadIdx.x == 0) {
    A.iters[J.model] = spmv;
    A.epoch[J.model] = base + 2 * (unsigned long long)spmv + 16;  // above every number used
  }
  __syncthreads();
  return true;
}

template <typename R, bool kHalves = false>
__global__ void __launch_bounds__(kPcgThreads, 2) pcg_kernel(PcgArgs<R> A) {
  __shared__ double wsm[kPcgWarps * 4];
  __shared__ double tot[4];
  __shared__ PcgScalars<R> sc;
  __shared__ int ok_s;
  extern __shared__ __align__(16) unsigned char pcg_smem[];
  R* rs = reinterpret_cast<R*>(pcg_smem);
  // Fault injection (tests of the timeout path): this CTA never arrives, so
  // the other members of its group give up after A.spin cycles.
  if (A.hold_cta > 0 && (int32_t)blockIdx.x == A.hold_cta - 1) return;
  for (int jb = A.cta_job0[blockIdx.x]; jb < A.cta_job0[blockIdx.x + 1]; ++jb) {
    const PcgJob J = A.jobs[jb];
    if (!A.active[J.model]) continue;
    if (J.row1 - J.row0 > A.smem_rows) {  // the planner never does this; fail loudly
      if (threadIdx.x == 0) atomicOr(A.err, ERR_STRUCTURE);
      return;
    }
    const bool all = pcg_blocks(A.row_ptr, J, A.lens_row[J.model]) <= A.smem_blocks;
    bool on;
    if constexpr (kHalves)
      on = pcg_job<R, true, true>(A, J, wsm, tot, sc, &ok_s, rs);
    else
      on = all ? pcg_job<R, true, false>(A, J, wsm, tot, sc, &ok_s, rs)
               : pcg_job<R, false, false>(A, J, wsm, tot, sc, &ok_s, rs);
    if (!on) return;
  }
}

// lens_pos[row] = index of the block (row, lens row of its model), or -1.
__global__ static void lens_pos_kernel(int64_t nb, const uint32_t* row_ptr,
                                       const uint32_t* col_idx, const uint32_t* blk_model,
                                       const int32_t* lens_row, int32_t* lens_pos) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nb) return;
  const int32_t L = lens_row[blk_model[r]];
  int32_t pos = -1;
  if (L >= 0 && L != (int32_t)r)
    for (uint32_t k = row_ptr[r]; k < row_ptr[r + 1]; ++k)
      if ((int32_t)col_idx[k] == L) {
        pos = (int32_t)k;
        break;
      }
  lens_pos[r] = pos;
}

}  // namespace ba
