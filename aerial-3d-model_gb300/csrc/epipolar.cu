// Epipolar geometry ahead of bundle adjustment, on the device:
//
//  * fundamental-matrix RANSAC of every photo pair's putative matches
//    (ransac_fundamental, geometry.rs:248-300, called per pair at
//    sparse.rs:290 with threshold 1.5 px, 600 iterations, seed i*7919 + j);
//  * the pair check of the third round (pair_fits, sparse.rs:620-645): the
//    median Sampson error of a pair's matches under the current poses.
//
// RANSAC is split into its data-parallel parts.  Hypothesis samples depend
// on one xorshift stream per pair; a warp draws from 32 places of it at once
// and writes all of its pair's samples first.  Then a thread per hypothesis
// fits the normalised 8-point F (the null vector of its 8x9
// system, rank 2 by removing the smallest singular value); a warp counts a
// hypothesis' inliers over the pair's correspondences (FP32 with an
// error bound, FP64 near the threshold: the decisions are the FP64 ones); a
// CTA per pair takes the first hypothesis with the most inliers and refits on
// its inliers (normal matrix, smallest eigenvector).  Geometry in FP64, as
// the reference.
#include <algorithm>
#include <cmath>
#include <vector>

#include "ba_gb300.h"
#include "context.cuh"
#include "primitives.cuh"
#include "select.cuh"
#include "undistort.cuh"

namespace ba {
namespace {

constexpr double kF64Max = 1.7976931348623157e308;
constexpr int kFitThreads = 64;
constexpr int kCountThreads = 256;
constexpr int kRefitThreads = 128;
constexpr int64_t kMaxChunkHyp = int64_t(1) << 22;

// ---- shared device math -------------------------------------------------------

// normalise (geometry.rs:161-183) of side `side` (0: first photo, 1: second)
// of the eight correspondences idx[0..8): centroid as a running sum of p/8,
// mean distance to it, scale sqrt(2)/d.  Division by 8 is the exact
// multiplication by 0.125.  Writes the similarity T (row-major) and the
// centroid/scale (mx, my, s) used to map points on the fly.
__device__ void ep_normalise8(const double* uv, const uint32_t* idx, int side, double* T,
                              double& mx, double& my, double& s) {
  mx = 0.0, my = 0.0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const double* p = uv + 4 * (size_t)idx[i] + 2 * side;
    mx = mx + p[0] * 0.125;
    my = my + p[1] * 0.125;
  }
  double d = 0.0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const double* p = uv + 4 * (size_t)idx[i] + 2 * side;
    const double dx = p[0] - mx, dy = p[1] - my;
    d += sqrt(dx * dx + dy * dy);
  }
  d *= 0.125;
  s = d > 1e-12 ? 1.4142135623730951 / d : 1.0;
  T[0] = s, T[1] = 0.0, T[2] = -s * mx;
  T[3] = 0.0, T[4] = s, T[5] = -s * my;
  T[6] = 0.0, T[7] = 0.0, T[8] = 1.0;
}

__device__ __forceinline__ void mul3(const double* A, const double* B, double* C) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      C[3 * i + j] = A[3 * i] * B[j] + A[3 * i + 1] * B[3 + j] + A[3 * i + 2] * B[6 + j];
}

// a x + b y + c.  Fused throughout, or with the rounding of the products of
// the plain expression, two of the FP64 pipe's operations either way.
template <bool kFused>
__device__ __forceinline__ double affine(double a, double x, double b, double y, double c) {
  return kFused ? fma(a, x, fma(b, y, c)) : sum2(a, x, b, y) + c;
}

// sampson (geometry.rs:233-246).  The inlier tests take the fused form, for
// its shorter code in their kernels (the count 2.15 ms, with the other 2.46);
// the pair check, whose errors are results, keeps the plain expression's
// roundings.
template <bool kFused>
__device__ __forceinline__ double ep_sampson(const double* F, double ax, double ay, double bx,
                                             double by) {
  const double f0 = affine<kFused>(F[0], ax, F[1], ay, F[2]);
  const double f1 = affine<kFused>(F[3], ax, F[4], ay, F[5]);
  const double f2 = affine<kFused>(F[6], ax, F[7], ay, F[8]);
  const double g0 = affine<kFused>(F[0], bx, F[3], by, F[6]);
  const double g1 = affine<kFused>(F[1], bx, F[4], by, F[7]);
  const double e = affine<kFused>(bx, f0, by, f1, f2);
  const double d = fma(g1, g1, fma(g0, g0, sum2(f0, f0, f1, f1)));
  return d < 1e-18 ? kF64Max : quotient_by(mul_any(e, e), d, reciprocal_near(d));
}

// ---- RANSAC -------------------------------------------------------------------

struct RansacArgs {
  int64_t p0, np;  // pairs [p0, p0 + np) of this chunk
  const uint32_t* match_ptr;
  const double* uv;
  const uint64_t* seed;
  int iters;
  double t2;
  uint32_t* samples;  // [np * iters * 8]
  double* F;          // [np * iters * 9]
  float4* F32;        // [np * iters * 3] the same in FP32 (9 of 12 values)
  uint8_t* valid;     // [np * iters]
  int32_t* count;     // [np * iters]
  uint32_t* scratch;  // [n_matches] inlier index lists
  uint8_t* inlier;    // [n_matches]
  int32_t* n_inl;     // [n_pairs]
  int32_t* best;      // [n_pairs]
  uint8_t* refit;     // [n_pairs]
  uint32_t* err;
};

// A pair's draws are one sequential xorshift stream, but a step of it is a
// linear map of 64 bits, so a lane can start anywhere: lane l begins 64 l
// steps ahead (its five bits choose among the map's powers) and draws 64
// residues, 2048 a warp.  Samples then take eight residues each, 32 samples
// at a time, up to the first one with a repeated index (28 / n of them), which
// takes the distinct ones of the next 32.  A warp per pair; a thread per pair, one draw
// after the other, held 1603 pairs of 600 samples for 0.68 ms.
constexpr int kLaneDraws = 64;
constexpr int kDraws = 32 * kLaneDraws;

// m[k][b]: the state 64 2^k steps after the state with bit b alone.
struct DrawJump {
  uint64_t m[5][64];
};

__host__ __device__ __forceinline__ uint64_t xorshift64(uint64_t s) {
  s ^= s << 13;
  s ^= s >> 7;
  s ^= s << 17;
  return s;
}

const DrawJump& draw_jump() {
  static const DrawJump j = [] {
    DrawJump d;
    uint64_t t[64];
    for (int b = 0; b < 64; ++b) t[b] = xorshift64(uint64_t(1) << b);
    auto apply = [](const uint64_t* m, uint64_t v) {
      uint64_t r = 0;
      for (int b = 0; b < 64; ++b)
        if ((v >> b) & 1) r ^= m[b];
      return r;
    };
    for (int e = 0; e < 11; ++e) {  // t: 2^e steps
      if (e >= 6) std::copy(t, t + 64, d.m[e - 6]);
      uint64_t u[64];
      for (int b = 0; b < 64; ++b) u[b] = apply(t, t[b]);
      std::copy(u, u + 64, t);
    }
    return d;
  }();
  return j;
}

__global__ void __launch_bounds__(32) ransac_sample_kernel(RansacArgs A,
                                                           const __grid_constant__ DrawJump J) {
  __shared__ uint32_t buf[2 * kDraws];  // residues not used yet
  const int lane = threadIdx.x;
  const int64_t q = blockIdx.x, p = A.p0 + q;
  const uint32_t n = A.match_ptr[p + 1] - A.match_ptr[p];
  if (n < 12) return;
  uint64_t s = A.seed[p] | 1;  // state after the residues drawn so far
  uint4* out = reinterpret_cast<uint4*>(A.samples + (size_t)q * A.iters * 8);
  // s % n without a 64-bit division: with M = floor((2^64 - 1) / n),
  // umulhi(s, M) is floor(s / n) or one less, so one correction is exact.
  const uint64_t M = ~0ull / n;
  int have = 0, pos = 0;
  bool more = true;
  for (int it = 0; it < A.iters;) {
    if (more || have - pos < 8) {
      const int left = have - pos;
      if (left > kDraws) {  // a sample that 2048 draws do not fill: not with n >= 12
        if (lane == 0) atomicOr(A.err, ERR_STRUCTURE);
        for (; it + lane < A.iters; it += 32) {  // (the fit reads every sample)
          out[2 * (it + lane)] = make_uint4(0, 1, 2, 3);
          out[2 * (it + lane) + 1] = make_uint4(4, 5, 6, 7);
        }
        return;
      }
      for (int i0 = 0; i0 < left; i0 += 32) {  // to the front (pos >= 32, or the buffer is empty)
        const uint32_t v = i0 + lane < left ? buf[pos + i0 + lane] : 0u;
        __syncwarp();
        if (i0 + lane < left) buf[i0 + lane] = v;
        __syncwarp();
      }
      uint64_t t = s;
#pragma unroll 1
      for (int k = 0; k < 5; ++k) {
        uint64_t r = 0;
#pragma unroll 8
        for (int b = 0; b < 64; ++b) r ^= J.m[k][b] & (0ull - ((t >> b) & 1));
        if ((lane >> k) & 1) t = r;
      }
#pragma unroll 4
      for (int i = 0; i < kLaneDraws; ++i) {
        t = xorshift64(t);
        uint64_t r = t - __umul64hi(t, M) * n;
        if (r >= n) r -= n;
        buf[left + kLaneDraws * lane + i] = (uint32_t)r;
      }
      s = __shfl_sync(kFull, t, 31);
      have = left + kDraws, pos = 0, more = false;
      __syncwarp();
    }
    const int w = min(min(32, (have - pos) / 8), A.iters - it);
    uint32_t idx[8];
    bool dup = false;
    if (lane < w) {
#pragma unroll
      for (int j = 0; j < 8; ++j) idx[j] = buf[pos + 8 * lane + j];
#pragma unroll
      for (int j = 1; j < 8; ++j)
#pragma unroll
        for (int i = 0; i < j; ++i) dup |= idx[i] == idx[j];
    }
    const unsigned bad = __ballot_sync(kFull, dup);
    const int first = bad ? __ffs(bad) - 1 : w;
    if (lane < first) {
      out[2 * (it + lane)] = make_uint4(idx[0], idx[1], idx[2], idx[3]);
      out[2 * (it + lane) + 1] = make_uint4(idx[4], idx[5], idx[6], idx[7]);
    }
    it += first, pos += 8 * first;
    if (!bad) continue;
    // The sample with a repeated index: a lane per residue, of which it takes
    // the first eight that no earlier lane has.
    const uint32_t c = pos + lane < have ? buf[pos + lane] : 0xffffffffu;
    const unsigned same = __match_any_sync(kFull, c);
    unsigned fresh = __ballot_sync(kFull, pos + lane < have && lane == __ffs(same) - 1);
    if (__popc(fresh) >= 8) {
      const int rank = __popc(fresh & ((1u << lane) - 1u));
      if (((fresh >> lane) & 1u) && rank < 8) reinterpret_cast<uint32_t*>(out + 2 * it)[rank] = c;
      const unsigned eighth = __ballot_sync(kFull, ((fresh >> lane) & 1u) && rank == 7);
      ++it, pos += __ffs(eighth);
      continue;
    }
    // More than 32 residues: one after the other (every lane the same).
    int k = 0, d = pos;
    uint32_t got[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (; d < have && k < 8; ++d) {
      const uint32_t v = buf[d];
      bool again = false;
#pragma unroll
      for (int j = 0; j < 8; ++j) again |= (j < k) & (got[j] == v);
      if (!again) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j == k) got[j] = v;
        ++k;
      }
    }
    more = k < 8;  // ran out of residues: this sample begins again with more
    if (!more) {
      if (lane == 0) {
        out[2 * it] = make_uint4(got[0], got[1], got[2], got[3]);
        out[2 * it + 1] = make_uint4(got[4], got[5], got[6], got[7]);
      }
      ++it, pos = d;
    }
  }
}

// Symmetric 3x3 eigen-decomposition by cyclic Jacobi rotations (registers; the
// upper triangle of A is used, its diagonal returns the eigenvalues).  The
// rotation of (p, q) by the smaller angle, t = tan = 2 a / (|d| + sqrt(d^2 +
// 4 a^2)) with a = A_pq, d = A_qq - A_pp and the sign of a d, moves t a
// between the two diagonal entries (Golub and Van Loan, Matrix Computations,
// 8.5): some 46 FP64 operations where rotating rows and columns and dividing
// by 2 a took 81 (the fit of 1603 pairs by 600 samples: 3.24 -> 2.62 ms).  An
// off-diagonal entry below 1e-140 is left (A has a trace near 1 here, and
// the loop ends when they are below 1e-17).
__device__ void jacobi3(double (&A)[3][3], double (&V)[3][3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) V[i][j] = i == j ? 1.0 : 0.0;
  for (int sweep = 0; sweep < 50; ++sweep) {
    const double off = A[0][1] * A[0][1] + A[0][2] * A[0][2] + A[1][2] * A[1][2];
    const double diag = A[0][0] * A[0][0] + A[1][1] * A[1][1] + A[2][2] * A[2][2];
    if (off <= 1e-34 * diag || off == 0.0) break;
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
      for (int q = p + 1; q < 3; ++q) {
        const double a = A[p][q];
        if (fabs(a) < 1e-140) continue;
        const double d = A[q][q] - A[p][p], a2 = a + a;
        const double u = a2 * __drcp_rn(fabs(d) + sqrt(d * d + a2 * a2));
        const double t = d >= 0.0 ? u : -u;
        const double c = rsqrt(t * t + 1.0), sn = t * c;
        A[p][p] -= t * a;
        A[q][q] += t * a;
        A[p][q] = 0.0;
        const int r = 3 - p - q;
        double& rp = r < p ? A[r][p] : A[p][r];
        double& rq = r < q ? A[r][q] : A[q][r];
        const double x = rp, y = rq;
        rp = c * x - sn * y;
        rq = sn * x + c * y;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const double vkp = V[k][p], vkq = V[k][q];
          V[k][p] = c * vkp - sn * vkq;
          V[k][q] = sn * vkp + c * vkq;
        }
      }
  }
}

// Sum of a value that lanes 0 .. 8 of a warp hold (the others 0), in every lane.
__device__ __forceinline__ double sum9(double v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return __shfl_sync(kFull, v, 0);
}

// Eigenvector of the smallest eigenvalue of the symmetric positive
// semi-definite 9 x 9 matrix M (row-major, in shared memory, overwritten) by
// inverse iteration on its pivoted Cholesky factor.  A pivot below 1e-30
// trace(M) is raised to that floor, so an exactly singular M yields a null
// vector.  The reference takes this eigenvector from nalgebra's
// symmetric_eigen (geometry.rs:209-215); any accurate method gives it up to
// sign and rounding when the smallest eigenvalue is simple.
//
// By a warp: lane i < 9 has row i of the factor's column, of the solves and of
// the result x_i, which it returns; the 36 entries that a column changes are a
// lane's each (four of them a second one).  On one thread the same 1200
// operations and more took half of the pair's time.
__device__ double smallest_eigvec9(double* M) {
  const int lane = threadIdx.x & 31;
  const bool row = lane < 9;
  const int li = row ? lane : 0;
  // entries (ei, ej), 1 <= ej <= ei <= 8, number e = ei (ei - 1) / 2 + ej - 1
  int ei[2], ej[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    int e = lane + 32 * h;
    ei[h] = 1;
    while (e >= ei[h] && ei[h] < 9) e -= ei[h], ++ei[h];
    ej[h] = e + 1;  // (ei 9: none)
  }
  const double tr = sum9(row ? M[10 * li] : 0.0);
  const double floor_d = 1e-30 * tr + 1e-300;
  int perm = lane;      // column `lane` of the factor is x's entry perm
  double rdiag = 0.0;   // of row `lane`
  for (int k = 0; k < 9; ++k) {
    // The largest remaining diagonal entry, the first of equals (negative ones,
    // rounding's, count as zero: a positive double's bits are in its order).
    const double dk = row && lane >= k ? fmax(M[10 * li], 0.0) : 0.0;
    unsigned long long key = (unsigned long long)__double_as_longlong(dk);
    int pk = row && lane >= k ? lane : 31;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      const unsigned long long ok = __shfl_xor_sync(kFull, key, o);
      const int op = __shfl_xor_sync(kFull, pk, o);
      if (ok > key || (ok == key && op < pk)) key = ok, pk = op;
    }
    pk = __shfl_sync(kFull, pk, 0);
    if (pk != k) {  // symmetric swap of rows and columns k and pk
      if (row) {
        const double t = M[9 * k + li];
        M[9 * k + li] = M[9 * pk + li], M[9 * pk + li] = t;
      }
      __syncwarp();
      if (row) {
        const double t = M[9 * li + k];
        M[9 * li + k] = M[9 * li + pk], M[9 * li + pk] = t;
      }
      const int a = __shfl_sync(kFull, perm, k), b = __shfl_sync(kFull, perm, pk);
      perm = lane == k ? b : lane == pk ? a : perm;
      __syncwarp();
    }
    const double lkk = sqrt(fmax(M[10 * k], floor_d));
    const double rk = __drcp_rn(lkk);
    if (lane == k) rdiag = rk;
    __syncwarp();
    if (row && lane > k) M[9 * li + k] *= rk;
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (ei[h] < 9 && ej[h] > k) {
        const double v = M[9 * ei[h] + ej[h]] - M[9 * ei[h] + k] * M[9 * ej[h] + k];
        M[9 * ei[h] + ej[h]] = v, M[9 * ej[h] + ei[h]] = v;
      }
    __syncwarp();
  }
  // L in the lower triangle: P^T M P = L L^T.  The iterate in the factor's
  // order: lane i has entry perm of x.
  double x = row ? 1.0 - 0.0625 * perm : 0.0;
  x *= rsqrt(sum9(x * x));
  for (int it = 0; it < 60; ++it) {
    double y = x;
    for (int j = 0; j < 9; ++j) {  // L z = x
      const double z = __shfl_sync(kFull, y * rdiag, j);
      y = lane == j ? z : row && lane > j ? y - M[9 * li + j] * z : y;
    }
    for (int j = 8; j >= 0; --j) {  // L^T w = z
      const double w = __shfl_sync(kFull, y * rdiag, j);
      y = lane == j ? w : lane < j ? y - M[9 * j + li] * w : y;
    }
    y = row ? y : 0.0;
    y *= rsqrt(sum9(y * y));
    if (sum9(y * x) < 0.0) y = -y;
    const bool done = !row || fabs(y - x) <= 1e-15;
    x = y;
    if (__all_sync(kFull, done)) break;
  }
  // back to x's own order
  double out = 0.0;
  for (int j = 0; j < 9; ++j) {
    const double v = __shfl_sync(kFull, x, j);
    const int at = __shfl_sync(kFull, perm, j);
    if (lane == at) out = v;
  }
  return out;
}

// Rank 2, denormalisation and unit norm of the 8-point solution f
// (geometry.rs:216-229), as ep_fundamental does after its eigenvector.
__device__ bool ep_finish(const double* fm, const double* ta, const double* tb, double* F) {
  // Right singular vector of fm's smallest singular value: the eigenvector
  // of fm^T fm's smallest eigenvalue.
  double ftf[3][3], W[3][3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c)
      ftf[r][c] = fm[r] * fm[c] + fm[3 + r] * fm[3 + c] + fm[6 + r] * fm[6 + c];
  jacobi3(ftf, W);
  int j = 0;
  if (ftf[1][1] < ftf[j][j]) j = 1;
  if (ftf[2][2] < ftf[j][j]) j = 2;
  const double v0 = j == 0 ? W[0][0] : j == 1 ? W[0][1] : W[0][2];
  const double v1 = j == 0 ? W[1][0] : j == 1 ? W[1][1] : W[1][2];
  const double v2 = j == 0 ? W[2][0] : j == 1 ? W[2][1] : W[2][2];
  double f2[9];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const double fv = fm[3 * r] * v0 + fm[3 * r + 1] * v1 + fm[3 * r + 2] * v2;
    f2[3 * r] = fm[3 * r] - fv * v0;
    f2[3 * r + 1] = fm[3 * r + 1] - fv * v1;
    f2[3 * r + 2] = fm[3 * r + 2] - fv * v2;
  }
  double tbt[9], tmp[9], full[9];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) tbt[3 * r + c] = tb[3 * c + r];
  mul3(tbt, f2, tmp);
  mul3(tmp, ta, full);
  double nrm = 0.0;
#pragma unroll
  for (int i = 0; i < 9; ++i) nrm += full[i] * full[i];
  nrm = sqrt(nrm);
  if (!(nrm > 1e-15)) return false;
  const double rn = __drcp_rn(nrm);
#pragma unroll
  for (int i = 0; i < 9; ++i) F[i] = quotient_by(full[i], nrm, rn);
  return true;
}

// |x| rounded to FP32, as an integer in the same order (-1 for NaN): the FP64
// pipe, the bound of the fit, also executes the hardware's conversion.
__device__ __forceinline__ int magnitude_f32(double x) {
  const uint32_t hi = (uint32_t)__double2hiint(x) & 0x7fffffffu;
  if (hi - (898u << 20) < (252u << 20)) {  // well inside FP32's normal range
    const uint64_t b = ((uint64_t)(hi - (896u << 20)) << 32) | (uint32_t)__double2loint(x);
    return (int)((b + 0x0fffffffull + ((b >> 29) & 1)) >> 29);  // to nearest, ties to even
  }
  const float f = fabsf((float)x);
  return f == f ? __float_as_int(f) : -1;
}

// The 8-point hypothesis (geometry.rs:186-230 on eight correspondences).
// Its normal matrix M = A^T A has the null vector of the 8x9 system A as the
// eigenvector of its zero eigenvalue, which is the one the reference takes;
// here that null vector comes from A directly, by Gaussian elimination with
// full pivoting (about 500 operations instead of a 9x9 eigen-decomposition).
// The two agree to rounding for any sample of rank 8; for a rank-deficient
// sample both return some vector of the null space.  A lives in shared
// memory, element (r, c) at As[(9 r + c) * stride].
__device__ bool ep_fundamental8(const double* uv, const uint32_t* idx, double* As, int stride,
                                double* F) {
  double ta[9], tb[9], ax, ay, as, bx, by, bs;
  ep_normalise8(uv, idx, 0, ta, ax, ay, as);
  ep_normalise8(uv, idx, 1, tb, bx, by, bs);
#define AS(r, c) As[(9 * (r) + (c)) * stride]
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const double* u = uv + 4 * (size_t)idx[i];
    const double p0 = (u[0] - ax) * as, p1 = (u[1] - ay) * as;
    const double q0 = (u[2] - bx) * bs, q1 = (u[3] - by) * bs;
    AS(i, 0) = q0 * p0, AS(i, 1) = q0 * p1, AS(i, 2) = q0;
    AS(i, 3) = q1 * p0, AS(i, 4) = q1 * p1, AS(i, 5) = q1;
    AS(i, 6) = p0, AS(i, 7) = p1, AS(i, 8) = 1.0;
  }
  uint64_t perm = 0;  // 4 bits per column: original index of column k
#pragma unroll
  for (int c = 0; c < 9; ++c) perm |= (uint64_t)c << (4 * c);
  int rank = 8;
  double rpiv = 0.0;
  for (int k = 0; k < 8; ++k) {
    // Pivot choice on FP32 magnitudes (the choice only steers stability);
    // a zero pivot is tested exactly.
    int pr = k, pc = k, best = -1;
    for (int r = k; r < 8; ++r)
      for (int c = k; c < 9; ++c) {
        const int v = magnitude_f32(AS(r, c));
        if (v > best) best = v, pr = r, pc = c;
      }
    if (AS(pr, pc) == 0.0) {
      rank = k;
      break;
    }
    if (pr != k)
      for (int c = k; c < 9; ++c) {
        const double t = AS(k, c);
        AS(k, c) = AS(pr, c), AS(pr, c) = t;
      }
    if (pc != k) {
      for (int r = 0; r < 8; ++r) {
        const double t = AS(r, k);
        AS(r, k) = AS(r, pc), AS(r, pc) = t;
      }
      const uint64_t a = (perm >> (4 * k)) & 15, b = (perm >> (4 * pc)) & 15;
      perm &= ~((uint64_t)15 << (4 * k)) & ~((uint64_t)15 << (4 * pc));
      perm |= (b << (4 * k)) | (a << (4 * pc));
    }
    rpiv = __drcp_rn(AS(k, k));
    for (int r = k + 1; r < 8; ++r) {
      const double m = AS(r, k) * rpiv;
      for (int c = k + 1; c < 9; ++c) AS(r, c) -= m * AS(k, c);
    }
    if (k < 7) AS(k + 1, k) = rpiv;  // kept for the back-substitution
  }
  // Null vector: the free (last unpivoted) unknown is 1, the rest follow by
  // back-substitution through the upper-triangular rows 0..rank-1.
  double x[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) x[c] = c == rank ? 1.0 : 0.0;
  for (int k = rank - 1; k >= 0; --k) {
    double acc = 0.0;
    for (int c = k + 1; c < 9; ++c) acc += AS(k, c) * (c == rank ? 1.0 : (c < rank ? x[c] : 0.0));
    x[k] = quotient_by(-acc, AS(k, k), k < 7 ? AS(k + 1, k) : rpiv);
  }
#undef AS
  double fm[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) fm[c] = 0.0;
  for (int c = 0; c < 9; ++c) {
    const int o = (int)((perm >> (4 * c)) & 15);
#pragma unroll
    for (int t = 0; t < 9; ++t)
      if (t == o) fm[t] = x[c];
  }
  double nn = 0.0;
#pragma unroll
  for (int c = 0; c < 9; ++c) nn += fm[c] * fm[c];
  nn = sqrt(nn);
  const double rnn = __drcp_rn(nn);
#pragma unroll
  for (int c = 0; c < 9; ++c) fm[c] = quotient_by(fm[c], nn, rnn);
  return ep_finish(fm, ta, tb, F);
}

__global__ void __launch_bounds__(kFitThreads) ransac_fit_kernel(RansacArgs A) {
  __shared__ double As[72 * kFitThreads];
  const int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= A.np * A.iters) return;
  const int64_t p = A.p0 + h / A.iters;
  const uint32_t b = A.match_ptr[p], n = A.match_ptr[p + 1] - b;
  A.valid[h] = 0;
  if (n < 12) return;
  uint32_t idx[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) idx[j] = A.samples[8 * h + j];
  double F[9];
  if (!ep_fundamental8(A.uv + 4 * (size_t)b, idx, As + threadIdx.x, kFitThreads, F)) return;
#pragma unroll
  for (int j = 0; j < 9; ++j) A.F[9 * h + j] = F[j];
  float4* f = A.F32 + 3 * h;
  f[0] = make_float4((float)F[0], (float)F[1], (float)F[2], (float)F[3]);
  f[1] = make_float4((float)F[4], (float)F[5], (float)F[6], (float)F[7]);
  f[2] = make_float4((float)F[8], 0.0f, 0.0f, 0.0f);
  A.valid[h] = 1;
}

// Inlier test of one correspondence against one hypothesis, decided in FP32
// with a rounding-error bound and in FP64 (ep_sampson, as the reference) only
// when the FP32 value is too close to the threshold to be sure.  With
// u = 2^-24, each FP32 value x_hat of the test carries a bound dx on
// |x_hat - x| (x exact from the FP64 inputs): inputs rounded to FP32 and a
// three-term FMA dot product stay within 8u of the sum of the terms'
// magnitudes, and e = b^T F a, d = |(F a)_xy|^2 + |(F^T b)_xy|^2 propagate
// those.  "Surely in" means e^2 < t^2 d (1 - 32u) for every e, d in their
// intervals; "surely out" the converse; the FP64 evaluation's own error
// (about 2^-50 relative) is far inside those margins, so the decisions
// equal the FP64 ones.
struct Hyp32 {
  float f[9];
};

// 1: surely an inlier, 0: surely not, -1: evaluate in FP64.
__device__ __forceinline__ int inlier_fp32(const Hyp32& H, float4 c, float t2) {
  constexpr float u = 5.9604645e-8f;  // 2^-24
  const float* f = H.f;
  const float ax = c.x, ay = c.y, bx = c.z, by = c.w;
  const float f0 = fmaf(f[0], ax, fmaf(f[1], ay, f[2]));
  const float f1 = fmaf(f[3], ax, fmaf(f[4], ay, f[5]));
  const float f2 = fmaf(f[6], ax, fmaf(f[7], ay, f[8]));
  const float g0 = fmaf(f[0], bx, fmaf(f[3], by, f[6]));
  const float g1 = fmaf(f[1], bx, fmaf(f[4], by, f[7]));
  const float af = fabsf(ax), ag = fabsf(ay), bf = fabsf(bx), bg = fabsf(by);
  const float d0 = 8.0f * u * fmaf(fabsf(f[0]), af, fmaf(fabsf(f[1]), ag, fabsf(f[2])));
  const float d1 = 8.0f * u * fmaf(fabsf(f[3]), af, fmaf(fabsf(f[4]), ag, fabsf(f[5])));
  const float d2 = 8.0f * u * fmaf(fabsf(f[6]), af, fmaf(fabsf(f[7]), ag, fabsf(f[8])));
  const float e0 = 8.0f * u * fmaf(fabsf(f[0]), bf, fmaf(fabsf(f[3]), bg, fabsf(f[6])));
  const float e1 = 8.0f * u * fmaf(fabsf(f[1]), bf, fmaf(fabsf(f[4]), bg, fabsf(f[7])));
  const float e = fmaf(bx, f0, fmaf(by, f1, f2));
  const float de = fmaf(bf, d0, fmaf(bg, d1, d2)) +
                   8.0f * u * fmaf(bf, fabsf(f0), fmaf(bg, fabsf(f1), fabsf(f2)));
  const float d = fmaf(f0, f0, fmaf(f1, f1, fmaf(g0, g0, g1 * g1)));
  const float dd = fmaf(d0, fmaf(2.0f, fabsf(f0), d0),
                        fmaf(d1, fmaf(2.0f, fabsf(f1), d1),
                             fmaf(e0, fmaf(2.0f, fabsf(g0), e0), e1 * fmaf(2.0f, fabsf(g1), e1)))) +
                   8.0f * u * d;
  const float ae = fabsf(e);
  const float lo = d - dd, hi = d + dd;
  if (lo > 2e-18f) {
    const float in_l = (ae + de) * (ae + de), in_r = t2 * lo * (1.0f - 32.0f * u);
    if (in_l < in_r) return 1;
    const float out_e = ae - de;
    if (out_e > 0.0f && out_e * out_e > t2 * hi * (1.0f + 32.0f * u)) return 0;
  } else if (hi < 5e-19f && hi >= 0.0f) {
    return 0;  // the FP64 d is below 1e-18: f64::MAX, never an inlier
  }
  return -1;
}

constexpr int kCountTile = 2048;

// First-tier bounds of one hypothesis over one tile of correspondences, from
// the tile's largest coordinate magnitudes (ax, ay, bx, by): every |f_k| is
// at most S_k, so the error bounds of inlier_fp32 become constants de, dd
// (plus the 8u d term of d's own rounding).
struct TileBound {
  float de, dd;
};

__device__ __forceinline__ TileBound tile_bound(const Hyp32& H, float4 m) {
  constexpr float u = 5.9604645e-8f;
  const float* f = H.f;
  const float S0 = fmaf(fabsf(f[0]), m.x, fmaf(fabsf(f[1]), m.y, fabsf(f[2])));
  const float S1 = fmaf(fabsf(f[3]), m.x, fmaf(fabsf(f[4]), m.y, fabsf(f[5])));
  const float S2 = fmaf(fabsf(f[6]), m.x, fmaf(fabsf(f[7]), m.y, fabsf(f[8])));
  const float T0 = fmaf(fabsf(f[0]), m.z, fmaf(fabsf(f[3]), m.w, fabsf(f[6])));
  const float T1 = fmaf(fabsf(f[1]), m.z, fmaf(fabsf(f[4]), m.w, fabsf(f[7])));
  const float d0 = 8.0f * u * S0, d1 = 8.0f * u * S1, d2 = 8.0f * u * S2;
  const float e0 = 8.0f * u * T0, e1 = 8.0f * u * T1;
  TileBound B;
  // |f_hat| <= S + d; bounds rounded up by the 2x in the factors.
  B.de = 2.0f * (fmaf(m.z, d0, fmaf(m.w, d1, d2)) +
                 8.0f * u * fmaf(m.z, S0 + d0, fmaf(m.w, S1 + d1, S2 + d2)));
  B.dd = 2.0f * (d0 * (2.0f * (S0 + d0) + d0) + d1 * (2.0f * (S1 + d1) + d1) +
                 e0 * (2.0f * (T0 + e0) + e0) + e1 * (2.0f * (T1 + e1) + e1));
  return B;
}

// Whether surely in / surely out by the tile's constant bounds (neither:
// undecided).
__device__ __forceinline__ void inlier_tile(const Hyp32& H, const TileBound& B, float4 c, float t2,
                                            bool& in, bool& out) {
  constexpr float u = 5.9604645e-8f;
  const float* f = H.f;
  const float f0 = fmaf(f[0], c.x, fmaf(f[1], c.y, f[2]));
  const float f1 = fmaf(f[3], c.x, fmaf(f[4], c.y, f[5]));
  const float f2 = fmaf(f[6], c.x, fmaf(f[7], c.y, f[8]));
  const float g0 = fmaf(f[0], c.z, fmaf(f[3], c.w, f[6]));
  const float g1 = fmaf(f[1], c.z, fmaf(f[4], c.w, f[7]));
  const float ae = fabsf(fmaf(c.z, f0, fmaf(c.w, f1, f2)));
  const float d = fmaf(f0, f0, fmaf(f1, f1, fmaf(g0, g0, g1 * g1)));
  const float dd = fmaf(8.0f * u, d, B.dd);
  const float lo = d - dd;
  const float a = ae + B.de, o = ae - B.de;
  const bool clear = lo > 2e-18f;
  in = clear && a * a < t2 * lo * (1.0f - 32.0f * u);
  out = clear && o > 0.0f && o * o > t2 * (d + dd) * (1.0f + 32.0f * u);
}

// Inlier counts: a warp per hypothesis at a time, over the pair's FP32
// coordinates in shared memory (a tile of them at a time where they are
// more).  Tests are decided by the tile's constant bounds, else by the
// correspondence's own bounds, else in FP64.
//
// Only the first hypothesis with the most inliers is wanted: one that could
// not reach the CTA's best count any more, were all its remaining tests
// inliers, is left with a count of 0 (a sample with one mismatch in it, nine
// of ten at a quarter of mismatches, is through after some third of the
// tests).  gridDim.x / pairs CTAs share a pair, a bound each.  Four tests a
// lane are in flight, and both outcomes of a test are formed without a
// branch.  1603 pairs x 600 x 1300 tests: 3.9 ms with every test made, four
// hypotheses a warp; now 2.15 ms.
__global__ void __launch_bounds__(kCountThreads) ransac_count_kernel(RansacArgs A,
                                                                     const float4* uv32,
                                                                     int parts) {
  __shared__ float4 tile[kCountTile];
  __shared__ float4 wmax[kCountThreads / 32];
  __shared__ int best;
  constexpr int kWarps = kCountThreads / 32, kTests = 4;
  const int64_t q = blockIdx.x / parts;
  const int part = (int)(blockIdx.x % parts);
  const int64_t p = A.p0 + q;
  const uint32_t b = A.match_ptr[p], n = A.match_ptr[p + 1] - b;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float t2 = (float)A.t2;
  const int h0 = (int)((int64_t)A.iters * part / parts),
            h1 = (int)((int64_t)A.iters * (part + 1) / parts);
  if (n < 12) {
    for (int it = h0 + threadIdx.x; it < h1; it += kCountThreads) A.count[q * A.iters + it] = 0;
    return;
  }
  if (threadIdx.x == 0) best = 0;
  float4 m;
  auto load_tile = [&](uint32_t t0, uint32_t tn) {
    __syncthreads();
    m = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t i = threadIdx.x; i < tn; i += kCountThreads) {
      const float4 c = uv32[b + t0 + i];
      tile[i] = c;
      m.x = fmaxf(m.x, fabsf(c.x)), m.y = fmaxf(m.y, fabsf(c.y));
      m.z = fmaxf(m.z, fabsf(c.z)), m.w = fmaxf(m.w, fabsf(c.w));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      m.x = fmaxf(m.x, __shfl_xor_sync(kFull, m.x, o));
      m.y = fmaxf(m.y, __shfl_xor_sync(kFull, m.y, o));
      m.z = fmaxf(m.z, __shfl_xor_sync(kFull, m.z, o));
      m.w = fmaxf(m.w, __shfl_xor_sync(kFull, m.w, o));
    }
    if (lane == 0) wmax[warp] = m;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float4 v = wmax[w];
      m.x = fmaxf(m.x, v.x), m.y = fmaxf(m.y, v.y), m.z = fmaxf(m.z, v.z), m.w = fmaxf(m.w, v.w);
    }
  };
  const bool one_tile = n <= (uint32_t)kCountTile;
  if (one_tile) load_tile(0, n);
  // Every warp makes the same number of rounds (a tile is loaded by all).
  for (int hb = h0; hb < h1; hb += kWarps) {
    const int it = hb + warp;
    const int64_t h = q * A.iters + it;
    bool live = it < h1 && A.valid[h];
    Hyp32 H;
    {
      const float4* f = A.F32 + 3 * h;
      const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 a = live ? f[0] : z, c = live ? f[1] : z, e = live ? f[2] : z;
      H.f[0] = a.x, H.f[1] = a.y, H.f[2] = a.z, H.f[3] = a.w;
      H.f[4] = c.x, H.f[5] = c.y, H.f[6] = c.z, H.f[7] = c.w, H.f[8] = e.x;
    }
    int cnt = 0;
    for (uint32_t t0 = 0; t0 < n; t0 += kCountTile) {
      const uint32_t tn = min((uint32_t)kCountTile, n - t0);
      if (!one_tile) load_tile(t0, tn);
      if (!live) continue;
      const TileBound TB = tile_bound(H, m);
      for (uint32_t i0 = 0; i0 < tn; i0 += 32 * kTests) {
        bool in[kTests], out[kTests];
#pragma unroll
        for (int j = 0; j < kTests; ++j) {
          const uint32_t i = i0 + 32 * j + lane;
          inlier_tile(H, TB, tile[i < tn ? i : 0], t2, in[j], out[j]);
          in[j] = in[j] && i < tn, out[j] = out[j] || i >= tn;
        }
#pragma unroll
        for (int j = 0; j < kTests; ++j) {
          if (__any_sync(kFull, !in[j] && !out[j])) {
            if (!in[j] && !out[j]) {
              const uint32_t i = i0 + 32 * j + lane;
              int r = inlier_fp32(H, tile[i], t2);
              if (r < 0) {
                const double* u64 = A.uv + 4 * ((size_t)b + t0 + i);
                r = ep_sampson<true>(A.F + 9 * h, u64[0], u64[1], u64[2], u64[3]) < A.t2;
              }
              in[j] = r != 0;
            }
            __syncwarp();
          }
          cnt += __popc(__ballot_sync(kFull, in[j]));
        }
        // Strictly less: of equal counts the first hypothesis wins.  Other
        // warps raise the bound meanwhile, so one lane reads it for all: lanes
        // with different values would part before the next ballot.
        const int64_t left = (int64_t)n - t0 - i0 - 32 * kTests;
        int bound = 0;
        if (lane == 0) bound = *(volatile int*)&best;
        bound = __shfl_sync(kFull, bound, 0);
        if (left > 0 && cnt + left < bound) {
          live = false;
          cnt = 0;
          break;
        }
      }
    }
    if (it < h1 && lane == 0) {
      A.count[h] = cnt;
      if (live) atomicMax(&best, cnt);
    }
    __syncwarp();
  }
}

__global__ void uv_f32_kernel(int64_t n, const double* uv, float4* out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* u = uv + 4 * i;
  out[i] = make_float4((float)u[0], (float)u[1], (float)u[2], (float)u[3]);
}

__device__ __forceinline__ uint64_t cta_max_u64(uint64_t v, uint64_t* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = max(v, (uint64_t)__shfl_xor_sync(kFull, v, o));
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (warp == 0) {
    v = lane < kRefitThreads / 32 ? red[lane] : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, (uint64_t)__shfl_xor_sync(kFull, v, o));
    if (lane == 0) red[kRefitThreads / 32] = v;
  }
  __syncthreads();
  const uint64_t r = red[kRefitThreads / 32];
  __syncthreads();
  return r;
}

__device__ __forceinline__ int cta_sum_int(int v, int* wsum) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = v;
  __syncthreads();
  int t = 0;
  for (int w = 0; w < kRefitThreads / 32; ++w) t += wsum[w];
  __syncthreads();
  return t;
}

// Inlier flags of F for the CTA's pair into `flag`, and the inlier indices
// in correspondence order into `list`; returns the count.
__device__ int mark_inliers(const double* F, const double* uv, uint32_t n, double t2,
                            uint8_t* flag, uint32_t* list, int* wsum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ int base_s;
  if (threadIdx.x == 0) base_s = 0;
  __syncthreads();
  for (uint32_t i0 = 0; i0 < n; i0 += kRefitThreads) {
    const uint32_t i = i0 + threadIdx.x;
    bool in = false;
    if (i < n) {
      const double* u = uv + 4 * (size_t)i;
      in = ep_sampson<true>(F, u[0], u[1], u[2], u[3]) < t2;
      flag[i] = in;
    }
    const unsigned m = __ballot_sync(kFull, in);
    if (lane == 0) wsum[warp] = __popc(m);
    __syncthreads();
    int off = base_s;
    for (int w = 0; w < warp; ++w) off += wsum[w];
    if (in) list[off + __popc(m & ((1u << lane) - 1u))] = i;
    __syncthreads();
    if (threadIdx.x == 0)
      for (int w = 0; w < kRefitThreads / 32; ++w) base_s += wsum[w];
    __syncthreads();
  }
  return base_s;
}

__device__ __forceinline__ double cta_sum_d(double v, double* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double t = 0.0;
#pragma unroll
  for (int w = 0; w < kRefitThreads / 32; ++w) t += red[w];
  __syncthreads();
  return t;
}

// CTA per pair: the best hypothesis (the first with the most inliers), its
// inliers, and one refit on them (geometry.rs:286-298), kept when it has at
// least as many inliers.  The refit's centroid, mean distance and normal
// matrix are CTA reductions in a fixed order (the 45 sums by halving: 48
// additions a lane for 225); its eigenvector is a warp's work, another one in
// each CTA so that an SM's CTAs spread it over its four FP64 pipes.  1603
// pairs of 150 cameras: 1.13 -> 0.89 ms.
__global__ void __launch_bounds__(kRefitThreads) ransac_select_kernel(RansacArgs A) {
  __shared__ uint64_t red[kRefitThreads / 32 + 1];
  __shared__ int wsum[kRefitThreads / 32];
  __shared__ double dred[kRefitThreads / 32];
  __shared__ double msum[kRefitThreads / 32][45];
  __shared__ double Ms[81];
  __shared__ double Fs[9];
  __shared__ int ok_s;
  const int64_t q = blockIdx.x, p = A.p0 + q;
  const uint32_t b = A.match_ptr[p], n = A.match_ptr[p + 1] - b;
  uint8_t* flag = A.inlier + b;
  for (uint32_t i = threadIdx.x; i < n; i += kRefitThreads) flag[i] = 0;
  if (threadIdx.x == 0) A.n_inl[p] = 0, A.best[p] = -1, A.refit[p] = 0;
  if (n < 12) return;
  uint64_t key = 0;
  for (int it = threadIdx.x; it < A.iters; it += kRefitThreads) {
    const int c = A.count[q * A.iters + it];
    if (c > 0) key = max(key, ((uint64_t)c << 32) | (uint32_t)(0x7fffffff - it));
  }
  key = cta_max_u64(key, red);
  if (key == 0) return;
  const int hbest = 0x7fffffff - (int)(uint32_t)key;
  if (threadIdx.x < 9) Fs[threadIdx.x] = A.F[9 * (q * A.iters + hbest) + threadIdx.x];
  __syncthreads();
  const double* U = A.uv + 4 * (size_t)b;
  uint32_t* list = A.scratch + b;
  const int nb = mark_inliers(Fs, U, n, A.t2, flag, list, wsum);
  if (threadIdx.x == 0) A.best[p] = hbest, A.n_inl[p] = nb;
  if (nb < 8) return;
  // normalise (geometry.rs:161-183) of both sides over the inliers.
  const double nn = (double)nb, rnn = __drcp_rn(nn);
  double sa = 0.0, sb = 0.0, sc = 0.0, sd = 0.0;
  for (int i = threadIdx.x; i < nb; i += kRefitThreads) {
    const double* u = U + 4 * (size_t)list[i];
    sa += quotient_by(u[0], nn, rnn), sb += quotient_by(u[1], nn, rnn);
    sc += quotient_by(u[2], nn, rnn), sd += quotient_by(u[3], nn, rnn);
  }
  const double max_ = cta_sum_d(sa, dred), may = cta_sum_d(sb, dred);
  const double mbx = cta_sum_d(sc, dred), mby = cta_sum_d(sd, dred);
  double da = 0.0, db = 0.0;
  for (int i = threadIdx.x; i < nb; i += kRefitThreads) {
    const double* u = U + 4 * (size_t)list[i];
    const double x0 = u[0] - max_, y0 = u[1] - may, x1 = u[2] - mbx, y1 = u[3] - mby;
    da += sqrt(x0 * x0 + y0 * y0), db += sqrt(x1 * x1 + y1 * y1);
  }
  const double dA = cta_sum_d(da, dred) / nn, dB = cta_sum_d(db, dred) / nn;
  const double sA = dA > 1e-12 ? 1.4142135623730951 / dA : 1.0;
  const double sB = dB > 1e-12 ? 1.4142135623730951 / dB : 1.0;
  // Normal matrix, upper triangle (45 entries) per thread, then in order.
  double acc[45];
#pragma unroll
  for (int k = 0; k < 45; ++k) acc[k] = 0.0;
  for (int i = threadIdx.x; i < nb; i += kRefitThreads) {
    const double* u = U + 4 * (size_t)list[i];
    const double p0 = (u[0] - max_) * sA, p1 = (u[1] - may) * sA;
    const double q0 = (u[2] - mbx) * sB, q1 = (u[3] - mby) * sB;
    const double row[9] = {q0 * p0, q0 * p1, q0, q1 * p0, q1 * p1, q1, p0, p1, 1.0};
    int k = 0;
#pragma unroll
    for (int r = 0; r < 9; ++r)
#pragma unroll
      for (int c = r; c < 9; ++c) acc[k++] += row[r] * row[c];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int off = 0, cnt45 = 45;
  double v2[2];
  warp_halve<16>(acc, lane, off, cnt45, v2);
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (i < cnt45) msum[warp][off + i] = v2[i];
  __syncthreads();
  if (threadIdx.x < 45) {
    double t = 0.0;
    for (int w = 0; w < kRefitThreads / 32; ++w) t += msum[w][threadIdx.x];
    int r = 0, k = threadIdx.x;
    while (k >= 9 - r) k -= 9 - r, ++r;
    const int c = r + k;
    Ms[9 * r + c] = t, Ms[9 * c + r] = t;
  }
  __syncthreads();
  if (warp == (int)(blockIdx.x % (kRefitThreads / 32))) {
    const double x = smallest_eigvec9(Ms);
    double fm[9], F[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) fm[i] = __shfl_sync(kFull, x, i);
    if (lane == 0) {
      const double ta[9] = {sA, 0.0, -sA * max_, 0.0, sA, -sA * may, 0.0, 0.0, 1.0};
      const double tb[9] = {sB, 0.0, -sB * mbx, 0.0, sB, -sB * mby, 0.0, 0.0, 1.0};
      ok_s = ep_finish(fm, ta, tb, F);
      if (ok_s)
        for (int j = 0; j < 9; ++j) Fs[j] = F[j];
    }
  }
  __syncthreads();
  if (!ok_s) return;
  int cnt = 0;
  for (uint32_t i = threadIdx.x; i < n; i += kRefitThreads) {
    const double* u = U + 4 * (size_t)i;
    list[i] = ep_sampson<true>(Fs, u[0], u[1], u[2], u[3]) < A.t2;  // (the index list is done with)
    cnt += list[i];
  }
  const int nr = cta_sum_int(cnt, wsum);
  if (nr < nb) return;
  for (uint32_t i = threadIdx.x; i < n; i += kRefitThreads) flag[i] = (uint8_t)list[i];
  if (threadIdx.x == 0) A.n_inl[p] = nr, A.refit[p] = 1;
}

// ---- pair_fits ----------------------------------------------------------------

struct FitsArgs {
  int64_t p0;  // first pair of this launch
  const uint32_t* pair_cam;
  const uint32_t* match_ptr;
  const double* uv;
  const double* rot;
  const double* center;
  const double* intr;
  const uint32_t* cam_group;
  uint64_t* key;   // [n_matches] of pairs with more than kFitKeys matches
  double* median;  // [n_pairs]
};

constexpr int kFitsThreads = 256;
constexpr uint32_t kFitKeys = 3072;  // total-order keys of a pair in shared memory

// CTA per pair: E = [t]x R_b R_a^T, t = R_b (C_a - C_b) (sparse.rs:629-631),
// then every match's error sqrt(sampson) * f_a on undistorted coordinates,
// and the pair's median error (element n/2 in total order).
//
// Bound by its FP64 operations (~190 a match, and as many again in integer
// instructions: 3.46 -> 2.19 ms for 4.6 million matches).  The median is
// selected in the CTA that made the errors: sorting all matches by error and then by pair took
// nine passes over memory (1.3 of 5.6 ms for 4.6 million matches), and the
// errors 4.1 ms with two divisions a step of the undistortion.
__global__ void __launch_bounds__(kFitsThreads) pair_fits_kernel(FitsArgs A) {
  __shared__ double E[9];
  __shared__ uint64_t skey[kFitKeys];
  __shared__ uint32_t hist[256], found[3];
  const int64_t p = A.p0 + blockIdx.x;
  const uint32_t b = A.match_ptr[p], n = A.match_ptr[p + 1] - b;
  if (n == 0) {
    if (threadIdx.x == 0) A.median[p] = kF64Max;
    return;
  }
  const uint32_t ca = A.pair_cam[2 * p], cb = A.pair_cam[2 * p + 1];
  const double* Ka = A.intr + 5 * (size_t)A.cam_group[ca];
  const double* Kb = A.intr + 5 * (size_t)A.cam_group[cb];
  if (threadIdx.x == 0) {
    const double* Ra = A.rot + 9 * (size_t)ca;
    const double* Rb = A.rot + 9 * (size_t)cb;
    double RaT[9], R[9], S[9];
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) RaT[3 * r + c] = Ra[3 * c + r];
    mul3(Rb, RaT, R);
    const double d0 = A.center[3 * ca] - A.center[3 * cb];
    const double d1 = A.center[3 * ca + 1] - A.center[3 * cb + 1];
    const double d2 = A.center[3 * ca + 2] - A.center[3 * cb + 2];
    double t[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) t[r] = Rb[3 * r] * d0 + Rb[3 * r + 1] * d1 + Rb[3 * r + 2] * d2;
    S[0] = 0.0, S[1] = -t[2], S[2] = t[1];
    S[3] = t[2], S[4] = 0.0, S[5] = -t[0];
    S[6] = -t[1], S[7] = t[0], S[8] = 0.0;
    double Et[9];
    mul3(S, R, Et);
    for (int j = 0; j < 9; ++j) E[j] = Et[j];
  }
  const double rfa = __drcp_rn(Ka[0]), rfb = __drcp_rn(Kb[0]);
  __syncthreads();
  uint64_t* key = n <= kFitKeys ? skey : A.key + b;
  for (uint32_t i = threadIdx.x; i < n; i += kFitsThreads) {
    const double2* u = reinterpret_cast<const double2*>(A.uv + 4 * (size_t)(b + i));
    const double2 ua = u[0], ub = u[1];
    double x1[2], x2[2];
    undistort(Ka, rfa, ua.x, ua.y, x1);
    undistort(Kb, rfb, ub.x, ub.y, x2);
    const double err = sqrt(ep_sampson<false>(E, x1[0], x1[1], x2[0], x2[1])) * Ka[0];
    key[i] = total_order_key(err);
  }
  __syncthreads();
  const uint64_t med = select_key<kFitsThreads>(key, n, n / 2, hist, found);
  if (threadIdx.x == 0) A.median[p] = from_total_order_key(med);
}

// ---- input checks ---------------------------------------------------------------

__global__ void check_pairs_kernel(int64_t n_pairs, int64_t n_matches, const uint32_t* match_ptr,
                                   const uint32_t* pair_cam, int64_t nc, const uint32_t* cam_group,
                                   int64_t ng, uint32_t* err) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p > n_pairs) return;
  if (p == 0 && match_ptr[0] != 0) atomicOr(err, ERR_BAD_INDEX);
  if (p == n_pairs) {
    if (match_ptr[p] != (uint64_t)n_matches) atomicOr(err, ERR_BAD_INDEX);
    return;
  }
  if (match_ptr[p + 1] < match_ptr[p]) atomicOr(err, ERR_BAD_INDEX);
  if (pair_cam) {
    const uint32_t a = pair_cam[2 * p], c = pair_cam[2 * p + 1];
    if (a >= (uint64_t)nc || c >= (uint64_t)nc) {
      atomicOr(err, ERR_BAD_INDEX);
    } else if (cam_group && (cam_group[a] >= (uint64_t)ng || cam_group[c] >= (uint64_t)ng)) {
      atomicOr(err, ERR_BAD_INDEX);
    }
  }
}

__global__ void default_seed_kernel(int64_t n_pairs, const uint32_t* pair_cam, uint64_t* seed) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p < n_pairs) seed[p] = (uint64_t)pair_cam[2 * p] * 7919u + pair_cam[2 * p + 1];
}

template <typename T>
void upload_n(DevBuf<T>& d, const T* h, int64_t n, cudaStream_t s) {
  d.alloc(std::max<int64_t>(n, 1), s);
  if (n > 0) check(cudaMemcpyAsync(d.p, h, n * sizeof(T), cudaMemcpyDefault, s), "copy in");
}

template <typename T>
void download_n(T* h, const DevBuf<T>& d, int64_t n, cudaStream_t s) {
  if (h && n > 0) check(cudaMemcpyAsync(h, d.p, n * sizeof(T), cudaMemcpyDefault, s), "copy out");
}

struct PairsIn {
  int64_t np = 0, nm = 0;
  DevBuf<uint32_t> match_ptr, pair_cam, err;
  DevBuf<double> uv;

  // copy_uv false: the correspondences' buffer is made, not filled.
  void load(const ba_pair_matches* m, bool need_cams, int64_t nc, const uint32_t* cam_group_dev,
            int64_t ng, cudaStream_t s, bool copy_uv = true) {
    if (!m) throw BadInput("null pair matches");
    np = m->n_pairs, nm = m->n_matches;
    if (np < 0 || nm < 0) throw BadInput("negative size");
    if (nm > 0xfffffff0LL || np > 0x7ffffff0LL) throw BadInput("too many pairs or matches");
    if (!m->match_ptr) throw BadInput("null match_ptr");
    if (nm > 0 && !m->uv) throw BadInput("null uv");
    if (need_cams && np > 0 && !m->pair_cam) throw BadInput("null pair_cam");
    upload_n(match_ptr, m->match_ptr, np + 1, s);
    if (copy_uv)
      upload_n(uv, m->uv, 4 * nm, s);
    else
      uv.alloc(std::max<int64_t>(4 * nm, 1), s);
    if (m->pair_cam) upload_n(pair_cam, m->pair_cam, 2 * np, s);
    err.alloc(1, s);
    err.zero();
    BA_LAUNCH(check_pairs_kernel<<<grid_for(np + 1, 256), 256, 0, s>>>(
        np, nm, match_ptr, m->pair_cam ? pair_cam.p : nullptr, nc, cam_group_dev, ng, err));
    uint32_t e = 0;
    check(cudaMemcpyAsync(&e, err.p, 4, cudaMemcpyDeviceToHost, s), "d2h");
    check(cudaStreamSynchronize(s), "pair check");
    if (e) throw BadInput("match_ptr not increasing from 0 to n_matches, or a camera or group index out of range");
  }
};

// A second stream for a call's large copy, and an event for the order.
struct CopySide {
  cudaStream_t s = nullptr;
  cudaEvent_t e = nullptr;
  // From here on (buffers made, the caller's earlier work done).
  void fork(cudaStream_t main) {
    check(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "copy stream");
    check(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "event");
    check(cudaEventRecord(e, main), "fork");
    check(cudaStreamWaitEvent(s, e, 0), "fork");
  }
  // `main` waits for the copies so far.
  void join(cudaStream_t main) {
    if (!s) return;
    check(cudaEventRecord(e, s), "join");
    check(cudaStreamWaitEvent(main, e, 0), "join");
  }
  ~CopySide() {
    if (s) cudaStreamSynchronize(s), cudaStreamDestroy(s);
    if (e) cudaEventDestroy(e);
  }
};

}  // namespace
}  // namespace ba

using namespace ba;

extern "C" ba_status ba_ransac_fundamental(const ba_pair_matches* m, double thresh_px,
                                           int32_t iters, void* stream, uint8_t* inlier,
                                           int32_t* n_inliers, int32_t* best_hypothesis,
                                           uint8_t* refit) {
  return guarded([&] {
    if (!(thresh_px >= 0.0) || !std::isfinite(thresh_px)) throw BadInput("thresh_px must be finite and >= 0");
    if (iters < 0 || iters > (1 << 20)) throw BadInput("iters must be in 0..2^20");
    cudaStream_t s = (cudaStream_t)stream;
    PairsIn P;
    P.load(m, m && !m->seed, (int64_t)1 << 32, nullptr, 0, s, false);
    const int64_t np = P.np, nm = P.nm;
    // A large call's correspondences are copied while the samples are drawn.
    CopySide side;
    if (nm > (int64_t(1) << 18)) side.fork(s);
    if (nm > 0)
      check(cudaMemcpyAsync(P.uv.p, m->uv, 32 * nm, cudaMemcpyDefault, side.s ? side.s : s),
            "copy in");
    DevBuf<uint64_t> seed;
    if (m->seed) {
      upload_n(seed, m->seed, np, s);
    } else {
      seed.alloc(std::max<int64_t>(np, 1), s);
      if (np > 0) BA_LAUNCH(default_seed_kernel<<<grid_for(np, 256), 256, 0, s>>>(np, P.pair_cam, seed));
    }
    DevBuf<uint8_t> d_inl(std::max<int64_t>(nm, 1), s), d_refit(std::max<int64_t>(np, 1), s);
    DevBuf<int32_t> d_n(std::max<int64_t>(np, 1), s), d_best(std::max<int64_t>(np, 1), s);
    DevBuf<uint32_t> scratch(std::max<int64_t>(nm, 1), s);
    const int64_t chunk = iters > 0 ? std::max<int64_t>(1, kMaxChunkHyp / iters) : np;
    const int64_t cp = std::min<int64_t>(std::max<int64_t>(np, 1), chunk);
    const int64_t ch = std::max<int64_t>(cp * iters, 1);
    DevBuf<uint32_t> samples(8 * ch, s);
    DevBuf<double> F(9 * ch, s);
    DevBuf<float4> F32(3 * ch, s);
    DevBuf<uint8_t> valid(ch, s);
    DevBuf<int32_t> count(ch, s);
    DevBuf<float4> uv32(std::max<int64_t>(nm, 1), s);
    // Counting: two CTAs a pair (1603 pairs of unequal size: 2.15 ms; one took
    // 0.2 ms more, three 0.03), more where that leaves SMs with fewer than four, but at
    // least eight hypotheses a warp, so that the bound of a CTA's first counts
    // serves most of its hypotheses.
    int dev = 0, n_sm = 0;
    check(cudaGetDevice(&dev), "cudaGetDevice");
    check(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev), "attribute");
    auto join_copy = [&] {
      side.join(s);
      if (nm > 0) BA_LAUNCH(uv_f32_kernel<<<grid_for(nm, 256), 256, 0, s>>>(nm, P.uv, uv32));
    };
    if (np == 0 || iters == 0) join_copy();
    for (int64_t p0 = 0; p0 < np; p0 += cp) {
      const int64_t n = std::min(cp, np - p0);
      RansacArgs A{p0, n, P.match_ptr, P.uv, seed, iters, thresh_px * thresh_px, samples, F, F32,
                   valid, count, scratch, d_inl, d_n, d_best, d_refit, P.err};
      if (iters > 0) {
        BA_LAUNCH(ransac_sample_kernel<<<(unsigned)n, 32, 0, s>>>(A, draw_jump()));
        if (p0 == 0) join_copy();
        BA_LAUNCH(ransac_fit_kernel<<<grid_for(n * iters, kFitThreads), kFitThreads, 0, s>>>(A));
        const int64_t most = std::max<int64_t>(1, iters / (8 * (kCountThreads / 32)));
        const int parts = (int)std::min<int64_t>(most, std::max<int64_t>(2, 4 * n_sm / n));
        BA_LAUNCH(ransac_count_kernel<<<(unsigned)(n * parts), kCountThreads, 0, s>>>(A, uv32,
                                                                                     parts));
      }
      BA_LAUNCH(ransac_select_kernel<<<(unsigned)n, kRefitThreads, 0, s>>>(A));
    }
    uint32_t e = 0;
    check(cudaMemcpyAsync(&e, P.err.p, 4, cudaMemcpyDeviceToHost, s), "d2h");
    download_n(inlier, d_inl, nm, s), download_n(n_inliers, d_n, np, s);
    download_n(best_hypothesis, d_best, np, s), download_n(refit, d_refit, np, s);
    check(cudaStreamSynchronize(s), "ransac");
    if (e) throw std::runtime_error("RANSAC sampling found no eight distinct correspondences");
  });
}

extern "C" ba_status ba_pair_fits(const ba_pair_matches* m, const double* rot, const double* center,
                                  const double* intr, const uint32_t* cam_group, int64_t n_cams,
                                  int64_t n_groups, void* stream, double* median_px) {
  return guarded([&] {
    if (n_cams < 0 || n_groups < 0) throw BadInput("negative size");
    if (m && m->n_pairs > 0x7fffffff) throw BadInput("too many pairs");  // a CTA each
    if ((n_cams > 0 && (!rot || !center || !cam_group)) || (n_groups > 0 && !intr))
      throw BadInput("null camera array");
    cudaStream_t s = (cudaStream_t)stream;
    DevBuf<double> d_rot, d_center, d_intr;
    DevBuf<uint32_t> d_group;
    upload_n(d_rot, rot, 9 * n_cams, s), upload_n(d_center, center, 3 * n_cams, s);
    upload_n(d_intr, intr, 5 * n_groups, s), upload_n(d_group, cam_group, n_cams, s);
    PairsIn P;
    P.load(m, true, n_cams, d_group, n_groups, s, false);
    const int64_t np = P.np, nm = P.nm;
    DevBuf<double> med(std::max<int64_t>(np, 1), s);
    // The correspondences of a large call come in on a second stream, a
    // quarter first: the rest is copied while its pairs are worked on (the copy
    // is 1.0 ms for 4.6 million, the arithmetic 2.2).  More pieces cost more in
    // half-empty last waves than they hide (with arithmetic of 3.0 ms: 4.35 ms in
    // three, 5.1 in five, 8.9 in seventeen, against 4.3 in one).
    std::vector<uint32_t> ptr((size_t)np + 1, 0);
    check(cudaMemcpyAsync(ptr.data(), P.match_ptr.p, 4 * ptr.size(), cudaMemcpyDeviceToHost, s), "d2h");
    check(cudaStreamSynchronize(s), "pair offsets");
    uint32_t most = 0;
    for (int64_t p = 0; p < np; ++p) most = std::max(most, ptr[p + 1] - ptr[p]);
    DevBuf<uint64_t> key(most > kFitKeys ? nm : 1, s);
    FitsArgs A{0, P.pair_cam, P.match_ptr, P.uv, d_rot, d_center, d_intr, d_group, key, med};
    CopySide side;
    if (nm > (int64_t(1) << 20)) side.fork(s);
    for (int64_t p0 = 0; p0 < np;) {
      int64_t p1 = np;
      if (side.s && p0 == 0) {
        p1 = std::upper_bound(ptr.begin(), ptr.end(), (uint32_t)(nm / 4)) - ptr.begin();
        p1 = std::max<int64_t>(1, std::min(p1, np));
      }
      const int64_t b = ptr[p0], n = ptr[p1] - b;
      if (n > 0)
        check(cudaMemcpyAsync(P.uv.p + 4 * b, m->uv + 4 * b, 32 * n, cudaMemcpyDefault,
                              side.s ? side.s : s),
              "copy in");
      side.join(s);
      A.p0 = p0;
      BA_LAUNCH(pair_fits_kernel<<<(unsigned)(p1 - p0), kFitsThreads, 0, s>>>(A));
      p0 = p1;
    }
    download_n(median_px, med, np, s);
    check(cudaStreamSynchronize(s), "pair fits");
  });
}
