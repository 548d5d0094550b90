// Exclusive scan, stable LSD radix sort and batched lower_bound.
#include <vector>

#include "ba_common.cuh"
#include "primitives.cuh"

namespace ba {

thread_local int64_t g_launches = 0;


namespace {

constexpr int kScanThreads = 512;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;  // 2048

// Exclusive scan of one 2048-element tile; writes the tile total.
__global__ void __launch_bounds__(kScanThreads)
    scan_tile_kernel(const uint32_t* in, uint32_t* out, uint32_t* tile_sums,
                     size_t n) {
  __shared__ uint32_t warp_tot[kScanThreads / 32];
  const size_t base = (size_t)blockIdx.x * kScanTile + (size_t)threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t sum = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    v[i] = (base + i < n) ? in[base + i] : 0u;
    sum += v[i];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t t = (lane < kScanThreads / 32) ? warp_tot[lane] : 0u;
    uint32_t ti = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(kFull, ti, o);
      if (lane >= o) ti += u;
    }
    if (lane < kScanThreads / 32) warp_tot[lane] = ti - t;  // exclusive
    if (lane == kScanThreads / 32 - 1 && tile_sums) tile_sums[blockIdx.x] = ti;
  }
  __syncthreads();
  uint32_t run = warp_tot[warp] + incl - sum;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    if (base + i < n) out[base + i] = run;
    run += v[i];
  }
}

__global__ void scan_add_kernel(uint32_t* out, const uint32_t* tile_off,
                                size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] += tile_off[i / kScanTile];
}

void scan_rec(const uint32_t* in, uint32_t* out, size_t n, cudaStream_t s) {
  const size_t tiles = (n + kScanTile - 1) / kScanTile;
  if (tiles <= 1) {
    BA_LAUNCH(scan_tile_kernel<<<1, kScanThreads, 0, s>>>(in, out, nullptr, n));
    return;
  }
  DevBuf<uint32_t> sums(tiles, s);
  BA_LAUNCH(scan_tile_kernel<<<(unsigned)tiles, kScanThreads, 0, s>>>(in, out, sums, n));
  scan_rec(sums, sums, tiles, s);
  BA_LAUNCH(scan_add_kernel<<<grid_for(n, 256), 256, 0, s>>>(out, sums, n));
}

// ---- radix sort ------------------------------------------------------------

// The passes share the key's bits evenly (21 bits: three digits of seven), so
// that a tile of 4096 items leaves runs of some 8 to 32 items in each bucket.
constexpr int kSortThreads = 512;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 8;
constexpr int kSortTile = kSortThreads * kSortItems;  // 4096
constexpr int kRadixBits = 9;                         // of a digit, at most
constexpr int kRadix = 1 << kRadixBits;               // 512
static_assert(kRadix <= kSortThreads, "a thread per bucket");

__global__ void __launch_bounds__(kSortThreads)
    radix_hist_kernel(const uint64_t* keys, size_t n, int shift, int radix,
                      uint32_t* hist, size_t ntiles) {
  __shared__ uint32_t cnt[kRadix];
  const int t = threadIdx.x;
  cnt[t < radix ? t : 0] = 0;
  __syncthreads();
  const size_t base = (size_t)blockIdx.x * kSortTile;
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const size_t i = base + (size_t)r * kSortThreads + t;
    if (i < n) atomicAdd(&cnt[(int)(keys[i] >> shift) & (radix - 1)], 1u);
  }
  __syncthreads();
  if (t < radix) hist[(size_t)t * ntiles + blockIdx.x] = cnt[t];
}

// Stable scatter of a tile.  A warp takes 256 consecutive items, 32 at a
// time, and counts its own digits, so items are ranked in index order with
// two CTA barriers in all; the tile is then put in order in shared memory,
// keys first and values after them, and leaves it in runs of consecutive
// addresses.  Bound by the stores' sectors: the form before this one stored
// every item where its rank came up, 256 items between barriers (60.3 M pairs
// of 1200 cameras: 980 us a pass, now 555 us; the histogram is half as long a
// list of fewer buckets, and so its scan).
template <typename V>
__global__ void __launch_bounds__(kSortThreads)
    radix_scatter_kernel(const uint64_t* keys, const V* vals, uint64_t* okeys,
                         V* ovals, size_t n, int shift, int radix, const uint32_t* offs,
                         size_t ntiles) {
  __shared__ union Stage {
    uint32_t cnt[kSortWarps][kRadix];  // per warp: items of a digit so far
    uint64_t key[kSortTile];
    V val[kSortTile];
  } st;
  __shared__ uint32_t start[kRadix];  // first place of a digit in the ordered tile
  __shared__ uint32_t to[kRadix];     // its global offset less that place
  __shared__ uint32_t wsum[kSortWarps];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  for (int i = t; i < kSortWarps * kRadix; i += kSortThreads) (&st.cnt[0][0])[i] = 0;
  __syncthreads();
  const size_t tbase = (size_t)blockIdx.x * kSortTile;
  const int nt = n - tbase < (size_t)kSortTile ? (int)(n - tbase) : kSortTile;
  const int first = warp * (32 * kSortItems) + lane;
  uint64_t k[kSortItems];
  uint32_t place[kSortItems];
#pragma unroll
  for (int r = 0; r < kSortItems; ++r)
    k[r] = first + 32 * r < nt ? keys[tbase + first + 32 * r] : 0;
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const bool valid = first + 32 * r < nt;
    const unsigned d = valid ? (unsigned)(k[r] >> shift) & (radix - 1) : kRadix;
    const unsigned peers = __match_any_sync(kFull, d);
    const unsigned before = __popc(peers & ((1u << lane) - 1u));
    const uint32_t had = valid ? st.cnt[warp][d] : 0u;
    __syncwarp();
    if (valid && before == 0) st.cnt[warp][d] = had + __popc(peers);
    __syncwarp();
    place[r] = had + before;
  }
  __syncthreads();
  // A thread per digit: the warps' counts become their first places among the
  // digit's items, and the digits' totals their first places in the tile.
  uint32_t total = 0;
  if (t < radix)
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
      const uint32_t c = st.cnt[w][t];
      st.cnt[w][t] = total;
      total += c;
    }
  uint32_t incl = total;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  uint32_t at = incl - total;
  for (int w = 0; w < warp; ++w) at += wsum[w];
  if (t < radix) {
    start[t] = at;
    to[t] = offs[(size_t)t * ntiles + blockIdx.x] - at;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortItems; ++r)
    if (first + 32 * r < nt) {
      const unsigned d = (unsigned)(k[r] >> shift) & (radix - 1);
      place[r] += start[d] + st.cnt[warp][d];
    }
  __syncthreads();  // the counts are done with
#pragma unroll
  for (int r = 0; r < kSortItems; ++r)
    if (first + 32 * r < nt) st.key[place[r]] = k[r];
  __syncthreads();
  uint32_t dst[kSortItems];
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int q = t + r * kSortThreads;
    dst[r] = 0;
    if (q < nt) {
      const uint64_t key = st.key[q];
      dst[r] = to[(unsigned)(key >> shift) & (radix - 1)] + (uint32_t)q;
      if (dst[r] < n) okeys[dst[r]] = key;  // always true for a consistent histogram
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortItems; ++r)
    if (first + 32 * r < nt) st.val[place[r]] = vals[tbase + first + 32 * r];
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortItems; ++r) {
    const int q = t + r * kSortThreads;
    if (q < nt && dst[r] < n) ovals[dst[r]] = st.val[q];
  }
}

// Returns whether the result is in the *_tmp arrays.
template <typename V>
bool radix_passes(uint64_t* keys, V* vals, uint64_t* keys_tmp, V* vals_tmp,
                  size_t n, int bits, cudaStream_t s) {
  if (n <= 1 || bits <= 0) return false;
  const size_t ntiles = (n + kSortTile - 1) / kSortTile;
  const int passes = (bits + kRadixBits - 1) / kRadixBits;
  const int digit = (bits + passes - 1) / passes, radix = 1 << digit;
  DevBuf<uint32_t> hist(ntiles * radix, s);
  uint64_t *ki = keys, *ko = keys_tmp;
  V *vi = vals, *vo = vals_tmp;
  for (int p = 0; p < passes; ++p) {
    const int shift = p * digit;
    BA_LAUNCH(radix_hist_kernel<<<(unsigned)ntiles, kSortThreads, 0, s>>>(ki, n, shift, radix,
                                                                      hist, ntiles));
    scan_rec(hist, hist, ntiles * radix, s);
    BA_LAUNCH((radix_scatter_kernel<V><<<(unsigned)ntiles, kSortThreads, 0, s>>>(
        ki, vi, ko, vo, n, shift, radix, hist, ntiles)));
    std::swap(ki, ko);
    std::swap(vi, vo);
  }
  return passes & 1;
}

template <typename K>
__global__ void lower_bounds_kernel(const K* sorted, size_t n, uint32_t* p,
                                    size_t m, uint64_t mul) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i > m) return;
  const uint64_t key = (uint64_t)i * mul;
  size_t lo = 0, hi = n;
  while (lo < hi) {
    const size_t mid = (lo + hi) >> 1;
    if ((uint64_t)sorted[mid] < key)
      lo = mid + 1;
    else
      hi = mid;
  }
  p[i] = (uint32_t)lo;
}

}  // namespace

uint64_t exclusive_scan_u32(const uint32_t* in, uint32_t* out, size_t n,
                            cudaStream_t s) {
  if (n == 0) return 0;
  uint32_t last_in = 0, last_out = 0;
  check(cudaMemcpyAsync(&last_in, in + n - 1, 4, cudaMemcpyDeviceToHost, s), "scan");
  scan_rec(in, out, n, s);
  check(cudaMemcpyAsync(&last_out, out + n - 1, 4, cudaMemcpyDeviceToHost, s), "scan");
  check(cudaStreamSynchronize(s), "scan sync");
  return (uint64_t)last_out + last_in;
}

void radix_sort_u64_u32(uint64_t* keys, uint32_t* vals, uint64_t* kt,
                        uint32_t* vt, size_t n, int bits, cudaStream_t s) {
  if (!radix_passes<uint32_t>(keys, vals, kt, vt, n, bits, s)) return;
  check(cudaMemcpyAsync(keys, kt, n * sizeof(uint64_t), cudaMemcpyDeviceToDevice, s),
        "sort copy");
  check(cudaMemcpyAsync(vals, vt, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, s),
        "sort copy");
}
void radix_sort_u64_u64(DevBuf<uint64_t>& keys, DevBuf<uint64_t>& vals, DevBuf<uint64_t>& kt,
                        DevBuf<uint64_t>& vt, size_t n, int bits, cudaStream_t s) {
  if (!radix_passes<uint64_t>(keys, vals, kt, vt, n, bits, s)) return;
  std::swap(keys, kt);
  std::swap(vals, vt);
}

void lower_bounds_u32(const uint32_t* sorted, size_t n, uint32_t* p, size_t m,
                      cudaStream_t s) {
  BA_LAUNCH(lower_bounds_kernel<uint32_t><<<grid_for(m + 1, 256), 256, 0, s>>>(sorted, n, p,
                                                                          m, 1));
}
void lower_bounds_u64(const uint64_t* sorted, size_t n, uint32_t* p, size_t m,
                      uint64_t key_mul, cudaStream_t s) {
  BA_LAUNCH(lower_bounds_kernel<uint64_t><<<grid_for(m + 1, 256), 256, 0, s>>>(sorted, n, p,
                                                                          m, key_mul));
}

}  // namespace ba
