// HISTOGRAM (counts[bins[i]] += 1) and MULTI_REDUCE (values[bins[i]] +=
// data[i]): per-bin reductions over a bin index per item.
//
// HISTOGRAM: up to 16 bins (the suite's default is 10), each thread counts in
// packed 8-bit register counters; up to 16384 bins (55000 for long arrays), a CTA
// counts into a shared-memory histogram, lanes of one bin together where a warp
// holds many of them (kCountTogether: 2^24 items in 50 bins, random bins, one bin
// in long runs, two in turn, nine tenths in one: 28, 26, 28, 29 us; always
// together 92, 29, 29, 31; only where all 32 lanes agree 30, 29, 43, 66); the CTA
// then adds its counts to the global counters with 64-bit atomics.  Integer
// sums do not depend on order, so the counts are exact.  The global counters
// start from counts_init (one small copy kernel).
//
// MULTI_REDUCE: deterministic.  Every thread accumulates into its own row of
// bins in shared memory (bin-major, thread-minor: a warp's 32 accesses hit
// 32 banks whatever the bins), visiting its items in index order; the CTA
// sums the 256 rows per bin in a fixed tree and writes one partial per bin;
// the last CTA to finish sums the partials per bin in a fixed tree and adds
// values_init.
// Up to kPrivateBins bins; beyond that, up to kSharedSums, the items are added
// with FP64 atomics to a CTA's bins in shared memory, and those to the global
// ones; beyond that with global FP64 atomics (order-dependent rounding, within
// the reassociation bound).
//
// Items whose bin is outside [0, num_bins) are skipped (the suite's loop
// would write out of bounds).
#include "b200_internal.cuh"
#include "b200_reduce.cuh"

#include <algorithm>

using namespace b200;

namespace {

constexpr int kBlock = 256;
constexpr int kItems = 8;
constexpr int64_t kSharedBins = 16384;  // HISTOGRAM: 64 KB of 32-bit counters,
constexpr int64_t kMaxSharedBins = 55000;  // for 64 items a bin and more 215 KB
constexpr int64_t kBlockBins = 2048;    // in CTAs of kBlock threads up to here, of 1024 above
constexpr int64_t kPrivateBins = 96;    // MULTI_REDUCE: 256 x 96 x 8 B = 192 KB
constexpr int64_t kSharedSums = 28000;  // a multiple of 4; MULTI_REDUCE: 224 KB of sums
constexpr int kSumThreads = 1024;

int bin_grid(int64_t n) {
  int64_t g = ceil_div(n > 0 ? n : 1, static_cast<int64_t>(kBlock) * kItems);
  const int64_t cap = static_cast<int64_t>(device_info().sm_count) * 4;
  return static_cast<int>(g < cap ? g : cap);
}

__global__ void copy_u64_kernel(const unsigned long long* __restrict__ src,
                                unsigned long long* __restrict__ dst, int64_t m) {
  for (int64_t b = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; b < m;
       b += static_cast<int64_t>(gridDim.x) * blockDim.x)
    dst[b] = src[b];
}

constexpr unsigned int kNoBin = 0xffffffffu;  // the key of an item outside the bins

// An add to shared memory takes a cycle or two per lane that hits the same
// counter, __match_any_sync a step per bin that the warp's lanes hold: from this
// many lanes of one bin on (a middle lane's, the likeliest to lie in a run or in
// a frequent bin) the lanes of a bin are counted together.
constexpr int kCountTogether = 12;

template <int BS>
__global__ void __launch_bounds__(BS)
histogram_shared_kernel(const int64_t* __restrict__ bins, int64_t n, int64_t num_bins,
                        unsigned long long* __restrict__ counts) {
  extern __shared__ unsigned int s_cnt[];
  for (int64_t b = threadIdx.x; b < num_bins; b += BS) s_cnt[b] = 0u;
  __syncthreads();
  const unsigned int lane = threadIdx.x & 31u;
  for (int64_t t0 = static_cast<int64_t>(blockIdx.x) * (BS * kItems); t0 < n;
       t0 += static_cast<int64_t>(gridDim.x) * (BS * kItems)) {
    int64_t b[kItems];
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
      const int64_t i = t0 + u * BS + threadIdx.x;
      b[u] = (i < n) ? __ldcs(bins + i) : -1;
    }
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
      const bool ok = b[u] >= 0 && b[u] < num_bins;
      const unsigned int key = ok ? static_cast<unsigned int>(b[u]) : kNoBin;
      unsigned int peers = __ballot_sync(0xffffffffu, key == __shfl_sync(0xffffffffu, key, 16));
      if (peers == 0xffffffffu) {
        if (ok && lane == 0u) atomicAdd(&s_cnt[key], 32u);
      } else if (__popc(peers) >= kCountTogether) {
        peers = __match_any_sync(0xffffffffu, key);
        if (ok && lane == __ffs(peers) - 1u) atomicAdd(&s_cnt[key], __popc(peers));
      } else if (ok) {
        atomicAdd(&s_cnt[key], 1u);
      }
    }
  }
  __syncthreads();
  for (int64_t b = threadIdx.x; b < num_bins; b += BS)
    if (s_cnt[b]) atomicAdd(&counts[b], static_cast<unsigned long long>(s_cnt[b]));
}

// Up to 16 bins: every thread counts in two 64-bit words of 8-bit counters
// (bin b adds 1 << 8*(b mod 8) to word b / 8: a shift and an add per item),
// unpacked into 32-bit totals before any byte can overflow; warp and CTA
// sums follow, and one 64-bit atomic per bin and CTA.
constexpr int64_t kRegisterBins = 16;

__global__ void __launch_bounds__(kBlock)
histogram_register_kernel(const int64_t* __restrict__ bins, int64_t n, int num_bins,
                          bool vec, unsigned long long* __restrict__ counts) {
  __shared__ unsigned int s_tot[kBlock / 32][kRegisterBins];
  unsigned int acc[kRegisterBins];
#pragma unroll
  for (int k = 0; k < kRegisterBins; ++k) acc[k] = 0u;
  unsigned long long lo = 0ull, hi = 0ull;
  int pending = 0;
  auto flush = [&]() {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      acc[k] += static_cast<unsigned int>((lo >> (8 * k)) & 0xffull);
      acc[8 + k] += static_cast<unsigned int>((hi >> (8 * k)) & 0xffull);
    }
    lo = hi = 0ull;
    pending = 0;
  };
  auto count = [&](int64_t b) {
    const bool ok = b >= 0 && b < num_bins;
    const unsigned long long one = ok ? (1ull << (8 * (b & 7))) : 0ull;
    if (b < 8) lo += one; else hi += one;
  };
  // item pairs with 16-byte loads (bins is 16-byte aligned when `vec`)
  const int64_t units = vec ? (n >> 1) : n;
  for (int64_t t0 = static_cast<int64_t>(blockIdx.x) * (kBlock * kItems); t0 < units;
       t0 += static_cast<int64_t>(gridDim.x) * (kBlock * kItems)) {
    longlong2 b[kItems];
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
      const int64_t i = t0 + u * kBlock + threadIdx.x;
      if (vec) {
        b[u] = (i < units) ? __ldcs(reinterpret_cast<const longlong2*>(bins) + i)
                           : make_longlong2(-1, -1);
      } else {
        b[u] = make_longlong2((i < units) ? __ldcs(bins + i) : -1, -1);
      }
    }
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
      count(b[u].x);
      count(b[u].y);
    }
    pending += 2 * kItems;
    if (pending > 255 - 2 * kItems) flush();
  }
  if (vec && (n & 1) && blockIdx.x == 0 && threadIdx.x == 0) count(__ldcs(bins + n - 1));
  flush();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < kRegisterBins; ++k) {
    unsigned int v = acc[k];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if (lane == 0) s_tot[warp][k] = v;
  }
  __syncthreads();
  if (threadIdx.x < num_bins) {
    unsigned long long t = 0ull;
#pragma unroll
    for (int w = 0; w < kBlock / 32; ++w) t += s_tot[w][threadIdx.x];
    if (t) atomicAdd(&counts[threadIdx.x], t);
  }
}

__global__ void histogram_global_kernel(const int64_t* __restrict__ bins, int64_t n,
                                        int64_t num_bins,
                                        unsigned long long* __restrict__ counts) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t b = __ldcs(bins + i);
    if (b >= 0 && b < num_bins) atomicAdd(&counts[b], 1ull);
  }
}

// s_rows: num_bins x kBlock doubles (bin-major).  partials: gridDim.x x num_bins.
__global__ void __launch_bounds__(kBlock)
multi_reduce_private_kernel(const int64_t* __restrict__ bins, const double* __restrict__ data,
                            int64_t n, int num_bins, const double* __restrict__ values_init,
                            double* __restrict__ values, double* __restrict__ partials,
                            unsigned int* __restrict__ counter) {
  extern __shared__ double s_rows[];
  __shared__ bool last_flag;
  for (int k = threadIdx.x; k < num_bins * kBlock; k += kBlock) s_rows[k] = 0.0;
  __syncthreads();
  for (int64_t t0 = static_cast<int64_t>(blockIdx.x) * (kBlock * kItems); t0 < n;
       t0 += static_cast<int64_t>(gridDim.x) * (kBlock * kItems)) {
    int64_t b[kItems];
    double v[kItems];
#pragma unroll
    for (int u = 0; u < kItems; ++u) {
      const int64_t i = t0 + u * kBlock + threadIdx.x;
      b[u] = (i < n) ? __ldcs(bins + i) : -1;
      v[u] = (i < n) ? __ldcs(data + i) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kItems; ++u)
      if (b[u] >= 0 && b[u] < num_bins) s_rows[b[u] * kBlock + threadIdx.x] += v[u];
  }
  __syncthreads();
  // per bin: lane l sums rows l, l+32, ..., then a fixed warp tree
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int bb = warp; bb < num_bins; bb += kBlock / 32) {
    double s = 0.0;
#pragma unroll
    for (int r = lane; r < kBlock; r += 32) s += s_rows[bb * kBlock + r];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (lane == 0) {
      partials[static_cast<int64_t>(blockIdx.x) * num_bins + bb] = s;
      __threadfence();  // every writer's partial is visible before the arrival
    }
  }
  if (arrive_last(counter, &last_flag)) {
    // per bin: lane l sums the partials of CTAs l, l+32, ..., then a fixed tree
    for (int bb = warp; bb < num_bins; bb += kBlock / 32) {
      double s = 0.0;
      for (int c = lane; c < static_cast<int>(gridDim.x); c += 32 * 10) {
        double v[10];  // loads in flight together, added in order
#pragma unroll
        for (int u = 0; u < 10; ++u)
          v[u] = c + 32 * u < static_cast<int>(gridDim.x)
                     ? __ldcg(partials + static_cast<int64_t>(c + 32 * u) * num_bins + bb)
                     : 0.0;
#pragma unroll
        for (int u = 0; u < 10; ++u) s += v[u];
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
      if (lane == 0) values[bb] = values_init[bb] + s;
    }
    if (threadIdx.x == 0) *counter = 0u;
  }
}

__global__ void copy_f64_kernel(const double* __restrict__ src, double* __restrict__ dst,
                                int64_t m) {
  for (int64_t b = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; b < m;
       b += static_cast<int64_t>(gridDim.x) * blockDim.x)
    dst[b] = src[b];
}

__global__ void multi_reduce_global_kernel(const int64_t* __restrict__ bins,
                                           const double* __restrict__ data, int64_t n,
                                           int64_t num_bins, double* __restrict__ values) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t b = __ldcs(bins + i);
    if (b >= 0 && b < num_bins) atomicAdd(&values[b], __ldcs(data + i));
  }
}

// The lanes of `rest` (not empty) with one of its lanes' key, the middle one's
// if it is in there.
__device__ __forceinline__ unsigned int peers_of(unsigned int key, unsigned int rest) {
  const int lane = (rest >> 16) & 1u ? 16 : __ffs(rest) - 1;
  return rest & __ballot_sync(0xffffffffu, key == __shfl_sync(0xffffffffu, key, lane));
}

// `copies` sets of the CTA's sums, one for every few warps: an FP64 add to
// shared memory is a compare-and-swap loop, which lanes and warps that hit one
// bin make each other repeat (2^24 items in 97 random bins: 2724 us with global
// atomics, 449 with one set, 103 with 32; in 3000 bins: 306, 97 and 83).  A thread
// takes four consecutive items and adds up neighbours of one bin; lanes whose four
// items continue the bin of the lane before add up along the warp; and where many
// lanes of a step still hold one bin, the warp sums them.
constexpr int kRun = 4;
// Where a bin's sum lies in a set: the low two bits are turned so that bins 4
// apart, as the lanes of a step hold them where bins follow each other, fall
// into different banks (2^24 items over 16384 bins in turn: 82 -> 70 us).
__host__ __device__ constexpr int sum_at(unsigned int bin) {
  return static_cast<int>(bin ^ ((bin >> 4) & 3u));
}
__host__ __device__ constexpr int sum_set(int num_bins) { return (num_bins + 3) & ~3; }
constexpr int kRunLanes = 8;      // lanes with neighbours of one bin that make it worth while
constexpr int kSumTogether = 12;  // lanes of one bin: five adds on the FP64 pipe against as many

__global__ void __launch_bounds__(kSumThreads)
multi_reduce_shared_kernel(const int64_t* __restrict__ bins, const double* __restrict__ data,
                           int64_t n, int num_bins, int copies, bool vec,
                           double* __restrict__ values) {
  extern __shared__ double s_sum[];
  const int set = sum_set(num_bins);
  for (int b = threadIdx.x; b < copies * set; b += kSumThreads) s_sum[b] = 0.0;
  __syncthreads();
  constexpr unsigned int kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  double* sums = s_sum + (threadIdx.x >> 5) % copies * set;
  unsigned int held = kNoBin;  // the bin of the lanes' `acc`: the warp's last items were all of it
  double acc = 0.0;
  auto flush = [&] {
    if (held != kNoBin) {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(kAll, acc, off);
      if (lane == 0) atomicAdd(&sums[sum_at(held)], acc);
    }
    acc = 0.0;
  };
  constexpr int kGroups = kItems / kRun;
  constexpr int64_t kStep = static_cast<int64_t>(kSumThreads) * kRun;
  for (int64_t t0 = static_cast<int64_t>(blockIdx.x) * (kGroups * kStep); t0 < n;
       t0 += static_cast<int64_t>(gridDim.x) * (kGroups * kStep)) {
    int64_t b[kGroups][kRun];
    double v[kGroups][kRun];
#pragma unroll
    for (int g = 0; g < kGroups; ++g) {
      const int64_t i = t0 + g * kStep + threadIdx.x * kRun;
      if (vec && i + kRun <= n) {
#pragma unroll
        for (int q = 0; q < kRun; q += 2) {
          const longlong2 k2 = __ldcs(reinterpret_cast<const longlong2*>(bins + i + q));
          const double2 v2 = __ldcs(reinterpret_cast<const double2*>(data + i + q));
          b[g][q] = k2.x;
          b[g][q + 1] = k2.y;
          v[g][q] = v2.x;
          v[g][q + 1] = v2.y;
        }
      } else {
#pragma unroll
        for (int q = 0; q < kRun; ++q) {
          b[g][q] = i + q < n ? __ldcs(bins + i + q) : -1;
          v[g][q] = i + q < n ? __ldcs(data + i + q) : 0.0;
        }
      }
    }
#pragma unroll
    for (int g = 0; g < kGroups; ++g) {
      unsigned int key[kRun];
#pragma unroll
      for (int q = 0; q < kRun; ++q)
        key[q] = b[g][q] >= 0 && b[g][q] < num_bins ? static_cast<unsigned int>(b[g][q]) : kNoBin;
      constexpr int kLast = kRun - 1;
      bool equal = false, whole = true;  // neighbours in one bin: any, all
#pragma unroll
      for (int q = 1; q < kRun; ++q) {
        equal |= key[q] == key[q - 1];
        whole &= key[q] == key[q - 1];
      }
      const unsigned int step = __ballot_sync(kAll, key[1] != kNoBin);
      const bool together = step && __popc(peers_of(key[1], step)) >= kSumTogether;
      if (__popc(__ballot_sync(kAll, equal)) >= kRunLanes) {
#pragma unroll
        for (int q = 1; q < kRun; ++q) {
          if (key[q] == key[q - 1]) {
            v[g][q] += v[g][q - 1];
            key[q - 1] = kNoBin;
          }
        }
        const unsigned int before = __shfl_up_sync(kAll, key[kLast], 1);
        const unsigned int heads =
            __ballot_sync(kAll, lane == 0 || !whole || before != key[kLast]);
        if (heads == 1u && __all_sync(kAll, whole)) {
          if (key[kLast] != held) {
            flush();
            held = key[kLast];
          }
          acc += v[g][kLast];
          continue;
        }
        const int start = 31 - __clz(static_cast<int>(heads & (kAll >> (31 - lane))));
        for (int off = 1; __any_sync(kAll, lane - off >= start); off *= 2) {
          const double left = __shfl_up_sync(kAll, v[g][kLast], off);
          if (lane - off >= start) v[g][kLast] += left;
        }
        if (lane < 31 && !((heads >> (lane + 1)) & 1u)) key[kLast] = kNoBin;  // added to the next
      }
#pragma unroll
      for (int q = 0; q < kRun; ++q) {
        bool mine = key[q] != kNoBin;
        if (together) {
          unsigned int rest = __ballot_sync(kAll, mine);
          while (rest) {  // the same in every lane
            const unsigned int peers = peers_of(key[q], rest);
            if (__popc(peers) < kSumTogether) break;
            double sum = (peers >> lane) & 1u ? v[g][q] : 0.0;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(kAll, sum, off);
            if (lane == __ffs(peers) - 1) atomicAdd(&sums[sum_at(key[q])], sum);
            rest &= ~peers;
          }
          mine = (rest >> lane) & 1u;
        }
        if (mine) atomicAdd(&sums[sum_at(key[q])], v[g][q]);
      }
    }
  }
  flush();
  __syncthreads();
  for (int b = threadIdx.x; b < num_bins; b += kSumThreads) {
    double s = 0.0;
    for (int c = 0; c < copies; ++c) s += s_sum[c * set + sum_at(b)];
    if (s != 0.0) atomicAdd(&values[b], s);
  }
}

int small_grid(int64_t m) {
  const int64_t g = ceil_div(m > 0 ? m : 1, 256);
  return static_cast<int>(g < 1024 ? g : 1024);
}

}  // namespace

extern "C" {

int b200_algorithm_histogram(const int64_t* bins, int64_t n, int64_t num_bins,
                             const unsigned long long* counts_init, unsigned long long* counts,
                             const b200_tune* tune, b200_stream_t stream) {
  (void)tune;
  if (n < 0 || num_bins < 1 || !counts_init || !counts || (n > 0 && !bins))
    return invalid("b200_algorithm_histogram: bad args");
  cudaStream_t st = as_stream(stream);
  copy_u64_kernel<<<small_grid(num_bins), 256, 0, st>>>(counts_init, counts, num_bins);
  int launches = 1;
  if (n > 0) {
    if (num_bins <= kRegisterBins) {
      histogram_register_kernel<<<bin_grid(n), kBlock, 0, st>>>(
          bins, n, static_cast<int>(num_bins), aligned16(bins), counts);
    } else if (num_bins <= kSharedBins || (num_bins <= kMaxSharedBins && n >= 64 * num_bins)) {
      const size_t smem = static_cast<size_t>(num_bins) * sizeof(unsigned int);
      // many bins: few large CTAs, since each adds all its bins to the global ones
      const bool large = num_bins > kBlockBins;
      const void* kernel = large ? reinterpret_cast<const void*>(histogram_shared_kernel<1024>)
                                 : reinterpret_cast<const void*>(histogram_shared_kernel<kBlock>);
      if (smem > 48 * 1024) {
        const int rc = allow_dynamic_smem(kernel, smem, "b200_algorithm_histogram");
        if (rc != B200_OK) return rc;
      }
      if (large) {
        const int64_t grid = std::min<int64_t>(ceil_div(n, 1024 * kItems),
                                               device_info().sm_count * (smem <= 110000 ? 2 : 1));
        histogram_shared_kernel<1024><<<static_cast<int>(grid), 1024, smem, st>>>(bins, n, num_bins,
                                                                                 counts);
      } else {
        // (2^24 items in 50 bins: 28 us with eight CTAs per SM, 31 with four; in 1000,
        // where every CTA has more to add to the global bins: 35 and 33)
        const int64_t grid = std::min<int64_t>(ceil_div(n, kBlock * kItems),
                                               device_info().sm_count * (num_bins <= 64 ? 8 : 4));
        histogram_shared_kernel<kBlock><<<static_cast<int>(grid), kBlock, smem, st>>>(
            bins, n, num_bins, counts);
      }
    } else {
      histogram_global_kernel<<<bin_grid(n) * 4, kBlock, 0, st>>>(bins, n, num_bins, counts);
    }
    ++launches;
  }
  return after_launch("b200_algorithm_histogram", launches);
}

size_t b200_multi_reduce_workspace_bytes(int64_t n, int64_t num_bins) {
  if (num_bins < 1 || num_bins > kPrivateBins) return 256;
  return 256 + static_cast<size_t>(bin_grid(n)) * static_cast<size_t>(num_bins) * 8;
}

int b200_basic_multi_reduce(const int64_t* bins, const double* data, int64_t n,
                            int64_t num_bins, const double* values_init, double* values,
                            void* workspace, size_t workspace_bytes, const b200_tune* tune,
                            b200_stream_t stream) {
  (void)tune;
  if (n < 0 || num_bins < 1 || !values_init || !values || (n > 0 && (!bins || !data)))
    return invalid("b200_basic_multi_reduce: bad args");
  cudaStream_t st = as_stream(stream);
  if (num_bins > kPrivateBins || n == 0) {
    copy_f64_kernel<<<small_grid(num_bins), 256, 0, st>>>(values_init, values, num_bins);
    // each CTA clears and adds all its sums: from 350 items a bin on (random bins,
    // against global atomics: 2^20 items in 2049 bins 22 us and 33; 2^18 in 1000 bins
    // 22 and 18)
    if (n >= (1 << 18) && num_bins <= kSharedSums && n >= 350 * num_bins) {
      const int set = sum_set(static_cast<int>(num_bins));
      const int copies = std::min<int>(32, static_cast<int>(kSharedSums) / set);
      const size_t smem = static_cast<size_t>(copies * set) * sizeof(double);
      const int rc = allow_dynamic_smem(
          reinterpret_cast<const void*>(multi_reduce_shared_kernel), smem,
          "b200_basic_multi_reduce");
      if (rc != B200_OK) return rc;
      const int64_t fit = smem <= 110000 ? 2 : 1;  // CTAs per SM
      const int64_t grid = std::min<int64_t>(ceil_div(n, kSumThreads * kItems),
                                             fit * device_info().sm_count);
      multi_reduce_shared_kernel<<<static_cast<int>(grid), kSumThreads, smem, st>>>(
          bins, data, n, static_cast<int>(num_bins), copies, aligned16(bins) && aligned16(data),
          values);
    } else if (n > 0)
      multi_reduce_global_kernel<<<bin_grid(n) * 4, kBlock, 0, st>>>(bins, data, n, num_bins,
                                                                      values);
    return after_launch("b200_basic_multi_reduce", n > 0 ? 2 : 1);
  }
  const size_t need = b200_multi_reduce_workspace_bytes(n, num_bins);
  if (!workspace || workspace_bytes < need) {
    set_error("b200_basic_multi_reduce: workspace %zu bytes, need %zu", workspace_bytes, need);
    return B200_ERR_WORKSPACE;
  }
  const size_t smem = static_cast<size_t>(num_bins) * kBlock * sizeof(double);
  if (smem > 48 * 1024) {
    const int rc = allow_dynamic_smem(reinterpret_cast<const void*>(multi_reduce_private_kernel),
                                      smem, "b200_basic_multi_reduce");
    if (rc != B200_OK) return rc;
  }
  char* w = static_cast<char*>(workspace);
  // no more CTAs than are resident at once: the last one sums a partial of each
  // (50 bins, 2^24 items: 133 us with 608 CTAs, 91 with 304)
  const int64_t resident = device_info().sm_count * std::max<int64_t>(1, 220000 / (smem + 1024));
  multi_reduce_private_kernel<<<static_cast<int>(std::min<int64_t>(bin_grid(n), resident)),
                                kBlock, smem, st>>>(
      bins, data, n, static_cast<int>(num_bins), values_init, values,
      reinterpret_cast<double*>(w + 256), reinterpret_cast<unsigned int*>(w));
  return after_launch("b200_basic_multi_reduce");
}

}  // extern "C"
