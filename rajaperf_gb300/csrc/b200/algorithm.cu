// Algorithm group: SCAN (exclusive prefix sum, FP64 and int64) and REDUCE_SUM.
//
// SCAN is a single-pass scan: every CTA takes the next tile id from a counter
// (so a CTA only ever waits on tiles already owned by running CTAs).  Three
// kernels: one CTA per tile with a lookback warp (scan_kernel), and two
// persistent ones on a ring of shared-memory stages with one scanner warp that
// gives all tiles their prefixes, for int64 (pipe::scan_pipelined) and for FP64
// (pipe64::scan_pipelined_f64).  Flags carry a launch
// epoch, so the workspace never needs re-zeroing between calls (and the call
// can be captured in a CUDA graph): the CTA that draws the launch's last tile
// id resets the tile counter and advances the epoch.  Every wait is bounded; a
// wait that gives up sets the error word of the workspace header (byte offset
// 16) and the call's results are invalid.
#include "b200_internal.cuh"
#include "b200_fma_form.cuh"
#include "b200_async.cuh"
#include "b200_f64emu.cuh"
#include "b200_launch.cuh"
#include "b200_lookback.cuh"
#include "b200_pipeline.cuh"
#include "b200_reduce.cuh"

#include <type_traits>

using namespace b200;

namespace {

constexpr int kScanBlock = 256;                         // loader threads
constexpr int kScanThreads = kScanBlock + 32;           // + the lookback warp
constexpr int kScanItemsMin = 16;                       // smallest tile: 4096 items
constexpr int kScanItemsDefault = 32;                   // default tile: 8192 items
constexpr int kScanTileMin = kScanBlock * kScanItemsMin;

// One CTA per tile of kScanBlock * IT items.  Warp 0 is the lookback warp:
// it walks the predecessors' flags as soon as the tile id is known, while
// warps 1..8 (the loaders) stage the tile in shared memory (padded so the
// per-thread runs of IT consecutive items are conflict-free), reduce it and
// publish the aggregate.  The lookback warp then publishes the inclusive
// prefix, and the loaders write the tile out.  Named barriers: 1 = loaders
// only, 2 = aggregate ready (loaders arrive, lookback warp waits), 3 =
// exclusive prefix ready (lookback warp arrives, loaders wait).
// 16-byte vector of two T (double2 / longlong2).
template <typename T> struct Vec2;
template <> struct Vec2<double> { using type = double2; };
template <> struct Vec2<long long> { using type = longlong2; };

template <typename T, int IT, bool VEC>
__global__ void __launch_bounds__(kScanThreads, 3)
scan_kernel(const T* __restrict__ x, T* __restrict__ y, int64_t n, T init,
            ScanHeader* __restrict__ hdr, TileDesc* __restrict__ descs, uint64_t limit_ns) {
  using V2 = typename Vec2<T>::type;
  constexpr int kTile = kScanBlock * IT;
  constexpr int kPadShift = (IT == 32) ? 5 : 4;
  extern __shared__ __align__(16) unsigned char s_raw[];
  T* s_tile = reinterpret_cast<T*>(s_raw);
  __shared__ T s_warp[kScanBlock / 32];
  __shared__ T s_excl;
  __shared__ T s_agg;
  __shared__ unsigned int s_tile_id;
  __shared__ unsigned long long s_epoch;
  auto pad = [](int i) { return i + (i >> kPadShift); };

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  take_tile(hdr, &s_tile_id, &s_epoch);
  const unsigned int tile = s_tile_id;
  const unsigned long long epoch = s_epoch;
  const unsigned long long AGG = epoch * 4 + 1, INC = epoch * 4 + 2;
  const int64_t base = static_cast<int64_t>(tile) * kTile;

  if (warp == 0) {
    // ---- lookback warp ----
    // One round examines 32 * kLookbackPerLane predecessors, nearest first
    // (window slot w = j * 32 + lane is predecessor p_hi - w).
    const T exclusive =
        (tile > 0) ? lookback_exclusive<T>(descs, tile, AGG, INC, hdr, limit_ns) : init;
    named_sync(2, kScanThreads);  // the loaders have the tile aggregate
    if (lane == 0) {
      desc_store(descs + tile, INC, to_bits<T>(exclusive + s_agg));
      s_excl = exclusive;
    }
    named_arrive(3, kScanThreads);
  } else {
    // ---- loaders ----
    const int ltid = tid - 32, lwarp = warp - 1;
    if (VEC && base + kTile <= n) {
      // 16-byte loads of item pairs (x 16-byte aligned, tiles start even)
      const V2* xv = reinterpret_cast<const V2*>(x + base);
#pragma unroll
      for (int u = 0; u < IT / 2; ++u) {
        const int k2 = u * kScanBlock + ltid;
        const V2 v = __ldcs(xv + k2);
        s_tile[pad(2 * k2)] = v.x;
        s_tile[pad(2 * k2 + 1)] = v.y;
      }
    } else if (base + kTile <= n) {
#pragma unroll
      for (int u = 0; u < IT; ++u) {
        const int k = u * kScanBlock + ltid;
        s_tile[pad(k)] = __ldcs(x + base + k);
      }
    } else {
#pragma unroll
      for (int u = 0; u < IT; ++u) {
        const int k = u * kScanBlock + ltid;
        const int64_t i = base + k;
        s_tile[pad(k)] = (i < n) ? __ldcs(x + i) : T(0);
      }
    }
    named_sync(1, kScanBlock);
    // Each thread sums its IT consecutive items; a scan of the thread totals
    // gives every thread its offset inside the tile.
    T run = T(0);
#pragma unroll
    for (int u = 0; u < IT; ++u) run += s_tile[pad(ltid * IT + u)];
    const T incl = warp_inclusive_scan(run);
    if (lane == 31) s_warp[lwarp] = incl;
    named_sync(1, kScanBlock);
    if (lwarp == 0) {
      const T w = (lane < kScanBlock / 32) ? s_warp[lane] : T(0);
      const T wi = warp_inclusive_scan(w);
      if (lane < kScanBlock / 32) s_warp[lane] = wi - w;  // exclusive warp offsets
      if (lane == kScanBlock / 32 - 1) {
        s_agg = wi;                                       // tile aggregate
        if (tile > 0) desc_store(descs + tile, AGG, to_bits<T>(wi));
      }
    }
    named_sync(1, kScanBlock);
    named_arrive(2, kScanThreads);
    // tile-local exclusive prefixes, in place
    {
      T r = s_warp[lwarp] + (incl - run);
#pragma unroll
      for (int u = 0; u < IT; ++u) {
        const int k = pad(ltid * IT + u);
        const T xv = s_tile[k];
        s_tile[k] = r;
        r += xv;
      }
    }
    named_sync(1, kScanBlock);
    named_sync(3, kScanThreads);  // the lookback warp has the exclusive prefix
    const T prefix = s_excl;
    if (VEC && base + kTile <= n) {
      V2* yv = reinterpret_cast<V2*>(y + base);
#pragma unroll
      for (int u = 0; u < IT / 2; ++u) {
        const int k2 = u * kScanBlock + ltid;
        V2 v;
        v.x = prefix + s_tile[pad(2 * k2)];
        v.y = prefix + s_tile[pad(2 * k2 + 1)];
        __stcs(yv + k2, v);
      }
    } else if (base + kTile <= n) {
#pragma unroll
      for (int u = 0; u < IT; ++u) {
        const int k = u * kScanBlock + ltid;
        __stcs(y + base + k, prefix + s_tile[pad(k)]);
      }
    } else {
#pragma unroll
      for (int u = 0; u < IT; ++u) {
        const int k = u * kScanBlock + ltid;
        const int64_t i = base + k;
        if (i < n) __stcs(y + i, prefix + s_tile[pad(k)]);
      }
    }
  }

}

// ---- pipelined persistent SCAN, int64 -----------------------------------------
// One CTA per SM, but the scanner's, on the stage ring of b200_pipeline.cuh
// (producer warp 0, prefix warp 2), plus:
//  * aggregator (warp 1): sums each tile as it lands and publishes the
//    aggregate at once;
//  * compute (warps 3-6): a thread owns a run of 32 consecutive items (16
//    item pairs), sums it, scans the run sums across the tile and, when the
//    tile's exclusive prefix arrives, writes every item's prefix in place;
//  * store (warp 7): writes a finished tile back with one bulk store and
//    frees the stage once the store has read it (mbarrier ready[s]: compute
//    -> store).
// A compute thread visits its pairs rotated by (run mod 16), so every 16-byte
// shared-memory access of a warp is conflict-free without padding the
// bulk-copied tile.
namespace pipe {

using ring::kStages;
using ring::kTile;
using ring::kEnd;
constexpr int kComputeWarps = 4;
constexpr int kFirstCompute = 3;
constexpr int kStoreWarp = kFirstCompute + kComputeWarps;
constexpr int kThreads = 32 * (kStoreWarp + 1);
constexpr int kRuns = 32 * kComputeWarps;    // 128 runs per tile
constexpr int kPairs = kTile / kRuns / 2;    // 16 pairs per run

template <typename T>
struct Smem {
  ring::Ring<T, T> r;
  T warp_total[kComputeWarps];
  uint64_t ready[kStages];  // compute -> store warp: the stage holds results
  int fail_loaded;          // compute group: a wait before its first barrier gave up
  int fail_prefix;          // compute group: a wait before its second barrier gave up
  unsigned long long ticket;  // the CTA's first
};

template <typename T>
constexpr size_t smem_bytes() { return sizeof(Smem<T>) + 128; }
static_assert(sizeof(Smem<long long>) + 128 <= 232448, "shared memory budget");

template <typename T>
__global__ void __launch_bounds__(kThreads, 1)
scan_pipelined(const T* x, T* y, int64_t n, T init, unsigned int tiles, ScanHeader* hdr,
               TileDesc* descs, uint64_t limit_ns) {
  using V2 = typename Vec2<T>::type;
  extern __shared__ unsigned char s_raw[];
  Smem<T>& sm = *reinterpret_cast<Smem<T>*>(
      (reinterpret_cast<uintptr_t>(s_raw) + 127) & ~static_cast<uintptr_t>(127));
  ring::Ring<T, T>& r = sm.r;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  if (tid == 0) {
    ring::init(r, limit_ns);
    for (int s = 0; s < kStages; ++s) mbar_init(&sm.ready[s], 1);
    sm.fail_loaded = 0;
    sm.fail_prefix = 0;
    mbar_init_fence();
  }
  const unsigned int z = begin_early();
  x += z;
  hdr += z;
  descs += z;
  if (tid == 0) ring::first_ticket(hdr, tiles, &sm.ticket);
  __syncthreads();
  // the CTA with the first ticket scans the aggregates of all the others (a
  // single tile needs no scanner)
  const unsigned int bias = tiles > 1u ? 1u : 0u;
  if (static_cast<unsigned int>(sm.ticket) < bias) {
    if (warp == 0) ring::scan_aggregates(descs, tiles, init, sm.ticket >> 32, hdr, limit_ns);
    return;
  }

  if (warp == 0) {
    ring::produce(r, x, n, tiles, hdr, 1, &sm.ticket, bias);
  } else if (warp == 1) {
    // ---- aggregator: lane L sums pairs L, L + 32, ... (conflict-free) ----
    for (int k = 0;; ++k) {
      const int s = k % kStages;
      if (!ring::wait(r, &r.full[s], (k / kStages) & 1, hdr)) break;
      const unsigned int tile = r.ticket[s];
      if (tile == kEnd) break;
      const V2* tv = reinterpret_cast<const V2*>(r.tile[s]);
      T total = T(0);
#pragma unroll 16
      for (int q = lane; q < kTile / 2; q += 32) {
        const V2 v = tv[q];
        total += v.x;
        total += v.y;
      }
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) total += __shfl_xor_sync(0xffffffffu, total, off);
      if (lane == 0) {
        desc_store(descs + tile, r.epoch * 4 + 1, to_bits<T>(total));
        mbar_arrive(&r.summed[s]);  // the tile is read: it may be overwritten
      }
      __syncwarp();
    }
  } else if (warp < kFirstCompute) {
    ring::fetch_prefixes(r, descs, init, hdr);
  } else if (warp < kStoreWarp) {
    // ---- compute ----
    // The four warps decide together whether to go on: a warp whose wait
    // gave up sets a flag before the next group barrier and every thread
    // reads it after that barrier, so no thread is left at a later barrier.
    // The two barriers of an iteration use separate flags: a failure in the
    // next iteration can only be recorded after every thread has passed
    // this iteration's reads of the flag it sets.
    const int ct = tid - 32 * kFirstCompute, cw = ct >> 5;
    const int rot = ct & (kPairs - 1);
    volatile int* fail_loaded = &sm.fail_loaded;
    volatile int* fail_prefix = &sm.fail_prefix;
    for (int k = 0;; ++k) {
      const int s = k % kStages;
      const uint32_t par = (k / kStages) & 1;
      const bool loaded = ring::wait(r, &r.full[s], par, hdr);
      const unsigned int tile = r.ticket[s];
      if (!loaded) *fail_loaded = 1;
      V2* tv = reinterpret_cast<V2*>(r.tile[s]) + ct * kPairs;
      V2 v[kPairs];
      T head = T(0), tail = T(0);  // pairs q < rot come first in index order
      if (loaded && tile != kEnd) {
#pragma unroll
        for (int w = 0; w < kPairs; ++w) v[w] = tv[(w + rot) & (kPairs - 1)];
#pragma unroll
        for (int w = 0; w < kPairs; ++w) {
          if (w >= kPairs - rot) {
            head += v[w].x;
            head += v[w].y;
          } else {
            tail += v[w].x;
            tail += v[w].y;
          }
        }
      }
      const T rs = head + tail;
      const T inc = warp_inclusive_scan(rs);
      if (lane == 31) sm.warp_total[cw] = inc;
      named_sync(1, 32 * kComputeWarps);
      if (*fail_loaded || tile == kEnd) {
        if (ct == 0 && !*fail_loaded) mbar_arrive(&sm.ready[s]);  // end marker for the store warp
        break;
      }
      T woff = T(0);
      for (int w = 0; w < cw; ++w) woff += sm.warp_total[w];
      const bool have_prefix =
          ring::wait(r, &r.prefix[s], par, hdr) && ring::wait(r, &r.summed[s], par, hdr);
      if (have_prefix) {
        const T base = r.excl[s] + (woff + (inc - rs));
        T run = base + head;
#pragma unroll
        for (int w = 0; w < kPairs; ++w) {
          if (w == kPairs - rot) run = base;
          V2 o;
          o.x = run;
          run += v[w].x;
          o.y = run;
          run += v[w].y;
          tv[(w + rot) & (kPairs - 1)] = o;
        }
        fence_proxy_async_smem();
      } else {
        *fail_prefix = 1;
      }
      named_sync(2, 32 * kComputeWarps);
      if (*fail_prefix) break;
      const int64_t first = static_cast<int64_t>(tile) * kTile;
      if (first + kTile > n) {
        // the ragged last tile: plain stores
        for (int i = ct; first + i < n; i += 32 * kComputeWarps) y[first + i] = r.tile[s][i];
      }
      if (ct == 0) mbar_arrive(&sm.ready[s]);
    }
  } else {
    // ---- store: one bulk store per finished tile, then the stage is free ----
    for (int k = 0;; ++k) {
      const int s = k % kStages;
      if (!ring::wait(r, &sm.ready[s], (k / kStages) & 1, hdr)) break;
      const unsigned int tile = r.ticket[s];
      if (tile == kEnd) break;
      const int64_t first = static_cast<int64_t>(tile) * kTile;
      if (lane == 0) {
        if (first + kTile <= n) {
          bulk_store(y + first, r.tile[s], kTile * sizeof(T));
          bulk_commit();
          bulk_wait_read<0>();
        }
        mbar_arrive(&r.empty[s]);
      }
      __syncwarp();
    }
    if (lane == 0) bulk_wait_all();
  }

  __syncthreads();
  if (tid == 0) ring::drain(r);
}

}  // namespace pipe

// ---- pipelined persistent SCAN, FP64 ----------------------------------------
// The ring again, arranged around the FP64 pipe, which bounds an FP64 scan: at
// 2 thread instructions per clock and SM (595 G/s), the tile kernel's three
// adds per item (run total, prefix in the tile, plus the tile's prefix) take
// 0.40 ms at 2^26 items, the memory traffic 0.16 ms.  Here an item costs one
// or two:
//  * four aggregator warps total the runs on the integer pipes.  Items of one
//    sign add as integers in units of 2^-56 of the largest one's binade, and
//    the total is rounded once, where a chain of FP64 adds rounds 34 times.
//    What an item more than 4 binades below the largest has under that unit is
//    cut, so the total is low by less than 33 units, 2^-51 of itself; measured
//    against exact prefixes, the scan's error is the tile kernel's or less, for
//    uniform, log-normal and integer items.  A run of both signs, whose total may cancel, or with an
//    infinity, a NaN or nothing above 2^-960, is totalled with FP64 adds.
//  * two groups of four compute warps take alternate tiles, a thread a run of
//    34 consecutive items.  Where the tile's exclusive prefix has the run's
//    sign and is at least 2^16 times its largest item's binade, the prefix in
//    the tile is summed as an integer too (units of 2^-49 of that binade 2^e,
//    rounded to 2^-38 of it: at most an eighth of the result's last place), set
//    as the low bits of a double D = 2^(e+14) + prefix, and the result is
//    (exclusive - 2^(e+14)) + D: the difference is exact, so one FP64 add and
//    one rounding per item.  Elsewhere (the first tiles, mixed signs) a chain
//    of FP64 adds gives the prefix in the tile and one more the result.
// 17 pairs per run: an odd stride of 16-byte accesses is free of bank
// conflicts with every run in order.  No barrier joins the warps of a role;
// each arrives on the stage's mbarrier by itself.
namespace pipe64 {

using ring::kEnd;
constexpr int kAggWarps = 4;
constexpr int kGroups = 2;                    // compute groups, alternate tiles
constexpr int kGroupWarps = kAggWarps;        // a run has the same lane in both roles
constexpr int kFirstAgg = 2;                  // after the producer and the prefix warp
constexpr int kFirstCompute = kFirstAgg + kAggWarps;
constexpr int kStoreWarp = kFirstCompute + kGroups * kGroupWarps;
constexpr int kThreads = 32 * (kStoreWarp + 1);
constexpr int kRuns = 32 * kAggWarps;         // 128 runs per tile
constexpr int kPairs = 17;
constexpr int kTile = kRuns * kPairs * 2;     // 4352 items
constexpr int kStages = 6;
static_assert(kAggWarps == 4, "warp totals are summed as four");
static_assert(kTile >= kScanTileMin, "the workspace has a descriptor per kScanTileMin items");

struct Smem {
  ring::Ring<double, double, kTile, kStages> r;
  double before[kStages][kRuns];           // total of the warp's runs before this one
  double warp_total[kStages][kAggWarps];
  unsigned int top[kStages][kRuns];        // sign and exponent of the run's largest item, or 0
  unsigned int arrived[kStages];           // aggregator warps done with the stage
  uint64_t ready[kStages];                 // compute -> store warp: the stage holds results
  unsigned long long ticket;               // the CTA's first
};
constexpr size_t kSmemBytes = sizeof(Smem) + 128;
static_assert(kSmemBytes <= 232448, "shared memory budget");

// v >> s for any s (0 from 64 on)
__device__ __forceinline__ uint64_t shr(uint64_t v, uint32_t s) {
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
  return r;
}

// The item's significand in units of 2^-UNIT of `top`'s binade; `top` is the
// sign and exponent field of an item of the same sign that is no smaller, at
// least 64, so that a zero's or subnormal's hidden bit is shifted out.
template <int UNIT>
__device__ __forceinline__ uint64_t fixed(uint64_t item, uint32_t top) {
  const uint64_t m = (item & f64emu::kFrac) | f64emu::kHidden;
  const uint32_t d = top - static_cast<uint32_t>(item >> 52);
  if constexpr (UNIT >= 52) return shr(m << (UNIT - 52), d);
  return shr(m, d + (52u - UNIT));
}

// v * 2^(unit - 1023), rounded to nearest even, on the integer pipes; `unit`
// carries the sign above its 11 bits, and the result is a normal number.
__device__ __forceinline__ double to_double(uint64_t v, uint32_t unit) {
  if (v == 0u) return 0.0;
  const uint32_t lz = static_cast<uint32_t>(__clzll(static_cast<long long>(v)));
  const uint64_t w = v << lz, m = w >> 11;
  const uint32_t up = ((static_cast<uint32_t>(w) & 0x7ffu) + 0x3ffu +
                       (static_cast<uint32_t>(m) & 1u)) >> 11;
  return f64emu::from_bits((static_cast<uint64_t>(unit + 62u - lz) << 52) + m + up);
}

// Prefix sums over a warp that stay off the FP64 pipe, where the aggregates'
// dependent adds would queue behind the compute warps': one non-negative
// integer per lane in units of 2^(top - 1023 - UNIT), all lanes' signs equal,
// is brought to the warp's largest `top` (`all`) and, where 32 of them could
// overflow, to a coarser unit.
struct WarpFixed {
  uint64_t v;
  uint32_t unit;
};
template <int UNIT>
__device__ __forceinline__ WarpFixed warp_align(uint64_t v, uint32_t top, uint32_t all) {
  v = shr(v, all - top);
  const uint32_t big = __reduce_max_sync(0xffffffffu, static_cast<uint32_t>(v >> 32));
  const int lz = __clz(static_cast<int>(big));
  const uint32_t s = lz < 5 ? 5u - lz : 0u;
  return {(v + ((1ull << s) >> 1)) >> s, all - UNIT + s};
}

__global__ void __launch_bounds__(kThreads, 1)
scan_pipelined_f64(const double* x, double* y, int64_t n, double init, unsigned int tiles,
                   ScanHeader* hdr, TileDesc* descs, uint64_t limit_ns, int zero) {
  extern __shared__ unsigned char s_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(
      (reinterpret_cast<uintptr_t>(s_raw) + 127) & ~static_cast<uintptr_t>(127));
  auto& r = sm.r;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  if (tid == 0) {
    ring::init(r, limit_ns);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&sm.ready[s], kGroupWarps);
      sm.arrived[s] = 0u;
    }
    mbar_init_fence();
  }
  const unsigned int z = begin_early();
  x += z;
  hdr += z;
  descs += z;
  if (tid == 0) ring::first_ticket(hdr, tiles, &sm.ticket);
  __syncthreads();
  // the CTA with the first ticket scans the aggregates of all the others (a
  // single tile needs no scanner)
  const unsigned int bias = tiles > 1u ? 1u : 0u;
  if (static_cast<unsigned int>(sm.ticket) < bias) {
    if (warp == 0) ring::scan_aggregates(descs, tiles, init, sm.ticket >> 32, hdr, limit_ns);
    return;
  }

  if (warp == 0) {
    ring::produce(r, x, n, tiles, hdr, kGroups, &sm.ticket, bias);
  } else if (warp < kFirstAgg) {
    ring::fetch_prefixes(r, descs, init, hdr);
  } else if (warp < kFirstCompute) {
    // ---- aggregators ----
    const int aw = warp - kFirstAgg, run = aw * 32 + lane;
    for (int k = 0;; ++k) {
      const int s = k % kStages;
      if (!ring::wait(r, &r.full[s], (k / kStages) & 1, hdr)) break;
      const unsigned int tile = r.ticket[s];
      if (tile == kEnd) break;
      const ulonglong2* tv = reinterpret_cast<const ulonglong2*>(r.tile[s]) + run * kPairs;
      ulonglong2 v[kPairs];
      uint32_t top = 0u, differ = 0u;  // largest high word; its sign bit: signs differ
#pragma unroll
      for (int q = 0; q < kPairs; ++q) v[q] = tv[q];
      const uint32_t first = static_cast<uint32_t>(v[0].x >> 32);
#pragma unroll
      for (int q = 0; q < kPairs; ++q) {
        const uint32_t a = static_cast<uint32_t>(v[q].x >> 32);
        const uint32_t b = static_cast<uint32_t>(v[q].y >> 32);
        top = max(top, max(a, b));
        differ |= (a ^ first) | (b ^ first);
      }
      top >>= 20;
      const uint32_t e = top & 0x7ffu;
      double before, inc;  // totals of the warp's runs before this one, and up to it
      const bool one_sign = (differ >> 31) == 0u && e - 64u < 2032u - 64u;
      uint64_t acc = 0;  // at most 34 * (2^57 - 1)
      if (one_sign) {
#pragma unroll
        for (int q = 0; q < kPairs; ++q) acc += fixed<56>(v[q].x, top) + fixed<56>(v[q].y, top);
      } else {
        top = 0u;
      }
      const uint32_t most = __reduce_max_sync(0xffffffffu, top);
      // runs of one size and sign: no run loses bits to a later one
      if (__all_sync(0xffffffffu, one_sign && most - top < 4u)) {
        const WarpFixed f = warp_align<56>(acc, top, most);
        const uint64_t up_to = warp_inclusive_scan(f.v);
        inc = to_double(up_to, f.unit);
        before = to_double(up_to - f.v, f.unit);
      } else {
        double total;
        if (one_sign) {
          total = to_double(acc, top - 56u);
        } else {
          total = 0.0;
#pragma unroll
          for (int q = 0; q < kPairs; ++q) {
            total += f64emu::from_bits(v[q].x);
            total += f64emu::from_bits(v[q].y);
          }
        }
        inc = warp_inclusive_scan(total);
        before = __shfl_up_sync(0xffffffffu, inc, 1);
        if (lane == 0) before = 0.0;
      }
      sm.before[s][run] = before;
      sm.top[s][run] = top;
      if (lane == 31) sm.warp_total[s][aw] = inc;
      __syncwarp();
      if (lane == 0) {
        __threadfence_block();
        if (atomicAdd(&sm.arrived[s], 1u) == kAggWarps - 1u) {  // the last of the four
          __threadfence_block();
          sm.arrived[s] = 0u;
          volatile double* wt = sm.warp_total[s];
          const double w0 = wt[0], w1 = wt[1], w2 = wt[2], w3 = wt[3], w01 = w0 + w1;
          desc_store(descs + tile, r.epoch * 4 + 1, to_bits<double>(w01 + (w2 + w3)));
          wt[0] = 0.0;  // now the totals of the warps before
          wt[1] = w0;
          wt[2] = w01;
          wt[3] = w01 + w2;
          mbar_arrive(&r.summed[s]);
        }
      }
      __syncwarp();
    }
  } else if (warp < kStoreWarp) {
    // ---- compute ----
    const int group = (warp - kFirstCompute) / kGroupWarps;
    const int cw = (warp - kFirstCompute) % kGroupWarps, run = cw * 32 + lane;
    const fform::Regs rg = fform::regs(zero);
    for (int k = group;; k += kGroups) {
      const int s = k % kStages;
      const uint32_t par = (k / kStages) & 1;
      if (!ring::wait(r, &r.drawn[s], par, hdr)) break;
      const unsigned int tile = r.ticket[s];
      if (tile == kEnd) break;
      if (!ring::wait(r, &r.full[s], par, hdr)) break;
      if (!ring::wait(r, &r.summed[s], par, hdr)) break;
      double2* tv = reinterpret_cast<double2*>(r.tile[s]) + run * kPairs;
      double2 v[kPairs];
#pragma unroll
      for (int q = 0; q < kPairs; ++q) v[q] = tv[q];
      double off = sm.before[s][run] + sm.warp_total[s][cw];  // the tile's total before this run
      // signs and exponents: of the run's largest item, of off
      const uint32_t top = sm.top[s][run], e = top & 0x7ffu;
      const uint64_t ob = f64emu::bits(off);
      const uint32_t oe = static_cast<uint32_t>(ob >> 52);
      const uint64_t head = static_cast<uint64_t>(top + 14u) << 52;  // 2^(e+14)
      auto chain = [&] {
        double o = off;
#pragma unroll
        for (int q = 0; q < kPairs; ++q) {
          const double a = v[q].x, b = v[q].y;
          v[q].x = o;
          o = fform::add(a, o, rg);
          v[q].y = o;
          o = fform::add(b, o, rg);
        }
      };
      // off is below 2^(e+13), the run's total below 2^(e+7)
      bool whole = top != 0u && (ob == 0u || oe - (top & 0x800u) < e + 13u);
      if (whole) {
        uint64_t acc = 1024u;
        if (ob != 0u)
          acc += shr(((ob & f64emu::kFrac) | f64emu::kHidden) << 10, e + 13u - (oe & 0x7ffu));
#pragma unroll
        for (int q = 0; q < kPairs; ++q) {
          const uint64_t a = f64emu::bits(v[q].x), b = f64emu::bits(v[q].y);
          v[q].x = f64emu::from_bits(head | (acc >> 11));
          acc += fixed<49>(a, top);
          v[q].y = f64emu::from_bits(head | (acc >> 11));
          acc += fixed<49>(b, top);
        }
      } else {
        chain();
      }
      if (!ring::wait(r, &r.prefix[s], par, hdr)) break;
      double rest = r.excl[s];
      const uint32_t xe = static_cast<uint32_t>(f64emu::bits(rest) >> 52);
      if (whole) {
        // up to xe = e + 66, 2^(e+14) is a multiple of the prefix's last place
        if (xe - (top + 16u) <= 50u && ((xe ^ top) & 0x800u) == 0u) {
          rest -= f64emu::from_bits(head);
        } else {
#pragma unroll
          for (int q = 0; q < kPairs; ++q) v[q] = tv[q];
          chain();
        }
      }
#pragma unroll
      for (int q = 0; q < kPairs; ++q) {
        v[q].x = fform::add(v[q].x, rest, rg);
        v[q].y = fform::add(v[q].y, rest, rg);
      }
#pragma unroll
      for (int q = 0; q < kPairs; ++q) tv[q] = v[q];
      fence_proxy_async_smem();
      __syncwarp();
      const int64_t first = static_cast<int64_t>(tile) * kTile;
      if (first + kTile > n) {  // the ragged last tile: plain stores of the warp's own items
        constexpr int kOwn = 32 * 2 * kPairs;
        for (int i = cw * kOwn + lane; i < (cw + 1) * kOwn; i += 32)
          if (first + i < n) y[first + i] = r.tile[s][i];
        __syncwarp();
      }
      if (lane == 0) mbar_arrive(&sm.ready[s]);
    }
  } else {
    // ---- store: one bulk store per finished tile, then the stage is free ----
    for (int k = 0;; ++k) {
      const int s = k % kStages;
      const uint32_t par = (k / kStages) & 1;
      if (!ring::wait(r, &r.drawn[s], par, hdr)) break;
      const unsigned int tile = r.ticket[s];
      if (tile == kEnd) break;
      if (!ring::wait(r, &sm.ready[s], par, hdr)) break;
      const int64_t first = static_cast<int64_t>(tile) * kTile;
      if (lane == 0) {
        if (first + kTile <= n) {
          bulk_store(y + first, r.tile[s], kTile * sizeof(double));
          bulk_commit();
          bulk_wait_read<0>();
        }
        mbar_arrive(&r.empty[s]);
      }
      __syncwarp();
    }
    if (lane == 0) bulk_wait_all();
  }

  __syncthreads();
  if (tid == 0) ring::drain(r);
}

}  // namespace pipe64

// The workspace is sized for the smallest tile, so it serves every tile size.
int64_t scan_tiles_max(int64_t n) { return ceil_div(n > 0 ? n : 1, kScanTileMin); }

template <typename T, int IT, bool VEC>
int launch_scan_it(const T* x, T* y, int64_t n, T init, char* w, uint64_t limit_ns,
                   cudaStream_t st) {
  constexpr int kTile = kScanBlock * IT;
  constexpr size_t kSmem = static_cast<size_t>(kTile + kTile / IT) * sizeof(T);
  const int rc = allow_dynamic_smem(reinterpret_cast<const void*>(scan_kernel<T, IT, VEC>),
                                    kSmem, "scan");
  if (rc != B200_OK) return rc;
  const int64_t tiles = ceil_div(n, kTile);
  ScanHeader* hdr = reinterpret_cast<ScanHeader*>(w);
  TileDesc* descs = reinterpret_cast<TileDesc*>(w + 256);
  scan_kernel<T, IT, VEC><<<static_cast<int>(tiles), kScanThreads, kSmem, st>>>(
      x, y, n, init, hdr, descs, limit_ns);
  return B200_OK;
}

int launch_scan_pipelined(const long long* x, long long* y, int64_t n, long long init, char* w,
                          uint64_t limit_ns, cudaStream_t st) {
  constexpr size_t kSmem = pipe::smem_bytes<long long>();
  const int rc = allow_dynamic_smem(
      reinterpret_cast<const void*>(pipe::scan_pipelined<long long>), kSmem, "scan");
  if (rc != B200_OK) return rc;
  const int64_t tiles = ceil_div(n, pipe::kTile);
  const int grid =
      static_cast<int>(std::min<int64_t>(tiles > 1 ? tiles + 1 : 1, device_info().sm_count));
  launch(pipe::scan_pipelined<long long>, grid, pipe::kThreads, kSmem, st, x, y, n, init,
         static_cast<unsigned int>(tiles), reinterpret_cast<ScanHeader*>(w),
         reinterpret_cast<TileDesc*>(w + 256), limit_ns);
  return B200_OK;
}

int launch_scan_pipelined(const double* x, double* y, int64_t n, double init, char* w,
                          uint64_t limit_ns, cudaStream_t st) {
  const int rc = allow_dynamic_smem(reinterpret_cast<const void*>(pipe64::scan_pipelined_f64),
                                    pipe64::kSmemBytes, "scan");
  if (rc != B200_OK) return rc;
  const int64_t tiles = ceil_div(n, pipe64::kTile);
  const int grid =
      static_cast<int>(std::min<int64_t>(tiles > 1 ? tiles + 1 : 1, device_info().sm_count));
  launch(pipe64::scan_pipelined_f64, grid, pipe64::kThreads, pipe64::kSmemBytes, st, x, y, n,
         init, static_cast<unsigned int>(tiles), reinterpret_cast<ScanHeader*>(w),
         reinterpret_cast<TileDesc*>(w + 256), limit_ns, 0);
  return B200_OK;
}

template <typename T>
int launch_scan(const char* name, const T* x, T* y, int64_t n, T init, void* ws,
                size_t ws_bytes, const b200_tune* tune, cudaStream_t st) {
  if (n < 0 || (n > 0 && (!x || !y))) return invalid("%s: bad args", name);
  if (n == 0) return B200_OK;
  const int64_t slots = scan_tiles_max(n);
  if (slots > 0x7fffffffLL) return invalid("%s: n too large", name);
  const int algo = tune ? tune->algo : 0;
  if (algo < 0 || algo > 2) return invalid("%s: algo %d (0, 1 or 2)", name, algo);
  if (tune && tune->block_size && tune->block_size != kScanBlock)
    return invalid("%s: block size %d (only %d)", name, tune->block_size, kScanBlock);
  // up to one tile of 4096 items per SM the tile kernel takes those (500001
  // items of FP64: 9.9 us against 12.4 with 8192)
  const bool one_wave = n <= static_cast<int64_t>(device_info().sm_count) * kScanTileMin;
  const int items = (tune && tune->items) ? tune->items
                                          : (one_wave ? kScanItemsMin : kScanItemsDefault);
  if (items != 16 && items != 32) return invalid("%s: items %d (16 or 32)", name, items);
  size_t need = 256 + static_cast<size_t>(slots) * sizeof(TileDesc);
  if (ws && !aligned16(ws)) return invalid("%s: workspace not 16-byte aligned", name);
  if (!ws || ws_bytes < need) {
    set_error("%s: workspace %zu bytes, need %zu", name, ws_bytes, need);
    return B200_ERR_WORKSPACE;
  }
  char* w = static_cast<char*>(ws);
  const bool vec = aligned16(x) && aligned16(y) && !(tune && tune->vec == 1);
  const uint64_t lim = wait_limit_ns(tune, kDefaultWaitNs);
  int rc;
  // FP64 takes the tile kernel for as long as it is one wave (65536 items: 8.4
  // us, the ring 11 us; 700001: 13.4 and 11.1 us; 2^26: 467 and 203 us)
  const bool ring =
      vec && (algo == 2 || (algo == 0 && (std::is_same<T, long long>::value || !one_wave)));
  if (ring)
    rc = launch_scan_pipelined(x, y, n, init, w, lim, st);
  else
    rc = (items == 16) ? (vec ? launch_scan_it<T, 16, true>(x, y, n, init, w, lim, st)
                              : launch_scan_it<T, 16, false>(x, y, n, init, w, lim, st))
                       : (vec ? launch_scan_it<T, 32, true>(x, y, n, init, w, lim, st)
                              : launch_scan_it<T, 32, false>(x, y, n, init, w, lim, st));
  if (rc != B200_OK) return rc;
  return after_launch(name);
}

// ---- REDUCE_SUM -------------------------------------------------------------
template <int BS, int IT>
__global__ void __launch_bounds__(BS)
reduce_sum_kernel(const double* x, int64_t n, double init, double* out, double* partials,
                  unsigned int* counter, int zero) {
  __shared__ double smem[BS / 32];
  __shared__ bool last_flag;
  const int64_t first = begin() + threadIdx.x;
  double s = 0.0;
  // s + v as a register-operand FMA (fform: bit-identical, full FP64 rate
  // where DADD gets 5/6 of it); `zero` is 0 at run time
  const double one = fform::regs(zero).one;
  for (int64_t t0 = static_cast<int64_t>(blockIdx.x) * (BS * IT); t0 < n;
       t0 += static_cast<int64_t>(gridDim.x) * (BS * IT)) {
    double v[IT];
#pragma unroll
    for (int u = 0; u < IT; ++u) {
      const int64_t i = t0 + u * BS + first;
      v[u] = (i < n) ? x[i] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < IT; ++u) s = fma(v[u], one, s);  // s + v[u]
  }
  s = block_sum<BS>(s, smem);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
  if (arrive_last(counter, &last_flag)) {
    double t = 0.0;
    for (int i = threadIdx.x; i < static_cast<int>(gridDim.x); i += BS)
      t += __ldcg(partials + i);
    t = block_sum<BS>(t, smem);
    if (threadIdx.x == 0) {
      *out = init + t;
      *counter = 0u;
    }
  }
}

}  // namespace

extern "C" {

size_t b200_scan_workspace_bytes(int64_t n) {
  return 256 + static_cast<size_t>(scan_tiles_max(n)) * sizeof(TileDesc);
}

int b200_algorithm_scan(const double* x, double* y, int64_t n, double init,
                        void* workspace, size_t workspace_bytes, const b200_tune* tune,
                        b200_stream_t stream) {
  return launch_scan<double>("b200_algorithm_scan", x, y, n, init, workspace,
                             workspace_bytes, tune, as_stream(stream));
}

int b200_algorithm_scan_i64(const int64_t* x, int64_t* y, int64_t n, int64_t init,
                            void* workspace, size_t workspace_bytes,
                            const b200_tune* tune, b200_stream_t stream) {
  return launch_scan<long long>("b200_algorithm_scan_i64",
                                reinterpret_cast<const long long*>(x),
                                reinterpret_cast<long long*>(y), n,
                                static_cast<long long>(init), workspace, workspace_bytes,
                                tune, as_stream(stream));
}

int b200_algorithm_reduce_sum(const double* x, int64_t n, double sum_init, double* sum,
                              void* workspace, size_t workspace_bytes,
                              const b200_tune* tune, b200_stream_t stream) {
  if (n < 0 || (n > 0 && !x) || !sum) return invalid("b200_algorithm_reduce_sum: bad args");
  int block = (tune && tune->block_size) ? tune->block_size : 256;
  int items = (tune && tune->items) ? tune->items : 8;
  if (!valid_block(block))
    return invalid("b200_algorithm_reduce_sum: bad block size %d", block);
  int grid = reduce_grid(n, tune, block, items);
  size_t need = reduce_ws_bytes_for_grid(grid);
  if (!workspace || workspace_bytes < need) {
    set_error("b200_algorithm_reduce_sum: workspace %zu bytes, need %zu", workspace_bytes,
              need);
    return B200_ERR_WORKSPACE;
  }
  unsigned int* counter = static_cast<unsigned int*>(workspace);
  double* partials = reinterpret_cast<double*>(static_cast<char*>(workspace) + 256);
  cudaStream_t st = as_stream(stream);
  B200_DISPATCH_BLOCK(block, BS, B200_DISPATCH_ITEMS(items, IT,
    launch(reduce_sum_kernel<BS, IT>, grid, BS, 0, st, x, n, sum_init, sum, partials, counter,
           0)));
  return after_launch("b200_algorithm_reduce_sum");
}

}  // extern "C"
