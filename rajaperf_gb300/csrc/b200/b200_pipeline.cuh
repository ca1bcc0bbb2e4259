// The stage ring of SCAN's persistent single-pass kernels: one CTA per SM
// streams tiles of a 1-D array (4096 items by default) through its
// shared-memory stages (seven by default), and one more CTA scans the tiles'
// aggregates.  This header holds the ring's layout and bounded waits, the
// producer warp (draws tile ids, issues one bulk copy per tile), the scanner
// and the prefix warp (takes a tile's exclusive prefix from the scanner); the
// kernel adds the aggregators (publish a tile's aggregate as soon as it
// lands), its compute warps, and the role that frees a stage.  INDEXLIST's
// persistent kernel (indexlist.cu) keeps its own slots and producer.
//
// Per stage s, mbarriers link the roles (one arrival each):
//   drawn[s]  producer -> prefix        the stage's tile id is set
//   full[s]   producer (TMA) -> all     the tile's items have landed
//   summed[s] aggregator -> compute     the tile's aggregate is published
//   prefix[s] prefix -> compute         its exclusive prefix is in excl[s]
//   empty[s]  kernel -> producer        the stage may be refilled
// A tile id is drawn only once its stage is free: an id held while waiting
// would delay that tile's aggregate and the prefixes of its successors.
// A parity wait for phase p of a barrier passes at once while phase p-1 is
// still open, so a warp that takes alternate tiles (k, k + W, ...) must know
// that stage s's previous tile is done before waiting on s: drawn[s] gives
// that (the producer draws in order and refills a stage only after its
// tile is done), so such a warp waits on drawn[s] before any other barrier
// of stage s.  full[s] alone does not: bulk copies can complete out of order.
// After the last tile the producer places one end marker (tile id kEnd) per
// group of the role with the most groups taking alternate tiles.  Every wait
// is bounded (Ring::limit_ns); one that gives up sets the workspace error word
// and stops every role of the CTA.
#pragma once

#include <cstdint>

#include <type_traits>

#include "b200_async.cuh"
#include "b200_f64emu.cuh"
#include "b200_lookback.cuh"

namespace b200 {
namespace ring {

constexpr int kTile = 4096;                  // items per tile, unless a kernel says otherwise
constexpr int kStages = 7;
constexpr unsigned int kEnd = 0xffffffffu;   // end marker in ticket[]

template <typename In, typename Acc, int TILE = kTile, int STAGES = kStages>
struct Ring {
  using InT = In;
  using AccT = Acc;
  static constexpr int kTile = TILE;
  static constexpr int kStages = STAGES;
  In tile[kStages][kTile];
  Acc excl[kStages];
  unsigned int ticket[kStages];
  unsigned int phases[kStages];  // full-barrier phases started per stage
  uint64_t drawn[kStages];
  uint64_t full[kStages];
  uint64_t summed[kStages];
  uint64_t prefix[kStages];
  uint64_t empty[kStages];
  unsigned long long epoch;
  uint64_t limit_ns;  // limit of every bounded wait of the launch
  int abort;
};

// Thread 0, before the CTA's first barrier.
template <class R>
__device__ __forceinline__ void init(R& r, uint64_t limit_ns) {
  for (int s = 0; s < R::kStages; ++s) {
    mbar_init(&r.drawn[s], 1);
    mbar_init(&r.full[s], 1);
    mbar_init(&r.summed[s], 1);
    mbar_init(&r.prefix[s], 1);
    mbar_init(&r.empty[s], 1);
    r.phases[s] = 0u;
  }
  r.limit_ns = limit_ns;
  r.abort = 0;
}

// Bounded wait by a whole warp; the result is the same in every lane (a lane
// that gave up fails the warp).  On expiry records the error and stops every
// role of the CTA.  R: a Ring, or any struct with its limit_ns and abort.
template <class R>
__device__ __forceinline__ bool wait(R& r, uint64_t* bar, uint32_t parity, ScanHeader* hdr) {
  const bool ok = __all_sync(0xffffffffu, mbar_wait_for(bar, parity, r.limit_ns));
  if (!ok && (threadIdx.x & 31) == 0) {
    atomicExch(&hdr->error, 1u);
    *reinterpret_cast<volatile int*>(&r.abort) = 1;
  }
  return ok;
}

// A whole warp fills a tile's stage with its `left` < TILE items and zeros
// behind: a bulk copy of the whole 16-byte units, a plain load of what is left
// (a loop of plain loads over the tile took the single warp some 17 us).
template <typename In, int TILE>
__device__ __forceinline__ void load_ragged(In* stage, const In* src, int left, uint64_t* full) {
  constexpr int kUnit = 16 / static_cast<int>(sizeof(In));
  static_assert(TILE % kUnit == 0, "a tile is whole 16-byte units");
  const int lane = threadIdx.x & 31, bulk = left / kUnit * kUnit;
  if (lane < kUnit && bulk < left)
    stage[bulk + lane] = bulk + lane < left ? src[bulk + lane] : In(0);
  uint4* rest = reinterpret_cast<uint4*>(stage) + (left + kUnit - 1) / kUnit;
  const int units = (TILE - left) / kUnit;
#pragma unroll 4
  for (int i = lane; i < units; i += 32) rest[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncwarp();
  if (lane == 0) {
    if (bulk > 0) {
      mbar_arrive_expect_tx(full, bulk * static_cast<uint32_t>(sizeof(In)));
      bulk_load(stage, src, bulk * static_cast<uint32_t>(sizeof(In)), full);
    } else {
      mbar_arrive(full);
    }
  }
}

// Warp 0: for k = 0, 1, ... waits for stage k mod kStages to be free, draws
// the next tile id and fills the stage with one bulk copy (the ragged last
// tile zero-filled), then places `end_markers` end markers
// (at least the number of warps of any role that takes alternate tiles, and
// fewer than kStages).  The CTA
// that draws the launch's last ticket (tiles + gridDim.x draws: every CTA
// draws exactly one id past the end) resets the count and advances the epoch.
// `first`: the CTA's first ticket, already drawn; a ticket's tile id is the
// ticket less `bias`.
template <class R>
__device__ void produce(R& r, const typename R::InT* x, int64_t n, unsigned int tiles,
                        ScanHeader* hdr, int end_markers,
                        const unsigned long long* first, unsigned int bias) {
  using In = typename R::InT;
  constexpr int kTile = R::kTile, kStages = R::kStages;
  const int lane = threadIdx.x & 31;
  const unsigned long long draws = static_cast<unsigned long long>(tiles) + gridDim.x;
  volatile int* abort_flag = &r.abort;
  int ends = 0;
  for (int k = 0; ends < end_markers && !__any_sync(0xffffffffu, *abort_flag); ++k) {
    const int s = k % kStages;
    if (k >= kStages && !wait(r, &r.empty[s], ((k / kStages) - 1) & 1, hdr)) break;
    unsigned int tile = kEnd;
    if (ends == 0) {
      unsigned long long t = 0;
      if (k == 0) {
        t = *first;
      } else if (lane == 0) {
        t = atomicAdd(&hdr->ticket, 1ull);
        if (static_cast<unsigned int>(t) == draws - 1)
          atomicAdd(&hdr->ticket, (1ull << 32) - draws);
      }
      t = __shfl_sync(0xffffffffu, t, 0);
      if (k == 0 && lane == 0) r.epoch = t >> 32;
      const unsigned int id = static_cast<unsigned int>(t) - bias;
      if (id < tiles) tile = id;
    }
    if (lane == 0) {
      r.ticket[s] = tile;
      mbar_arrive(&r.drawn[s]);
    }
    if (tile == kEnd) {  // end markers in consecutive stages, one per warp of a role
      ++ends;
      __syncwarp();
      if (lane == 0) {
        ++r.phases[s];
        mbar_arrive(&r.full[s]);
      }
      continue;
    }
    const int64_t base = static_cast<int64_t>(tile) * kTile;
    if (base + kTile <= n) {
      if (lane == 0) {
        ++r.phases[s];
        mbar_arrive_expect_tx(&r.full[s], kTile * sizeof(In));
        bulk_load(r.tile[s], x + base, kTile * sizeof(In), &r.full[s]);
      }
    } else {
      if (lane == 0) ++r.phases[s];
      load_ragged<In, kTile>(r.tile[s], x + base, static_cast<int>(n - base), &r.full[s]);
    }
  }
}

// The scanner: one warp, in a CTA that takes no tiles, turns the tiles'
// aggregates, as they are published, into exclusive prefixes, in tile order.
// Each tile's prefix warp then polls one descriptor, where a lookback re-reads
// hundreds: at 2^26 items lookback warps in every CTA left the kernel at
// 238-275 us (2 to 5 warps, 128 to 256 predecessors a round), the scanner at
// 203 us (2, 4, 8 tiles per lane: 267, 203, 227 us; no prefixes at all: 173
// us; the copy alone: 157 us).  int64, 2^26 items: 189 and 160 us.  A round takes the published tiles
// from p on, up to kPerLane per lane.  The running FP64 prefix is kept in two parts
// (Dekker's two-sum, larger operand first, compared as integers), so that its
// roundings do not add up over the rounds.
constexpr int kPerLane = 4;

template <typename T>
__device__ void scan_aggregates(TileDesc* descs, unsigned int tiles, T init,
                                unsigned long long epoch, ScanHeader* hdr, uint64_t limit_ns) {
  const int lane = threadIdx.x & 31;
  const unsigned long long AGG = epoch * 4 + 1, INC = epoch * 4 + 2;
  T hi = init, lo = T(0);
  uint64_t t0 = 0;  // time of the first empty round since the last full one
  for (unsigned int p = 0; p < tiles;) {
    T v[kPerLane];
    unsigned int have = 0;  // the lane's published tiles before its first other one
    {
      unsigned long long f[kPerLane], bits[kPerLane];
      const unsigned int t = p + lane * kPerLane;
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) {
        f[j] = bits[j] = 0ull;
        if (t + j < tiles) desc_load(descs + t + j, f[j], bits[j]);
      }
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) {
        if (have == j && f[j] == AGG) ++have;
        v[j] = have > j ? from_bits<T>(bits[j]) : T(0);
      }
    }
    const unsigned int part = __ballot_sync(0xffffffffu, have < kPerLane);
    const int last = part ? __ffs(part) - 1 : 31;  // the last lane that counts
    if (lane > last) have = 0;
    const unsigned int found = last * kPerLane + __shfl_sync(0xffffffffu, have, last);
    if (found == 0) {
      uint64_t now = 0;
      if (lane == 0) now = globaltimer();
      now = __shfl_sync(0xffffffffu, now, 0);
      if (t0 == 0) t0 = now;
      if (now - t0 > limit_ns) {
        if (lane == 0) atomicExch(&hdr->error, 1u);
        return;
      }
      continue;
    }
    t0 = 0;
    if (lane > last) {
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) v[j] = T(0);
    }
    T before[kPerLane];
    T sum = T(0);
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
      before[j] = sum;
      sum += v[j];
    }
    const T inc = warp_inclusive_scan(sum);
    T left = __shfl_up_sync(0xffffffffu, inc, 1);
    left = lane == 0 ? lo : left + lo;
#pragma unroll
    for (int j = 0; j < kPerLane; ++j)
      if (j < have)
        desc_store(descs + p + lane * kPerLane + j, INC, to_bits<T>(hi + (left + before[j])));
    const T all = __shfl_sync(0xffffffffu, inc, 31);
    if constexpr (std::is_same<T, double>::value) {
      const bool first = (f64emu::bits_opaque(hi) << 1) >= (f64emu::bits_opaque(all) << 1);
      const double a = first ? hi : all, b = first ? all : hi;
      hi = a + b;
      const double err = b - (hi - a);
      lo += fabs(err) < INFINITY ? err : 0.0;
    } else {
      hi += all;
    }
    p += found;
  }
}

// The prefix warp: takes each tile's exclusive prefix from the scanner.
template <class R>
__device__ void fetch_prefixes(R& r, const TileDesc* descs, typename R::AccT init,
                               ScanHeader* hdr) {
  using T = typename R::AccT;
  const int lane = threadIdx.x & 31;
  for (int k = 0;; ++k) {
    const int s = k % R::kStages;
    if (!wait(r, &r.drawn[s], (k / R::kStages) & 1, hdr)) return;
    const unsigned int tile = r.ticket[s];
    if (tile == kEnd) return;
    if (lane == 0) {
      const unsigned long long INC = r.epoch * 4 + 2;
      T excl = init;
      bool ok = true;
      if (tile > 0) {
        unsigned long long f, bits;
        desc_load(descs + tile, f, bits);
        if (f != INC) {
          const uint64_t t0 = globaltimer();
          while (ok && f != INC) {
            desc_load(descs + tile, f, bits);
            ok = globaltimer() - t0 <= r.limit_ns;
          }
        }
        excl = from_bits<T>(bits);
      }
      if (ok) {
        r.excl[s] = excl;
        mbar_arrive(&r.prefix[s]);
      } else {
        atomicExch(&hdr->error, 1u);
        *reinterpret_cast<volatile int*>(&r.abort) = 1;
      }
    }
    __syncwarp();
    if (*reinterpret_cast<volatile int*>(&r.abort)) return;
  }
}

// Thread 0 draws the CTA's first ticket, a run of `run` tiles: the launch makes
// floor(tiles / run) + gridDim.x draws, one of them the scanner's.
__device__ __forceinline__ void first_ticket(ScanHeader* hdr, unsigned int tiles,
                                             unsigned long long* ticket, unsigned int run = 1u) {
  const unsigned long long draws = static_cast<unsigned long long>(tiles / run) + gridDim.x;
  const unsigned long long t = atomicAdd(&hdr->ticket, static_cast<unsigned long long>(run));
  if (static_cast<unsigned int>(t) == run * (draws - 1))
    atomicAdd(&hdr->ticket, (1ull << 32) - run * draws);
  *ticket = t;
}

// Thread 0 after the CTA's final barrier: after an abort, bulk copies may
// still be landing; wait (bounded) for the last phase started in each stage.
template <class R>
__device__ __forceinline__ void drain(R& r) {
  if (!r.abort) return;
  for (int s = 0; s < R::kStages; ++s)
    if (r.phases[s] > 0u) mbar_wait_for(&r.full[s], (r.phases[s] - 1u) & 1u, r.limit_ns);
}

}  // namespace ring
}  // namespace b200
