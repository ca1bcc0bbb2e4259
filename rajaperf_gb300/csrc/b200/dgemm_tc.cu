// C = A * B in FP64 on the FP8 tensor cores, every element as accurate as one
// rounding of the exact product.
//
// GB300's FP64 pipe gives 1.25 TFLOP/s; its e4m3 tensor cores give 4.5 PFLOP/s
// and, on integers, exact sums.  A value x of a row of A (column of B) whose
// largest magnitude lies in binade e is rounded to an integer in units of
// 2^(e+1-74), and that is cut into 15 balanced base-32 digits -15 .. 16, each
// with x's sign.  The e4m3 code of a digit is its magnitude (codes 0 .. 16 are the
// linear range 0 .. 16 of 2^-9) and a sign bit, so cutting takes shifts, masks
// and byte permutes only.  For every weight w = s + t = 2 .. 17 the digit products
// A_s * B_t sum to an integer that FP32 holds exactly (at most 15 * 256 * k <
// 2^24), and the 16 sums combine into one integer and one rounding.
//
// Error: the weights from 18 on leave out at most 108 k units of the combined
// integer (kDropped), a value that lies more than 21 binades below its row's
// largest and so lost bits at most 256 (kPerCut).  An element at least 2^55
// times what may be missing from it is stored: it errs by its one rounding and
// at most a quarter of 2^-53 of itself, whatever the values, where a chain of
// FP64 FMAs rounds k times.  The others (one in 30000 for k = 1000 uniform values
// of either sign) are computed again as FP64 dot products, one by one; a tile with
// many of them (max_redo), or with a row or column that the cut does not take
// (infinities, NaNs, magnitudes outside 2^-400 .. 2^400), is computed whole on
// the FP64 pipe.  Where most elements are like that (a diagonal matrix, say, whose
// products are mostly zeros), four of them, computed first, tell, and the tile
// skips the digits (1000^3 each, a diagonal matrix: 6600 us against 7150 without
// them, and 6120 on the FP64 pipe alone; they take 1.3 % of other calls).
// (16 unsigned base-16 digits, cut off below, took 508 us where this takes 705,
// 1000^3 each, but what they left out, of one sign and 2^-60 of the largest
// products, cost up to 9 bits where one large value of a row met a small one.)
//
// A CTA owns a 128 x 32 tile of C: with 16 weights its sums fill tensor memory
// (16 x 32 FP32 columns), so nothing is folded before the end, and the digits
// of B stand one slice under the other, so that one MMA multiplies A_s by all
// the slices it meets: columns 32 (s - 1) .. of the sums.  Eight warps cut the
// operands of a k step of 32 into shared memory (128-byte swizzle, two stages)
// while one thread issues the MMAs of the other stage.
//
// Measured, E = A B, F = C D, G = E F (us, against the FP64 pipe's kernel):
// 1000 x 1100 x 1010 x 1200 x 1000  787 / 7360; 1000^3 each, uniform, normal,
// Student-t (3) and log-normal values 705 - 766 / 6120, 500^3 145 / 1560, 250^3 86 /
// 790, 100^3 50 / 320, 32^3 27 / 113.  The cutting is the bound (some
// 46 integer instructions a value), the MMAs alone take 38 us of a tile of
// k = 1000, at 4.5 PFLOP/s.  Extracting the fields by spreading 20 bits over
// four bytes of each value was 14 % slower than two fields of four values at a
// time, by byte permutes.
#include "b200_dgemm.cuh"
#include "b200_f64emu.cuh"
#include "b200_launch.cuh"
#include "b200_tcgen05.cuh"

using namespace b200;

namespace {

using namespace tcgen05;

constexpr int TM = 128, TN = 32, KS = 32;     // tile of C, k per step
constexpr int kDigits = 15, kWeights = 16;
constexpr int kCutters = 8;                   // warps that cut and, at the end, combine
constexpr int kThreads = 32 * (1 + kCutters);
constexpr int kStages = 2;
constexpr int kQuads = TM / 4 / kCutters;  // quads of A per thread and step
constexpr uint32_t kATile = TM * 128;                      // four digits: 128 rows x 128 bytes
constexpr uint32_t kAStage = kATile * ((kDigits + 3) / 4);   // 64 KB
constexpr uint32_t kBBytes = kDigits * TN * 128;           // 60 KB: the stages side by side
constexpr uint32_t kTmemCols = 512;
constexpr int64_t kMaxK = 4096;
constexpr int kProbes = 4;
constexpr int kProbesBad = 3;                 // probes that fail before a tile skips the digits
// Bounds of what a sum leaves out, in its last unit (see above).
constexpr int kDropped = 108;                 // per k: 256 (13/32 + 12/32^2 + 11/32^3 + ..)
constexpr int kPerCut = 1 << 8;               // per value that lost bits
constexpr uint64_t kWaitNs = 1000000000ull;

struct Smem {
  uint64_t full[kStages], empty[kStages], done;
  uint32_t tmem;
  int abort, bad, redo;
  int ea[TM], eb[TN];        // biased exponents of the rows' and columns' largest values; 0: all zero
  int cut_a[TM], cut_b[TN];  // how many of their values lost bits
  double probe[kProbes];     // some of the tile's elements as FP64 dot products
  uint16_t list[TM * TN];
};
constexpr uint32_t kOperands = kStages * kAStage + kBBytes;
constexpr size_t kSmemBytes = 1024 + kOperands + sizeof(Smem);
static_assert(kSmemBytes <= 232448, "shared memory budget");
static_assert(kDigits * 256 * kMaxK < (1 << 24), "sums are exact in FP32");
static_assert(kWeights * TN <= kTmemCols, "the sums fit in tensor memory");

struct Products {
  Product p[2];
  int tiles0;  // tiles of p[0]
};

// Elements redone one by one; more: the whole tile.  Where the two cost the same
// (us per tile beyond the digits' pass, an element and the tile): k = 32 0.11 and
// 47, 100 0.12 and 100, 250 0.22 and 260, 1000 1.0 and 1080, 4000 5 and 4270.
__device__ __forceinline__ int max_redo(int64_t k) { return k < 100 ? 512 : 896; }

// The row and column of probe p, one in every quarter of the tile's.
__device__ __forceinline__ int probe_row(int p) { return p * (TM / kProbes + 1); }
__device__ __forceinline__ int probe_col(int p) { return p * (TN / kProbes); }

// The key of x's magnitude: above zero for any non-zero x, ordered by binade.
__device__ __forceinline__ uint32_t key(double x) {
  const uint64_t b = f64emu::bits_opaque(x);
  return (static_cast<uint32_t>(b >> 32) & 0x7fffffffu) | (static_cast<uint32_t>(b) ? 1u : 0u);
}

// A row's exponent from its largest key; sets `bad` for one that is not cut.
__device__ __forceinline__ int exponent(uint32_t key, int* bad) {
  const int e = static_cast<int>(key >> 20);
  if (key != 0u && (e < 1023 - 400 || e > 1023 + 400)) *bad = 1;
  return key == 0u ? 0 : e;
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t s) {
  return __byte_perm(a, b, s);
}

// 15 in every 5-bit field of 75 bits (32-bit words, the lowest first): added to
// an integer, it makes the fields the balanced digits -15 .. 16 plus 15.
constexpr uint32_t kFifteens0 = 0xdef7bdefu, kFifteens1 = 0xf7bdef7bu, kFifteens2 = 0x3deu;

// Two values' bits `at` .. `at` + 9 of a word, side by side in 16 bits each.
__device__ __forceinline__ uint32_t pair(uint32_t a, uint32_t b, int at) {
  const uint32_t y = at / 8;
  return prmt(a, b, y * 0x1111u + 0x5410u) >> (at % 8);
}

// The e4m3 codes of four digits from their fields (digit + 15 in the low bits
// of each byte): a digit of magnitude m up to 16 has the code m, with the sign
// in bit 7.  `flip` holds 0x80 in the bytes of the non-negative values.
__device__ __forceinline__ uint32_t codes(uint32_t fields, uint32_t flip) {
  const uint32_t p = (fields >> 4) & 0x01010101u;  // digit > 0
  const uint32_t m = ((fields & 0x0f0f0f0fu) ^ 0x0f0f0f0fu) ^ (p * 15u);
  return (p * 0x81u + m) ^ flip;
}

// A value more than 21 binades below its row's (column's) largest, `below` of
// them further: its significand in the unit, rounded to nearest.
__device__ __forceinline__ uint64_t far_below(uint64_t bits, uint32_t below, int* lost) {
  const uint64_t m = (bits & f64emu::kFrac) | f64emu::kHidden;
  if ((bits << 1) == 0u) return 0u;
  uint64_t v = 0;
  if ((bits << 1 >> 53) != 0u && below <= 54u) v = (m + (1ull << (below - 1u))) >> below;
  if (v == 0u || v << below != m) atomicAdd(lost, 1);
  return v;
}

// Digits 1 .. 15 (most significant first) of a quad, four values of a row or
// column: out[d] holds digit d + 1 of all four, as e4m3 codes.  `lost` counts
// the values that lost bits.
__device__ __forceinline__ void cut4(const double (&x)[4], int e, int* lost,
                                     uint32_t (&out)[kDigits]) {
  uint32_t hi[4], mh[4], ml[4];
  int up[4];  // the significand's shift to the unit 2^(e + 1 - 74)
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    const uint64_t b = f64emu::bits_opaque(x[m]);
    hi[m] = static_cast<uint32_t>(b >> 32);
    ml[m] = static_cast<uint32_t>(b);
    mh[m] = (hi[m] & 0xfffffu) | 0x100000u;
    up[m] = static_cast<int>((hi[m] >> 20) & 0x7ffu) - (e - 21);
  }
  if (min(min(up[0], up[1]), min(up[2], up[3])) < 0) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      if (up[m] < 0) {
        const uint64_t v = far_below(f64emu::bits_opaque(x[m]), static_cast<uint32_t>(-up[m]), lost);
        mh[m] = static_cast<uint32_t>(v >> 32);
        ml[m] = static_cast<uint32_t>(v);
        up[m] = 0;
      }
    }
  }
  uint32_t t[5][4];  // 75 bits in three words; bits 30 .. 61 and 60 .. 91
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    t[0][m] = __funnelshift_l(0u, ml[m], up[m]);
    t[1][m] = __funnelshift_l(ml[m], mh[m], up[m]);
    t[2][m] = __funnelshift_l(mh[m], 0u, up[m]);
    asm("add.cc.u32 %0, %0, %3;\n\t"
        "addc.cc.u32 %1, %1, %4;\n\t"
        "addc.u32 %2, %2, %5;"
        : "+r"(t[0][m]), "+r"(t[1][m]), "+r"(t[2][m])
        : "n"(kFifteens0), "n"(kFifteens1), "n"(kFifteens2));
    t[3][m] = __funnelshift_r(t[0][m], t[1][m], 30);
    t[4][m] = __funnelshift_r(t[1][m], t[2][m], 28);
  }
  // the bytes of a word of codes: values 0, 2, 1, 3 of the quad
  const uint32_t signs = prmt(prmt(hi[0], hi[2], 0x0073), prmt(hi[1], hi[3], 0x0073), 0x5410);
  const uint32_t flip = ~signs & 0x80808080u;
  // two fields at a time: word and bit where they start
  constexpr int kWord[8] = {0, 0, 0, 3, 1, 1, 4, 2}, kBit[8] = {0, 10, 20, 0, 8, 18, 0, 6};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t* v = t[kWord[j]];
    const uint32_t a = pair(v[0], v[1], kBit[j]), b = pair(v[2], v[3], kBit[j]);
    out[kDigits - 1 - 2 * j] = codes((a & 0x00ff00ffu) | ((b << 8) & 0xff00ff00u), flip);
    if (j < 7)
      out[kDigits - 2 - 2 * j] = codes(((a >> 5) & 0x00ff00ffu) | ((b << 3) & 0xff00ff00u), flip);
  }
}

__device__ __forceinline__ void st32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t n) {
  // FP32 sums, e4m3 operands, both K-major; n >> 3 at bit 17, m >> 4 at bit 24
  const uint32_t idesc = (1u << 4) | ((n >> 3) << 17) | (static_cast<uint32_t>(TM >> 4) << 24);
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.eq.u32 p, 0, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc)
      : "memory");
}

// The tile on the FP64 pipe: 256 threads of 4 x 4 elements, k in order.
__device__ void fp64_tile(const Product& g, int64_t i0, int64_t j0, unsigned char* smem) {
  constexpr int GK = 16;
  double (*As)[TM + 1] = reinterpret_cast<double (*)[TM + 1]>(smem);
  double (*Bs)[TN] = reinterpret_cast<double (*)[TN]>(smem + sizeof(double) * GK * (TM + 1));
  const int t = threadIdx.x, tx = t % 8, ty = t / 8;
  double acc[4][4] = {};
  for (int64_t k0 = 0; k0 < g.k; k0 += GK) {
    __syncthreads();
    if (t < 256) {
#pragma unroll
      for (int u = 0; u < TM * GK / 256; ++u) {
        const int id = u * 256 + t, kk = id % GK, i = id / GK;
        As[kk][i] = (i0 + i < g.m && k0 + kk < g.k) ? g.A[(i0 + i) * g.k + k0 + kk] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < TN * GK / 256; ++u) {
        const int id = u * 256 + t, j = id % TN, kk = id / TN;
        Bs[kk][j] = (j0 + j < g.n && k0 + kk < g.k) ? g.B[(k0 + kk) * g.n + j0 + j] : 0.0;
      }
    }
    __syncthreads();
    if (t < 256) {
      const int kn = static_cast<int>(g.k - k0 < GK ? g.k - k0 : GK);
      for (int kk = 0; kk < kn; ++kk)
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c)
            acc[r][c] = fma(As[kk][ty + 32 * r], Bs[kk][tx + 8 * c], acc[r][c]);
    }
  }
  if (t < 256)
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int64_t i = i0 + ty + 32 * r, j = j0 + tx + 8 * c;
        if (i < g.m && j < g.n) g.C[i * g.n + j] = acc[r][c];
      }
}

__global__ void __launch_bounds__(kThreads, 1) dgemm_tc_kernel(const Products ps) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  Smem& sm = *reinterpret_cast<Smem*>(base + kOperands);
  const uint32_t a_smem = smem_u32(base), b_smem = a_smem + kStages * kAStage;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&sm.full[s], kCutters);
      mbar_init(&sm.empty[s], 1);
    }
    mbar_init(&sm.done, 1);
    sm.abort = sm.bad = sm.redo = 0;
    for (int i = 0; i < TN; ++i) sm.cut_b[i] = 0;
    mbar_init_fence();
  }
  if (tid < TM) sm.cut_a[tid] = 0;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&sm.tmem)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  int tile = static_cast<int>(begin_early()) + static_cast<int>(blockIdx.x);
  const bool second = tile >= ps.tiles0;
  Product g = second ? ps.p[1] : ps.p[0];
  if (second) tile -= ps.tiles0;
  const int nt = static_cast<int>((g.n + TN - 1) / TN);
  const int64_t i0 = static_cast<int64_t>(tile / nt) * TM, j0 = static_cast<int64_t>(tile % nt) * TN;
  const int steps = static_cast<int>((g.k + KS - 1) / KS);
  volatile int* abort_flag = &sm.abort;

  // ---- the rows' and columns' exponents ----
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp > 0) {
    const int cw = warp - 1;
    // 32 loads in flight per thread: the pass is bound by their latency
    constexpr int R = TM / kCutters, U = 32 / R;
    uint32_t most[R];
    const double* rows[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      most[r] = 0u;
      const int64_t i = i0 + r * kCutters + cw;
      rows[r] = g.A + (i < g.m ? i : g.m - 1) * g.k;
    }
    for (int64_t k = lane; k < g.k; k += 32 * U) {
      double x[U][R];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int64_t ku = k + 32 * u;
          x[u][r] = ku < g.k ? rows[r][ku] : 0.0;
        }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int r = 0; r < R; ++r) most[r] = max(most[r], key(x[u][r]));
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t all = __reduce_max_sync(0xffffffffu, most[r]);
      if (lane == 0) sm.ea[r * kCutters + cw] = exponent(all, &sm.bad);
    }
    // columns: a lane's column, every kCutters-th k; the warps meet in cols[]
    uint32_t col = 0u;
    for (int64_t k = cw; k < g.k; k += 32 * kCutters) {
      double x[32];
#pragma unroll
      for (int u = 0; u < 32; ++u) {
        const int64_t ku = k + u * kCutters;
        x[u] = (j0 + lane < g.n && ku < g.k) ? g.B[ku * g.n + j0 + lane] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 32; ++u) col = max(col, key(x[u]));
    }
    uint32_t* cols = reinterpret_cast<uint32_t*>(base);  // [kCutters][TN], before the operands
    cols[cw * TN + lane] = col;
  } else {
    // the probes: kLanes lanes each, 32 loads in flight per lane
    constexpr int kLanes = 32 / kProbes;
    const int p = lane / kLanes;
    const int64_t i = i0 + probe_row(p), j = j0 + probe_col(p);
    const double* a = g.A + (i < g.m ? i : g.m - 1) * g.k;
    const double* b = g.B + (j < g.n ? j : g.n - 1);
    double dot = 0.0;
    for (int64_t k = lane % kLanes; k < g.k; k += kLanes * 16) {
      double x[16], y[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int64_t ku = k + kLanes * u;
        x[u] = ku < g.k ? a[ku] : 0.0;
        y[u] = ku < g.k ? b[ku * g.n] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 16; ++u) dot = fma(x[u], y[u], dot);
    }
#pragma unroll
    for (int off = kLanes / 2; off > 0; off >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, off);
    if (lane % kLanes == 0) sm.probe[p] = dot;
  }
  // the sums start at zero
  if (warp >= 1 && warp <= 4) {  // one warp per quadrant of tensor memory's lanes
    const uint32_t zero[16] = {};
    const uint32_t at = sm.tmem + (static_cast<uint32_t>(32 * (warp & 3)) << 16);
    for (uint32_t c = 0; c < kTmemCols; c += 16) tmem_st16(at + c, zero);
    tmem_st_wait();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (tid < TN) {
    const uint32_t* cols = reinterpret_cast<const uint32_t*>(base);
    uint32_t all = 0u;
    for (int w = 0; w < kCutters; ++w) all = max(all, cols[w * TN + tid]);
    sm.eb[tid] = exponent(all, &sm.bad);
    __syncwarp();
    // how many of the probes would be computed again
    bool again = false;
    if (tid < kProbes) {
      const int e = sm.ea[probe_row(tid)], f = sm.eb[probe_col(tid)];
      const double least = f64emu::from_bits(
          static_cast<uint64_t>(e + f - 1023 + 4 - 85 + 55) << 52) * (kDropped * static_cast<double>(g.k));
      again = e != 0 && f != 0 && fabs(sm.probe[tid]) < least;
    }
    const int count = __popc(__ballot_sync(0xffffffffu, again));
    if (tid == 0 && count >= kProbesBad) sm.bad = 1;
  }
  __syncthreads();
  const uint32_t tmem = sm.tmem;
  bool whole = sm.bad != 0;  // the tile on the FP64 pipe

  if (!whole && warp == 0) {
    if (lane == 0) {
      // ---- MMAs ----
      bool ok = true;
      for (int t = 0; ok && t < steps; ++t) {
        const uint32_t s = t % kStages;
        ok = mbar_wait(&sm.full[s], (t / kStages) & 1, abort_flag, kWaitNs);
        if (!ok) break;
        tc_fence_after();
        const uint64_t bd = sw128_desc(b_smem) + 2u * s;
        for (int d = 0; d < kDigits; ++d) {
          const uint64_t ad = sw128_desc(a_smem + s * kAStage + (d >> 2) * kATile) + 2u * (d & 3u);
          const uint32_t n = TN * min(kDigits, kWeights - d);
          mma(tmem + TN * d, ad, bd, n < 256u ? n : 256u);
          if (n > 256u) mma(tmem + TN * d + 256u, ad, bd + (256u * 128u >> 4), n - 256u);
        }
        umma_commit(&sm.empty[s]);
      }
      umma_commit(&sm.done);
      if (!mbar_wait_drain(&sm.done, 0u, kWaitNs)) *abort_flag = 1;
    }
    __syncwarp();
  } else if (!whole) {
    // ---- cut ----
    const int cw = warp - 1, quad = lane & 7;
    // A quad is k = q, q + 8, q + 16, q + 24 of a step: the order of k inside a
    // step is free, as long as A and B agree, and lanes then load neighbours.
    // Rows r, r + 2, r + 4, r + 6 at a time: their 16-byte units fall into
    // different banks under the swizzle.
    int row[kQuads], ea[kQuads];
    // Rows and columns past the matrix read its last ones: their sums are not
    // written.  Only the last step can reach past k.
    const double* ap[kQuads];
#pragma unroll
    for (int u = 0; u < kQuads; ++u) {
      const int grp = cw * kQuads + u;
      row[u] = (grp >> 1) * 8 + (grp & 1) + 2 * (lane >> 3);
      ea[u] = sm.ea[row[u]] ? sm.ea[row[u]] : 1023;
      const int64_t i = i0 + row[u] < g.m ? i0 + row[u] : g.m - 1;
      ap[u] = g.A + i * g.k + quad;
    }
    // each warp also cuts a quad of B: k = cw, column `lane`
    static_assert(kCutters == KS / 4, "a quad of B per warp");
    const int eb = sm.eb[lane] ? sm.eb[lane] : 1023;
    const int64_t j = j0 + lane < g.n ? j0 + lane : g.n - 1;
    const double* bp = g.B + cw * g.n + j;
    const int64_t b8 = 8 * g.n;
    struct Values {
      double a[kQuads][4], b[4];
    };
    auto load = [&](int t, Values& v) {
      const int64_t k0 = static_cast<int64_t>(t) * KS;
      if (k0 + KS <= g.k) {
#pragma unroll
        for (int u = 0; u < kQuads; ++u)
#pragma unroll
          for (int m = 0; m < 4; ++m) v.a[u][m] = ap[u][8 * m];
#pragma unroll
        for (int m = 0; m < 4; ++m) v.b[m] = bp[m * b8];
      } else {
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const int64_t k = k0 + 8 * m;
#pragma unroll
          for (int u = 0; u < kQuads; ++u) v.a[u][m] = k + quad < g.k ? ap[u][8 * m] : 0.0;
          v.b[m] = k + cw < g.k ? bp[m * b8] : 0.0;
        }
      }
#pragma unroll
      for (int u = 0; u < kQuads; ++u) ap[u] += KS;
      bp += 4 * b8;
    };
    auto cut = [&](int t, const Values& v) -> bool {
      const uint32_t s = t % kStages;
      if (t >= kStages &&
          !__all_sync(0xffffffffu, mbar_wait(&sm.empty[s], ((t / kStages) - 1) & 1, abort_flag,
                                             kWaitNs)))
        return false;
      uint32_t out[kDigits];
#pragma unroll
      for (int u = 0; u < kQuads; ++u) {
        cut4(v.a[u], ea[u], &sm.cut_a[row[u]], out);
        const uint32_t at = a_smem + s * kAStage + row[u] * 128 + (quad & 3) * 4;
#pragma unroll
        for (int d = 0; d < kDigits; ++d)
          st32(at + (d >> 2) * kATile +
                   ((((d & 3) * 2 + (quad >> 2)) ^ (row[u] & 7)) << 4),
               out[d]);
      }
      cut4(v.b, eb, &sm.cut_b[lane], out);
      const uint32_t bt =
          b_smem + lane * 128 + (((s * 2 + (cw >> 2)) ^ (lane & 7)) << 4) + (cw & 3) * 4;
#pragma unroll
      for (int d = 0; d < kDigits; ++d) st32(bt + d * TN * 128, out[d]);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sm.full[s]);
      return true;
    };
    // loads run one step ahead
    Values next;
    load(0, next);
    for (int t = 0; t < steps; ++t) {
      const Values now = next;
      if (t + 1 < steps) load(t + 1, next);
      if (!cut(t, now)) break;
    }
    // ---- combine ----
    asm volatile("bar.sync 1, %0;" ::"n"(32 * kCutters) : "memory");  // cut_a and cut_b are whole
    if (__all_sync(0xffffffffu, mbar_wait(&sm.done, 0u, abort_flag, kWaitNs))) {
      tc_fence_after();
      constexpr int NC = 4 * TN / kCutters;  // columns per thread
      const int r = 32 * (warp & 3) + lane, c0 = NC * (cw >> 2);
      const uint32_t at = tmem + (static_cast<uint32_t>(32 * (warp & 3)) << 16) + c0;
      long long half[2][NC];  // weights 2..9 and 10..17, the last in units of one
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int c = 0; c < NC; ++c) half[h][c] = 0;
#pragma unroll
        for (int w = 0; w < 8; w += 2) {
          uint32_t f[NC], f1[NC];
          tmem_ld16(at + TN * (8 * h + w), f);
          tmem_ld16(at + TN * (8 * h + w + 1), f1);
          tmem_ld_wait(f);
          tmem_keep(f1);
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const int n = __float2int_rn(__uint_as_float(f[c]) * 262144.0f);
            const int n1 = __float2int_rn(__uint_as_float(f1[c]) * 262144.0f);
            half[h][c] = half[h][c] * 1024 + (n * 32 + n1);
          }
        }
      }
      const int64_t i = i0 + r;
      if (i < g.m) {
        const int e = sm.ea[r], lost = sm.cut_a[r];
        const int left_out = kDropped * static_cast<int>(g.k);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const int64_t j = j0 + c0 + c;
          if (j < g.n) {
            const int f = sm.eb[c0 + c];
            // 2^(ea + 2) * 2^(eb + 2) * 32^-17
            const double unit = f64emu::from_bits(static_cast<uint64_t>(e + f - 1023 + 4 - 85) << 52);
            const long long low = ((half[0][c] & 0xfffffll) << 40) + half[1][c];
            const double v = fma(static_cast<double>(half[0][c] >> 20), 0x1p60,
                                 static_cast<double>(low));
            const float least = static_cast<float>(left_out + kPerCut * (lost + sm.cut_b[c0 + c]));
            // the upper word of 2^55 times `least`, rounded up
            const uint32_t keep =
                (__float_as_uint(least) >> 3) + ((1023u - 127u + 55u) << 20) + 1u;
            if (e == 0 || f == 0) {
              g.C[i * g.n + j] = 0.0;
            } else if ((static_cast<uint32_t>(__double2hiint(v)) & 0x7fffffffu) >= keep) {
              g.C[i * g.n + j] = v * unit;
            } else {
              const int at_list = atomicAdd(&sm.redo, 1);
              sm.list[at_list] = static_cast<uint16_t>(r * TN + c0 + c);
            }
          }
        }
      }
      tc_fence_before();
    }
  }
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTmemCols)
                 : "memory");
  }
  whole = whole || sm.abort || sm.redo > max_redo(g.k);
  if (whole) {
    fp64_tile(g, i0, j0, base);
    return;
  }
  for (int q = warp; q < sm.redo; q += kThreads / 32) {
    const int64_t i = i0 + sm.list[q] / TN, j = j0 + sm.list[q] % TN;
    double dot = 0.0;
    for (int64_t k = lane; k < g.k; k += 32 * 8) {  // 16 loads in flight per lane
      double x[8], y[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int64_t ku = k + 32 * u;
        x[u] = ku < g.k ? g.A[i * g.k + ku] : 0.0;
        y[u] = ku < g.k ? g.B[ku * g.n + j] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) dot = fma(x[u], y[u], dot);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, off);
    if (lane == 0) g.C[i * g.n + j] = dot;
  }
}

int64_t tiles(const Product& p) {
  return ceil_div(p.m, TM) * ceil_div(p.n, TN);
}

}  // namespace

namespace b200 {

// From one step and a quarter of a tile on (1 x 1 x 1, all three: 24 us here, 14
// us on the FP64 pipe; 32 x 32 x 32: 71 and 112 us).
bool dgemm_tc_takes(const Product& p) {
  return p.k >= KS && p.k <= kMaxK && p.m > 0 && p.n > 0 && p.m * p.n >= TM * TN / 4 &&
         tiles(p) < (1 << 30);
}

int launch_dgemm_tc(const Product* p, int count, cudaStream_t st) {
  const int rc = allow_dynamic_smem(reinterpret_cast<const void*>(dgemm_tc_kernel), kSmemBytes,
                                    "dgemm");
  if (rc != B200_OK) return rc;
  Products ps{};
  int64_t all = 0;
  for (int i = 0; i < count; ++i) {
    ps.p[i] = p[i];
    if (i == 0) ps.tiles0 = static_cast<int>(tiles(p[0]));
    all += tiles(p[i]);
  }
  launch(dgemm_tc_kernel, static_cast<unsigned>(all), kThreads, kSmemBytes, st, ps);
  return B200_OK;
}

}  // namespace b200
