// tcgen05 decode attention over the packed tiles of a cache, on the integer tensor cores: head_dim 64 or 128, group 64, 1- to 4-bit codes,
// 1 / 2 / 4 / 8 query heads per kv head (sm_100a).
//
// Both contractions reduce over the packed rows (keys: over channels, values: over tokens), and a row of 64 codes runs along the
// dimension that is kept.  So one thread owns a row: it builds the row's book of dequantized values (fixed point, relative to the
// row's larger side S) in registers, expands the codes four at a time with byte permutes, and stores the bytes of the values, each
// in a plane of its own, as they stand into operands in shared memory that are major along the kept dimension.  The other operand is
// the query (the probabilities) times S, as a fixed-point number in signed bytes, so that the products and their sums are exact integers:
//   * a worker is two teams of four warps; a step is 128 tokens of a (batch, kv head) pair.  One team expands the keys (thread r = channel
//     r of the step's two groups) one step ahead of the other, which finishes the logits, keeps the softmax and expands the values (thread
//     r = token r with its two channel groups).  A CTA has two or three workers and a warp per worker that only issues MMAs: one
//     thread needs 55 cycles for each
//   * tcgen05.mma.kind::i8, M 128 x N 32 x K 32: M = 2 groups x 64 tokens (2 x 64 channels), N = 2 groups x 4 heads x 4 bytes; the
//     group of a row of the result picks its half of the columns
//   * the top byte is signed, the others unsigned; each plane has an accumulator of its own, and column_sum adds products of equal weight
//   * online softmax with one thread per token, the running output in registers (thread = channel); MMA completion is tracked with
//     mbarriers, and so is what the teams hand to their issuing warp.  Every wait on one is bounded: whichever warp's runs out tells its worker,
//     which poisons its records from then on (the merged output becomes NaN), issues no more products, waits for those in flight, frees its
//     tensor memory and returns.  (The named barriers left are within a team, whose warps keep step whatever runs out.)
//   * the residual window is un-quantized: its tiles have CTAs of their own (mz_dense_tiles.cuh)
//
// What bounds it: issue (58 % of the cycles; per row of 64 two-bit codes about 290 instructions, residual tiles included) and the logic pipe
// (47 %, two cycles per instruction); integer MMAs take 40 cycles each, all of it reading their operands, 31 %.  A thread that spills
// is dear: 227 KB of shared memory leave 28 KB of L1, and 20 bytes of spill per thread cost 10 %.  Hence the register split.
// 64 x 8 pairs x 4224 tokens, 4 heads, us per call: 1 bit 202 -> 108 (before: SIMT kernel), 2 bits 148 -> 134 (before: unrolled mma.sync
// kernel), 3 bits 230 -> 208 (SIMT); 24 x 8 x 1537, 3 bits: 53 -> 41.  About 7 % of these are the folds' own scales (put_folds).
//
// Precision: three planes hold a value to 2^-24 of its row's larger side and a product to 4e-9 of the step's largest for its head and group, which
// is no worse than the fp32 kernels (relative error against 64 bits 2e-7 to 7e-7 where those have 2e-7 to 1.1e-6, attention sinks, outlier
// channels and tokens of unlike range included; 1 bit is exact in one plane).  Two planes (2 bits, calls that the unrolled kernel served): 2^-15
// and 1e-6, 1e-5 to 4e-5 where the unrolled kernel has 5e-5 to 2e-4.  Any range is served: folds and query are scaled by powers of two.
#include <atomic>

#include "mz_dense_tiles.cuh"

namespace mzu {
using namespace mzm;

constexpr int STEP_GROUPS = 2;                   // groups of 64 tokens per step
constexpr int SPIN_LIMIT = 1000000;              // looks of a wait before it gives up
#ifdef MZ_BOUNDS
constexpr int SHORT_LIMIT = 0;                   // and once one has: none, so that a test fails every wait
#else
constexpr int SHORT_LIMIT = 1;
#endif
constexpr int PLANE_BYTES = 16384;               // [16-byte chunk of the kept dimension, 8][row 128][16]
constexpr int FOLD_BYTES = 4096;                 // [group 2][row 128][4 heads x 4 bytes]
constexpr float MAGIC = 12582912.0f;             // 1.5 * 2^23: adding it rounds to an integer that stands in the low mantissa bits

constexpr int DENSE_WARPS = 12, DENSE_REGS = 128;          // of a CTA that has residual tiles

// How a code width is run.  A CTA has WORKERS workers, each with four warps for the keys and four for softmax and values, and one more group
// of four warps that issue the workers' MMAs (one each).  The registers that the warps are launched with (LAUNCH each) are
// redistributed: KEY * 4 W + VALUE * 4 W + ISSUE * 4 <= LAUNCH * (8 W + 4).
template <int BITS, int P>
struct Cfg {
  static constexpr int NE = 1 << BITS, TOP = NE - 1, ZC = NE / 2;
  static constexpr int PLANES = P;                                       // bytes per value
  static constexpr int WORKERS = PLANES == 3 ? 2 : 3;
  static constexpr int WARPS = 8 * WORKERS + 4, THREADS = 32 * WARPS;
  static constexpr int LAUNCH = WORKERS == 3 ? 72 : 96, KEY = WORKERS == 3 ? 56 : BITS == 4 ? 96 : 88, VALUE = WORKERS == 3 ? 104 : BITS == 4 ? 128 : 136, ISSUE = 24;
  static_assert(DENSE_REGS * DENSE_WARPS + 24 * (WARPS - DENSE_WARPS) <= LAUNCH * WARPS, "register split of a residual CTA");
  static_assert(KEY * 4 * WORKERS + VALUE * 4 * WORKERS + ISSUE * 4 <= LAUNCH * WARPS, "register split");
  // book table: per zero code up to the middle (rows above are mirrored) slopes and offsets of the entries that may lie on the row's
  // smaller side, and for 4 bits the bytes of the upper eight entries, plane by plane
  static constexpr int MIXED = NE < 8 ? NE : 8, BOOK_ROW = BITS == 4 ? 96 : 8 * NE, BOOK_BYTES = ZC * BOOK_ROW;
  static constexpr float FULL = PLANES == 1 ? 1.0f : PLANES == 2 ? 32766.0f : 8388600.0f;      // fixed-point value of S
  // fixed-point value of 1 in the folded operand (two planes: half of it; else its upper half), and what a unit of column_sum is worth.  The
  // largest number that the digits hold is 1.129 (two planes) or 1.125 of it: scales are powers of two, found to within a factor of 1.125
  static constexpr float FOLD_FULL = PLANES == 2 ? 3700000.0f : 29000.0f;
  static constexpr float UNIT = (PLANES == 1 ? 1.0f / 65536.0f : PLANES == 2 ? 128.0f : 256.0f) / (FULL * FOLD_FULL);
  static constexpr int TM_SIDE = 32 * PLANES, TM_WORKER = 2 * TM_SIDE;   // tensor-memory columns: one accumulator per plane
  static constexpr int TM_ALLOC = WORKERS * TM_WORKER <= 256 ? 256 : 512;
  static constexpr int OFF_FOLD = PLANES * PLANE_BYTES, SIDE_BYTES = OFF_FOLD + FOLD_BYTES;      // operands of one side
  static constexpr int OFF_RED = 2 * SIDE_BYTES, WORKER_BYTES = OFF_RED + 1792;
  static constexpr int BOOKS_BYTES = (2 * BOOK_BYTES + 127) / 128 * 128;
  static constexpr int SMEM = BOOKS_BYTES + WORKERS * WORKER_BYTES;
};
// exchange between a worker's warps, doubled by the step's parity where a fast warp may be a step ahead
constexpr int RED_SK = 0;                        // [parity][warp][group][4] largest |query * S| of the keys, as the sum of the two bit patterns
constexpr int RED_SV = RED_SK + 256;             // [parity][warp][group][4] largest log2 (probability * |S|) of the values, before the maximum is taken off
constexpr int RED_MAX = RED_SV + 256;            // [parity][warp][4] largest logit
constexpr int RED_EX = RED_MAX + 128;            // [parity][group][4] what a unit of the keys' column_sum is worth
constexpr int RED_FLAG = RED_EX + 64, RED_CA = RED_FLAG + 32;      // [parity][warp] whether there is a constant term; [parity][warp][group][4] its parts
constexpr int RED_QS = RED_CA + 256;             // [4] logit (base 2) per unit of the scaled query times a key
constexpr int RED_RUN = RED_QS + 16;             // [parity][4] running maximum of the logits (base 2)
constexpr int RED_END = RED_RUN + 32;            // [warp][16]: constant terms of the output [group][4], sum of probabilities [4]
constexpr int RED_KFOLD = RED_END + 256;         // [warp of the keys][group][4] factors of the step's folds
constexpr int RED_VFOLD = RED_KFOLD + 128;       // [warp of the values]: factors of the step's folds [group][4], worth of a unit of their column_sum [group][4]
// mbarriers: products of the keys / values are done, the keys' accumulators have been read, the operands of the keys / values are written, no
// product of this worker is in flight
constexpr int RED_BARS = RED_VFOLD + 256, BAR_KDONE = RED_BARS, BAR_KFREE = RED_BARS + 8, BAR_VDONE = RED_BARS + 16, BAR_KREADY = RED_BARS + 24,
              BAR_VREADY = RED_BARS + 32, BAR_END = RED_BARS + 40, RED_TMEM = RED_BARS + 48;
constexpr int RED_FAILED = RED_TMEM + 4;         // not 0: a wait of this worker has run out
static_assert(RED_FAILED + 4 <= 1792, "exchange area");

// ---- tcgen05 / mbarrier wrappers
// this lane's row of every plane's accumulator: the 8 columns of two heads
template <int P>
__device__ __forceinline__ void tm_ld8(uint32_t taddr, int (&c)[P][8]) {
#define MZ_LD8(q) \
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];" \
               : "=r"(c[q][0]), "=r"(c[q][1]), "=r"(c[q][2]), "=r"(c[q][3]), "=r"(c[q][4]), "=r"(c[q][5]), "=r"(c[q][6]), "=r"(c[q][7]) \
               : "r"(taddr + 32 * (q)) : "memory")
  MZ_LD8(0);
  if (P > 1) MZ_LD8(P > 1 ? 1 : 0);
  if (P > 2) MZ_LD8(P > 2 ? 2 : 0);
#undef MZ_LD8
  // the wait names the registers, so that nothing reads them above it
#pragma unroll
  for (int q = 0; q < P; ++q)
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(c[q][0]), "+r"(c[q][1]), "+r"(c[q][2]), "+r"(c[q][3]), "+r"(c[q][4]), "+r"(c[q][5]), "+r"(c[q][6]), "+r"(c[q][7]) :: "memory");
}
__device__ __forceinline__ void tm_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tm_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// among the four warps of a team
__device__ __forceinline__ void team_barrier(int team) { asm volatile("bar.sync %0, 128;" ::"r"(team + 1) : "memory"); }
template <int N>
__device__ __forceinline__ void more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N>
__device__ __forceinline__ void fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
  return p != 0;
}
// table reads: constant after the set-up, so they may be moved and merged
__device__ __forceinline__ uint4 book128(uint32_t a) {
  uint4 v;
  asm("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
// shared-memory operand, not swizzled, major along the kept dimension: core matrices of 8 rows x 16 bytes, 128 bytes apart along the
// reduction (leading offset), 2048 bytes along the kept dimension (stride offset)
__device__ __forceinline__ uint64_t descriptor(uint32_t sa) {
  return (uint64_t)((sa >> 4) & 0x3FFF) | (128ull >> 4) << 16 | (2048ull >> 4) << 32 | 1ull << 46;
}
// D[128 x 32] (+)= A[128 x 32] * B[32 x 32], 8-bit integers into 32-bit
template <bool SIGNED_A>
__device__ __forceinline__ void umma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t accumulate) {
  const uint32_t idesc = (2u << 4) | ((SIGNED_A ? 1u : 0u) << 7) | (1u << 10) | (1u << 15) | (1u << 16) | (4u << 17) | (8u << 24);
  const uint32_t zero = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(zero), "r"(zero), "r"(zero), "r"(zero) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// the products of a side: its rows in slices of 32, each plane on an accumulator of its own
template <int BITS, int P, int SLICES>
__device__ __forceinline__ void umma_side(uint32_t d_tmem, uint64_t values, uint64_t folds) {
#pragma unroll
  for (int j = 0; j < SLICES; ++j)
#pragma unroll
    for (int q = 0; q < Cfg<BITS, P>::PLANES; ++q) {
      const uint64_t a = values + ((q * PLANE_BYTES + j * 512) >> 4), b = folds + j * (512 >> 4);
      if (q == 0) umma<true>(d_tmem, a, b, j > 0);
      else umma<false>(d_tmem + 32 * q, a, b, j > 0);
    }
}
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
  asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.shared::cta.b64 t, [%0];\n\t}\n" ::"r"(bar) : "memory");
}
// waits for phase `parity` of an mbarrier with a limit.  Who gives up says so to the whole worker before it goes on, so that what it spoils
// from then on is in a record that is poisoned; its later waits are short.  SLEEP: ns between looks, for a team that is ahead anyway.  (What
// stands here is dear: a limit or first value of `failed` that only the launch knows costs 2 to 15 % of a call.)
template <int SLEEP = 0>
__device__ __forceinline__ void bar_wait(uint32_t bar, uint32_t parity, uint32_t red, bool& failed) {
  const int limit = failed ? SHORT_LIMIT : SPIN_LIMIT;
  for (int it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return;
    if (SLEEP > 0) __nanosleep(SLEEP);
  }
  failed = true;
  sts32(red + RED_FAILED, 1u);
}

// ---- books.  A row's zero code is brought to the lower half by mirroring (code -> TOP - code, S -> -S): then the side above it is the
// larger one, its fixed-point values FULL * u are the same for every row with that zero code, and the values below are FULL * u *
// (smaller / larger side).
__device__ __forceinline__ float unit_value(float alpha, int e, int zc, int top) {
  const int room = max(e >= zc ? top - zc : zc, 1), n = min(abs(e - zc), room);
  const float grow = expm1f((float)n / (float)room * log1pf(alpha)) / alpha;
  return e >= zc ? grow : -grow;
}
template <int BITS, int P>
__device__ __forceinline__ void fill_books(uint32_t table, float alpha, int first, int n) {
  using C = Cfg<BITS, P>;
  for (int i = first; BITS > 1 && i < C::ZC * C::NE; i += n) {
    const int zc = i / C::NE, e = i % C::NE;
    const float u = C::FULL * unit_value(alpha, e, zc, C::TOP);
    const uint32_t row = table + zc * C::BOOK_ROW;
    if (e < C::MIXED) {
      stsf(row + e * 4, e < zc ? u : 0.0f);
      stsf(row + C::MIXED * 4 + e * 4, (P == 2 ? MAGIC : 0.0f) + (e < zc ? 0.0f : rintf(u)));
    } else {
      for (int q = 0; q < P; ++q) sts8(row + 64 + 8 * q + (e - 8), (uint32_t)(__float2int_rn(u) >> (8 * (P - 1 - q))) & 0xff);
    }
  }
}

// constants of one row: signed scale, ratio of the smaller to the larger side, value of the zero code, mirrored zero code
struct Row { float s, ratio, A; uint32_t zc; };
template <int BITS, int P, bool EXACT>
__device__ __forceinline__ Row prepare_row(float lo, float span) {
  constexpr int TOP = Cfg<BITS, P>::TOP;
  Row r;
  float bup, bdn;
  int zc;
  bool wild = false;       // never with 16-bit floats of 5 exponent bits
  row_split(lo, span, (float)TOP, r.A, bup, bdn, zc, wild);
  if (EXACT) zc = exact_zero_code(lo, span, (float)TOP);
  const bool mirrored = zc > TOP / 2 && bup < INFINITY;              // an infinite range has no zero code; it stays S = inf
  const float big = mirrored ? bdn : bup, small = mirrored ? bup : bdn;
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(big));
  r.ratio = small * y;
  r.s = mirrored ? -big : big;
  r.zc = min((uint32_t)(mirrored ? TOP - zc : zc), (uint32_t)(TOP / 2));
  return r;
}
// a book entry: offset + slope * ratio as an integer.  Two planes: in the low mantissa bits, by magic addition in the offset; three: 24 bits
template <int P>
__device__ __forceinline__ uint32_t book_entry(uint32_t slope, float ratio, uint32_t offset) {
  const float v = fmaf(__uint_as_float(slope), ratio, __uint_as_float(offset));
  return P == 2 ? __float_as_uint(v) : (uint32_t)__float2int_rn(v);
}
// four book entries -> their bytes, plane by plane, top byte first
template <int P>
__device__ __forceinline__ void pack4(const uint32_t* v, uint32_t* plane) {
  const uint32_t a = prmt(v[0], v[1], 0x5140u), b = prmt(v[2], v[3], 0x5140u);
  plane[P - 1] = prmt(a, b, 0x5410u);
  plane[P - 2] = prmt(a, b, 0x7632u);
  if (P == 3) plane[0] = prmt(prmt(v[0], v[1], 0x0062u), prmt(v[2], v[3], 0x0062u), 0x5410u);
}
// expands the 64 codes of one row: `dst` is the row's 16 bytes in the first chunk of its group's half of the first plane.  The permutes
// take their selector from the low half of a register; `two16` is 2^16 as a run-time value, so that the multiplier brings the
// upper half down: the logic pipe is the busy one
template <int BITS, int P, int NW>
__device__ __forceinline__ void expand_row(const uint32_t (&w)[NW], const Row& r, uint32_t table, uint32_t dst, uint32_t two16) {
  using C = Cfg<BITS, P>;
  const uint32_t flip = (uint32_t)(__float_as_int(r.s) >> 31);       // mirrored rows: TOP - code is the complement
  if constexpr (BITS == 1) {
    // the zero code is the first (mirrored: the last) code, so a value is S times the (complemented) code
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      // 16 codes: four nibble fields of one bit; position 4 k + j of the chunk is code k + 4 j
      const uint32_t c = (q & 1) ? __umulhi(w[q >> 1] ^ flip, two16) : w[q >> 1] ^ flip;
      sts128(dst + q * 2048, make_uint4(prmt(0x00000100u, 0u, c & 0x1111u), prmt(0x00000100u, 0u, c >> 1 & 0x1111u),
                                        prmt(0x00000100u, 0u, c >> 2 & 0x1111u), prmt(0x00000100u, 0u, c >> 3 & 0x1111u)));
    }
  } else {
    const uint32_t row = table + r.zc * C::BOOK_ROW;
    constexpr int Q = C::MIXED / 4;
    uint32_t book[P][Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const uint4 t = book128(row + 16 * q), c = book128(row + C::MIXED * 4 + 16 * q);
      uint32_t v[4], b[P];
      v[0] = book_entry<P>(t.x, r.ratio, c.x);
      v[1] = book_entry<P>(t.y, r.ratio, c.y);
      v[2] = book_entry<P>(t.z, r.ratio, c.z);
      v[3] = book_entry<P>(t.w, r.ratio, c.w);
      pack4<P>(v, b);
#pragma unroll
      for (int k = 0; k < P; ++k) book[k][q] = b[k];
    }
    if constexpr (BITS == 2) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t even = (w[q] ^ flip) & 0x33333333u, odd = ((w[q] >> 2) ^ flip) & 0x33333333u;
        const uint32_t even2 = __umulhi(even, two16), odd2 = __umulhi(odd, two16);
#pragma unroll
        for (int k = 0; k < P; ++k)
          sts128(dst + k * PLANE_BYTES + q * 2048, make_uint4(prmt(book[k][0], 0u, even), prmt(book[k][0], 0u, even2), prmt(book[k][0], 0u, odd), prmt(book[k][0], 0u, odd2)));
      }
    } else if constexpr (BITS == 4) {
      // lower eight entries from the registers, upper eight from the table; a code's top bit says which
      const uint4 a = book128(row + 64), b = book128(row + 80);
      const uint32_t up[3][2] = {{a.x, a.y}, {a.z, a.w}, {b.x, b.y}};
      const uint32_t flip4 = flip & 0x44444444u;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t o[P][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t c = w[2 * q + (k >> 1)];
          uint32_t sel = (c ^ flip) & 0x77777777u, top = ((c >> 1) & 0x44444444u) ^ flip4;
          if (k & 1) { sel = __umulhi(sel, two16); top = __umulhi(top, two16); }
          const uint32_t m = prmt(0u, 0xFFFFFFFFu, top);
#pragma unroll
          for (int p = 0; p < P; ++p) o[p][k] = (prmt(book[p][0], book[p][Q - 1], sel) & ~m) | (prmt(up[p][0], up[p][1], sel) & m);
        }
#pragma unroll
        for (int p = 0; p < P; ++p) sts128(dst + p * PLANE_BYTES + q * 2048, make_uint4(o[p][0], o[p][1], o[p][2], o[p][3]));
      }
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t o[P][4];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          // 24 bits from bit 24 (2 q + k) on, spread to eight nibbles: the multiplier adds what has to move
          constexpr uint32_t M12 = 0x00FFF000u, M6 = 0x0FC00FC0u, M3 = 0x38383838u;
          const int bit = 24 * (2 * q + k), word = bit >> 5, sh = bit & 31;
          uint32_t x = sh == 0 ? w[word] : sh <= 8 ? w[word] >> sh : __funnelshift_r(w[word], w[(word + 1) % NW], sh);
          x = (x ^ flip) & 0x00FFFFFFu;
          x = (x & M12) * 15u + x;
          x = (x & M6) * 3u + x;
          x = (x & M3) * 1u + x;
          const uint32_t x2 = __umulhi(x, two16);
#pragma unroll
          for (int b = 0; b < P; ++b) { o[b][2 * k] = prmt(book[b][0], book[b][Q - 1], x); o[b][2 * k + 1] = prmt(book[b][0], book[b][Q - 1], x2); }
        }
#pragma unroll
        for (int b = 0; b < P; ++b) sts128(dst + b * PLANE_BYTES + q * 2048, make_uint4(o[b][0], o[b][1], o[b][2], o[b][3]));
      }
    }
  }
}
// position inside a 16-byte chunk of the kept dimension -> code of the row
template <int BITS>
__device__ __forceinline__ int chunk_code(int i) {
  if (BITS == 1) return (i >> 2) + 4 * (i & 3);
  if (BITS > 2) return i;
  return (i & 8) ? 2 * (i & 7) + 1 : 2 * (i & 7);
}

// fold value x * s, |x| <= FOLD_FULL, |s| < 1, in signed base-256 digits, low digit first.  Two planes: 2 x s rounded (24 bits) in three
// digits, the top byte is of no use (its columns of the result are not read).  Else 2^16 x s rounded (31 bits) in four: the upper half is
// rounded off by one magic addition, what is left by another, and the constants add up to 0x80808080.
template <int P>
__device__ __forceinline__ uint32_t fold_digits(float x, float s) {
  if (P == 2) return (__float_as_uint(fmaf(x, s, MAGIC + 16448.0f)) << 1) ^ 0x00808080u;
  constexpr float HIGH = MAGIC + 13632.0f, LOW = MAGIC + 32896.0f;
  const float h = fmaf(x, s, HIGH), rest = fmaf(x, s, -(h - HIGH));
  return (__float_as_uint(h) * 65536u + __float_as_uint(fmaf(rest, 65536.0f, LOW))) ^ 0x80808080u;
}
// a result row's accumulators of one head -> sum of value * fold in units of UNIT.  Column k of plane q counts digit k of the fold with byte
// q of the values; products of equal weight are added, the largest three weights (and for three planes the fourth) count.
template <int P>
__device__ __forceinline__ float column_sum(const int (&c)[P][8], int at) {
  const int* a = c[0] + at;
  if (P == 1) return fmaf((float)a[3], 16777216.0f, fmaf((float)a[2], 65536.0f, (float)(a[0] + a[1] * 256)));
  const int* b = c[P > 1 ? 1 : 0] + at;
  if (P == 2) return fmaf((float)a[2], 65536.0f, (float)(a[0] + b[1] + 256 * (a[1] + b[2])));
  const int* d = c[P > 2 ? 2 : 0] + at;
  return fmaf((float)a[3], 65536.0f, (float)(a[1] + b[2] + d[3] + 256 * (a[2] + b[3]) + ((a[0] + b[1] + d[2]) >> 8)));
}

// power of two that brings a positive number of exponent field `ex` (up to 255) into [0.5, 1), and half its inverse.  What is not finite has no
// digits: its inverse is NaN, and so is every sum that it has a part in
__device__ __forceinline__ float scale_down(uint32_t ex) {
  return __uint_as_float(ex <= 252u ? (253u - max(ex, 1u)) << 23 : 0x00800000u >> (ex - 252u));
}
__device__ __forceinline__ float half_scale_up(uint32_t ex) { return __uint_as_float(ex < 255u ? max(ex, 1u) << 23 : 0x7FFFFFFFu); }
__device__ __forceinline__ float lg2f(float x) {
  float y;
  asm("lg2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// maxima that keep a NaN
__device__ __forceinline__ float max_nan(float a, float b) {
  float y;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
  return y;
}
__device__ __forceinline__ float warp_max_nan(float a) {
  float y;
  asm("redux.sync.max.NaN.f32 %0, %1, 0xffffffff;" : "=f"(y) : "f"(a));
  return y;
}
// exponent field of the largest magnitude of a head's query (HD elements of 16 bits)
template <int HD>
__device__ __forceinline__ uint32_t query_exponent(const uint16_t* q, int lane, int dtype) {
  const uint32_t a = *((const uint32_t*)q + lane), b = HD == 128 ? *((const uint32_t*)q + 32 + lane) : 0u;
  const uint32_t mx = __reduce_max_sync(0xffffffffu, max(max(a & 0x7FFFu, a >> 16 & 0x7FFFu), max(b & 0x7FFFu, b >> 16 & 0x7FFFu)));
  return __float_as_uint(mz_u16_to_float((uint16_t)mx, dtype)) >> 23;
}


struct Place { int pair, step, b, kvh; };
std::atomic<int> g_fail_waits{0};                // mz_debug_fail_waits (checked build)

template <int BITS, int P, int HD, int GQA, bool HALF_META>
__global__ void __launch_bounds__(Cfg<BITS, P>::THREADS, 1) decode_umma_kernel(const MzDecodeParams p, const uint32_t two16) {
  using C = Cfg<BITS, P>;
  constexpr int WORKERS = C::WORKERS;
  constexpr int QB = G * BITS / 8;            // bytes of a packed row of 64 codes
  constexpr int NW = QB / 4;                  // words of it
  constexpr int NG = HD / G;                  // channel groups of a token
  constexpr int CODE_BYTES = HD * QB;         // packed bytes of one tile side
  constexpr int VROW = NG * QB;               // bytes of one token's value codes
  extern __shared__ __align__(128) uint8_t smem[];
  const mz_kv_store& s = p.s;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);            // uniform: the descriptors stay in uniform registers
  const bool issuer = warp >= 8 * WORKERS;
  const int lane = threadIdx.x & 31, w = warp & 3, team = warp >> 2, wk = issuer ? min(w, WORKERS - 1) : warp >> 3;
  const bool keys = (team & 1) == 0;
  const int r = w * 32 + lane;                                                    // row of the operands and of the results
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (p.hetero > 0 && (int)blockIdx.x >= p.hetero) {
    // ================= a CTA of the residual tiles: twelve warps of its own plan =================
    if (warp >= DENSE_WARPS) {
      fewer_registers<24>();
      return;
    }
    more_registers<DENSE_REGS>();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    mzd::dense_tiles<HD, GQA>(p, p.tp2, p.slots_a, ((int)blockIdx.x - p.hetero) * DENSE_WARPS + warp,
                          (uint32_t)__cvta_generic_to_shared(smem) + warp * mzd::WARP_BYTES);
    return;
  }

  const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);
  const uint32_t book = base + (keys ? 0 : C::BOOK_BYTES);
  const uint32_t worker = base + C::BOOKS_BYTES + wk * C::WORKER_BYTES;
  const uint32_t side = worker + (keys ? 0 : C::SIDE_BYTES), red = worker + C::OFF_RED;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(red + RED_TMEM), "r"(C::TM_ALLOC));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  if (!issuer && keys && r == 0) {
    bar_init(red + BAR_KDONE, 2); bar_init(red + BAR_KFREE, 4); bar_init(red + BAR_VDONE, 1);
    bar_init(red + BAR_KREADY, 4); bar_init(red + BAR_VREADY, 4); bar_init(red + BAR_END, 1);
    sts32(red + RED_FAILED, 0u);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  fill_books<BITS, P>(base, s.alpha_key, threadIdx.x, C::THREADS);
  fill_books<BITS, P>(base + C::BOOK_BYTES, s.alpha_value, threadIdx.x, C::THREADS);
  tm_fence_before();
  __syncthreads();
  tm_fence_after();
  const uint32_t tm_base = lds32(red - wk * C::WORKER_BYTES + RED_TMEM);             // kept by worker 0
  const uint32_t tm_k = tm_base + wk * C::TM_WORKER, tm_v = tm_k + C::TM_SIDE;

  const int T = p.tp.tiles_per_pair;          // steps per (batch, kv head) pair
  const int kt = s.k_groups;
  const int gwk = blockIdx.x * WORKERS + wk;
  long long f0 = 0, f1 = 0;
  if (gwk < p.tp.total_warps) mz_warp_tiles(p.tp, gwk, &f0, &f1);
  const int steps = (int)(f1 - f0);
  Place cur;
  cur.pair = (int)((unsigned)f0 / (unsigned)T); cur.step = (int)((unsigned)f0 % (unsigned)T);
  cur.b = cur.pair / s.kv_heads; cur.kvh = cur.pair % s.kv_heads;
  auto advance = [&](Place& c) {
    if (++c.step == T) {
      c.step = 0; ++c.pair;
      if (++c.kvh == s.kv_heads) { c.kvh = 0; ++c.b; }
    }
  };
#ifdef MZ_BOUNDS
  bool failed = p.fail_waits != 0;
#else
  bool failed = false;
#endif
  const bool meta32 = s.meta_dtype == MZ_F32;
  // everything above reads kernel parameters only and may run while the grid before drains
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // rows in flight, one of either group: codes and metadata as loaded (16-bit metadata in the low half)
  uint32_t code[2][NW], lo[2], span[2];
  const int channel = r & (HD - 1);                                   // keys: its channel (64 of them: the other threads have no rows)
  const int half = r >> 6;                                            // values: group of this thread's token; also of its row of the results
  const int spot = (r & 0x70) + chunk_code<BITS>(r & 15);             // values: its token of a step, and its channel of the output
  // Keys: channel r of the step's two groups (a last half step reads its group twice); values: token `spot` with its two channel groups (in a
  // last half step the tokens of the first group twice, the second time with probability zero).
  // The cursor of the loads runs ahead: pointers of the step `ahead`, advanced with it.
  Place ahead = cur;
  const int msz = HALF_META ? 2 : meta32 ? 4 : 2;
  const uint8_t *code_at, *mn_at, *span_at;
  auto point = [&]() {
    const int kvh = ahead.kvh >> p.kv_share;
    const long long tile = STEP_GROUPS * ahead.step;
    const long long row = keys ? channel : half * G + (spot & 63);
    const long long m = keys ? ahead.b * s.km_stride_b + kvh * s.km_stride_h + tile * HD + row : ahead.b * s.vm_stride_b + kvh * s.vm_stride_h + (tile * G + row) * NG;
    code_at = keys ? s.packed_k + ahead.b * s.pk_stride_b + kvh * s.pk_stride_h + tile * CODE_BYTES + row * QB
                   : s.packed_v + ahead.b * s.pv_stride_b + kvh * s.pv_stride_h + (tile * G + row) * VROW;
    mn_at = (const uint8_t*)(keys ? s.k_mn : s.v_mn) + m * msz;
    span_at = (const uint8_t*)(keys ? s.k_scale : s.v_scale) + m * msz;
  };
  auto move_ahead = [&]() {
    if (++ahead.step == T) {
      ahead.step = 0; ++ahead.pair;
      if (++ahead.kvh == s.kv_heads) { ahead.kvh = 0; ++ahead.b; }
      point();
    } else {
      code_at += STEP_GROUPS * CODE_BYTES;
      mn_at += STEP_GROUPS * HD * msz;
      span_at += STEP_GROUPS * HD * msz;
    }
  };
  // bytes (codes) / elements (metadata) from the first row's to this thread's row of either group
  const int x_codes = keys ? CODE_BYTES : (NG - 1) * QB, x_meta = keys ? HD : NG - 1;     // (one channel group: the row twice, not used)
  const uint8_t* code_next;                                           // codes of the step that comes next
  int code_second;
  auto load_meta = [&]() {                                            // and keeps where the codes are
    int back = 0, second = x_meta;                                    // tokens back from the first row, elements on to the second
    code_next = code_at; code_second = x_codes;
    if (STEP_GROUPS * ahead.step + 1 >= kt) {                         // a last half step
      if (keys) second = code_second = 0;
      else if (half) back = -G;
      code_next += back * VROW;
    }
    const uint8_t* a = mn_at + back * NG * msz;
    const uint8_t* b = span_at + back * NG * msz;
    if (HALF_META || !meta32) {
      lo[0] = __ldg((const uint16_t*)a); lo[1] = __ldg((const uint16_t*)a + second);
      span[0] = __ldg((const uint16_t*)b); span[1] = __ldg((const uint16_t*)b + second);
    } else {
      lo[0] = __ldg((const uint32_t*)a); lo[1] = __ldg((const uint32_t*)a + second);
      span[0] = __ldg((const uint32_t*)b); span[1] = __ldg((const uint32_t*)b + second);
    }
  };
  auto load_codes = [&](int x) {
    if constexpr (QB % 16 == 0) {
      const uint4* src = (const uint4*)(code_next + (x ? code_second : 0));
#pragma unroll
      for (int i = 0; i < NW / 4; ++i) {
        const uint4 v = __ldg(src + i);
        code[x][4 * i] = v.x; code[x][4 * i + 1] = v.y; code[x][4 * i + 2] = v.z; code[x][4 * i + 3] = v.w;
      }
    } else {
      const uint2* src = (const uint2*)(code_next + (x ? code_second : 0));
#pragma unroll
      for (int i = 0; i < NW / 2; ++i) {
        const uint2 v = __ldg(src + i);
        code[x][2 * i] = v.x; code[x][2 * i + 1] = v.y;
      }
    }
  };
  Row rows[2];
  // row constants from the metadata in flight
  auto prepare = [&]() {
#pragma unroll
    for (int x = 0; x < 2; ++x)
      rows[x] = HALF_META ? prepare_row<BITS, P, false>(mz_u16_to_float((uint16_t)lo[x], MZ_F16), mz_u16_to_float((uint16_t)span[x], MZ_F16))
                : meta32  ? prepare_row<BITS, P, true>(__uint_as_float(lo[x]), __uint_as_float(span[x]))
                          : prepare_row<BITS, P, true>(mz_u16_to_float((uint16_t)lo[x], s.meta_dtype), mz_u16_to_float((uint16_t)span[x], s.meta_dtype));
  };
  auto magnitude = [&](int x) { return __float_as_uint(rows[x].s) & 0x7FFFFFFFu; };
  // Folds are scaled by their largest product, per head and group of the step: rounding and dropped low products of digits then come to 1e-6 (two
  // planes) or 4e-9 of the largest addend of a sum (rms), whatever the sides and queries or probabilities beside it.  (One scale for the largest side times the
  // largest query or probability lost 2 to 40 times the fp32 kernels' error where these do not meet: a token that
  // dominates and has a small value, an outlier channel with a small query.  Finding the products costs 7 % of a call: 8 x 8 pairs x 131072
  // tokens at 2 bits 408 -> 437 us.  Their factors before the output of the step before, instead of behind it: 444.)  They are kept per
  // warp at `factors`.
  auto put_folds = [&](const float (&x)[GQA], uint32_t factors, int groups) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (k >= groups) break;
      const uint4 f = lds128(factors + 16 * k);
      uint32_t d[4] = {0, 0, 0, 0};
#pragma unroll
      for (int g = 0; g < GQA; ++g) d[g] = fold_digits<P>(x[g] * __uint_as_float(g == 0 ? f.x : g == 1 ? f.y : g == 2 ? f.z : f.w), rows[k].s);
      sts128(side + C::OFF_FOLD + k * 2048 + r * 16, make_uint4(d[0], d[1], d[2], d[3]));
    }
  };

  if (issuer) {
    // ================= the issuing warps: keys of step i + 1, then values of step i =================
    fewer_registers<C::ISSUE>();
    if (w < WORKERS) {
      const uint64_t key_values = descriptor(worker), key_folds = descriptor(worker + C::OFF_FOLD);
      const uint64_t value_values = descriptor(worker + C::SIDE_BYTES), value_folds = descriptor(worker + C::SIDE_BYTES + C::OFF_FOLD);
      for (int i = -1; i < steps; ++i) {
        if (i + 1 < steps) {
          bar_wait(red + BAR_KREADY, (uint32_t)(i + 1) & 1, red, failed);
          if (i >= 0) bar_wait(red + BAR_KFREE, (uint32_t)i & 1, red, failed);        // the logits before have been read
          tm_fence_after();
          if (elect_one()) {
            bar_arrive(red + BAR_KDONE);                              // hands on what the team has noted
            if (!failed) umma_side<BITS, P, HD / 32>(tm_k, key_values, key_folds);
            umma_commit(red + BAR_KDONE);
          }
          __syncwarp();
        }
        if (i >= 0) {
          bar_wait(red + BAR_VREADY, (uint32_t)i & 1, red, failed);
          tm_fence_after();
          if (elect_one()) {
            if (!failed) umma_side<BITS, P, 4>(tm_v, value_values, value_folds);
            umma_commit(red + BAR_VDONE);
          }
          __syncwarp();
        }
      }
      // no product may be in flight when the tensor memory goes back, whoever has given up before
      if (elect_one()) umma_commit(red + BAR_END);
      __syncwarp();
      bool given_up = false;
      bar_wait(red + BAR_END, 0, red, given_up);
    }
  } else if (keys) {
    fewer_registers<C::KEY>();
    if (steps > 0) {
    // ================= keys: channel r of the step's groups, one step ahead of the values =================
    float qn[GQA];                                                    // query of this channel, scaled per head into (-1, 1)
    auto load_query = [&](const Place& c) {
#pragma unroll
      for (int g = 0; g < GQA; ++g) {
        const uint16_t* q = (const uint16_t*)p.query + c.b * p.q_stride_b + (long long)(c.kvh * GQA + g) * p.q_stride_h;
        qn[g] = mz_u16_to_float(q[channel], s.kv_dtype) * scale_down(query_exponent<HD>(q, lane, s.kv_dtype));
      }
    };
    // the warp's largest products: bit patterns of positive numbers add up to that of their product but for a factor in [8/9, 1].  A side
    // that is not finite outweighs every finite product
    auto publish_products = [&](uint32_t at) {
      uint32_t m[2][4];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const uint32_t a = magnitude(x) < 0x7F800000u ? magnitude(x) : 0xC0000000u;
#pragma unroll
        for (int g = 0; g < 4; ++g) m[x][g] = g < GQA ? __reduce_max_sync(0xffffffffu, a + (__float_as_uint(qn[g % GQA]) & 0x7FFFFFFFu)) : 0u;
      }
      if (lane == 0) {
        sts128(at + 32 * w, make_uint4(m[0][0], m[0][1], m[0][2], m[0][3]));
        sts128(at + 32 * w + 16, make_uint4(m[1][0], m[1][1], m[1][2], m[1][3]));
      }
    };
    point();
    load_meta();
    load_codes(0);
    load_codes(1);
    load_query(cur);
    prepare();
    publish_products(red + RED_SK);
    if (steps > 1) { move_ahead(); load_meta(); }
    team_barrier(team);
    for (int i = 0; i < steps; ++i) {
      const int par = i & 1;
      const bool more = i + 1 < steps;
      // lane l has group and head l mod 8
      uint32_t most = lds32(red + RED_SK + 128 * par + 4 * lane);
      most = max(most, __shfl_xor_sync(0xffffffffu, most, 8));
      most = max(most, __shfl_xor_sync(0xffffffffu, most, 16));
      const uint32_t ex = (uint32_t)min(max((int)(most >> 23) - 127, 1), 255);
      if (lane < 8) stsf(red + RED_KFOLD + 32 * w + 4 * lane, scale_down(ex) * C::FOLD_FULL);
      __syncwarp();
      if (i > 0) bar_wait<64>(red + BAR_KDONE, (uint32_t)(i - 1) & 1, red, failed);       // the operands have been read
      const bool own = HD == 128 || w < 2;                            // this warp has rows
      if (own) expand_row<BITS, P, NW>(code[0], rows[0], book, side + r * 16, two16);
      if (more) load_codes(0);
      if (own) expand_row<BITS, P, NW>(code[1], rows[1], book, side + 8192 + r * 16, two16);
      if (more) load_codes(1);
      if (own) put_folds(qn, red + RED_KFOLD + 32 * w, 2);
      // constant term sum_d q[h][d] A_d per group and head (rows whose range does not straddle zero): this warp's part
      const bool any = own && __any_sync(0xffffffffu, rows[0].A != 0.0f || rows[1].A != 0.0f);
      if (any) {
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int g = 0; g < GQA; ++g) {
            float v = qn[g] * rows[x].A;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            if (lane == 0) stsf(red + RED_CA + par * 128 + ((w * 2 + x) * 4 + g) * 4, v);
          }
      }
      if (lane == 0) sts32(red + RED_FLAG + par * 16 + 4 * w, any ? 1u : 0u);
      if (w == 0 && lane < 8) stsf(red + RED_EX + 32 * par + 4 * lane, half_scale_up(ex) * (2.0f * C::UNIT));
      const int pair = cur.pair;
      advance(cur);
      if (more) {
        prepare();
        if (cur.pair != pair) load_query(cur);
        publish_products(red + RED_SK + 128 * (par ^ 1));
      }
      if (i + 2 < steps) { move_ahead(); load_meta(); }
      proxy_fence();
      __syncwarp();
      if (lane == 0) bar_arrive(red + BAR_KREADY);
      team_barrier(team);
    }
    }
  } else {
    more_registers<C::VALUE>();
    if (steps > 0) {
    // ================= softmax and values: thread r has row r of the results =================
    const uint32_t tm_mine = ((uint32_t)(32 * w) << 16) + 16 * half;
    float l_part[GQA], out[GQA];                                      // this thread's sum of probabilities, output
    float base_sum = 0.f;                                             // lane 4 x + g: sum p * A of the warp's tokens, channel group x and head g
    bool has_base = false;
    int seg = 0;
    auto start_pair = [&](const Place& c) {
#pragma unroll
      for (int g = 0; g < GQA; ++g) {
        l_part[g] = out[g] = 0.f;
        const uint16_t* q = (const uint16_t*)p.query + c.b * p.q_stride_b + (long long)(c.kvh * GQA + g) * p.q_stride_h;
        const uint32_t ex = query_exponent<HD>(q, lane, s.kv_dtype);
        if (r == 0) stsf(red + RED_QS + 4 * g, half_scale_up(ex) * p.scaling * (2.0f * LOG2E));     // read behind the next barrier but one
      }
      if (r < 2) sts128(red + RED_RUN + 16 * r, make_uint4(0xFF800000u, 0xFF800000u, 0xFF800000u, 0xFF800000u));
      base_sum = 0.f; has_base = false;
      team_barrier(team);
    };
    // adds the products of step v's values to the output
    auto drain = [&](int v) {
      bar_wait(red + BAR_VDONE, (uint32_t)v & 1, red, failed);
      tm_fence_after();
#pragma unroll
      for (int g = 0; g < GQA; g += 2) {
        int c[P][8];
        tm_ld8<P>(tm_v + tm_mine + 4 * g, c);
        const uint2 up = lds64(red + RED_VFOLD + 64 * w + 32 + 16 * half + 4 * g);
        out[g] = fmaf(column_sum<P>(c, 0), __uint_as_float(up.x), out[g]);
        if (g + 1 < GQA) out[(g + 1) % GQA] = fmaf(column_sum<P>(c, 4), __uint_as_float(up.y), out[(g + 1) % GQA]);
      }
      tm_fence_before();
    };
    // ---- end of a segment: the partial record (m, l, acc) of this worker for the pair it just left
    auto write_partial = [&](int par) {
#pragma unroll
      for (int g = 0; g < GQA; ++g) {
        float lsum = l_part[g];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, off);
        if (lane == 0) stsf(red + RED_END + w * 64 + 32 + 4 * g, lsum);
      }
      if (lane < 8) stsf(red + RED_END + w * 64 + 4 * lane, base_sum);
      team_barrier(team);
      const long long slot0 = ((long long)gwk * p.tp.max_segs + seg) * GQA;
      if (MZ_IN_BOUNDS(slot0 + GQA - 1, p.part.slots, 12)) {          // always true outside the checked build
#pragma unroll
        for (int g = 0; g < GQA; ++g) {
          float bs = 0.f, lt = 0.f;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            bs += ldsf(red + RED_END + k * 64 + 16 * half + 4 * g);
            lt += ldsf(red + RED_END + k * 64 + 32 + 4 * g);
          }
          // a NaN probability has no digits either: what shows it is their sum
          if (HD == 128 || r < HD) p.part.acc[(slot0 + g) * HD + spot] = lt == lt ? out[g] + bs : lt;
          if (r == 0) {
            // a wait of any of the worker's warps ran out: +inf turns the merged output into NaN
            p.part.m[slot0 + g] = lds32(red + RED_FAILED) != 0 ? INFINITY : ldsf(red + RED_RUN + 16 * par + 4 * g) * (1.0f / LOG2E);
            p.part.l[slot0 + g] = lt;
          }
        }
      }
      team_barrier(team);
    };
    point();
    load_meta();
    load_codes(0);
    load_codes(1);
    start_pair(cur);
    bool pending = false;                                             // the last step's values are not in the output yet
    for (int i = 0; i < steps; ++i) {
      const int par = i & 1;
      Place nxt = cur;
      advance(nxt);
      prepare();
      const bool more = i + 1 < steps;
      if (more) { move_ahead(); load_meta(); }
      const bool live = STEP_GROUPS * cur.step + half < kt;
      float mask = 0.f;
      if (p.mask && live)
        mask = mz_load_as_float(p.mask, cur.b * p.mask_stride_b + (long long)cur.step * (STEP_GROUPS * G) + spot, p.mask_dtype) * LOG2E;
      // ================= logits of token `spot` =================
      bar_wait(red + BAR_KDONE, (uint32_t)par, red, failed);
      tm_fence_after();
      float lg[GQA];
      {
#pragma unroll
        for (int g = 0; g < GQA; g += 2) {
          int c[P][8];
          tm_ld8<P>(tm_k + tm_mine + 4 * g, c);
          lg[g] = column_sum<P>(c, 0);
          if (g + 1 < GQA) lg[(g + 1) % GQA] = column_sum<P>(c, 4);
        }
        const uint4 up = lds128(red + RED_EX + 32 * par + 16 * half);
        const uint4 fl = lds128(red + RED_FLAG + 16 * par);
        float ca[GQA];
#pragma unroll
        for (int g = 0; g < GQA; ++g) ca[g] = 0.f;
        if (fl.x | fl.y | fl.z | fl.w) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const bool on = (k == 0 ? fl.x : k == 1 ? fl.y : k == 2 ? fl.z : fl.w) != 0;
#pragma unroll
            for (int g = 0; g < GQA; ++g) ca[g] += on ? ldsf(red + RED_CA + par * 128 + ((k * 2 + half) * 4 + g) * 4) : 0.f;
          }
        }
        tm_fence_before();
        __syncwarp();
        if (lane == 0) bar_arrive(red + BAR_KFREE);
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        const uint4 qs = lds128(red + RED_QS);
#pragma unroll
        for (int g = 0; g < GQA; ++g) {
          const float v = fmaf(lg[g], __uint_as_float(g == 0 ? up.x : g == 1 ? up.y : g == 2 ? up.z : up.w), ca[g]);
          lg[g] = live ? fmaf(v, __uint_as_float(g == 0 ? qs.x : g == 1 ? qs.y : g == 2 ? qs.z : qs.w), mask) : -INFINITY;
          asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(mx[g]) : "f"(lg[g]));
        }
        if (lane == 0) sts128(red + RED_MAX + par * 64 + w * 16, make_uint4(__float_as_uint(mx[0]), __float_as_uint(mx[1]), __float_as_uint(mx[2]), __float_as_uint(mx[3])));
        // the warp's largest products of a probability and a side, in logarithms
#pragma unroll
        for (int x = 0; x < NG; ++x) {
          const float a = lg2f(fabsf(rows[x].s));
          float m[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int g = 0; g < GQA; ++g) m[g] = warp_max_nan(lg[g] + a);
          if (lane == 0) sts128(red + RED_SV + par * 128 + w * 32 + x * 16, make_uint4(__float_as_uint(m[0]), __float_as_uint(m[1]), __float_as_uint(m[2]), __float_as_uint(m[3])));
        }
      }
      team_barrier(team);
      float most = ldsf(red + RED_SV + 128 * par + 4 * lane);         // lane l has group and head l mod 8
      if (pending) drain(i - 1);                                      // and its operands have been read
      // ================= softmax =================
      {
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint4 a = lds128(red + RED_MAX + par * 64 + k * 16);
          mx[0] = fmaxf(mx[0], __uint_as_float(a.x)); mx[1] = fmaxf(mx[1], __uint_as_float(a.y));
          mx[2] = fmaxf(mx[2], __uint_as_float(a.z)); mx[3] = fmaxf(mx[3], __uint_as_float(a.w));
        }
        const uint4 run = lds128(red + RED_RUN + 16 * (par ^ 1));
        const float before[4] = {__uint_as_float(run.x), __uint_as_float(run.y), __uint_as_float(run.z), __uint_as_float(run.w)};
#pragma unroll
        for (int g = 0; g < 4; ++g) mx[g] = fmaxf(mx[g], before[g]);
        // scale of the folds: the power of two above the largest product; the logits' own rounding (a logit of 2^20 has steps of 1/8) is
        // made up for
        most = max_nan(most, __shfl_xor_sync(0xffffffffu, most, 8));
        most = max_nan(most, __shfl_xor_sync(0xffffffffu, most, 16));
        const float high = fmaxf((lane & 2) ? ((lane & 1) ? mx[3] : mx[2]) : ((lane & 1) ? mx[1] : mx[0]), -3.0e38f);
        most = fmaf(fabsf(high), 2.4e-7f, most - high);
        const uint32_t ex = most < 200.0f ? (uint32_t)(min(max(__float2int_ru(most), -100), 128) + 126) : 255u;      // (a NaN has none)
        if (lane < 16) stsf(red + RED_VFOLD + 64 * w + 4 * lane, lane < 8 ? scale_down(ex) * C::FOLD_FULL : half_scale_up(ex) * (2.0f * C::UNIT));
        __syncwarp();
        if (r == 0) sts128(red + RED_RUN + 16 * par, make_uint4(__float_as_uint(mx[0]), __float_as_uint(mx[1]), __float_as_uint(mx[2]), __float_as_uint(mx[3])));
#pragma unroll
        for (int g = 0; g < GQA; ++g) {
          const float top = fmaxf(mx[g], -3.0e38f);                  // -inf as long as every token is masked: then the probabilities are 0
          const float c = ex2f(before[g] - top);
          lg[g] = ex2f(lg[g] - top);
          l_part[g] = fmaf(l_part[g], c, lg[g]);
          out[g] *= c;
          if (has_base && (lane & 3) == g) base_sum *= c;
        }
        // constant terms of the output (rows whose range does not straddle zero)
        has_base |= __any_sync(0xffffffffu, rows[0].A != 0.0f || (NG == 2 && rows[1].A != 0.0f));
        if (has_base) {
#pragma unroll
          for (int x = 0; x < NG; ++x)
#pragma unroll
            for (int g = 0; g < GQA; ++g) {
              float v = lg[g] * rows[x].A;
#pragma unroll
              for (int off = 1; off < 32; off <<= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
              if (lane == 4 * x + g) base_sum += v;
            }
        }
      }
      // ================= values: token `spot`, its two channel groups =================
      put_folds(lg, red + RED_VFOLD + 64 * w, NG);
      expand_row<BITS, P, NW>(code[0], rows[0], book, side + r * 16, two16);
      if (more) load_codes(0);
      if (NG == 2) {
        expand_row<BITS, P, NW>(code[1], rows[1], book, side + 8192 + r * 16, two16);
        if (more) load_codes(1);
      }
      proxy_fence();
      tm_fence_before();
      __syncwarp();
      if (lane == 0) bar_arrive(red + BAR_VREADY);
      pending = true;
      if (!more || nxt.pair != cur.pair) {
        drain(i);
        write_partial(par);
        ++seg;
        pending = false;
        if (more) start_pair(nxt);
      }
      cur = nxt;
    }
    }
  }
  tm_fence_before();
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm_base), "r"(C::TM_ALLOC));
}

template <int BITS, int P, int HD, int GQA, bool HALF_META>
int launch_one(const MzDecodeParams& p, cudaStream_t st) {
  auto kern = decode_umma_kernel<BITS, P, HD, GQA, HALF_META>;
  MZ_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BITS, P>::SMEM));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.hetero > 0 ? p.tp.ctas + p.tp2.ctas : p.tp.ctas));
  cfg.blockDim = dim3(Cfg<BITS, P>::THREADS);
  cfg.dynamicSmemBytes = Cfg<BITS, P>::SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MZ_CUDA(cudaLaunchKernelEx(&cfg, kern, p, 65536u));
  MZ_LAUNCH_CHECK("decode_umma");
  return MZ_OK;
}
template <int BITS, int P, int HD>
int launch_gqa(const MzDecodeParams& p, cudaStream_t st) {
  const bool half = p.s.meta_dtype == MZ_F16;
  switch (p.gqa) {
    case 1: return half ? launch_one<BITS, P, HD, 1, true>(p, st) : launch_one<BITS, P, HD, 1, false>(p, st);
    case 2: return half ? launch_one<BITS, P, HD, 2, true>(p, st) : launch_one<BITS, P, HD, 2, false>(p, st);
    case 4: return half ? launch_one<BITS, P, HD, 4, true>(p, st) : launch_one<BITS, P, HD, 4, false>(p, st);
  }
  return mz_fail(MZ_ERR_UNSUPPORTED, "gqa %d", p.gqa);
}
}  // namespace mzu

bool mz_decode_umma_supported(const MzDecodeParams& p) {
  return mz_decode_mma_supported(p) && (p.s.head_dim == 64 || p.s.head_dim == 128) && p.s.group == 64 && p.s.bits <= 4 &&
         (p.gqa == 1 || p.gqa == 2 || p.gqa == 4 || p.gqa == 8) && p.s.k_groups > 0;
}

// us of one residual tile in a CTA of residual tiles (12 warps, 3 us each; swept 0.20 .. 0.36: 64 x 8 pairs x 4224 tokens at 3 bits 215, 186, 186,
// 185, 187 us), and of a step of 128 packed tokens on an SM: [bits][planes]
constexpr float kDenseTileUs = 0.26f;
constexpr float step_us(int bits, int planes) { return bits == 1 ? 0.55f : planes == 2 ? 0.88f : bits < 4 ? 1.35f : 1.7f; }

namespace {
// even cut of `tiles` tiles per pair over W workers
int cut(MzTilesPlan& t, long long pairs, int tiles, long long W) {
  t = MzTilesPlan{};
  t.kind = 2;
  t.tiles_per_pair = tiles;
  // in 64ths of a tile, so that the merge kernel finds a pair's workers within a narrow range (it divides by the whole units per worker)
  t.cost_q = t.cost_d = 64;
  t.pair_cost = 64LL * tiles;
  t.total_tiles = pairs * tiles;
  t.total_cost = pairs * t.pair_cost;
  if (t.total_cost >= (1LL << 31)) return mz_fail(MZ_ERR_UNSUPPORTED, "cache too large for the tiled kernel");
  if (W > t.total_tiles) W = t.total_tiles;
  if (W < 1) W = 1;
  if (W > (1LL << 30)) return mz_fail(MZ_ERR_ARG, "too many splits");
  t.total_warps = (int)W;
  t.cost_quot = (unsigned)(t.total_cost / W);
  t.cost_rem = (unsigned)(t.total_cost % W);
  const long long len = t.total_cost / W + 2;
  t.max_segs = (int)((len - 1) / t.pair_cost + 2);
  return MZ_OK;
}
}  // namespace

// One launch over two plans: the packed tiles (p.tp, workers = warp groups, tiles = steps of 128 tokens) and, when there is a residual
// window, its tiles on CTAs of their own (p.tp2, workers = warps); the records of the second plan follow those of the first.
int mz_plan_umma(MzDecodeParams& p, bool full_precision, int splits_request, int sm_count, size_t* slots) {
  const mz_kv_store& s = p.s;
  if (p.gqa == 8) {       // eight heads are two times four, each with the kv head to itself
    p.gqa = 4;
    p.s.kv_heads *= 2;
    p.kv_share = 1;
  }
  p.planes = s.bits == 1 ? 1 : s.bits == 2 && s.head_dim == 128 && !full_precision ? 2 : 3;
  const int workers = p.planes == 3 ? mzu::Cfg<3, 3>::WORKERS : mzu::Cfg<2, 2>::WORKERS;
  const int steps = (s.k_groups + mzu::STEP_GROUPS - 1) / mzu::STEP_GROUPS;
  const long long pairs = (long long)s.batch * s.kv_heads;
  const int dense_tiles = (s.res_len + mzd::DT - 1) / mzd::DT;
  int n_d = 0;
  if (dense_tiles > 0) {
    const float dense = (float)dense_tiles * kDenseTileUs, packed = (float)steps * step_us(s.bits, p.planes) * (s.head_dim == 64 ? 0.6f : 1.0f);
    n_d = (int)((float)sm_count * dense / (dense + packed) + 0.5f);
    if (n_d < 1) n_d = 1;
    if (n_d > sm_count / 2) n_d = sm_count / 2;
  }
  p.cluster = 0;
  p.hetero = 0;
  p.fail_waits = mzu::g_fail_waits.load(std::memory_order_relaxed);
  int rc = cut(p.tp, pairs, steps, splits_request > 0 ? pairs * splits_request : (long long)(sm_count - n_d) * workers);
  if (rc) return rc;
  p.tp.packed_tiles = steps;
  p.tp.ctas = (p.tp.total_warps + workers - 1) / workers;
  *slots = (size_t)p.tp.total_warps * p.tp.max_segs * p.gqa;
  p.slots_a = (long long)*slots;
  p.tp2 = MzTilesPlan{};
  if (dense_tiles > 0) {
    if ((rc = cut(p.tp2, pairs, dense_tiles, splits_request > 0 ? pairs * splits_request : (long long)n_d * mzu::DENSE_WARPS))) return rc;
    p.tp2.ctas = (p.tp2.total_warps + mzu::DENSE_WARPS - 1) / mzu::DENSE_WARPS;
    p.hetero = p.tp.ctas;
    *slots += (size_t)p.tp2.total_warps * p.tp2.max_segs * p.gqa;
  }
  return MZ_OK;
}

int mz_launch_decode_umma(const MzDecodeParams& p, cudaStream_t st) {
  const int which = p.s.bits * 16 + p.planes;
  if (p.s.head_dim == 64) {
    switch (which) {
      case 0x11: return mzu::launch_gqa<1, 1, 64>(p, st);
      case 0x23: return mzu::launch_gqa<2, 3, 64>(p, st);
      case 0x33: return mzu::launch_gqa<3, 3, 64>(p, st);
      case 0x43: return mzu::launch_gqa<4, 3, 64>(p, st);
    }
  } else {
    switch (which) {
      case 0x11: return mzu::launch_gqa<1, 1, 128>(p, st);
      case 0x22: return mzu::launch_gqa<2, 2, 128>(p, st);
      case 0x23: return mzu::launch_gqa<2, 3, 128>(p, st);
      case 0x33: return mzu::launch_gqa<3, 3, 128>(p, st);
      case 0x43: return mzu::launch_gqa<4, 3, 128>(p, st);
    }
  }
  return mz_fail(MZ_ERR_UNSUPPORTED, "bits %d, %d planes", p.s.bits, p.planes);
}

extern "C" int mz_debug_fail_waits(int on) {
#ifdef MZ_BOUNDS
  return mzu::g_fail_waits.exchange(on != 0);
#else
  (void)on;
  return -1;
#endif
}
