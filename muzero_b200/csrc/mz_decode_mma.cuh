// Tensor-core decode attention for head_dim 64 / 128, groups of 32 / 64 / 128, 1..8-bit codes, up to 8 query heads per
// kv head (sm_100a).
//
// The dequantized value of code e in a row with metadata (lo, span) is
//     A + Bup * u+[zc][e] + Bdn * u-[zc][e]
// where zc is the row's zero code, A / Bup / Bdn are per-row constants and u+ / u- are the positive
// and negative part of ONE normalised table that depends on (zc, e) only.  Key rows run along the
// tokens and value rows along the channels, i.e. always along the dimension a contraction does NOT
// reduce over, so the per-row constants can be folded into the other operand:
//     logit[h,t]  = sum_d  (q[h,d]*Bup_d) u+  +  (q[h,d]*Bdn_d) u-   + sum_d q[h,d] A_d
//     out[h,c]    = sum_t  (p[h,t]*Bup_tg) u+ +  (p[h,t]*Bdn_tg) u-  + sum_t p[h,t] A_tg
// Both contractions run on the tensor cores (mma.sync m16n8k16, fp16 operands, fp32 accumulate):
//   * the A operand holds table values; one code = a 64-bit shared-memory lookup that returns the fp16 pair (u+, u-),
//     which is one A-fragment register (the reduction index is doubled: one slot for the part above the zero code, one
//     for the part below it), and the pair of what rounding to fp16 dropped
//   * the table is replicated once per lane of a half warp, so no lookup pattern can cause a bank conflict, and it sits
//     at shared-window address 65536 with a stride of 256 bytes, so that the address of a lookup is one byte
//     permute: byte 1 of the address <- (zc, code)
//   * the B operand holds the folded query (keys) or folded probabilities (values); its 8 columns are
//     4 heads x {product rounded to fp16, its exact fp16 remainder (+ the remainders of the constant and of the
//     probability)};
//     5 to 8 heads per kv head use a second set of 8 columns on the same A fragments
//   * a second product takes the fp16 remainders of the table values (the upper half of the 64-bit entry).  With constants,
//     query products and probabilities as value + remainder too, and the running sums kept outside the tensor cores, the
//     result has the error of the fp32 kernels (a few 1e-7)
//   * M rows are tokens (keys) or channels (values), permuted so that one load of packed codes
//     feeds a thread's rows of all M tiles.
// Codes of 5 to 8 bits have no table (2^16 entries): their value (v - A) / span is computed per code (one ex2) and
// enters as an fp16 pair value + remainder, two MMAs over 16 rows instead of one over 8 doubled ones.
// Residual (un-quantized) tiles of 16 tokens use fragments of the cache's own 16-bit type.
//
// Work: tiles of G packed tokens or 16 residual tokens of one (batch, kv head) pair.  Either the flat list of all
// tiles is cut by cost into one contiguous range per warp of a machine-filling grid and a merge kernel combines the
// partial records, or (few pairs) a cluster of CTAs owns a pair and merges through distributed shared memory.
// Measured (8 kv heads, call included): one sequence of 500 tokens, 4 bits 27.8 us as cut + merge on the unrolled kernel, 14.5 us
// here; 6 x 1777 with 8 heads per kv head under a mask 43.0 us on the SIMT kernel, 38.1 us here (and 32.8 on the tcgen05
// kernel, which has that call now); head_dim 64, 16 x 2050 333 us on the
// shape-generic kernel, 23.8 us here.  Without the second product (error 1e-5 instead of 5e-7): 13.8, 32.7 and 19.9 us.
// Bound by the latency of a tile's chain: no unit is busy (issue 30 to 51 %, shared-memory pipe 17 to 39 %).
#pragma once
#include <type_traits>

#include "mz_mma_common.cuh"

namespace mzm {
constexpr int DT = 16;                      // tokens per residual tile
constexpr uint32_t WIDE_ROW = 32;           // row constants of a wide code: 8 words
// Operands are kept away from fp16's subnormals (2^-24) and its largest value (65504): the query's largest element is
// scaled by a power of two into [64, 128), the largest range among the rows of a tile (of each value group) into
// [128, 256), probabilities by 128.  Products stay below 2^15, and what a remainder can lose is 2^-40 of the largest
// product.  The powers of two are taken back in the fp32 sums.
constexpr float P_SCALE = 128.0f;

// BITS: 1..4 and 8, or 0 for 5..7 (code width at run time)
template <int BITS, int D_, int G_, int NT_>
struct Cfg {
  static constexpr bool WIDE = BITS == 0 || BITS > 4;
  static constexpr int D = D_, G = G_, NT = NT_;
  static constexpr int NG = D / G;            // value groups of a token
  static constexpr int CPL = G / 8;           // consecutive positions of a row per lane
  static constexpr int MT = G / 16;           // M tiles along a row
  static constexpr int NB = D / 8;            // reduction blocks of 8 rows per tile side (both sides have D rows)
  static constexpr int MAXW = NT == 1 ? 12 : 8;
  static constexpr int NE = 1 << (WIDE ? 1 : BITS);
  // table: entries (zero code, code) in 256-byte slots, keys' copies in the lower, values' in the upper half
  static constexpr int ENTRIES = WIDE ? 0 : NE * NE;
  static constexpr uint32_t TABLE_BYTES = ENTRIES * 256u;
  // row constants, and the folded-query source (the block loops are not unrolled over it)
  static constexpr uint32_t Q_BYTES = NT * NB * 64;
  static constexpr uint32_t RI_BYTES = D * (WIDE ? WIDE_ROW : 10) + Q_BYTES;       // table path: constants (8), zero-code byte, padding
  static constexpr uint32_t A_BYTES = D * 4;
  static constexpr uint32_t P_BYTES = G * 16 * NT;             // probabilities: [G/8][4 x 8 NT] half2
};
struct Layout { uint32_t kbuf, vbuf, ri, a, pbuf, q; };

// One B-operand register of a lane: x * B for the pair B = (Bup, Bdn).  mask = 0 (even column): the fp16
// product; mask = all ones (odd column): what that rounding dropped, exactly.
// `lo` is the remainder of the constants, `xm` = x in the odd columns, else 0.
__device__ __forceinline__ uint32_t fold_pair(__half2 x, __half2 xm, uint32_t B, uint32_t lo, uint32_t mask) {
  const uint32_t h = h2_bits(__hmul2(x, bits_h2(B))) & mask;
  return h2_bits(__hfma2(xm, bits_h2(lo), __hfma2(x, bits_h2(B), __hneg2(bits_h2(h)))));
}

// table lookups: the table never changes after the fill, so the compiler may move them freely
__device__ __forceinline__ uint2 tab64(uint32_t a) {
  uint2 v;
  asm("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t pack_u16(uint32_t lo, uint32_t hi) { return prmt(lo, hi, 0x5410u); }

// ---- lookups.  A thread (g = lane / 4, t = lane % 4) holds, per reduction block, the codes of two rows (slot 0 and 1)
// for the CPL consecutive positions CPL*g + i along the row; position i belongs to M tile i / 2, fragment row
// g + 8 * (i & 1).  `row0` / `row1` are the shared addresses of the lane's first code byte in the two rows.  Codes are
// loaded a quad of M tiles at a time (8 positions; 4 when the group is 32) and looked up half a quad at a time: half h
// has the positions 4 h + i, a[4 (i / 2) + 2 slot + (i & 1)].
template <int BITS, int CPL>
struct Quad;
// 4-bit codes: 8 positions = one word
template <int CPL>
struct Quad<4, CPL> {
  uint32_t w0, w1;
  __device__ __forceinline__ void load(uint32_t row0, uint32_t row1, int q) {
    if (CPL == 4) { w0 = lds16(row0); w1 = lds16(row1); }
    else { w0 = lds32(row0 + 4 * q); w1 = lds32(row1 + 4 * q); }
  }
  __device__ __forceinline__ void look(int h, uint32_t z0, uint32_t z1, uint32_t base, uint2 (&a)[8]) const {
    const uint32_t c[4] = {(w0 & 0x0F0F0F0Fu) | z0, ((w0 >> 4) & 0x0F0F0F0Fu) | z0, (w1 & 0x0F0F0F0Fu) | z1, ((w1 >> 4) & 0x0F0F0F0Fu) | z1};
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int k = 0; k < 4; ++k) a[4 * m + k] = tab64(prmt(c[k], base, 0x7604u | (uint32_t)((2 * h + m) << 4)));
  }
};
// 3-bit codes: 8 positions = 24 bits at any bit address
template <int CPL>
struct Quad<3, CPL> {
  uint32_t w0, w1;
  static __device__ __forceinline__ uint32_t fetch(uint32_t row, uint32_t bit) {
    // two words of the row (the second may lie past its end, still inside the staged tile)
    const uint32_t at = row + (bit >> 5) * 4;
    return __funnelshift_r(lds32(at), lds32(at + 4), bit & 31);
  }
  __device__ __forceinline__ void load(uint32_t row0, uint32_t row1, int q, int g) {
    const uint32_t bit = (uint32_t)(g * CPL + 8 * q) * 3;
    w0 = fetch(row0, bit); w1 = fetch(row1, bit);
  }
  // four 3-bit codes -> four bytes
  static __device__ __forceinline__ uint32_t spread(uint32_t x) {
    x = (x | (x << 10)) & 0x003F003Fu;
    return (x | (x << 5)) & 0x07070707u;
  }
  __device__ __forceinline__ void look(int h, uint32_t z0, uint32_t z1, uint32_t base, uint2 (&a)[8]) const {
    const uint32_t c0 = spread((w0 >> (12 * h)) & 0xfffu) | z0, c1 = spread((w1 >> (12 * h)) & 0xfffu) | z1;
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        a[4 * m + r] = tab64(prmt(c0, base, 0x7604u | (uint32_t)((2 * m + r) << 4)));
        a[4 * m + 2 + r] = tab64(prmt(c1, base, 0x7604u | (uint32_t)((2 * m + r) << 4)));
      }
  }
};
// 2-bit codes: 8 positions = 16 bits; byte 2 slot + h of c is position 4 h + k
template <int CPL>
struct Quad<2, CPL> {
  uint32_t w;                 // low half: slot 0, high half: slot 1
  __device__ __forceinline__ void load(uint32_t row0, uint32_t row1, int q) {
    if (CPL == 4) w = pack_u16(lds8(row0), lds8(row1));
    else w = pack_u16(lds16(row0 + 2 * q), lds16(row1 + 2 * q));
  }
  __device__ __forceinline__ void look(int h, uint32_t z0, uint32_t z1, uint32_t base, uint2 (&a)[8]) const {
    const uint32_t z = pack_u16(z0, z1);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t c = ((w >> (2 * k)) & 0x03030303u) | z;
#pragma unroll
      for (int slot = 0; slot < 2; ++slot) a[4 * (k >> 1) + 2 * slot + (k & 1)] = tab64(prmt(c, base, 0x7604u | (uint32_t)((2 * slot + h) << 4)));
    }
  }
};
// 1-bit codes: 8 positions = one byte, spread like the 2-bit ones
template <int CPL>
struct Quad<1, CPL> {
  uint32_t w;                 // bytes: slot 0 positions 0.., 4.., slot 1 positions 0.., 4..
  __device__ __forceinline__ void load(uint32_t row0, uint32_t row1, int q, int g = 0) {
    const uint32_t sh = CPL == 4 ? 4 * (g & 1) : 0, b0 = lds8(row0 + q) >> sh, b1 = lds8(row1 + q) >> sh, b = pack_u16(b0, b1);
    w = prmt(b, b >> 4, 0x6240u);
  }
  __device__ __forceinline__ void look(int h, uint32_t z0, uint32_t z1, uint32_t base, uint2 (&a)[8]) const {
    const uint32_t z = pack_u16(z0, z1);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t c = ((w >> k) & 0x01010101u) | z;
#pragma unroll
      for (int slot = 0; slot < 2; ++slot) a[4 * (k >> 1) + 2 * slot + (k & 1)] = tab64(prmt(c, base, 0x7604u | (uint32_t)((2 * slot + h) << 4)));
    }
  }
};

// byte offset of lane row-position g inside a packed row (the part handled by Quad itself excepted)
template <int BITS, int CPL>
__device__ __forceinline__ uint32_t lane_offset(int g) {
  if (BITS == 3) return 0;                                   // addressed by Quad
  if (BITS == 1 && CPL == 4) return g >> 1;
  return (uint32_t)(g * (CPL * BITS)) >> 3;
}

// the table values of half a quad; zz: zero-code bytes of slot 0 and 1
template <class Q>
__device__ __forceinline__ void look_step(const Q& w, int h, uint32_t zz, uint32_t base, uint2 (&a)[8]) {
  w.look(h, prmt(zz, 0u, 0x0000u), prmt(zz, 0u, 0x1111u), base, a);
}

// One step's product with M tile `m` of half a quad, added to c: the remainders first, then the rounded values, on a
// fresh accumulator, so that the running sum is rounded to nearest.  The tensor cores truncate theirs: with the keys' sums left
// on them the error against 64 bits is 2.0e-6 instead of 4.5e-7 (4 bits, head_dim 128), for 0 to 3 % of the time.
template <bool SCALED = false>
__device__ __forceinline__ void mma_step(float (&c)[4], const uint2 (&a)[8], int m, uint32_t b0, uint32_t b1, float unit = 1.0f) {
  float x[4];
  mma_f16_first(x, a[4 * m].y, a[4 * m + 1].y, a[4 * m + 2].y, a[4 * m + 3].y, b0, b1);
  mma_f16(x, a[4 * m].x, a[4 * m + 1].x, a[4 * m + 2].x, a[4 * m + 3].x, b0, b1);
  if (SCALED) fma4(c, x, unit);
  else add4(c, x);
}

// ---- the lookup table, from the entries [2][ENTRIES] = (keys' alpha, values' alpha) in global memory (nullptr: they
// are computed here).  A thread takes whole entries: the loads of up to four are in flight together (one by one their
// latency was most of a small call), then 16-byte stores of the copies, rotated so that eight neighbouring threads hit
// eight different bank groups.
template <class C, int BITS>
__device__ __forceinline__ void fill_tables(uint32_t table, const uint2* __restrict__ lut, float alpha_key, float alpha_value) {
  constexpr int PER = C::ENTRIES, CHUNKS = 8;
  const int n = alpha_key == alpha_value ? PER : 2 * PER;        // equal alphas: one table, in the lower halves
  for (int i0 = threadIdx.x; i0 < n; i0 += 4 * blockDim.x) {
    uint2 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = min(i0 + k * (int)blockDim.x, n - 1);
      v[k] = lut != nullptr ? lut[i] : split_entry<BITS>(i / PER ? alpha_value : alpha_key, i % PER);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = i0 + k * blockDim.x, which = i / PER, idx = i % PER;
      if (i < n) {
        const uint32_t row = table + idx * 256 + which * 128;
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) sts128(row + (((c + threadIdx.x) & (CHUNKS - 1)) << 4), make_uint4(v[k].x, v[k].y, v[k].x, v[k].y));
      }
    }
  }
}

// ---- wide codes: (v - A) / span of code e.  Row constants {zc, kup, kdn, cup, cdn}: above the zero code
// cup * (2^(n kup) - 1), below it cdn * (2^(n kdn) - 1) with n = |e - zc| and cdn < 0.
struct WideRow { float zc, kup, kdn, cup, cdn; };        // zc: 2^23 + zero code
// f: 2^23 + code
__device__ __forceinline__ float wide_value(float f, const WideRow& r) {
  const float n = f - r.zc;
  const bool up = n >= 0.0f;
  const float x = ex2f(fabsf(n) * (up ? r.kup : r.kdn));
  return (x - 1.0f) * (up ? r.cup : r.cdn);
}
// two values as fp16 pairs: rounded, and what the rounding dropped
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(a, b);
  const float2 f = __half22float2(h);
  hi = h2_bits(h);
  lo = h2_bits(__floats2half2_rn(a - f.x, b - f.y));
}
// One tile side of wide codes: blocks of 16 rows, a lane holds rows 4 s + t (s = 0..3).  INNER consecutive blocks are
// unrolled (the value groups of a token block).  row(blk, s): byte offset of the row; fold(blk, spans, b): the B operand;
// mma(k, m, hi, lo, b): multiply M tile m of inner block k.
template <class C, int BITS, int INNER, class RowF, class FoldF, class MmaF>
__device__ __forceinline__ void wide_side(uint32_t buf, uint32_t ri, int g, int t, int bits, RowF row, FoldF fold, MmaF mma) {
  constexpr int PER = C::CPL < 8 ? C::CPL : 8;          // codes of a row taken at once
#pragma unroll 1
  for (int j = 0; j < C::NB / 2 / INNER; ++j) {
#pragma unroll
    for (int k = 0; k < INNER; ++k) {
      const int blk = j * INNER + k;
      WideRow r[4];
      uint32_t sp[4], at[4];
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const uint4 c0 = lds128(ri + (blk * 4 + s) * 128 + t * 16), c1 = lds128(ri + (blk * 4 + s) * 128 + 64 + t * 16);
        r[s] = {__uint_as_float(c0.x), __uint_as_float(c0.y), __uint_as_float(c0.z), __uint_as_float(c0.w), __uint_as_float(c1.x)};
        sp[s] = c1.y;
        at[s] = buf + row(blk, s);
      }
      uint32_t bb[C::NT][2];
      fold(blk, sp, bb);
#pragma unroll
      for (int q = 0; q < C::CPL / PER; ++q) {
        uint2 w[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          if (BITS == 8) {
            if (PER == 8) w[s] = lds64(at[s] + g * C::CPL + 8 * q);
            else w[s] = make_uint2(lds32(at[s] + g * C::CPL), 0u);
          } else {
            const uint32_t bit = (uint32_t)(g * C::CPL + 8 * q) * bits, ad = at[s] + (bit >> 5) * 4;
            const uint32_t x0 = lds32(ad), x1 = lds32(ad + 4), x2 = lds32(ad + 8);
            w[s] = make_uint2(__funnelshift_r(x0, x1, bit & 31), __funnelshift_r(x1, x2, bit & 31));
          }
        }
#pragma unroll
        for (int m = 0; m < PER / 2; ++m) {
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int rr = 0; rr < 2; ++rr) {
            const int i = 2 * m + rr;
            float v[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              uint32_t e;
              if (BITS == 8) e = prmt(i < 4 ? w[s].x : w[s].y, 0x4B000000u, 0x7440u | (uint32_t)(i & 3));
              else e = ((uint32_t)((((unsigned long long)w[s].y << 32) | w[s].x) >> (i * bits)) & ((1u << bits) - 1u)) | 0x4B000000u;
              v[s] = wide_value(__uint_as_float(e), r[s]);
            }
            split_pair(v[0], v[1], hi[rr], lo[rr]);
            split_pair(v[2], v[3], hi[2 + rr], lo[2 + rr]);
          }
          mma(k, q * (PER / 2) + m, hi, lo, bb);
        }
      }
    }
  }
}

// ---- a residual tile: up to 16 un-quantized tokens, staged in shared memory as rows of 2 D bytes whose 16-byte chunks are
// swizzled by the row (keys: chunk ^ 4 (row & 1), values: chunk ^ (row & 6)) so that the fragment loads below have no bank
// conflicts.  The reduction order of the keys is permuted (lane t takes channels 32 i + 8 t .. + 7) so that every load
// is 16 bytes; values are loaded by (token, channel) and paired over tokens by byte permutes.
// The newest token may still be in the caller's tensors (p.new_k / new_v): it is staged from there, and stored into the
// window by the warp that works on its tile.
template <class C>
__device__ __forceinline__ void stage_dense(const MzDecodeParams& p, uint32_t dst, bool values, int b, int kvh, int dt, int lane) {
  constexpr int CH = C::D / 8;
  const mz_kv_store& s = p.s;
  const int tok0 = dt * DT, ntok = min(DT, s.res_len - tok0);
  const int fresh = p.new_k != nullptr ? s.res_len - 1 - tok0 : -1;
  const uint16_t* src = (const uint16_t*)(values ? s.res_v : s.res_k) + b * s.res_stride_b + kvh * s.res_stride_h +
                        (long long)(s.res_start + tok0) * s.res_stride_t;
  const uint16_t* fresh_row = (const uint16_t*)(values ? p.new_v : p.new_k) + b * p.new_sb + kvh * p.new_sh;
#pragma unroll
  for (int i = lane; i < DT * CH; i += 32) {
    const int row = i / CH, c = i % CH;
    const uint32_t at = dst + row * (2 * C::D) + ((c ^ (values ? row & 6 : (row & 1) << 2)) << 4);
    // rows past the end are zeroed (they are multiplied by probability 0, which must not meet a NaN bit pattern)
    if (row < ntok) cp16(at, (row == fresh ? fresh_row : src + (long long)row * s.res_stride_t) + c * 8);
    else sts128(at, make_uint4(0, 0, 0, 0));
  }
}
template <class C, class SoftmaxF, class KeysDoneF, class ValuesReadyF>
__device__ __forceinline__ void dense_tile(const MzDecodeParams& p, uint32_t kbuf, uint32_t vbuf, int dt, int b, int kvh, int g, int t, int hq,
                                           bool bf, long long mask0, const uint16_t* q0, float (&out)[C::NT][C::D / 16][4],
                                           SoftmaxF& softmax_update, KeysDoneF keys_done, ValuesReadyF values_ready) {
  constexpr int D = C::D, NT = C::NT, NG = C::NG, CPL = C::CPL, MT = C::MT;
  const mz_kv_store& s = p.s;
  const int tok0 = dt * DT, ntok = min(DT, s.res_len - tok0), gqa = p.gqa;
  const int fresh = p.new_k != nullptr ? s.res_len - 1 - tok0 : -1;      // row of the token that is not in the window yet
  uint16_t* rk = (uint16_t*)s.res_k + b * s.res_stride_b + kvh * s.res_stride_h + (long long)(s.res_start + tok0) * s.res_stride_t;
  uint16_t* rv = (uint16_t*)s.res_v + (rk - (uint16_t*)s.res_k);
  uint4 kx[2][D / 32];
#pragma unroll
  for (int r = 0; r < 2; ++r)
#pragma unroll
    for (int i = 0; i < D / 32; ++i) kx[r][i] = lds128(kbuf + (g + 8 * r) * (2 * D) + (((4 * i + t) ^ ((g & 1) << 2)) << 4));
  if (fresh >= 0 && fresh < DT) {
#pragma unroll
    for (int r = 0; r < 2; ++r)
      if (g + 8 * r == fresh && MZ_IN_BOUNDS(s.res_start + tok0 + fresh, p.new_rows, 15)) {
#pragma unroll
        for (int i = 0; i < D / 32; ++i) *(uint4*)(rk + (g + 8 * r) * s.res_stride_t + 32 * i + 8 * t) = kx[r][i];
      }
  }
  warp_sync();                    // every lane has its keys
  keys_done();
  float sv[NT][2];
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    const int h = 4 * n + hq;
    const bool mine = (g & 1) == 0 && h < gqa;
    const uint16_t* qrow = q0 + min(h, gqa - 1) * p.q_stride_h + 8 * t;
    float dacc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    uint32_t qx[D / 32][4];
#pragma unroll
    for (int i = 0; i < D / 32; ++i)
#pragma unroll
      for (int k = 0; k < 4; ++k) qx[i][k] = mine ? *(const uint32_t*)(qrow + 32 * i + 2 * k) : 0u;
#pragma unroll
    for (int i = 0; i < D / 32; ++i) {
      const uint4 lo = kx[0][i], hi = kx[1][i];
      if (bf) {
        mma_bf16(dacc[0], lo.x, hi.x, lo.y, hi.y, qx[i][0], qx[i][1]);
        mma_bf16(dacc[1], lo.z, hi.z, lo.w, hi.w, qx[i][2], qx[i][3]);
      } else {
        mma_f16(dacc[0], lo.x, hi.x, lo.y, hi.y, qx[i][0], qx[i][1]);
        mma_f16(dacc[1], lo.z, hi.z, lo.w, hi.w, qx[i][2], qx[i][3]);
      }
    }
    // this lane: head 4 n + t, tokens g and g + 8
    const float sc = p.scaling * LOG2E;
    sv[n][0] = (dacc[0][0] + dacc[1][0]) * sc;
    sv[n][1] = (dacc[0][2] + dacc[1][2]) * sc;
    if (p.mask) {
      if (g < ntok) sv[n][0] += mz_load_as_float(p.mask, mask0 + g, p.mask_dtype) * LOG2E;
      if (g + 8 < ntok) sv[n][1] += mz_load_as_float(p.mask, mask0 + g + 8, p.mask_dtype) * LOG2E;
    }
    if (g >= ntok) sv[n][0] = -INFINITY;
    if (g + 8 >= ntok) sv[n][1] = -INFINITY;
    softmax_update(n, sv[n]);
  }
  values_ready();
  uint32_t vx[4][NG * MT];       // channel pairs of tokens 2t, 2t + 1, 2t + 8, 2t + 9
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int row = 2 * t + (k & 1) + 8 * (k >> 1);
#pragma unroll
    for (int n = 0; n < NG; ++n) {
      const uint32_t off = (n * C::G + CPL * g) * 2;           // byte offset inside the row
      if (CPL == 4) {
        const uint2 v = lds64(vbuf + row * (2 * D) + (((off >> 4) ^ (row & 6)) << 4) + (off & 8));
        vx[k][n * MT] = v.x; vx[k][(n * MT + 1) % (NG * MT)] = v.y;
      } else {
#pragma unroll
        for (int c = 0; c < CPL / 8; ++c) {
          const uint4 v = lds128(vbuf + row * (2 * D) + ((((off >> 4) + c) ^ (row & 6)) << 4));
          vx[k][n * MT + 4 * c] = v.x; vx[k][(n * MT + 4 * c + 1) % (NG * MT)] = v.y;
          vx[k][(n * MT + 4 * c + 2) % (NG * MT)] = v.z; vx[k][(n * MT + 4 * c + 3) % (NG * MT)] = v.w;
        }
      }
    }
    if (row == fresh && MZ_IN_BOUNDS(s.res_start + tok0 + fresh, p.new_rows, 16)) {
#pragma unroll
      for (int n = 0; n < NG; ++n)
#pragma unroll
        for (int m = 0; m < MT; ++m) *(uint32_t*)(rv + row * s.res_stride_t + n * C::G + CPL * g + 2 * m) = vx[k][n * MT + m];
    }
  }
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    // B operand: probabilities of head 4 n + hq, split into the 16-bit value (even columns) and its remainder; bf16 pairs
    // leave a third part of 8 bits, which goes through a product of its own
    uint32_t bb[2], b3[2];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float pv[2], rest[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float pf = P_SCALE * __shfl_sync(0xffffffffu, sv[n][half], 4 * (2 * t + k) + hq);
        const float hi = bf ? __bfloat162float(__float2bfloat16_rn(pf)) : __half2float(__float2half_rn(pf));
        pv[k] = (g & 1) ? pf - hi : hi;
        rest[k] = (g & 1) ? pv[k] - __bfloat162float(__float2bfloat16_rn(pv[k])) : 0.f;
      }
      if (bf) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(pv[0], pv[1]), r = __floats2bfloat162_rn(rest[0], rest[1]);
        bb[half] = *reinterpret_cast<const uint32_t*>(&v);
        b3[half] = *reinterpret_cast<const uint32_t*>(&r);
      } else {
        bb[half] = h2_bits(__floats2half2_rn(pv[0], pv[1]));
      }
    }
#pragma unroll
    for (int m = 0; m < NG * MT; ++m) {
      // rows g / g+8 = channels 2m / 2m+1 of the lane's; columns = tokens (2t, 2t+1) and (2t+8, 2t+9)
      const uint32_t a0 = prmt(vx[0][m], vx[1][m], 0x5410u), a1 = prmt(vx[0][m], vx[1][m], 0x7632u);
      const uint32_t a2 = prmt(vx[2][m], vx[3][m], 0x5410u), a3 = prmt(vx[2][m], vx[3][m], 0x7632u);
      float x[4];
      if (bf) {
        mma_bf16_first(x, a0, a1, a2, a3, b3[0], b3[1]);
        mma_bf16(x, a0, a1, a2, a3, bb[0], bb[1]);
      } else {
        mma_f16_first(x, a0, a1, a2, a3, bb[0], bb[1]);
      }
      fma4(out[n][m], x, 1.0f / P_SCALE);
    }
  }
}

// ---- cluster mode: the warps' states become records {acc[D], m, l} per head in shared memory, each CTA merges its own,
// and CTA `rank` writes its share of the pair's outputs from the records of all CTAs (distributed shared memory).
__device__ __forceinline__ uint32_t remote(uint32_t addr, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float2 ld_remote2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_remote4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float4 lds4f(uint32_t a) {
  const uint4 v = lds128(a);
  return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
__device__ __forceinline__ float2 lds2f(uint32_t a) {
  const uint2 v = lds64(a);
  return make_float2(__uint_as_float(v.x), __uint_as_float(v.y));
}
// every thread of the cluster; the lanes of a warp may come out of a divergent loop, so not the .aligned form (a warp that
// is not converged there is an illegal instruction)
__device__ __forceinline__ void cluster_sync() {
  __syncthreads();
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
template <class C, class ReduceF>
__device__ __forceinline__ void finish_cluster(const MzDecodeParams& p, uint32_t window, int rank, int nw, int warp, int lane, int g, int t, bool active,
                                               const float (&out)[C::NT][C::D / 16][4], const float (&m_st)[C::NT], ReduceF& reduce_state) {
  constexpr int D = C::D, NG = C::NG, CPL = C::CPL, MT = C::MT;
  constexpr int REC = (D + 4) * 4;              // bytes of one head's record
  const int gqa = p.gqa, cs = p.cluster;
  const MzTilesPlan& tp = p.tp;
  const uint32_t per_high = tp.stage_bytes + C::RI_BYTES + C::A_BYTES + C::P_BYTES;
  const uint32_t low = window + tp.low_base, high = window + tp.high_base, mine = high + warp * per_high;
  __syncthreads();                              // every warp is done with its buffers
#pragma unroll
  for (int n = 0; n < C::NT; ++n) {
    float lsum, bv[NG];
    reduce_state(n, lsum, bv);
    const int h = 4 * n + t;
    if (h < gqa) {
      const uint32_t dst = mine + h * REC + CPL * g * 4;
#pragma unroll
      for (int k = 0; k < NG; ++k)
#pragma unroll
        for (int m = 0; m < MT; m += 2) {
          const float(&x)[4] = out[n][k * MT + m];
          const float(&y)[4] = out[n][k * MT + m + 1];
          sts128(dst + (k * C::G + 2 * m) * 4, make_uint4(__float_as_uint(x[0] + x[1] + bv[k]), __float_as_uint(x[2] + x[3] + bv[k]),
                                                         __float_as_uint(y[0] + y[1] + bv[k]), __float_as_uint(y[2] + y[3] + bv[k])));
        }
      if (g == 0) {
        stsf(mine + h * REC + D * 4, active ? m_st[n] : -INFINITY);
        stsf(mine + h * REC + D * 4 + 4, lsum);
      }
    }
  }
  __syncthreads();
  const int pair = (int)blockIdx.x / cs;
  const int total = gqa * D;
  // merges the records 0 .. n-1 (at most N) of four neighbouring elements of a head; base-2 maxima.  All maxima, then all
  // accumulators are in flight together.
  auto merge = [&](auto nmax, int n, auto&& ml, auto&& acc, float& mx, float& lsum, float4& a) {
    constexpr int N = decltype(nmax)::value;
    float2 v[N];
    mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = i < n ? ml(i) : make_float2(-INFINITY, 0.f);
#pragma unroll
    for (int i = 0; i < N; ++i) mx = fmaxf(mx, v[i].x);
    lsum = 0.f;
    a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      if (i < n) {
        const float w = v[i].x > -INFINITY ? ex2f(v[i].x - mx) : 0.f;
        const float4 x = acc(i);
        lsum = fmaf(v[i].y, w, lsum);
        a.x = fmaf(x.x, w, a.x); a.y = fmaf(x.y, w, a.y); a.z = fmaf(x.z, w, a.z); a.w = fmaf(x.w, w, a.w);
      }
    }
  };
  auto write_out = [&](int h, int d, float mx, float lsum, float4 a) {
    const long long row = (long long)pair * gqa + h;
    const MzDecodeOut& o = p.o;
    if (!MZ_IN_BOUNDS(row, (long long)p.s.batch * p.H, 17)) return;
    if (o.out) {
      const float den = fmaxf(lsum, 1e-20f);
      mz_store_from_float(o.out, row * D + d, a.x / den, o.out_dt);
      mz_store_from_float(o.out, row * D + d + 1, a.y / den, o.out_dt);
      mz_store_from_float(o.out, row * D + d + 2, a.z / den, o.out_dt);
      mz_store_from_float(o.out, row * D + d + 3, a.w / den, o.out_dt);
    } else {
      float* dst = o.acc + row * o.acc_stride + d;
      dst[0] = a.x; dst[1] = a.y; dst[2] = a.z; dst[3] = a.w;
      if (d == 0) { o.m[row * o.ml_stride] = mx * (1.0f / LOG2E); o.l[row * o.ml_stride] = lsum; }
    }
  };
  const int units = total / 4;
  for (int i = threadIdx.x; i < units; i += blockDim.x) {
    const int h = i / (D / 4), d = i % (D / 4) * 4;
    float mx, lsum;
    float4 a;
    merge(std::integral_constant<int, C::MAXW>{}, nw, [&](int w) { return lds2f(high + w * per_high + h * REC + D * 4); },
          [&](int w) { return lds4f(high + w * per_high + h * REC + d * 4); }, mx, lsum, a);
    if (cs == 1) {
      write_out(h, d, mx, lsum, a);
    } else {
      sts128(low + h * REC + d * 4, make_uint4(__float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(a.z), __float_as_uint(a.w)));
      if (d == 0) { stsf(low + h * REC + D * 4, mx); stsf(low + h * REC + D * 4 + 4, lsum); }
    }
  }
  if (cs == 1) return;
  cluster_sync();
  const int i0 = units * rank / cs, i1 = units * (rank + 1) / cs;
  for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
    const int h = i / (D / 4), d = i % (D / 4) * 4;
    float mx, lsum;
    float4 a;
    merge(std::integral_constant<int, 8>{}, cs, [&](int r) { return ld_remote2(remote(low + h * REC + D * 4, r)); },
          [&](int r) { return ld_remote4(remote(low + h * REC + d * 4, r)); }, mx, lsum, a);
    write_out(h, d, mx, lsum, a);
  }
  cluster_sync();                               // nobody leaves while its shared memory may still be read
}

// swizzle of the folded-probability buffer: word w of block j lives at w ^ pswz(j), which spreads both the softmax lanes'
// stores (j = their g) and the fold's loads over all banks
__host__ __device__ constexpr int pswz(int j) { return (j & 1) | (((j >> 1) & 3) << 3); }

template <int BITS, int D_, int G_, int NT>
__global__ void __launch_bounds__(Cfg<BITS, D_, G_, NT>::MAXW * 32, 1) decode_mma_kernel(const __grid_constant__ MzDecodeParams p) {
  using C = Cfg<BITS, D_, G_, NT>;
  constexpr int D = D_, G = G_, NG = C::NG, CPL = C::CPL, MT = C::MT, NB = C::NB;
  constexpr int QT = 2;                       // M tiles of a step: half a quad of lookups
  constexpr int NQ = MT / QT;                 // steps along a row
  constexpr int SPQ = MT < 4 ? 1 : 2;         // steps of a quad
  const mz_kv_store& s = p.s;
  const int bits = BITS == 0 ? s.bits : BITS;
  const int QB = G * bits / 8;                // bytes of one packed row
  const int CODE_BYTES = D * QB;              // one tile side
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int gqa = p.gqa;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  // ---- this warp's share.  Cluster mode: the cluster owns one pair and its warps cut the pair's tiles, interleaved
  // over the CTAs; otherwise the flat list of all tiles is cut.  One launch may carry two plans: the first p.hetero
  // CTAs take the packed tiles, the others the residual tiles (a residual tile is a short latency-bound chain; kept
  // apart it does not sit in the packed tiles' warps).
  const bool clustered = p.cluster > 0;
  const bool second = !clustered && p.hetero > 0 && (int)blockIdx.x >= p.hetero;
  const MzTilesPlan& tp = second ? p.tp2 : p.tp;
  const long long first_record = second ? p.slots_a : 0;      // in records of one head
  const int kt = tp.packed_tiles;
  const int W = tp.total_warps, T = tp.tiles_per_pair;
  const uint32_t nw = blockDim.x >> 5;
  const int rank = clustered ? (int)blockIdx.x % p.cluster : 0;
  const int gw = clustered ? warp * p.cluster + rank : ((int)blockIdx.x - (second ? p.hetero : 0)) * (int)nw + warp;
  long long f0 = 0, f1 = 0;
  if (gw < W) mz_warp_tiles(tp, gw, &f0, &f1);
  const bool active = gw < W && f0 < f1;

  // ---- this warp's buffers (shared-window addresses; the planner sized the pools).  In a cluster a CTA's own window
  // starts at its rank << 24 (the offset below is the same in every CTA), and st.shared / ld.shared want it there.
  extern __shared__ __align__(128) uint8_t smem[];
  const uint32_t window = (uint32_t)__cvta_generic_to_shared(smem) & 0xff000000u;
  const int msz = s.meta_dtype == MZ_F32 ? 4 : 2;
  const uint32_t SB = tp.stage_bytes;
  Layout L;
  L.kbuf = window + tp.low_base + warp * SB;
  L.vbuf = window + tp.high_base + warp * (SB + C::RI_BYTES + C::A_BYTES + C::P_BYTES);
  L.ri = L.vbuf + SB;
  L.q = L.ri + C::RI_BYTES - C::Q_BYTES;
  L.a = L.ri + C::RI_BYTES;
  L.pbuf = L.a + C::A_BYTES;
  // a 64-bit load is served one half of the warp at a time: 16 copies are enough to keep the lookups free of conflicts
  const uint32_t lbK = window + TBL + (lane & 15) * 8;
  const uint32_t lbV = lbK + (s.alpha_key == s.alpha_value ? 0u : 128u);      // equal alphas: one table, in the lower halves
  const int hq = g >> 1;                       // head (of each column set) this lane folds for (B operand column g)
  const uint32_t rem_mask = (g & 1) ? 0xFFFFFFFFu : 0u;   // odd columns carry the fp16 remainder of the folded query
  const bool bf = s.kv_dtype == MZ_BF16;
  const int nq = s.k_groups * G;

  struct Cursor { int pair, tile, b, kvh; };
  auto advance = [&](Cursor& c) {
    if (++c.tile == T) {
      c.tile = 0; ++c.pair;
      if (++c.kvh == s.kv_heads) { c.kvh = 0; ++c.b; }
    }
  };
  auto stage_meta = [&](uint32_t dst, const void* mn, const void* sc, long long m0) {
    for (int off = lane * 16; off < D * msz; off += 512) {
      cp16(dst + off, (const uint8_t*)mn + m0 + off);
      cp16(dst + D * msz + off, (const uint8_t*)sc + m0 + off);
    }
  };
  auto stage_k = [&](const Cursor& c, bool valid) {
    if (valid && c.tile >= kt) stage_dense<C>(p, L.kbuf, false, c.b, c.kvh, c.tile - kt, lane);
    else if (valid) {
      const uint8_t* src = s.packed_k + c.b * s.pk_stride_b + c.kvh * s.pk_stride_h + (long long)c.tile * CODE_BYTES;
      for (int off = lane * 16; off < CODE_BYTES; off += 512) cp16(L.kbuf + off, src + off);
      stage_meta(L.kbuf + CODE_BYTES, s.k_mn, s.k_scale, (c.b * s.km_stride_b + c.kvh * s.km_stride_h + (long long)c.tile * D) * msz);
    }
    cp_async_commit();
  };
  // value rows are regrouped on the way: [group][token] instead of [token][group], so that the rows one load
  // instruction touches are contiguous (rows that are not whole 16-byte chunks keep their order)
  const bool regroup = NG > 1 && QB % 16 == 0;
  auto stage_v = [&](const Cursor& c, bool valid) {
    if (valid && c.tile >= kt) stage_dense<C>(p, L.vbuf, true, c.b, c.kvh, c.tile - kt, lane);
    else if (valid) {
      const uint8_t* src = s.packed_v + c.b * s.pv_stride_b + c.kvh * s.pv_stride_h + (long long)c.tile * CODE_BYTES;
      if (regroup) {
        const int cpr = QB >> 4;               // 16-byte chunks of a row
        for (int i = lane; i < CODE_BYTES / 16; i += 32) {
          const int row = i / cpr, ch = i % cpr;
          cp16(L.vbuf + ((row % NG) * G + row / NG) * QB + ch * 16, src + i * 16);
        }
      } else {
        for (int off = lane * 16; off < CODE_BYTES; off += 512) cp16(L.vbuf + off, src + off);
      }
      stage_meta(L.vbuf + CODE_BYTES, s.v_mn, s.v_scale, (c.b * s.vm_stride_b + c.kvh * s.vm_stride_h + (long long)c.tile * D) * msz);
    }
    cp_async_commit();
  };

  // ---- per-row constants of one staged tile side -> L.ri; row r of the side: keys r = channel, values r = token * NG +
  // group.  Returns whether any row has a real A (then they are in L.a: keys by channel, values [group][token]).
  // unit: what one unit of the scaled constants stands for, in the rows of this lane's value group (lane % NG).
  auto prep_rows = [&](uint32_t buf, bool values, float alpha, float& unit) -> bool {
    const int top = (1 << bits) - 1;
    const float lg = C::WIDE ? log2f(1.0f + alpha) : 0.f, inv_alpha = C::WIDE ? 1.0f / alpha : 0.f;
    auto load_row = [&](int r, float& lo, float& span) {
      if (msz == 4) {
        lo = ldsf(buf + CODE_BYTES + r * 4);
        span = ldsf(buf + CODE_BYTES + D * 4 + r * 4);
      } else {
        lo = mz_u16_to_float((uint16_t)lds16(buf + CODE_BYTES + r * 2), s.meta_dtype);
        span = mz_u16_to_float((uint16_t)lds16(buf + CODE_BYTES + D * 2 + r * 2), s.meta_dtype);
      }
    };
    auto put_row = [&](int r, float span, float bup, float bdn, int zc) {
      const int pos = values ? r / NG : r, grp = values ? r % NG : 0;
      if (C::WIDE) {
        const int blk = values ? (pos >> 4) * NG + grp : pos >> 4;
        const uint32_t at = L.ri + (blk * 4 + ((pos >> 2) & 3)) * 128 + (pos & 3) * 16;
        const float inv = __fdiv_rn(inv_alpha, span);
        sts128(at, make_uint4(__float_as_uint(8388608.0f + (float)zc), __float_as_uint(__fdiv_rn(lg, (float)max(top - zc, 1))),
                              __float_as_uint(__fdiv_rn(lg, (float)max(zc, 1))), __float_as_uint(bup * inv)));
        const __half sh = __float2half_rn(span);
        sts128(at + 64, make_uint4(__float_as_uint(-bdn * inv), pack_u16(__half_as_ushort(sh), __half_as_ushort(__float2half_rn(span - __half2float(sh)))), 0u, 0u));
      } else {
        const int blk = values ? (pos >> 3) * NG + grp : pos >> 3;
        const __half2 hi = __floats2half2_rn(bup, bdn);
        const float2 hf = __half22float2(hi);
        const uint32_t lo = h2_bits(__floats2half2_rn(bup - hf.x, bdn - hf.y)), at = (blk * 4 + (pos & 3)) * 2 + ((pos >> 2) & 1);
        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(L.ri + at * 8), "r"(h2_bits(hi)), "r"(lo) : "memory");
        sts8(L.ri + D * 8 + at, (uint32_t)(zc << BITS));
      }
    };
    float A[D / 32], sp[D / 32], bup[D / 32], bdn[D / 32];
    int zc[D / 32];
    bool any = false, wild = msz == 4;        // fp32 metadata: see row_split
    float most = 0.f;
#pragma unroll
    for (int i = 0; i < D / 32; ++i) {
      float lo;
      load_row(lane + 32 * i, lo, sp[i]);
      row_split(lo, sp[i], (float)top, A[i], bup[i], bdn[i], zc[i], wild);
      any |= A[i] != 0.0f;
      sp[i] = fmaxf(sp[i], 1e-8f);
      most = fmaxf(most, sp[i] < INFINITY ? sp[i] : 0.f);
    }
    if (__any_sync(0xffffffffu, wild)) {
#pragma unroll
      for (int i = 0; i < D / 32; ++i) {
        float lo, span;
        load_row(lane + 32 * i, lo, span);
        zc[i] = exact_zero_code(lo, span, (float)top);
      }
    }
    // the largest range of the tile side (keys) or of the value group
#pragma unroll
    for (int off = values ? NG : 1; off < 32; off <<= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, off));
    const int ex = max(__float_as_int(most) >> 23, 64);              // most in [2^(ex-127), 2^(ex-126)), at least 1e-8 unless no range is finite
    const float scale = __int_as_float((261 - ex) << 23);           // most * scale in [128, 256)
    unit = __int_as_float((ex - 7) << 23);
#pragma unroll
    for (int i = 0; i < D / 32; ++i) put_row(lane + 32 * i, sp[i] * scale, bup[i] * scale, bdn[i] * scale, zc[i]);
    any = __any_sync(0xffffffffu, any);
    if (any) {
#pragma unroll
      for (int i = 0; i < D / 32; ++i) {
        const int r = lane + 32 * i;
        stsf(L.a + (values ? (r % NG) * G + r / NG : r) * 4, A[i]);
      }
    }
    return any;
  };

  float out[NT][D / 16][4];  // M tile grp * MT + m: channels grp * G + CPL * g + 2m + {0,1}, head 4 nt + t, columns {value, 0-column}
  float m_st[NT], l_st[NT];  // softmax state of head 4 nt + t (l: this lane's tokens only, reduced at the end)
  float base_v[NT][NG];      // sum p * A of the channel groups (this lane's tokens only)
  float qs[NT];              // logit scale of head 4 nt + t for packed tiles: 2^k * scaling * log2(e)
  int cur_pair = -1, seg = 0;

  auto reset_state = [&]() {
#pragma unroll
    for (int n = 0; n < NT; ++n) {
#pragma unroll
      for (int m = 0; m < D / 16; ++m)
#pragma unroll
        for (int k = 0; k < 4; ++k) out[n][m][k] = 0.f;
      m_st[n] = -INFINITY; l_st[n] = 0.f;
#pragma unroll
      for (int k = 0; k < NG; ++k) base_v[n][k] = 0.f;
    }
  };
  // lane-wise sums of the state over the lanes that share a head
  auto reduce_state = [&](int n, float& lsum, float (&bv)[NG]) {
    lsum = l_st[n];
#pragma unroll
    for (int k = 0; k < NG; ++k) bv[k] = base_v[n][k];
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) {
      lsum += __shfl_xor_sync(0xffffffffu, lsum, off);
#pragma unroll
      for (int k = 0; k < NG; ++k) bv[k] += __shfl_xor_sync(0xffffffffu, bv[k], off);
    }
  };
  auto write_partial = [&]() {
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      float lsum, bv[NG];
      reduce_state(n, lsum, bv);
      const int h = 4 * n + t;
      if (h < gqa) {
        const long long slot = first_record + ((long long)gw * tp.max_segs + seg) * gqa + h;
        if (!MZ_IN_BOUNDS(slot, p.part.slots, 10)) return;
        float* dst = p.part.acc + slot * D + CPL * g;
#pragma unroll
        for (int k = 0; k < NG; ++k)
#pragma unroll
          for (int m = 0; m < MT; m += 2) {
            const float(&x)[4] = out[n][k * MT + m];
            const float(&y)[4] = out[n][k * MT + m + 1];
            *(float4*)(dst + k * G + 2 * m) = make_float4(x[0] + x[1] + bv[k], x[2] + x[3] + bv[k], y[0] + y[1] + bv[k], y[2] + y[3] + bv[k]);
          }
        if (g == 0) {
          p.part.m[slot] = m_st[n] * (1.0f / LOG2E);   // back to natural-log units
          p.part.l[slot] = lsum;
        }
      }
    }
  };
  // online-softmax update of head 4 n + t with this lane's logits (base 2): the logits become probabilities in
  // place and the running state is rescaled
  auto softmax_update = [&](int n, auto& sv) {
    constexpr int cnt = (int)(sizeof(sv) / sizeof(float));
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < cnt; ++i) mx = fmaxf(mx, sv[i]);
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    const float m_new = fmaxf(m_st[n], mx);
    const bool dead = !(m_new > -INFINITY);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < cnt; ++i) {
      sv[i] = dead ? 0.f : ex2f(sv[i] - m_new);
      sum += sv[i];
    }
    const float c = dead ? 1.0f : ex2f(m_st[n] - m_new);   // m_st = -inf -> 0
    l_st[n] = l_st[n] * c + sum;
    m_st[n] = m_new;
    if (__any_sync(0xffffffffu, c != 1.0f)) {
#pragma unroll
      for (int m = 0; m < D / 16; ++m)
#pragma unroll
        for (int k = 0; k < 4; ++k) out[n][m][k] *= c;
#pragma unroll
      for (int k = 0; k < NG; ++k) base_v[n][k] *= c;
    }
  };

  Cursor cur;
  if (clustered) {
    cur.pair = (int)blockIdx.x / p.cluster;
    cur.tile = (int)f0;
  } else {
    cur.pair = (int)((unsigned)f0 / (unsigned)T); cur.tile = (int)((unsigned)f0 % (unsigned)T);
  }
  cur.b = cur.pair / s.kv_heads; cur.kvh = cur.pair % s.kv_heads;
  Cursor nxt = cur;
  // Everything up to here reads kernel parameters only, and the table build touches shared memory only: when the
  // kernel was launched as a programmatic dependent of the previous kernel in the stream (the merge kernel of the
  // previous call, the flush of this step) this prologue runs while that kernel drains.  Global memory is first
  // touched after the wait (the table entries were written long before).
  if (!C::WIDE && kt > 0) fill_tables<C, C::WIDE ? 1 : BITS>(window + TBL, (const uint2*)p.lut, s.alpha_key, s.alpha_value);
  for (int i = lane; i < (int)C::P_BYTES / 4; i += 32) sts32(L.pbuf + i * 4, 0u);   // columns of absent heads stay zero for good
  asm volatile("griddepcontrol.wait;" ::: "memory");
  stage_k(cur, active);
  stage_v(cur, active);
  __syncthreads();
  reset_state();
  for (int left = active ? (int)(f1 - f0) : 0; left > 0; --left, cur = nxt) {
    const int pair = cur.pair, tile = cur.tile, b = cur.b, kvh = cur.kvh;
    advance(nxt);
    const uint16_t* q0 = (const uint16_t*)p.query + b * p.q_stride_b + (long long)(kvh * gqa) * p.q_stride_h;
    if (pair != cur_pair) {
      if (cur_pair >= 0) { write_partial(); ++seg; }
      cur_pair = pair;
      reset_state();
      // folded-query source: half2(q[8j+t], q[8j+4+t]) of head 4 n + hq, scaled by a power of two into [64, 128)
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const int h = 4 * n + hq;
        const uint16_t* qrow = q0 + min(h, gqa - 1) * p.q_stride_h;
        float qv[2 * NB];
        float amax = 0.f;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          qv[2 * j] = h < gqa ? mz_u16_to_float(qrow[8 * j + t], s.kv_dtype) : 0.f;
          qv[2 * j + 1] = h < gqa ? mz_u16_to_float(qrow[8 * j + 4 + t], s.kv_dtype) : 0.f;
          amax = fmaxf(amax, fmaxf(fabsf(qv[2 * j]), fabsf(qv[2 * j + 1])));
        }
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        int ex = (__float_as_int(amax) >> 23) & 0xff;            // amax in [2^(ex-127), 2^(ex-126))
        ex = min(max(ex, 7), 254);
        const float down = __int_as_float((260 - ex) << 23);     // 2^(133-ex): amax*down in [64, 128)
        const float up = __int_as_float((ex - 6) << 23);         // 2^(ex-133)
#pragma unroll
        for (int j = 0; j < NB; ++j)
          if ((g & 1) == 0) sts32(L.q + (n * NB + j) * 64 + (hq * 4 + t) * 4, h2_bits(__floats2half2_rn(qv[2 * j] * down, qv[2 * j + 1] * down)));
        // head t's scale sits in the lanes that fold for head t (g = 2t)
        qs[n] = __shfl_sync(0xffffffffu, up, 8 * t) * p.scaling * LOG2E;
      }
      warp_sync();
    }
    const bool dense = tile >= kt;
    const int tok0 = dense ? (tile - kt) * DT : tile * G;
    const long long mask0 = p.mask ? b * p.mask_stride_b + (dense ? nq : 0) + tok0 : 0;

    cp_async_wait<1>();
    warp_sync();
    if (!dense) {
      // additive mask of this lane's tokens, in flight during the key phase
      float mv[CPL];
      if (p.mask) {
#pragma unroll
        for (int i = 0; i < CPL; ++i) mv[i] = mz_load_as_float(p.mask, mask0 + CPL * g + i, p.mask_dtype);
      }
      // ================= keys =================
      float un_k;
      const bool hasA = prep_rows(L.kbuf, false, s.alpha_key, un_k);
      warp_sync();
      float acc[NT][MT][4];
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int k = 0; k < 4; ++k) acc[n][m][k] = 0.f;
      if constexpr (!C::WIDE) {
        // steps (block, half a quad), a loop of two blocks: the code words and constants of step i+2 and the table values of
        // step i+1 are in flight while the tensor cores work on step i.  (Unrolled over all blocks the kernel was 48 KB of
        // code and 168 registers; instruction fetch and three warps per scheduler were what it waited for.)
        constexpr int NS = NB * NQ, SPI = 2 * NQ;
        Quad<BITS, CPL> cw[2];
        uint4 rc[2];
        uint2 av[2][8];
        uint32_t zz[2], qq[2][NT], bfr[2][NT][2];
        auto load_step = [&](int blk, int u) {            // u: static step number, blk: its block
          const int q = u % NQ;
          if (q % SPQ == 0) {
            const uint32_t r0 = L.kbuf + (8 * blk + t) * QB + lane_offset<BITS, CPL>(g);
            if constexpr (BITS == 3 || BITS == 1) cw[(u / SPQ) & 1].load(r0, r0 + 4 * QB, q / SPQ, g);
            else cw[(u / SPQ) & 1].load(r0, r0 + 4 * QB, q / SPQ);
          }
          if (q == 0) {
            rc[(u / NQ) & 1] = lds128(L.ri + (blk * 4 + t) * 16);
            zz[(u / NQ) & 1] = lds16(L.ri + D * 8 + (blk * 4 + t) * 2);
#pragma unroll
            for (int n = 0; n < NT; ++n) qq[(u / NQ) & 1][n] = lds32(L.q + (n * NB + blk) * 64 + (hq * 4 + t) * 4);
          }
        };
        auto open_step = [&](int u) {
          const int o = (u / NQ) & 1;
          look_step(cw[(u / SPQ) & 1], u % SPQ, zz[o], lbK, av[u & 1]);
          // fold q * B: even columns the product rounded to fp16, odd columns what that rounding dropped
          if (u % NQ == 0) {
#pragma unroll
            for (int n = 0; n < NT; ++n) {
              const uint32_t x = qq[o][n], xm = x & rem_mask;
              bfr[o][n][0] = fold_pair(dup_lo(x), dup_lo(xm), rc[o].x, rc[o].y, rem_mask);
              bfr[o][n][1] = fold_pair(dup_hi(x), dup_hi(xm), rc[o].z, rc[o].w, rem_mask);
            }
          }
        };
        load_step(0, 0);
        load_step(1 / NQ, 1);
        open_step(0);
#pragma unroll 1
        for (int i0 = 0; i0 < NS; i0 += SPI) {
#pragma unroll
          for (int u = 0; u < SPI; ++u) {
            const int blk2 = (i0 + u + 2) / NQ;
            if (u + 2 < SPI || i0 + SPI < NS) load_step(blk2, u + 2);
            if (u + 1 < SPI || i0 + SPI < NS) open_step(u + 1);
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
              for (int m = 0; m < QT; ++m) mma_step(acc[n][(u % NQ) * QT + m], av[u & 1], m, bfr[(u / NQ) & 1][n][0], bfr[(u / NQ) & 1][n][1]);
          }
        }
      } else {
        wide_side<C, BITS, 1>(L.kbuf, L.ri, g, t, bits, [&](int blk, int sl) { return (16 * blk + 4 * sl + t) * QB; },
                           [&](int blk, const uint32_t (&sp)[4], uint32_t (&bb)[NT][2]) {
#pragma unroll
          for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int k = 0; k < 2; ++k)
            {
              const uint32_t x = lds32(L.q + (n * NB + 2 * blk + k) * 64 + (hq * 4 + t) * 4);
              bb[n][k] = fold_pair(bits_h2(x), bits_h2(x & rem_mask), pack_u16(sp[2 * k], sp[2 * k + 1]), prmt(sp[2 * k], sp[2 * k + 1], 0x7632u), rem_mask);
            }
        }, [&](int, int m, const uint32_t (&hi)[4], const uint32_t (&lo)[4], const uint32_t (&bb)[NT][2]) {
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            float x[4];
            mma_f16_first(x, lo[0], lo[1], lo[2], lo[3], bb[n][0], bb[n][1]);
            mma_f16(x, hi[0], hi[1], hi[2], hi[3], bb[n][0], bb[n][1]);
            add4(acc[n][m], x);
          }
        });
      }
      // constant term sum_d q[t][d] * A_d (rows whose range does not straddle zero)
      float cA[NT];
#pragma unroll
      for (int n = 0; n < NT; ++n) cA[n] = 0.f;
      if (hasA) {
        for (int h = 0; h < gqa; ++h) {
          float part = 0.f;
#pragma unroll
          for (int i = 0; i < D / 32; ++i) part = fmaf(mz_u16_to_float(q0[h * p.q_stride_h + lane + 32 * i], s.kv_dtype), ldsf(L.a + (lane + 32 * i) * 4), part);
#pragma unroll
          for (int off = 1; off < 32; off <<= 1) part += __shfl_xor_sync(0xffffffffu, part, off);
#pragma unroll
          for (int n = 0; n < NT; ++n)
            if (h == 4 * n + t) cA[n] = part * p.scaling * LOG2E;
        }
      }
      warp_sync();                  // every lane is done with kbuf and the row constants
      stage_k(nxt, left > 1);
      // ================= softmax: this lane has head 4 n + t, tokens CPL g .. CPL g + CPL - 1 =================
      float sv[NT][CPL];
#pragma unroll
      for (int n = 0; n < NT; ++n) {
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          sv[n][2 * m] = fmaf(acc[n][m][0] + acc[n][m][1], qs[n] * un_k, cA[n]);
          sv[n][2 * m + 1] = fmaf(acc[n][m][2] + acc[n][m][3], qs[n] * un_k, cA[n]);
        }
        if (p.mask) {
#pragma unroll
          for (int i = 0; i < CPL; ++i) sv[n][i] += mv[i] * LOG2E;
        }
        softmax_update(n, sv[n]);
        if (4 * n + t < gqa) {
          // scaled probabilities as fp16 pairs (p[8j+i], p[8j+4+i]): column 2t the rounded values, column 2t+1 their
          // remainders; word (j, i, column) is swizzled over the banks by j
          auto put = [&](int j, int i, float a, float b2) {
            a *= P_SCALE; b2 *= P_SCALE;
            const __half2 ph = __floats2half2_rn(a, b2);
            const float2 phf = __half22float2(ph);
            const uint32_t wa = L.pbuf + j * (128 * NT), wi = (8 * NT) * i + 8 * n + 2 * t;
            sts32(wa + ((wi ^ pswz(j)) << 2), h2_bits(ph));
            sts32(wa + (((wi + 1) ^ pswz(j)) << 2), h2_bits(__floats2half2_rn(a - phf.x, b2 - phf.y)));
          };
          if (CPL >= 8) {
#pragma unroll
            for (int jj = 0; jj < CPL / 8; ++jj)
#pragma unroll
              for (int i = 0; i < 4; ++i) put(g * (CPL / 8) + jj, i, sv[n][(8 * jj + i) % CPL], sv[n][(8 * jj + i + 4) % CPL]);
          } else {
            // this lane has one half of each word
            const int j = g >> 1;
            const uint32_t wa = L.pbuf + j * (128 * NT) + 2 * (g & 1);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t wi = (8 * NT) * i + 8 * n + 2 * t;
              const float a = sv[n][i % CPL] * P_SCALE;
              const __half ph = __float2half_rn(a);
              sts16(wa + ((wi ^ pswz(j)) << 2), __half_as_ushort(ph));
              sts16(wa + (((wi + 1) ^ pswz(j)) << 2), __half_as_ushort(__float2half_rn(a - __half2float(ph))));
            }
          }
        }
      }
      cp_async_wait<1>();
      warp_sync();                  // value tile landed; probabilities visible
      // ================= values =================
      float un_mine, un_v[NG];
      const bool hasAV = prep_rows(L.vbuf, true, s.alpha_value, un_mine);
      warp_sync();
#pragma unroll
      for (int k = 0; k < NG; ++k) un_v[k] = __shfl_sync(0xffffffffu, un_mine, k) * (1.0f / P_SCALE);
      if (hasAV) {
#pragma unroll
        for (int n = 0; n < NT; ++n)
          if (4 * n + t < gqa) {
#pragma unroll
            for (int i = 0; i < CPL; ++i)
#pragma unroll
              for (int k = 0; k < NG; ++k) base_v[n][k] = fmaf(sv[n][i], ldsf(L.a + (k * G + CPL * g + i) * 4), base_v[n][k]);
          }
      }
      // this lane folds for head 4 n + hq: the rounded probabilities sit in column 2 hq, their remainders in 2 hq + 1
      auto probs = [&](int n, int j, uint32_t& hi, uint32_t& lo) {
        const uint32_t wa = L.pbuf + j * (128 * NT), wi = (8 * NT) * t + 8 * n + (g & ~1);
        hi = lds32(wa + ((wi ^ pswz(j)) << 2));
        lo = lds32(wa + (((wi + 1) ^ pswz(j)) << 2)) & rem_mask;
      };
      const uint32_t v_row = regroup ? QB : NG * QB, v_grp = regroup ? G * QB : QB;     // token and group strides in the staged tile
      if constexpr (!C::WIDE) {
        // steps (token block j, group, half a quad), a loop of one or two token blocks; the probabilities of a token block
        // are read once
        constexpr int NS = NB * NQ, BPI = NG > 2 ? NG : 2, SPI = BPI * NQ;       // blocks and steps of an iteration
        Quad<BITS, CPL> cw[2];
        uint4 rc[2];
        uint2 av[2][8];
        uint32_t zz[2], bfr[2][NT][2], ph[2][NT], pl[2][NT];
        auto load_step = [&](int blk, int u) {
          const int q = u % NQ, grp = (u / NQ) % NG, j = blk / NG;
          if (q % SPQ == 0) {
            const uint32_t r0 = L.vbuf + (8 * j + t) * v_row + grp * v_grp + lane_offset<BITS, CPL>(g);
            if constexpr (BITS == 3 || BITS == 1) cw[(u / SPQ) & 1].load(r0, r0 + 4 * v_row, q / SPQ, g);
            else cw[(u / SPQ) & 1].load(r0, r0 + 4 * v_row, q / SPQ);
          }
          if (q == 0) {
            rc[(u / NQ) & 1] = lds128(L.ri + (blk * 4 + t) * 16);
            zz[(u / NQ) & 1] = lds16(L.ri + D * 8 + (blk * 4 + t) * 2);
            if (grp == 0) {
#pragma unroll
              for (int n = 0; n < NT; ++n) probs(n, j, ph[(u / NQ / NG) & 1][n], pl[(u / NQ / NG) & 1][n]);
            }
          }
        };
        auto open_step = [&](int u) {
          const int o = (u / NQ) & 1;
          look_step(cw[(u / SPQ) & 1], u % SPQ, zz[o], lbV, av[u & 1]);
          // fold (ph + pl) * B: even columns fp16(ph * B), odd columns its remainder + pl * B
          if (u % NQ == 0) {
#pragma unroll
            for (int n = 0; n < NT; ++n) {
              const uint32_t hi = ph[(u / NQ / NG) & 1][n], lo = pl[(u / NQ / NG) & 1][n];
              const uint32_t hm = hi & rem_mask;
              bfr[o][n][0] = h2_bits(__hfma2(dup_lo(lo), bits_h2(rc[o].x), bits_h2(fold_pair(dup_lo(hi), dup_lo(hm), rc[o].x, rc[o].y, rem_mask))));
              bfr[o][n][1] = h2_bits(__hfma2(dup_hi(lo), bits_h2(rc[o].z), bits_h2(fold_pair(dup_hi(hi), dup_hi(hm), rc[o].z, rc[o].w, rem_mask))));
            }
          }
        };
        // two iterations are unrolled where a token block's probabilities alternate between two registers across them
        constexpr int TWO = (BPI / NG) & 1 ? 2 : 1;
        load_step(0, 0);
        load_step(1 / NQ, 1);
        open_step(0);
#pragma unroll 1
        for (int i0 = 0; i0 < NS; i0 += TWO * SPI) {
#pragma unroll
          for (int u = 0; u < TWO * SPI; ++u) {
            const int blk2 = (i0 + u + 2) / NQ;
            if (u + 2 < TWO * SPI || i0 + TWO * SPI < NS) load_step(blk2, u + 2);
            if (u + 1 < TWO * SPI || i0 + TWO * SPI < NS) open_step(u + 1);
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
              for (int m = 0; m < QT; ++m)
                mma_step<true>(out[n][((u / NQ) % NG) * MT + (u % NQ) * QT + m], av[u & 1], m, bfr[(u / NQ) & 1][n][0], bfr[(u / NQ) & 1][n][1], un_v[(u / NQ) % NG]);
          }
        }
      } else {
        wide_side<C, BITS, NG>(L.vbuf, L.ri, g, t, bits,
                           [&](int blk, int sl) { return (16 * (blk / NG) + 4 * sl + t) * v_row + (blk % NG) * v_grp; },
                           [&](int blk, const uint32_t (&sp)[4], uint32_t (&bb)[NT][2]) {
          const int j = blk / NG;
#pragma unroll
          for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              uint32_t hi, lo;
              probs(n, 2 * j + k, hi, lo);
              const uint32_t S = pack_u16(sp[2 * k], sp[2 * k + 1]);
              bb[n][k] = h2_bits(__hfma2(bits_h2(lo), bits_h2(S), bits_h2(fold_pair(bits_h2(hi), bits_h2(hi & rem_mask), S, prmt(sp[2 * k], sp[2 * k + 1], 0x7632u), rem_mask))));
            }
        }, [&](int k, int m, const uint32_t (&hi)[4], const uint32_t (&lo)[4], const uint32_t (&bb)[NT][2]) {
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            float x[4];
            mma_f16_first(x, lo[0], lo[1], lo[2], lo[3], bb[n][0], bb[n][1]);
            mma_f16(x, hi[0], hi[1], hi[2], hi[3], bb[n][0], bb[n][1]);
            fma4(out[n][k * MT + m], x, un_v[k]);
          }
        });
      }
      warp_sync();                  // every lane is done with vbuf, the row constants and the probabilities
      stage_v(nxt, left > 1);
    } else {
      dense_tile<C>(p, L.kbuf, L.vbuf, tile - kt, b, kvh, g, t, hq, bf, mask0, q0, out, softmax_update, [&]() { stage_k(nxt, left > 1); },
                    [&]() { cp_async_wait<1>(); warp_sync(); });
      warp_sync();                  // every lane is done with vbuf
      stage_v(nxt, left > 1);
    }
  }
  cp_async_wait<0>();
  if (!clustered) {
    if (active) write_partial();
    return;
  }
  finish_cluster<C>(p, window, rank, (int)nw, warp, lane, g, t, active, out, m_st, reduce_state);
}

template <int BITS, int D_, int G_, int NT>
void describe(MzMmaKernel* k) {
  using C = Cfg<BITS, D_, G_, NT>;
  *k = {(const void*)decode_mma_kernel<BITS, D_, G_, NT>, C::RI_BYTES, C::A_BYTES, C::P_BYTES, C::TABLE_BYTES, C::MAXW};
}
template <int BITS>
bool pick_instance(int D, int G, int nt, MzMmaKernel* k) {
#define MZ_MMA_CASE(d, g)                          \
  if (D == d && G == g) {                          \
    if (nt == 1) describe<BITS, d, g, 1>(k);       \
    else describe<BITS, d, g, 2>(k);               \
    return true;                                   \
  }
  MZ_MMA_CASE(128, 64)
  MZ_MMA_CASE(128, 32)
  MZ_MMA_CASE(128, 128)
  MZ_MMA_CASE(64, 64)
  MZ_MMA_CASE(64, 32)
#undef MZ_MMA_CASE
  return false;
}
}  // namespace mzm
