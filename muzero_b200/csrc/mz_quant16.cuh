// Quantizer of 16-bit rows on packed pairs (two values per register), bit-exact with MzQuantRow.
//
// The reference's chain rounds to the 16-bit type after every operation.  Two facts make it cheap:
//   * R(x - lo), R(1 - a) and the like are one packed 16-bit instruction: the fp32 difference of two 16-bit values
//     is exact unless the smaller one is below 2^-13 of the larger, and then neither rounding can cross a tie
//   * everything after unit = R(R(x - lo) / span) depends on the row through ONE 16-bit number, the zero anchor
//     (zero code, steps and side extents all follow from it), and the code never decreases as unit grows.
//     So the code is the number of thresholds U_k(anchor) = min{unit : code >= k} that unit reaches.  The
//     thresholds of every anchor in [0, 1] are a table (15 x 2 bytes per anchor at 4 bits, 0.5 MB, L2 resident)
//     built once per device by evaluating the chain itself; a binary search over it takes BITS packed compares.
// Wider codes (5..8 bits) would need hundreds of thresholds per row and evaluate the chain on the unit instead.
// Bound by instruction issue; the chain itself takes about 100 instructions per value and most of a prompt's time.
#pragma once
#include "mz_quant_math.cuh"

namespace mzq {

template <int DT> struct P2;   // packed pair of the 16-bit type, as raw bits
template <> struct P2<MZ_BF16> {
  static constexpr uint32_t ONE = 0x3F80u, INF2 = 0x7F807F80u;
  static __device__ __forceinline__ __nv_bfloat162 h(uint32_t v) { return *reinterpret_cast<__nv_bfloat162*>(&v); }
  static __device__ __forceinline__ uint32_t b(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t*>(&v); }
  static __device__ __forceinline__ uint32_t sub(uint32_t x, uint32_t y) { return b(__hsub2(h(x), h(y))); }
  static __device__ __forceinline__ uint32_t mn(uint32_t x, uint32_t y) { return b(__hmin2(h(x), h(y))); }
  static __device__ __forceinline__ uint32_t mx(uint32_t x, uint32_t y) { return b(__hmax2(h(x), h(y))); }
  static __device__ __forceinline__ uint32_t mx_nan(uint32_t x, uint32_t y) { return b(__hmax2_nan(h(x), h(y))); }
  static __device__ __forceinline__ uint32_t ge(uint32_t x, uint32_t y) { return __hge2_mask(h(x), h(y)); }
  static __device__ __forceinline__ float lo(uint32_t v) { return __uint_as_float(v << 16); }
  static __device__ __forceinline__ float hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
  static __device__ __forceinline__ uint32_t pack(float a, float c) { return b(__floats2bfloat162_rn(a, c)); }
  // low half-words of two fp32 quotients -> zero in a half whose value lies within 4 fp32 ulps of a rounding
  // boundary of the type (a borrow out of the low half moves the high half's window by one, still inside)
  static __device__ __forceinline__ uint32_t near_tie(uint32_t ya, uint32_t yb, uint32_t) {
    return (__byte_perm(ya, yb, 0x5410) - 0x7FFC7FFCu) & 0xFFF8FFF8u;
  }
};
template <> struct P2<MZ_F16> {
  static constexpr uint32_t ONE = 0x3C00u, INF2 = 0x7C007C00u;
  static __device__ __forceinline__ __half2 h(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
  static __device__ __forceinline__ uint32_t b(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
  static __device__ __forceinline__ uint32_t sub(uint32_t x, uint32_t y) { return b(__hsub2(h(x), h(y))); }
  static __device__ __forceinline__ uint32_t mn(uint32_t x, uint32_t y) { return b(__hmin2(h(x), h(y))); }
  static __device__ __forceinline__ uint32_t mx(uint32_t x, uint32_t y) { return b(__hmax2(h(x), h(y))); }
  static __device__ __forceinline__ uint32_t mx_nan(uint32_t x, uint32_t y) { return b(__hmax2_nan(h(x), h(y))); }
  static __device__ __forceinline__ uint32_t ge(uint32_t x, uint32_t y) { return __hge2_mask(h(x), h(y)); }
  static __device__ __forceinline__ float lo(uint32_t v) { return __low2float(h(v)); }
  static __device__ __forceinline__ float hi(uint32_t v) { return __high2float(h(v)); }
  static __device__ __forceinline__ uint32_t pack(float a, float c) { return b(__floats2half2_rn(a, c)); }
  // as above for the 13 dropped bits of a normal fp16 result; results in (0, 2^-14] (subnormal, other boundaries)
  // always count as near a boundary
  static __device__ __forceinline__ uint32_t near_tie(uint32_t ya, uint32_t yb, uint32_t r) {
    const uint32_t m = (__byte_perm(ya, yb, 0x5410) + 0x10041004u) & 0x1FF81FF8u;
    const uint32_t a = r & 0xffffu, c = r >> 16;
    return (a - 1u < 0x400u || c - 1u < 0x400u) ? 0u : m;
  }
};

// per-row constants shared by the thresholds builder and both code paths
template <int DT>
struct Anchor {
  float anchor, zero_code, steps_up, steps_dn, room_up, room_dn;
  __device__ __forceinline__ void set(float a, float top, float eps_t) {
    using TT = MzType<DT>;
    anchor = a;
    zero_code = rintf(TT::round(__fmul_rn(a, top)));
    steps_up = fmaxf(TT::round(__fsub_rn(top, zero_code)), 1.0f);
    steps_dn = fmaxf(zero_code, 1.0f);
    room_up = fmaxf(TT::round(__fsub_rn(1.0f, a)), eps_t);
    room_dn = fmaxf(a, eps_t);
  }
};

// round-half-even of a value in [0, 2^22) left in the low mantissa bits
constexpr float kMagic = 12582912.0f;

// Code of `unit` (clamped to [0, 1], not NaN) for the row constants `c`; p_up / p_dn select the quotient.  The plain
// form of the chain's second half, used by the table builder (IEEE divisions).
template <int DT>
__device__ __forceinline__ int code_of_unit(float unit, const Anchor<DT>& c, float top, const uint16_t* __restrict__ ctab, int ctab_n) {
  using TT = MzType<DT>;
  const bool up = unit >= c.anchor;
  const float num = fabsf(TT::round(__fsub_rn(unit, c.anchor)));
  float p = TT::round(__fdiv_rn(num, up ? c.room_up : c.room_dn));
  if (p != p) return 0;
  p = fminf(fmaxf(p, 0.0f), 1.0f);
  uint32_t idx = DT == MZ_BF16 ? __float_as_uint(p) >> 16 : (uint32_t)__half_as_ushort(__float2half_rn(p));
  idx = min(idx, (uint32_t)(ctab_n - 1));
  const float rr = rintf(TT::round(__fmul_rn(mz_u16_to_float(ctab[idx], DT), up ? c.steps_up : c.steps_dn)));
  const float q = up ? c.zero_code + rr : c.zero_code - rr;
  return (int)fminf(fmaxf(q, 0.0f), top);
}

// What a row's min / max determine.  `special`: the packed path does not apply (non-finite range, or an extent that
// rounds to zero in the type, where the reference's chain goes through NaN) and every value takes MzQuantRow::code.
template <int DT>
struct RowHead {
  float lo, span, inv_span;
  uint32_t anchor_bits;    // index of the row's thresholds
  bool special;
  __device__ __forceinline__ void set(float mn, float mx, float eps) {
    using TT = MzType<DT>;
    const float eps_t = TT::round(eps);
    lo = mn;
    span = fmaxf(TT::round(__fsub_rn(mx, mn)), eps_t);
    const float a = TT::round(__fdiv_rn(TT::round(__fsub_rn(0.0f, mn)), span));
    const float anchor = fminf(fmaxf(a, 0.0f), 1.0f);
    inv_span = __frcp_rn(span);
    anchor_bits = DT == MZ_BF16 ? __float_as_uint(anchor) >> 16 : (uint32_t)__half_as_ushort(__float2half_rn(anchor));
    special = !(span > 0.0f && span < INFINITY) || a != a || !(inv_span < INFINITY && inv_span > 1.2e-38f) ||
              (eps_t == 0.0f && anchor == 1.0f);
  }
};

// ---- thresholds held by a thread: T[k - 1] = (U_k of the row in the low half, U_k of the row in the high half)
template <int DT, int BITS>
struct Thresholds {
  static constexpr int N = (1 << BITS) - 1;
  uint32_t T[N];
  static __device__ __forceinline__ uint32_t sel(uint32_t m, uint32_t a, uint32_t b) { return (a & m) | (b & ~m); }
  // the codes of a pair of units, each shifted left by SH inside its half-word
  template <int SH>
  __device__ __forceinline__ uint32_t codes(uint32_t u) const {
    using P = P2<DT>;
    constexpr uint32_t B0 = 0x00010001u << SH;
    if (BITS == 1) return P::ge(u, T[0]) & B0;
    if (BITS == 2) {
      const uint32_t m1 = P::ge(u, T[1]);
      const uint32_t m0 = P::ge(u, sel(m1, T[2], T[0]));
      return (m1 & (B0 << 1)) | (m0 & B0);
    }
    if (BITS == 3) {
      const uint32_t m2 = P::ge(u, T[3 % N]);
      const uint32_t m1 = P::ge(u, sel(m2, T[5 % N], T[1 % N]));
      const uint32_t m0 = P::ge(u, sel(m2, sel(m1, T[6 % N], T[4 % N]), sel(m1, T[2 % N], T[0])));
      return (m2 & (B0 << 2)) | (m1 & (B0 << 1)) | (m0 & B0);
    }
    const uint32_t m3 = P::ge(u, T[7 % N]);
    const uint32_t m2 = P::ge(u, sel(m3, T[11 % N], T[3 % N]));
    const uint32_t m1 = P::ge(u, sel(m3, sel(m2, T[13 % N], T[9 % N]), sel(m2, T[5 % N], T[1 % N])));
    const uint32_t m0 = P::ge(u, sel(m3, sel(m2, sel(m1, T[14 % N], T[12 % N]), sel(m1, T[10 % N], T[8 % N])),
                                     sel(m2, sel(m1, T[6 % N], T[4 % N]), sel(m1, T[2 % N], T[0]))));
    return (m3 & (B0 << 3)) | (m2 & (B0 << 2)) | (m1 & (B0 << 1)) | (m0 & B0);
  }
};

// ---- wider codes: the chain's second half on a pair of units; the two halves may belong to two rows
template <int DT>
struct WideRow {
  float anchor, zero_code, steps_up, steps_dn, room_up, room_dn, inv_up, inv_dn;
  __device__ __forceinline__ void set(float a, float top, float eps_t) {
    Anchor<DT> c;
    c.set(a, top, eps_t);
    anchor = a; zero_code = c.zero_code; steps_up = c.steps_up; steps_dn = c.steps_dn; room_up = c.room_up; room_dn = c.room_dn;
    inv_up = __frcp_rn(room_up); inv_dn = __frcp_rn(room_dn);
  }
};
// units (in [0, 1]) -> codes of the low / high half as bytes 0 / 2
template <int DT>
__device__ __forceinline__ uint32_t wide_codes(uint32_t u, const WideRow<DT>& a, const WideRow<DT>& b, float top,
                                               const uint16_t* __restrict__ ctab) {
  using P = P2<DT>;
  const float ua = P::lo(u), ub = P::hi(u);
  const bool upa = ua >= a.anchor, upb = ub >= b.anchor;
  const uint32_t num = P::pack(fabsf(ua - a.anchor), fabsf(ub - b.anchor));
  const float na = P::lo(num), nb = P::hi(num);
  const float ya = __fmul_rn(na, upa ? a.inv_up : a.inv_dn), yb = __fmul_rn(nb, upb ? b.inv_up : b.inv_dn);
  uint32_t p = P::pack(ya, yb);
  const uint32_t tie = P::near_tie(__float_as_uint(ya), __float_as_uint(yb), p);
  if ((tie & 0xffffu) == 0u || (tie >> 16) == 0u)
    p = P::pack(__fdiv_rn(na, upa ? a.room_up : a.room_dn), __fdiv_rn(nb, upb ? b.room_up : b.room_dn));
  const uint32_t pa = min(p & 0xffffu, P::ONE), pb = min(p >> 16, P::ONE);     // p >= 0: ordered as integers
  const uint32_t r = P::pack(__fmul_rn(mz_u16_to_float(ctab[pa], DT), upa ? a.steps_up : a.steps_dn),
                             __fmul_rn(mz_u16_to_float(ctab[pb], DT), upb ? b.steps_up : b.steps_dn));
  const float ra = __fsub_rn(__fadd_rn(P::lo(r), kMagic), kMagic), rb = __fsub_rn(__fadd_rn(P::hi(r), kMagic), kMagic);
  const float qa = fminf(fmaxf(upa ? a.zero_code + ra : a.zero_code - ra, 0.0f), top);
  const float qb = fminf(fmaxf(upb ? b.zero_code + rb : b.zero_code - rb, 0.0f), top);
  return __byte_perm(__float_as_uint(__fadd_rn(qa, kMagic)), __float_as_uint(__fadd_rn(qb, kMagic)), 0x7410) & 0x00ff00ffu;
}
__device__ __forceinline__ uint32_t min_u16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("min.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// units of W pairs: u = R(R(x - lo) / span), one multiply per value; when a product lies near a rounding boundary of
// the type (1 in 8000) the group is divided out
template <int DT, int W>
__device__ __forceinline__ void units_of(const uint32_t (&x)[W], uint32_t lo2, float inv_a, float inv_b, float span_a, float span_b,
                                         uint32_t (&u)[W]) {
  using P = P2<DT>;
  uint32_t tie = 0xffffffffu;
#pragma unroll
  for (int i = 0; i < W; ++i) {
    const uint32_t d = P::sub(x[i], lo2);
    const float ya = __fmul_rn(P::lo(d), inv_a), yb = __fmul_rn(P::hi(d), inv_b);
    u[i] = P::pack(ya, yb);
    tie = min_u16x2(tie, P::near_tie(__float_as_uint(ya), __float_as_uint(yb), u[i]));
  }
  if ((tie & 0xffffu) == 0u || tie < 0x10000u) {
#pragma unroll
    for (int i = 0; i < W; ++i) {
      const uint32_t d = P::sub(x[i], lo2);
      u[i] = P::pack(__fdiv_rn(P::lo(d), span_a), __fdiv_rn(P::hi(d), span_b));
    }
  }
}

// eight codes (four pairs of units of one row) -> `bits` bytes
template <int DT, int BITS>
__device__ __forceinline__ unsigned long long pack_octet(const Thresholds<DT, BITS>& th, const uint32_t (&u)[4]) {
  if constexpr (BITS == 4) {
    // byte w of a half: the low half's code in the low nibble, the high half's moves into the high nibble
    const uint32_t a = th.template codes<0>(u[0]) | th.template codes<8>(u[1]);
    const uint32_t b = th.template codes<0>(u[2]) | th.template codes<8>(u[3]);
    return __byte_perm(a | (a >> 12), b | (b >> 12), 0x5410);
  } else if constexpr (BITS == 3) {
    const uint32_t a = th.template codes<0>(u[0]) | th.template codes<6>(u[1]);
    const uint32_t b = th.template codes<0>(u[2]) | th.template codes<6>(u[3]);
    return ((a | (a >> 13)) & 0xfffu) | (((b | (b >> 13)) & 0xfffu) << 12);
  } else {
    const uint32_t a = th.template codes<0>(u[0]) | th.template codes<2 * BITS>(u[1]) | th.template codes<4 * BITS>(u[2]) |
                       th.template codes<6 * BITS>(u[3]);
    return (a | (a >> (16 - BITS))) & ((1u << (8 * BITS)) - 1u);
  }
}

// One lane's share of a value row: chunks sub and sub + lpr of eight values, in x[0..3] and x[4..7]; `word[c]` receives
// the packed codes of chunk c.  All lanes of a row call it (shuffles over lpr lanes).
template <int DT, int BITS>
__device__ __forceinline__ void quantize_row16(const uint32_t (&x)[8], int lpr, float alpha, float eps, const uint16_t* __restrict__ thr,
                                               const uint16_t* __restrict__ ctab, int ctab_n, RowHead<DT>& head,
                                               unsigned long long (&word)[2]) {
  using P = P2<DT>;
  constexpr bool WIDE = BITS > 4;
  uint32_t mn = x[0], mx = x[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) { mn = P::mn(mn, x[i]); mx = P::mx(mx, x[i]); }
  for (int off = lpr >> 1; off > 0; off >>= 1) {
    mn = P::mn(mn, __shfl_xor_sync(0xffffffffu, mn, off));
    mx = P::mx(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  }
  const float fmn = fminf(P::lo(mn), P::hi(mn)), fmx = fmaxf(P::lo(mx), P::hi(mx));
  head.set(fmn, fmx, eps);
  if (head.special) {
    MzQuantRow<DT> r;
    r.setup(fmn, fmx, BITS, alpha, eps, ctab, ctab_n);
    word[0] = word[1] = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      word[i >> 2] |= (unsigned long long)r.code(P::lo(x[i])) << ((2 * (i & 3)) * BITS);
      word[i >> 2] |= (unsigned long long)r.code(P::hi(x[i])) << ((2 * (i & 3) + 1) * BITS);
    }
    return;
  }
  const uint32_t lo2 = P::pack(head.lo, head.lo);
  uint32_t u[2][4];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const uint32_t xx[4] = {x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]};
    units_of<DT, 4>(xx, lo2, head.inv_span, head.inv_span, head.span, head.span, u[c]);
  }
  if constexpr (!WIDE) {
    Thresholds<DT, BITS> th;
    const uint16_t* t = thr + ((size_t)head.anchor_bits << BITS);
    uint32_t w[1 << (BITS - 1)];
    if constexpr (BITS >= 3) {
#pragma unroll
      for (int k = 0; k < (1 << (BITS - 3)); ++k) {
        const uint4 a = *((const uint4*)t + k);
        w[4 * k] = a.x; w[4 * k + 1] = a.y; w[4 * k + 2] = a.z; w[4 * k + 3] = a.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < BITS; ++k) w[k] = *((const uint32_t*)t + k);
    }
#pragma unroll
    for (int k = 0; k < (1 << BITS) - 1; ++k) th.T[k] = __byte_perm(w[k >> 1], 0u, (k & 1) ? 0x3232 : 0x1010);
#pragma unroll
    for (int c = 0; c < 2; ++c) word[c] = pack_octet<DT, BITS>(th, u[c]);
  } else {
    WideRow<DT> r;
    r.set(mz_u16_to_float((uint16_t)head.anchor_bits, DT), (float)((1 << BITS) - 1), MzType<DT>::round(eps));
    const uint32_t one = P::ONE | (P::ONE << 16);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      word[c] = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t nn = P::ge(u[c][k], 0u);           // a NaN value has code 0
        const uint32_t q = wide_codes<DT>(P::mn(P::mx(u[c][k], 0u), one), r, r, (float)((1 << BITS) - 1), ctab) & nn;
        word[c] |= ((unsigned long long)(q & 0xffffu) << (2 * k * BITS)) | ((unsigned long long)(q >> 16) << ((2 * k + 1) * BITS));
      }
    }
  }
}

}  // namespace mzq

// Device table of thresholds: [anchor bits 0 .. bits_of(1.0)][2^bits] of 16-bit values, entry k - 1 = U_k(anchor),
// the type's infinity where no unit in [0, 1] reaches k; the last entry of a row is unused.  bits 1..4.
int mz_get_unit_thresholds(int dtype, int bits, float alpha, float eps, const uint16_t** dev_table);
