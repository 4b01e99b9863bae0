// Quantizer of fp32 rows.  The reference's fp32 chain is one rounding per operation with log1p taken correctly
// rounded; its result is an integer, so it only has to be followed exactly where the un-rounded code position comes
// near a half.  F32Row evaluates the position with the hardware log2 and one reciprocal per row, bounds its own error,
// and leaves the (rare) values inside that bound to MzQuantRow<MZ_F32>, which carries a double-precision log1p.
#pragma once
#include "mz_quant_math.cuh"

namespace mzq {
struct F32Row {
  float lo, span, inv_span, anchor, a_up, a_dn, k_up, k_dn, zero_code, top, limit;
  __device__ __forceinline__ void set(float mn, float mx, int bits, float alpha, float eps) {
    top = (float)((1 << bits) - 1);
    lo = mn;
    span = fmaxf(__fsub_rn(mx, mn), eps);
    inv_span = __frcp_rn(span);
    anchor = fminf(fmaxf(__fdiv_rn(__fsub_rn(0.0f, mn), span), 0.0f), 1.0f);
    zero_code = rintf(__fmul_rn(anchor, top));
    const float lb = log1pf(alpha);
    a_up = __fdividef(alpha, fmaxf(1.0f - anchor, eps));
    a_dn = __fdividef(alpha, fmaxf(anchor, eps));
    const float per_log2 = 0.693147182f / lb;
    k_up = fmaxf(top - zero_code, 1.0f) * per_log2;
    k_dn = fmaxf(zero_code, 1.0f) * per_log2;
    // distance from a half below which the position is not trusted: a position is steps * log1p(alpha * s / room) / lb,
    // steps / room < 2 top on the side that matters (on the other side every position clamps to the end code), so an
    // error of 4e-7 in s moves it by less than 8e-7 * top * alpha / lb; log2 and the products add a few 1e-7 * top
    limit = 0.5f - (2e-6f * top * (1.0f + alpha / lb) + 1e-5f);
    // a row outside the ordinary range (non-finite, or a reciprocal that over/underflows): every value the exact way
    if (!(span < 1e37f && inv_span < 1e37f && lo > -1e37f && lo < 1e37f && a_up < 1e30f && a_dn < 1e30f && limit > 0.0f)) limit = -1.0f;
  }
  static __device__ __noinline__ int exact(float x, float mn, float mx, int bits, float alpha, float eps) {
    MzQuantRow<MZ_F32> r;
    r.setup(mn, mx, bits, alpha, eps, nullptr, 0);
    return r.code(x);
  }
  __device__ __forceinline__ int code(float x, float mn, float mx, int bits, float alpha, float eps) const {
    const float s = __fmul_rn(__fsub_rn(x, lo), inv_span) - anchor;
    const bool up = s >= 0.0f;
    const float y = __log2f(fmaf(fabsf(s), up ? a_up : a_dn, 1.0f)) * (up ? k_up : k_dn);
    constexpr float magic = 12582912.0f;
    const float r = (y + magic) - magic;
    if (!(fabsf(y - r) < limit)) return exact(x, mn, mx, bits, alpha, eps);
    const float q = fminf(fmaxf(up ? zero_code + r : zero_code - r, 0.0f), top);
    return __float_as_int(q + magic) & 0x1ff;
  }
};
}  // namespace mzq
