// Helpers shared by the two tensor-core decode kernels (mma.sync and tcgen05): shared memory by
// shared-window address, the replicated lookup table, the per-row constants of the folded dequantizer.
#pragma once
#include "mz_tiles_common.cuh"

namespace mzm {
using mzt::cp_async_commit;
using mzt::cp_async_wait;
using mzt::D;
using mzt::ex2f;
using mzt::LOG2E;
using mzt::prmt;

constexpr int G = 64;                       // tokens per packed tile
constexpr uint32_t TBL = 65536;             // shared-window address of the lookup table

// ---- shared memory by shared-window address (no generic-address arithmetic in the loops) ----
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t lds8(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ float ldsf(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory"); }
__device__ __forceinline__ void sts16(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(a), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ void sts8(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u8 [%0], %1;" ::"r"(a), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ void stsf(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
__device__ __forceinline__ void sts128(uint32_t a, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void cp16(uint32_t sa, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(g) : "memory");
}
__device__ __forceinline__ void warp_sync() { __syncwarp(); }

// D(16x8, fp32) += A(16x16) * B(16x8), 16-bit operands of the named type; the _first forms start from zero
__device__ __forceinline__ void mma_f16_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mma_bf16_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// c += t * f, rounded to nearest
__device__ __forceinline__ void fma4(float (&c)[4], const float (&t)[4], float f) {
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 z, {%8, %8};\n\t"
      "mov.b64 x, {%0, %1};\n\tmov.b64 y, {%4, %5};\n\tfma.rn.f32x2 x, y, z, x;\n\tmov.b64 {%0, %1}, x;\n\t"
      "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%6, %7};\n\tfma.rn.f32x2 x, y, z, x;\n\tmov.b64 {%2, %3}, x;\n\t}"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "f"(t[0]), "f"(t[1]), "f"(t[2]), "f"(t[3]), "f"(f));
}
// c += t, rounded to nearest (the tensor cores' own accumulation truncates)
__device__ __forceinline__ void add4(float (&c)[4], const float (&t)[4]) {
  asm("{\n\t.reg .b64 x, y;\n\t"
      "mov.b64 x, {%0, %1};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t"
      "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%6, %7};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%2, %3}, x;\n\t}"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "f"(t[0]), "f"(t[1]), "f"(t[2]), "f"(t[3]));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ __half2 dup_lo(uint32_t v) { return __half2half2(__low2half(bits_h2(v))); }
__device__ __forceinline__ __half2 dup_hi(uint32_t v) { return __half2half2(__high2half(bits_h2(v))); }

// ---- the lookup table at shared-window address TBL: entry (zc, e) -> half2(u+, u-), one copy per lane for the
// keys' alpha (first 128 bytes of an entry's 256) and for the values' alpha (second 128 bytes).  The idle half
// of an entry carries the fp16 remainder of the active half, pre-scaled by the nominal ratio Bdn / Bup of a row
// in that zero-code bin (anchor at the bin centre); the end bins have codes on one side only and row_constants
// makes their two constants equal.  Called by every thread of the CTA; the caller synchronises afterwards.
// entry idx = (zc, e) of the table for `alpha`, as the bits of half2(u+, u-)
template <int BITS>
__device__ __forceinline__ uint32_t lookup_entry(float alpha, int idx) {
  constexpr int NE = 1 << BITS, TOP = NE - 1;
  const int zc = idx >> BITS, e = idx & TOP;
  const float lb = log1pf(alpha);
  const float zac = (float)zc / (float)TOP;    // middle of the bin
  const float ratio = (zc == 0 || zc == TOP) ? 1.0f : zac / (1.0f - zac);
  __half2 ent;
  if (e >= zc) {
    const int up = max(TOP - zc, 1);
    const float u = expm1f((float)min(e - zc, up) / (float)up * lb) / alpha;
    const float uh = __half2float(__float2half_rn(u));
    ent = __floats2half2_rn(uh, (u - uh) / ratio);
  } else {
    const int dn = max(zc, 1);
    const float u = -expm1f((float)(zc - e) / (float)dn * lb) / alpha;
    const float uh = __half2float(__float2half_rn(u));
    ent = __floats2half2_rn((u - uh) * ratio, uh);
  }
  return h2_bits(ent);
}
// entry idx = (zc, e) of the general kernel's table: half2(u+, u-) rounded, and what the rounding dropped
template <int BITS>
__device__ __forceinline__ uint2 split_entry(float alpha, int idx) {
  constexpr int NE = 1 << BITS, TOP = NE - 1;
  const int zc = idx >> BITS, e = idx & TOP;
  const int room = max(e >= zc ? TOP - zc : zc, 1), n = min(abs(e - zc), room);
  const float grow = expm1f((float)n / (float)room * log1pf(alpha)) / alpha, u = e >= zc ? grow : -grow;
  const __half h = __float2half_rn(u), l = __float2half_rn(u - __half2float(h)), z = __ushort_as_half(0);
  return e >= zc ? make_uint2(h2_bits(__halves2half2(h, z)), h2_bits(__halves2half2(l, z)))
                 : make_uint2(h2_bits(__halves2half2(z, h)), h2_bits(__halves2half2(z, l)));
}
// stores one entry to the 32 lane copies of its slot half (rotated so that the lanes of a warp, which hold
// consecutive entries, hit different banks)
__device__ __forceinline__ void store_entry_copies(uint32_t row, uint32_t bits) {
#pragma unroll 4
  for (int c = 0; c < 32; ++c) sts32(row + (((c + threadIdx.x) & 31) << 2), bits);
}
template <int BITS>
__device__ __forceinline__ void fill_lookup_table(float alpha_key, float alpha_value) {
  constexpr int NE = 1 << BITS;
  // one table when keys and values use the same alpha (the usual case): each entry is computed once and stored
  // to both halves of its 256-byte slot
  const bool same = alpha_key == alpha_value;
  const int n = same ? NE * NE : 2 * NE * NE;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int which = i / (NE * NE), idx = i % (NE * NE);
    const uint32_t bits = lookup_entry<BITS>(which ? alpha_value : alpha_key, idx);
    store_entry_copies(TBL + idx * 256 + which * 128, bits);
    if (same) store_entry_copies(TBL + idx * 256 + 128, bits);
  }
}
// the same table from a copy in global memory: [2][NE * NE] entries (keys' alpha, values' alpha), built once
// per device and (bits, alphas) by the host side
template <int BITS>
__device__ __forceinline__ void fill_lookup_table_from(const uint32_t* __restrict__ entries) {
  constexpr int NE = 1 << BITS;
  for (int i = threadIdx.x; i < 2 * NE * NE; i += blockDim.x) {
    const int which = i / (NE * NE), idx = i % (NE * NE);
    store_entry_copies(TBL + idx * 256 + which * 128, entries[i]);
  }
}

// ---- per-row constants of the folded dequantizer: value(code e) = A + Bup * u+[zc][e] + Bdn * u-[zc][e].
// A is the value of the zero code: exactly 0 when the row's range straddles zero, up to the rounding of the
// anchor (a few 2^-24 of |lo|), which is dropped.  IEEE division and multiply: the zero code must round exactly
// as the dequantizer's does.
template <int BITS>
__device__ __forceinline__ void row_constants(float lo, float span, int& zc, float& A, float& Bup, float& Bdn) {
  constexpr int TOP = (1 << BITS) - 1;
  float anchor = __fdiv_rn(__fsub_rn(0.0f, lo), fmaxf(span, 1e-8f));
  anchor = fminf(fmaxf(anchor, 0.0f), 1.0f);
  zc = __float2int_rn(__fmul_rn(anchor, (float)TOP));
  A = fmaf(span, anchor, lo);
  if (fabsf(A) <= 9.5367431640625e-7f * fmaxf(fabsf(lo), span)) A = 0.0f;
  Bup = fminf(span * fmaxf(1.0f - anchor, 1e-8f), 65504.f);
  Bdn = fminf(span * fmaxf(anchor, 1e-8f), 65504.f);
  // a row whose zero code is the first / last code has no codes on the other side: that side's constant only
  // ever multiplies the remainder half of the table entries
  if (zc == 0) Bdn = Bup;
  if (zc == TOP) Bup = Bdn;
}
// ---- row constants: Bdn = clamp(-lo, 0, span) is the part of the range below zero, Bup the part above, A the value of the
// zero code (0 when the range straddles zero).  The zero code is rint(RN(RN(-lo / span) * TOP)) as the dequantizer has it.
// The quotient takes Markstein's final step (IBM J. Res. Dev. 34(1), 1990), q0 + (b - q0 s) y with y close to 1/s, which is
// branch-free, where the IEEE division costs a range test and a slow path per row.  Ties matter: 16-bit extremes often give
// a quotient that lies exactly on a code boundary.  For 16-bit metadata the step is correctly rounded whatever the last bits of
// y: b and s have at most 11 significant bits, so b/s is at least 2^-13 ulp away from every rounding boundary (a quotient
// with 25 bits would need a dividend of more than 11), and the step's value before rounding is within 2^-20 ulp of b/s.
// fp32 metadata has no such gap: its rows, and spans from 2^125 on, which would flush the reciprocal, take the
// division (`wild`).
__device__ __forceinline__ void row_split(float lo, float span, float top, float& A, float& bup, float& bdn, int& zc, bool& wild) {
  span = fmaxf(span, 1e-8f);
  bdn = fminf(fmaxf(-lo, 0.0f), span);
  bup = span - bdn;
  A = lo + bdn;
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(span));
  y = fmaf(fmaf(-span, y, 1.0f), y, y);
  const float q0 = bdn * y;
  const float q = fmaf(fmaf(-q0, span, bdn), y, q0);
  const float pos = __fmul_rn(q, top), r = pos + 12582912.0f;
  zc = __float_as_int(r) & 0xff;
  wild |= !(span < 4e37f);
}
__device__ __forceinline__ int exact_zero_code(float lo, float span, float top) {
  const float anchor = fminf(fmaxf(__fdiv_rn(__fsub_rn(0.0f, lo), fmaxf(span, 1e-8f)), 0.0f), 1.0f);
  return __float2int_rn(__fmul_rn(anchor, top));
}
}  // namespace mzm
