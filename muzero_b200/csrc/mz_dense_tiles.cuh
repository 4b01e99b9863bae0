// Residual (un-quantized) tiles of 16 tokens on mma.sync, head_dim HD (64 or 128): one warp walks the tiles of a plan that has no packed
// tiles and leaves a partial record per (batch, kv head) pair.  A tile is a short latency-bound chain (3 us), so a launch
// gives these warps CTAs of their own beside the packed tiles'.
//
// M rows are tokens (keys) / channels (values); B columns are 4 heads x {query or probability rounded to 16 bits, remainder}.  A bf16
// probability has a third part, and products go to a fresh accumulator that is added in round-to-nearest (the tensor cores truncate their
// running sums), so that no more is lost than to fp32.
#pragma once
#include "mz_mma_common.cuh"

namespace mzd {
using namespace mzm;
constexpr int DT = 16;                      // tokens per tile
constexpr int TILE_BYTES = DT * (2 * 128 + 16);            // rows are padded (bank spread)
constexpr int PROB_BYTES = DT * 16;         // probabilities [16 tokens][4 heads]
constexpr int WARP_BYTES = 2 * TILE_BYTES + PROB_BYTES;

// warp `gw` of plan `tp`; `buf` is the shared-window address of its WARP_BYTES, records from `first_record` (in records of one head) on
template <int HD, int GQA>
__device__ __forceinline__ void dense_tiles(const MzDecodeParams& p, const MzTilesPlan& tp, long long first_record, int gw, uint32_t buf) {
  constexpr int STRIDE = 2 * HD + 16, PIECES = HD / 8;
  const mz_kv_store& s = p.s;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int hq = g >> 1;                    // head whose query and probabilities this lane supplies (B column g)
  const bool bf = s.kv_dtype == MZ_BF16;
  const uint32_t kbuf = buf, vbuf = buf + TILE_BYTES, dbuf = buf + 2 * TILE_BYTES;
  const int T = tp.tiles_per_pair;
  const int nq = s.k_groups * G;
  long long f0 = 0, f1 = 0;
  if (gw < tp.total_warps) mz_warp_tiles(tp, gw, &f0, &f1);
  if (f0 >= f1) return;

  struct Cursor { int pair, tile, b, kvh; };
  auto advance = [&](Cursor& c) {
    if (++c.tile == T) {
      c.tile = 0; ++c.pair;
      if (++c.kvh == s.kv_heads) { c.kvh = 0; ++c.b; }
    }
  };
  // up to 16 rows of HD elements; rows past the end are zeroed (they meet probability 0, which must not meet a NaN bit pattern).  The
  // newest token may still be in the caller's tensors (p.new_k / new_v): it is staged from there, and stored into the window
  auto stage = [&](uint32_t dst, void* window, const void* fresh, const Cursor& c, bool valid) {
    if (valid) {
      const int tok0 = c.tile * DT, ntok = min(DT, s.res_len - tok0), kvh = c.kvh >> p.kv_share;
      const int newest = fresh != nullptr ? s.res_len - 1 - tok0 : -1;
      uint16_t* src = (uint16_t*)window + c.b * s.res_stride_b + kvh * s.res_stride_h + (long long)(s.res_start + tok0) * s.res_stride_t;
      for (int i = lane; i < DT * PIECES; i += 32) {
        const int row = i / PIECES, k = i % PIECES;
        if (row < ntok) {
          const uint16_t* from = src + (long long)row * s.res_stride_t + k * 8;
          if (row == newest) {
            from = (const uint16_t*)fresh + c.b * p.new_sb + kvh * p.new_sh + k * 8;
            if (kvh << p.kv_share == c.kvh && MZ_IN_BOUNDS(s.res_start + tok0 + row, p.new_rows, 15))
              *(uint4*)(src + (long long)row * s.res_stride_t + k * 8) = *(const uint4*)from;
          }
          cp16(dst + row * STRIDE + k * 16, from);
        } else sts128(dst + row * STRIDE + k * 16, make_uint4(0, 0, 0, 0));
      }
    }
    cp_async_commit();
  };

  float out[HD / 16][4];    // M tile m: channels (m < 4 ? 0 : 64) + 8g + 2(m%4) + {0,1}, head t, columns {value, remainder}
  float m_st = -INFINITY, l_st = 0.f;       // softmax state of head t (l: this lane's tokens only)
  int cur_pair = -1, seg = 0;
  auto reset = [&]() {
#pragma unroll
    for (int m = 0; m < HD / 16; ++m)
#pragma unroll
      for (int k = 0; k < 4; ++k) out[m][k] = 0.f;
    m_st = -INFINITY; l_st = 0.f;
  };
  auto write_partial = [&]() {
    float lsum = l_st;
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, off);
    if (t < GQA) {
      const long long slot = first_record + ((long long)gw * tp.max_segs + seg) * GQA + t;
      if (!MZ_IN_BOUNDS(slot, p.part.slots, 10)) return;
      float* dst = p.part.acc + slot * HD + 8 * g;
#pragma unroll
      for (int h = 0; h < HD / 32; ++h)     // channels 0..3, 4..7 of the lower and of the upper half
        *(float4*)(dst + (h >> 1) * 64 + (h & 1) * 4) = make_float4(out[2 * h][0] + out[2 * h][1], out[2 * h][2] + out[2 * h][3],
                                                                    out[2 * h + 1][0] + out[2 * h + 1][1], out[2 * h + 1][2] + out[2 * h + 1][3]);
      if (g == 0) {
        p.part.m[slot] = m_st * (1.0f / LOG2E);   // back to natural-log units
        p.part.l[slot] = lsum;
      }
    }
  };

  Cursor cur;
  cur.pair = (int)((unsigned)f0 / (unsigned)T); cur.tile = (int)((unsigned)f0 % (unsigned)T);
  cur.b = cur.pair / s.kv_heads; cur.kvh = cur.pair % s.kv_heads;
  Cursor nxt = cur;
  stage(kbuf, s.res_k, p.new_k, cur, true);
  stage(vbuf, s.res_v, p.new_v, cur, true);
  reset();
  const uint16_t* qrow = nullptr;
  for (int left = (int)(f1 - f0); left > 0; --left, cur = nxt) {
    advance(nxt);
    if (cur.pair != cur_pair) {
      if (cur_pair >= 0) { write_partial(); ++seg; }
      cur_pair = cur.pair;
      reset();
      qrow = (const uint16_t*)p.query + cur.b * p.q_stride_b + (long long)(cur.kvh * GQA + min(hq, GQA - 1)) * p.q_stride_h;
    }
    const int tok0 = cur.tile * DT, ntok = min(DT, s.res_len - tok0);
    cp_async_wait<1>();
    warp_sync();
    // ---- keys
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    const bool fold_lane = (g & 1) == 0 && hq < GQA;
#pragma unroll
    for (int j = 0; j < HD / 16; ++j) {
      const uint32_t ka = kbuf + g * STRIDE + (16 * j + 2 * t) * 2;
      const uint32_t a0 = lds32(ka), a1 = lds32(ka + 8 * STRIDE), a2 = lds32(ka + 16), a3 = lds32(ka + 8 * STRIDE + 16);
      const uint32_t b0 = fold_lane ? *(const uint32_t*)(qrow + 16 * j + 2 * t) : 0u;
      const uint32_t b1 = fold_lane ? *(const uint32_t*)(qrow + 16 * j + 8 + 2 * t) : 0u;
      float part[4];
      if (bf) mma_bf16_first(part, a0, a1, a2, a3, b0, b1);
      else mma_f16_first(part, a0, a1, a2, a3, b0, b1);
      add4(acc, part);
    }
    warp_sync();
    stage(kbuf, s.res_k, p.new_k, nxt, left > 1);
    // ---- softmax: this lane has head t, tokens g and g + 8
    float sv[2] = {acc[0] * p.scaling * LOG2E, acc[2] * p.scaling * LOG2E};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (g + 8 * i >= ntok) sv[i] = -INFINITY;
      else if (p.mask) sv[i] += mz_load_as_float(p.mask, cur.b * p.mask_stride_b + nq + tok0 + g + 8 * i, p.mask_dtype) * LOG2E;
    }
    float mx = fmaxf(sv[0], sv[1]);
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    const float m_new = fmaxf(m_st, mx);
    const bool dead = !(m_new > -INFINITY);
    sv[0] = dead ? 0.f : ex2f(sv[0] - m_new);
    sv[1] = dead ? 0.f : ex2f(sv[1] - m_new);
    const float c = dead ? 1.0f : ex2f(m_st - m_new);   // m_st = -inf -> 0
    l_st = l_st * c + sv[0] + sv[1];
    m_st = m_new;
    if (__any_sync(0xffffffffu, c != 1.0f)) {
#pragma unroll
      for (int m = 0; m < HD / 16; ++m)
#pragma unroll
        for (int k = 0; k < 4; ++k) out[m][k] *= c;
    }
    if (t < GQA) {
      stsf(dbuf + (g * 4 + t) * 4, sv[0]);
      stsf(dbuf + ((g + 8) * 4 + t) * 4, sv[1]);
    }
    cp_async_wait<1>();
    warp_sync();
    // ---- values: B holds the probabilities of head hq, rounded (even columns) and what that dropped (odd columns); bf16: b3 what that
    // dropped again (even columns)
    uint32_t bb[2], b3[2];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float pv[2], rest[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float pf = hq < GQA ? ldsf(dbuf + ((2 * t + 8 * half + k) * 4 + hq) * 4) : 0.f;
        const float hi = bf ? __bfloat162float(__float2bfloat16_rn(pf)) : __half2float(__float2half_rn(pf));
        pv[k] = (g & 1) ? pf - hi : hi;
        rest[k] = (g & 1) ? 0.f : (pf - hi) - __bfloat162float(__float2bfloat16_rn(pf - hi));
      }
      if (bf) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(pv[0], pv[1]), w = __floats2bfloat162_rn(rest[0], rest[1]);
        bb[half] = *reinterpret_cast<const uint32_t*>(&v);
        b3[half] = *reinterpret_cast<const uint32_t*>(&w);
      } else {
        bb[half] = h2_bits(__floats2half2_rn(pv[0], pv[1]));
        b3[half] = 0u;
      }
    }
#pragma unroll
    for (int grp = 0; grp < HD / 64; ++grp) {
      const uint32_t va = vbuf + (2 * t) * STRIDE + (grp * 64 + 8 * g) * 2;
      const uint4 x0 = lds128(va), x1 = lds128(va + STRIDE), x2 = lds128(va + 8 * STRIDE), x3 = lds128(va + 9 * STRIDE);
      const uint32_t c0[4] = {x0.x, x0.y, x0.z, x0.w}, c1[4] = {x1.x, x1.y, x1.z, x1.w};
      const uint32_t c2[4] = {x2.x, x2.y, x2.z, x2.w}, c3[4] = {x3.x, x3.y, x3.z, x3.w};
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        // rows g / g + 8 = channels 8g + 2m / 8g + 2m + 1; columns = tokens (2t, 2t + 1) and (2t + 8, 2t + 9)
        const uint32_t a0 = prmt(c0[m], c1[m], 0x5410u), a1 = prmt(c0[m], c1[m], 0x7632u);
        const uint32_t a2 = prmt(c2[m], c3[m], 0x5410u), a3 = prmt(c2[m], c3[m], 0x7632u);
        float part[4];
        if (bf) {
          mma_bf16_first(part, a0, a1, a2, a3, b3[0], b3[1]);
          mma_bf16(part, a0, a1, a2, a3, bb[0], bb[1]);
        } else {
          mma_f16_first(part, a0, a1, a2, a3, bb[0], bb[1]);
        }
        add4(out[grp * 4 + m], part);
      }
    }
    warp_sync();
    stage(vbuf, s.res_v, p.new_v, nxt, left > 1);
  }
  cp_async_wait<0>();
  write_partial();
}
}  // namespace mzd
