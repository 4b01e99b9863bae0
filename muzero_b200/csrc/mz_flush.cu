// Residual-window flush and single-token append.
//
// Flush is one launch.  flush16_kernel below serves the usual shapes; any other takes flush_kv_kernel: the first n_k CTAs each take one key tile
// [G tokens x D channels] of one (b, kvh): the tile is staged in shared memory
// with 16-byte row loads, then one thread per channel reduces min/max down its
// column, quantizes it and writes the packed row straight into the store (the
// transpose never touches global memory).  The remaining CTAs quantize value
// rows (G contiguous channels of one token) with G/8 lanes per row.
#include "mz_quant16.cuh"
#include "mz_store.cuh"

namespace {

// the rows of the window that a flush leaves dense, copied to a new window (dst_k == nullptr: not asked for)
struct MoveParams {
  uint16_t* dst_k; uint16_t* dst_v;
  long long sb, sh, st;      // element strides of the new window
  int k_first, v_first;      // first key / value row that stays; key row k_first becomes row 0 of the new window
  // checked build: element `rel` of head h's rows lies inside the head's slab (heads outermost) or the batch entry's
  __device__ __forceinline__ bool holds(int h, long long rel) const {
    return sh >= st ? MZ_IN_BOUNDS(rel, sh, 23) : MZ_IN_BOUNDS(h * sh + rel, sb, 23);
  }
};

struct FlushParams {
  mz_kv_store s;
  MoveParams mv;
  int n_tiles;               // key tiles (groups of G tokens) to flush, from the window's first token
  int v_first, n_vtokens;    // value tokens to flush: window rows [v_first, v_first + n_vtokens)
  int QB, NG;
  float eps;
  const uint16_t* ctab_k; int ctab_k_n;
  const uint16_t* ctab_v; int ctab_v_n;
  unsigned n_k_blocks;
  long long v_rows;          // B*KVH*n_vtokens*NG
  int v_fast;                // G/8 lanes per value row, D % 8 == 0
  int k_vec;                 // key tile rows can be loaded as 16-byte vectors
};

template <int DT>
__device__ void flush_key_tile(const FlushParams& p, uint16_t* tile) {
  const mz_kv_store& s = p.s;
  const int G = s.group, D = s.head_dim;
  unsigned blk = blockIdx.x;
  const int j = blk % p.n_tiles; blk /= p.n_tiles;
  const int h = blk % s.kv_heads;
  const int b = blk / s.kv_heads;
  const uint16_t* src = (const uint16_t*)s.res_k + b * s.res_stride_b + h * s.res_stride_h +
                        (long long)(s.res_start + j * G) * s.res_stride_t;
  if (p.k_vec) {
    const int vec_per_row = D >> 3;
    for (int i = threadIdx.x; i < G * vec_per_row; i += blockDim.x) {
      const int t = i / vec_per_row, c = i % vec_per_row;
      ((uint4*)tile)[i] = *(const uint4*)(src + (long long)t * s.res_stride_t + c * 8);
    }
  } else {
    for (int i = threadIdx.x; i < G * D; i += blockDim.x) tile[i] = src[(long long)(i / D) * s.res_stride_t + (i % D)];
  }
  __syncthreads();
  const int grp = s.k_groups + j;
  uint8_t* dst_rows = s.packed_k + b * s.pk_stride_b + h * s.pk_stride_h + (long long)grp * D * p.QB;
  const long long meta0 = b * s.km_stride_b + h * s.km_stride_h + (long long)grp * D;
  // checked build: the last byte of this group's rows and its last metadata element lie inside the pair's slab
  if (!MZ_IN_BOUNDS((long long)(grp + 1) * D * p.QB - 1, s.pk_stride_h, 1) ||
      !MZ_IN_BOUNDS((long long)(grp + 1) * D - 1, s.km_stride_h, 2)) return;
  // A channel's G tokens are split over `parts` threads when the CTA has more threads than channels (2 for
  // head_dim 128 and 256 threads): partial min/max meet in shared memory, then each thread quantizes and packs
  // its own share of the row (whole octets, so the byte ranges of the parts do not overlap).
  const int parts = (blockDim.x >= 2 * D && G % 16 == 0) ? 2 : 1;
  float* red = (float*)(tile + ((G * D + 1) & ~1));          // [parts][2][D]
  const int share = G / parts;
  for (int idx = threadIdx.x; idx < D * parts; idx += blockDim.x) {
    const int d = idx % D, part = idx / D;
    float mn = INFINITY, mx = -INFINITY;
    for (int t = part * share; t < (part + 1) * share; ++t) {
      const float v = mz_u16_to_float(tile[t * D + d], DT);
      mn = fminf(mn, v); mx = fmaxf(mx, v);
    }
    red[(part * 2) * D + d] = mn;
    red[(part * 2 + 1) * D + d] = mx;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < D * parts; idx += blockDim.x) {
    const int d = idx % D, part = idx / D;
    float mn = red[d], mx = red[D + d];
    if (parts == 2) { mn = fminf(mn, red[2 * D + d]); mx = fmaxf(mx, red[3 * D + d]); }
    MzQuantRow<DT> r;
    r.setup(mn, mx, s.bits, s.alpha_key, p.eps, p.ctab_k, p.ctab_k_n);
    uint8_t* dst = dst_rows + (long long)d * p.QB;
    for (int t0 = part * share; t0 < (part + 1) * share; t0 += 8) {
      const int n = min(8, (part + 1) * share - t0);
      unsigned long long word = 0;
      for (int k = 0; k < n; ++k)
        word |= ((unsigned long long)r.code(mz_u16_to_float(tile[(t0 + k) * D + d], DT))) << (k * s.bits);
      uint8_t* o = dst + (t0 >> 3) * s.bits;
      if (n == 8) mz_store_octet(o, word, s.bits);
      else {
        const int nb = (n * s.bits + 7) >> 3;
        for (int i = 0; i < nb; ++i) o[i] = (uint8_t)(word >> (8 * i));
      }
    }
    if (part == 0) {
      mz_store_from_float(s.k_mn, meta0 + d, r.lo, s.meta_dtype);
      mz_store_from_float(s.k_scale, meta0 + d, r.span, s.meta_dtype);
    }
  }
}

// value rows, G/8 lanes per row (G power of two in 8..256, D % 8 == 0)
template <int DT>
__device__ void flush_value_rows_fast(const FlushParams& p) {
  const mz_kv_store& s = p.s;
  const int G = s.group, D = s.head_dim, lpr = G >> 3;
  const int rows_per_cta = blockDim.x / lpr;
  const int sub = threadIdx.x % lpr;
  const long long row = (long long)(blockIdx.x - p.n_k_blocks) * rows_per_cta + threadIdx.x / lpr;
  const bool live = row < p.v_rows;
  long long r = live ? row : 0;
  const int grp = (int)(r % p.NG); r /= p.NG;
  const int t = (int)(r % p.n_vtokens); r /= p.n_vtokens;
  const int h = (int)(r % s.kv_heads);
  const int b = (int)(r / s.kv_heads);
  const int c0 = grp * G + sub * 8;
  float v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = 0.f;
  if (live && c0 < D) {
    const uint16_t* src = (const uint16_t*)s.res_v + b * s.res_stride_b + h * s.res_stride_h +
                          (long long)(s.res_start + p.v_first + t) * s.res_stride_t + c0;
    if (p.k_vec) {
      const uint4 raw = *(const uint4*)src;
      const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[2 * i] = mz_u16_to_float((uint16_t)(w[i] & 0xffffu), DT);
        v[2 * i + 1] = mz_u16_to_float((uint16_t)(w[i] >> 16), DT);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = mz_u16_to_float(src[i], DT);
    }
  }
  float mn = v[0], mx = v[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) { mn = fminf(mn, v[i]); mx = fmaxf(mx, v[i]); }
  for (int off = lpr >> 1; off > 0; off >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, off));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  }
  if (!live) return;
  MzQuantRow<DT> q;
  q.setup(mn, mx, s.bits, s.alpha_value, p.eps, p.ctab_v, p.ctab_v_n);
  unsigned long long word = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) word |= ((unsigned long long)q.code(v[i])) << (i * s.bits);
  const long long tok = s.v_tokens + t;
  uint8_t* dst = s.packed_v + b * s.pv_stride_b + h * s.pv_stride_h + (tok * p.NG + grp) * p.QB + sub * s.bits;
  if (!MZ_IN_BOUNDS((tok * p.NG + grp + 1) * p.QB - 1, s.pv_stride_h, 3) || !MZ_IN_BOUNDS(tok * p.NG + grp, s.vm_stride_h, 4)) return;
  mz_store_octet(dst, word, s.bits);
  if (sub == 0) {
    const long long m = b * s.vm_stride_b + h * s.vm_stride_h + tok * p.NG + grp;
    mz_store_from_float(s.v_mn, m, q.lo, s.meta_dtype);
    mz_store_from_float(s.v_scale, m, q.span, s.meta_dtype);
  }
}

// value rows, any G / D: one warp per row, bits written one byte at a time
template <int DT>
__device__ void flush_value_rows_generic(const FlushParams& p) {
  const mz_kv_store& s = p.s;
  const int G = s.group, D = s.head_dim;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long row = (long long)(blockIdx.x - p.n_k_blocks) * (blockDim.x >> 5) + warp;
  if (row >= p.v_rows) return;
  long long r = row;
  const int grp = (int)(r % p.NG); r /= p.NG;
  const int t = (int)(r % p.n_vtokens); r /= p.n_vtokens;
  const int h = (int)(r % s.kv_heads);
  const int b = (int)(r / s.kv_heads);
  const uint16_t* src = (const uint16_t*)s.res_v + b * s.res_stride_b + h * s.res_stride_h +
                        (long long)(s.res_start + p.v_first + t) * s.res_stride_t;
  float mn = INFINITY, mx = -INFINITY;
  for (int i = lane; i < G; i += 32) {
    const int c = grp * G + i;
    const float v = c < D ? mz_u16_to_float(src[c], DT) : 0.f;
    mn = fminf(mn, v); mx = fmaxf(mx, v);
  }
  for (int off = 16; off > 0; off >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, off));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  }
  MzQuantRow<DT> q;
  q.setup(mn, mx, s.bits, s.alpha_value, p.eps, p.ctab_v, p.ctab_v_n);
  const long long tok = s.v_tokens + t;
  uint8_t* dst = s.packed_v + b * s.pv_stride_b + h * s.pv_stride_h + (tok * p.NG + grp) * p.QB;
  if (!MZ_IN_BOUNDS((tok * p.NG + grp + 1) * p.QB - 1, s.pv_stride_h, 5) || !MZ_IN_BOUNDS(tok * p.NG + grp, s.vm_stride_h, 6)) return;
  for (int byte = lane; byte < p.QB; byte += 32) {
    uint32_t out = 0;
    const int first = (byte * 8) / s.bits, last = min(G - 1, (byte * 8 + 7) / s.bits);
    for (int i = first; i <= last; ++i) {
      const int c = grp * G + i;
      const uint32_t code = (uint32_t)q.code(c < D ? mz_u16_to_float(src[c], DT) : 0.f);
      const int sh = i * s.bits - byte * 8;
      out |= sh >= 0 ? (code << sh) : (code >> (-sh));
    }
    dst[byte] = (uint8_t)out;
  }
  if (lane == 0) {
    const long long m = b * s.vm_stride_b + h * s.vm_stride_h + tok * p.NG + grp;
    mz_store_from_float(s.v_mn, m, q.lo, s.meta_dtype);
    mz_store_from_float(s.v_scale, m, q.span, s.meta_dtype);
  }
}

template <int DT>
__global__ void __launch_bounds__(256) flush_kv_kernel(const FlushParams p) {
  extern __shared__ __align__(16) uint16_t s_tile[];
  if (blockIdx.x < p.n_k_blocks) flush_key_tile<DT>(p, s_tile);
  else if (p.v_fast) flush_value_rows_fast<DT>(p);
  else flush_value_rows_generic<DT>(p);
}

// ---- head_dim 64 / 128, groups of 32 / 64 / 128 that divide it: the packed quantizer (mz_quant16.cuh).
//
// Bound by instruction issue (HBM traffic is 2.6 bytes per value at 4 bits): the point of the layout is that every
// step works on two values per register and that nothing is staged that can stay in registers.
//   keys    a thread owns two neighbouring channels (the two halves of a register) of TPT tokens, so the loads of a
//           warp are whole 128-byte rows and the transpose happens in the packing; the parts of a channel meet in
//           shared memory for the min / max, one thread per channel then prepares the row (metadata, reciprocal,
//           thresholds) and the finished codes go through shared memory into whole-line stores
//   values  a thread owns 16 channels of one row (two 16-byte loads), G / 16 lanes per row, shuffles for min / max
struct Flush16Params {
  mz_kv_store s;
  int n_tiles;               // key tiles per pair
  int v_first, n_vtokens;    // value tokens: window rows [v_first, v_first + n_vtokens)
  float eps;
  const uint16_t* thr_k; const uint16_t* thr_v;
  const uint16_t* ctab_k; const uint16_t* ctab_v; int ctab_k_n, ctab_v_n;
  unsigned n_k_blocks, tiles;       // key CTAs; key tiles in all
  unsigned v_blocks_per_pair;
  unsigned n_v_blocks, mv_per_pair;   // value CTAs; CTAs per pair of the rows that stay
  MoveParams mv;
};

template <int DT, int BITS, int TPT>
__device__ __forceinline__ void flush16_keys(const Flush16Params& p, uint8_t* smem) {
  using P = mzq::P2<DT>;
  constexpr bool WIDE = BITS > 4;
  constexpr int NT = WIDE ? 1 : (1 << BITS) - 1;
  constexpr int CB = TPT * BITS / 8;                      // packed bytes of one channel in one thread
  const mz_kv_store& s = p.s;
  const int G = s.group, D = s.head_dim, QB = G * BITS / 8;
  const int pairs = D >> 1, parts = G / TPT, tt = pairs * parts, per_cta = 256 / tt, rows = per_cta * D;
  const int tid = threadIdx.x;
  const int local = tid / tt, part = (tid % tt) / pairs, cp = tid % pairs;
  // shared memory: partial min / max, row constants, thresholds (or the wide rows' constants), code tile
  uint32_t* red = (uint32_t*)smem;                        // [per_cta][parts][2][pairs]
  float* s_inv = (float*)(red + 512);                     // [rows]
  float* s_span = s_inv + 256;                            // [rows], negative: special row
  uint16_t* s_lo = (uint16_t*)(s_span + 256);             // [rows]
  uint32_t* s_thr = (uint32_t*)(s_lo + 256);              // [NT][rows / 2] pairs, or floats [8][rows]
  uint8_t* s_code = (uint8_t*)(s_thr + (WIDE ? 8 * 256 : NT * 128));   // even channels, then odd ones, padded rows
  const int stride = QB + 8;
  const unsigned tile0 = blockIdx.x * per_cta;
  auto locate = [&](unsigned tile, int& j, int& h, int& b) {
    j = tile % p.n_tiles; tile /= p.n_tiles;
    h = tile % s.kv_heads; b = tile / s.kv_heads;
  };
  const bool live = tile0 + local < p.tiles;
  uint32_t x[TPT];
  const uint16_t* src = nullptr;
  if (live) {
    int j, h, b;
    locate(tile0 + local, j, h, b);
    src = (const uint16_t*)s.res_k + b * s.res_stride_b + h * s.res_stride_h + (long long)(s.res_start + j * G + part * TPT) * s.res_stride_t + 2 * cp;
    uint32_t mn = P::INF2, mx = P::INF2 | 0x80008000u;
#pragma unroll
    for (int i = 0; i < TPT; ++i) x[i] = *(const uint32_t*)(src + i * s.res_stride_t);
#pragma unroll
    for (int i = 0; i < TPT; ++i) { mn = P::mn(mn, x[i]); mx = P::mx(mx, x[i]); }
    red[((local * parts + part) * 2) * pairs + cp] = mn;
    red[((local * parts + part) * 2 + 1) * pairs + cp] = mx;
  }
  __syncthreads();
  if (tid < rows && tile0 + tid / D < p.tiles) {
    const int l = tid / D, d = tid % D;
    const uint16_t* r16 = (const uint16_t*)(red + l * parts * 2 * pairs);
    float mn = mz_u16_to_float(r16[d], DT), mx = mz_u16_to_float(r16[D + d], DT);
    for (int k = 1; k < parts; ++k) {
      mn = fminf(mn, mz_u16_to_float(r16[2 * k * D + d], DT));
      mx = fmaxf(mx, mz_u16_to_float(r16[(2 * k + 1) * D + d], DT));
    }
    mzq::RowHead<DT> head;
    head.set(mn, mx, p.eps);
    s_inv[tid] = head.inv_span;
    s_span[tid] = head.special ? -1.0f : head.span;
    s_lo[tid] = (uint16_t)(P::pack(head.lo, head.lo) & 0xffffu);
    if constexpr (WIDE) {
      mzq::WideRow<DT> w;
      w.set(mz_u16_to_float((uint16_t)head.anchor_bits, DT), (float)((1 << BITS) - 1), MzType<DT>::round(p.eps));
      float* f = (float*)s_thr + tid;
      f[0] = w.anchor; f[256] = w.zero_code; f[512] = w.steps_up; f[768] = w.steps_dn;
      f[1024] = w.room_up; f[1280] = w.room_dn; f[1536] = w.inv_up; f[1792] = w.inv_dn;
    } else {
      const uint16_t* t = p.thr_k + ((size_t)(head.special ? 0 : head.anchor_bits) << BITS);
      uint16_t* o = (uint16_t*)s_thr + tid;
      if constexpr (BITS == 4) {
        const uint4 a = *(const uint4*)t, b = *(const uint4*)(t + 8);
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int k = 0; k < NT; ++k) o[k * 256] = (uint16_t)(w[k >> 1] >> ((k & 1) * 16));
      } else {
#pragma unroll
        for (int k = 0; k < NT; ++k) o[k * 256] = t[k];
      }
    }
    int j, h, b;
    locate(tile0 + l, j, h, b);
    const long long grp = s.k_groups + j;
    if (MZ_IN_BOUNDS((grp + 1) * D - 1, s.km_stride_h, 2)) {
      const long long m = b * s.km_stride_b + h * s.km_stride_h + grp * D + d;
      mz_store_from_float(s.k_mn, m, head.lo, s.meta_dtype);
      mz_store_from_float(s.k_scale, m, head.span, s.meta_dtype);
    }
  }
  __syncthreads();
  if (live) {
    const int row = local * D + 2 * cp;
    const uint32_t lo2 = *(const uint32_t*)(s_lo + row);
    const float2 inv = *(const float2*)(s_inv + row), span = *(const float2*)(s_span + row);
    uint8_t* dst = s_code + (size_t)(local * pairs + cp) * stride + part * CB;
    uint8_t* dst_odd = dst + (size_t)per_cta * pairs * stride;
    if (span.x < 0.f || span.y < 0.f) {
      // a row outside the packed path's domain: value by value
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        float mn = INFINITY, mx = -INFINITY;
        const uint16_t* r16 = (const uint16_t*)(red + local * parts * 2 * pairs);
        for (int k = 0; k < parts; ++k) {
          mn = fminf(mn, mz_u16_to_float(r16[2 * k * D + 2 * cp + c], DT));
          mx = fmaxf(mx, mz_u16_to_float(r16[(2 * k + 1) * D + 2 * cp + c], DT));
        }
        MzQuantRow<DT> r;
        r.setup(mn, mx, BITS, s.alpha_key, p.eps, p.ctab_k, p.ctab_k_n);
#pragma unroll 1
        for (int t0 = 0; t0 < TPT; t0 += 8) {
          unsigned long long word = 0;
#pragma unroll 1
          for (int k = 0; k < 8; ++k)
            word |= ((unsigned long long)r.code(mz_u16_to_float(src[(t0 + k) * s.res_stride_t + c], DT))) << (k * BITS);
          for (int k = 0; k < BITS; ++k) (c ? dst_odd : dst)[(t0 >> 3) * BITS + k] = (uint8_t)(word >> (8 * k));
        }
      }
    } else if constexpr (!WIDE) {
      mzq::Thresholds<DT, BITS> th;
#pragma unroll
      for (int k = 0; k < NT; ++k) th.T[k] = s_thr[k * 128 + (row >> 1)];
#pragma unroll
      for (int t0 = 0; t0 < TPT; t0 += 16) {
        unsigned long long ca = 0, cb = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t xx[4] = {x[t0 + 4 * q], x[t0 + 4 * q + 1], x[t0 + 4 * q + 2], x[t0 + 4 * q + 3]};
          uint32_t u[4];
          mzq::units_of<DT, 4>(xx, lo2, inv.x, inv.y, span.x, span.y, u);
          // four codes of each channel in the two halves
          const uint32_t acc = th.template codes<0>(u[0]) | th.template codes<BITS>(u[1]) |
                               th.template codes<2 * BITS>(u[2]) | th.template codes<3 * BITS>(u[3]);
          ca |= (unsigned long long)(acc & 0xffffu) << (4 * BITS * q);
          cb |= (unsigned long long)(acc >> 16) << (4 * BITS * q);
        }
        uint8_t* da = dst + t0 * BITS / 8;
        uint8_t* db = dst_odd + t0 * BITS / 8;
        if (BITS == 4) { *(unsigned long long*)da = ca; *(unsigned long long*)db = cb; }
        else if (BITS == 2) { *(uint32_t*)da = (uint32_t)ca; *(uint32_t*)db = (uint32_t)cb; }
        else {
#pragma unroll
          for (int k = 0; k < BITS; ++k) {
            *(uint16_t*)(da + 2 * k) = (uint16_t)(ca >> (16 * k));
            *(uint16_t*)(db + 2 * k) = (uint16_t)(cb >> (16 * k));
          }
        }
      }
    } else {
      mzq::WideRow<DT> ra, rb;
      const float* f = (const float*)s_thr + row;
      ra = {f[0], f[256], f[512], f[768], f[1024], f[1280], f[1536], f[1792]};
      rb = {f[1], f[257], f[513], f[769], f[1025], f[1281], f[1537], f[1793]};
#pragma unroll
      for (int t0 = 0; t0 < TPT; t0 += 8) {
        unsigned long long ca = 0, cb = 0;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const uint32_t xx[4] = {x[t0 + 4 * q], x[t0 + 4 * q + 1], x[t0 + 4 * q + 2], x[t0 + 4 * q + 3]};
          uint32_t u[4];
          mzq::units_of<DT, 4>(xx, lo2, inv.x, inv.y, span.x, span.y, u);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t one = P::ONE | (P::ONE << 16);
            // a NaN value has code 0
            const uint32_t nn = P::ge(u[k], 0u);
            const uint32_t c = mzq::wide_codes<DT>(P::mn(P::mx(u[k], 0u), one), ra, rb, (float)((1 << BITS) - 1), p.ctab_k) & nn;
            ca |= (unsigned long long)(c & 0xffffu) << (BITS * (4 * q + k));
            cb |= (unsigned long long)(c >> 16) << (BITS * (4 * q + k));
          }
        }
        uint8_t* da = dst + (t0 >> 3) * BITS;
        uint8_t* db = dst_odd + (t0 >> 3) * BITS;
        if (BITS == 8) { *(unsigned long long*)da = ca; *(unsigned long long*)db = cb; }
        else {
#pragma unroll
          for (int k = 0; k < BITS; ++k) { da[k] = (uint8_t)(ca >> (8 * k)); db[k] = (uint8_t)(cb >> (8 * k)); }
        }
      }
    }
  }
  __syncthreads();
  // code tile -> store: the D rows of a tile are contiguous there
  // i / wpr by multiplication: exact for i < 4096 and wpr <= 32
  const int words = D * QB / 4, wpr = QB / 4;
  const unsigned wpr_inv = ((1u << 20) + wpr - 1) / wpr;
  for (int l = 0; l < per_cta && tile0 + l < p.tiles; ++l) {
    int j, h, b;
    locate(tile0 + l, j, h, b);
    const long long grp = s.k_groups + j;
    if (!MZ_IN_BOUNDS((grp + 1) * D * QB - 1, s.pk_stride_h, 1)) continue;
    uint32_t* out = (uint32_t*)(s.packed_k + b * s.pk_stride_b + h * s.pk_stride_h + grp * D * QB);
    for (int i = tid; i < words; i += 256) {
      const int d = (int)(((unsigned)i * wpr_inv) >> 20), w = i - d * wpr;
      out[i] = *(const uint32_t*)(s_code + (size_t)((d & 1) * per_cta * pairs + l * pairs + (d >> 1)) * stride + 4 * w);
    }
  }
}

template <int DT, int BITS>
__device__ __forceinline__ void flush16_values(const Flush16Params& p) {
  const mz_kv_store& s = p.s;
  const int G = s.group, D = s.head_dim, NG = D / G, QB = G * BITS / 8, lpr = G >> 4;
  const unsigned blk = blockIdx.x - p.n_k_blocks;
  const unsigned pair = blk / p.v_blocks_per_pair, chunk = blk % p.v_blocks_per_pair;
  const int b = pair / s.kv_heads, h = pair % s.kv_heads;
  const int r = chunk * (256 / lpr) + threadIdx.x / lpr, sub = threadIdx.x % lpr;   // row inside the pair: token * NG + group
  const bool live = r < p.n_vtokens * NG;
  const int t = live ? r / NG : 0, grp = live ? r % NG : 0;
  uint32_t x[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (live) {
    const uint16_t* src = (const uint16_t*)s.res_v + b * s.res_stride_b + h * s.res_stride_h +
                          (long long)(s.res_start + p.v_first + t) * s.res_stride_t + grp * G + sub * 8;
    const uint4 a = *(const uint4*)src, c = *(const uint4*)(src + lpr * 8);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = c.x; x[5] = c.y; x[6] = c.z; x[7] = c.w;
  }
  mzq::RowHead<DT> head;
  unsigned long long word[2];
  mzq::quantize_row16<DT, BITS>(x, lpr, s.alpha_value, p.eps, p.thr_v, p.ctab_v, p.ctab_v_n, head, word);
  if (!live) return;
  const long long row = (long long)(s.v_tokens + t) * NG + grp;
  if (!MZ_IN_BOUNDS((row + 1) * QB - 1, s.pv_stride_h, 3) || !MZ_IN_BOUNDS(row, s.vm_stride_h, 4)) return;
  uint8_t* dst = s.packed_v + b * s.pv_stride_b + h * s.pv_stride_h + row * QB + sub * BITS;
  mz_store_octet(dst, word[0], BITS);
  mz_store_octet(dst + lpr * BITS, word[1], BITS);
  if (sub == 0) {
    const long long m = b * s.vm_stride_b + h * s.vm_stride_h + row;
    mz_store_from_float(s.v_mn, m, head.lo, s.meta_dtype);
    mz_store_from_float(s.v_scale, m, head.span, s.meta_dtype);
  }
}

// rows that stay dense: 16 bytes of the key row and of the value row per thread
__device__ __forceinline__ void move_rows16(const mz_kv_store& s, const MoveParams& m, unsigned blk, unsigned per_pair) {
  const unsigned pair = blk / per_pair;
  const int vpr = s.head_dim >> 3, i = (int)(blk % per_pair) * 256 + threadIdx.x, row = m.k_first + i / vpr, c = (i % vpr) * 8;
  if (row >= s.res_len) return;
  const int b = pair / s.kv_heads, h = pair % s.kv_heads;
  const long long src = b * s.res_stride_b + h * s.res_stride_h + (long long)(s.res_start + row) * s.res_stride_t + c;
  if (!m.holds(h, (long long)(row - m.k_first) * m.st + c + 7)) return;
  const long long dst = b * m.sb + h * m.sh + (long long)(row - m.k_first) * m.st + c;
  *(uint4*)(m.dst_k + dst) = *(const uint4*)((const uint16_t*)s.res_k + src);
  if (row >= m.v_first) *(uint4*)(m.dst_v + dst) = *(const uint4*)((const uint16_t*)s.res_v + src);
}

template <int DT, int BITS, int TPT>
__global__ void __launch_bounds__(256) flush16_kernel(const Flush16Params p) {
  extern __shared__ __align__(16) uint8_t s_flush[];
  if (blockIdx.x < p.n_k_blocks) flush16_keys<DT, BITS, TPT>(p, s_flush);
  else if (blockIdx.x < p.n_k_blocks + p.n_v_blocks) flush16_values<DT, BITS>(p);
  else move_rows16(p.s, p.mv, blockIdx.x - p.n_k_blocks - p.n_v_blocks, p.mv_per_pair);
}

__global__ void __launch_bounds__(256) move_rows_kernel(const mz_kv_store s, const MoveParams m) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int D = s.head_dim, nk = s.res_len - m.k_first;
  if (i >= (long long)s.batch * s.kv_heads * nk * D) return;
  const int d = (int)(i % D), row = (int)(i / D % nk) + m.k_first;
  const long long pair = i / D / nk;
  const long long src = (pair / s.kv_heads) * s.res_stride_b + (pair % s.kv_heads) * s.res_stride_h + (long long)(s.res_start + row) * s.res_stride_t + d;
  const long long dst = (pair / s.kv_heads) * m.sb + (pair % s.kv_heads) * m.sh + (long long)(row - m.k_first) * m.st + d;
  if (!m.holds((int)(pair % s.kv_heads), (long long)(row - m.k_first) * m.st + d)) return;
  m.dst_k[dst] = ((const uint16_t*)s.res_k)[src];
  if (row >= m.v_first) m.dst_v[dst] = ((const uint16_t*)s.res_v)[src];
}

__global__ void append_kv_kernel(const mz_kv_store s, const uint16_t* __restrict__ k_new, const uint16_t* __restrict__ v_new,
                                 long long nsb, long long nsh) {
  // launched as a programmatic dependent: nothing is read or written before the previous kernel has completed,
  // and the next kernel (the decode attention) may start its own prologue right away
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int D = s.head_dim;
  const long long n = (long long)s.batch * s.kv_heads * D;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int d = (int)(i % D);
  const int h = (int)((i / D) % s.kv_heads);
  const int b = (int)(i / ((long long)D * s.kv_heads));
  const long long dst = b * s.res_stride_b + h * s.res_stride_h + (long long)(s.res_start + s.res_len) * s.res_stride_t + d;
  const long long src = b * nsb + h * nsh + d;
  ((uint16_t*)s.res_k)[dst] = k_new[src];
  ((uint16_t*)s.res_v)[dst] = v_new[src];
}

bool pow2(int v) { return v > 0 && (v & (v - 1)) == 0; }

bool flush16_serves(const mz_kv_store& s, const FlushParams& p) {
  return (s.head_dim == 64 || s.head_dim == 128) && (s.group == 32 || s.group == 64 || s.group == 128) && s.head_dim % s.group == 0 &&
         p.k_vec && ((uintptr_t)s.packed_k & 3) == 0 && ((s.pk_stride_b | s.pk_stride_h) & 3) == 0 && p.n_vtokens < (1 << 28);
}
template <int DT, int BITS>
int launch_flush16(const Flush16Params& p, unsigned blocks, cudaStream_t st) {
  const int per_cta = 256 / ((p.s.head_dim / 2) * (p.s.group / (p.s.group == 128 ? 32 : 16)));
  const size_t smem = 2048 + 2 * 1024 + 512 + (BITS > 4 ? 8192 : ((1 << BITS) - 1) * 512) +
                      (size_t)per_cta * p.s.head_dim * (p.s.group * BITS / 8 + 8);
  if (p.s.group == 128) flush16_kernel<DT, BITS, 32><<<blocks, 256, smem, st>>>(p);
  else flush16_kernel<DT, BITS, 16><<<blocks, 256, smem, st>>>(p);
  MZ_LAUNCH_CHECK("flush16");
  return MZ_OK;
}
template <int DT>
int launch_flush16_bits(const Flush16Params& p, unsigned blocks, cudaStream_t st) {
  switch (p.s.bits) {
    case 1: return launch_flush16<DT, 1>(p, blocks, st);
    case 2: return launch_flush16<DT, 2>(p, blocks, st);
    case 3: return launch_flush16<DT, 3>(p, blocks, st);
    case 4: return launch_flush16<DT, 4>(p, blocks, st);
    case 5: return launch_flush16<DT, 5>(p, blocks, st);
    case 6: return launch_flush16<DT, 6>(p, blocks, st);
    case 7: return launch_flush16<DT, 7>(p, blocks, st);
    default: return launch_flush16<DT, 8>(p, blocks, st);
  }
}
// *done = 0 when the thresholds table is not available: the caller takes the per-value kernel
int flush16(const mz_kv_store& s, const FlushParams& f, cudaStream_t st, int* done) {
  Flush16Params p;
  p.s = s; p.n_tiles = f.n_tiles; p.v_first = f.v_first; p.n_vtokens = f.n_vtokens; p.eps = f.eps;
  p.ctab_k = f.ctab_k; p.ctab_k_n = f.ctab_k_n; p.ctab_v = f.ctab_v; p.ctab_v_n = f.ctab_v_n;
  p.thr_k = p.thr_v = nullptr;
  int rc;
  if (s.bits <= 4) {
    if ((rc = mz_get_unit_thresholds(s.kv_dtype, s.bits, s.alpha_key, f.eps, &p.thr_k))) return rc;
    if ((rc = mz_get_unit_thresholds(s.kv_dtype, s.bits, s.alpha_value, f.eps, &p.thr_v))) return rc;
    if (!p.thr_k || !p.thr_v) return MZ_OK;
  }
  const int tpt = s.group == 128 ? 32 : 16, per_cta = 256 / ((s.head_dim / 2) * (s.group / tpt));
  const long long pairs = (long long)s.batch * s.kv_heads, tiles = pairs * p.n_tiles;
  const int rows_per_cta = 256 / (s.group / 16);
  p.v_blocks_per_pair = (unsigned)(((long long)p.n_vtokens * (s.head_dim / s.group) + rows_per_cta - 1) / rows_per_cta);
  const long long kb = (tiles + per_cta - 1) / per_cta, vb = pairs * p.v_blocks_per_pair;
  p.mv = f.mv;
  p.mv_per_pair = f.mv.dst_k ? (unsigned)(((s.res_len - f.mv.k_first) * (s.head_dim / 8) + 255) / 256) : 0;
  const long long mb = pairs * p.mv_per_pair;
  if (tiles >= (1LL << 31) || kb + vb + mb >= (1LL << 31)) return MZ_OK;
  p.tiles = (unsigned)tiles; p.n_k_blocks = (unsigned)kb; p.n_v_blocks = (unsigned)vb;
  *done = 1;
  return s.kv_dtype == MZ_BF16 ? launch_flush16_bits<MZ_BF16>(p, (unsigned)(kb + vb + mb), st) : launch_flush16_bits<MZ_F16>(p, (unsigned)(kb + vb + mb), st);
}
}  // namespace

namespace {
int flush(const mz_kv_store* s, int n_key_tokens, int value_first, int n_value_tokens, float eps, const MoveParams& mv, void* stream) {
  int rc = mz_check_store_basic(s);
  if (rc) return rc;
  if ((rc = mz_check_store_quantized(s))) return rc;
  if ((rc = mz_check_store_residual(s))) return rc;
  MZ_REQUIRE(n_key_tokens >= 0 && n_key_tokens % s->group == 0, "n_key_tokens %d is not a multiple of group %d", n_key_tokens,
             s->group);
  MZ_REQUIRE(n_key_tokens <= s->res_len, "flush of %d key tokens but residual holds %d", n_key_tokens, s->res_len);
  MZ_REQUIRE(value_first >= 0 && n_value_tokens >= 0 && value_first + n_value_tokens <= s->res_len,
             "value tokens [%d, %d) outside the residual window of %d", value_first, value_first + n_value_tokens, s->res_len);
  if (n_key_tokens == 0 && n_value_tokens == 0) return MZ_OK;
  const MzStoreGeom g = mz_geom(*s);
  FlushParams p;
  p.s = *s; p.n_tiles = n_key_tokens / g.G; p.v_first = value_first; p.n_vtokens = n_value_tokens;
  p.QB = g.QB; p.NG = g.NG; p.eps = eps; p.mv = mv;
  if ((rc = mz_get_compand_table(g.kv_dt, s->alpha_key, &p.ctab_k, &p.ctab_k_n))) return rc;
  if ((rc = mz_get_compand_table(g.kv_dt, s->alpha_value, &p.ctab_v, &p.ctab_v_n))) return rc;
  const long long kb = (long long)g.B * g.KVH * p.n_tiles;
  p.v_rows = (long long)g.B * g.KVH * n_value_tokens * g.NG;
  p.v_fast = pow2(g.G) && g.G >= 8 && g.G <= 256 && g.D % 8 == 0;
  p.k_vec = g.D % 8 == 0 && s->res_stride_t % 8 == 0 && s->res_stride_h % 8 == 0 && s->res_stride_b % 8 == 0 &&
            (uintptr_t)s->res_k % 16 == 0 && (uintptr_t)s->res_v % 16 == 0;
  const bool mv_vec = !mv.dst_k || ((((uintptr_t)mv.dst_k | (uintptr_t)mv.dst_v) & 15) == 0 && ((mv.sb | mv.sh | mv.st) & 7) == 0);
  if (mv_vec && flush16_serves(*s, p)) {
    int done = 0;
    if ((rc = flush16(*s, p, (cudaStream_t)stream, &done)) || done) return rc;
  }
  const int rows_per_cta = p.v_fast ? 256 / (g.G / 8) : 8;
  const long long vb = (p.v_rows + rows_per_cta - 1) / rows_per_cta;
  MZ_REQUIRE(kb + vb < (1LL << 31), "flush too large");
  p.n_k_blocks = (unsigned)kb;
  const size_t smem = (size_t)((g.G * g.D + 1) & ~1) * 2 + (size_t)g.D * 4 * sizeof(float);   // key tile + partial min/max of two parts
  if (smem > 200 * 1024) return mz_fail(MZ_ERR_UNSUPPORTED, "key tile of %zu bytes exceeds shared memory", smem);
  cudaStream_t st = (cudaStream_t)stream;
  if (g.kv_dt == MZ_BF16) {
    if (smem > 48 * 1024) MZ_CUDA(cudaFuncSetAttribute(flush_kv_kernel<MZ_BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    flush_kv_kernel<MZ_BF16><<<(unsigned)(kb + vb), 256, smem, st>>>(p);
  } else {
    if (smem > 48 * 1024) MZ_CUDA(cudaFuncSetAttribute(flush_kv_kernel<MZ_F16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    flush_kv_kernel<MZ_F16><<<(unsigned)(kb + vb), 256, smem, st>>>(p);
  }
  MZ_LAUNCH_CHECK("flush_kv");
  if (mv.dst_k && s->res_len > mv.k_first) {
    const long long n = (long long)g.B * g.KVH * (s->res_len - mv.k_first) * g.D;
    MZ_REQUIRE((n + 255) / 256 < (1LL << 31), "window too large");
    move_rows_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(*s, mv);
    MZ_LAUNCH_CHECK("move_rows");
  }
  return MZ_OK;
}
}  // namespace

extern "C" int mz_flush_kv_parts(const mz_kv_store* s, int n_key_tokens, int value_first, int n_value_tokens, float eps,
                                 void* stream) {
  MZ_RANGE("mz_flush_kv_parts");
  return flush(s, n_key_tokens, value_first, n_value_tokens, eps, MoveParams{}, stream);
}

extern "C" int mz_flush_kv_move(const mz_kv_store* s, int n_key_tokens, int value_first, int n_value_tokens, void* dst_k, void* dst_v,
                                long long dst_stride_b, long long dst_stride_h, long long dst_stride_t, float eps, void* stream) {
  MZ_RANGE("mz_flush_kv_move");
  MZ_REQUIRE(s != nullptr && dst_k && dst_v && dst_stride_t >= s->head_dim, "bad destination window");
  const MoveParams mv = {(uint16_t*)dst_k, (uint16_t*)dst_v, dst_stride_b, dst_stride_h, dst_stride_t, n_key_tokens, value_first + n_value_tokens};
  MZ_REQUIRE(n_key_tokens + n_value_tokens > 0 && mv.v_first >= mv.k_first, "nothing to flush, or values behind the keys");
  return flush(s, n_key_tokens, value_first, n_value_tokens, eps, mv, stream);
}

extern "C" int mz_flush_kv(const mz_kv_store* s, int n_tokens, float eps, void* stream) {
  return mz_flush_kv_parts(s, n_tokens, 0, n_tokens, eps, stream);
}

extern "C" int mz_append_kv(const mz_kv_store* s, const void* k_new, const void* v_new, long long nsb, long long nsh, void* stream) {
  MZ_RANGE("mz_append_kv");
  int rc = mz_check_store_basic(s);
  if (rc) return rc;
  if ((rc = mz_check_store_residual(s))) return rc;
  MZ_REQUIRE(k_new && v_new, "NULL new token pointer");
  const long long n = (long long)s->batch * s->kv_heads * s->head_dim;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((n + 255) / 256));
  cfg.blockDim = dim3(256);
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  MZ_CUDA(cudaLaunchKernelEx(&cfg, append_kv_kernel, *s, (const uint16_t*)k_new, (const uint16_t*)v_new, nsb, nsh));
  MZ_LAUNCH_CHECK("append_kv");
  return MZ_OK;
}
