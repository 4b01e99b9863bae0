// Store -> dense keys and values: a range of the packed prefix, optionally followed by the residual window, in one
// launch.  Bit-exact with the reference's fp32 dequantizer (muzero/quantizer.py:229-266).
// Measured (8 x 8 x 4224 tokens, head_dim 128, 4 bits, call included): 721 us as two dequantizers, conversions and
// concatenations, 65.6 us with every value evaluated, 61.0 us now (0.45 of the copy rate).
//
// head_dim 64 / 128, groups of 32 / 64 / 128 that divide it, 16-bit output: bound by HBM (the output is 4 to 16 times
// the packed input).  Keys are packed along tokens and written along channels, so a key tile is staged in shared
// memory and a thread takes two neighbouring channels of 16 tokens (one 4-byte store per token, 128 bytes per warp
// row); with codes of up to 4 bits each channel gets a 2^bits-entry book of finished 16-bit values, laid out entry-major
// so that the 32 lanes of a lookup always hit 32 different half-bank pairs.  Values are packed the way they are
// written; a thread takes 16 channels of a row.  Up to 4 bits the row's lanes share out the evaluation of its 2^bits entries and look
// them up by byte permute; wider codes are evaluated one by one.
#include "mz_quant_math.cuh"
#include "mz_store.cuh"

namespace {

struct DenseParams {
  mz_kv_store s;
  int g0, n_groups, t0, n_tok;            // packed ranges
  int res_k, res_v, v_skip;               // residual tokens appended to each side; values skip the window's first v_skip
  long long sk, sv;                       // output tokens per pair
  void* out_k; void* out_v;
  int QB, NG;
  float eps;
  const float* tab_k; const float* tab_v;
  unsigned b_key, b_kres, b_val, b_vres;  // CTAs of each part
  unsigned key_tiles, val_per_pair, kres_per_pair, vres_per_pair;
};

template <int DT> __device__ __forceinline__ uint32_t to16(float v) {
  return DT == MZ_BF16 ? (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(v)) : (uint32_t)__half_as_ushort(__float2half_rn(v));
}
template <int DT> __device__ __forceinline__ uint32_t pack16(float a, float b) {
  if (DT == MZ_BF16) { __nv_bfloat162 v = __floats2bfloat162_rn(a, b); return *reinterpret_cast<uint32_t*>(&v); }
  __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float meta16(const void* p, long long i, int dt) { return mz_load_as_float(p, i, dt); }

template <int DT, int BITS>
__device__ __forceinline__ void dense_keys(const DenseParams& p, uint8_t* smem) {
  constexpr bool BOOK = BITS <= 4;
  constexpr int NE = 1 << BITS, TPT = 16, CB = 2 * BITS;
  const mz_kv_store& s = p.s;
  const int G = s.group, D = s.head_dim, QB = p.QB, top = NE - 1;
  // a tile of more than 256 threads' worth of work (group 128 at head_dim 128) is walked in two steps
  const int pairs = D >> 1, parts = G / TPT, tt = pairs * parts, per_cta = tt >= 256 ? 1 : 256 / tt, rows = per_cta * D;
  const int tid = threadIdx.x, stride = QB + 8;
  float* s_row = (float*)smem;                               // wide codes: {lo, span, anchor, room_up, room_dn, zero code} x 256
  uint16_t* s_book = (uint16_t*)smem;                        // [NE][256]
  uint8_t* s_code = smem + (BOOK ? NE * 512 : 6 * 1024);
  const unsigned tile0 = blockIdx.x * per_cta;
  auto locate = [&](unsigned tile, int& j, int& h, int& b) {
    j = tile % p.n_groups; tile /= p.n_groups;
    h = tile % s.kv_heads; b = tile / s.kv_heads;
  };
  // i / wpr by multiplication: exact for i < 4096 and wpr <= 32
  const int words = D * QB / 4, wpr = QB / 4;
  const unsigned wpr_inv = ((1u << 20) + wpr - 1) / wpr;
  for (int l = 0; l < per_cta && tile0 + l < p.key_tiles; ++l) {
    int j, h, b;
    locate(tile0 + l, j, h, b);
    const uint32_t* src = (const uint32_t*)(s.packed_k + b * s.pk_stride_b + h * s.pk_stride_h + (long long)(p.g0 + j) * D * QB);
    for (int i = tid; i < words; i += 256) {
      const int d = (int)(((unsigned)i * wpr_inv) >> 20), w = i - d * wpr;
      *(uint32_t*)(s_code + (size_t)((d & 1) * per_cta * pairs + l * pairs + (d >> 1)) * stride + 4 * w) = __ldg(src + i);
    }
  }
  const int share = BOOK && rows == 128 ? 2 : 1;             // threads per row for the book
  if (tid < rows * share && tile0 + (tid % rows) / D < p.key_tiles) {
    const int row = tid % rows, half = tid / rows;
    int j, h, b;
    locate(tile0 + row / D, j, h, b);
    const long long m = b * s.km_stride_b + h * s.km_stride_h + (long long)(p.g0 + j) * D + row % D;
    const MzRowParams r = mz_row_params(meta16(s.k_mn, m, s.meta_dtype), meta16(s.k_scale, m, s.meta_dtype), top, p.eps);
    if (BOOK) {
      const int n = NE / share;
#pragma unroll 4
      for (int e = half * n; e < half * n + n; ++e) s_book[e * 256 + row] = (uint16_t)to16<DT>(mz_dequant_exact(r, e, p.tab_k, NE));
    } else {
      s_row[row] = r.lo; s_row[256 + row] = r.span; s_row[512 + row] = r.anchor; s_row[768 + row] = r.room_up;
      s_row[1024 + row] = r.room_dn; s_row[1280 + row] = __int_as_float(r.zero_code);
    }
  }
  __syncthreads();
  for (int w = tid; w < per_cta * tt; w += 256) {
    const int local = w / tt, part = (w % tt) / pairs, cp = w % pairs;
    if (tile0 + local >= p.key_tiles) break;
    int j, h, b;
    locate(tile0 + local, j, h, b);
    const uint8_t* ca = s_code + (size_t)(local * pairs + cp) * stride + part * CB;
    const uint8_t* cb = ca + (size_t)per_cta * pairs * stride;
    const int row = local * D + 2 * cp;
    const long long at = (((long long)b * s.kv_heads + h) * p.sk + (long long)j * G + part * TPT) * D + 2 * cp;
    if (!MZ_IN_BOUNDS(at + (TPT - 1) * D + 1, (long long)s.batch * s.kv_heads * p.sk * D, 18)) continue;
    uint32_t* dst = (uint32_t*)((uint16_t*)p.out_k + at);
    if (BOOK) {
      // 16 codes of each channel, LSB first
      unsigned long long a, c;
      if (BITS == 4) { a = *(const unsigned long long*)ca; c = *(const unsigned long long*)cb; }
      else if (BITS == 2) { a = *(const uint32_t*)ca; c = *(const uint32_t*)cb; }
      else {
        a = c = 0;
#pragma unroll
        for (int k = 0; k < BITS; ++k) {
          a |= (unsigned long long)*(const uint16_t*)(ca + 2 * k) << (16 * k);
          c |= (unsigned long long)*(const uint16_t*)(cb + 2 * k) << (16 * k);
        }
      }
#pragma unroll
      for (int i = 0; i < TPT; ++i) {
        const uint32_t ea = (uint32_t)(a >> (BITS * i)) & top, ec = (uint32_t)(c >> (BITS * i)) & top;
        dst[(size_t)i * pairs] = (uint32_t)s_book[ea * 256 + row] | ((uint32_t)s_book[ec * 256 + row + 1] << 16);
      }
    } else {
      MzRowParams r[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float* f = s_row + row + k;
        r[k].lo = f[0]; r[k].span = f[256]; r[k].anchor = f[512]; r[k].room_up = f[768]; r[k].room_dn = f[1024];
        r[k].zero_code = __float_as_int(f[1280]);
        r[k].steps_up = max(top - r[k].zero_code, 1); r[k].steps_dn = max(r[k].zero_code, 1);
      }
#pragma unroll
      for (int o = 0; o < TPT; o += 8) {
        unsigned long long a = 0, c = 0;
        if (BITS == 8) { a = *(const unsigned long long*)(ca + o); c = *(const unsigned long long*)(cb + o); }
        else {
#pragma unroll
          for (int k = 0; k < BITS; ++k) {
            a |= (unsigned long long)ca[(o >> 3) * BITS + k] << (8 * k);
            c |= (unsigned long long)cb[(o >> 3) * BITS + k] << (8 * k);
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float va = mz_dequant_exact(r[0], (int)(a >> (BITS * i)) & top, p.tab_k, NE);
          const float vc = mz_dequant_exact(r[1], (int)(c >> (BITS * i)) & top, p.tab_k, NE);
          dst[(size_t)(o + i) * pairs] = pack16<DT>(va, vc);
        }
      }
    }
  }
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}
// eight codes (LSB first) in the nibbles of a word
template <int BITS>
__device__ __forceinline__ uint32_t nibbles(uint32_t x) {
  if (BITS == 4) return x;
  if (BITS == 3) {
    x = (x & 0x00FFF000u) * 15u + x;
    x = (x & 0x0FC00FC0u) * 3u + x;
    return (x & 0x38383838u) + x;
  }
  if (BITS == 2) {
    x = (x | x << 8) & 0x00FF00FFu;
    x = (x | x << 4) & 0x0F0F0F0Fu;
    return (x | x << 2) & 0x33333333u;
  }
  x = (x | x << 12) & 0x000F000Fu;
  x = (x | x << 6) & 0x03030303u;
  return (x | x << 3) & 0x11111111u;
}
// eight codes -> eight 16-bit values, out of a book in registers (low and high bytes of its entries, four to a word)
template <int BITS, int N>
__device__ __forceinline__ uint4 book_values(uint32_t codes, const uint32_t (&lo)[N], const uint32_t (&hi)[N]) {
  const uint32_t x = nibbles<BITS>(codes);
  uint32_t v[4];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    uint32_t l, h;
    if (BITS == 4) {
      const uint32_t sel = (x >> (16 * k)) & 0x7777u, m = prmt(0u, 0xFFFFFFFFu, (x >> (16 * k + 1)) & 0x4444u);
      l = (prmt(lo[0], lo[1 % N], sel) & ~m) | (prmt(lo[N / 2], lo[N - 1], sel) & m);
      h = (prmt(hi[0], hi[1 % N], sel) & ~m) | (prmt(hi[N / 2], hi[N - 1], sel) & m);
    } else {
      const uint32_t sel = x >> (16 * k);
      l = prmt(lo[0], lo[N - 1], sel);
      h = prmt(hi[0], hi[N - 1], sel);
    }
    v[2 * k] = prmt(l, h, 0x5140u);
    v[2 * k + 1] = prmt(l, h, 0x7362u);
  }
  return make_uint4(v[0], v[1], v[2], v[3]);
}

// A CTA takes kValChunks x 256 / lanes-per-row rows; the codes and metadata of all of a thread's rows are in flight before the
// table is staged (one chunk per CTA spent most of its life in those two latencies).
constexpr int kValChunks = 4;
template <int DT, int BITS>
__device__ __forceinline__ void dense_values(const DenseParams& p, unsigned blk, uint8_t* smem) {
  constexpr int NE = 1 << BITS, top = NE - 1;
  const mz_kv_store& s = p.s;
  const int G = s.group, D = s.head_dim, NG = p.NG, lpr = G >> 4, rows = 256 / lpr;
  const unsigned pair = blk / p.val_per_pair, chunk = blk % p.val_per_pair;
  const int b = pair / s.kv_heads, h = pair % s.kv_heads;
  const int row0 = chunk * (rows * kValChunks) + threadIdx.x / lpr, sub = threadIdx.x % lpr, n_rows = p.n_tok * NG;
  const uint8_t* pv = s.packed_v + b * s.pv_stride_b + h * s.pv_stride_h;
  const long long m0 = b * s.vm_stride_b + h * s.vm_stride_h, at0 = (long long)p.t0 * NG;
  unsigned long long w[kValChunks][2];
  float lo[kValChunks], span[kValChunks];
#pragma unroll
  for (int k = 0; k < kValChunks; ++k) {
    const int row = min(row0 + k * rows, n_rows - 1);
    const uint8_t* src = pv + (at0 + row) * p.QB;
    w[k][0] = mz_load_octet(src + sub * BITS, BITS);
    w[k][1] = mz_load_octet(src + (sub + lpr) * BITS, BITS);
    lo[k] = meta16(s.v_mn, m0 + at0 + row, s.meta_dtype);
    span[k] = meta16(s.v_scale, m0 + at0 + row, s.meta_dtype);
  }
  const float* table = p.tab_v;
  if (BITS <= 4) {
    float* t = (float*)smem;
    for (int i = threadIdx.x; i < NE * NE; i += 256) t[i] = table[i];
    __syncthreads();
    table = t;
  }
#pragma unroll
  for (int k = 0; k < kValChunks; ++k) {
    const int row = row0 + k * rows;
    if (row >= n_rows) return;
    const MzRowParams r = mz_row_params(lo[k], span[k], top, p.eps);
    const long long at = (long long)pair * p.sv * D + (long long)row * G;
    if (!MZ_IN_BOUNDS(at + G - 1, (long long)s.batch * s.kv_heads * p.sv * D, 19)) continue;
    uint16_t* dst = (uint16_t*)p.out_v + at;
    if constexpr (BITS <= 4) {
      // the row's book of finished values, four entries to a word; its lanes (2, 4 or 8) share the words out.  16 codes per lane took 16
      // evaluations of the exact chain, 4 (4 bits in groups of 32: 8) and a permute lookup are what is left
      constexpr int N = NE < 4 ? 1 : NE / 4;
      const int share = min(lpr, N), lane = threadIdx.x & 31;
      uint32_t lo_own[2] = {0, 0}, hi_own[2] = {0, 0}, blo[N], bhi[N];
#pragma unroll
      for (int c = 0; c < (N == 4 ? 2 : 1); ++c) {
        const int word = sub % share + c * share;
        if (word >= N) break;
#pragma unroll
        for (int e = 0; e < 4 && e < NE; ++e) {
          const uint32_t v = to16<DT>(mz_dequant_exact(r, 4 * word + e, table, NE));
          lo_own[c] |= (v & 0xff) << (8 * e);
          hi_own[c] |= (v >> 8) << (8 * e);
        }
      }
      if (N == 1) {
        blo[0] = lo_own[0]; bhi[0] = hi_own[0];
      } else {
        const unsigned row_lanes = ((1u << lpr) - 1u) << (lane & ~(lpr - 1));
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const int from = (lane & ~(lpr - 1)) | (j % share);
          const bool second = j >= share;
          blo[j] = __shfl_sync(row_lanes, second ? lo_own[1] : lo_own[0], from);
          bhi[j] = __shfl_sync(row_lanes, second ? hi_own[1] : hi_own[0], from);
        }
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) *(uint4*)(dst + (sub + c * lpr) * 8) = book_values<BITS, N>((uint32_t)w[k][c], blo, bhi);
    } else {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          v[i] = pack16<DT>(mz_dequant_exact(r, (int)(w[k][c] >> (2 * i * BITS)) & top, table, NE),
                            mz_dequant_exact(r, (int)(w[k][c] >> ((2 * i + 1) * BITS)) & top, table, NE));
        *(uint4*)(dst + (sub + c * lpr) * 8) = make_uint4(v[0], v[1], v[2], v[3]);
      }
    }
  }
}

// residual rows -> the tail of the output, 16 bytes per thread
__device__ __forceinline__ void dense_residual(const mz_kv_store& s, const void* res, int first, int n, unsigned blk, unsigned per_pair,
                                               long long s_out, long long prefix, void* out) {
  const unsigned pair = blk / per_pair;
  const int i = (int)(blk % per_pair) * 256 + threadIdx.x, vpr = s.head_dim >> 3;
  if (i >= n * vpr) return;
  const int t = i / vpr, c = i % vpr;
  const int b = pair / s.kv_heads, h = pair % s.kv_heads;
  const long long at = (pair * s_out + prefix + t) * s.head_dim + c * 8;
  if (!MZ_IN_BOUNDS(at + 7, (long long)s.batch * s.kv_heads * s_out * s.head_dim, 20)) return;
  *(uint4*)((uint16_t*)out + at) =
      *(const uint4*)((const uint16_t*)res + b * s.res_stride_b + h * s.res_stride_h + (long long)(s.res_start + first + t) * s.res_stride_t + c * 8);
}

template <int DT, int BITS>
__global__ void __launch_bounds__(256) dense16_kernel(const DenseParams p) {
  extern __shared__ __align__(16) uint8_t s_dense[];
  unsigned blk = blockIdx.x;
  if (blk < p.b_key) { dense_keys<DT, BITS>(p, s_dense); return; }
  blk -= p.b_key;
  if (blk < p.b_val) { dense_values<DT, BITS>(p, blk, s_dense); return; }
  blk -= p.b_val;
  if (blk < p.b_kres) { dense_residual(p.s, p.s.res_k, 0, p.res_k, blk, p.kres_per_pair, p.sk, p.sk - p.res_k, p.out_k); return; }
  dense_residual(p.s, p.s.res_v, p.v_skip, p.res_v, blk - p.b_kres, p.vres_per_pair, p.sv, p.sv - p.res_v, p.out_v);
}

// ---- any shape: one thread per octet (keys: channel fastest; values: channel octets)
__global__ void __launch_bounds__(256) dequant_keys_kernel(const DenseParams p, int out_dt) {
  const mz_kv_store& s = p.s;
  const int G = s.group, D = s.head_dim, octs = (G + 7) >> 3, top = (1 << s.bits) - 1;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)p.n_groups * octs * D * s.batch * s.kv_heads) return;
  const int d = (int)(i % D); i /= D;
  const int oct = (int)(i % octs); i /= octs;
  const int g = p.g0 + (int)(i % p.n_groups); i /= p.n_groups;
  const int h = (int)(i % s.kv_heads);
  const int b = (int)(i / s.kv_heads);
  const long long m = b * s.km_stride_b + h * s.km_stride_h + (long long)g * D + d;
  const MzRowParams r = mz_row_params(mz_load_as_float(s.k_mn, m, s.meta_dtype), mz_load_as_float(s.k_scale, m, s.meta_dtype), top, p.eps);
  const uint8_t* row = s.packed_k + b * s.pk_stride_b + h * s.pk_stride_h + ((long long)g * D + d) * p.QB;
  const long long o0 = (((long long)b * s.kv_heads + h) * p.sk + (long long)(g - p.g0) * G + oct * 8) * D + d;
  const int n = min(8, G - oct * 8);
  if (!MZ_IN_BOUNDS(o0 + (long long)(n - 1) * D, (long long)s.batch * s.kv_heads * p.sk * D, 18)) return;
  for (int k = 0; k < n; ++k) {
    const int q = mz_extract_code(row, oct * 8 + k, s.bits, p.QB);
    mz_store_from_float(p.out_k, o0 + (long long)k * D, mz_dequant_exact(r, q, p.tab_k, top + 1), out_dt);
  }
}

__global__ void __launch_bounds__(256) dequant_values_kernel(const DenseParams p, int out_dt) {
  const mz_kv_store& s = p.s;
  const int G = s.group, D = s.head_dim, octs = (G + 7) >> 3, top = (1 << s.bits) - 1;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)s.batch * s.kv_heads * p.n_tok * p.NG * octs) return;
  const int oct = (int)(i % octs); i /= octs;
  const int grp = (int)(i % p.NG); i /= p.NG;
  const int t = (int)(i % p.n_tok); i /= p.n_tok;
  const int h = (int)(i % s.kv_heads);
  const int b = (int)(i / s.kv_heads);
  const long long at = (long long)(p.t0 + t) * p.NG + grp;
  const long long m = b * s.vm_stride_b + h * s.vm_stride_h + at;
  const MzRowParams r = mz_row_params(mz_load_as_float(s.v_mn, m, s.meta_dtype), mz_load_as_float(s.v_scale, m, s.meta_dtype), top, p.eps);
  const uint8_t* row = s.packed_v + b * s.pv_stride_b + h * s.pv_stride_h + at * p.QB;
  const long long o0 = (((long long)b * s.kv_heads + h) * p.sv + t) * D;
  for (int k = 0; k < 8; ++k) {
    const int idx = oct * 8 + k, c = grp * G + idx;
    if (idx >= G || c >= D || !MZ_IN_BOUNDS(o0 + c, (long long)s.batch * s.kv_heads * p.sv * D, 19)) break;
    const int q = mz_extract_code(row, idx, s.bits, p.QB);
    mz_store_from_float(p.out_v, o0 + c, mz_dequant_exact(r, q, p.tab_v, top + 1), out_dt);
  }
}

__global__ void __launch_bounds__(256) copy_residual_kernel(const mz_kv_store s, const uint16_t* res, int first, int n, long long s_out,
                                                            void* out, int out_dt) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int D = s.head_dim;
  if (i >= (long long)s.batch * s.kv_heads * n * D) return;
  const int d = (int)(i % D), t = (int)(i / D % n);
  const long long pair = i / D / n;
  const int b = (int)(pair / s.kv_heads), h = (int)(pair % s.kv_heads);
  const float v = mz_u16_to_float(res[b * s.res_stride_b + h * s.res_stride_h + (long long)(s.res_start + first + t) * s.res_stride_t + d], s.kv_dtype);
  const long long at = (pair * s_out + (s_out - n) + t) * D + d;
  if (MZ_IN_BOUNDS(at, (long long)s.batch * s.kv_heads * s_out * D, 20)) mz_store_from_float(out, at, v, out_dt);
}

template <int DT>
int launch_dense16(const DenseParams& p, cudaStream_t st) {
  const unsigned blocks = p.b_key + p.b_kres + p.b_val + p.b_vres;
  const int tt = (p.s.head_dim / 2) * (p.s.group / 16), per_cta = tt >= 256 ? 1 : 256 / tt;
  const size_t smem = (p.s.bits <= 4 ? (512u << p.s.bits) : 6144u) + (size_t)per_cta * p.s.head_dim * (p.QB + 8);
  switch (p.s.bits) {
    case 1: dense16_kernel<DT, 1><<<blocks, 256, smem, st>>>(p); break;
    case 2: dense16_kernel<DT, 2><<<blocks, 256, smem, st>>>(p); break;
    case 3: dense16_kernel<DT, 3><<<blocks, 256, smem, st>>>(p); break;
    case 4: dense16_kernel<DT, 4><<<blocks, 256, smem, st>>>(p); break;
    case 5: dense16_kernel<DT, 5><<<blocks, 256, smem, st>>>(p); break;
    case 6: dense16_kernel<DT, 6><<<blocks, 256, smem, st>>>(p); break;
    case 7: dense16_kernel<DT, 7><<<blocks, 256, smem, st>>>(p); break;
    default: dense16_kernel<DT, 8><<<blocks, 256, smem, st>>>(p); break;
  }
  MZ_LAUNCH_CHECK("dense16");
  return MZ_OK;
}

// p.g0 / n_groups / t0 / n_tok / res_* / v_skip / out_* are set; fills the rest and launches
int run_dense(DenseParams& p, int out_dtype, float eps, cudaStream_t st) {
  const mz_kv_store& s = p.s;
  const MzStoreGeom g = mz_geom(s);
  const long long pairs = (long long)g.B * g.KVH;
  p.QB = g.QB; p.NG = g.NG; p.eps = eps;
  p.sk = (long long)p.n_groups * g.G + p.res_k;
  p.sv = (long long)p.n_tok + p.res_v;
  p.tab_k = p.tab_v = nullptr;
  int rc;
  if (p.n_groups > 0 && (rc = mz_get_expand_table(g.bits, s.alpha_key, &p.tab_k))) return rc;
  if (p.n_tok > 0 && (rc = mz_get_expand_table(g.bits, s.alpha_value, &p.tab_v))) return rc;
  auto al = [](const void* q, int n) { return ((uintptr_t)q & (n - 1)) == 0; };
  const bool fast = (g.D == 64 || g.D == 128) && (g.G == 32 || g.G == 64 || g.G == 128) && g.D % g.G == 0 && out_dtype != MZ_F32 &&
                    (!(p.res_k | p.res_v) || (out_dtype == g.kv_dt && !((s.res_stride_b | s.res_stride_h | s.res_stride_t) & 7) &&
                                              al(s.res_k, 16) && al(s.res_v, 16))) &&
                    (!p.n_groups || (al(s.packed_k, 4) && !((s.pk_stride_b | s.pk_stride_h) & 3))) &&
                    (!p.n_tok || (al(s.packed_v, 8) && !((s.pv_stride_b | s.pv_stride_h) & 7))) &&
                    al(p.out_k, 16) && al(p.out_v, 16) && p.n_tok < (1 << 28);
  if (fast) {
    const int tt = (g.D / 2) * (g.G / 16), per_cta = tt >= 256 ? 1 : 256 / tt, rows_per_cta = 256 / (g.G / 16) * kValChunks, vpr = g.D / 8;
    const long long tiles = pairs * p.n_groups;
    p.val_per_pair = (unsigned)(((long long)p.n_tok * g.NG + rows_per_cta - 1) / rows_per_cta);
    p.kres_per_pair = (unsigned)((p.res_k * vpr + 255) / 256);
    p.vres_per_pair = (unsigned)((p.res_v * vpr + 255) / 256);
    const long long bk = (tiles + per_cta - 1) / per_cta, bv = pairs * p.val_per_pair, br = pairs * p.kres_per_pair, bs = pairs * p.vres_per_pair;
    MZ_REQUIRE(tiles < (1LL << 31) && bk + bv + br + bs < (1LL << 31), "problem too large");
    p.key_tiles = (unsigned)tiles;
    p.b_key = (unsigned)bk; p.b_val = (unsigned)bv; p.b_kres = (unsigned)br; p.b_vres = (unsigned)bs;
    if (bk + bv + br + bs == 0) return MZ_OK;
    return out_dtype == MZ_BF16 ? launch_dense16<MZ_BF16>(p, st) : launch_dense16<MZ_F16>(p, st);
  }
  if (p.n_groups > 0) {
    const long long n = pairs * p.n_groups * ((g.G + 7) / 8) * g.D;
    dequant_keys_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(p, out_dtype);
    MZ_LAUNCH_CHECK("dequant_keys");
  }
  if (p.n_tok > 0) {
    const long long n = pairs * p.n_tok * g.NG * ((g.G + 7) / 8);
    dequant_values_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(p, out_dtype);
    MZ_LAUNCH_CHECK("dequant_values");
  }
  if (p.res_k > 0) {
    const long long n = pairs * p.res_k * g.D;
    copy_residual_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(s, (const uint16_t*)s.res_k, 0, p.res_k, p.sk, p.out_k, out_dtype);
    MZ_LAUNCH_CHECK("copy_residual");
  }
  if (p.res_v > 0) {
    const long long n = pairs * p.res_v * g.D;
    copy_residual_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(s, (const uint16_t*)s.res_v, p.v_skip, p.res_v, p.sv, p.out_v, out_dtype);
    MZ_LAUNCH_CHECK("copy_residual");
  }
  return MZ_OK;
}
}  // namespace

extern "C" int mz_dequantize_kv(const mz_kv_store* s, int g0, int g1, void* out_k, int t0, int t1, void* out_v, int out_dtype,
                                float eps, void* stream) {
  MZ_RANGE("mz_dequantize_kv");
  int rc = mz_check_store_basic(s);
  if (rc) return rc;
  if ((rc = mz_check_store_quantized(s))) return rc;
  MZ_REQUIRE(mz_dtype_ok(out_dtype), "bad out_dtype");
  DenseParams p = {};
  p.s = *s; p.out_k = out_k; p.out_v = out_v;
  if (out_k && g1 > g0) {
    MZ_REQUIRE(g0 >= 0 && g1 <= s->k_groups, "key group range [%d,%d) outside [0,%d)", g0, g1, s->k_groups);
    p.g0 = g0; p.n_groups = g1 - g0;
  }
  if (out_v && t1 > t0) {
    MZ_REQUIRE(t0 >= 0 && t1 <= s->v_tokens, "value token range [%d,%d) outside [0,%d)", t0, t1, s->v_tokens);
    p.t0 = t0; p.n_tok = t1 - t0;
  }
  return run_dense(p, out_dtype, eps, (cudaStream_t)stream);
}

extern "C" int mz_materialize_kv(const mz_kv_store* s, void* out_k, void* out_v, int out_dtype, float eps, void* stream) {
  MZ_RANGE("mz_materialize_kv");
  int rc = mz_check_store_basic(s);
  if (rc) return rc;
  const int lead = s->v_tokens - s->k_groups * s->group;
  MZ_REQUIRE(lead >= 0 && lead <= s->res_len, "value prefix (%d tokens) must cover the key prefix (%d tokens) and end inside the residual window (%d tokens)",
             s->v_tokens, s->k_groups * s->group, s->res_len);
  if (s->v_tokens > 0 && (rc = mz_check_store_quantized(s))) return rc;
  if (s->res_len > 0 && (rc = mz_check_store_residual(s))) return rc;
  MZ_REQUIRE(out_k && out_v && mz_dtype_ok(out_dtype), "bad output");
  DenseParams p = {};
  p.s = *s; p.out_k = out_k; p.out_v = out_v;
  p.n_groups = s->k_groups; p.n_tok = s->v_tokens;
  p.res_k = s->res_len; p.res_v = s->res_len - lead; p.v_skip = lead;
  return run_dense(p, out_dtype, eps, (cudaStream_t)stream);
}
