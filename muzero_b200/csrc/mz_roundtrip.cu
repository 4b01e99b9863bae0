// Quantize -> dequantize of a 16-bit K or V block in fp32 (the quality tool's path), without materialising fp32 rows,
// a transposed copy, codes or metadata.  Bound by instruction issue (about 40 per value, most of them the exact
// dequantizer); HBM traffic is the block once in and once out.
// One launch for a K and a V block (either may be absent): the two halves fill each other's last waves.
// Keys: thread = two neighbouring channels of 16 tokens, the parts of a channel meet in shared memory; values: thread =
// 16 channels of one row, shuffles over the row's lanes (the layouts of the flush).
// Measured (2 x 8 x 2048 tokens, head_dim 128, 4 bits, K and V, call included): 185 us as quantizer, dequantizer and copies,
// 28.7 us now.
#include "mz_quant16.cuh"
#include "mz_quant_f32.cuh"

namespace {
struct RoundtripParams {
  const uint16_t* x;
  long long sb, sh, st;
  int B, H, S, D, G, bits, meta_dtype;
  float alpha, eps;
  const float* table;
  uint16_t* out;
  unsigned tiles, per_pair;
};

__device__ __forceinline__ float through_meta(float v, int dt) {
  if (dt == MZ_F16) return __half2float(__float2half_rn(v));
  if (dt == MZ_BF16) return __bfloat162float(__float2bfloat16_rn(v));
  return v;
}

// a row's constants as floats in shared memory: the quantizer's, then the dequantizer's
constexpr int kRowFloats = 18;
struct Row {
  mzq::F32Row q;
  float hi;
  MzRowParams d;
};
__device__ __forceinline__ void make_row(Row& r, float mn, float mx, const RoundtripParams& p) {
  r.q.set(mn, mx, p.bits, p.alpha, p.eps);
  r.hi = mx;
  r.d = mz_row_params(through_meta(r.q.lo, p.meta_dtype), through_meta(r.q.span, p.meta_dtype), (1 << p.bits) - 1, p.eps);
}
__device__ __forceinline__ void put_row(float* f, const Row& r) {
  const float v[kRowFloats] = {r.q.lo, r.q.span, r.q.inv_span, r.q.anchor, r.q.a_up, r.q.a_dn, r.q.k_up, r.q.k_dn, r.q.zero_code,
                               r.q.limit, r.hi, r.d.lo, r.d.span, r.d.anchor, r.d.room_up, r.d.room_dn, __int_as_float(r.d.zero_code), 0.f};
#pragma unroll
  for (int k = 0; k < kRowFloats - 1; ++k) f[k * 256] = v[k];
}
__device__ __forceinline__ void get_row(Row& r, const float* f, int bits) {
  const int top = (1 << bits) - 1;
  r.q.lo = f[0]; r.q.span = f[256]; r.q.inv_span = f[512]; r.q.anchor = f[768]; r.q.a_up = f[1024]; r.q.a_dn = f[1280];
  r.q.k_up = f[1536]; r.q.k_dn = f[1792]; r.q.zero_code = f[2048]; r.q.limit = f[2304]; r.q.top = (float)top;
  r.hi = f[2560];
  r.d.lo = f[2816]; r.d.span = f[3072]; r.d.anchor = f[3328]; r.d.room_up = f[3584]; r.d.room_dn = f[3840];
  r.d.zero_code = __float_as_int(f[4096]);
  r.d.steps_up = max(top - r.d.zero_code, 1); r.d.steps_dn = max(r.d.zero_code, 1);
}
__device__ __forceinline__ float back(float x, const Row& r, const RoundtripParams& p, const float* table) {
  return mz_dequant_exact(r.d, r.q.code(x, r.q.lo, r.hi, p.bits, p.alpha, p.eps), table, 1 << p.bits);
}
__device__ __forceinline__ const float* stage_table(const RoundtripParams& p, float* s_table) {
  if (p.bits > 4) return p.table;
  for (int i = threadIdx.x; i < (1 << (2 * p.bits)); i += 256) s_table[i] = p.table[i];
  return s_table;
}

template <int DT>
__device__ __forceinline__ void roundtrip_keys(const RoundtripParams& p, uint32_t* s_red, float* s_row, float* s_table) {
  using P = mzq::P2<DT>;
  constexpr int TPT = 16;
  const int G = p.G, D = p.D, pairs = D >> 1, parts = G / TPT, tt = pairs * parts, per_cta = tt >= 256 ? 1 : 256 / tt, rows = per_cta * D;
  const int nsg = p.S / G, tid = threadIdx.x;
  const float* table = stage_table(p, s_table);
  const unsigned tile0 = blockIdx.x * per_cta;
  for (int w = tid; w < per_cta * tt; w += 256) {
    const int local = w / tt, part = (w % tt) / pairs, cp = w % pairs;
    const unsigned tile = tile0 + local;
    if (tile >= p.tiles) break;
    const int j = tile % nsg, pair = tile / nsg;
    const uint16_t* src = p.x + (pair / p.H) * p.sb + (pair % p.H) * p.sh + (long long)(j * G + part * TPT) * p.st + 2 * cp;
    uint32_t mn = P::INF2, mx = P::INF2 | 0x80008000u;
#pragma unroll
    for (int i = 0; i < TPT; ++i) {
      const uint32_t v = *(const uint32_t*)(src + i * p.st);
      mn = P::mn(mn, v); mx = P::mx(mx, v);
    }
    s_red[((local * parts + part) * 2) * pairs + cp] = mn;
    s_red[((local * parts + part) * 2 + 1) * pairs + cp] = mx;
  }
  __syncthreads();
  if (tid < rows && tile0 + tid / D < p.tiles) {
    const uint16_t* r16 = (const uint16_t*)(s_red + (tid / D) * parts * 2 * pairs);
    const int d = tid % D;
    float mn = INFINITY, mx = -INFINITY;
    for (int k = 0; k < parts; ++k) {
      mn = fminf(mn, mz_u16_to_float(r16[2 * k * D + d], DT));
      mx = fmaxf(mx, mz_u16_to_float(r16[(2 * k + 1) * D + d], DT));
    }
    Row r;
    make_row(r, mn, mx, p);
    put_row(s_row + tid, r);
  }
  __syncthreads();
  for (int w = tid; w < per_cta * tt; w += 256) {
    const int local = w / tt, part = (w % tt) / pairs, cp = w % pairs;
    const unsigned tile = tile0 + local;
    if (tile >= p.tiles) break;
    const int j = tile % nsg, pair = tile / nsg;
    const uint16_t* src = p.x + (pair / p.H) * p.sb + (pair % p.H) * p.sh + (long long)(j * G + part * TPT) * p.st + 2 * cp;
    const long long at = ((long long)pair * p.S + j * G + part * TPT) * D + 2 * cp;
    if (!MZ_IN_BOUNDS(at + (TPT - 1) * D + 1, (long long)p.B * p.H * p.S * D, 21)) continue;
    uint32_t* dst = (uint32_t*)(p.out + at);
    Row ra, rb;
    get_row(ra, s_row + local * D + 2 * cp, p.bits);
    get_row(rb, s_row + local * D + 2 * cp + 1, p.bits);
#pragma unroll 4
    for (int i = 0; i < TPT; ++i) {
      const uint32_t v = *(const uint32_t*)(src + i * p.st);
      dst[i * pairs] = P::pack(back(P::lo(v), ra, p, table), back(P::hi(v), rb, p, table));
    }
  }
}

template <int DT>
__device__ __forceinline__ void roundtrip_values(const RoundtripParams& p, unsigned block, float* s_table) {
  using P = mzq::P2<DT>;
  const float* table = stage_table(p, s_table);
  __syncthreads();
  const int G = p.G, D = p.D, NG = D / G, lpr = G >> 4;
  const unsigned pair = block / p.per_pair, chunk = block % p.per_pair;
  const int row = chunk * (256 / lpr) + threadIdx.x / lpr, sub = threadIdx.x % lpr;
  const bool live = row < p.S * NG;
  uint32_t x[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (live) {
    const uint16_t* src = p.x + (pair / p.H) * p.sb + (pair % p.H) * p.sh + (long long)(row / NG) * p.st + (row % NG) * G + sub * 8;
    const uint4 a = *(const uint4*)src, c = *(const uint4*)(src + lpr * 8);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = c.x; x[5] = c.y; x[6] = c.z; x[7] = c.w;
  }
  uint32_t mn = x[0], mx = x[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) { mn = P::mn(mn, x[i]); mx = P::mx(mx, x[i]); }
  for (int off = lpr >> 1; off > 0; off >>= 1) {
    mn = P::mn(mn, __shfl_xor_sync(0xffffffffu, mn, off));
    mx = P::mx(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  }
  if (!live) return;
  Row r;
  make_row(r, fminf(P::lo(mn), P::hi(mn)), fmaxf(P::lo(mx), P::hi(mx)), p);
  const long long at = ((long long)pair * p.S * NG + row) * G + sub * 8;
  if (!MZ_IN_BOUNDS(at + lpr * 8 + 7, (long long)p.B * p.H * p.S * D, 22)) return;
  uint16_t* dst = p.out + at;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = P::pack(back(P::lo(x[4 * c + i]), r, p, table), back(P::hi(x[4 * c + i]), r, p, table));
    *(uint4*)(dst + c * lpr * 8) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

template <int DT>
__global__ void __launch_bounds__(256, 4) roundtrip_kernel(const RoundtripParams k, const RoundtripParams v, unsigned key_blocks) {
  __shared__ uint32_t s_red[1024];
  __shared__ float s_row[(kRowFloats - 1) * 256];
  __shared__ float s_table[256];
  if (blockIdx.x < key_blocks) roundtrip_keys<DT>(k, s_red, s_row, s_table);
  else roundtrip_values<DT>(v, blockIdx.x - key_blocks, s_table);
}

// fills the parameters of one block and the CTAs it takes
int prepare(const void* x, const int* shape, const long long* strides, int group, int bits, float alpha, float eps, int meta_dtype, int keys,
            void* out, RoundtripParams* q, long long* blocks) {
  MZ_REQUIRE(x && shape && strides && out, "NULL pointer");
  MZ_REQUIRE(shape[0] > 0 && shape[1] > 0 && shape[2] > 0, "bad shape");
  MZ_REQUIRE(alpha > 0.f && eps > 0.f, "alpha and eps must be > 0");
  const int D = shape[3], S = shape[2];
  const int unit = keys ? 1 : 7;             // element granularity of the loads
  if ((D != 64 && D != 128) || (group != 32 && group != 64 && group != 128) || D % group != 0 || (keys && S % group != 0) ||
      ((strides[0] | strides[1] | strides[2]) & unit) || ((uintptr_t)x & (keys ? 3 : 15)) || ((uintptr_t)out & 15) || S >= (1 << 27))
    return mz_fail(MZ_ERR_UNSUPPORTED, "shape served by mz_quantize_rows / mz_dequantize_rows: head_dim %d, group %d, %d tokens", D, group, S);
  RoundtripParams& p = *q;
  p.x = (const uint16_t*)x; p.sb = strides[0]; p.sh = strides[1]; p.st = strides[2];
  p.B = shape[0]; p.H = shape[1]; p.S = S; p.D = D; p.G = group; p.bits = bits; p.meta_dtype = meta_dtype;
  p.alpha = alpha; p.eps = eps; p.out = (uint16_t*)out;
  int rc = mz_get_expand_table(bits, alpha, &p.table);
  if (rc) return rc;
  const long long pairs = (long long)p.B * p.H;
  if (keys) {
    const int tt = (D / 2) * (group / 16), per_cta = tt >= 256 ? 1 : 256 / tt;
    const long long tiles = pairs * (S / group);
    MZ_REQUIRE(tiles < (1LL << 31), "problem too large");
    p.tiles = (unsigned)tiles; p.per_pair = 0;
    *blocks = (tiles + per_cta - 1) / per_cta;
  } else {
    const int rows_per_cta = 256 / (group / 16);
    p.tiles = 0;
    p.per_pair = (unsigned)(((long long)S * (D / group) + rows_per_cta - 1) / rows_per_cta);
    *blocks = pairs * p.per_pair;
  }
  return MZ_OK;
}
}  // namespace

extern "C" int mz_roundtrip_kv(const void* k, const int* k_shape, const long long* k_strides, float alpha_key, void* k_out, const void* v,
                               const int* v_shape, const long long* v_strides, float alpha_value, void* v_out, int dtype, int group, int bits,
                               float eps, int meta_dtype, void* stream) {
  MZ_RANGE("mz_roundtrip_kv");
  MZ_REQUIRE((dtype == MZ_BF16 || dtype == MZ_F16) && mz_dtype_ok(meta_dtype), "bad dtype code");
  MZ_REQUIRE(bits >= 1 && bits <= 8, "bits must be 1..8, got %d", bits);
  MZ_REQUIRE(k != nullptr || v != nullptr, "neither keys nor values");
  RoundtripParams pk = {}, pv = {};
  long long kb = 0, vb = 0;
  int rc;
  if (k && (rc = prepare(k, k_shape, k_strides, group, bits, alpha_key, eps, meta_dtype, 1, k_out, &pk, &kb))) return rc;
  if (v && (rc = prepare(v, v_shape, v_strides, group, bits, alpha_value, eps, meta_dtype, 0, v_out, &pv, &vb))) return rc;
  MZ_REQUIRE(kb + vb < (1LL << 31), "problem too large");
  if (dtype == MZ_BF16) roundtrip_kernel<MZ_BF16><<<(unsigned)(kb + vb), 256, 0, (cudaStream_t)stream>>>(pk, pv, (unsigned)kb);
  else roundtrip_kernel<MZ_F16><<<(unsigned)(kb + vb), 256, 0, (cudaStream_t)stream>>>(pk, pv, (unsigned)kb);
  MZ_LAUNCH_CHECK("roundtrip");
  return MZ_OK;
}
