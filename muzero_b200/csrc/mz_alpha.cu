// Statistics of a 16-bit K or V block that the log-compander alpha is chosen from: order statistics of |x| over a
// strided sample, and the mean distance of the groups' zero anchors from 0.5.
//
// |x| of a 16-bit type has 32768 patterns that sort like the magnitudes, so the order statistics are exact ranks in
// a histogram (65,536 samples at most by default): one launch instead of a gather, a radix sort and index arithmetic
// in 64-bit tensors (25 launches).  The last CTA to finish walks the histogram and leaves it zeroed for the next call.
// The anchor pass reads the block once and is bound by that; per-CTA sums are added in CTA order by the last CTA.
// Taken for 1-, 3- and 8-bit caches only: the other widths have one alpha whatever the data is.
#include "mz_common.cuh"

namespace {
constexpr int kBins = 32768;
constexpr int kMaxCtas = 2048;
struct AlphaParams {
  const uint16_t* x;
  long long sb, sh, st;          // element strides of [B, H, S, D]
  int B, H, S, D, G, dt;
  int rows_order;                // sample order: 1 = key rows (b, h, group, channel, token), 0 = (b, h, token, channel up to d_pad)
  int d_pad;
  long long total, step; int n;  // sample i = element i * step of that order, i < n
  unsigned* hist; unsigned* ticket; double* partial;
  float* out;                    // {p50, p95, p99, anchor offset}
  int k50, k95, k99;             // 1-based ranks
  int vec;                       // channel groups of whole, aligned 16-byte vectors: G / 8 lanes per group
};

__device__ __forceinline__ bool last_cta(unsigned* ticket) {
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  __syncthreads();
  return s_last;
}

__global__ void __launch_bounds__(1024) alpha_ratios_kernel(const AlphaParams p) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < p.n; i += (long long)gridDim.x * blockDim.x) {
    long long r = i * p.step;
    long long at;
    bool zero = false;
    if (p.rows_order) {
      const int nsg = p.S / p.G;
      const int t = (int)(r % p.G); r /= p.G;
      const int d = (int)(r % p.D); r /= p.D;
      const int g = (int)(r % nsg); r /= nsg;
      at = (r / p.H) * p.sb + (r % p.H) * p.sh + (long long)(g * p.G + t) * p.st + d;
    } else {
      const int d = (int)(r % p.d_pad); r /= p.d_pad;
      const int t = (int)(r % p.S); r /= p.S;
      zero = d >= p.D;
      at = (r / p.H) * p.sb + (r % p.H) * p.sh + (long long)t * p.st + (zero ? 0 : d);
    }
    atomicAdd(p.hist + (zero ? 0 : (p.x[at] & 0x7fffu)), 1u);
  }
  if (!last_cta(p.ticket)) return;
  // thread t owns 32 bins; prefix over the 1024 threads, then each rank falls into one thread's bins
  __shared__ unsigned s_warp[32];
  unsigned c[32], sum = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint4 v = __ldcg((const uint4*)(p.hist + threadIdx.x * 32) + k);
    c[4 * k] = v.x; c[4 * k + 1] = v.y; c[4 * k + 2] = v.z; c[4 * k + 3] = v.w;
    ((uint4*)(p.hist + threadIdx.x * 32))[k] = make_uint4(0, 0, 0, 0);
    sum += v.x + v.y + v.z + v.w;
  }
  if (threadIdx.x == 0) *p.ticket = 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned pre = sum;
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned o = __shfl_up_sync(0xffffffffu, pre, off);
    if (lane >= off) pre += o;
  }
  if (lane == 31) s_warp[warp] = pre;
  __syncthreads();
  unsigned base = 0;
  for (int w = 0; w < warp; ++w) base += s_warp[w];
  unsigned below = base + pre - sum;
  const int ks[3] = {p.k50, p.k95, p.k99};
#pragma unroll
  for (int k = 0; k < 32; ++k) {
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if ((unsigned)ks[j] > below && (unsigned)ks[j] <= below + c[k]) p.out[j] = mz_u16_to_float((uint16_t)(threadIdx.x * 32 + k), p.dt);
    below += c[k];
  }
}

__device__ __forceinline__ float anchor_offset(float lo, float hi) {
  const float a = __fdiv_rn(__fsub_rn(0.0f, lo), fmaxf(__fsub_rn(hi, lo), 1e-8f));
  return fabsf(fminf(fmaxf(a, 0.0f), 1.0f) - 0.5f);
}
// groups along tokens (KEYS; a ragged last group is padded with zeros) or along channels (padded likewise)
template <bool KEYS>
__global__ void __launch_bounds__(256) alpha_anchor_kernel(const AlphaParams p) {
  const long long ng = KEYS ? (p.S + p.G - 1) / p.G : (p.D + p.G - 1) / p.G;
  const long long groups = (long long)p.B * p.H * ng * (KEYS ? p.D : p.S);
  double sum = 0.0;
  const int lane = threadIdx.x & 31;
  if (KEYS) {
    // thread = one channel of one group, channels fastest
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < groups; i += (long long)gridDim.x * blockDim.x) {
      const int d = (int)(i % p.D);
      long long r = i / p.D;
      const int g = (int)(r % ng); r /= ng;
      const uint16_t* src = p.x + (r / p.H) * p.sb + (r % p.H) * p.sh + d;
      const int t0 = g * p.G, t1 = min(t0 + p.G, p.S);
      float lo = INFINITY, hi = -INFINITY;
#pragma unroll 8
      for (int t = t0; t < t1; ++t) {
        const float v = mz_u16_to_float(src[(long long)t * p.st], p.dt);
        lo = fminf(lo, v); hi = fmaxf(hi, v);
      }
      if (t1 - t0 < p.G) { lo = fminf(lo, 0.f); hi = fmaxf(hi, 0.f); }
      sum += anchor_offset(lo, hi);
    }
  } else if (p.vec) {
    // G / 8 lanes per group, one 16-byte load each
    const int lpg = p.G >> 3, sub = threadIdx.x % lpg;
    const long long per_pass = (long long)gridDim.x * (blockDim.x / lpg), passes = (groups + per_pass - 1) / per_pass;
    long long i = (long long)blockIdx.x * (blockDim.x / lpg) + threadIdx.x / lpg;
    for (long long k = 0; k < passes; ++k, i += per_pass) {
      const bool live = i < groups;
      const long long at = live ? i : 0;
      const long long row = at / ng, pair = row / p.S;
      const uint16_t* src = p.x + (pair / p.H) * p.sb + (pair % p.H) * p.sh + (row % p.S) * p.st + (at % ng) * p.G + sub * 8;
      const uint4 v = *(const uint4*)src;
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
      float lo = INFINITY, hi = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float a = mz_u16_to_float((uint16_t)(w[j] & 0xffffu), p.dt), b = mz_u16_to_float((uint16_t)(w[j] >> 16), p.dt);
        lo = fminf(lo, fminf(a, b)); hi = fmaxf(hi, fmaxf(a, b));
      }
      for (int off = lpg >> 1; off > 0; off >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, off));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, off));
      }
      if (live && sub == 0) sum += anchor_offset(lo, hi);
    }
  } else {
    // warp = one group of one token at a time
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long i = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < groups; i += warps) {
      const int g = (int)(i % ng);
      long long r = i / ng;
      const int t = (int)(r % p.S); r /= p.S;
      const uint16_t* src = p.x + (r / p.H) * p.sb + (r % p.H) * p.sh + (long long)t * p.st + g * p.G;
      const int n = min(p.G, p.D - g * p.G);
      float lo = INFINITY, hi = -INFINITY;
      for (int c = lane; c < p.G; c += 32) {
        const float v = c < n ? mz_u16_to_float(src[c], p.dt) : 0.f;
        lo = fminf(lo, v); hi = fmaxf(hi, v);
      }
      for (int off = 16; off > 0; off >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, off));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, off));
      }
      if (lane == 0) sum += anchor_offset(lo, hi);
    }
  }
  __shared__ double s_sum[8];
  for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
  if (lane == 0) s_sum[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0;
    for (int w = 0; w < 8; ++w) a += s_sum[w];
    p.partial[blockIdx.x] = a;
  }
  if (!last_cta(p.ticket + 1)) return;
  double a = 0.0;
  for (unsigned c = threadIdx.x; c < gridDim.x; c += blockDim.x) a += __ldcg(p.partial + c);
  for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
  if (lane == 0) s_sum[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    a = 0.0;
    for (int w = 0; w < 8; ++w) a += s_sum[w];
    p.out[3] = (float)(a / (double)groups);
    p.ticket[1] = 0;
  }
}
}  // namespace

extern "C" size_t mz_alpha_stats_workspace_bytes(void) {
  return kBins * sizeof(unsigned) + 16 + kMaxCtas * sizeof(double);
}

extern "C" int mz_alpha_stats(const void* block, int dtype, const int* shape, const long long* strides, int group, int keys, int rows_order,
                              int max_points, int want, void* workspace, float* stats, void* stream) {
  MZ_RANGE("mz_alpha_stats");
  MZ_REQUIRE(block && shape && strides && workspace && stats, "NULL pointer");
  MZ_REQUIRE(dtype == MZ_BF16 || dtype == MZ_F16, "dtype must be bf16 or fp16");
  MZ_REQUIRE(shape[0] > 0 && shape[1] > 0 && shape[2] > 0 && shape[3] > 0 && group > 0 && max_points > 0, "bad shape");
  MZ_REQUIRE((uintptr_t)workspace % 16 == 0, "workspace must be 16-byte aligned");
  AlphaParams p = {};
  p.x = (const uint16_t*)block;
  p.B = shape[0]; p.H = shape[1]; p.S = shape[2]; p.D = shape[3];
  p.sb = strides[0]; p.sh = strides[1]; p.st = strides[2];
  p.G = group; p.dt = dtype; p.rows_order = rows_order;
  p.d_pad = keys || rows_order < 0 ? p.D : (p.D + group - 1) / group * group;
  if (rows_order < 0) p.rows_order = 0;
  p.hist = (unsigned*)workspace;
  p.ticket = p.hist + kBins;
  p.partial = (double*)(p.ticket + 4);
  p.out = stats;
  cudaStream_t st = (cudaStream_t)stream;
  if (want & 1) {
    MZ_REQUIRE(!p.rows_order || p.S >= group, "no whole group of tokens");
    p.total = (long long)p.B * p.H * (p.rows_order ? (long long)(p.S / group) * group * p.D : (long long)p.S * p.d_pad);
    p.step = p.total > max_points ? p.total / max_points : 1;
    const long long n = (p.total + p.step - 1) / p.step;
    p.n = (int)(n < max_points ? n : max_points);
    auto rank = [&](double q) { const int k = (int)(q * p.n); return k < 1 ? 1 : k; };
    p.k50 = rank(0.50); p.k95 = rank(0.95); p.k99 = rank(0.99);
    int ctas = (p.n + 1023) / 1024;
    if (ctas > 148) ctas = 148;
    alpha_ratios_kernel<<<ctas, 1024, 0, st>>>(p);
    MZ_LAUNCH_CHECK("alpha_ratios");
  }
  if (want & 2) {
    const long long ng = keys ? (p.S + group - 1) / group : (p.D + group - 1) / group;
    const long long groups = (long long)p.B * p.H * ng * (keys ? p.D : p.S);
    long long ctas = keys ? (groups + 255) / 256 : (groups + 63) / 64;
    if (ctas > 148 * 8) ctas = 148 * 8;
    p.vec = !keys && p.D % group == 0 && (group & (group - 1)) == 0 && group >= 8 && group <= 256 && ((uintptr_t)block & 15) == 0 &&
            !((p.sb | p.sh | p.st) & 7);
    if (keys) alpha_anchor_kernel<true><<<(unsigned)ctas, 256, 0, st>>>(p);
    else alpha_anchor_kernel<false><<<(unsigned)ctas, 256, 0, st>>>(p);
    MZ_LAUNCH_CHECK("alpha_anchor");
  }
  return MZ_OK;
}
