// Merge of the partial softmax records that the tiled decode kernels write (head_dim 64 or 128).
#include "mz_decode.cuh"

namespace {
// ---- merge of the records of one (batch, kv head) pair and head: one CTA, whose groups of D threads each merge every n-th chunk
// of records; their partial states are merged in a fixed order at the end.  The warps of the main kernel that hold records of the pair are found from
// the partition functions the main kernel uses: warp g owns the tiles whose start cost lies in
// [cost(g), cost(g+1)), and cost(g) is within [g*quot, g*(quot+1)), so every contributor lies in the
// candidate range [c_lo/(quot+1) - 1, (c_hi-1)/quot + 1], c_lo..c_hi being the pair's cost interval.
// All threads test candidates at once; the list keeps the candidates' order (a fixed merge order).
constexpr int kMaxCombineSlots = 4096;
// The workers of plan `tp` that can hold records of `pair` lie in [first, last] (a superset; see above).
struct WorkerRange { long long first, last; };
__device__ __forceinline__ WorkerRange candidate_workers(const MzTilesPlan& tp, int pair) {
  WorkerRange r = {0, -1};
  if (tp.total_warps <= 0) return r;
  const unsigned quot = tp.cost_quot ? tp.cost_quot : 1u;
  const unsigned c_lo = (unsigned)pair * (unsigned)tp.pair_cost, c_hi = c_lo + (unsigned)tp.pair_cost;
  r.first = (long long)(c_lo / (quot + 1u)) - 1;
  r.last = (long long)((c_hi - 1u) / quot) + 1;
  if (r.first < 0 || tp.cost_quot == 0) r.first = 0;
  if (r.last > tp.total_warps - 1 || tp.cost_quot == 0) r.last = tp.total_warps - 1;   // more workers than cost units: test them all
  return r;
}
// record index of worker gw's segment for `pair` (first_record = index of the plan's first record), or -1
__device__ __forceinline__ long long record_of(const MzTilesPlan& tp, long long gw, int pair, long long first_record) {
  const int T = tp.tiles_per_pair;
  const long long lo = (long long)pair * T, hi = lo + T;
  long long f0, f1;
  mz_warp_tiles(tp, gw, &f0, &f1);
  if (!(f0 < hi && f1 > lo && f0 < f1)) return -1;
  return first_record + gw * tp.max_segs + (pair - (int)((unsigned)f0 / (unsigned)T));
}
template <int D>
__global__ void __launch_bounds__(512, 4) combine_tiles_kernel(const MzDecodeParams p, const MzDecodeOut o) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // a dependent waits for this grid's completion itself
  __shared__ int s_slot[kMaxCombineSlots];     // record of candidate i, or -1
  __shared__ float s_part[512 / D][D + 2];
  const int gqa = p.gqa, pair = blockIdx.x / gqa, h = blockIdx.x % gqa;
  // candidates of the main plan, then of the residual-tile plan of the tcgen05 route (its records follow)
  const WorkerRange ra = candidate_workers(p.tp, pair), rb = candidate_workers(p.tp2, pair);
  const long long cand_a = ra.last - ra.first + 1, cand_b = rb.last - rb.first + 1;
  const long long cand = cand_a + cand_b;
  const long long first_b = p.slots_a / gqa;
  const bool listed = cand <= kMaxCombineSlots &&
                      first_b + (long long)p.tp.total_warps * p.tp.max_segs + (long long)p.tp2.total_warps * p.tp2.max_segs < (1LL << 31);
  if (listed) {
    for (int i = threadIdx.x; i < cand; i += blockDim.x)
      s_slot[i] = (int)(i < cand_a ? record_of(p.tp, ra.first + i, pair, 0) : record_of(p.tp2, rb.first + (i - cand_a), pair, first_b));
  }
  // everything above is arithmetic on the plans; the records themselves are the main kernels' output
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __syncthreads();
  const int n = (int)cand;
  // more candidates than the list holds (a huge explicit split count): every thread walks them itself
  auto for_each_slot = [&](auto&& fn) {
    for (long long gw = ra.first; gw <= ra.last; ++gw) {
      const long long rec = record_of(p.tp, gw, pair, 0);
      if (rec >= 0) fn(rec);
    }
    for (long long gw = rb.first; gw <= rb.last; ++gw) {
      const long long rec = record_of(p.tp2, gw, pair, first_b);
      if (rec >= 0) fn(rec);
    }
  };
  const int quad = threadIdx.x / D, quads = blockDim.x / D, d = threadIdx.x % D;
  float mx = -INFINITY, lsum = 0.f, a = 0.f;
  if (listed) {
    // four records at a time: their loads are independent and in flight together; the running
    // maximum is carried along (one pass)
    for (int i0 = 4 * quad; i0 < n; i0 += 4 * quads) {
      float mi[4], li[4], ai[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int sl = i0 + j < n ? s_slot[i0 + j] : -1;
        const bool on = sl >= 0;
        const long long slot = on ? (long long)sl * gqa + h : 0;
        mi[j] = on ? p.part.m[slot] : -INFINITY;
        li[j] = on ? p.part.l[slot] : 0.f;
        ai[j] = on ? p.part.acc[slot * D + d] : 0.f;
      }
      const float m_new = fmaxf(fmaxf(mx, fmaxf(mi[0], mi[1])), fmaxf(mi[2], mi[3]));
      const float keep = mx > -INFINITY ? __expf(mx - m_new) : 0.f;
      lsum *= keep; a *= keep;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float wgt = mi[j] > -INFINITY ? __expf(mi[j] - m_new) : 0.f;
        lsum = fmaf(li[j], wgt, lsum);
        a = fmaf(ai[j], wgt, a);
      }
      mx = m_new;
    }
    // the groups' states, merged in order by the first
    s_part[quad][d] = a;
    if (d == 0) { s_part[quad][D] = mx; s_part[quad][D + 1] = lsum; }
    __syncthreads();
    if (quad != 0) return;
    float m_all = -INFINITY;
    for (int k = 0; k < quads; ++k) m_all = fmaxf(m_all, s_part[k][D]);
    lsum = 0.f; a = 0.f;
    for (int k = 0; k < quads; ++k) {
      const float mk = s_part[k][D];
      const float wgt = mk > -INFINITY ? __expf(mk - m_all) : 0.f;
      lsum = fmaf(s_part[k][D + 1], wgt, lsum);
      a = fmaf(s_part[k][d], wgt, a);
    }
    mx = m_all;
  } else {
    if (quad != 0) return;
    for_each_slot([&](long long sl) { mx = fmaxf(mx, p.part.m[sl * gqa + h]); });
    for_each_slot([&](long long sl) {
      const long long slot = sl * gqa + h;
      const float mi = p.part.m[slot];
      const float wgt = mi > -INFINITY ? __expf(mi - mx) : 0.f;
      lsum = fmaf(p.part.l[slot], wgt, lsum);
      a = fmaf(p.part.acc[slot * D + d], wgt, a);
    });
  }
  const long long row = (long long)pair * gqa + h;
  if (o.out) mz_store_from_float(o.out, row * D + d, a / fmaxf(lsum, 1e-20f), o.out_dt);
  else {
    o.acc[row * o.acc_stride + d] = a;
    if (d == 0) { o.m[row * o.ml_stride] = mx; o.l[row * o.ml_stride] = lsum; }
  }
}

template <int V>
__device__ __forceinline__ void load_vec(const float* src, bool on, float (&v)[V]) {
  if (V == 4) {
    const float4 x = on ? *(const float4*)src : make_float4(0.f, 0.f, 0.f, 0.f);
    v[0] = x.x; v[1] = x.y; v[2 % V] = x.z; v[3 % V] = x.w;
  } else {
    const float2 x = on ? *(const float2*)src : make_float2(0.f, 0.f);
    v[0] = x.x; v[1] = x.y;
  }
}

// The common case (a handful of records per pair): one WARP per (pair, head), no shared memory and no block
// barrier.  Each lane finds one candidate's record before the wait (pure arithmetic), then up to eight records
// are loaded at once (their m / l words and D / 32 floats of acc per lane) and merged in candidate order; the
// records of a second plan (residual tiles of a split launch) follow those of the first.
template <int D>
__global__ void __launch_bounds__(256) combine_tiles_warp_kernel(const MzDecodeParams p, const MzDecodeOut o) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // a dependent waits for this grid's completion itself
  const int lane = threadIdx.x & 31;
  const long long row = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long rows = (long long)p.s.batch * p.H;
  const int gqa = p.gqa;
  const int pair = (int)(row / gqa), h = (int)(row % gqa);
  const bool live = row < rows;
  const WorkerRange ca = live ? candidate_workers(p.tp, pair) : WorkerRange{0, -1};
  const WorkerRange cb = live ? candidate_workers(p.tp2, pair) : WorkerRange{0, -1};
  const long long first_b = p.slots_a / gqa;
  // first chunk of candidates of each plan (one per lane); nearly always the only chunk
  long long rec_a = -1, rec_b = -1;
  if (ca.first + lane <= ca.last) rec_a = record_of(p.tp, ca.first + lane, pair, 0);
  if (cb.first + lane <= cb.last) rec_b = record_of(p.tp2, cb.first + lane, pair, first_b);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (!live) return;
  float mx = -INFINITY, lsum = 0.f;
  constexpr int V = D / 32;
  float a[V];
#pragma unroll
  for (int k = 0; k < V; ++k) a[k] = 0.f;
  auto merge_chunk = [&](long long my_rec) {
    unsigned todo = __ballot_sync(0xffffffffu, my_rec >= 0);
    while (todo) {
      float mi[8], li[8];
      float ai[8][V];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const bool on = todo != 0;
        const int src = on ? __ffs(todo) - 1 : 0;
        if (on) todo &= todo - 1;
        const long long rec = __shfl_sync(0xffffffffu, my_rec, src);
        const long long slot = on ? rec * gqa + h : 0;
        mi[j] = on ? p.part.m[slot] : -INFINITY;
        li[j] = on ? p.part.l[slot] : 0.f;
        load_vec<V>(p.part.acc + slot * D + V * lane, on, ai[j]);
      }
      float m_new = mx;
#pragma unroll
      for (int j = 0; j < 8; ++j) m_new = fmaxf(m_new, mi[j]);
      const float keep = mx > -INFINITY ? __expf(mx - m_new) : 0.f;
      lsum *= keep;
#pragma unroll
      for (int k = 0; k < V; ++k) a[k] *= keep;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float wgt = mi[j] > -INFINITY ? __expf(mi[j] - m_new) : 0.f;
        lsum = fmaf(li[j], wgt, lsum);
#pragma unroll
        for (int k = 0; k < V; ++k) a[k] = fmaf(ai[j][k], wgt, a[k]);
      }
      mx = m_new;
    }
  };
  for (long long base = ca.first; base <= ca.last; base += 32) {
    if (base != ca.first) rec_a = base + lane <= ca.last ? record_of(p.tp, base + lane, pair, 0) : -1;
    merge_chunk(rec_a);
  }
  for (long long base = cb.first; base <= cb.last; base += 32) {
    if (base != cb.first) rec_b = base + lane <= cb.last ? record_of(p.tp2, base + lane, pair, first_b) : -1;
    merge_chunk(rec_b);
  }
  const int d = V * lane;
  if (o.out) {
    const float den = fmaxf(lsum, 1e-20f);
#pragma unroll
    for (int k = 0; k < V; ++k) mz_store_from_float(o.out, row * D + d + k, a[k] / den, o.out_dt);
  } else {
    float* dst = o.acc + row * o.acc_stride + d;
#pragma unroll
    for (int k = 0; k < V; ++k) dst[k] = a[k];
    if (lane == 0) { o.m[row * o.ml_stride] = mx; o.l[row * o.ml_stride] = lsum; }
  }
}
}  // namespace

int mz_combine_tiles(const MzDecodeParams& p, const MzDecodeOut& o, cudaStream_t st) {
  if (p.tp.max_segs < 1) return mz_fail(MZ_ERR_ARG, "bad plan");
  // programmatic dependent launch: the merge grid may start while the main kernel drains; it finds its
  // records (pure arithmetic) and then waits for the main grid's results (griddepcontrol.wait)
  cudaLaunchConfig_t cfg = {};
  // A warp per (pair, head) takes eight records at a time and pays while that is about one turn: below eight workers per pair.  From there on a
  // CTA per (pair, head) shares them (12 x 8 pairs x 3000 tokens at 4 bits, 19 workers per pair: 35.2 us per call with warps,
  // 34.3 with CTAs; 16 x 8 x 4224, 13 per pair: 49.5 and 47.9; 48 x 8 x 2100, 4 per pair: 70.9 and 76.9; 64 pairs with 27 records
  // 150 and 140).  One CTA per pair for all heads, which had served 8 to 24 workers per pair, took 22 us on its own: 48.2 and 58.2.
  const long long pairs = (long long)p.s.batch * p.s.kv_heads;
  const bool per_warp = p.tp.total_warps / pairs < 8;
  const int D = p.s.head_dim;
  cfg.gridDim = dim3((unsigned)(per_warp ? (pairs * p.gqa + 7) / 8 : pairs * p.gqa));
  cfg.blockDim = dim3(per_warp ? 256 : 512);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (D == 128) {
    if (per_warp) MZ_CUDA(cudaLaunchKernelEx(&cfg, combine_tiles_warp_kernel<128>, p, o));
    else MZ_CUDA(cudaLaunchKernelEx(&cfg, combine_tiles_kernel<128>, p, o));
  } else {
    if (per_warp) MZ_CUDA(cudaLaunchKernelEx(&cfg, combine_tiles_warp_kernel<64>, p, o));
    else MZ_CUDA(cudaLaunchKernelEx(&cfg, combine_tiles_kernel<64>, p, o));
  }
  MZ_LAUNCH_CHECK("combine_tiles");
  return MZ_OK;
}
