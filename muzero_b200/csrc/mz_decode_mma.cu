// Host side of the tensor-core decode kernel: which shapes it serves, the shared-memory layout, the cut of the work over
// warps, and the launch.  The kernel itself is in mz_decode_mma.cuh, its instances in mz_decode_mma_*.cu.
#include <map>
#include <mutex>
#include <tuple>

#include "mz_mma_common.cuh"

namespace mzm {
constexpr int DT = 16;                      // tokens per residual tile
// first byte of a kernel's dynamic shared memory inside the shared window
__global__ void smem_base_probe_kernel(unsigned* out) {
  extern __shared__ __align__(128) uint8_t smem[];
  *out = (unsigned)__cvta_generic_to_shared(smem);
}
__device__ unsigned g_probe_result;

constexpr int kMaxDevices = 64;
std::mutex g_mu;
int g_window_base[kMaxDevices];      // 0 = not probed yet, -1 = probe failed, else the address

// Lookup-table entries kept in a static device array (no allocation): one slot per (bits, form, alpha of keys, alpha
// of values) seen on a device.  Form: 32-bit entries of the unrolled kernel, or 64-bit entries of the general one.
constexpr int kLutSlots = 16, kLutWords = 1024;
__device__ __align__(16) uint32_t g_lut[kLutSlots][kLutWords];
template <int BITS, bool SPLIT>
__global__ void build_lut_kernel(int slot, float alpha_key, float alpha_value) {
  constexpr int N = 1 << (2 * BITS);
  for (int i = threadIdx.x; i < 2 * N; i += blockDim.x) {
    const float alpha = i / N ? alpha_value : alpha_key;
    if (SPLIT) ((uint2*)g_lut[slot])[i] = split_entry<BITS>(alpha, i % N);
    else g_lut[slot][i] = lookup_entry<BITS>(alpha, i % N);
  }
}
struct LutKey { int bits; bool split; float ak, av; };
struct LutDevice { uint32_t* base; int used; LutKey keys[kLutSlots]; };
LutDevice g_lut_dev[kMaxDevices];
}  // namespace mzm

// Device pointer to the table entries for (bits, form, alphas) on the current device, or nullptr when they cannot be
// provided (all slots taken, or the one-time build is not possible right now, e.g. during stream capture): the
// kernel then computes the entries in every CTA.  The first request for a combination launches a one-block
// kernel on the default stream and waits for it, so that any stream may use the entries afterwards.
const unsigned* mz_mma_lookup_entries(int bits, bool split, float alpha_key, float alpha_value) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= mzm::kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lk(mzm::g_mu);
  mzm::LutDevice& d = mzm::g_lut_dev[dev];
  for (int i = 0; i < d.used; ++i)
    if (d.keys[i].bits == bits && d.keys[i].split == split && d.keys[i].ak == alpha_key && d.keys[i].av == alpha_value) return d.base + i * mzm::kLutWords;
  if (d.used >= mzm::kLutSlots) return nullptr;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(cudaStreamLegacy, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
    (void)cudaGetLastError();
    return nullptr;
  }
  if (d.base == nullptr && cudaGetSymbolAddress((void**)&d.base, mzm::g_lut) != cudaSuccess) {
    (void)cudaGetLastError();
    d.base = nullptr;
    return nullptr;
  }
  const int slot = d.used;
  if (!split && bits == 2) mzm::build_lut_kernel<2, false><<<1, 32>>>(slot, alpha_key, alpha_value);
  else if (!split) mzm::build_lut_kernel<4, false><<<1, 256>>>(slot, alpha_key, alpha_value);
  else if (bits == 1) mzm::build_lut_kernel<1, true><<<1, 32>>>(slot, alpha_key, alpha_value);
  else if (bits == 2) mzm::build_lut_kernel<2, true><<<1, 32>>>(slot, alpha_key, alpha_value);
  else if (bits == 3) mzm::build_lut_kernel<3, true><<<1, 128>>>(slot, alpha_key, alpha_value);
  else mzm::build_lut_kernel<4, true><<<1, 256>>>(slot, alpha_key, alpha_value);
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  d.keys[slot] = {bits, split, alpha_key, alpha_value};
  d.used = slot + 1;
  return d.base + slot * mzm::kLutWords;
}

// Shared-window address at which this device places dynamic shared memory (a kernel without static shared
// memory).  The tensor-core kernel addresses its buffers absolutely (the lookup table must sit at 65536),
// so the planner needs the number; it is measured once per device with a one-thread kernel and a
// synchronous 4-byte read of a device variable, no allocation.
int mz_smem_window_base() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= mzm::kMaxDevices) return -1;
  std::lock_guard<std::mutex> lk(mzm::g_mu);
  if (mzm::g_window_base[dev] == 0) {
    unsigned* dptr = nullptr;
    unsigned v = 0;
    cudaError_t e = cudaGetSymbolAddress((void**)&dptr, mzm::g_probe_result);
    if (e == cudaSuccess) {
      mzm::smem_base_probe_kernel<<<1, 1, 1024>>>(dptr);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyFromSymbol(&v, mzm::g_probe_result, sizeof(v));
    mzm::g_window_base[dev] = (e == cudaSuccess && v > 0 && v < 8192) ? (int)v : -1;
    if (e != cudaSuccess) (void)cudaGetLastError();
  }
  return mzm::g_window_base[dev];
}


namespace {
bool find_kernel(const MzDecodeParams& p, MzMmaKernel* k) {
  const int D = p.s.head_dim, G = p.s.group, nt = p.gqa > 4 ? 2 : 1;
  switch (p.s.bits) {
    case 1: return mz_mma_kernel_b1(D, G, nt, k);
    case 2: return mz_mma_kernel_b2(D, G, nt, k);
    case 3: return mz_mma_kernel_b3(D, G, nt, k);
    case 4: return mz_mma_kernel_b4(D, G, nt, k);
    case 8: return mz_mma_kernel_b8(D, G, nt, k);
    default: return mz_mma_kernel_wide(D, G, nt, k);
  }
}
}  // namespace

bool mz_decode_mma_supported(const MzDecodeParams& p) {
  const mz_kv_store& s = p.s;
  if ((s.head_dim != 64 && s.head_dim != 128) || (s.group != 32 && s.group != 64 && s.group != 128) || s.head_dim % s.group != 0) return false;
  if (p.gqa < 1 || p.gqa > 8 || p.v_lead != 0) return false;
  auto al16 = [](const void* q) { return ((uintptr_t)q & 15) == 0; };
  const int msz = s.meta_dtype == MZ_F32 ? 4 : 2;
  if (s.k_groups > 0) {
    if (!al16(s.packed_k) || !al16(s.packed_v) || !al16(s.k_mn) || !al16(s.k_scale) || !al16(s.v_mn) || !al16(s.v_scale)) return false;
    if ((s.pk_stride_b | s.pk_stride_h | s.pv_stride_b | s.pv_stride_h) & 15) return false;
    if (((s.km_stride_b | s.km_stride_h | s.vm_stride_b | s.vm_stride_h) * msz) & 15) return false;
  }
  if (s.res_len > 0) {
    if (!al16(s.res_k) || !al16(s.res_v)) return false;
    if ((s.res_stride_b | s.res_stride_h | s.res_stride_t) & 7) return false;
  }
  // the residual-tile path reads the query in 4-byte pieces
  if (((uintptr_t)p.query & 3) || ((p.q_stride_b | p.q_stride_h) & 1)) return false;
  return mz_smem_window_base() > 0;
}

namespace {
constexpr int kCostPacked = 64;      // relative cost of a packed tile of 64 tokens at head_dim 128
constexpr int kCostDense = 20;       // of a residual tile of 16 tokens among busy warps

// shared-memory layout of `t` for up to `warps` warps (0: as many as fit); returns the warp count, 0 if a tile does not fit
int layout(MzTilesPlan& t, const MzDecodeParams& p, const MzMmaKernel& k, int warps, unsigned min_stage) {
  const mz_kv_store& s = p.s;
  const int msz = s.meta_dtype == MZ_F32 ? 4 : 2;
  unsigned sb = (unsigned)(s.head_dim * p.QB + 2 * s.head_dim * msz);
  if (sb < min_stage) sb = min_stage;
  if (s.res_len > 0 && sb < (unsigned)(mzm::DT * 2 * s.head_dim)) sb = mzm::DT * 2 * s.head_dim;     // a residual tile
  sb = (sb + 127u) & ~127u;
  const unsigned wb = (unsigned)mz_smem_window_base();
  const unsigned window_end = wb + 227u * 1024u;      // the most dynamic shared memory a block may ask for
  const unsigned per_high = sb + k.ri_bytes + k.a_bytes + k.p_bytes;
  const int most = warps > 0 && warps < k.max_warps ? warps : k.max_warps;
  warps = most;
  t.stage_bytes = sb;
  t.low_base = (wb + 127u) & ~127u;
  if (k.table_bytes > 0) {
    t.high_base = mzm::TBL + k.table_bytes;
    const int fit_low = (int)((mzm::TBL - t.low_base) / sb), fit_high = (int)((window_end - t.high_base) / per_high);
    if (warps > fit_low) warps = fit_low;
    if (warps > fit_high) warps = fit_high;
  } else {
    const int fit = (int)((window_end - t.low_base) / (sb + per_high));
    if (warps > fit) warps = fit;
    t.high_base = t.low_base + warps * sb;
  }
  t.smem_per_warp = sb + per_high;
  t.smem_bytes = t.high_base + per_high * warps - wb;
  return warps;
}

void describe_tiles(MzTilesPlan& t, const MzDecodeParams& p) {
  const mz_kv_store& s = p.s;
  t.kind = 1;
  t.packed_tiles = s.k_groups;
  t.dense_tokens = mzm::DT;
  const int dense_tiles = (s.res_len + mzm::DT - 1) / mzm::DT;
  t.tiles_per_pair = t.packed_tiles + dense_tiles;
  // a tile of 32 tokens still prepares as many rows: measured ratios (64 x 8 pairs x 4224 tokens, 4 bits)
  t.cost_q = s.group == 32 ? 54 : s.group == 64 ? kCostPacked : 140;
  if (s.head_dim == 64) t.cost_q = t.cost_q * 6 / 10;
  t.cost_d = kCostDense;
  t.pair_cost = (long long)t.packed_tiles * t.cost_q + (long long)dense_tiles * t.cost_d;
  if (t.pair_cost < 1) t.pair_cost = 1;
}
int cut(MzTilesPlan& t, long long pairs, long long W) {
  t.total_tiles = pairs * t.tiles_per_pair;
  t.total_cost = pairs * t.pair_cost;
  if (t.total_cost >= (1LL << 31)) return mz_fail(MZ_ERR_UNSUPPORTED, "cache too large for the tiled kernel");
  if (W > (1LL << 30)) return mz_fail(MZ_ERR_ARG, "too many splits");
  t.total_warps = (int)W;
  t.cost_quot = (unsigned)(t.total_cost / W);
  t.cost_rem = (unsigned)(t.total_cost % W);
  const long long len = t.total_cost / W + 2;
  t.max_segs = (int)((len - 1) / t.pair_cost + 2);
  return MZ_OK;
}

int plan_single(MzDecodeParams& p, const MzMmaKernel& k, int splits_request, int sm_count, size_t* slots, unsigned min_stage = 0) {
  MzTilesPlan& t = p.tp;
  describe_tiles(t, p);
  int warps = layout(t, p, k, 0, min_stage);
  if (warps < 1) return mz_fail(MZ_ERR_UNSUPPORTED, "tile does not fit shared memory");
  const long long pairs = (long long)p.s.batch * p.s.kv_heads;
  long long W;
  if (splits_request > 0) {
    W = pairs * splits_request;
  } else {
    W = (long long)sm_count * warps;                             // one resident CTA per SM
    const long long one_tile = pairs * t.pair_cost / t.cost_q;   // at least one packed tile's worth per warp
    if (W > one_tile) W = one_tile;
    if (W < 1) W = 1;
  }
  int rc = cut(t, pairs, W);
  if (rc) return rc;
  if (W < (long long)sm_count * warps) warps = layout(t, p, k, (int)((W + sm_count - 1) / sm_count), min_stage);
  t.warps_per_cta = warps;
  t.ctas = (int)((W + warps - 1) / warps);
  *slots = (size_t)W * t.max_segs * p.gqa;
  return MZ_OK;
}

// clusters of `cs` CTAs with this much shared memory that the device holds at once (asked once per configuration)
int clusters_at_once(const MzMmaKernel& k, int cs, int threads, unsigned smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, const void*, int, int, unsigned>, int> seen;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_tuple(dev, k.fn, cs, threads, smem);
  const auto it = seen.find(key);
  if (it != seen.end()) return it->second;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cs);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, k.fn, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    n = 0;
  }
  if (seen.size() > 4096) seen.clear();
  seen[key] = n;
  return n;
}

// ---- choice between cluster mode and an even cut of the tiles over all SMs, and of the kernel for the cut, by measured
// cost.  The constants are least-squares fits, in us, to device times of calls of 1..40 sequences x 2, 4 or 8 kv heads x
// 260..40000 tokens at head_dim 128 (1060 shapes, each run in every form that serves it).  x = packed tiles per SM, a residual
// tile counted by its cost.
// SIMT cut: base (launch, prologue, last turn, merge kernel) + tile * x; within 9 to 19 % (rms).  [group 32, 64, 128], then
// [heads per kv head: 1 and 2, 4, 8] and [bits]
constexpr float kSimtBase[3][3] = {{18.2f, 21.7f, 24.8f}, {22.4f, 26.1f, 34.6f}, {28.1f, 33.2f, 44.7f}};
constexpr float kSimtTile[3][3][8] = {{{0.56f, 0.54f, 0.59f, 0.72f, 0.91f, 0.93f, 0.95f, 0.89f},
                                       {0.60f, 0.57f, 0.67f, 0.80f, 1.02f, 0.98f, 0.99f, 0.95f},
                                       {0.96f, 0.95f, 1.12f, 1.15f, 1.40f, 1.35f, 1.36f, 1.30f}},
                                      {{0.85f, 0.88f, 1.01f, 0.90f, 1.36f, 1.43f, 1.72f, 1.53f},
                                       {0.92f, 0.84f, 1.04f, 1.02f, 1.72f, 1.93f, 1.99f, 1.35f},
                                       {1.57f, 1.51f, 1.65f, 1.76f, 2.50f, 2.46f, 2.25f, 2.22f}},
                                      {{1.43f, 1.57f, 1.58f, 1.37f, 2.77f, 3.15f, 4.71f, 2.87f},
                                       {1.71f, 1.58f, 2.09f, 1.84f, 3.42f, 3.67f, 6.23f, 3.81f},
                                       {3.00f, 3.08f, 2.98f, 3.53f, 5.29f, 5.68f, 7.26f, 4.21f}}};
constexpr float kUnrolledBase = 18.f, kUnrolledTile = 0.69f;      // 14 %
// Cluster mode: base + tile * warps * turns, a turn being one packed tile for every warp of the cluster; within 5 to 10 %.
// [group][up to 4 heads, up to 8][bits].  Tiles of head_dim 64 take 0.6 of it.
constexpr float kClusterBase[2] = {10.5f, 13.f};
constexpr float kClusterTile[3][2][8] = {{{0.60f, 0.57f, 0.61f, 0.59f, 1.01f, 1.00f, 1.00f, 0.89f}, {1.02f, 0.94f, 1.04f, 0.99f, 1.40f, 1.39f, 1.36f, 1.25f}},
                                         {{0.77f, 0.88f, 0.89f, 0.88f, 1.50f, 1.86f, 1.85f, 1.69f}, {1.53f, 1.57f, 1.63f, 1.50f, 2.19f, 2.28f, 2.12f, 1.89f}},
                                         {{1.44f, 1.49f, 2.20f, 1.95f, 4.20f, 4.88f, 4.78f, 4.36f}, {2.87f, 2.89f, 3.15f, 3.47f, 4.92f, 5.52f, 5.39f, 5.10f}}};
// The general kernel's own cut: a tile costs 1.25 of the cluster's (its turns are not aligned), its base is 24 / 35 us.
constexpr float kGeneralBase[2] = {24.f, 35.f}, kGeneralTile = 1.25f;

int group_index(int group) { return group == 32 ? 0 : group == 64 ? 1 : 2; }
float cluster_tile_us(const MzDecodeParams& p) {
  return kClusterTile[group_index(p.s.group)][p.gqa > 4][p.s.bits - 1] * (p.s.head_dim == 64 ? 0.6f : 1.0f);
}

// The kernel of an even cut: the unrolled kernel where it serves; else the SIMT kernel where it serves.  The general kernel's base is
// larger and its tiles cost as much or more (3 bits, 4 heads, groups of 32: 0.81 against 0.67 us; 64: 1.09 against 1.04; 128: 2.7
// against 2.1; 8 bits, 64: 2.4 against 1.35), but its residual tiles have CTAs of their own once every warp has two
// packed tiles, which is worth a turn.  Codes of up to 4 bits in groups of 64 with 4 or 8 heads gain by that between about 28 and 52
// tiles per SM (20 shapes: 0.79 to 1.06 of the SIMT kernel's time, 0.96 on average; 1 bit, 24 x 8 x 1537 48 against 62 us); below
// (1.04 on average) and above (1.04; 3 bits, 2 x 8 x 60000 144 against 126) they don't.  (1 to 3 bits at head_dim 128 come here with explicit splits or under a
// scratch limit only, 4 bits with 8 heads also where choose_umma leaves them; the other calls of this family are the tcgen05 kernel's.)
enum class Cut { kUnrolled, kSimt, kGeneral };
Cut choose_cut(const MzDecodeParams& p, float x) {
  if (mz_decode_flat_supported(p)) return Cut::kUnrolled;
  if (!mz_decode_tiles_supported(p)) return Cut::kGeneral;
  return p.s.bits <= 4 && p.s.group == 64 && p.gqa >= 4 && x >= 28.f && x < 52.f ? Cut::kGeneral : Cut::kSimt;
}
float cut_us(const MzDecodeParams& p, float x) {
  const int g = group_index(p.s.group), heads = p.gqa > 4 ? 2 : p.gqa == 4 ? 1 : 0;
  switch (choose_cut(p, x)) {
    case Cut::kUnrolled: return kUnrolledBase + kUnrolledTile * x;
    case Cut::kSimt: return kSimtBase[g][heads] + kSimtTile[g][heads][p.s.bits - 1] * x;
    default: return kGeneralBase[p.gqa > 4] + kGeneralTile * cluster_tile_us(p) * x;
  }
}
float tiles_per_sm(const MzDecodeParams& p, const MzTilesPlan& t, int sm_count) {
  return (float)((double)p.s.batch * p.s.kv_heads * (double)t.pair_cost / t.cost_q / sm_count);
}

// estimate for clusters of `cs` CTAs of `nw` warps
float cluster_us(const MzDecodeParams& p, const MzTilesPlan& t, int cs, int nw) {
  const long long turn = (long long)cs * nw * t.cost_q, pair_cost = (long long)t.packed_tiles * t.cost_q + (long long)(t.tiles_per_pair - t.packed_tiles) * t.cost_d;
  return kClusterBase[p.gqa > 4] + cluster_tile_us(p) * (float)(nw * ((pair_cost + turn - 1) / turn));
}
float cluster_us(const MzDecodeParams& c) { return cluster_us(c, c.tp, c.cluster, c.tp.warps_per_cta); }

// Cluster mode: one cluster per pair, no partial records in memory and no merge kernel; taken where the estimates above say that it
// is not slower than the cut, or at any cost.
bool plan_cluster(MzDecodeParams& p, const MzMmaKernel& k, int sm_count, bool any_cost = false) {
  const long long pairs = (long long)p.s.batch * p.s.kv_heads;
  if (pairs > sm_count) return false;
  MzTilesPlan& t = p.tp;
  describe_tiles(t, p);
  const int T = t.tiles_per_pair;
  const float limit = any_cost ? INFINITY : cut_us(p, tiles_per_sm(p, t, sm_count));
  int cs = 1;
  while (cs < 8 && cs * 2 * pairs <= sm_count && cs * 4 < T) cs *= 2;
  const unsigned rec = (unsigned)(p.gqa * (p.s.head_dim + 4) * 4);
  for (; cs >= 1; cs >>= 1) {
    // one warp per tile where that fits; at least four warps to fill the tables
    int want = (T + cs - 1) / cs;
    if (want < 4) want = 4;
    const int nw = layout(t, p, k, want, rec);
    if (nw < 1) return false;
    if (cluster_us(p, t, cs, nw) > limit) return false;    // smaller clusters are heavier still
    if (cs > 1 && clusters_at_once(k, cs, nw * 32, t.smem_bytes) < pairs) continue;
    // tiles are dealt to the cluster's warps by cost; every warp gets at most about one residual tile's cost more than its share
    if (cut(t, 1, (long long)cs * nw) != MZ_OK) return false;
    t.warps_per_cta = nw;
    t.ctas = (int)pairs * cs;
    p.cluster = cs;
    return true;
  }
  return false;
}
// Whether the tcgen05 kernel takes a call that it serves; `clusters`: the choice without it is cluster mode, planned in `c`.
// head_dim 128, 1 to 3 bits: always but for the smallest calls (kOneLaunchTiles).  On the device, over 51 shapes of 3 to 120 tiles per SM it needs 0.56 (1 bit), 0.68 (2 bits) and
// 0.62 (3 bits) of the time of the other choice, and was behind it in one (34 x 4 x 673 at 1 bit: 19.5 against 17.8 us).
// 4 bits need two lookups per code, and three planes because the unrolled kernel's error (3e-5) is out of reach of two (4e-5 to 6e-5).
// With up to four heads the unrolled kernel keeps its calls (64 x 8 pairs x 4224 tokens 149 us; 28 x 8 x 9800 49.9 against 72.7); cluster mode's
// go by cost (1 x 8 x 17879 54 -> 30 us, 5 x 4 x 4988 30 -> 22; 15 x 8 x 459 would be 17.2 -> 19.5; all before the folds had scales of their own, which
// cost this kernel 7 %).  Eight heads run as two times four.
// head_dim 64 halves the expansion and not the softmax, and cluster mode has less to gain from (48 shapes: 0.40 to 0.9 from about 8 tiles per
// SM on, up to 1.5 below): by cost at every width.
// One launch against two (kernel and merge): a small call takes less time on the device than the host needs for it, and there the second
// launch costs about 2 us whatever the kernel does.  Drawn by packed tiles per SM (cluster mode's estimate does not tell these apart):
// 16 steps of a generation at 2 bits in cluster mode and here, 0.3 tiles per SM (1 x 8 x 500 tokens) 361 and 389 us, 2.6 (4 x 8 x 900) 333 and
// 370, 4.0 (2 x 8 x 2500) 405 and 366; one call at 3.1 (2 x 8 x 2000) 18.9 and 15.1.  These are eager loops at 2 bits; a captured graph, where the host is
// not the limit, would gain by this kernel below the line too.
// Bytes per value (planes) at 2 bits, head_dim 128 and up to four heads: three where cluster mode was the choice without this kernel, whose error is that of
// an fp32 evaluation, two where the unrolled kernel was (5e-5 to 2e-4 there, 1e-5 to 4e-5 with two planes).  So no call is less precise than by
// the choice between those two, and the line between the two errors is theirs (3 x 2 pairs: 4928 tokens two planes, 4992 three).
constexpr float kOneLaunchTiles = 3.f;
constexpr float kUmmaBase = 14.5f, kUmmaBase8 = 15.0f;                          // us
constexpr float kUmmaTile[4] = {0.30f, 0.55f, 0.72f, 1.0f}, kUmmaTile64 = 0.9f;  // us per packed tile on an SM [bits]; at head_dim 64 of it
// At head_dim 64 a residual tile weighs more than the 0.31 of a packed one that it counts for everywhere (33 x 8 x 592 at 4 bits has 16 of them on an SM
// beside 12 packed ones: 31.9 us here and 22.0 by the general kernel's cut), and the estimates of that cut and of clusters are high there (1.0 to 1.7 of
// the device time), as this kernel's is (1.0 to 1.4).  Over 190 calls that go by cost the choice without this weight and these margins was slower than the
// other kernel by more than 3 % in 25 (up to 1.45), with them in 6 (up to 1.11); what both lose to the better of the two is 2.4 % on average.
// Of 195 other calls it gives 76 to this kernel, at 0.73 of the other's time on average, 7 of them slower by more than 3 % (up to 1.28).
constexpr float kUmmaDense64 = 0.6f;                                            // us per residual tile on an SM, besides
constexpr float kUmmaMargin = 0.95f, kUmmaMarginCut64 = 0.9f;
bool choose_umma(const MzDecodeParams& p, const MzDecodeParams& c, bool clusters, int sm_count) {
  if (clusters && (float)((long long)p.s.batch * p.s.kv_heads * p.s.k_groups) < kOneLaunchTiles * (float)sm_count) return false;
  if (p.s.head_dim == 128 && p.s.bits < 4) return true;
  if (!clusters && mz_decode_flat_supported(p)) return false;
  MzTilesPlan t = {};
  describe_tiles(t, p);
  const float x = tiles_per_sm(p, t, sm_count), tile = kUmmaTile[p.s.bits - 1] * (p.s.head_dim == 64 ? kUmmaTile64 : 1.0f);
  float us = p.gqa > 4 ? kUmmaBase8 + 2.0f * tile * x : kUmmaBase + tile * x;
  if (p.s.head_dim == 64) us += kUmmaDense64 * (float)((double)p.s.batch * p.s.kv_heads * (t.tiles_per_pair - t.packed_tiles) / sm_count);
  return us < (!clusters && p.s.head_dim == 64 ? kUmmaMarginCut64 : kUmmaMargin) * (clusters ? cluster_us(c) : cut_us(p, x));
}

}  // namespace

// Cost of a residual tile in CTAs that hold residual tiles only, in units of a packed tile among busy warps.  Such a
// warp is bound by memory latency.
constexpr int kDenseCtaCost = 36;

// the general kernel's table; asked for by the plans that run it only (a build costs a synchronisation and one of 16 slots)
static void take_lookup_entries(MzDecodeParams& p) {
  p.lut = p.s.k_groups > 0 && p.s.bits <= 4 ? mz_mma_lookup_entries(p.s.bits, true, p.s.alpha_key, p.s.alpha_value) : nullptr;
}

// an even cut by the kernel that serves it best
static int plan_cut(MzDecodeParams& p, const MzMmaKernel& k, int splits_request, int sm_count, size_t* slots) {
  const mz_kv_store& s = p.s;
  describe_tiles(p.tp, p);
  switch (choose_cut(p, tiles_per_sm(p, p.tp, sm_count))) {
    case Cut::kUnrolled: return mz_plan_flat(p, splits_request, sm_count, slots);
    case Cut::kSimt: return mz_plan_tiles(p, splits_request, sm_count, slots);
    case Cut::kGeneral: break;
  }
  take_lookup_entries(p);
  const long long pairs = (long long)s.batch * s.kv_heads;
  const int dense_tiles = (s.res_len + mzm::DT - 1) / mzm::DT;
  // enough packed work to fill every warp of the machine, and a residual window: split the CTAs
  if (splits_request == 0 && s.k_groups > 0 && dense_tiles > 0 && sm_count >= 8 &&
      pairs * s.k_groups >= (long long)sm_count * k.max_warps * 2) {
    describe_tiles(p.tp, p);
    const long long cost_d = (long long)dense_tiles * kDenseCtaCost, cost_p = (long long)s.k_groups * p.tp.cost_q;
    int n_d = (int)((sm_count * cost_d + cost_d + cost_p - 1) / (cost_d + cost_p));
    if (n_d < 1) n_d = 1;
    if (n_d > sm_count / 2) n_d = sm_count / 2;
    MzDecodeParams a = p, b = p;
    a.s.res_len = 0;
    b.s.k_groups = 0; b.s.v_tokens = 0;
    size_t slots_a = 0, slots_b = 0;
    const unsigned stage = (unsigned)(mzm::DT * 2 * s.head_dim);      // both plans lay out the shared memory alike
    int rc = plan_single(a, k, 0, sm_count - n_d, &slots_a, stage);
    if (rc == MZ_OK) rc = plan_single(b, k, 0, n_d, &slots_b, stage);
    const bool same_shape = rc == MZ_OK && a.tp.warps_per_cta == b.tp.warps_per_cta && a.tp.smem_bytes == b.tp.smem_bytes &&
                            a.tp.stage_bytes == b.tp.stage_bytes && a.tp.low_base == b.tp.low_base && a.tp.high_base == b.tp.high_base;
    if (same_shape) {
      p.tp = a.tp;
      p.tp2 = b.tp;
      p.slots_a = (long long)slots_a;
      p.hetero = a.tp.ctas;
      *slots = slots_a + slots_b;
      return MZ_OK;
    }
  }
  return plan_single(p, k, splits_request, sm_count, slots);
}

int mz_plan_mma(MzDecodeParams& p, int splits_request, int sm_count, size_t* slots) {
  p.hetero = 0;
  p.cluster = 0;
  MzMmaKernel k;
  if (!find_kernel(p, &k)) return mz_fail(MZ_ERR_UNSUPPORTED, "no tensor-core kernel for this shape");
  auto clustered = [&](MzDecodeParams& q, bool any_cost) {
    if (splits_request != 0 || !plan_cluster(q, k, sm_count, any_cost)) return false;
    *slots = 4;                                   // no records; a workspace is still asked for, so that its size is never 0
    take_lookup_entries(q);
    return true;
  };
  bool decided = false;                           // cluster mode has been planned already, and does not pay
  if (splits_request == 0 && mz_decode_umma_supported(p)) {
    MzDecodeParams c = p;
    const bool clusters = plan_cluster(c, k, sm_count);
    if (choose_umma(p, c, clusters, sm_count)) {
      MzDecodeParams t = p;
      size_t n = 0;
      if (mz_plan_umma(t, clusters || !mz_decode_flat_supported(p), 0, sm_count, &n) == MZ_OK &&
          (p.scratch_limit == 0 || n * sizeof(float) * (2 + (size_t)p.s.head_dim) <= p.scratch_limit)) {
        p = t;
        *slots = n;
        return MZ_OK;
      }
    }
    if (clusters) {
      p = c;
      *slots = 4;
      take_lookup_entries(p);
      return MZ_OK;
    }
    decided = true;
  }
  if (!decided && clustered(p, false)) return MZ_OK;
  p.cluster = 0;
  MzDecodeParams other = p;
  const int rc = plan_cut(p, k, splits_request, sm_count, slots);
  if (rc == MZ_OK && p.scratch_limit > 0 && *slots * sizeof(float) * (2 + (size_t)p.s.head_dim) > p.scratch_limit) {
    const size_t cut_slots = *slots;
    if (clustered(other, true)) p = other;
    else *slots = cut_slots;
  }
  return rc;
}

int mz_launch_decode_mma(const MzDecodeParams& p, cudaStream_t st) {
  if (p.tp.kind == 3) return mz_launch_decode_flat(p, st);
  MzMmaKernel k;
  if (!find_kernel(p, &k)) return mz_fail(MZ_ERR_UNSUPPORTED, "no tensor-core kernel for this shape");
  if (p.tp.smem_bytes > 48 * 1024) {
    // the limit is a property of the function on a device: raised to the most any plan uses, once
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, bool> raised;
    int dev = 0;
    MZ_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    bool& done = raised[{dev, k.fn}];
    if (!done) {
      MZ_CUDA(cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
      done = true;
    }
  }
  // programmatic dependent launch: harmless after a kernel that never signals (the launch then happens at its
  // completion, as usual); after one that does, the prologue overlaps it
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.hetero > 0 ? p.tp.ctas + p.tp2.ctas : p.tp.ctas));
  cfg.blockDim = dim3((unsigned)p.tp.warps_per_cta * 32);
  cfg.dynamicSmemBytes = p.tp.smem_bytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)p.cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.cluster > 1 ? 2 : 1;
  void* args[] = {(void*)&p};
  MZ_CUDA(cudaLaunchKernelExC(&cfg, k.fn, args));
  MZ_LAUNCH_CHECK("decode_mma");
  return MZ_OK;
}
