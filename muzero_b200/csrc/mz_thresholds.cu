// The unit-space thresholds of the packed quantizer (see mz_quant16.cuh): built on the device, once per
// (device, type, bits, alpha, eps), by bisecting the reference's chain over the 16-bit units in [0, 1].
#include <map>
#include <mutex>
#include <tuple>

#include "mz_quant16.cuh"

namespace {
// thread = (anchor, k): the smallest unit whose code reaches k + 1
template <int DT>
__global__ void build_thresholds_kernel(uint16_t* __restrict__ out, int bits, float eps, const uint16_t* __restrict__ ctab, int n) {
  const int per_row = 1 << bits;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n * per_row) return;
  const int k = i % per_row + 1, top = per_row - 1;
  const float eps_t = MzType<DT>::round(eps);
  mzq::Anchor<DT> c;
  c.set(mz_u16_to_float((uint16_t)(i / per_row), DT), (float)top, eps_t);
  int lo = 0, hi = n;                       // first unit index with code >= k; n = none
  if (k > top) lo = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (mzq::code_of_unit<DT>(mz_u16_to_float((uint16_t)mid, DT), c, (float)top, ctab, n) >= k) hi = mid;
    else lo = mid + 1;
  }
  out[i] = lo < n ? (uint16_t)lo : (uint16_t)(mzq::P2<DT>::INF2 & 0xffffu);
}

std::mutex g_mu;
constexpr size_t kMaxTables = 32;           // per process; further (alpha, eps) combinations use the plain chain
std::map<std::tuple<int, int, int, float, float>, uint16_t*> g_tables;
}  // namespace

// *dev_table = nullptr when no table can be provided (bits above 4, all slots taken, stream capture in progress): the
// caller then runs the plain chain.  The first request launches one kernel on the default stream and waits for it.
int mz_get_unit_thresholds(int dtype, int bits, float alpha, float eps, const uint16_t** dev_table) {
  *dev_table = nullptr;
  if (bits > 4) return MZ_OK;
  int dev = 0;
  MZ_CUDA(cudaGetDevice(&dev));
  const uint16_t* ctab;
  int n;
  int rc = mz_get_compand_table(dtype, alpha, &ctab, &n);
  if (rc) return rc;
  std::lock_guard<std::mutex> lk(g_mu);
  const auto key = std::make_tuple(dev, dtype, bits, alpha, eps);
  auto it = g_tables.find(key);
  if (it == g_tables.end()) {
    if (g_tables.size() >= kMaxTables) return MZ_OK;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(cudaStreamLegacy, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
      (void)cudaGetLastError();
      return MZ_OK;
    }
    uint16_t* d = nullptr;
    const int total = n << bits;
    MZ_CUDA(cudaMalloc(&d, (size_t)total * sizeof(uint16_t)));
    if (dtype == MZ_BF16) build_thresholds_kernel<MZ_BF16><<<(total + 255) / 256, 256>>>(d, bits, eps, ctab, n);
    else build_thresholds_kernel<MZ_F16><<<(total + 255) / 256, 256>>>(d, bits, eps, ctab, n);
    MZ_LAUNCH_CHECK("build_thresholds");
    MZ_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
    it = g_tables.emplace(key, d).first;
  }
  *dev_table = it->second;
  return MZ_OK;
}
