// Host side of the tensor-memory kernels: what the device offers, kernel attributes, launches and copy-engine descriptors.
#pragma once
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <stdint.h>
#include <string.h>

#include <mutex>

#include "epilogue.cuh"

namespace vb {

inline PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  });
  return g_encode;
}

struct DeviceInfo {
  int sms = 0, cc_major = 0, cc_minor = 0, max_smem = 0, smem_per_sm = 0, l2_bytes = 0;
  bool ok = false;
};
inline DeviceInfo device_info() {
  static DeviceInfo cache[64];
  static std::mutex mu;
  int dev = 0;
  DeviceInfo none;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return none;
  std::lock_guard<std::mutex> lock(mu);   // a record is filled and read under the lock: no half-written fields
  if (!cache[dev].ok) {
    DeviceInfo d;
    if (cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return none;
    cudaDeviceGetAttribute(&d.cc_major, cudaDevAttrComputeCapabilityMajor, dev);
    cudaDeviceGetAttribute(&d.cc_minor, cudaDevAttrComputeCapabilityMinor, dev);
    cudaDeviceGetAttribute(&d.max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&d.smem_per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&d.l2_bytes, cudaDevAttrL2CacheSize, dev);
    d.ok = true;
    cache[dev] = d;
  }
  return cache[dev];
}

// cudaFuncSetAttribute per (kernel, device), repeated only when a larger ring is asked for.
// All kernels share one C++ function-pointer type, so the record is keyed by the pointer value.  The table
// holds every instantiation of the library on up to 16 devices; beyond that the attribute is simply set again
// on every launch of the pairs that found no room (correct, a little slower).
inline int ensure_smem(const void* kernel, int bytes) {
  struct Rec { const void* fn; int dev; int bytes; };
  constexpr int kRecs = 192 * 16;
  static Rec recs[kRecs];
  static int n_recs = 0;
  static std::mutex mu;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -1;
  std::lock_guard<std::mutex> lock(mu);
  Rec* r = nullptr;
  for (int i = 0; i < n_recs; ++i)
    if (recs[i].fn == kernel && recs[i].dev == dev) r = &recs[i];
  if (r != nullptr && r->bytes >= bytes) return 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return -1;
  if (r == nullptr && n_recs < kRecs) r = &recs[n_recs++];
  if (r != nullptr) { r->fn = kernel; r->dev = dev; r->bytes = bytes; }
  return 0;
}

template <typename T>
struct same_type { using type = T; };
// overlapped: the launch may start beside the end of the kernel before it.
template <typename... P>
cudaError_t launch_kernel(bool overlapped, void (*kernel)(P...), dim3 grid, int threads, int smem_bytes, cudaStream_t stream, const typename same_type<P>::type&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlapped ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <typename... P>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, int threads, int smem_bytes, cudaStream_t stream, const typename same_type<P>::type&... args) {
  return launch_kernel<P...>(true, kernel, grid, threads, smem_bytes, stream, args...);
}
// Every launch reports its own status.  (The runtime's last error is the last call's that failed, which may be an earlier entry's:
// cudaGetLastError behind a launch would report that one.)
inline int status_of(cudaError_t rc) { return rc == cudaSuccess ? VOID_OK : VOID_ERR_CUDA; }
// Launches that follow one another on a stream; none after the first that failed.
class Launches {
 public:
  explicit Launches(cudaStream_t stream) : stream_(stream) {}
  template <typename... P>
  void run(void (*kernel)(P...), dim3 grid, int threads, const typename same_type<P>::type&... args) {
    if (rc_ == cudaSuccess) rc_ = launch_kernel<P...>(false, kernel, grid, threads, 0, stream_, args...);
  }
  int status() const { return status_of(rc_); }

 private:
  cudaStream_t stream_;
  cudaError_t rc_ = cudaSuccess;
};

// B as a tensor for the copy engine, 128-byte swizzle, zero fill outside [K, N].  Elements of es bytes: every box is 128
// bytes (kPanelN / es columns) wide, a panel takes es of them.
//   whole (asked for when N is a multiple of a box): 3-D, dim0 = the columns of a box, dim1 = k, dim2 = box; one copy
//   fetches the 32 k-rows of np panels.  Otherwise, or when the driver refuses that view: 2-D, one box per copy.
inline bool panel_map(CUtensorMap* m, const void* b, int64_t ldb, int K, int N, int es, int np, bool* whole) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = get_encode();
  if (enc == nullptr) return false;
  const CUtensorMapDataType dt = (es == 1) ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                 : (es == 2) ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT32;
  const int box_n = kPanelN / es;
  const CUtensorMapSwizzle swz = (es == 4) ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B;
  if (*whole) {
    const cuuint64_t gdim[3] = {(cuuint64_t)box_n, (cuuint64_t)K, (cuuint64_t)(N / box_n)};
    const cuuint64_t gstride[2] = {(cuuint64_t)ldb, (cuuint64_t)kPanelN};
    const cuuint32_t box[3] = {(cuuint32_t)box_n, (cuuint32_t)kTile, (cuuint32_t)(np * es)};
    const cuuint32_t estride[3] = {1, 1, 1};
    if (enc(m, dt, 3, const_cast<void*>(b), gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS)
      return true;
    *whole = false;
  }
  const cuuint64_t gdim[2] = {(cuuint64_t)N, (cuuint64_t)K};
  const cuuint64_t gstride[1] = {(cuuint64_t)ldb};
  const cuuint32_t box[2] = {(cuuint32_t)box_n, (cuuint32_t)kTile};
  const cuuint32_t estride[2] = {1, 1};
  return enc(m, dt, 2, const_cast<void*>(b), gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// B stored [N, K]: dim0 = k, dim1 = n; box 32 k x 128 n, swizzle span = the 32 * es bytes of a row
inline bool panel_map_transposed(CUtensorMap* m, const void* b, int64_t ldb, int K, int N, int es) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = get_encode();
  if (enc == nullptr) return false;
  const CUtensorMapDataType dt = (es == 1) ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                 : (es == 2) ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT32;
  const cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)N};
  const cuuint64_t gstride[1] = {(cuuint64_t)ldb};
  const cuuint32_t box[2] = {(cuuint32_t)kTile, (cuuint32_t)kPanelN};
  const cuuint32_t estride[2] = {1, 1};
  const CUtensorMapSwizzle sw = (es == 4) ? CU_TENSOR_MAP_SWIZZLE_128B
                                : (es == 2) ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
  return enc(m, dt, 2, const_cast<void*>(b), gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// C of 16-bit elements for tiled stores of 32 rows x 32 columns, 64-byte swizzle
inline bool store_map(CUtensorMap* m, void* out, int64_t ldc, int M, int N) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = get_encode();
  if (enc == nullptr) return false;
  const cuuint64_t gdim[2] = {(cuuint64_t)N, (cuuint64_t)M};
  const cuuint64_t gstride[1] = {(cuuint64_t)ldc * 2};
  const cuuint32_t box[2] = {32, (cuuint32_t)kTile};
  const cuuint32_t estride[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, out, gdim, gstride, box, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace vb
