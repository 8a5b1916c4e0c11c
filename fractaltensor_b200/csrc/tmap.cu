#include "tmap.h"

#include <atomic>
#include <mutex>

#include "ptx.cuh"

namespace ftb {

namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(p);
    }
  });
  return fn;
}

CUtensorMapDataType tmap_dtype(int dt) {
  switch (dt) {
    case FTB_F32: return CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    case FTB_F16: return CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    default: return CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  }
}
}  // namespace

namespace {
int encode_2d(CUtensorMap* out, const void* base, int dtype, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows,
              uint32_t box_cols, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return FTB_ERR_DRIVER;
  const size_t es = dtype_size(dtype);
  if ((reinterpret_cast<uintptr_t>(base) & 15) || ((ld * es) & 15)) return FTB_ERR_ALIGN;
  if (box_rows > 256 || box_cols > 256 || (swizzle == CU_TENSOR_MAP_SWIZZLE_128B && box_cols * es > 128)) return FTB_ERR_ARG;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * es};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(out, tmap_dtype(dtype), 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? FTB_OK : FTB_ERR_DRIVER;
}
}  // namespace

int make_tmap_2d(CUtensorMap* out, const void* base, int dtype, uint64_t rows, uint64_t cols, uint64_t ld,
                 uint32_t box_rows, uint32_t box_cols, bool swizzle128) {
  return encode_2d(out, base, dtype, rows, cols, ld, box_rows, box_cols,
                   swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE);
}

int make_tmap_2d_sw64(CUtensorMap* out, const void* base, int dtype, uint64_t rows, uint64_t cols, uint64_t ld,
                      uint32_t box_rows) {
  return encode_2d(out, base, dtype, rows, cols, ld, box_rows, static_cast<uint32_t>(64 / dtype_size(dtype)), CU_TENSOR_MAP_SWIZZLE_64B);
}

int make_tmap_3d(CUtensorMap* out, const void* base, int dtype, uint64_t cols, uint64_t rows, uint64_t planes,
                 uint64_t row_stride_bytes, uint64_t plane_stride_bytes, uint32_t box_cols, uint32_t box_rows,
                 uint32_t box_planes, bool swizzle128) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return FTB_ERR_DRIVER;
  const size_t es = dtype_size(dtype);
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (row_stride_bytes & 15) || (plane_stride_bytes & 15))
    return FTB_ERR_ALIGN;
  if (box_rows > 256 || box_cols > 256 || box_planes > 256 || (swizzle128 && box_cols * es > 128))
    return FTB_ERR_ARG;
  cuuint64_t dims[3] = {cols, rows, planes};
  cuuint64_t strides[2] = {row_stride_bytes, plane_stride_bytes};
  cuuint32_t box[3] = {box_cols, box_rows, box_planes};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(out, tmap_dtype(dtype), 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? FTB_OK : FTB_ERR_DRIVER;
}

int make_tmap_steps(CUtensorMap* out, const void* base, int dtype, uint64_t steps, uint64_t rows, uint64_t K, uint32_t box_rows,
                    uint32_t box_planes) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return FTB_ERR_DRIVER;
  const size_t row = K * dtype_size(dtype);
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (row & 15)) return FTB_ERR_ALIGN;
  if (K % 64 != 0 || box_rows > 256 || box_planes > 256) return FTB_ERR_ARG;
  cuuint64_t dims[4] = {64, rows, K / 64, steps};
  cuuint64_t strides[3] = {row, 128, rows * row};
  cuuint32_t box[4] = {64, box_rows, box_planes, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(out, tmap_dtype(dtype), 4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? FTB_OK : FTB_ERR_DRIVER;
}

int make_tmap_gates(CUtensorMap* out, const void* base, int dtype, uint64_t rows, uint64_t K) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return FTB_ERR_DRIVER;
  const size_t row = K * dtype_size(dtype);
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (row & 15)) return FTB_ERR_ALIGN;
  if (rows % 32 != 0) return FTB_ERR_ARG;
  cuuint64_t dims[4] = {K, 8, 4, rows / 32};
  cuuint64_t strides[3] = {4 * row, row, 32 * row};
  cuuint32_t box[4] = {64, 8, 4, 4};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(out, tmap_dtype(dtype), 4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? FTB_OK : FTB_ERR_DRIVER;
}

namespace {
// What a device is does not change: its attributes are asked for once (0 = not asked yet).  Devices
// past the table are asked on every call.
constexpr int kKnownDevices = 64;
std::atomic<int> g_major[kKnownDevices], g_sms[kKnownDevices];

int device_attribute(cudaDeviceAttr attr, std::atomic<int>* known) {
  int dev = 0, v = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return 0;
  if (dev < kKnownDevices && (v = known[dev].load(std::memory_order_relaxed)) != 0) return v;
  if (cudaDeviceGetAttribute(&v, attr, dev) != cudaSuccess) return 0;
  if (dev < kKnownDevices) known[dev].store(v, std::memory_order_relaxed);
  return v;
}
}  // namespace

int check_device_sm100() {
  return device_attribute(cudaDevAttrComputeCapabilityMajor, g_major) == 10 ? FTB_OK : FTB_ERR_ARCH;
}

namespace {
std::atomic<long long> g_launches{0};
}
void count_launch(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
long long launches_so_far() { return g_launches.load(std::memory_order_relaxed); }

int current_sm_count() { return device_attribute(cudaDevAttrMultiProcessorCount, g_sms); }

}  // namespace ftb
