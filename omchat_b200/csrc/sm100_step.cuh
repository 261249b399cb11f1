// What the tcgen05 kernels of the sequence-step library share: waits that end by themselves, and tensor maps made per launch.
#pragma once
#include <cuda.h>

#include "ptx.cuh"
#include "seq_common.cuh"

namespace omc {

// A wait gives up after this many tries (each lets the hardware suspend the thread for a while), or at once where another wait of the CTA
// has, and returns whether its phase has come. Who was refused issues no more copies and no more products; the CTA runs on to its end
// through the same sequence of block barriers. What it wrote is not valid, and `failures` (a counter in device memory) says so.
constexpr uint32_t kWaitTries = 1u << 22, kDrainTries = 1u << 20;
__device__ __forceinline__ bool wait_bounded(uint64_t* bar, uint32_t parity, uint32_t* dead, unsigned int* failures, uint32_t tries = kWaitTries) {
  for (uint32_t i = 0; !mbar_try_wait(bar, parity); ++i) {
    if (i >= tries && atomicExch(dead, 1u) == 0u) atomicAdd(failures, 1u);
    if (*reinterpret_cast<volatile uint32_t*>(dead)) return false;
  }
  return true;
}
// For copies and products that have been issued: none may be under way into shared or tensor memory when the CTA gives these back, so these
// waits have tries of their own whether or not another wait has given up.
__device__ __forceinline__ bool drain_bounded(uint64_t* bar, uint32_t parity, uint32_t* dead, unsigned int* failures) {
  for (uint32_t i = 0; i < kDrainTries; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  if (atomicExch(dead, 1u) == 0u) atomicAdd(failures, 1u);
  return false;
}

typedef CUresult (*TensorMapEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                      const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline TensorMapEncodeFn tensor_map_encode_fn() {
  static TensorMapEncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
    return reinterpret_cast<TensorMapEncodeFn>(p);
  }();
  return fn;
}

// bf16 [batch][rows][cols] (row and batch strides in elements, multiples of 8), boxes of 64 columns x box_rows rows, 128-byte swizzle.
inline int step_tensor_map(CUtensorMap* tm, const void* p, unsigned long long cols, unsigned long long rows, unsigned long long ld, int batch,
                           unsigned long long batch_stride, int box_rows) {
  TensorMapEncodeFn enc = tensor_map_encode_fn();
  if (enc == nullptr) return set_error(OMC_ERR_DRIVER, "cuTensorMapEncodeTiled entry point unavailable");
  cuuint64_t dim[3] = {cols, rows, (cuuint64_t)batch}, stride[2] = {ld * 2, batch > 1 ? batch_stride * 2 : ld * 2};
  cuuint32_t box[3] = {64u, (cuuint32_t)box_rows, 1u}, one[3] = {1u, 1u, 1u};
  if (enc(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(p), dim, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return set_error(OMC_ERR_DRIVER, "cuTensorMapEncodeTiled failed");
  return OMC_OK;
}
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const void* tmap, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(smem_dst)), "l"(tmap),
      "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

}  // namespace omc
