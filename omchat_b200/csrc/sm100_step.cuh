// What the tcgen05 kernels of the sequence-step library share: waits that end by themselves, and tensor maps made per launch.
#pragma once
#include <cuda.h>
#include <string.h>

#include "ptx.cuh"
#include "seq_common.cuh"

namespace omc {

// A wait gives up after this many tries (each lets the hardware suspend the thread for a while), or at once where another wait of the CTA
// has, and returns whether its phase has come. Who was refused issues no more copies and no more products; the CTA runs on to its end
// through the same sequence of block barriers. What it wrote is not valid, and a counter in device memory and a word in host memory say so:
// the launches of the library refuse while the word is set, and who has waited for a step's results can read it without waiting again.
constexpr uint32_t kWaitTries = 1u << 22, kDrainTries = 1u << 20;
struct WaitReport {
  uint32_t* dead;         // shared memory: a wait of this CTA has given up
  unsigned int* count;    // device memory
  unsigned int* host;     // this device's word of step_failure_words()
};
__device__ __forceinline__ void wait_ran_out(const WaitReport& r) {
  if (atomicExch(r.dead, 1u) != 0u) return;
  atomicAdd(r.count, 1u);
  *reinterpret_cast<volatile unsigned int*>(r.host) = 1u;
  __threadfence_system();
}
__device__ __forceinline__ bool wait_bounded(uint64_t* bar, uint32_t parity, const WaitReport& r, uint32_t tries = kWaitTries) {
  for (uint32_t i = 0; !mbar_try_wait(bar, parity); ++i) {
    if (i >= tries) wait_ran_out(r);
    if (*reinterpret_cast<volatile uint32_t*>(r.dead)) return false;
  }
  return true;
}
// A wait of all 32 lanes, with one answer for them all: whether every lane's phase has come. Where a wait gives up, lanes of a warp can see different
// answers of wait_bounded (a phase that comes at that moment); lanes that then went different ways would leave the others in the next barrier of
// the warp, or reach tensor memory without them.
__device__ __forceinline__ bool wait_bounded_warp(uint64_t* bar, uint32_t parity, const WaitReport& r, uint32_t tries = kWaitTries) {
  const bool come = wait_bounded(bar, parity, r, tries);
  return __all_sync(0xffffffffu, come);
}
// For copies and products that have been issued: none may be under way into shared or tensor memory when the CTA gives these back, so these
// waits have tries of their own whether or not another wait has given up.
__device__ __forceinline__ bool drain_bounded(uint64_t* bar, uint32_t parity, const WaitReport& r) {
  for (uint32_t i = 0; i < kDrainTries; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  wait_ran_out(r);
  return false;
}

// One word per device, in host memory that every device can write; nullptr where there is none to be had.
inline unsigned int* step_failure_words() {
  static unsigned int* words = [] {
    void* p = nullptr;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;   // the first launch may be one that is captured
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (cudaHostAlloc(&p, kMaxDevices * sizeof(unsigned int), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
      memset(p, 0, kMaxDevices * sizeof(unsigned int));
    } else {
      cudaGetLastError();
      p = nullptr;
    }
    cudaThreadExchangeStreamCaptureMode(&mode);
    return static_cast<unsigned int*>(p);
  }();
  return words;
}
// The current device's word, for a launch; an error where there is none or it is set.
inline int step_failure_word(unsigned int** word) {
  unsigned int* words = step_failure_words();
  if (words == nullptr) return set_error(OMC_ERR_CUDA, "no host memory for the step kernels' failure words");
  *word = words + cur_device();
  if (*reinterpret_cast<volatile unsigned int*>(*word) != 0u) return set_error(OMC_ERR_CUDA, "a wait of an earlier step kernel ran out on this device; what was computed since is not valid");
  return OMC_OK;
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
