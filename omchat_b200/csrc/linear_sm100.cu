// bf16 x bf16 products of omc_linear on tcgen05: Y[b] = act(alpha X[b] W[b]^T + bias) (* sigmoid(gate)) for a batch of problems that are column slices
// of shared buffers (the heads of a latent attention: W_uk absorbed into the query, W_uv behind the attention).
//
// One CTA per 128 x BN tile, several CTAs per SM instead of a persistent loop: K is short (128 to 512), so a tile is a load, a few MMAs and an
// epilogue, and another CTA's epilogue hides the load. Warp 0: TMA (three-dimensional maps: K, rows, batch; edges arrive as zeros). Warp 1:
// MMA issuer. Warps 2..5: epilogue, thread = row. The K terms of an output are added in one order whatever the tile, so a row's result does
// not depend on M.
// What bounds it: the output's and the gate's bytes (51 MB, 1.4 TB/s), behind the set-up and the first load of a tile. 3126 rows x 16 heads, 128 -> 512:
// 38 us = 172 TFLOP/s; 512 -> 128 with a gate per element 48 us; 32 rows: 6 us each (mma.sync with a two-stage cp.async ring before: 140, 141, 21).
#include "linear_args.cuh"
#include "sm100_step.cuh"

namespace omc {

constexpr int kHgThreads = 192, kHgBM = 128, kHgBK = 64, kHgMaxStages = 4;
constexpr int kHgPitch = 68, kHgSlabs = 4 * 32 * kHgPitch * 4;   // the epilogue's [32 rows][64 columns] fp32 per warp

static __device__ unsigned int g_linear_failures;   // waits that ran out

struct HgShared {
  uint64_t full[kHgMaxStages], empty[kHgMaxStages], done;
  uint32_t tmem, dead;
};

__device__ __forceinline__ void hg_row(const float* src, float alpha, float (&f)[8]) {
  const float4 lo = *reinterpret_cast<const float4*>(src), hi = *reinterpret_cast<const float4*>(src + 4);
  f[0] = lo.x * alpha, f[1] = lo.y * alpha, f[2] = lo.z * alpha, f[3] = lo.w * alpha, f[4] = hi.x * alpha, f[5] = hi.y * alpha, f[6] = hi.z * alpha, f[7] = hi.w * alpha;
}
__device__ __forceinline__ void hg_gates(const LinearArgs& a, long long at, float (&z)[8]) {   // eight neighbours from a 16-byte boundary
  if (a.gate_dt == OMC_DT_F32) {
    const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(a.gate) + at);
    const float4 g0 = p[0], g1 = p[1];
    z[0] = g0.x, z[1] = g0.y, z[2] = g0.z, z[3] = g0.w, z[4] = g1.x, z[5] = g1.y, z[6] = g1.z, z[7] = g1.w;
  } else {
    const uint4 g = *reinterpret_cast<const uint4*>(static_cast<const bf16_t*>(a.gate) + at);
    const float2 g0 = unpack_bf16(g.x), g1 = unpack_bf16(g.y), g2 = unpack_bf16(g.z), g3 = unpack_bf16(g.w);
    z[0] = g0.x, z[1] = g0.y, z[2] = g1.x, z[3] = g1.y, z[4] = g2.x, z[5] = g2.y, z[6] = g3.x, z[7] = g3.y;
  }
}
__device__ __forceinline__ void hg_store(float* y, const float (&f)[8]) {
  reinterpret_cast<float4*>(y)[0] = make_float4(f[0], f[1], f[2], f[3]);
  reinterpret_cast<float4*>(y)[1] = make_float4(f[4], f[5], f[6], f[7]);
}
__device__ __forceinline__ void hg_store(bf16_t* y, const float (&f)[8]) {
  *reinterpret_cast<uint4*>(y) = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
}

template <int BN, typename TY>
__global__ void __launch_bounds__(kHgThreads) linear_sm100_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w, LinearArgs a,
                                                                  int stages, bool x_shared, bool w_shared, bool vec_out, bool vec_gate, bool pair_gate, unsigned int* failed) {
  constexpr int kA = kHgBM * 128, kStage = kA + BN * 128;
  extern __shared__ uint8_t hg_raw[];
  __shared__ HgShared shared;
  HgShared* sh = &shared;
  uint8_t* ring = hg_raw + ((1024u - (smem_u32(hg_raw) & 1023u)) & 1023u);
  const int m0 = blockIdx.y * kHgBM, n0 = blockIdx.x * BN, b = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nk = (a.K + kHgBK - 1) / kHgBK;
  const WaitReport report{&sh->dead, &g_linear_failures, failed};
  auto wait = [&](uint64_t* bar, uint32_t parity) { return wait_bounded(bar, parity, report); };
  auto drain = [&](uint64_t* bar, uint32_t parity) { drain_bounded(bar, parity, report); };
  auto load = [&](int kb) {
    uint8_t* sa = ring + (kb % stages) * kStage;
    uint64_t* bar = &sh->full[kb % stages];
    mbar_arrive_expect_tx(bar, kStage);
    tma_load_3d(sa, &tm_x, bar, kb * kHgBK, m0, x_shared ? 0 : b);
    tma_load_3d(sa + kA, &tm_w, bar, kb * kHgBK, n0, w_shared ? 0 : b);
  };
  if (tid == 0) {
    tma_prefetch_desc(&tm_x);
    tma_prefetch_desc(&tm_w);
    for (int s = 0; s < stages; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    mbar_init(&sh->done, 1);
    sh->dead = 0u;
    fence_barrier_init();
    fence_proxy_async();
    for (int kb = 0; kb < min(stages, nk); ++kb) load(kb);
  }
  if (warp == 1) {
    tmem_alloc<1>(&sh->tmem, BN);
    tmem_relinquish<1>();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem;
  if (warp == 0) {
    if (lane == 0) {
      int issued = min(stages, nk);
      for (; issued < nk && wait(&sh->empty[issued % stages], (issued / stages - 1) & 1); ++issued) load(issued);
      for (int kb = max(0, issued - stages); kb < issued; ++kb) drain(&sh->full[kb % stages], (kb / stages) & 1);   // nothing is on its way any more
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(kHgBM, BN);
      for (int kb = 0; kb < nk; ++kb) {
        if (!wait(&sh->full[kb % stages], (kb / stages) & 1)) break;
        tc_fence_after();
        const uint32_t sa = smem_u32(ring + (kb % stages) * kStage);
        const uint64_t da = make_sw128_kmajor_desc(sa), db = make_sw128_kmajor_desc(sa + kA);
#pragma unroll
        for (int k = 0; k < kHgBK / 16; ++k) umma_bf16<1>(tmem, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
        umma_commit(&sh->empty[kb % stages]);
      }
      umma_commit(&sh->done);
      drain(&sh->done, 0);   // every product that was issued is done
    }
  } else {
    // thread = row while the accumulator is read, eight neighbouring threads = one row of 64 columns while gates come in and outputs go out
    // (lines of 32 rows per store otherwise); the ring is free by then
    const int quarter = warp & 3;
    float* slab = reinterpret_cast<float*>(ring) + quarter * 32 * kHgPitch;
    const bool plain = vec_out && a.act == OMC_ACT_NONE && a.bias == nullptr && (a.gate == nullptr || vec_gate);
    const bool done = wait_bounded_warp(&sh->done, 0, report);
    tc_fence_after();
    for (int c = 0; done && c < BN && n0 + c < a.N; c += 64) {
#pragma unroll
      for (int part = 0; part < 2; ++part) {
        uint32_t v[32];
        tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + c + 32 * part, v);
        tmem_ld_wait();
        uint4* dst = reinterpret_cast<uint4*>(slab + lane * kHgPitch + 32 * part);
#pragma unroll
        for (int j = 0; j < 8; ++j) dst[j] = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      }
      __syncwarp();
      const int n = n0 + c + (lane & 7) * 8, left = min(8, a.N - n);
      const bf16_t* bias = a.bias != nullptr ? static_cast<const bf16_t*>(a.bias) + b * a.sbias : nullptr;
      if (plain && n0 + c + 64 <= a.N && m0 + quarter * 32 + 32 <= a.M) {
        // a whole piece without activation or bias: no branch between the loads and the stores of its 8 x 4 rows
        const long long m = m0 + quarter * 32 + (lane >> 3);
        const float* src = slab + (lane >> 3) * kHgPitch + (lane & 7) * 8;
        TY* y = static_cast<TY*>(a.Y) + (long long)b * a.sy + m * a.ldy + n;
        if (a.gate == nullptr) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            float f[8];
            hg_row(src + i * 4 * kHgPitch, a.alpha, f);
            hg_store(y + (long long)(i * 4) * a.ldy, f);
          }
        } else {
          const long long at = m * a.ldg + (long long)b * a.sg + n;
#pragma unroll
          for (int i0 = 0; i0 < 8; i0 += 4) {
            float z[4][8];
#pragma unroll
            for (int i = 0; i < 4; ++i) hg_gates(a, at + (long long)((i0 + i) * 4) * a.ldg, z[i]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float f[8];
              hg_row(src + (i0 + i) * 4 * kHgPitch, a.alpha, f);
#pragma unroll
              for (int j = 0; j < 8; ++j) f[j] /= 1.f + __expf(-z[i][j]);   // as at the edges: bits do not depend on the tile
              hg_store(y + (long long)((i0 + i) * 4) * a.ldy, f);
            }
          }
        }
        __syncwarp();
        continue;
      }
#pragma unroll 2
      for (int i = 0; i < 8 && left > 0; ++i) {
        const int row = i * 4 + (lane >> 3), m = m0 + quarter * 32 + row;
        if (m >= a.M) break;
        float f[8];
        hg_row(slab + row * kHgPitch + (lane & 7) * 8, a.alpha, f);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = apply_act(f[j] + (bias != nullptr && j < left ? __bfloat162float(bias[n + j]) : 0.f), a.act);
        if (a.gate != nullptr) {
          const long long at = (long long)m * a.ldg + (long long)b * a.sg + n;
          float z[8];
          if (vec_gate && left == 8) {
            hg_gates(a, at, z);
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              z[j] = j >= left ? 0.f : (a.gate_dt == OMC_DT_F32 ? static_cast<const float*>(a.gate)[at + j] : ldf(static_cast<const bf16_t*>(a.gate) + at + j));
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] /= 1.f + (pair_gate && n + (j | 1) < a.N ? __expf(-z[j]) : expf(-z[j]));
        }
        TY* y = static_cast<TY*>(a.Y) + (long long)b * a.sy + (long long)m * a.ldy + n;
        if (vec_out && left == 8) {
          hg_store(y, f);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j < left) stf(y + j, f[j]);
        }
      }
      __syncwarp();
    }
    tc_fence_before();
  }
  __syncwarp();
  __syncthreads();
  if (warp == 1) tmem_dealloc<1>(tmem, BN);
}

template <int BN, typename TY>
static int hg_launch(const LinearArgs& a, int batch, cudaStream_t st) {
  CUtensorMap tx, tw;
  unsigned int* failed = nullptr;
  int rc = step_failure_word(&failed);
  if (rc == OMC_OK) rc = step_tensor_map(&tx, a.X, a.K, a.M, a.ldx, a.sx > 0 ? batch : 1, a.sx, kHgBM);   // stride 0: the batch shares the operand
  if (rc == OMC_OK) rc = step_tensor_map(&tw, a.W, a.K, a.N, a.ldw, a.sw > 0 ? batch : 1, a.sw, BN);
  if (rc != OMC_OK) return rc;
  constexpr int stage = (kHgBM + BN) * 128, max_smem = kHgMaxStages * stage + 1024;
  static_assert(max_smem >= kHgSlabs + 1024, "the ring holds the epilogue's slabs");
  static bool done[kMaxDevices] = {};
  const int dev = cur_device();
  if (!done[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(linear_sm100_kernel<BN, TY>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
    if (e != cudaSuccess) return set_error(OMC_ERR_CUDA, cudaGetErrorString(e));
    done[dev] = true;
  }
  // two CTAs per SM: 2 stages of 48 KB, 3 of 32 KB, 4 of 24 KB - and no more than K needs
  const int fits = BN == 256 ? 2 : (BN == 128 ? 3 : 4), nk = (a.K + kHgBK - 1) / kHgBK, stages = nk < fits ? nk : fits;
  auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  const int ye = 16 / (int)sizeof(TY), ge = a.gate_dt == OMC_DT_F32 ? 4 : 8;
  const bool vec_out = aligned(a.Y) && a.ldy % ye == 0 && a.sy % ye == 0, vec_gate = aligned(a.gate) && a.ldg % ge == 0 && a.sg % ge == 0;
  // the hardware exponential for gates that come in pairs on 8-byte boundaries, the precise one for those at odd strides and an odd last column
  const bool pair_gate = a.ldg % 2 == 0 && a.sg % 2 == 0 && reinterpret_cast<uintptr_t>(a.gate) % 8 == 0;
  const dim3 grid((a.N + BN - 1) / BN, (a.M + kHgBM - 1) / kHgBM, batch);
  const int smem = (stages * stage > kHgSlabs ? stages * stage : kHgSlabs) + 1024;
  linear_sm100_kernel<BN, TY><<<grid, kHgThreads, smem, st>>>(tx, tw, a, stages, a.sx == 0, a.sw == 0, vec_out, vec_gate, pair_gate, failed);
  return check_launch("omc_linear");
}

template <typename TY>
static int hg_launch_typed(const LinearArgs& a, int batch, cudaStream_t st) {
  // the widest tile that still gives every SM a CTA (steps of few rows are a matter of CTAs, not of reuse)
  const long long rows = (a.M + kHgBM - 1) / kHgBM;
  if (a.N > 128 && rows * ((a.N + 255) / 256) * batch >= 148) return hg_launch<256, TY>(a, batch, st);
  if (a.N > 64 && rows * ((a.N + 127) / 128) * batch >= 148) return hg_launch<128, TY>(a, batch, st);
  return hg_launch<64, TY>(a, batch, st);
}

// X and W bf16 with rows and batch items on 16-byte boundaries (sm100_operands_ok of linear_any.cu)
int linear_sm100(const LinearArgs& a, int y_dt, int batch, cudaStream_t st) {
  if (y_dt == OMC_DT_F32) return hg_launch_typed<float>(a, batch, st);
  if (y_dt == OMC_DT_BF16) return hg_launch_typed<bf16_t>(a, batch, st);
  return set_error(OMC_ERR_ARG, "omc_linear: unknown output dtype");
}

int latent_sm100_failures(unsigned int* n);   // latent_attention_sm100.cu
int window_sm100_failures(unsigned int* n);   // window_attention_sm100.cu

// out: a wait for a barrier that nothing arrives at; the next one for it; one for a barrier that another thread arrives at only behind it; a drain of
// that one
__global__ void step_wait_selfcheck_kernel(int32_t* out, unsigned int* failed) {
  __shared__ uint64_t never, late;
  __shared__ uint32_t dead, refused;
  if (threadIdx.x == 0) {
    mbar_init(&never, 1);
    mbar_init(&late, 1);
    dead = refused = 0u;
    fence_barrier_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const WaitReport report{&dead, &g_linear_failures, failed};
    out[0] = wait_bounded(&never, 0, report, 8);
    out[1] = wait_bounded(&never, 0, report);
    out[2] = wait_bounded(&late, 0, report);
    *reinterpret_cast<volatile uint32_t*>(&refused) = 1u;
    out[3] = drain_bounded(&late, 0, report);
  } else if (threadIdx.x == 32) {
    for (int i = 0; i < 1000000 && !*reinterpret_cast<volatile uint32_t*>(&refused); ++i) __nanosleep(1000);   // thread 0 sets it after its eight tries
    __nanosleep(20000);
    mbar_arrive(&late);
  }
}

// One warp whose lanes wait for different barriers, the lower half for one whose phase has come, the others for one that nothing arrives at. out: every
// lane's answer.
__global__ void step_wait_warp_selfcheck_kernel(int32_t* out, unsigned int* failed) {
  __shared__ uint64_t come, never;
  __shared__ uint32_t dead;
  if (threadIdx.x == 0) {
    mbar_init(&come, 1);
    mbar_init(&never, 1);
    dead = 0u;
    fence_barrier_init();
    mbar_arrive(&come);
  }
  __syncwarp();
  const WaitReport report{&dead, &g_linear_failures, failed};
  out[threadIdx.x] = wait_bounded_warp(threadIdx.x < 16 ? &come : &never, 0, report, 8);
}

}  // namespace omc

extern "C" int omc_step_wait_failed(void) {
  const volatile unsigned int* words = omc::step_failure_words();
  int any = 0;
  for (int dev = 0; words != nullptr && dev < omc::kMaxDevices; ++dev) any |= words[dev] != 0u;
  return any;
}

extern "C" int omc_step_wait_selfcheck(int32_t* out, void* stream) {
  if (out == nullptr) return omc::set_error(OMC_ERR_ARG, "omc_step_wait_selfcheck: bad argument");
  unsigned int* failed = nullptr;
  if (const int rc = omc::step_failure_word(&failed); rc != OMC_OK) return rc;
  omc::step_wait_selfcheck_kernel<<<1, 64, 0, static_cast<cudaStream_t>(stream)>>>(out, failed);
  return omc::check_launch("omc_step_wait_selfcheck");
}

extern "C" int omc_step_wait_warp_selfcheck(int32_t* out, void* stream) {
  if (out == nullptr) return omc::set_error(OMC_ERR_ARG, "omc_step_wait_warp_selfcheck: bad argument");
  unsigned int* failed = nullptr;
  if (const int rc = omc::step_failure_word(&failed); rc != OMC_OK) return rc;
  omc::step_wait_warp_selfcheck_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(out, failed);
  return omc::check_launch("omc_step_wait_warp_selfcheck");
}

extern "C" int omc_step_wait_failures(unsigned int* count) {
  unsigned int linear = 0, latent = 0, window = 0;
  if (count == nullptr) return omc::set_error(OMC_ERR_ARG, "omc_step_wait_failures: bad argument");
  if (cudaMemcpyFromSymbol(&linear, omc::g_linear_failures, sizeof(linear)) != cudaSuccess || omc::latent_sm100_failures(&latent) != OMC_OK ||
      omc::window_sm100_failures(&window) != OMC_OK)
    return omc::set_error(OMC_ERR_CUDA, "omc_step_wait_failures: the counters could not be read");
  *count = linear + latent + window;
  return OMC_OK;
}
