// bf16 x bf16 products of omc_linear on tcgen05: Y[b] = act(alpha X[b] W[b]^T + bias) (* sigmoid(gate)) for a batch of problems that are column slices
// of shared buffers (the heads of a latent attention: W_uk absorbed into the query, W_uv behind the attention).
//
// One CTA per 128 x BN tile, several CTAs per SM instead of a persistent loop: K is short (128 to 512), so a tile is a load, a few MMAs and an
// epilogue, and another CTA's epilogue hides the load. Warp 0: TMA (three-dimensional maps: K, rows, batch; edges arrive as zeros). Warp 1:
// MMA issuer. Warps 2..5: epilogue, thread = row. The K terms of an output are added in one order whatever the tile, so a row's result does
// not depend on M.
// What bounds it: the output's and the gate's bytes. RATE
#include "linear_args.cuh"
#include "sm100_step.cuh"

namespace omc {

constexpr int kHgThreads = 192, kHgBM = 128, kHgBK = 64, kHgMaxStages = 4;

static __device__ unsigned int g_linear_failures;   // waits that ran out

struct HgShared {
  uint64_t full[kHgMaxStages], empty[kHgMaxStages], done;
  uint32_t tmem, dead;
};

template <int BN, typename TY>
__global__ void __launch_bounds__(kHgThreads) linear_sm100_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w, LinearArgs a,
                                                                  int stages, bool x_shared, bool w_shared, bool vec_out, bool vec_gate) {
  constexpr int kA = kHgBM * 128, kStage = kA + BN * 128;
  extern __shared__ uint8_t hg_raw[];
  __shared__ HgShared shared;
  HgShared* sh = &shared;
  uint8_t* ring = hg_raw + ((1024u - (smem_u32(hg_raw) & 1023u)) & 1023u);
  const int m0 = blockIdx.y * kHgBM, n0 = blockIdx.x * BN, b = blockIdx.z;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nk = (a.K + kHgBK - 1) / kHgBK;
  auto wait = [&](uint64_t* bar, uint32_t parity) { wait_bounded(bar, parity, &sh->dead, &g_linear_failures); };
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
      for (int kb = stages; kb < nk; ++kb) {
        wait(&sh->empty[kb % stages], (kb / stages - 1) & 1);
        load(kb);
      }
      for (int kb = max(0, nk - stages); kb < nk; ++kb) wait(&sh->full[kb % stages], (kb / stages) & 1);   // nothing is on its way any more
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(kHgBM, BN);
      for (int kb = 0; kb < nk; ++kb) {
        wait(&sh->full[kb % stages], (kb / stages) & 1);
        tc_fence_after();
        const uint32_t sa = smem_u32(ring + (kb % stages) * kStage);
        const uint64_t da = make_sw128_kmajor_desc(sa), db = make_sw128_kmajor_desc(sa + kA);
#pragma unroll
        for (int k = 0; k < kHgBK / 16; ++k) umma_bf16<1>(tmem, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
        umma_commit(&sh->empty[kb % stages]);
      }
      umma_commit(&sh->done);
    }
  } else {
    const int quarter = warp & 3, m = m0 + quarter * 32 + lane;
    const bool row_ok = m < a.M;
    TY* y = static_cast<TY*>(a.Y) + (long long)b * a.sy + (long long)m * a.ldy;
    const long long g0 = (long long)m * a.ldg + (long long)b * a.sg;
    const bf16_t* bias = a.bias != nullptr ? static_cast<const bf16_t*>(a.bias) + b * a.sbias : nullptr;
    wait(&sh->done, 0);
    tc_fence_after();
    for (int c = 0; c < BN && n0 + c < a.N; c += 32) {
      uint32_t v[32];
      tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + c, v);
      tmem_ld_wait();
      if (!row_ok) continue;
      const int n = n0 + c, left = min(32, a.N - n);
      float f[32];
#pragma unroll
      for (int j = 0; j < 32; ++j)
        f[j] = apply_act(__uint_as_float(v[j]) * a.alpha + (bias != nullptr && j < left ? __bfloat162float(bias[n + j]) : 0.f), a.act);
      if (a.gate != nullptr) {
        if (vec_gate && left == 32) {
          if (a.gate_dt == OMC_DT_F32) {
            const float4* g = reinterpret_cast<const float4*>(static_cast<const float*>(a.gate) + g0 + n);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float4 z = g[j];
              f[4 * j] /= 1.f + __expf(-z.x), f[4 * j + 1] /= 1.f + __expf(-z.y), f[4 * j + 2] /= 1.f + __expf(-z.z), f[4 * j + 3] /= 1.f + __expf(-z.w);
            }
          } else {
            const uint4* g = reinterpret_cast<const uint4*>(static_cast<const bf16_t*>(a.gate) + g0 + n);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 z = g[j];
              const uint32_t w[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float2 e = unpack_bf16(w[i]);
                f[8 * j + 2 * i] /= 1.f + __expf(-e.x), f[8 * j + 2 * i + 1] /= 1.f + __expf(-e.y);
              }
            }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (j < left) {
              const float z = a.gate_dt == OMC_DT_F32 ? static_cast<const float*>(a.gate)[g0 + n + j] : ldf(static_cast<const bf16_t*>(a.gate) + g0 + n + j);
              f[j] /= 1.f + __expf(-z);
            }
        }
      }
      if (vec_out && left == 32) {
        if constexpr (sizeof(TY) == 4) {
#pragma unroll
          for (int j = 0; j < 8; ++j) reinterpret_cast<float4*>(y + n)[j] = make_float4(f[4 * j], f[4 * j + 1], f[4 * j + 2], f[4 * j + 3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            reinterpret_cast<uint4*>(y + n)[j] = make_uint4(pack_bf16(f[8 * j], f[8 * j + 1]), pack_bf16(f[8 * j + 2], f[8 * j + 3]),
                                                            pack_bf16(f[8 * j + 4], f[8 * j + 5]), pack_bf16(f[8 * j + 6], f[8 * j + 7]));
        }
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (j < left) stf(y + n + j, f[j]);
      }
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
  int rc = step_tensor_map(&tx, a.X, a.K, a.M, a.ldx, a.sx > 0 ? batch : 1, a.sx, kHgBM);   // stride 0: the batch shares the operand
  if (rc == OMC_OK) rc = step_tensor_map(&tw, a.W, a.K, a.N, a.ldw, a.sw > 0 ? batch : 1, a.sw, BN);
  if (rc != OMC_OK) return rc;
  constexpr int stage = (kHgBM + BN) * 128, max_smem = kHgMaxStages * stage + 1024;
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
  const dim3 grid((a.N + BN - 1) / BN, (a.M + kHgBM - 1) / kHgBM, batch);
  linear_sm100_kernel<BN, TY><<<grid, kHgThreads, stages * stage + 1024, st>>>(tx, tw, a, stages, a.sx == 0, a.sw == 0, vec_out, vec_gate);
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

// X and W bf16 with rows and batch items on 16-byte boundaries (mma_operands_ok of linear_any.cu)
int linear_sm100(const LinearArgs& a, int y_dt, int batch, cudaStream_t st) {
  if (y_dt == OMC_DT_F32) return hg_launch_typed<float>(a, batch, st);
  if (y_dt == OMC_DT_BF16) return hg_launch_typed<bf16_t>(a, batch, st);
  return set_error(OMC_ERR_ARG, "omc_linear: unknown output dtype");
}

int latent_sm100_failures(unsigned int* n);   // latent_attention_sm100.cu

}  // namespace omc

extern "C" int omc_step_wait_failures(unsigned int* count) {
  unsigned int linear = 0, latent = 0;
  if (count == nullptr) return omc::set_error(OMC_ERR_ARG, "omc_step_wait_failures: bad argument");
  if (cudaMemcpyFromSymbol(&linear, omc::g_linear_failures, sizeof(linear)) != cudaSuccess || omc::latent_sm100_failures(&latent) != OMC_OK)
    return omc::set_error(OMC_ERR_CUDA, "omc_step_wait_failures: the counters could not be read");
  *count = linear + latent;
  return OMC_OK;
}
