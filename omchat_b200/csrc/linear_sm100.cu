// bf16 x bf16 products of omc_linear on tcgen05: Y[b] = act(alpha X[b] W[b]^T + bias) (* sigmoid(gate)) for a batch of problems that are column slices
// of shared buffers (the heads of a latent attention: W_uk absorbed into the query, W_uv behind the attention).
//
// One CTA per SM walks over tiles of 128 x BN: K is short (128 to 512), so a tile is a load, a few MMAs and an epilogue, and what overlaps them is the next tile.
// Warp 0: TMA (three-dimensional maps: K, rows, batch; edges arrive as zeros), as far ahead as the ring goes. Warp 1: MMA issuer, into one of two accumulators.
// The others: epilogue, thread = row; gates are asked for before the accumulator is waited for. The K terms of an output are added in one order whatever
// the tile, so a row's result does not depend on M.
// What bounds it: bytes (103 MB from L2 and 26 MB of output and gate in 19 to 21 us) behind 8 us of set-up, first load and last epilogue; before, one tile per CTA and two CTAs per SM, a tile's
// load (2.9 us) and epilogue (4.3, with a gate 11.5: fp32 slabs read with two-way bank conflicts, gates asked for behind the accumulator, divisions of 10
// instructions) followed one another. 3126 rows x 16 heads, us (before): 128 -> 512 19.3 (39.5); 512 -> 128 with a gate per element 20.6 (45.0; 26.8 with the quotients as plain divisions); 1338 rows without
// a gate 12.4 (31.0), 10.4 (18.6); 300 rows 7.6 (10.5), 10.3 (12.5); 94 rows 7.8 (10.5), 9.4 (19.6); 1 row 7.7 (8.0), 8.4 (8.9). 206 shapes of 1 to 3000 rows, 1 to 32 problems, 64 to 2048 terms
// and 64 to 4096 columns: 0.64 of the time before on average, 1.05 at most.
#include "fp32_pairs.cuh"
#include "linear_args.cuh"
#include "sm100_step.cuh"

namespace omc {

constexpr int kHgBM = 128, kHgBK = 64, kHgMaxStages = 6;
constexpr int kHgPitch = 68, kHgPitch16 = 36, kHgSlab = 32 * kHgPitch * 4;   // the epilogue's [32 rows][64 columns] per warp, fp32, or bf16 in rows of 36 words
// epilogue warps: two per quarter of the rows where a tile has columns for both
__host__ __device__ constexpr int hg_epilogue(int bn) { return bn == 64 ? 4 : 8; }
__host__ __device__ constexpr int hg_stages(int bn) { return bn == 256 ? 3 : (bn == 128 ? 4 : 6); }

static __device__ unsigned int g_linear_failures;   // waits that ran out

struct HgShared {
  uint64_t full[kHgMaxStages], empty[kHgMaxStages], acc_full[2], acc_empty[2], done;
  uint32_t tmem, dead;
};

// Where four columns (chunk c of a row's sixteen) lie in a slab's row: the upper eight chunks change places in pairs, so that the even (the odd) chunks of a row, which
// eight threads read at a time, are on different banks
__device__ __forceinline__ int hg_chunk(int c) { return (c ^ (c >> 3)) * 4; }
__device__ __forceinline__ void hg_row(const float* row, int eight, float alpha, float (&f)[8]) {   // columns 8 eight .. + 7
  const float4 lo = *reinterpret_cast<const float4*>(row + hg_chunk(2 * eight)), hi = *reinterpret_cast<const float4*>(row + hg_chunk(2 * eight + 1));
  f[0] = lo.x * alpha, f[1] = lo.y * alpha, f[2] = lo.z * alpha, f[3] = lo.w * alpha, f[4] = hi.x * alpha, f[5] = hi.y * alpha, f[6] = hi.z * alpha, f[7] = hi.w * alpha;
}
// eight neighbours from a 16-byte boundary, as they lie and as numbers
__device__ __forceinline__ void hg_gates_load(const LinearArgs& a, long long at, uint4 (&g)[2]) {
  if (a.gate_dt == OMC_DT_F32) {
    const uint4* p = reinterpret_cast<const uint4*>(static_cast<const float*>(a.gate) + at);
    g[0] = p[0], g[1] = p[1];
  } else {
    g[0] = *reinterpret_cast<const uint4*>(static_cast<const bf16_t*>(a.gate) + at);
  }
}
__device__ __forceinline__ void hg_gates(const LinearArgs& a, const uint4 (&g)[2], float (&z)[8]) {
  if (a.gate_dt == OMC_DT_F32) {
    z[0] = __uint_as_float(g[0].x), z[1] = __uint_as_float(g[0].y), z[2] = __uint_as_float(g[0].z), z[3] = __uint_as_float(g[0].w);
    z[4] = __uint_as_float(g[1].x), z[5] = __uint_as_float(g[1].y), z[6] = __uint_as_float(g[1].z), z[7] = __uint_as_float(g[1].w);
  } else {
    const float2 g0 = unpack_bf16(g[0].x), g1 = unpack_bf16(g[0].y), g2 = unpack_bf16(g[0].z), g3 = unpack_bf16(g[0].w);
    z[0] = g0.x, z[1] = g0.y, z[2] = g1.x, z[3] = g1.y, z[4] = g2.x, z[5] = g2.y, z[6] = g3.x, z[7] = g3.y;
  }
}
// f[e] / y[e], y >= 1 behind a gate, the bits of a division: by quotients2 unless one of the eight is out of its range
__device__ __forceinline__ void hg_divide(float (&f)[8], const float (&y)[8]) {
  float most = fabsf(f[0]), least = most, top = y[0];
#pragma unroll
  for (int e = 1; e < 8; ++e) most = fmaxf(most, fabsf(f[e])), least = fminf(least, fabsf(f[e])), top = fmaxf(top, y[e]);
  if (most <= 0x1p100f && least >= 0x1p-60f && top <= 0x1p62f) {
#pragma unroll
    for (int e = 0; e < 8; e += 2) quotients2(-f[e], -f[e + 1], y[e], y[e + 1], f[e], f[e + 1]);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] /= y[e];
  }
}
__device__ __forceinline__ void hg_store(float* y, const float (&f)[8]) {
  reinterpret_cast<float4*>(y)[0] = make_float4(f[0], f[1], f[2], f[3]);
  reinterpret_cast<float4*>(y)[1] = make_float4(f[4], f[5], f[6], f[7]);
}
__device__ __forceinline__ void hg_store(bf16_t* y, const float (&f)[8]) {
  *reinterpret_cast<uint4*>(y) = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
}

// The tiles of a launch and how many of them a CTA has, and their division: a CTA places its first tile, and every copy in its ring, in front of the first load, where divisions by
// numbers known at run time took 0.7 us
struct HgTiles {
  int n, m, each, more;        // tiles along N and M; tiles of every CTA, CTAs that have one more
  uint32_t by_n, by_m;         // ceil(2^32 / n), ceil(2^32 / m): exact for fewer than 2^16 tiles; 0 for more
  __device__ __forceinline__ static int over(int t, int d, uint32_t by) { return d == 1 ? t : (by != 0 ? (int)__umulhi((uint32_t)t, by) : t / d); }
};

template <int BN, typename TY>
__global__ void __launch_bounds__(64 + 32 * hg_epilogue(BN)) linear_sm100_kernel(const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_w, LinearArgs a,
                                                                                HgTiles tiles, bool x_shared, bool w_shared, bool vec_out, bool vec_gate, bool pair_gate,
                                                                                unsigned int* failed) {
  constexpr int kA = kHgBM * 128, kStage = kA + BN * 128, EP = hg_epilogue(BN);
  extern __shared__ uint8_t hg_raw[];
  __shared__ HgShared shared;
  HgShared* sh = &shared;
  uint8_t* ring = hg_raw + ((1024u - (smem_u32(hg_raw) & 1023u)) & 1023u);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nk = (a.K + kHgBK - 1) / kHgBK;
  constexpr int stages = hg_stages(BN);
  const int mine = tiles.each + ((int)blockIdx.x < tiles.more);   // this CTA's tiles: blockIdx.x, + gridDim.x, ...
  auto place = [&](int i, int& n0, int& m0, int& b) {
    const int t = blockIdx.x + i * gridDim.x, row = HgTiles::over(t, tiles.n, tiles.by_n);
    n0 = (t - row * tiles.n) * BN, b = HgTiles::over(row, tiles.m, tiles.by_m), m0 = (row - b * tiles.m) * kHgBM;
  };
  const WaitReport report{&sh->dead, &g_linear_failures, failed};
  auto wait = [&](uint64_t* bar, uint32_t parity) { return wait_bounded(bar, parity, report); };
  auto drain = [&](uint64_t* bar, uint32_t parity) { drain_bounded(bar, parity, report); };
  int n0 = 0, m0 = 0, b = 0;
  auto load = [&](int kb, int at) {   // piece kb of the tile at (m0, n0, b) as the at-th of this CTA's copies
    uint8_t* sa = ring + (at % stages) * kStage;
    uint64_t* bar = &sh->full[at % stages];
    mbar_arrive_expect_tx(bar, kStage);
    tma_load_3d(sa, &tm_x, bar, kb * kHgBK, m0, x_shared ? 0 : b);
    tma_load_3d(sa + kA, &tm_w, bar, kb * kHgBK, n0, w_shared ? 0 : b);
  };
  const int ahead = min(stages, mine * nk);   // copies that wait for nothing
  if (tid == 0) {
    tma_prefetch_desc(&tm_x);
    tma_prefetch_desc(&tm_w);
    for (int s = 0; s < stages; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sh->acc_full[s], 1);
      mbar_init(&sh->acc_empty[s], EP);
    }
    mbar_init(&sh->done, 1);
    sh->dead = 0u;
    fence_barrier_init();
    fence_proxy_async();
    for (int at = 0, kb = 0, i = 0; at < ahead; ++at, ++kb) {
      if (kb == nk) kb = 0, ++i;
      if (kb == 0) place(i, n0, m0, b);
      load(kb, at);
    }
  }
  if (warp == 1) {
    tmem_alloc<1>(&sh->tmem, 2 * BN);
    tmem_relinquish<1>();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem;
  if (warp == 0) {
    if (lane == 0) {
      int at = ahead, kb = ahead, i = 0;
      if (at < mine * nk) {
        for (; kb >= nk; kb -= nk) ++i;
        place(i, n0, m0, b);
      }
      for (; at < mine * nk && wait(&sh->empty[at % stages], (at / stages - 1) & 1); ++at, ++kb) {
        if (kb == nk) kb = 0, place(++i, n0, m0, b);
        load(kb, at);
      }
      for (int x = max(0, at - stages); x < at; ++x) drain(&sh->full[x % stages], (x / stages) & 1);   // nothing is on its way any more
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(kHgBM, BN);
      bool go = true;
      for (int i = 0, at = 0; go && i < mine; ++i) {
        if (i >= 2) go = wait(&sh->acc_empty[i & 1], ((i >> 1) - 1) & 1);   // the epilogue has read what this accumulator held
        if (!go) break;
        tc_fence_after();
        for (int kb = 0; kb < nk; ++kb, ++at) {
          go = wait(&sh->full[at % stages], (at / stages) & 1);
          if (!go) break;
          tc_fence_after();
          const uint32_t sa = smem_u32(ring + (at % stages) * kStage);
          const uint64_t da = make_sw128_kmajor_desc(sa), db = make_sw128_kmajor_desc(sa + kA);
#pragma unroll
          for (int k = 0; k < kHgBK / 16; ++k) umma_bf16<1>(tmem + (i & 1) * BN, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
          umma_commit(&sh->empty[at % stages]);
        }
        if (go) umma_commit(&sh->acc_full[i & 1]);
      }
      umma_commit(&sh->done);
      drain(&sh->done, 0);   // every product that was issued is done
    }
  } else {
    // thread = row while the accumulator is read, eight neighbouring threads = one row of 64 columns while gates come in and outputs go out
    // (lines of 32 rows per store otherwise)
    const int quarter = warp & 3, first = (warp - 2) / 4 * 64;
    constexpr int STEP = EP / 4 * 64;
    float* slab = reinterpret_cast<float*>(ring + stages * kStage + (warp - 2) * kHgSlab);
    const bool plain = vec_out && a.act == OMC_ACT_NONE && a.bias == nullptr && (a.gate == nullptr || vec_gate);
    bool go = true;
    for (int i = 0; go && i < mine; ++i) {
      place(i, n0, m0, b);
      const int left_rows = a.M - m0 - quarter * 32, r0 = lane >> 3;   // of this warp's 32; the first of the eight that a thread brings out
      const long long m = m0 + quarter * 32 + r0;
      // no branch between the loads and the stores of its 8 x 4 rows; a row's end lies between two threads' columns, or behind the piece
      auto whole = [&](int c) { return plain && left_rows > 0 && (n0 + c + 64 <= a.N || (a.N & 7) == 0); };
      uint4 gate[8][2];
      auto gates = [&](int c) {
        if (a.gate == nullptr || !whole(c)) return;
        const long long at = m * a.ldg + (long long)b * a.sg + min(n0 + c + (lane & 7) * 8, a.N - 8);
#pragma unroll
        for (int j = 0; j < 8; ++j) hg_gates_load(a, at + (long long)(min(r0 + j * 4, left_rows - 1) - r0) * a.ldg, gate[j]);
      };
      gates(first);
      go = wait_bounded_warp(&sh->acc_full[i & 1], (i >> 1) & 1, report);
      tc_fence_after();
      for (int c = first; go && c < BN && n0 + c < a.N; c += STEP) {
        if (c > first) gates(c);
        // bf16 without a gate is rounded on the way into the slab: half of its bytes
        const bool round_first = sizeof(TY) == 2 && a.gate == nullptr && whole(c);
#pragma unroll
        for (int part = 0; part < 2; ++part) {
          uint32_t v[32];
          tmem_ld32(tmem + (i & 1) * BN + ((uint32_t)(quarter * 32) << 16) + c + 32 * part, v);
          tmem_ld_wait();
          if (round_first) {
            uint4* dst = reinterpret_cast<uint4*>(slab + lane * kHgPitch16 + 16 * part);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint32_t o[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) o[e] = pack_bf16(__uint_as_float(v[8 * j + 2 * e]) * a.alpha, __uint_as_float(v[8 * j + 2 * e + 1]) * a.alpha);
              dst[j] = make_uint4(o[0], o[1], o[2], o[3]);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) *reinterpret_cast<uint4*>(slab + lane * kHgPitch + hg_chunk(8 * part + j)) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          }
        }
        if (c + STEP >= BN || n0 + c + STEP >= a.N) {   // that was the last of it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh->acc_empty[i & 1]);
        }
        __syncwarp();
        const int n = n0 + c + (lane & 7) * 8, left = min(8, a.N - n);
        const bf16_t* bias = a.bias != nullptr ? static_cast<const bf16_t*>(a.bias) + b * a.sbias : nullptr;
        if (whole(c)) {
          const int rows_here = left > 0 ? left_rows : 0;
          TY* y = static_cast<TY*>(a.Y) + (long long)b * a.sy + m * a.ldy + n;
          if (round_first) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const uint4 o = *reinterpret_cast<const uint4*>(slab + (r0 + j * 4) * kHgPitch16 + (lane & 7) * 4);
              if (r0 + j * 4 < rows_here) *reinterpret_cast<uint4*>(y + (long long)(j * 4) * a.ldy) = o;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              if (r0 + j * 4 >= rows_here) break;
              float f[8], z[8];
              hg_row(slab + (r0 + j * 4) * kHgPitch, lane & 7, a.alpha, f);
              if (a.gate != nullptr) {
                hg_gates(a, gate[j], z);
#pragma unroll
                for (int e = 0; e < 8; ++e) z[e] = 1.f + __expf(-z[e]);   // as at the edges: bits do not depend on the tile
                hg_divide(f, z);
              }
              hg_store(y + (long long)(j * 4) * a.ldy, f);
            }
          }
          __syncwarp();
          continue;
        }
#pragma unroll 2
        for (int j = 0; j < 8 && left > 0; ++j) {
          const int row = j * 4 + (lane >> 3), mr = m0 + quarter * 32 + row;
          if (mr >= a.M) break;
          float f[8];
          hg_row(slab + row * kHgPitch, lane & 7, a.alpha, f);
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = apply_act(f[e] + (bias != nullptr && e < left ? __bfloat162float(bias[n + e]) : 0.f), a.act);
          if (a.gate != nullptr) {
            const long long at = (long long)mr * a.ldg + (long long)b * a.sg + n;
            float z[8];
            if (vec_gate && left == 8) {
              uint4 g[2];
              hg_gates_load(a, at, g);
              hg_gates(a, g, z);
            } else {
#pragma unroll
              for (int e = 0; e < 8; ++e)
                z[e] = e >= left ? 0.f : (a.gate_dt == OMC_DT_F32 ? static_cast<const float*>(a.gate)[at + e] : ldf(static_cast<const bf16_t*>(a.gate) + at + e));
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] /= 1.f + (pair_gate && n + (e | 1) < a.N ? __expf(-z[e]) : expf(-z[e]));
          }
          TY* y = static_cast<TY*>(a.Y) + (long long)b * a.sy + (long long)mr * a.ldy + n;
          if (vec_out && left == 8) {
            hg_store(y, f);
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (e < left) stf(y + e, f[e]);
          }
        }
        __syncwarp();
      }
      if (go && (first >= BN || n0 + first >= a.N)) {   // a warp without columns in this tile
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->acc_empty[i & 1]);
      }
    }
    tc_fence_before();
  }
  __syncwarp();
  __syncthreads();
  if (warp == 1) tmem_dealloc<1>(tmem, 2 * BN);
}

template <int BN, typename TY>
static int hg_launch(const LinearArgs& a, int batch, cudaStream_t st) {
  CUtensorMap tx, tw;
  unsigned int* failed = nullptr;
  int rc = step_failure_word(&failed);
  if (rc == OMC_OK) rc = step_tensor_map(&tx, a.X, a.K, a.M, a.ldx, a.sx > 0 ? batch : 1, a.sx, kHgBM);   // stride 0: the batch shares the operand
  if (rc == OMC_OK) rc = step_tensor_map(&tw, a.W, a.K, a.N, a.ldw, a.sw > 0 ? batch : 1, a.sw, BN);
  if (rc != OMC_OK) return rc;
  constexpr int stage = (kHgBM + BN) * 128, smem = hg_stages(BN) * stage + hg_epilogue(BN) * kHgSlab + 1024;
  static_assert(smem + (int)sizeof(HgShared) <= 227 * 1024 && hg_stages(BN) <= kHgMaxStages, "");
  static bool done[kMaxDevices] = {};
  const int dev = cur_device();
  if (!done[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(linear_sm100_kernel<BN, TY>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return set_error(OMC_ERR_CUDA, cudaGetErrorString(e));
    done[dev] = true;
  }
  auto aligned = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  const int ye = 16 / (int)sizeof(TY), ge = a.gate_dt == OMC_DT_F32 ? 4 : 8;
  const bool vec_out = aligned(a.Y) && a.ldy % ye == 0 && a.sy % ye == 0, vec_gate = aligned(a.gate) && a.ldg % ge == 0 && a.sg % ge == 0;
  // the hardware exponential for gates that come in pairs on 8-byte boundaries, the precise one for those at odd strides and an odd last column
  const bool pair_gate = a.ldg % 2 == 0 && a.sg % 2 == 0 && reinterpret_cast<uintptr_t>(a.gate) % 8 == 0;
  HgTiles tiles{(a.N + BN - 1) / BN, (a.M + kHgBM - 1) / kHgBM, 0, 0, 0, 0};
  const long long total = (long long)tiles.n * tiles.m * batch;
  if (total > 0x7fffffffLL - 148) return set_error(OMC_ERR_SHAPE, "omc_linear: too many tiles");
  const int ctas = (int)(total < 148 ? total : 148);
  tiles.each = (int)(total / ctas), tiles.more = (int)(total % ctas);
  if (total < 1 << 16) tiles.by_n = (uint32_t)(((1ull << 32) + tiles.n - 1) / tiles.n), tiles.by_m = (uint32_t)(((1ull << 32) + tiles.m - 1) / tiles.m);
  linear_sm100_kernel<BN, TY><<<ctas, 64 + 32 * hg_epilogue(BN), smem, st>>>(tx, tw, a, tiles, a.sx == 0, a.sw == 0, vec_out, vec_gate, pair_gate, failed);
  return check_launch("omc_linear");
}

template <typename TY>
static int hg_launch_typed(const LinearArgs& a, int batch, cudaStream_t st) {
  // Tiles of 64, 128 and 256 columns take 4 : 5 : 8, and CTAs walk over them in waves of 148. 71 rows x 16, 128 -> 1024: 256 tiles of 64 10.3 us, 128 of 128 7.8, 64 of 256 10.4; 302 x 8,
  // 128 -> 1024: 384 14.1, 192 12.2, 96 10.5; 282 x 16, 256 -> 1024 with gates: 768 24.4, 384 18.6, 192 20.0
  const long long rows = (long long)((a.M + kHgBM - 1) / kHgBM) * batch;
  auto cost = [&](int bn, int each) { return (rows * ((a.N + bn - 1) / bn) + 147) / 148 * each; };
  const long long of64 = cost(64, 4), of128 = a.N > 64 ? cost(128, 5) : of64, of256 = a.N > 128 ? cost(256, 8) : of64;
  if (of256 < of64 && of256 < of128) return hg_launch<256, TY>(a, batch, st);
  if (of128 < of64) return hg_launch<128, TY>(a, batch, st);
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
