// Linear layer for any shape and for fp32 as well as bf16 storage: Y = act(alpha * X W^T), fp32 accumulation on the FMA pipe.
//
// This is the kernel a new decoder is brought up on, the true-fp32 path of the sequence-step models (no reduced-precision
// matrix mode anywhere), and the path for shapes the tcgen05 GEMM does not take (dimensions that are not multiples of 8, head
// slices of a few dozen columns). blockIdx.z walks a batch of independent problems that are column slices of the same buffers
// (attention heads); an optional tile -> group table turns it into the grouped product of expert-sorted rows.
//
// Two kernels share one order of sums, so that a row's result does not depend on the M of the call: K is cut into chunks of 64; in a
// chunk the even and the odd terms are summed separately in ascending order (one packed fma does both), their sum is the chunk's,
// and the chunks are added in ascending order.
#include "linear_args.cuh"

namespace omc {

constexpr int kLinBM = 64, kLinBN = 64, kLinBK = 32;   // BM: rows per tile, also of the grouped product's tile table
constexpr int kLinChunk = 64;                          // K terms per partial sum
constexpr int kLinPitch = kLinBK + 4, kLinStages = 3;

__device__ __forceinline__ float gate_out(float y, const LinearArgs& a, int m, int n) {
  if (a.gate == nullptr) return y;
  const long long at = (long long)m * a.ldg + (long long)blockIdx.z * a.sg + n;
  const float z = a.gate_dt == OMC_DT_F32 ? static_cast<const float*>(a.gate)[at] : ldf(static_cast<const bf16_t*>(a.gate) + at);
  return y / (1.f + expf(-z));
}

__device__ __forceinline__ uint32_t lin_smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

typedef unsigned long long f32x2_t;
__device__ __forceinline__ void fma2(f32x2_t& acc, f32x2_t x, f32x2_t w) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(w)); }
__device__ __forceinline__ float sum2(f32x2_t v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ void lds_pairs(const float* p, f32x2_t& lo, f32x2_t& hi) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  lo = v.x, hi = v.y;
}

// dst[0..3] (shared memory) <- row[k..k+3] as fp32, zero where !valid or past K. VEC: K and the row strides are multiples of four and the
// rows start on boundaries of four elements. fp32 goes by cp.async, which the caller commits: as one piece with VEC, as four without.
template <typename T, bool VEC>
__device__ __forceinline__ void stage4(float* dst, const T* row, int k, int K, bool valid) {
  if constexpr (VEC && sizeof(T) == 4) {
    const bool in = valid && k < K;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(lin_smem_u32(dst)), "l"(in ? row + k : row), "r"(in ? 16 : 0) : "memory");
  } else if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool in = valid && k + j < K;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(lin_smem_u32(dst + j)), "l"(in ? row + k + j : row), "r"(in ? 4 : 0) : "memory");
    }
  } else {
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (valid) {
      if (VEC) {
        if (k < K) ld4(row + k, v);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (k + j < K) v[j] = ldf(row + k + j);
      }
    }
    st4(dst, v);
  }
}

template <typename TW, typename TY>
__device__ __forceinline__ void finish_output(const LinearArgs& a, TY* Y, float sum, int m, int n) {
  const float b = a.bias != nullptr ? ldf(static_cast<const TW*>(a.bias) + blockIdx.z * a.sbias + n) : 0.f;
  stf(Y + (long long)m * a.ldy + n, gate_out(apply_act(sum * a.alpha + b, a.act), a, m, n));
}

// Many rows: 64 x 64 outputs per CTA of 128 threads, 4 x 8 each, K in slices of 32 that go through a ring of three buffers. A thread
// reads its rows and columns as 16-byte pieces along K (12 loads for 64 packed fma; a pitch of 36 floats puts eight neighbouring rows on
// different banks), so what bounds it is the shared-memory pipe behind the fma pipe and, with few tiles, the serial walk over K. Measured in
// fp32 (the kernel before it, 4 x 4 outputs of 256 threads with scalar loads and one buffer, in brackets): 4096 x 6144 x 2048 2463 us =
// 42 TFLOP/s (4036), 384 x 1024 x 1024 45 us (93).
template <typename TX, typename TW, typename TY, bool VEC, int NT>   // NT threads: 128 with 4 x 8 outputs each, 256 with 4 x 4
__global__ void __launch_bounds__(NT) linear_tile_kernel(LinearArgs a) {
  extern __shared__ __align__(16) float lin_sm[];   // [stages][64 rows of X | 64 rows of W][pitch]
  constexpr int kStage = (kLinBM + kLinBN) * kLinPitch;
  const int m0 = blockIdx.y * kLinBM, n0 = blockIdx.x * kLinBN;
  const TX* X = static_cast<const TX*>(a.X) + (long long)blockIdx.z * a.sx;
  const TW* W = static_cast<const TW*>(a.W) + (long long)blockIdx.z * a.sw;
  TY* Y = static_cast<TY*>(a.Y) + (long long)blockIdx.z * a.sy;
  if (a.tile_group != nullptr) {
    const int g = a.tile_group[blockIdx.y];
    if (g < 0) return;
    W += (long long)g * a.group_stride;
  }
  constexpr int NJ = kLinBM * kLinBN / 4 / NT, kTx = kLinBN / NJ, kRowsAtOnce = NT / 8;
  const int tid = threadIdx.x, tx = tid % kTx, ty = tid / kTx;   // ty < 16
  const int lk = (tid & 7) * 4, lr = tid >> 3;   // staging: 8 pieces of a row by 8 neighbouring threads
  auto stage = [&](int kt) {
    float* xs = lin_sm + (kt % kLinStages) * kStage;
    float* ws = xs + kLinBM * kLinPitch;
    const int k = kt * kLinBK + lk;
#pragma unroll
    for (int i = 0; i < kLinBM / kRowsAtOnce; ++i) {
      const int r = lr + i * kRowsAtOnce;
      stage4<TX, VEC>(xs + r * kLinPitch + lk, X + (long long)min(m0 + r, a.M - 1) * a.ldx, k, a.K, m0 + r < a.M);
    }
#pragma unroll
    for (int i = 0; i < kLinBN / kRowsAtOnce; ++i) {
      const int r = lr + i * kRowsAtOnce;
      stage4<TW, VEC>(ws + r * kLinPitch + lk, W + (long long)min(n0 + r, a.N - 1) * a.ldw, k, a.K, n0 + r < a.N);
    }
  };
  f32x2_t acc[4][NJ];
  float tot[4][NJ];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) acc[i][j] = 0ull, tot[i][j] = 0.f;
  const int nk = (a.K + kLinBK - 1) / kLinBK;
#pragma unroll
  for (int s = 0; s < kLinStages - 1; ++s) {
    if (s < nk) stage(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int kt = 0; kt < nk; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kLinStages - 2) : "memory");
    __syncthreads();   // slice kt is there for everyone, and everyone is done with the buffer that the next load overwrites
    if (kt + kLinStages - 1 < nk) stage(kt + kLinStages - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* xs = lin_sm + (kt % kLinStages) * kStage + ty * kLinPitch;
    const float* ws = lin_sm + (kt % kLinStages) * kStage + (kLinBM + tx) * kLinPitch;
#pragma unroll
    for (int k = 0; k < kLinBK; k += 4) {
      f32x2_t xl[4], xh[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) lds_pairs(xs + i * 16 * kLinPitch + k, xl[i], xh[i]);
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        f32x2_t wl, wh;
        lds_pairs(ws + j * kTx * kLinPitch + k, wl, wh);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          fma2(acc[i][j], xl[i], wl);
          fma2(acc[i][j], xh[i], wh);
        }
      }
    }
    if ((kt & 1) || kt + 1 == nk) {   // the end of a chunk
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) tot[i][j] += sum2(acc[i][j]), acc[i][j] = 0ull;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty + 16 * i;
    if (m >= a.M) continue;
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int n = n0 + tx + kTx * j;
      if (n < a.N) finish_output<TW, TY>(a, Y, tot[i][j], m, n);
    }
  }
}

// Few rows: what counts is how many bytes of W are on their way. A CTA owns 8 columns and up to MR rows and brings CHUNKS chunks of 64 terms at a time into
// shared memory, all of them in one go (16: 1024 terms and 64 threads; 32: 2048 and 128, for sums that long in few CTAs, see the launch); thread (p, c) sums chunk c of the
// columns p and p + 4 for every row, and the chunks' sums are added by one thread per output, in one order whatever CHUNKS. A pitch of 68 floats per chunk puts the chunks on different
// banks. 3 x 6144 x 2048 in fp32: 19 us = 2.6 TB/s of W (the tile kernel before: 145), 3 x 4096 x 1024 10 (76).
constexpr int kRowsCols = 8;

template <typename TX, typename TW, typename TY, int MR, bool VEC, int CHUNKS>
__global__ void __launch_bounds__(4 * CHUNKS) linear_rows_kernel(LinearArgs a) {
  constexpr int kRowsChunks = CHUNKS, kRowsPitch = CHUNKS * (kLinChunk + 4), kRowsThreads = 4 * CHUNKS;
  extern __shared__ __align__(16) float lin_sm[];   // W [8][pitch] | X [MR][pitch] | chunk sums [8][MR][CHUNKS + 1]
  float* ws = lin_sm;
  float* xs = ws + kRowsCols * kRowsPitch;
  float* part = xs + MR * kRowsPitch;
  const int m0 = blockIdx.y * MR, n0 = blockIdx.x * kRowsCols;
  const TX* X = static_cast<const TX*>(a.X) + (long long)blockIdx.z * a.sx;
  const TW* W = static_cast<const TW*>(a.W) + (long long)blockIdx.z * a.sw;
  TY* Y = static_cast<TY*>(a.Y) + (long long)blockIdx.z * a.sy;
  const int tid = threadIdx.x, c = tid % kRowsChunks, p = tid / kRowsChunks;
  const int out_n = tid & (kRowsCols - 1), out_m = tid / kRowsCols;   // the output whose chunks this thread adds
  float total = 0.f;
  for (int k0 = 0; k0 < a.K; k0 += kRowsChunks * kLinChunk) {
    const int chunks = min(kRowsChunks, (a.K - k0 + kLinChunk - 1) / kLinChunk);
    if (k0 > 0) __syncthreads();
    for (int e = tid; e < chunks * (kLinChunk / 4); e += kRowsThreads) {   // piece e of every row
      const int k = e * 4, at = k + (k >> 6) * 4;
#pragma unroll
      for (int r = 0; r < kRowsCols; ++r)
        stage4<TW, VEC>(ws + r * kRowsPitch + at, W + (long long)min(n0 + r, a.N - 1) * a.ldw, k0 + k, a.K, n0 + r < a.N);
#pragma unroll
      for (int r = 0; r < MR; ++r)
        stage4<TX, VEC>(xs + r * kRowsPitch + at, X + (long long)min(m0 + r, a.M - 1) * a.ldx, k0 + k, a.K, m0 + r < a.M);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (c < chunks) {
      f32x2_t acc[2][MR];
#pragma unroll
      for (int r = 0; r < MR; ++r) acc[0][r] = acc[1][r] = 0ull;
      const float* w0 = ws + p * kRowsPitch + c * (kLinChunk + 4);
      const float* x0 = xs + c * (kLinChunk + 4);
#pragma unroll 4
      for (int k = 0; k < kLinChunk; k += 4) {
        f32x2_t al, ah, bl, bh;
        lds_pairs(w0 + k, al, ah);
        lds_pairs(w0 + 4 * kRowsPitch + k, bl, bh);
#pragma unroll
        for (int r = 0; r < MR; ++r) {
          f32x2_t xl, xh;
          lds_pairs(x0 + r * kRowsPitch + k, xl, xh);
          fma2(acc[0][r], xl, al);
          fma2(acc[0][r], xh, ah);
          fma2(acc[1][r], xl, bl);
          fma2(acc[1][r], xh, bh);
        }
      }
#pragma unroll
      for (int r = 0; r < MR; ++r) {
        part[(p * MR + r) * (kRowsChunks + 1) + c] = sum2(acc[0][r]);
        part[((p + 4) * MR + r) * (kRowsChunks + 1) + c] = sum2(acc[1][r]);
      }
    }
    __syncthreads();
    if (out_m < MR) {
      const float* s = part + (out_n * MR + out_m) * (kRowsChunks + 1);
      for (int i = 0; i < chunks; ++i) total += s[i];
    }
  }
  if (out_m < MR && m0 + out_m < a.M && n0 + out_n < a.N) finish_output<TW, TY>(a, Y, total, m0 + out_m, n0 + out_n);
}

// ---- a few outputs per row (routers, gates, low-rank factors): the tile kernels would leave such a product to a handful of CTAs
// that each walk all of K. Here a CTA takes 8 rows and walks K in chunks of 1024 that it holds in shared memory as fp32; a warp owns
// up to 8 output columns (n = blockIdx.y * 8 + warp, then in strides of 8 * gridDim.y) with 8 accumulators each: it reads a chunk of
// that row of W once for all 8 rows. A lane takes four consecutive k at a time (one 8- or 16-byte load of W, float4 reads of the
// rows), the warp strides the chunk by 128, and a shuffle tree finishes the sums - the order of a sum depends on K alone, with or
// without the vector loads and however the columns are spread over CTAs (all columns in one CTA for long steps, eight per CTA for
// steps of a few rows, where there are few row blocks to fill the device with).
constexpr int kNarrowRows = 8, kNarrowMaxN = 64, kNarrowKC = 1024, kNarrowPerWarp = kNarrowMaxN / 8;

template <typename TX, typename TW, typename TY, bool VEC>
__global__ void __launch_bounds__(256, 2) linear_narrow_kernel(LinearArgs a) {
  __shared__ __align__(16) float nxs[kNarrowRows][kNarrowKC];
  const int m0 = blockIdx.x * kNarrowRows, nr = min(kNarrowRows, a.M - m0);
  const TX* X = static_cast<const TX*>(a.X) + (long long)blockIdx.z * a.sx;
  const TW* W = static_cast<const TW*>(a.W) + (long long)blockIdx.z * a.sw;
  TY* Y = static_cast<TY*>(a.Y) + (long long)blockIdx.z * a.sy;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.y * 8 + warp, stride = 8 * gridDim.y;
  float acc[kNarrowPerWarp][kNarrowRows];
#pragma unroll
  for (int i = 0; i < kNarrowPerWarp; ++i)
#pragma unroll
    for (int r = 0; r < kNarrowRows; ++r) acc[i][r] = 0.f;
  for (int kc = 0; kc < a.K; kc += kNarrowKC) {
    const int kn = min(kNarrowKC, a.K - kc), knp = (kn + 3) & ~3;   // the chunk's columns, rounded up to 4 with a zero tail
    if (kc > 0) __syncthreads();
    if (VEC) {
      const int k4n = knp >> 2;
      for (int e = threadIdx.x; e < kNarrowRows * k4n; e += blockDim.x) {
        const int r = e / k4n, k = (e - r * k4n) << 2;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (r < nr) ld4(X + (long long)(m0 + r) * a.ldx + kc + k, v);
        *reinterpret_cast<float4*>(&nxs[r][k]) = make_float4(v[0], v[1], v[2], v[3]);
      }
    } else {
      for (int e = threadIdx.x; e < kNarrowRows * knp; e += blockDim.x) {
        const int r = e / knp, k = e - r * knp;
        nxs[r][k] = (r < nr && k < kn) ? ldf(X + (long long)(m0 + r) * a.ldx + kc + k) : 0.f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kNarrowPerWarp; ++i) {
      const int n = n0 + i * stride;
      if (n < a.N) {
        const TW* wr = W + (long long)n * a.ldw + kc;
#pragma unroll 2
        for (int k = lane * 4; k < knp; k += 128) {
          float wv[4];
          if (VEC) {
            ld4(wr + k, wv);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) wv[j] = k + j < kn ? ldf(wr + k + j) : 0.f;
          }
#pragma unroll
          for (int r = 0; r < kNarrowRows; ++r) {
            const float4 xv = *reinterpret_cast<const float4*>(&nxs[r][k]);
            acc[i][r] = fmaf(xv.x, wv[0], acc[i][r]);
            acc[i][r] = fmaf(xv.y, wv[1], acc[i][r]);
            acc[i][r] = fmaf(xv.z, wv[2], acc[i][r]);
            acc[i][r] = fmaf(xv.w, wv[3], acc[i][r]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kNarrowPerWarp; ++i) {
    const int n = n0 + i * stride;
    if (n >= a.N) break;
    float mine = 0.f;
#pragma unroll
    for (int r = 0; r < kNarrowRows; ++r) {
      const float v = seq_warp_sum(acc[i][r]);
      if (lane == r) mine = v;
    }
    if (lane < nr) {
      const float b = a.bias != nullptr ? ldf(static_cast<const TW*>(a.bias) + blockIdx.z * a.sbias + n) : 0.f;
      stf(Y + (long long)(m0 + lane) * a.ldy + n, gate_out(apply_act(mine * a.alpha + b, a.act), a, m0 + lane, n));
    }
  }
}

// bf16 operands that the tensor-core kernel (linear_sm100.cu) can fetch: rows and batch items that start on 16-byte boundaries and do not
// overlap (its tensor maps know no stride of zero; a batch may share an operand).
int linear_sm100(const LinearArgs& a, int y_dt, int batch, cudaStream_t st);
static bool sm100_operands_ok(const LinearArgs& a) {
  return a.tile_group == nullptr && a.K % 8 == 0 && a.ldx % 8 == 0 && a.ldw % 8 == 0 && a.sx % 8 == 0 && a.sw % 8 == 0 && a.ldx >= a.K && a.ldw >= a.K &&
         a.sx >= 0 && a.sw >= 0 && reinterpret_cast<uintptr_t>(a.X) % 16 == 0 && reinterpret_cast<uintptr_t>(a.W) % 16 == 0;
}

template <typename TX, typename TW, typename TY>
static int launch_narrow_typed(const LinearArgs& a, int batch, cudaStream_t st) {
  // vector loads: rows of X and W that start on 8-byte (bf16) / 16-byte (fp32) boundaries and a K that is a multiple of four
  const bool vec = a.K % 4 == 0 && a.ldx % 4 == 0 && a.ldw % 4 == 0 && a.sx % 4 == 0 && a.sw % 4 == 0 &&
                   reinterpret_cast<uintptr_t>(a.X) % (4 * sizeof(TX)) == 0 && reinterpret_cast<uintptr_t>(a.W) % (4 * sizeof(TW)) == 0;
  // where the columns run is a matter of occupancy only: every column is summed by one warp in the same order either way
  const dim3 grid((a.M + kNarrowRows - 1) / kNarrowRows, a.M <= 64 ? (a.N + 7) / 8 : 1, batch);
  if (vec) linear_narrow_kernel<TX, TW, TY, true><<<grid, 256, 0, st>>>(a);
  else linear_narrow_kernel<TX, TW, TY, false><<<grid, 256, 0, st>>>(a);
  return check_launch("omc_linear");
}

template <typename TX, typename TW>
static int launch_narrow(const LinearArgs& a, int y_dt, int batch, cudaStream_t st) {
  if (y_dt == OMC_DT_F32) return launch_narrow_typed<TX, TW, float>(a, batch, st);
  if (y_dt == OMC_DT_BF16) return launch_narrow_typed<TX, TW, bf16_t>(a, batch, st);
  return set_error(OMC_ERR_ARG, "omc_linear: unknown output dtype");
}

// Rows kernel or tile kernel: the same results either way. Both were measured at K from 16 to 2048 (in us, rows / tile):
//   K =   64: 16 x 2048 outputs 5.9 / 4.6, 64 x 512 5.3 / 6.6, 100 x 2048 20.6 / 7.5, 32 x 4096 13.5 / 5.5
//   K =  256: 32 x 1024 7 / 14, 100 x 1024 14.5 / 14.1, 100 x 2048 26 / 14, 200 x 1024 25 / 14
//   K = 1024: 8 x 4096 13 / 37, 32 x 4096 28 / 40, 64 x 4096 48 / 44, 128 x 1024 29 / 44, 256 x 1024 49 / 45
// The tile kernel's time goes with K alone up to a first wave of 148 tiles, however few and empty they are, and in proportion above that. The rows
// kernel's goes with the outputs, and falls only slowly with K below its stage of 1024 terms (K / 64 of a CTA's 16 sums are at work, and its shared
// memory is the same): they meet at some 20,000 outputs plus 195 per K term and wave, whether the vector loads take the rows or not, and sooner where
// bf16 is converted on its way (K = 1001: 196,000 outputs in fp32, 150,000 with bf16 weights, 110,000 with bf16 rows too).
static long long lin_tiles(const LinearArgs& a, int batch) {
  return (long long)((a.N + kLinBN - 1) / kLinBN) * ((a.M + kLinBM - 1) / kLinBM) * batch;
}
static bool few_rows(const LinearArgs& a, int batch, int bf16_operands) {
  const long long tiles = lin_tiles(a, batch), outputs = (long long)a.M * a.N * batch;
  const long long meet = (20000 + 195LL * (a.K < 1024 ? a.K : 1024)) * (4 - bf16_operands) / 4;
  return a.tile_group == nullptr && 148 * outputs <= meet * (tiles > 148 ? tiles : 148) && a.M <= 8 * 65535;
}

// Dynamic shared memory above 48 KB is asked for once per kernel and device.
template <typename Kernel>
static int allow_smem(Kernel* kernel, int smem, bool (&done)[kMaxDevices]) {
  const int dev = cur_device();
  if (done[dev]) return OMC_OK;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return set_error(OMC_ERR_CUDA, cudaGetErrorString(e));
  done[dev] = true;
  return OMC_OK;
}

template <typename TX, typename TW, typename TY, int MR, bool VEC, int CHUNKS>
static int launch_rows(const LinearArgs& a, const dim3& grid, cudaStream_t st) {
  constexpr int smem = ((kRowsCols + MR) * CHUNKS * (kLinChunk + 4) + kRowsCols * MR * (CHUNKS + 1)) * 4;
  static bool done[kMaxDevices] = {};
  if (int rc = allow_smem(linear_rows_kernel<TX, TW, TY, MR, VEC, CHUNKS>, smem, done); rc != OMC_OK) return rc;
  linear_rows_kernel<TX, TW, TY, MR, VEC, CHUNKS><<<grid, 4 * CHUNKS, smem, st>>>(a);
  return check_launch("omc_linear");
}
// Sums of more than 1024 terms whose CTAs run in one wave have all of their terms under way at once: 3 x 1024 x 2048 8.5 -> 6.4 us, 8 x 1024 x 2048 10.5 -> 8.4, 100 x 77 x 4096
// 15.1 -> 11.5. With more CTAs than that the smaller ones, of which four share an SM, are as fast (3 x 4096 x 2048 14.2).
template <typename TX, typename TW, typename TY, int MR, bool VEC>
static int launch_rows(const LinearArgs& a, int batch, cudaStream_t st) {
  const dim3 grid((a.N + kRowsCols - 1) / kRowsCols, (a.M + MR - 1) / MR, batch);
  if (a.K > 1024 && (long long)grid.x * grid.y * batch <= (MR == 4 ? 296 : 148)) return launch_rows<TX, TW, TY, MR, VEC, 32>(a, grid, st);
  return launch_rows<TX, TW, TY, MR, VEC, 16>(a, grid, st);
}

template <typename TX, typename TW, typename TY, bool VEC, int NT>
static int launch_tile(const LinearArgs& a, int batch, cudaStream_t st) {
  constexpr int smem = kLinStages * (kLinBM + kLinBN) * kLinPitch * 4;
  static bool done[kMaxDevices] = {};
  if (int rc = allow_smem(linear_tile_kernel<TX, TW, TY, VEC, NT>, smem, done); rc != OMC_OK) return rc;
  const dim3 grid((a.N + kLinBN - 1) / kLinBN, (a.M + kLinBM - 1) / kLinBM, batch);
  linear_tile_kernel<TX, TW, TY, VEC, NT><<<grid, NT, smem, st>>>(a);
  return check_launch("omc_linear");
}

template <typename TX, typename TW, typename TY, bool VEC>
static int launch_any(const LinearArgs& a, int batch, cudaStream_t st) {
  constexpr int bf16_operands = (sizeof(TX) == 2) + (sizeof(TW) == 2);
  if (few_rows(a, batch, bf16_operands)) return a.M <= 4 ? launch_rows<TX, TW, TY, 4, VEC>(a, batch, st) : launch_rows<TX, TW, TY, 8, VEC>(a, batch, st);
  // the better reuse of 128 threads counts where a long sum over many tiles of fp32 leaves nothing else to wait for (in us, 128 / 256 threads: 4096 x
  // 6144 x 2048 2463 / 2646, 4096 x 2048 x 1024 432 / 454); the smaller tasks of 256 hide more elsewhere (the same at K = 256 142 / 127, at 64
  // 76 / 52, with bf16 weights at 257 244 / 189; 700 x 2000 x 256 43 / 32; 100 x 77 x 4096 17 / 13)
  if constexpr (bf16_operands == 0)
    if (a.K >= 768 && lin_tiles(a, batch) >= 296) return launch_tile<TX, TW, TY, VEC, 128>(a, batch, st);
  return launch_tile<TX, TW, TY, VEC, 256>(a, batch, st);
}

template <typename TX, typename TW, typename TY>
static int launch_linear_typed(const LinearArgs& a, int batch, cudaStream_t st) {
  // 16-byte (fp32) / 8-byte (bf16) pieces of rows that start on such boundaries and are a multiple of four long
  const bool vec = a.K % 4 == 0 && a.ldx % 4 == 0 && a.ldw % 4 == 0 && a.sx % 4 == 0 && a.sw % 4 == 0 && a.group_stride % 4 == 0 &&
                   reinterpret_cast<uintptr_t>(a.X) % (4 * sizeof(TX)) == 0 && reinterpret_cast<uintptr_t>(a.W) % (4 * sizeof(TW)) == 0;
  return vec ? launch_any<TX, TW, TY, true>(a, batch, st) : launch_any<TX, TW, TY, false>(a, batch, st);
}

template <typename TX, typename TW>
static int launch_linear(const LinearArgs& a, int y_dt, int batch, cudaStream_t st) {
  // few outputs over a long K: the choice depends on widths only, never on M
  if (a.tile_group == nullptr && a.N <= kNarrowMaxN && a.K >= 4 * a.N) return launch_narrow<TX, TW>(a, y_dt, batch, st);
  if (y_dt == OMC_DT_F32) return launch_linear_typed<TX, TW, float>(a, batch, st);
  if (y_dt == OMC_DT_BF16) return launch_linear_typed<TX, TW, bf16_t>(a, batch, st);
  return set_error(OMC_ERR_ARG, "omc_linear: unknown output dtype");
}

}  // namespace omc

static int run_linear(const void* X, int x_dt, long long ldx, long long sx, const void* W, int w_dt, long long ldw, long long sw, void* Y, int y_dt,
                      long long ldy, long long sy, int M, int N, int K, int batch, float alpha, int act, const int32_t* tile_group,
                      long long group_stride, const void* bias, long long sbias, const void* gate, int gate_dt, long long ldg, long long sg,
                      void* stream) {
  using namespace omc;
  if (X == nullptr || W == nullptr || Y == nullptr || N <= 0 || K <= 0 || M < 0 || batch <= 0)
    return set_error(OMC_ERR_ARG, "omc_linear: bad argument");
  if (M == 0) return OMC_OK;
  if (tile_group != nullptr && batch != 1) return set_error(OMC_ERR_ARG, "omc_linear: a tile table excludes a batch");
  if ((long long)((M + kLinBM - 1) / kLinBM) > 65535 || batch > 65535)
    return set_error(OMC_ERR_SHAPE, "omc_linear: more than 65535 row tiles or batch items");
  if (bias != nullptr && tile_group != nullptr) return set_error(OMC_ERR_ARG, "omc_linear: a bias excludes a tile table");
  LinearArgs a{X, W, Y, ldx, sx, ldw, sw, ldy, sy, group_stride, tile_group, M, N, K, alpha, act, bias, sbias, gate, gate_dt, ldg, sg};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (x_dt == OMC_DT_F32 && w_dt == OMC_DT_F32) return launch_linear<float, float>(a, y_dt, batch, st);
  if (x_dt == OMC_DT_F32 && w_dt == OMC_DT_BF16) return launch_linear<float, bf16_t>(a, y_dt, batch, st);
  if (x_dt == OMC_DT_BF16 && w_dt == OMC_DT_BF16) {
    // the choice depends on layout and widths only, never on M: a row is computed by the same kernel in every batch
    const bool narrow = tile_group == nullptr && N <= kNarrowMaxN && K >= 4 * N;
    if (!narrow && sm100_operands_ok(a) && (long long)N * K >= 4096) return linear_sm100(a, y_dt, batch, st);
    return launch_linear<bf16_t, bf16_t>(a, y_dt, batch, st);
  }
  return set_error(OMC_ERR_ARG, "omc_linear: operand dtypes must be (f32, f32), (f32, bf16) or (bf16, bf16)");
}

extern "C" int omc_linear_bias(const void* X, int x_dt, long long ldx, long long sx, const void* W, int w_dt, long long ldw,
                               long long sw, void* Y, int y_dt, long long ldy, long long sy, int M, int N, int K, int batch,
                               float alpha, int act, const int32_t* tile_group, long long group_stride, const void* bias,
                               long long sbias, void* stream) {
  return run_linear(X, x_dt, ldx, sx, W, w_dt, ldw, sw, Y, y_dt, ldy, sy, M, N, K, batch, alpha, act, tile_group, group_stride, bias, sbias, nullptr,
                    OMC_DT_F32, 0, 0, stream);
}

extern "C" int omc_linear_gate(const void* X, int x_dt, long long ldx, long long sx, const void* W, int w_dt, long long ldw, long long sw, void* Y,
                               int y_dt, long long ldy, long long sy, int M, int N, int K, int batch, float alpha, int act, const void* gate,
                               int gate_dt, long long ldg, long long sg, void* stream) {
  if (gate == nullptr || (gate_dt != OMC_DT_F32 && gate_dt != OMC_DT_BF16)) return omc::set_error(OMC_ERR_ARG, "omc_linear_gate: bad gate");
  return run_linear(X, x_dt, ldx, sx, W, w_dt, ldw, sw, Y, y_dt, ldy, sy, M, N, K, batch, alpha, act, nullptr, 0, nullptr, 0, gate, gate_dt, ldg, sg,
                    stream);
}

extern "C" int omc_linear(const void* X, int x_dt, long long ldx, long long sx, const void* W, int w_dt, long long ldw,
                          long long sw, void* Y, int y_dt, long long ldy, long long sy, int M, int N, int K, int batch,
                          float alpha, int act, const int32_t* tile_group, long long group_stride, void* stream) {
  return run_linear(X, x_dt, ldx, sx, W, w_dt, ldw, sw, Y, y_dt, ldy, sy, M, N, K, batch, alpha, act, tile_group, group_stride, nullptr, 0, nullptr,
                    OMC_DT_F32, 0, 0, stream);
}
