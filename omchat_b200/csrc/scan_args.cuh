// What the kernels of the linear-state recurrence share (state_mixers.cu describes it): their arguments, activations, asynchronous copies.
#pragma once
#include "fp32_pairs.cuh"
#include "seq_common.cuh"

namespace omc {

__device__ __forceinline__ float sigmoid_f(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }
// The same bits for four numbers at once: a division serves every exponent, in some ten instructions with a branch each, which these functions' callers wait for. Where a number
// is further from zero than 44 (or infinite) all four are divided.
template <bool SILU>
__device__ __forceinline__ void sigmoid4(float (&z)[4]) {
  float y[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) y[e] = 1.f + expf(-z[e]);
  if (fmaxf(fmaxf(fabsf(z[0]), fabsf(z[1])), fmaxf(fabsf(z[2]), fabsf(z[3]))) <= 44.f) {
#pragma unroll
    for (int e = 0; e < 4; e += 2) quotients2(SILU ? -z[e] : -1.f, SILU ? -z[e + 1] : -1.f, y[e], y[e + 1], z[e], z[e + 1]);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) z[e] = (SILU ? z[e] : 1.f) / y[e];
  }
}
__device__ __forceinline__ float softplus_f(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }

struct ScanArgs {
  const float* q;      // [T, ldq]: head g of kv_heads at columns g * dim
  const float* k;
  const float* v;      // [T, ldv]: head h at columns h * vdim
  long long ldq, ldk, ldv;
  int silu_in;         // q, k, v pass silu on the way in
  int decay_mode;      // 0: decay_const[h]; 1: a[t, h]; 2: a[t, h * dim + i]  (1, 2: g = exp(-exp(A_log[h]) softplus(a + dt_bias))); 3: g = a[t, h * dim + i];
                       // 4: g = sigmoid(a[t, h * dim + i] + dt_bias[h * dim + i])^decay_pow; 5: a[t, h * dim + i] holds g - 1
                       // (4 and 5 apply the decay as S + (g - 1) S); 6: dt = softplus(a[t, h] + dt_bias[h]), g = exp(-exp(A_log[h]) dt),
                       // u = dt v, o = S^T q + D[h] v (the decay as S + expm1(.) S)
  float decay_pow;     // mode 4
  float out_scale;     // o_t = out_scale * S^T q_t (a query scale, applied to the read-out)
  const float* decay_const;
  const float* a;
  long long lda;
  const float* A_log;    // fp32 [H]
  const float* dt_bias;  // fp32 [H] (modes 1, 6) or [H * dim] (mode 2)
  const float* D;        // fp32 [H] (mode 6) or NULL
  const float* beta;     // raw [T, ldb]: beta = sigmoid; NULL: no delta correction (u = v)
  long long ldb;
  float* state;          // [slots][H][dim][vdim]
  float* out;            // [T, ldo]
  long long ldo;
  const int32_t* row_begin;  // [P + 1] first row of every portion
  const int32_t* pos;
  const int32_t* slot;
  int H, G, dim, vdim;
  bool vec_state, vec_out;   // a thread's columns of the state / four outputs as one access
  int portions;              // P, where the CTAs take portions in the order of their lengths, the longest first; 0: in their own order
  int long_from;             // portions of this many rows and more are scan_chunk_kernel's, the others the token-by-token kernels' (0: all of them are theirs)
  int rows, all;             // the host's number of rows, by which scan_chunk_kernel has been launched; of portions
  int beside;                // 1, 2: the first and the second of the two kernels that share the portions of a step; 0: alone
};

// Whether a portion of n rows is scan_chunk_kernel's, for which the host has launched CTAs for rows / long_from portions: if row_begin has more rows than the host was told of,
// there may be more long portions than that, and the token-by-token kernels take them all.
__device__ __forceinline__ bool scan_is_long(const ScanArgs& a, int n) { return a.long_from > 0 && n >= a.long_from && a.row_begin[a.all] - a.row_begin[0] <= a.rows; }

// The two kernels of a step write different portions and slots, so the second may run beside the first: the first lets it start as soon as all of its own CTAs have, and the
// second ends behind the first, whose end nothing else would wait for: what comes next on the stream waits for the second alone. A CTA that does nothing else waits, in a layer of
// the grid behind the portions'; at the end of a CTA that has a portion the wait cost the token loops 5 % (64 channels, delta rule: 63 tokens 13.2 -> 13.9 us).
__device__ __forceinline__ void scan_begin(const ScanArgs& a) {
  if (a.beside == 1) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ bool scan_only_waits(const ScanArgs& a) {
  if (a.beside != 2 || (int)blockIdx.z < a.all) return false;
  if ((blockIdx.x | blockIdx.y) == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
  return true;
}
template <typename... Params, typename... Args>
int scan_launch(void (*kernel)(Params...), dim3 grid, int threads, int smem, cudaStream_t st, const ScanArgs& a, Args... args) {
  cudaLaunchConfig_t cfg{};
  if (a.beside == 2) ++grid.z;   // the layer that waits
  cfg.gridDim = grid, cfg.blockDim = dim3(threads), cfg.dynamicSmemBytes = smem, cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr, cfg.numAttrs = a.beside == 2 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, a, args...);
  return check_launch("omc_linear_state_scan");
}

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src));
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src));
}

// The portion whose length has the block's rank z, longest first (of up to as many portions as the block has threads): a long chain that starts last would run alone at the end.
// scratch: shared memory of that many words, free again behind it.
__device__ __forceinline__ int scan_portion(const int32_t* row_begin, int portions, int z, int* scratch) {
  const int p = threadIdx.x;
  if (p < portions) scratch[p] = row_begin[p + 1] - row_begin[p];
  __syncthreads();
  bool mine = false;
  if (p < portions) {
    const int n = scratch[p];
    int before = 0;
    for (int o = 0; o < portions; ++o) before += scratch[o] > n || (scratch[o] == n && o < p);
    mine = before == z;
  }
  __syncthreads();
  if (mine) scratch[0] = p;
  __syncthreads();
  const int found = scratch[0];
  __syncthreads();
  return found;
}

enum { kScanPlain = 0, kScanDelta = 1, kScanStep = 2 };
// Rows from which a portion goes eight tokens at a time: with decays per channel, and per head with the delta rule. A stage's overhead is gained back behind 15 to 35 tokens (per
// head 28 at 128 channels, 59 at 64). Where a step's portions lie on both sides of the line and CTAs are many its two kernels run one behind the other, so the line is low where it can
// be: 16 heads of 128 x 128 channels, portions of 64, 64 and 4 x 40 rows 1.56 of token by token with the line at 64 rows, 0.96 at 32; 32 heads, 64, 43, 30 rows 1.68 and 1.32, 8 x
// 40 rows 1.04 and 1.08. Per head 16 x 48 rows of 16 heads would take 1.16 of it with the line at 48; 64 and 63 rows take 1.42 with it at 64 (20 us).
constexpr int kScanLongChannel = 32, kScanLongHead = 64;
// The launch of scan_chunk.cu for the portions of at least a.long_from rows: the delta rule or per-channel decays (decay modes 1 with beta, 3, 5), 64 or 128 key
// channels, inputs that need no preparation of their own, 16-byte rows of k, q, v, decays, outputs and states. Returns check_launch's code.
int launch_scan_chunk(const ScanArgs& a, int rows, int portions, cudaStream_t st);

}  // namespace omc
