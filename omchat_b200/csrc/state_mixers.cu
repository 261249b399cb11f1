// Mixers that carry a fixed-size state per sequence instead of a growing cache: a short causal convolution per channel whose
// last inputs are state, and the family of linear-state recurrences
//     S <- diag(g_t) S;   u_t = beta_t (v_t - S^T k_t)  (delta rule)  or  u_t = v_t  (plain outer-product sum)
//                         or  u_t = dt_t v_t with g_t = exp(-A dt_t)  (state-space form: one step size per token and head);
//     S <- S + k_t u_t^T;   o_t = S^T q_t  (state-space form: + D v_t)
// with the decay g_t constant per head, one per token and head, or one per token, head and key channel, and the gated RMS norm
// that follows them. Rows of a step are addressed by (slot, position); the rows of one request are consecutive and ascending.
// A portion that starts at position 0 starts from a zero state, so a slot needs no clearing when it is handed to a new request.
// Everything here is fp32: state, decays and their logarithms, softplus / exponentials, step sizes, unit norms.
//
// The recurrence is evaluated token by token - prompt portions and single decoded tokens run the same instructions
// in the same order - except in portions of 64 rows and more of the delta rule, of 32 and more with a decay per key channel, which scan_chunk.cu takes eight tokens at a time: the
// same sums in another order. The result does not depend on how a prompt is cut but in these last bits. Its parallelism is over the
// independent COLUMNS of S: column j of a head's state only ever meets v[:, j], so a CTA owns 16, 32 or 64 columns of one head of one
// portion; a thread holds an eighth of the state elements of one, two or four neighbouring columns as packed fp32 pairs of key channels (a key or query value read from shared
// memory is used for each of its columns), and the eight lanes of a column finish the
// two dot products of a token with three shuffles each. Tokens are staged 8 or 16 at a time in shared memory by cp.async, one stage ahead of the one being
// computed (decays, sigmoid and silu applied on arrival), so the sequential loop touches registers and shared memory only.
// Recurrences whose channels carry one or a few states of their own (selective scan, gated linear recurrent unit) follow below.
#include <type_traits>

#include "scan_args.cuh"

namespace omc {

// sigmoid(z)^p - 1 = expm1(p * log sigmoid(z)), log sigmoid(z) = -softplus(-z). The decay is kept as its distance from 1: rounded to
// fp32 itself, a decay close to 1 loses most of the digits of 1 - decay, and the state multiplies by it once per token.
__device__ __forceinline__ float sigmoid_pow_m1_f(float z, float p) { return expm1f(-p * softplus_f(-z)); }

// ---- causal convolution (+ silu) (+ unit vectors) ---------------------------------------------------------------------------
// One CTA per (1 or 8 consecutive rows, block of channels; blocks are whole unit-vector groups). Tap j of `taps` multiplies the input
// `taps - 1 - j` positions back: an earlier row of the same step when that row belongs to the same request, else the state ring
// state[slot][position % (taps - 1)][channel], else (before position 0) zero. save_here: every row of the step is a request of
// its own, so the row's input goes into its ring from this kernel, after the reads (no other CTA reads that ring).
constexpr int kConvRows = 8;    // rows per CTA of a long step: neighbouring rows read each other's inputs, which then come from L1
constexpr int kConvMaxTaps = 32;

template <typename TW, typename TY>
__global__ void __launch_bounds__(256) causal_conv_silu_kernel(const float* __restrict__ x, long long ldx, int T, int ch, int ch_block,
                                                               int rows_per_cta, const TW* __restrict__ w, const TW* __restrict__ bias, int taps,
                                                               const int32_t* __restrict__ pos, const int32_t* __restrict__ slot,
                                                               float* __restrict__ state, TY* __restrict__ y, long long ldy,
                                                               int unit_channels, int unit_group, float unit_eps, int scaled_channels,
                                                               float unit_mult, int save_here, int act) {
  extern __shared__ float tile[];  // [rows_per_cta][ch_block]
  __shared__ const float* src[kConvRows][kConvMaxTaps];   // where tap j of row r reads: a row of x, a ring entry, or nothing
  const int t0 = blockIdx.x * rows_per_cta, nr = min(rows_per_cta, T - t0);
  const int c0 = blockIdx.y * ch_block, nc = min(ch_block, ch - c0);
  const int R = taps - 1;
  if (threadIdx.x < nr * taps) {
    const int r = threadIdx.x / taps, j = threadIdx.x - r * taps;
    const int t = t0 + r, p = pos[t], s = slot[t], back = R - j, sp = p - back;
    const float* q = nullptr;
    if (sp >= 0) q = (back == 0 || (t - back >= 0 && slot[t - back] == s)) ? x + (long long)(t - back) * ldx : state + ((long long)s * R + sp % R) * ch;
    src[r][j] = q;
  }
  __syncthreads();
  for (int cl = threadIdx.x; cl < nc; cl += blockDim.x) {
    const int c = c0 + cl;
    const float b0 = bias != nullptr ? ldf(bias + c) : 0.f;
    for (int r = 0; r < nr; ++r) {
      float acc = b0;
#pragma unroll 4
      for (int j = 0; j < taps; ++j) {
        const float* q = src[r][j];
        const float xv = q != nullptr ? q[c] : 0.f;
        acc = fmaf(ldf(w + (long long)c * taps + j), xv, acc);
      }
      tile[r * ch_block + cl] = act ? silu_f(acc) : acc;
      // this thread is the only one that touches channel c of the ring: its write follows its reads
      if (save_here && R > 0) state[((long long)slot[t0 + r] * R + pos[t0 + r] % R) * ch + c] = x[(long long)(t0 + r) * ldx + c];
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int unit_here = max(0, min(nc, unit_channels - c0));      // unit-vector channels of this block (whole groups)
  const int groups = unit_group > 0 ? unit_here / unit_group : 0;
  for (int rg = warp; rg < nr * groups; rg += nw) {
    const int r = rg / groups, g = rg - r * groups;
    float* row = tile + r * ch_block + g * unit_group;
    float ss = 0.f;
    for (int c = lane; c < unit_group; c += 32) ss = fmaf(row[c], row[c], ss);
    ss = seq_warp_sum(ss);
    const float f = (1.f / sqrtf(ss + unit_eps)) * (c0 + g * unit_group < scaled_channels ? unit_mult : 1.f);
    for (int c = lane; c < unit_group; c += 32) row[c] *= f;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nr * nc; e += blockDim.x) {
    const int r = e / nc, cl = e - r * nc;
    stf(y + (long long)(t0 + r) * ldy + c0 + cl, tile[r * ch_block + cl]);
  }
}

struct ConvUnit {   // unit vectors behind the convolution: the first `channels`, in groups of 4 * lanes, the first `scaled` of them times mult
  int channels, lanes, scaled;
  float eps, mult;
};

// The convolution with four neighbouring channels per thread: a thread walks ROWS consecutive rows with the last
// TAPS - 1 inputs in registers, so a row of x is read once per tile (plus TAPS - 1 rows in front of it), and nothing goes through
// shared memory. The same sums of taps as causal_conv_silu_kernel. UNIT: groups that a power of two of lanes of a warp holds are made unit vectors by
// shuffles among them (every warp is whole: ch is a multiple of 128); causal_conv_silu_kernel, a block of rows in shared memory, is for other
// groups. Nothing that a tile reads waits for another load of it, except for ring entries. 3126 rows of 4096 channels with unit queries and keys of
// 128: 73 us there, 31 here (3.3 TB/s; 34 with plain divisions in the activation, 42 with slots looked up in front of the rows before the tile); 6144 channels: 37
// (4.2 TB/s; 40 with plain divisions). What bounds it: half of the cycles the activation's instructions, otherwise the rows.
template <typename TW, typename TY, int TAPS, int ROWS, bool UNIT>
__global__ void __launch_bounds__(128) causal_conv_rows_kernel(const float* __restrict__ x, long long ldx, int T, int ch,
                                                               const TW* __restrict__ w, const TW* __restrict__ bias,
                                                               const int32_t* __restrict__ pos, const int32_t* __restrict__ slot,
                                                               float* __restrict__ state, TY* __restrict__ y, long long ldy, int save_here,
                                                               int act, ConvUnit unit, bool vec_w) {
  constexpr int R = TAPS - 1;
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
  if (!save_here) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // conv_state_save_kernel looks for its rows beside the last CTAs
  if (c >= ch) return;
  const int t0 = blockIdx.x * ROWS, nr = min(ROWS, T - t0);
  // everything that does not wait for anything else first: the rows, those in front of them, whose they are, the weights
  float4 xv[ROWS], h[R > 0 ? R : 1];   // h[j]: the input R - j positions back
#pragma unroll
  for (int r = 0; r < ROWS; ++r) xv[r] = r < nr ? *reinterpret_cast<const float4*>(x + (long long)(t0 + r) * ldx + c) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int j = 0; j < R; ++j) h[j] = t0 >= R - j ? *reinterpret_cast<const float4*>(x + (long long)(t0 - R + j) * ldx + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  int sl[R + ROWS];                    // slots of the rows from t0 - R on
#pragma unroll
  for (int j = 0; j < R + ROWS; ++j) sl[j] = t0 - R + j >= 0 && j < R + nr ? slot[t0 - R + j] : -1;
  float wv[TAPS][4], b4[4] = {0.f, 0.f, 0.f, 0.f};
  if constexpr (TAPS == 4) {
    if (vec_w) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float u[4];
        ld4(w + (long long)(c + i) * 4, u);
#pragma unroll
        for (int j = 0; j < 4; ++j) wv[j][i] = u[j];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (TAPS != 4 || !vec_w) {
#pragma unroll
      for (int j = 0; j < TAPS; ++j) wv[j][i] = ldf(w + (long long)(c + i) * TAPS + j);
    }
    if (bias != nullptr) b4[i] = ldf(bias + c + i);
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    if (r < nr) {
      const int t = t0 + r, s = sl[R + r], p = pos[t];
      if (r == 0) {                    // the inputs in front of the tile: rows of the same request, the ring or nothing
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const int sp = p - (R - j);
          if (sp < 0) h[j] = make_float4(0.f, 0.f, 0.f, 0.f);
          else if (sl[j] != s) h[j] = *reinterpret_cast<const float4*>(state + ((long long)s * R + sp % (R > 0 ? R : 1)) * ch + c);
        }
      } else if (s != sl[R + r - 1]) {   // first row of another request
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const int sp = p - (R - j);
          h[j] = sp >= 0 ? *reinterpret_cast<const float4*>(state + ((long long)s * R + sp % (R > 0 ? R : 1)) * ch + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      float o[4] = {b4[0], b4[1], b4[2], b4[3]};
#pragma unroll
      for (int j = 0; j < TAPS; ++j) {
        const float4 v = j < R ? h[j < R ? j : 0] : xv[r];
        o[0] = fmaf(wv[j][0], v.x, o[0]), o[1] = fmaf(wv[j][1], v.y, o[1]), o[2] = fmaf(wv[j][2], v.z, o[2]), o[3] = fmaf(wv[j][3], v.w, o[3]);
      }
      if (act) sigmoid4<true>(o);
      if (UNIT) {
        float ss = fmaf(o[0], o[0], fmaf(o[1], o[1], fmaf(o[2], o[2], o[3] * o[3])));
        for (int m = 1; m < unit.lanes; m <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, m);
        if (c < unit.channels) {
          const float f = (1.f / sqrtf(ss + unit.eps)) * (c < unit.scaled ? unit.mult : 1.f);
#pragma unroll
          for (int i = 0; i < 4; ++i) o[i] *= f;
        }
      }
      st4(y + (long long)t * ldy + c, o);
      // this thread is the only one that touches these channels of the ring: its write follows its reads
      if (save_here && R > 0) *reinterpret_cast<float4*>(state + ((long long)s * R + p % (R > 0 ? R : 1)) * ch + c) = xv[r];
#pragma unroll
      for (int j = 0; j + 1 < R; ++j) h[j] = h[j + 1];
      if (R > 0) h[R > 0 ? R - 1 : 0] = xv[r];
    }
  }
}

// The same convolution (no activation) in front of an attention: the first nq + nk channels are queries and keys that get an RMS norm
// per `group` channels (a head, or one score map of a head) with the weights wq / wk [group]; queries go to q_out, normed keys and the
// remaining channels (values) to the row of (slot, position) in the paged cache [pages][page_size][ch - nq]. One launch instead of
// convolution, norm and append, and the convolved rows never travel through memory.
template <typename TW, typename TC>
__global__ void __launch_bounds__(256) conv_qk_norm_store_kernel(const float* __restrict__ x, long long ldx, int T, int ch, int ch_block,
                                                                 int rows_per_cta, const TW* __restrict__ w, int taps,
                                                                 const int32_t* __restrict__ pos, const int32_t* __restrict__ slot,
                                                                 float* __restrict__ state, int nq, int nk, int group,
                                                                 const TW* __restrict__ wq, const TW* __restrict__ wk, float eps,
                                                                 const int32_t* __restrict__ block_table, int max_pages, int page_size,
                                                                 TC* __restrict__ pool, TC* __restrict__ q_out, long long ldqo,
                                                                 int save_here) {
  extern __shared__ float tile[];  // [rows_per_cta][ch_block]
  __shared__ const float* src[kConvRows][kConvMaxTaps];
  __shared__ TC* dst_row[kConvRows];   // the cache row of every row of this CTA
  const int t0 = blockIdx.x * rows_per_cta, nr = min(rows_per_cta, T - t0);
  const int c0 = blockIdx.y * ch_block, nc = min(ch_block, ch - c0);
  const int R = taps - 1;
  if (threadIdx.x < nr * taps) {
    const int r = threadIdx.x / taps, j = threadIdx.x - r * taps;
    const int t = t0 + r, p = pos[t], s = slot[t], back = R - j, sp = p - back;
    const float* q = nullptr;
    if (sp >= 0) q = (back == 0 || (t - back >= 0 && slot[t - back] == s)) ? x + (long long)(t - back) * ldx : state + ((long long)s * R + sp % R) * ch;
    src[r][j] = q;
  }
  if (threadIdx.x >= 224 && threadIdx.x - 224 < nr) {
    const int r = threadIdx.x - 224, p = pos[t0 + r];
    const int page = block_table[(long long)slot[t0 + r] * max_pages + p / page_size];
    dst_row[r] = pool + ((long long)page * page_size + p % page_size) * (ch - nq);
  }
  __syncthreads();
  for (int cl = threadIdx.x; cl < nc; cl += blockDim.x) {
    const int c = c0 + cl;
    for (int r = 0; r < nr; ++r) {
      float acc = 0.f;
#pragma unroll 4
      for (int j = 0; j < taps; ++j) {
        const float* q = src[r][j];
        const float xv = q != nullptr ? q[c] : 0.f;
        acc = fmaf(ldf(w + (long long)c * taps + j), xv, acc);
      }
      tile[r * ch_block + cl] = acc;
      if (save_here && R > 0) state[((long long)slot[t0 + r] * R + pos[t0 + r] % R) * ch + c] = x[(long long)(t0 + r) * ldx + c];
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int groups = max(0, min(nc, nq + nk - c0)) / group;      // normed groups of this block (blocks are whole groups)
  for (int rg = warp; rg < nr * groups; rg += nw) {
    const int r = rg / groups, g = rg - r * groups;
    float* row = tile + r * ch_block + g * group;
    const TW* wn = c0 + g * group < nq ? wq : wk;
    float ss = 0.f;
    for (int c = lane; c < group; c += 32) ss = fmaf(row[c], row[c], ss);
    ss = seq_warp_sum(ss);
    const float f = 1.f / sqrtf(ss / (float)group + eps);
    for (int c = lane; c < group; c += 32) row[c] = row[c] * f * ldf(wn + c);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nr * nc; e += blockDim.x) {
    const int r = e / nc, cl = e - r * nc, c = c0 + cl;
    const float v = tile[r * ch_block + cl];
    if (c < nq) stf(q_out + (long long)(t0 + r) * ldqo + c, v);
    else stf(dst_row[r] + (c - nq), v);
  }
}

// The last taps - 1 inputs of every request of the step go into its ring (rows that are followed by taps - 1 more rows of the
// same request are not among them). A launch of its own when a request may have several rows: a row's ring entry is read by
// CTAs of other rows of the convolution kernel.
constexpr int kSaveRows = 64;   // rows a CTA looks through
__global__ void __launch_bounds__(256) conv_state_save_kernel(const float* __restrict__ x, long long ldx, int ch, int R, int T,
                                                              const int32_t* __restrict__ pos, const int32_t* __restrict__ slot,
                                                              float* __restrict__ state) {
  __shared__ int s_last[kSaveRows];
  __shared__ int s_n;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  if (threadIdx.x < kSaveRows) {
    const int t = blockIdx.x * kSaveRows + threadIdx.x;
    if (t < T && !(t + R < T && slot[t + R] == slot[t])) s_last[atomicAdd(&s_n, 1)] = t;
  }
  __syncthreads();
  if (s_n == 0) return;
  asm volatile("griddepcontrol.wait;" ::: "memory");   // the convolution reads the rings. The step's last row is among the rows, so a CTA always waits, and this kernel ends behind it
  for (int i = 0; i < s_n; ++i) {   // every (row, channel) has a ring entry of its own: the order does not matter
    const int t = s_last[i];
    float* dst = state + ((long long)slot[t] * R + pos[t] % R) * ch;
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < ch; c += gridDim.y * blockDim.x) dst[c] = x[(long long)t * ldx + c];
  }
}
// Launched so that it may start beside the end of the convolution in front of it: both together 41.5 -> 39.2 us (3126 x 6144), 300 x 2048 10.7 -> 9.5.
static void save_conv_state(const float* x, long long ldx, int ch, int R, int T, const int32_t* pos, const int32_t* slot, float* state, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((T + kSaveRows - 1) / kSaveRows, (ch + 255) / 256), cfg.blockDim = dim3(256), cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr, cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, conv_state_save_kernel, x, ldx, ch, R, T, pos, slot, state);
}

// ---- linear-state recurrence ----------------------------------------------------------------------------------------------
constexpr int kScanLanes = 8, kScanGroups = 16, kScanThreads = kScanLanes * kScanGroups, kScanCpt = 2;

// Shared-memory place of key channel i: lane l = i / DPT owns DPT consecutive channels (read as float4), and a gap of four floats
// between the lanes' blocks moves them to different banks (the eight float4 reads of a quarter warp, at strides of 12, 20 or 36 floats, fall on different banks).
template <int DPT>
__device__ __forceinline__ int scan_place(int i) { return (i / DPT) * (DPT + 4) + (i % DPT); }

// Two stages of TOK tokens each: the raw inputs of the next chunk arrive by cp.async while the current chunk is computed;
// after arrival one pass turns them in place into what the recurrence uses (silu, decays, sigmoid). VEC: 16-byte copies
// (every row starts on a 16-byte boundary and the widths are multiples of four), else 4-byte copies.
// KIND: what enters the state - v itself, the delta rule's correction, or dt v (decay mode 6).
// TOK: tokens per stage; 1 for steps of one-token portions, whose CTAs then need little shared memory (more of them share
// an SM and keep state loads in flight: seven at 128 key channels, four at 256, which the launch bounds hold the registers to);
// any TOK is right for any portion.
//
// A thread owns DPT neighbouring key channels of CPT neighbouring columns: a packed register holds two neighbouring CHANNELS of one
// column, so that keys, queries and per-channel decays are used as they lie in shared memory, and only the numbers that all channels
// share (the input u of a column, a head's decay) are doubled. What bounds it is the issue of the three (delta: four) packed fma per
// state pair and token, behind them the latency of a token's chain; so what a token reads first is loaded during the token before it, and
// the read-out of a chunk is summed over the lanes once at its end, from shared memory, instead of by shuffles in every token. Portions of
// several tokens at 64 or 128 channels go to scan_rows_kernel below; measured here, 16 heads of 128 x 128, four portions of 1024, 777, 1024, 301
// tokens with per-channel decays: 435 us (560 with pairs of columns, a doubled key and a shuffled read-out per token); one token of 32 requests, step
// sizes: 22 us = 6.1 TB/s (42).
template <int DPT, int TOK>
__host__ __device__ constexpr int scan_stage_floats(bool chan, int cols) {
  return TOK * kScanLanes * (DPT + 4) * (chan ? 3 : 2) + TOK * cols + 2 * (TOK < 4 ? 4 : TOK);
}
template <int DPT, bool VEC, int KIND, bool CHAN, int TOK>   // CHAN: one decay per key channel
__global__ void __launch_bounds__(kScanThreads, TOK == 1 && DPT >= 16 ? (DPT == 32 ? 4 : 7) : 0) linear_state_scan_kernel(ScanArgs a) {
  constexpr bool LONG = CHAN || KIND == kScanDelta;   // long portions may be scan_chunk_kernel's
  if (LONG && scan_only_waits(a)) return;
  extern __shared__ __align__(16) float sm[];
  constexpr int PITCH = kScanLanes * (DPT + 4), CPT = kScanCpt, COLS = kScanGroups * CPT, DP = DPT / 2;
  constexpr int OPITCH = COLS + 4;           // a lane's partial read-outs of one token
  constexpr int HEADW = TOK < 4 ? 4 : TOK;   // one number per token, in whole 16-byte pieces
  const int dim = a.dim;
  constexpr bool WIDE = TOK == 1 && DPT <= 16;
  constexpr bool PRE = TOK > 1 && !CHAN;     // read ahead (per-channel decays fill the registers that this takes)
  const bool minus1 = KIND == kScanStep || a.decay_mode >= 4;  // the staged value is the decay minus one
  constexpr int stage_floats = scan_stage_floats<DPT, TOK>(CHAN, COLS);
  float* po = sm + 2 * stage_floats;         // [TOK][lanes][OPITCH] partial read-outs
  const int h = blockIdx.y, kvh = h / (a.H / a.G);
  const int col0 = blockIdx.x * COLS;
  const int r0 = a.row_begin[blockIdx.z], r1 = a.row_begin[blockIdx.z + 1];
  if (r1 <= r0 || (LONG && scan_is_long(a, r1 - r0))) return;
  // a decode step is a matter of reading and writing the states: there neighbouring threads take neighbouring columns (128 bytes of a row
  // of the state), and the lanes' sums meet in shared memory; otherwise the lanes of a column group are neighbours and meet by shuffles
  const int tid = threadIdx.x, lane = WIDE ? tid / kScanGroups : tid & (kScanLanes - 1), cg = WIDE ? tid % kScanGroups : tid / kScanLanes;
  const int col = col0 + CPT * cg;
  for (int e = tid; e < 2 * stage_floats; e += blockDim.x) sm[e] = 0.f;   // the pads stay zero: they meet zero state only
  float* S = a.state + (((long long)a.slot[r0] * a.H + h) * dim) * a.vdim;
  f32x2 st[CPT][DP];   // state elements (lane * DPT + 2 r, col + c) and (lane * DPT + 2 r + 1, col + c)
  const bool fresh = a.pos[r0] == 0;
#pragma unroll
  for (int r = 0; r < DP; ++r) {
    float e[2][CPT];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int i = lane * DPT + 2 * r + j;
      const float* row = S + (long long)i * a.vdim + col;
      const bool in = !fresh && i < dim;
      // the columns of a thread as one access (CPT divides vdim); one by one in a decode step, whose time is these loads: two columns at once have to
      // be taken apart into the registers that keep them, and fewer loads are on their way (256 requests, 64 heads of 128 x 64: 190 us, 307)
      if (a.vec_state && TOK != 1) {
        const float2 x = in && col < a.vdim ? *reinterpret_cast<const float2*>(row) : make_float2(0.f, 0.f);
        e[j][0] = x.x, e[j][1] = x.y;
      } else {
#pragma unroll
        for (int c = 0; c < CPT; ++c) e[j][c] = in && col + c < a.vdim ? row[c] : 0.f;
      }
    }
#pragma unroll
    for (int c = 0; c < CPT; ++c) st[c][r] = pack2(e[0][c], e[1][c]);
  }
  const float A = (KIND == kScanStep || a.decay_mode == 1 || a.decay_mode == 2) ? expf(a.A_log[h]) : 0.f;
  const float Dh = (KIND == kScanStep && a.D != nullptr) ? a.D[h] : 0.f;
  const float gconst = a.decay_mode == 0 ? a.decay_const[h] : 1.f;
  __syncthreads();

  // sum of a thread's numbers over the lanes, in the same order either way
  auto sum_lanes = [&](float (&x)[CPT]) {
    if constexpr (WIDE) {
      __syncthreads();   // the numbers of the sum before have been read
      *reinterpret_cast<float2*>(po + lane * OPITCH + CPT * cg) = make_float2(x[0], x[1]);
      __syncthreads();
      float2 s[kScanLanes];
#pragma unroll
      for (int l = 0; l < kScanLanes; ++l) s[l] = *reinterpret_cast<const float2*>(po + l * OPITCH + CPT * cg);
#pragma unroll
      for (int m = 1; m < kScanLanes; m <<= 1)
#pragma unroll
        for (int l = 0; l < kScanLanes; l += 2 * m) s[l].x += s[l + m].x, s[l].y += s[l + m].y;
      x[0] = s[0].x, x[1] = s[0].y;
    } else {
#pragma unroll
      for (int m = 1; m < kScanLanes; m <<= 1)
#pragma unroll
        for (int c = 0; c < CPT; ++c) x[c] += __shfl_xor_sync(0xffffffffu, x[c], m);
    }
  };
  auto issue = [&](int c0, int n, int stage) {
    float* sk = sm + stage * stage_floats;
    float* sq = sk + TOK * PITCH;
    float* sg = sq + TOK * PITCH;                       // [tok][PITCH] (per channel) or [tok]
    float* sv = sg + (CHAN ? TOK * PITCH : HEADW);
    float* sb = sv + TOK * COLS;
    if (VEC) {
      const int d4 = dim >> 2;
      for (int e = tid; e < n * d4; e += blockDim.x) {
        const int tt = e / d4, i = (e - tt * d4) << 2, at = tt * PITCH + scan_place<DPT>(i);
        cp_async16(sk + at, a.k + (long long)(c0 + tt) * a.ldk + kvh * dim + i);
        cp_async16(sq + at, a.q + (long long)(c0 + tt) * a.ldq + kvh * dim + i);
        if (CHAN) cp_async16(sg + at, a.a + (long long)(c0 + tt) * a.lda + h * dim + i);
      }
      for (int e = tid; e < n * (COLS / 4); e += blockDim.x) {
        const int tt = e / (COLS / 4), j = (e - tt * (COLS / 4)) << 2;
        if (col0 + j < a.vdim) cp_async16(sv + tt * COLS + j, a.v + (long long)(c0 + tt) * a.ldv + h * a.vdim + col0 + j);
      }
    } else {
      for (int e = tid; e < n * dim; e += blockDim.x) {
        const int tt = e / dim, i = e - tt * dim, at = tt * PITCH + scan_place<DPT>(i);
        cp_async4(sk + at, a.k + (long long)(c0 + tt) * a.ldk + kvh * dim + i);
        cp_async4(sq + at, a.q + (long long)(c0 + tt) * a.ldq + kvh * dim + i);
        if (CHAN) cp_async4(sg + at, a.a + (long long)(c0 + tt) * a.lda + h * dim + i);
      }
      for (int e = tid; e < n * COLS; e += blockDim.x) {
        const int tt = e / COLS, j = e - tt * COLS;
        if (col0 + j < a.vdim) cp_async4(sv + e, a.v + (long long)(c0 + tt) * a.ldv + h * a.vdim + col0 + j);
      }
    }
    if (tid < n) {
      if (KIND == kScanDelta) cp_async4(sb + tid, a.beta + (long long)(c0 + tid) * a.ldb + h);
      if (KIND == kScanStep || a.decay_mode == 1) cp_async4(sg + tid, a.a + (long long)(c0 + tid) * a.lda + h);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  issue(r0, min(TOK, r1 - r0), 0);
  int stage = 0;
  for (int c0 = r0; c0 < r1; c0 += TOK, stage ^= 1) {
    const int n = min(TOK, r1 - c0);
    if (c0 + TOK < r1) {
      issue(c0 + TOK, min(TOK, r1 - c0 - TOK), stage ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    float* sk = sm + stage * stage_floats;
    float* sq = sk + TOK * PITCH;
    float* sg = sq + TOK * PITCH;
    float* sv = sg + (CHAN ? TOK * PITCH : HEADW);
    float* sb = sv + TOK * COLS;
    // raw inputs -> what the recurrence uses
    if (a.silu_in || a.decay_mode == 2 || a.decay_mode == 4) {
      for (int e = tid; e < n * dim; e += blockDim.x) {
        const int tt = e / dim, i = e - tt * dim, at = tt * PITCH + scan_place<DPT>(i);
        if (a.silu_in) {
          sk[at] = silu_f(sk[at]);
          sq[at] = silu_f(sq[at]);
        }
        if (a.decay_mode == 2) sg[at] = expf(-A * softplus_f(sg[at] + a.dt_bias[h * dim + i]));
        else if (a.decay_mode == 4) sg[at] = sigmoid_pow_m1_f(sg[at] + (a.dt_bias != nullptr ? a.dt_bias[h * dim + i] : 0.f), a.decay_pow);
      }
    }
    if (a.silu_in)
      for (int e = tid; e < n * COLS; e += blockDim.x) sv[e] = silu_f(sv[e]);
    if (KIND == kScanStep) {
      if (tid < n) {
        const float dt = softplus_f(sg[tid] + a.dt_bias[h]);
        sb[tid] = dt;
        sg[tid] = expm1f(-A * dt);
      }
    } else if (tid < n) {
      sb[tid] = KIND == kScanDelta ? sigmoid_f(sb[tid]) : 1.f;
      if (a.decay_mode == 1) sg[tid] = expf(-A * softplus_f(sg[tid] + a.dt_bias[h]));
      else if (a.decay_mode == 0) sg[tid] = gconst;
    }
    __syncthreads();
    // what a token reads first - its key, input and shared numbers - is loaded while the token before it is computed
    f32x2 k2[DP];
    float un[CPT], gn, bn;
    auto fetch_key = [&](int tt) {
      const ulonglong2* kr = reinterpret_cast<const ulonglong2*>(sk + tt * PITCH + lane * (DPT + 4));
#pragma unroll
      for (int r = 0; r < DP; r += 2) {
        const ulonglong2 x = kr[r / 2];
        k2[r] = x.x, k2[r + 1] = x.y;
      }
    };
    auto fetch_shared = [&](int tt) {
#pragma unroll
      for (int c = 0; c < CPT; c += 2) {
        const float2 x = *reinterpret_cast<const float2*>(sv + tt * COLS + CPT * cg + c);
        un[c] = x.x, un[c + 1] = x.y;
      }
      gn = CHAN ? 0.f : sg[tt];
      bn = sb[tt];
    };
    if (PRE) fetch_key(0), fetch_shared(0);
    for (int tt = 0; tt < n; ++tt) {
      const int next = min(tt + 1, n - 1);
      if (!PRE) fetch_key(tt), fetch_shared(tt);
      float u[CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) u[c] = un[c];
      const float b = bn;
      if (CHAN) {
        const ulonglong2* gr = reinterpret_cast<const ulonglong2*>(sg + tt * PITCH + lane * (DPT + 4));
#pragma unroll
        for (int r = 0; r < DP; r += 2) {
          const ulonglong2 g = gr[r / 2];
#pragma unroll
          for (int c = 0; c < CPT; ++c) {
            st[c][r] = minus1 ? fma2(st[c][r], g.x, st[c][r]) : mul2(st[c][r], g.x);
            st[c][r + 1] = minus1 ? fma2(st[c][r + 1], g.y, st[c][r + 1]) : mul2(st[c][r + 1], g.y);
          }
        }
      } else {
        const f32x2 gh = pack2(gn, gn);
#pragma unroll
        for (int r = 0; r < DP; ++r)
#pragma unroll
          for (int c = 0; c < CPT; ++c) st[c][r] = minus1 ? fma2(st[c][r], gh, st[c][r]) : mul2(st[c][r], gh);
      }
      if (PRE) fetch_shared(next);
      const ulonglong2* qr = reinterpret_cast<const ulonglong2*>(sq + tt * PITCH + lane * (DPT + 4));
      f32x2 q2[DP];
      auto fetch_query = [&] {
#pragma unroll
        for (int r = 0; r < DP; r += 2) {
          const ulonglong2 x = qr[r / 2];
          q2[r] = x.x, q2[r + 1] = x.y;
        }
      };
      if (PRE) fetch_query();
      float vin[CPT];   // TOK == 1: what D multiplies
      if (KIND == kScanStep) {
#pragma unroll
        for (int c = 0; c < CPT; ++c) vin[c] = u[c], u[c] *= b;
      }
      if (KIND == kScanDelta) {
        float dot[CPT];
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          f32x2 d0 = 0ull, d1 = 0ull;   // two chains
#pragma unroll
          for (int r = 0; r < DP; r += 2) d0 = fma2(st[c][r], k2[r], d0), d1 = fma2(st[c][r + 1], k2[r + 1], d1);
          float w, x, y, z;
          unpack2(d0, w, x);
          unpack2(d1, y, z);
          dot[c] = (w + y) + (x + z);
        }
        sum_lanes(dot);
#pragma unroll
        for (int c = 0; c < CPT; ++c) u[c] = b * (u[c] - dot[c]);
      }
      f32x2 oa[CPT], ob[CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        const f32x2 u2 = pack2(u[c], u[c]);
        oa[c] = ob[c] = 0ull;
#pragma unroll
        for (int r = 0; r < DP; ++r) st[c][r] = fma2(k2[r], u2, st[c][r]);
      }
      if (PRE) fetch_key(next);
      else fetch_query();
#pragma unroll
      for (int r = 0; r < DP; r += 2)
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          oa[c] = fma2(st[c][r], q2[r], oa[c]);
          ob[c] = fma2(st[c][r + 1], q2[r + 1], ob[c]);
        }
      float o[CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        float w, x, y, z;
        unpack2(oa[c], w, x);
        unpack2(ob[c], y, z);
        o[c] = (w + y) + (x + z);
      }
      if constexpr (TOK == 1) {
        sum_lanes(o);
        if (lane == 0) {
          float* dst = a.out + (long long)(c0 + tt) * a.ldo + h * a.vdim + col;
#pragma unroll
          for (int c = 0; c < CPT; ++c) {
            if (KIND == kScanStep) o[c] = fmaf(Dh, vin[c], o[c]);
            if (col + c < a.vdim) dst[c] = o[c] * a.out_scale;
          }
        }
      } else {
        float* dst = po + (tt * kScanLanes + lane) * OPITCH + CPT * cg;
#pragma unroll
        for (int c = 0; c < CPT; c += 2) *reinterpret_cast<float2*>(dst + c) = make_float2(o[c], o[c + 1]);
      }
    }
    __syncthreads();   // the partial read-outs are there; the next iteration's copies overwrite the stage that was just read
    if constexpr (TOK > 1) {
      for (int e = tid; e < n * (COLS / 4); e += blockDim.x) {
        const int tt = e / (COLS / 4), j = (e - tt * (COLS / 4)) << 2;
        if (col0 + j >= a.vdim) continue;
        const float* src = po + tt * kScanLanes * OPITCH + j;
        float4 s[kScanLanes];
#pragma unroll
        for (int l = 0; l < kScanLanes; ++l) s[l] = *reinterpret_cast<const float4*>(src + l * OPITCH);
#pragma unroll
        for (int m = 1; m < kScanLanes; m <<= 1)   // the order of sum_lanes: the same bits
#pragma unroll
          for (int l = 0; l < kScanLanes; l += 2 * m) s[l].x += s[l + m].x, s[l].y += s[l + m].y, s[l].z += s[l + m].z, s[l].w += s[l + m].w;
        float4 o = s[0];
        if (KIND == kScanStep) {
          const float4 x = *reinterpret_cast<const float4*>(sv + tt * COLS + j);
          o.x = fmaf(Dh, x.x, o.x), o.y = fmaf(Dh, x.y, o.y), o.z = fmaf(Dh, x.z, o.z), o.w = fmaf(Dh, x.w, o.w);
        }
        o.x *= a.out_scale, o.y *= a.out_scale, o.z *= a.out_scale, o.w *= a.out_scale;
        float* dst = a.out + (long long)(c0 + tt) * a.ldo + h * a.vdim + col0 + j;
        if (a.vec_out) {
          *reinterpret_cast<float4*>(dst) = o;
        } else {
          dst[0] = o.x;
          if (col0 + j + 1 < a.vdim) dst[1] = o.y;
          if (col0 + j + 2 < a.vdim) dst[2] = o.z;
          if (col0 + j + 3 < a.vdim) dst[3] = o.w;
        }
      }
      if (KIND == kScanStep) __syncthreads();   // v is read here too
    }
  }
#pragma unroll
  for (int r = 0; r < DP; ++r) {
    float e[2][CPT];
#pragma unroll
    for (int c = 0; c < CPT; ++c) unpack2(st[c][r], e[0][c], e[1][c]);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int i = lane * DPT + 2 * r + j;
      float* row = S + (long long)i * a.vdim + col;
      if (i >= dim) continue;
      if (a.vec_state) {
        if (col < a.vdim) *reinterpret_cast<float2*>(row) = make_float2(e[j][0], e[j][1]);
      } else {
#pragma unroll
        for (int c = 0; c < CPT; ++c)
          if (col + c < a.vdim) row[c] = e[j][c];
      }
    }
  }
}

// The same recurrence for portions of several tokens at 64 or 128 key channels, inputs that need no preparation of their own (no silu, per-channel decays given)
// and 16-byte rows: the same sums in the same order, so the same bits, with what the general kernel spends beside them taken out (addresses and
// bookkeeping per token, a third barrier per stage, the decays' exponentials between two of them). Here the widths are constants, a stage is
// eight tokens without a loop around them, with two barriers, and the decays and step sizes of the next stage are formed in the shadow of this one. A CTA of four warps has
// CPT columns per group of eight lanes (see the launch). What bounds it: a token's chain through 92 instructions per warp (step sizes; delta rule 135), some three
// cycles each where a scheduler has one warp (4 heads, 1100 tokens: 440 cycles per token), with many CTAs the packed fma (58 % of the pipe's cycles) and the shared-memory
// reads of keys and queries (74 % of the data path's). Measured in us, the general kernel in brackets: step sizes, 64 heads of
// 128 x 64, portions of 1024, 777, 1024, 301 tokens 292 (340), 32 x 64 tokens 154 (228), 16 heads, 1100 tokens 149 (195). Long portions of the delta rule and with
// per-channel decays are scan_chunk.cu's.
constexpr int kSrTok = 8, kSrThreads = 128;
template <int DIM, int COLS, bool CHAN>
struct ScanRowsStage {
  static constexpr int PITCH = kScanLanes * (DIM / kScanLanes + 4);
  float k[kSrTok * PITCH], q[kSrTok * PITCH], g[CHAN ? kSrTok * PITCH : 4], v[kSrTok * COLS];
  float2 gb[kSrTok];   // a token's decay (or the decay minus one) and its beta or step size
};
template <int DIM, int COLS, bool CHAN>
struct ScanRowsShared {
  ScanRowsStage<DIM, COLS, CHAN> stage[2];
  float po[kSrTok * kScanLanes * (COLS + 4)];   // [token][lane][column]: partial read-outs
};

template <int DIM, int CPT, int KIND, bool CHAN>
__global__ void __launch_bounds__(kSrThreads) scan_rows_kernel(ScanArgs a) {
  constexpr bool LONG = CHAN || KIND == kScanDelta;   // long portions may be scan_chunk_kernel's
  if (LONG && scan_only_waits(a)) return;
  extern __shared__ __align__(16) float sm[];
  constexpr int COLS = kSrThreads / kScanLanes * CPT;
  typedef ScanRowsShared<DIM, COLS, CHAN> Shared;
  typedef ScanRowsStage<DIM, COLS, CHAN> Stage;
  Shared& sh = *reinterpret_cast<Shared*>(sm);
  constexpr int DPT = DIM / kScanLanes, DP = DPT / 2, PITCH = Stage::PITCH, OPITCH = COLS + 4;
  const bool minus1 = KIND == kScanStep || a.decay_mode == 5;
  const int h = blockIdx.y, kvh = h / (a.H / a.G), col0 = blockIdx.x * COLS;
  const int portion = a.portions > 1 ? scan_portion(a.row_begin, a.portions, blockIdx.z, reinterpret_cast<int*>(sm)) : blockIdx.z;
  const int r0 = a.row_begin[portion], r1 = a.row_begin[portion + 1];
  if (r1 <= r0 || (LONG && scan_is_long(a, r1 - r0))) return;
  const int tid = threadIdx.x, lane = tid & (kScanLanes - 1), cg = tid / kScanLanes, col = col0 + CPT * cg;
  const bool in = col < a.vdim;   // a thread's columns all exist or none does
  const float A = KIND == kScanStep || a.decay_mode == 1 ? expf(a.A_log[h]) : 0.f;
  const float bias = KIND == kScanStep || a.decay_mode == 1 ? a.dt_bias[h] : 0.f;
  const float Dh = KIND == kScanStep && a.D != nullptr ? a.D[h] : 0.f;
  const float gconst = a.decay_mode == 0 ? a.decay_const[h] : 1.f;

  // a thread copies the 16-byte pieces `piece` of tokens tok0, tok0 + STEP, ...
  constexpr int PIECES = DIM / 4, STEP = kSrThreads / PIECES;
  const int piece = tid % PIECES, tok0 = tid / PIECES, place = scan_place<DPT>(piece * 4);
  const float* kp = a.k + (long long)kvh * DIM + piece * 4;
  const float* qp = a.q + (long long)kvh * DIM + piece * 4;
  const float* gp = CHAN ? a.a + (long long)h * DIM + piece * 4 : nullptr;
  constexpr int VP = COLS / 4, PARTS = CHAN ? kSrThreads / (kSrTok * VP) : 1, PL = kScanLanes / PARTS;   // pieces of a token's columns; threads per token and piece of the
  const int vtok = tid / VP, vcol = tid % VP * 4, otok = tid / (VP * PARTS), opart = tid / VP % PARTS;   // read-out, and lanes that each of them adds up
  const float* vp = a.v + (long long)h * a.vdim + col0 + vcol;
  auto issue = [&](int c0, Stage& s) {
#pragma unroll
    for (int i = 0; i < kSrTok; i += STEP) {
      const int tt = tok0 + i;
      if (c0 + tt < r1) {
        cp_async16(s.k + tt * PITCH + place, kp + (long long)(c0 + tt) * a.ldk);
        cp_async16(s.q + tt * PITCH + place, qp + (long long)(c0 + tt) * a.ldq);
        if (CHAN) cp_async16(s.g + tt * PITCH + place, gp + (long long)(c0 + tt) * a.lda);
      }
    }
    if (vtok < kSrTok && c0 + vtok < r1 && col0 + vcol < a.vdim) cp_async16(s.v + vtok * COLS + vcol, vp + (long long)(c0 + vtok) * a.ldv);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // raw numbers of token c0 + tid, and what the recurrence makes of them
  float raw_a = 0.f, raw_b = 0.f;
  auto load_raw = [&](int c0) {
    const int t = c0 + tid;
    if (tid < kSrTok && t < r1) {
      if (KIND == kScanStep || a.decay_mode == 1) raw_a = a.a[(long long)t * a.lda + h];
      if (KIND == kScanDelta) raw_b = a.beta[(long long)t * a.ldb + h];
    }
  };
  auto put_raw = [&](Stage& s) {
    if (tid >= kSrTok) return;
    if (KIND == kScanStep) {
      const float dt = softplus_f(raw_a + bias);
      s.gb[tid] = make_float2(expm1f(-A * dt), dt);
    } else {
      s.gb[tid] = make_float2(a.decay_mode == 1 ? expf(-A * softplus_f(raw_a + bias)) : gconst, KIND == kScanDelta ? sigmoid_f(raw_b) : 1.f);
    }
  };

  issue(r0, sh.stage[0]);
  load_raw(r0);
  float* S = a.state + (((long long)a.slot[r0] * a.H + h) * DIM) * a.vdim;
  f32x2 st[CPT][DP];   // state elements (lane * DPT + 2 r, col + c) and (lane * DPT + 2 r + 1, col + c)
  const bool fresh = a.pos[r0] == 0;
#pragma unroll
  for (int r = 0; r < DP; ++r) {
    float e[2][CPT];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float* row = S + (long long)(lane * DPT + 2 * r + j) * a.vdim + col;
      const bool read = !fresh && in;
      if constexpr (CPT == 1) {
        e[j][0] = read ? *row : 0.f;
      } else if constexpr (CPT == 4) {
        const float4 x = read ? *reinterpret_cast<const float4*>(row) : make_float4(0.f, 0.f, 0.f, 0.f);
        e[j][0] = x.x, e[j][1] = x.y, e[j][2] = x.z, e[j][3] = x.w;
      } else {
        const float2 x = read ? *reinterpret_cast<const float2*>(row) : make_float2(0.f, 0.f);
        e[j][0] = x.x, e[j][1] = x.y;
      }
    }
#pragma unroll
    for (int c = 0; c < CPT; ++c) st[c][r] = pack2(e[0][c], e[1][c]);
  }
  put_raw(sh.stage[0]);
  load_raw(r0 + kSrTok);

  int at = 0;
  for (int c0 = r0; c0 < r1; c0 += kSrTok, at ^= 1) {
    const int n = min(kSrTok, r1 - c0);
    Stage& s = sh.stage[at];
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();   // this stage is there; the other one, and the partial read-outs, have been read by all
    if (c0 + kSrTok < r1) {
      issue(c0 + kSrTok, sh.stage[at ^ 1]);
      put_raw(sh.stage[at ^ 1]);
      load_raw(c0 + 2 * kSrTok);
    }
    f32x2 k2[DP];
    float un[CPT];
    float2 gb;
    auto fetch = [&](int tt) {   // what a token reads first, during the token before it
      const ulonglong2* kr = reinterpret_cast<const ulonglong2*>(s.k + tt * PITCH + lane * (DPT + 4));
#pragma unroll
      for (int r = 0; r < DP; r += 2) {
        const ulonglong2 x = kr[r / 2];
        k2[r] = x.x, k2[r + 1] = x.y;
      }
    };
    auto fetch_shared = [&](int tt) {
      const float* p = s.v + tt * COLS + CPT * cg;
      if constexpr (CPT == 1) {
        un[0] = *p;
      } else if constexpr (CPT == 4) {
        const float4 x = *reinterpret_cast<const float4*>(p);
        un[0] = x.x, un[1] = x.y, un[2] = x.z, un[3] = x.w;
      } else {
        const float2 x = *reinterpret_cast<const float2*>(p);
        un[0] = x.x, un[1] = x.y;
      }
      gb = s.gb[tt];
    };
    fetch(0);
    fetch_shared(0);
    auto token = [&](int tt, int next) {
      float u[CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) u[c] = KIND == kScanStep ? un[c] * gb.y : un[c];
      const float b = gb.y;
      if constexpr (CHAN) {
        const ulonglong2* gr = reinterpret_cast<const ulonglong2*>(s.g + tt * PITCH + lane * (DPT + 4));
#pragma unroll
        for (int r = 0; r < DP; r += 2) {
          const ulonglong2 g = gr[r / 2];
#pragma unroll
          for (int c = 0; c < CPT; ++c) {
            st[c][r] = minus1 ? fma2(st[c][r], g.x, st[c][r]) : mul2(st[c][r], g.x);
            st[c][r + 1] = minus1 ? fma2(st[c][r + 1], g.y, st[c][r + 1]) : mul2(st[c][r + 1], g.y);
          }
        }
      } else {
        const f32x2 gh = pack2(gb.x, gb.x);
#pragma unroll
        for (int r = 0; r < DP; ++r)
#pragma unroll
          for (int c = 0; c < CPT; ++c) st[c][r] = minus1 ? fma2(st[c][r], gh, st[c][r]) : mul2(st[c][r], gh);
      }
      fetch_shared(next);
      f32x2 q2[DP];
      const ulonglong2* qr = reinterpret_cast<const ulonglong2*>(s.q + tt * PITCH + lane * (DPT + 4));
#pragma unroll
      for (int r = 0; r < DP; r += 2) {
        const ulonglong2 x = qr[r / 2];
        q2[r] = x.x, q2[r + 1] = x.y;
      }
      auto columns = [&](const f32x2 (&with)[DP], float (&sum)[CPT]) {   // the general kernel's two chains per column
        f32x2 x0[CPT], x1[CPT];
#pragma unroll
        for (int c = 0; c < CPT; ++c) x0[c] = x1[c] = 0ull;
#pragma unroll
        for (int r = 0; r < DP; r += 2)
#pragma unroll
          for (int c = 0; c < CPT; ++c) x0[c] = fma2(st[c][r], with[r], x0[c]), x1[c] = fma2(st[c][r + 1], with[r + 1], x1[c]);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          float w, x, y, z;
          unpack2(x0[c], w, x);
          unpack2(x1[c], y, z);
          sum[c] = (w + y) + (x + z);
        }
      };
      if (KIND == kScanDelta) {
        float dot[CPT];
        columns(k2, dot);
#pragma unroll
        for (int m = 1; m < kScanLanes; m <<= 1)
#pragma unroll
          for (int c = 0; c < CPT; ++c) dot[c] += __shfl_xor_sync(0xffffffffu, dot[c], m);
#pragma unroll
        for (int c = 0; c < CPT; ++c) u[c] = b * (u[c] - dot[c]);
      }
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        const f32x2 u2 = pack2(u[c], u[c]);
#pragma unroll
        for (int r = 0; r < DP; ++r) st[c][r] = fma2(k2[r], u2, st[c][r]);
      }
      fetch(next);
      float o[CPT];
      columns(q2, o);
      float* dst = sh.po + (tt * kScanLanes + lane) * OPITCH + CPT * cg;
      if constexpr (CPT == 1) *dst = o[0];
      else if constexpr (CPT == 4) *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1], o[2], o[3]);
      else *reinterpret_cast<float2*>(dst) = make_float2(o[0], o[1]);
    };
    if (n == kSrTok) {
#pragma unroll (CHAN ? 1 : kSrTok)
      for (int tt = 0; tt < kSrTok; ++tt) token(tt, min(tt + 1, kSrTok - 1));
    } else {
#pragma unroll 1
      for (int tt = 0; tt < n; ++tt) token(tt, min(tt + 1, n - 1));
    }
    __syncthreads();   // the partial read-outs are there
    if (PARTS == 1 && otok >= n) continue;
    const float* src = sh.po + (otok * kScanLanes + opart * PL) * OPITCH + vcol;
    float4 x[PL];
#pragma unroll
    for (int l = 0; l < PL; ++l) x[l] = *reinterpret_cast<const float4*>(src + l * OPITCH);
#pragma unroll
    for (int m = 1; m < PL; m <<= 1)   // the order of the general kernel, through the threads that share a piece: the same bits
#pragma unroll
      for (int l = 0; l < PL; l += 2 * m) x[l].x += x[l + m].x, x[l].y += x[l + m].y, x[l].z += x[l + m].z, x[l].w += x[l + m].w;
    float4 o = x[0];
#pragma unroll
    for (int m = VP; m < VP * PARTS; m <<= 1) {
      o.x += __shfl_xor_sync(0xffffffffu, o.x, m), o.y += __shfl_xor_sync(0xffffffffu, o.y, m);
      o.z += __shfl_xor_sync(0xffffffffu, o.z, m), o.w += __shfl_xor_sync(0xffffffffu, o.w, m);
    }
    if (otok < n && opart == 0 && col0 + vcol < a.vdim) {
      if (KIND == kScanStep) {
        const float4 v = *reinterpret_cast<const float4*>(s.v + otok * COLS + vcol);
        o.x = fmaf(Dh, v.x, o.x), o.y = fmaf(Dh, v.y, o.y), o.z = fmaf(Dh, v.z, o.z), o.w = fmaf(Dh, v.w, o.w);
      }
      o.x *= a.out_scale, o.y *= a.out_scale, o.z *= a.out_scale, o.w *= a.out_scale;
      *reinterpret_cast<float4*>(a.out + (long long)(c0 + otok) * a.ldo + h * a.vdim + col0 + vcol) = o;
    }
  }
  if (!in) return;
#pragma unroll
  for (int r = 0; r < DP; ++r) {
    float e[2][CPT];
#pragma unroll
    for (int c = 0; c < CPT; ++c) unpack2(st[c][r], e[0][c], e[1][c]);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float* row = S + (long long)(lane * DPT + 2 * r + j) * a.vdim + col;
      if constexpr (CPT == 1) *row = e[j][0];
      else if constexpr (CPT == 4) *reinterpret_cast<float4*>(row) = make_float4(e[j][0], e[j][1], e[j][2], e[j][3]);
      else *reinterpret_cast<float2*>(row) = make_float2(e[j][0], e[j][1]);
    }
  }
}

// ---- elementwise preparation of a recurrence's inputs --------------------------------------------------------------------
// In place over x[t, :cols]: op 1: silu; op 2: x <- exp(-exp(A_log[c / group]) * softplus(x + bias[c])), the per-channel decay;
// op 3: x <- sigmoid(x + bias[c])^p - 1, the decay of a gated linear attention as its distance from 1.
// The recurrence can do both itself while it stages its inputs; for long portions one pass here is cheaper than doing it in
// every CTA that shares a head.
__global__ void __launch_bounds__(256) map_rows_kernel(float* __restrict__ x, long long ldx, int cols, long long total, int op,
                                                       const float* __restrict__ A_log, const float* __restrict__ bias, int group, float p_exp) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= total) return;
  const long long t = e / cols;
  const int c = (int)(e - t * cols);
  float* p = x + t * ldx + c;
  if (op == 1) *p = silu_f(*p);
  else if (op == 3) *p = sigmoid_pow_m1_f(*p + (bias != nullptr ? bias[c] : 0.f), p_exp);
  else *p = expf(-expf(A_log[c / group]) * softplus_f(*p + bias[c]));
}

// ---- gated RMS norm over groups of a row ----------------------------------------------------------------------------------
// y[t, g * n + c] = x[t, g * n + c] / sqrt(mean_c x^2 + eps) * w[c] * act(gate[t, g * n + c]); a warp per group.
template <typename TW, typename TY>
__global__ void __launch_bounds__(256) gated_rms_kernel(const float* __restrict__ x, long long ldx, int groups, int n,
                                                        const TW* __restrict__ w, float eps, const float* __restrict__ gate,
                                                        long long ldg, int gate_act, TY* __restrict__ y, long long ldy) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const long long t = blockIdx.x;
  for (int g = blockIdx.y * nw + warp; g < groups; g += nw * gridDim.y) {
    const float* xr = x + t * ldx + (long long)g * n;
    float ss = 0.f;
    for (int c = lane; c < n; c += 32) ss = fmaf(xr[c], xr[c], ss);
    ss = seq_warp_sum(ss);
    const float rstd = 1.f / sqrtf(ss / (float)n + eps);
    for (int c = lane; c < n; c += 32) {
      float v = xr[c] * rstd * ldf(w + c);
      if (gate != nullptr) {
        const float z = gate[t * ldg + (long long)g * n + c];
        v *= gate_act == 1 ? silu_f(z) : (gate_act == 2 ? sigmoid_f(z) : z);
      }
      stf(y + t * ldy + (long long)g * n + c, v);
    }
  }
}


// Both norms for groups that LANES neighbouring lanes hold in PIECES pieces of four columns each (n = 4 LANES PIECES): x and the gate are read once, all
// of it before anything is waited for, and no two warps meet. FRONT: the gate in front of the norm and a weight for every column of the row, else behind
// it and one weight of n columns for all groups. 3126 rows: 8 parts of 512 with a bf16 gate in front 38 -> 18 us (22 with plain divisions in the gate; 20 without the bound on
// registers, which the quotients' rare way out takes), 16 groups of 128 with an fp32 gate behind 29 -> 14 (16)
// (a block per part, a warp per group reading single columns twice).
template <typename TG, typename TW, typename TY, int LANES, int PIECES, bool FRONT>
__global__ void __launch_bounds__(256, FRONT && PIECES == 4 ? 5 : 0) group_rms_kernel(const float* __restrict__ x, long long ldx, int groups, long long total, const TW* __restrict__ w, float eps,
                                                        const TG* __restrict__ gate, long long ldg, int gate_act, TY* __restrict__ y, long long ldy) {
  constexpr int N = 4 * LANES * PIECES;
  const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / LANES;   // (row, group)
  const int lane = threadIdx.x % LANES;
  const bool live = i < total;
  const long long t = live ? i / groups : 0;
  const int c0 = live ? (int)(i - t * groups) * N : 0;
  float v[PIECES][4], g[PIECES][4], wv[PIECES][4];
#pragma unroll
  for (int p = 0; p < PIECES; ++p) {
    const int c = (p * LANES + lane) * 4;
    ld4(x + t * ldx + c0 + c, v[p]);
    if (gate != nullptr) ld4(gate + t * ldg + c0 + c, g[p]);
  }
  if (gate != nullptr && gate_act != 0) {
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      if (gate_act == 1) sigmoid4<true>(g[p]);
      else sigmoid4<false>(g[p]);
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int p = 0; p < PIECES; ++p)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (FRONT) v[p][e] *= g[p][e];
      ss = fmaf(v[p][e], v[p][e], ss);
    }
#pragma unroll
  for (int p = 0; p < PIECES; ++p) ld4(w + (FRONT ? c0 : 0) + (p * LANES + lane) * 4, wv[p]);   // where a gate in front has left its registers
#pragma unroll
  for (int m = LANES / 2; m > 0; m >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, m);
  const float rstd = 1.f / sqrtf(ss / (float)N + eps);
  if (!live) return;
#pragma unroll
  for (int p = 0; p < PIECES; ++p) {
    float o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      o[e] = v[p][e] * rstd * wv[p][e];
      if (!FRONT && gate != nullptr) o[e] *= g[p][e];
    }
    st4(y + t * ldy + c0 + (p * LANES + lane) * 4, o);
  }
}

// Launches it for the widths it takes (a power of two from 32 to 1024 columns, everything on 16 bytes); false: not one of them.
template <bool FRONT, typename TG, typename TW, typename TY>
static bool group_rms(const float* x, long long ldx, int rows, int groups, int n, const TW* w, float eps, const TG* gate, long long ldg, int gate_act, TY* y, long long ldy,
                      cudaStream_t st) {
  auto al = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  if (ldx % 4 || (gate != nullptr && ldg % 4) || ldy % 4 || !al(x) || !al(gate) || !al(y) || !al(w)) return false;
  const long long total = (long long)rows * groups;
  auto go = [&](auto lanes, auto pieces) {
    constexpr int L = decltype(lanes)::value, P = decltype(pieces)::value;
    const long long blocks = (total * L + 255) / 256;
    if (blocks >= 1ll << 31) return false;
    group_rms_kernel<TG, TW, TY, L, P, FRONT><<<(unsigned)blocks, 256, 0, st>>>(x, ldx, groups, total, w, eps, gate, ldg, gate_act, y, ldy);
    return true;
  };
  using std::integral_constant;
  if (n == 32) return go(integral_constant<int, 8>(), integral_constant<int, 1>());
  if (n == 64) return go(integral_constant<int, 16>(), integral_constant<int, 1>());
  if (n == 128) return go(integral_constant<int, 32>(), integral_constant<int, 1>());
  if (n == 256) return go(integral_constant<int, 32>(), integral_constant<int, 2>());
  if (n == 512) return go(integral_constant<int, 32>(), integral_constant<int, 4>());
  if (n == 1024) return go(integral_constant<int, 32>(), integral_constant<int, 8>());
  return false;
}

// The gate in front of the norm: v = x * act(gate), y = v / sqrt(mean(v^2) + eps) * w with the mean over each of `groups` equal parts of
// the row and a weight for every column. NT threads per (row, part); a thread keeps its elements in registers (VEC: four neighbours
// at a time), parts too wide for that are read twice.
constexpr int kGateRmsRegs = 8;   // elements (VEC: float4 pieces) a thread keeps
template <typename TG, typename TW, typename TY, bool VEC>
__global__ void __launch_bounds__(256) gate_rms_kernel(const float* __restrict__ x, long long ldx, int n, const TW* __restrict__ w, float eps,
                                                       const TG* __restrict__ gate, long long ldg, int gate_act, TY* __restrict__ y, long long ldy) {
  __shared__ float red[33];
  const long long t = blockIdx.x;
  const long long c0 = (long long)blockIdx.y * n;
  const float* xr = x + t * ldx + c0;
  const TG* gr = gate + t * ldg + c0;
  auto act = [&](float z) { return gate_act == 1 ? silu_f(z) : (gate_act == 2 ? sigmoid_f(z) : z); };
  constexpr int V = VEC ? 4 : 1;
  float keep[kGateRmsRegs][V];
  float ss = 0.f;
  auto value = [&](int c, float (&v)[V]) {
    if constexpr (VEC) {
      float g[4];
      ld4(xr + c, v);
      ld4(gr + c, g);
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] *= act(g[i]);
    } else {
      v[0] = xr[c] * act(ldf(gr + c));
    }
  };
#pragma unroll
  for (int i = 0; i < kGateRmsRegs; ++i) {
    const int c = (i * blockDim.x + threadIdx.x) * V;
    if (c < n) {
      value(c, keep[i]);
#pragma unroll
      for (int e = 0; e < V; ++e) ss = fmaf(keep[i][e], keep[i][e], ss);
    }
  }
  for (int c = (kGateRmsRegs * blockDim.x + threadIdx.x) * V; c < n; c += blockDim.x * V) {
    float v[V];
    value(c, v);
#pragma unroll
    for (int e = 0; e < V; ++e) ss = fmaf(v[e], v[e], ss);
  }
  const float rstd = 1.f / sqrtf(block_sum(ss, red) / (float)n + eps);
  auto put = [&](int c, const float (&v)[V]) {
    if constexpr (VEC) {
      float wv[4];
      ld4(w + c0 + c, wv);
      const float o[4] = {v[0] * rstd * wv[0], v[1] * rstd * wv[1], v[2] * rstd * wv[2], v[3] * rstd * wv[3]};
      st4(y + t * ldy + c0 + c, o);
    } else {
      stf(y + t * ldy + c0 + c, v[0] * rstd * ldf(w + c0 + c));
    }
  };
#pragma unroll
  for (int i = 0; i < kGateRmsRegs; ++i) {
    const int c = (i * blockDim.x + threadIdx.x) * V;
    if (c < n) put(c, keep[i]);
  }
  for (int c = (kGateRmsRegs * blockDim.x + threadIdx.x) * V; c < n; c += blockDim.x * V) {
    float v[V];
    value(c, v);
    put(c, v);
  }
}

// ---- tanh norm + input convolution of a sublayer ----------------------------------------------------------------------------
// What a sublayer of a "tanh-norm" decoder reads: with the stream row x (optionally first updated by the previous sublayer's
// output, x <- x + a1 y1 + a2 y2), h = tanh(alpha x) * nw + nb (a norm without statistics) and u = h + sum_j cw[:, j] h_(t - taps + 1 + j),
// a causal convolution over time per channel whose last taps - 1 inputs h live in a ring per slot like the other convolutions'.
// A CTA owns (1 or 8 consecutive rows + the taps - 1 rows in front of them, a block of channels): h is evaluated once per tile
// element into shared memory, then every row's taps read the tile, a ring entry or nothing.
// tanh for the norm. FAST (bf16 output): 1 - 2 / (exp(2x) + 1) through the hardware exponential, absolute error of a few 1e-7 -
// far below the rounding of the output; otherwise the library function.
template <bool FAST>
__device__ __forceinline__ float tanh_norm_f(float x) {
  if (FAST) {
    const float e = exp2f(fminf(x, 20.f) * 2.8853900817779268f);
    return 1.f - __fdividef(2.f, e + 1.f);
  }
  return tanhf(x);
}
template <bool FAST, typename TW>
__device__ __forceinline__ float dyt_f(float x, float alpha, const TW* __restrict__ nw, const TW* __restrict__ nb, int c) {
  return fmaf(tanh_norm_f<FAST>(alpha * x), ldf(nw + c), ldf(nb + c));
}
template <typename T>
struct is_bf16_t { static constexpr bool value = false; };
template <>
struct is_bf16_t<bf16_t> { static constexpr bool value = true; };

constexpr int kDytRegTaps = 8;   // convolutions of up to this many taps keep a channel's weights in registers across the rows
constexpr int kDytRows = 8;      // rows per CTA of a long step: the taps - 1 halo rows in front are evaluated once more per CTA (16 rows were slower)

template <typename TW, typename TU>
__global__ void __launch_bounds__(256) dyt_conv_kernel(const float* __restrict__ x, long long ldx, const float* __restrict__ y1, long long ld1,
                                                       float a1, const float* __restrict__ y2, long long ld2, float a2,
                                                       float* __restrict__ x_out, long long ldxo, const float* __restrict__ alpha_p,
                                                       const TW* __restrict__ nw, const TW* __restrict__ nb, const TW* __restrict__ cw, int taps,
                                                       const int32_t* __restrict__ pos, const int32_t* __restrict__ slot,
                                                       float* __restrict__ state, TU* __restrict__ u, long long ldu, int T, int C, int ch_block,
                                                       int rows_per_cta, int save_here) {
  constexpr bool FAST = is_bf16_t<TU>::value;
  extern __shared__ float tile[];  // [rows_per_cta + taps - 1][ch_block]: h of the halo rows, then of the CTA's own rows
  // where tap j of row r reads: a row of the tile (src_tile >= 0), a ring entry (src_ring != NULL, indexed by the channel), or nothing
  __shared__ int src_tile[kDytRows][kConvMaxTaps];
  __shared__ const float* src_ring[kDytRows][kConvMaxTaps];
  const int R = taps - 1;
  const int t0 = blockIdx.x * rows_per_cta, nr = min(rows_per_cta, T - t0);
  const int c0 = blockIdx.y * ch_block, nc = min(ch_block, C - c0);
  const float alpha = *alpha_p;
  for (int e = threadIdx.x; e < nr * taps; e += blockDim.x) {
    const int r = e / taps, j = e - r * taps;
    const int t = t0 + r, p = pos[t], s = slot[t], back = R - j, sp = p - back;
    int ti = -1;
    const float* q = nullptr;
    if (sp >= 0) {
      if (back == 0 || (t - back >= 0 && slot[t - back] == s)) ti = R + r - back;
      else q = state + ((long long)s * R + sp % R) * C;
    }
    src_tile[r][j] = ti;
    src_ring[r][j] = q;
  }
  for (int cl = threadIdx.x; cl < nc; cl += blockDim.x) {
    const int c = c0 + cl;
    const float w_n = ldf(nw + c), b_n = ldf(nb + c);
#pragma unroll 4
    for (int i = 0; i < nr + R; ++i) {
      const int t = t0 - R + i;
      float h = 0.f;
      if (t >= 0) {
        float xv = x[(long long)t * ldx + c];
        if (y1 != nullptr) xv = fmaf(a1, y1[(long long)t * ld1 + c], xv);
        if (y2 != nullptr) xv = fmaf(a2, y2[(long long)t * ld2 + c], xv);
        if (i >= R && x_out != nullptr) x_out[(long long)t * ldxo + c] = xv;
        h = fmaf(tanh_norm_f<FAST>(alpha * xv), w_n, b_n);
      }
      tile[i * ch_block + cl] = h;
    }
  }
  __syncthreads();   // a thread reads its own channel only, but the pointer table came from other threads
  for (int cl = threadIdx.x; cl < nc; cl += blockDim.x) {
    const int c = c0 + cl;
    float wreg[kDytRegTaps];
    if (taps <= kDytRegTaps) {
#pragma unroll
      for (int j = 0; j < kDytRegTaps; ++j) wreg[j] = j < taps ? ldf(cw + (long long)c * taps + j) : 0.f;
    }
    for (int r = 0; r < nr; ++r) {
      const float h = tile[(R + r) * ch_block + cl];
      float acc = h;
      if (taps <= kDytRegTaps) {
#pragma unroll
        for (int j = 0; j < kDytRegTaps; ++j) {
          if (j < taps) {
            const int ti = src_tile[r][j];
            const float* q = src_ring[r][j];
            if (ti >= 0) acc = fmaf(wreg[j], tile[ti * ch_block + cl], acc);
            else if (q != nullptr) acc = fmaf(wreg[j], q[c], acc);
          }
        }
      } else {
        for (int j = 0; j < taps; ++j) {
          const int ti = src_tile[r][j];
          const float* q = src_ring[r][j];
          const float wj = ldf(cw + (long long)c * taps + j);
          if (ti >= 0) acc = fmaf(wj, tile[ti * ch_block + cl], acc);
          else if (q != nullptr) acc = fmaf(wj, q[c], acc);
        }
      }
      stf(u + (long long)(t0 + r) * ldu + c, acc);
      // every row is a request of its own: nobody else reads this ring, and this thread's reads of channel c came first
      if (save_here && R > 0) state[((long long)slot[t0 + r] * R + pos[t0 + r] % R) * C + c] = h;
    }
  }
}

// The ring update of a step whose requests may have several rows: h of the last taps - 1 rows of every request, recomputed from the
// (already updated) stream rows.
template <bool FAST, typename TW>
__global__ void __launch_bounds__(256) dyt_state_save_kernel(const float* __restrict__ x, long long ldx, const float* __restrict__ alpha_p,
                                                             const TW* __restrict__ nw, const TW* __restrict__ nb, int C, int R, int T,
                                                             const int32_t* __restrict__ pos, const int32_t* __restrict__ slot,
                                                             float* __restrict__ state) {
  const int t = blockIdx.x;
  const int s = slot[t];
  if (t + R < T && slot[t + R] == s) return;
  const float alpha = *alpha_p;
  float* dst = state + ((long long)s * R + pos[t] % R) * C;
  for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < C; c += gridDim.y * blockDim.x) dst[c] = dyt_f<FAST>(x[(long long)t * ldx + c], alpha, nw, nb, c);
}

// ---- selective scan -------------------------------------------------------------------------------------------------------
// Per channel c a state S[c, :N] (fp32, in the request's slot):  S <- exp(dt_c A[c, :]) * S + dt_c x_c B_t;  y_c = S . C_t + D_c x_c,
// with dt = softplus(raw + bias) per channel and token, A = -exp(A_log), B_t / C_t shared by the channels; the output is gated,
// y * silu(z). Channels are independent: a CTA owns a block of channels of one request's portion, LANES neighbouring lanes share a
// channel (lane l holds the states l, l + LANES, ...), tokens go one after the other in chunks of kSelTok staged in shared memory.
// A portion whose first row has position 0 starts from S = 0.
constexpr int kSelTok = 16, kSelThreads = 128;

struct SelArgs {
  const void* x;
  long long ldx;
  const float* dt;
  long long lddt;
  const float* dt_bias;
  const float* B;
  long long ldb;
  const float* Cm;
  long long ldc;
  const float* A_log;
  const float* D;
  const float* z;
  long long ldz;
  float* state;
  void* y;
  long long ldy;
  const int32_t* row_begin;
  const int32_t* pos;
  const int32_t* slot;
  int inner, N;
};

// exp(x) - 1 for x <= 0 without losing the digits of a small x: a Taylor polynomial below 0.1 (truncation 1e-9 of x), the hardware
// exponential above, where its absolute error of ~1e-7 is small against the result and such a fast decay forgets within a few tokens.
__device__ __forceinline__ float expm1_decay_f(float x) {
  const float p = x * fmaf(x, fmaf(x, fmaf(x, fmaf(x, 1.f / 120.f, 1.f / 24.f), 1.f / 6.f), 0.5f), 1.f);
  const float e = exp2f(x * 1.4426950408889634f) - 1.f;
  return x > -0.1f ? p : e;
}

// LANES neighbouring lanes share a channel; lane l holds the states l, l + LANES, ... (P of them).
template <int LANES, int P, typename TD>
__global__ void __launch_bounds__(kSelThreads) selective_scan_kernel(SelArgs a) {
  constexpr int CH = kSelThreads / LANES;
  extern __shared__ float sm[];
  float* s_dt = sm;                          // [tok][CH]
  float* s_x = s_dt + kSelTok * CH;          // [tok][CH]
  float* s_y = s_x + kSelTok * CH;           // [tok][CH]
  float* s_B = s_y + kSelTok * CH;           // [tok][N]
  float* s_C = s_B + kSelTok * a.N;          // [tok][N]
  const int N = a.N, tid = threadIdx.x, lane = tid % LANES, cl = tid / LANES;
  const int c0 = blockIdx.x * CH, c = c0 + cl, ncl = min(CH, a.inner - c0);
  const bool live = c < a.inner;
  const int r0 = a.row_begin[blockIdx.y], r1 = a.row_begin[blockIdx.y + 1];
  if (r1 <= r0) return;
  const bool fresh = a.pos[r0] == 0;
  float* S = a.state + ((long long)a.slot[r0] * a.inner + (live ? c : 0)) * N;
  float st[P], A[P];
#pragma unroll
  for (int r = 0; r < P; ++r) {
    const int n = lane + r * LANES;
    const bool ok = live && n < N;
    st[r] = (ok && !fresh) ? S[n] : 0.f;
    A[r] = ok ? -expf(a.A_log[(long long)c * N + n]) : 0.f;
  }
  const float Dc = live ? a.D[c] : 0.f;
  const TD* xg = static_cast<const TD*>(a.x);
  TD* yg = static_cast<TD*>(a.y);
  for (int t0 = r0; t0 < r1; t0 += kSelTok) {
    const int n_tok = min(kSelTok, r1 - t0);
    for (int tt = tid / CH; tt < n_tok; tt += kSelThreads / CH) {
      const int j = tid % CH;
      if (j < ncl) {
        s_dt[tt * CH + j] = softplus_f(a.dt[(long long)(t0 + tt) * a.lddt + c0 + j] + a.dt_bias[c0 + j]);
        s_x[tt * CH + j] = ldf(xg + (long long)(t0 + tt) * a.ldx + c0 + j);
      }
    }
    for (int e = tid; e < n_tok * N; e += kSelThreads) {
      const int tt = e / N, n = e - tt * N;
      s_B[e] = a.B[(long long)(t0 + tt) * a.ldb + n];
      s_C[e] = a.Cm[(long long)(t0 + tt) * a.ldc + n];
    }
    __syncthreads();
    for (int tt = 0; tt < n_tok; ++tt) {
      const float dt = s_dt[tt * CH + cl], xv = s_x[tt * CH + cl], dx = dt * xv;
      const float* Bt = s_B + tt * N;
      const float* Ct = s_C + tt * N;
      float y = 0.f;
#pragma unroll
      for (int r = 0; r < P; ++r) {
        const int n = lane + r * LANES;
        if (n < N) {
          // the decay as S + (exp(dt A) - 1) S: a decay close to 1 would lose most of the digits of 1 - decay when rounded to
          // fp32 itself, and that error grows with every token the state remembers
          st[r] = fmaf(expm1_decay_f(dt * A[r]), st[r], st[r]) + dx * Bt[n];
          y = fmaf(st[r], Ct[n], y);
        }
      }
#pragma unroll
      for (int m = 1; m < LANES; m <<= 1) y += __shfl_xor_sync(0xffffffffu, y, m);
      if (lane == 0) s_y[tt * CH + cl] = fmaf(Dc, xv, y);
    }
    __syncthreads();
    for (int tt = tid / CH; tt < n_tok; tt += kSelThreads / CH) {
      const int j = tid % CH;
      if (j < ncl) {
        float y = s_y[tt * CH + j];
        if (a.z != nullptr) y *= silu_f(a.z[(long long)(t0 + tt) * a.ldz + c0 + j]);
        stf(yg + (long long)(t0 + tt) * a.ldy + c0 + j, y);
      }
    }
    // the next chunk's staging writes s_dt / s_x / s_B / s_C, which nobody reads any more; s_y is rewritten only after the next barrier
  }
  if (live) {
#pragma unroll
    for (int r = 0; r < P; ++r) {
      const int n = lane + r * LANES;
      if (n < N) S[n] = st[r];
    }
  }
}

// ---- real-gated linear recurrent unit -------------------------------------------------------------------------------------
// Per channel one state:  S <- a S + sqrt(1 - a^2) i u,  log a = -k r softplus(lam),  r and i sigmoids of raw gates that a block-
// diagonal product left in g. Nothing couples the channels, and the recurrence is linear in S: a CTA owns blockDim.x channels of one
// portion and blockDim.y consecutive runs of K tokens. Every thread evaluates its K tokens' (expm1(log a), input) in registers, runs
// them from a zero state, and leaves (sum of log a, local state) of its run in shared memory; with the runs in front of its own it
// gets its start state and goes over its K tokens once more from registers. A run's whole decay is applied as expm1 of the summed
// log a - never as a product of rounded decays - so the state keeps its digits however the tokens are spread over threads. The output
// is multiplied by gelu of the other branch. FAST (bf16 operands): hardware exponential, reciprocal and square root.
constexpr int kLruTok = 4, kLruSms = 148;

struct LruArgs {
  const void* u;
  int ldu;
  const float* g;
  int ldg;
  const float* gb;
  const float* lam;
  const float* y;
  int ldy;
  float* state;
  void* out;
  int ldo;
  const int32_t* row_begin;
  const int32_t* pos;
  const int32_t* slot;
  int width, n;   // n: channels per gate block
  float scale;
};

__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
template <bool FAST>
__device__ __forceinline__ float lru_sigmoid(float z) {
  return FAST ? rcp_approx(1.f + ex2_approx(-1.4426950408889634f * z)) : sigmoid_f(z);
}
template <bool FAST>
__device__ __forceinline__ float lru_sqrt(float z) {
  if (!FAST) return sqrtf(z);
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(z));
  return r;
}
// gelu in its tanh form: 0.5 z (1 + tanh(p)) = z sigmoid(2 p)
template <bool FAST>
__device__ __forceinline__ float lru_gelu(float z) {
  const float p = 0.7978845608028654f * fmaf(0.044715f * z * z, z, z);
  return FAST ? z * lru_sigmoid<true>(2.f * p) : 0.5f * z * (1.f + tanhf(p));
}
// exp(x) - 1 for x <= 0 (FAST: expm1_decay_f with the hardware exponential as it is)
template <bool FAST>
__device__ __forceinline__ float lru_expm1(float x) {
  if (!FAST) return expm1f(x);
  const float p = x * fmaf(x, fmaf(x, fmaf(x, fmaf(x, 1.f / 120.f, 1.f / 24.f), 1.f / 6.f), 0.5f), 1.f);
  const float e = ex2_approx(x * 1.4426950408889634f) - 1.f;
  return x > -0.1f ? p : e;
}

template <typename TD, bool FAST, int K>
__global__ void __launch_bounds__(512) rglru_scan_kernel(LruArgs a) {
  extern __shared__ float2 s_run[];  // [2][blockDim.y][blockDim.x]: (expm1 of the run's summed log a, its state from zero)
  const int cx = threadIdx.x, wy = threadIdx.y, CX = blockDim.x, W = blockDim.y;
  const int c = blockIdx.x * CX + cx;
  const bool live = c < a.width;
  const int r0 = a.row_begin[blockIdx.y], r1 = a.row_begin[blockIdx.y + 1];
  if (r1 <= r0) return;
  const int end = live ? r1 : r0, last = r1 - 1;   // channels past the last read channel 0 and take part in the barriers only
  const bool fresh = a.pos[r0] == 0;
  float* Sp = a.state + (long long)a.slot[r0] * a.width + c;
  float carry = (live && !fresh) ? *Sp : 0.f;
  const int blk = live ? c / a.n : 0, gr = blk * 2 * a.n + (live ? c - blk * a.n : 0);
  const float sp = live ? -a.scale * softplus_f(a.lam[c]) : 0.f;
  const float br = (live && a.gb != nullptr) ? a.gb[gr] : 0.f, bi = (live && a.gb != nullptr) ? a.gb[gr + a.n] : 0.f;
  const TD* ug = static_cast<const TD*>(a.u) + (long long)r0 * a.ldu + (live ? c : 0);
  const float* pr = a.g + (long long)r0 * a.ldg + gr;
  const float* pi = pr + a.n;
  const float* yg = a.y != nullptr ? a.y + (long long)r0 * a.ldy + (live ? c : 0) : nullptr;
  TD* og = static_cast<TD*>(a.out) + (long long)r0 * a.ldo + c;
  float zr[K], zi[K], uv[K], yv[K];   // the raw inputs of this thread's next run
  auto load = [&](int tb) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int t = min(tb + k, last) - r0;   // past the end: read the last row, whose copy contributes nothing below
      zr[k] = pr[(long long)t * a.ldg];
      zi[k] = pi[(long long)t * a.ldg];
      uv[k] = ldf(ug + (long long)t * a.ldu);
      yv[k] = yg != nullptr ? yg[(long long)t * a.ldy] : 0.f;
    }
  };
  load(r0 + wy * K);
  int buf = 0;
  for (int t0 = r0; t0 < r1; t0 += W * K, buf ^= 1) {
    const int tb = t0 + wy * K;
    float am1[K], in[K], yc[K];
    float L = 0.f, loc = 0.f;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const float la = tb + k < end ? sp * lru_sigmoid<FAST>(zr[k] + br) : 0.f;   // past the end: a = 1 and no input
      am1[k] = lru_expm1<FAST>(la);
      in[k] = lru_sqrt<FAST>(-am1[k] * (2.f + am1[k])) * (lru_sigmoid<FAST>(zi[k] + bi) * uv[k]);
      yc[k] = yv[k];
      L += la;
      loc = fmaf(am1[k], loc, loc) + in[k];
    }
    load(tb + W * K);   // on its way during the rest of this tile
    float S = carry;
    if (W > 1) {
      float2* run = s_run + (size_t)buf * W * CX;
      run[wy * CX + cx] = make_float2(lru_expm1<FAST>(L), loc);
      __syncthreads();   // the other buffer is rewritten only behind the next tile's barrier, which every reader of this one reaches first
      for (int w = 0; w < W; ++w) {
        if (w == wy) S = carry;
        const float2 v = run[w * CX + cx];
        carry = fmaf(v.x, carry, carry) + v.y;
      }
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (tb + k < end) {
        S = fmaf(am1[k], S, S) + in[k];
        stf(og + (long long)(tb + k - r0) * a.ldo, yg != nullptr ? S * lru_gelu<FAST>(yc[k]) : S);
      }
    }
    if (W == 1) carry = S;
  }
  if (live && wy == 0) *Sp = carry;
}

}  // namespace omc

using namespace omc;

extern "C" int omc_causal_conv(const float* x, long long ldx, int T, int ch, const void* w, const void* bias, int w_dt, int taps,
                               const int32_t* pos, const int32_t* slot, float* state, void* y, int y_dt, long long ldy, int act,
                               int unit_channels, int unit_group, float unit_eps, int scaled_channels, float unit_mult,
                               int single_rows, void* stream) {
  if (x == nullptr || w == nullptr || pos == nullptr || slot == nullptr || y == nullptr || T < 0 || ch <= 0 || taps < 1 || taps > kConvMaxTaps ||
      (taps > 1 && state == nullptr) || (act != OMC_CONV_LINEAR && act != OMC_CONV_SILU) || unit_channels < 0 || unit_channels > ch || (unit_channels > 0 && (unit_group <= 0 || unit_channels % unit_group)) ||
      (unit_channels > 0 && scaled_channels % unit_group))
    return set_error(OMC_ERR_ARG, "omc_causal_conv: bad argument");
  if (T == 0) return OMC_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // unit vectors of 4, 8, ... 128 channels lie in neighbouring lanes of one warp
  const bool unit = unit_channels > 0, unit_in_warp = unit && unit_group >= 4 && unit_group <= 128 && (unit_group & (unit_group - 1)) == 0 && ch % 128 == 0;
  const bool rows4 = (!unit || unit_in_warp) && taps <= 4 && ch % 4 == 0 && ldx % 4 == 0 && ldy % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0 &&
                     reinterpret_cast<uintptr_t>(y) % 16 == 0 && (state == nullptr || reinterpret_cast<uintptr_t>(state) % 16 == 0);
  if (rows4) {
    const int b4 = (ch / 4 + 127) / 128;
    if (b4 > 65535) return set_error(OMC_ERR_SHAPE, "omc_causal_conv: too many channel blocks");
    OMC_DT_SWITCH(w_dt, TW, OMC_DT_SWITCH(y_dt, TY, {
      const ConvUnit cu{unit_channels, unit ? unit_group / 4 : 0, scaled_channels, unit_eps, unit_mult};
      auto launch = [&](auto kernel, int rows) {
        kernel<<<dim3((T + rows - 1) / rows, b4), 128, 0, st>>>(x, ldx, T, ch, static_cast<const TW*>(w), static_cast<const TW*>(bias), pos, slot, state,
                                                              static_cast<TY*>(y), ldy, single_rows ? 1 : 0, act == OMC_CONV_SILU ? 1 : 0, cu,
                                                              reinterpret_cast<uintptr_t>(w) % 16 == 0);
      };
      auto go = [&](auto taps_c) {
        // four rows keep more warps on an SM than eight, whose thread reads its weights less often: with weights of 16 bits 38 and 39 us, of 32 bits 38 and 35 (3126 x 6144)
        constexpr int TAPS = decltype(taps_c)::value, ROWS = sizeof(TW) == 2 ? 4 : 8;
        if (T >= 256 && unit) launch(causal_conv_rows_kernel<TW, TY, TAPS, ROWS, true>, ROWS);
        else if (T >= 256) launch(causal_conv_rows_kernel<TW, TY, TAPS, ROWS, false>, ROWS);
        else if (unit) launch(causal_conv_rows_kernel<TW, TY, TAPS, 1, true>, 1);
        else launch(causal_conv_rows_kernel<TW, TY, TAPS, 1, false>, 1);
      };
      if (taps == 1) go(std::integral_constant<int, 1>());
      else if (taps == 2) go(std::integral_constant<int, 2>());
      else if (taps == 3) go(std::integral_constant<int, 3>());
      else go(std::integral_constant<int, 4>());
    }))
    if (taps > 1 && !single_rows) save_conv_state(x, ldx, ch, taps - 1, T, pos, slot, state, st);
    return check_launch("omc_causal_conv");
  }
  // channel blocks of about 512 channels, whole unit-vector groups each
  int ch_block = 512;
  if (unit_channels > 0) ch_block = unit_group >= 512 ? unit_group : (512 / unit_group) * unit_group;
  if (ch_block > ch) ch_block = ch;
  if ((size_t)ch_block * kConvRows * sizeof(float) > 200 * 1024) return set_error(OMC_ERR_SHAPE, "omc_causal_conv: unit-vector group too wide for shared memory");
  const int blocks = (ch + ch_block - 1) / ch_block;
  if (blocks > 65535) return set_error(OMC_ERR_SHAPE, "omc_causal_conv: too many channel blocks");
  const int rows_per_cta = T >= 256 ? kConvRows : 1;   // short steps (decode) keep one CTA per row: there are few rows to share anything
  const size_t smem = (size_t)ch_block * rows_per_cta * sizeof(float);
  OMC_DT_SWITCH(w_dt, TW, OMC_DT_SWITCH(y_dt, TY, {
    if (smem > 48 * 1024) cudaFuncSetAttribute(causal_conv_silu_kernel<TW, TY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    causal_conv_silu_kernel<TW, TY><<<dim3((T + rows_per_cta - 1) / rows_per_cta, blocks), 256, smem, st>>>(
        x, ldx, T, ch, ch_block, rows_per_cta, static_cast<const TW*>(w), static_cast<const TW*>(bias), taps, pos, slot, state,
        static_cast<TY*>(y), ldy, unit_channels, unit_group, unit_eps, scaled_channels, unit_mult, single_rows ? 1 : 0, act == OMC_CONV_SILU ? 1 : 0);
  }))
  if (taps > 1 && !single_rows) save_conv_state(x, ldx, ch, taps - 1, T, pos, slot, state, st);
  return check_launch("omc_causal_conv");
}

extern "C" int omc_conv_qk_norm_kv_store(const float* x, long long ldx, int T, int ch, const void* w, int w_dt, int taps, const int32_t* pos,
                                         const int32_t* slot, float* state, int nq, int nk, int group, const void* wq, const void* wk,
                                         float eps, const int32_t* block_table, int max_pages, int page_size, void* pool, void* q_out,
                                         long long ldqo, int dt, int single_rows, void* stream) {
  if (x == nullptr || w == nullptr || pos == nullptr || slot == nullptr || wq == nullptr || wk == nullptr || block_table == nullptr ||
      pool == nullptr || q_out == nullptr || T < 0 || taps < 1 || taps > kConvMaxTaps || (taps > 1 && state == nullptr) || group <= 0 ||
      nq <= 0 || nk <= 0 || nq % group || nk % group || ch <= nq + nk || page_size <= 0 || max_pages <= 0)
    return set_error(OMC_ERR_ARG, "omc_conv_qk_norm_kv_store: bad argument");
  if (T == 0) return OMC_OK;
  int ch_block = group >= 512 ? group : (512 / group) * group;
  if (ch_block > ch) ch_block = ch;
  if ((size_t)ch_block * kConvRows * sizeof(float) > 200 * 1024) return set_error(OMC_ERR_SHAPE, "omc_conv_qk_norm_kv_store: group too wide for shared memory");
  const int blocks = (ch + ch_block - 1) / ch_block;
  if (blocks > 65535) return set_error(OMC_ERR_SHAPE, "omc_conv_qk_norm_kv_store: too many channel blocks");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int rows_per_cta = T >= 256 ? kConvRows : 1;
  const size_t smem = (size_t)ch_block * rows_per_cta * sizeof(float);
  OMC_DT_SWITCH(w_dt, TW, OMC_DT_SWITCH(dt, TC, {
    if (smem > 48 * 1024) cudaFuncSetAttribute(conv_qk_norm_store_kernel<TW, TC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    conv_qk_norm_store_kernel<TW, TC><<<dim3((T + rows_per_cta - 1) / rows_per_cta, blocks), 256, smem, st>>>(
        x, ldx, T, ch, ch_block, rows_per_cta, static_cast<const TW*>(w), taps, pos, slot, state, nq, nk, group, static_cast<const TW*>(wq),
        static_cast<const TW*>(wk), eps, block_table, max_pages, page_size, static_cast<TC*>(pool), static_cast<TC*>(q_out), ldqo,
        single_rows ? 1 : 0);
  }))
  if (taps > 1 && !single_rows) save_conv_state(x, ldx, ch, taps - 1, T, pos, slot, state, st);
  return check_launch("omc_conv_qk_norm_kv_store");
}

extern "C" int omc_causal_conv_silu(const float* x, long long ldx, int T, int ch, const void* w, int w_dt, int taps,
                                    const int32_t* pos, const int32_t* slot, float* state, float* y, long long ldy,
                                    int unit_channels, int unit_group, float unit_eps, int scaled_channels, float unit_mult,
                                    int single_rows, void* stream) {
  return omc_causal_conv(x, ldx, T, ch, w, nullptr, w_dt, taps, pos, slot, state, y, OMC_DT_F32, ldy, OMC_CONV_SILU, unit_channels, unit_group,
                         unit_eps, scaled_channels, unit_mult, single_rows, stream);
}

extern "C" int omc_linear_state_scan(const float* q, long long ldq, const float* k, long long ldk, const float* v, long long ldv,
                                     int silu_in, int decay_mode, const float* decay_const, const float* a, long long lda,
                                     const float* A_log, const float* dt_bias, const float* D, const float* beta, long long ldb, float* state,
                                     float* out, long long ldo, const int32_t* row_begin, int portions, const int32_t* pos,
                                     const int32_t* slot, int rows, int H, int G, int dim, int vdim, float decay_pow, float out_scale, void* stream) {
  return omc_linear_state_scan_longest(q, ldq, k, ldk, v, ldv, silu_in, decay_mode, decay_const, a, lda, A_log, dt_bias, D, beta, ldb, state, out, ldo, row_begin, portions, pos,
                                       slot, rows, rows, H, G, dim, vdim, decay_pow, out_scale, stream);
}

extern "C" int omc_linear_state_scan_longest(const float* q, long long ldq, const float* k, long long ldk, const float* v, long long ldv,
                                             int silu_in, int decay_mode, const float* decay_const, const float* a, long long lda,
                                             const float* A_log, const float* dt_bias, const float* D, const float* beta, long long ldb, float* state,
                                             float* out, long long ldo, const int32_t* row_begin, int portions, const int32_t* pos, const int32_t* slot, int rows, int longest,
                                             int H, int G, int dim, int vdim, float decay_pow, float out_scale, void* stream) {
  if (q == nullptr || k == nullptr || v == nullptr || state == nullptr || out == nullptr || row_begin == nullptr || pos == nullptr ||
      slot == nullptr || portions < 0 || H <= 0 || G <= 0 || H % G || dim <= 0 || vdim <= 0 || decay_mode < 0 || decay_mode > 6 ||
      (decay_mode == 0 && decay_const == nullptr) || (decay_mode != 0 && a == nullptr) || (decay_mode == 6 && beta != nullptr) || (D != nullptr && decay_mode != 6) ||
      ((decay_mode == 1 || decay_mode == 2 || decay_mode == 6) && (A_log == nullptr || dt_bias == nullptr)))
    return set_error(OMC_ERR_ARG, "omc_linear_state_scan: bad argument");
  if (portions == 0) return OMC_OK;
  if (dim > 256) return set_error(OMC_ERR_SHAPE, "omc_linear_state_scan: key width above 256");
  if (portions > 65535 || H > 65535) return set_error(OMC_ERR_SHAPE, "omc_linear_state_scan: more than 65535 portions or heads");
  ScanArgs s{q, k, v, ldq, ldk, ldv, silu_in, decay_mode, decay_pow, out_scale, decay_const, a, lda, A_log, dt_bias, D, beta, ldb, state, out, ldo,
             row_begin, pos, slot, H, G, dim, vdim, false, false, 0, 0, rows, portions, 0};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int dpt = dim <= 32 ? 4 : (dim <= 64 ? 8 : (dim <= 128 ? 16 : 32));   // key channels per thread: dim / 8 lanes, rounded up to a float4
  const bool chan = decay_mode >= 2 && decay_mode <= 5;
  auto al16 = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  const bool vec = dim % 4 == 0 && vdim % 4 == 0 && ldq % 4 == 0 && ldk % 4 == 0 && ldv % 4 == 0 && al16(q) && al16(k) && al16(v) &&
                   (!chan || (lda % 4 == 0 && al16(a)));
  const bool one = vec && rows <= portions;   // every portion is one token
  s.vec_state = vdim % kScanCpt == 0 && al16(state);
  s.vec_out = vdim % 4 == 0 && ldo % 4 == 0 && al16(out);
  constexpr int cols = kScanGroups * kScanCpt;
  dim3 grid((vdim + cols - 1) / cols, H, portions);
  // 16 tokens per stage; with per-channel decays that is 85 KB and two CTAs per SM, so beyond 296 CTAs eight tokens (in us, 16 / 8 tokens,
  // 32 heads of 128 x 128, portions of 1024, 777, 1024, 301: 713 / 608; 16 heads: 435 / 476). Portions of few tokens have no use for 16, whose 63 KB
  // (39 at 32 channels) leave three CTAs to an SM: eight portions of three tokens, 16 heads of 128 x 128, 15.4 / 10.3
  const bool tight = chan && (long long)grid.x * H * portions > 296;
  const bool brief = rows <= 16LL * portions;
  // portions of several tokens whose inputs are ready: scan_rows_kernel
  const bool ready = !silu_in && (decay_mode == 0 || decay_mode == 1 || decay_mode == 3 || decay_mode >= 5);
  const bool several = !one && vec && ready && (dim == 64 || dim == 128) && s.vec_out && s.vec_state;
  auto tokens = [&]() -> int {   // token by token
    if (several) {
      // chains of hundreds of tokens, more CTAs than SMs: the longest portions first (32 heads of 128 x 64, portions of 1024, 777, 1024, 301 tokens: 197, in their own order 224)
      if (portions > 1 && portions <= kSrThreads && rows >= 128LL * portions && (long long)grid.x * H * portions > 148) s.portions = portions;
      auto go = [&](auto dim_c, auto cpt_c, auto kind_c, auto chan_c) {
        constexpr int DIM = decltype(dim_c)::value, CPT = decltype(cpt_c)::value, KIND = decltype(kind_c)::value, COLS = kSrThreads / kScanLanes * CPT;
        constexpr bool CHAN = decltype(chan_c)::value;
        static bool attr_done[kMaxDevices] = {};
        constexpr int smem = (int)sizeof(ScanRowsShared<DIM, COLS, CHAN>);
        if (!attr_done[cur_device()]) {
          cudaFuncSetAttribute(scan_rows_kernel<DIM, CPT, KIND, CHAN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
          attr_done[cur_device()] = true;
        }
        return scan_launch(scan_rows_kernel<DIM, CPT, KIND, CHAN>, dim3((vdim + COLS - 1) / COLS, H, portions), kSrThreads, smem, st, s);
      };
      using std::integral_constant;
      auto kinds = [&](auto dim_c, auto cpt_c) {
        if (decay_mode == 6) return go(dim_c, cpt_c, integral_constant<int, kScanStep>(), std::false_type());
        if (beta != nullptr) return go(dim_c, cpt_c, integral_constant<int, kScanDelta>(), std::false_type());
        return go(dim_c, cpt_c, integral_constant<int, kScanPlain>(), std::false_type());
      };
      auto channels = [&](auto dim_c) {
        typedef integral_constant<int, 1> One;
        if (beta != nullptr) return go(dim_c, One(), integral_constant<int, kScanDelta>(), std::true_type());
        return go(dim_c, One(), integral_constant<int, kScanPlain>(), std::true_type());
      };
      // 32 columns per CTA once CTAs of 16 would be more than the SMs: alone on an SM the smaller CTA is the faster one (in us, 16 / 32 columns: 16 heads of 128 x
      // 64, step sizes, 1100 tokens 149 / 162; delta rule 4 of 128 x 128 255 / 269, 4 of 64 x 64 195 / 213), two of them on it never (64 heads 230 / 163).
      // Per-channel decays take the registers of the larger one: there the general kernel is up to 12 % faster
      const bool small = (long long)grid.x * H * portions <= 74;
      typedef integral_constant<int, 1> One;
      typedef integral_constant<int, 2> Two;
      if (chan && small)
        return dim == 64 ? channels(integral_constant<int, 64>()) : channels(integral_constant<int, 128>());
      // 64 columns per CTA, four per thread, where such CTAs are many: half the shared-memory reads per column, which bound it then, but longer chains of a token, which do where
      // CTAs are few (in us, 32 / 64 columns: 64 heads of 128 x 64, 4 x 700 tokens 267 / 235, 32 x 64 184 / 154, 3 x 500 150 / 169; 80 heads, 3 x 600 230 / 203; 128 heads,
      // 8 x 400 517 / 427). Not where the last half of the columns would be empty (96: 181 / 205)
      const int blocks = (vdim + 63) / 64;
      if (!chan && beta == nullptr && (vdim + 31) / 32 == 2 * blocks && (long long)blocks * H * portions >= 240) {
        typedef integral_constant<int, 4> Four;
        auto plain = [&](auto dim_c) {
          if (decay_mode == 6) return go(dim_c, Four(), integral_constant<int, kScanStep>(), std::false_type());
          return go(dim_c, Four(), integral_constant<int, kScanPlain>(), std::false_type());
        };
        return dim == 64 ? plain(integral_constant<int, 64>()) : plain(integral_constant<int, 128>());
      }
      if (!chan && dim == 64) return small ? kinds(integral_constant<int, 64>(), One()) : kinds(integral_constant<int, 64>(), Two());
      if (!chan) return small ? kinds(integral_constant<int, 128>(), One()) : kinds(integral_constant<int, 128>(), Two());
    }
#define OMC_SCAN_LAUNCH(DPT, VEC, KIND, CHAN, TOK)                                                                                        \
  do {                                                                                                                                    \
    static bool attr_done[kMaxDevices] = {};                                                                                              \
    constexpr int smem = 4 * (2 * scan_stage_floats<DPT, TOK>(CHAN, cols) + TOK * kScanLanes * (cols + 4));                                \
    if (!attr_done[cur_device()]) {                                                                                                       \
      cudaFuncSetAttribute(linear_state_scan_kernel<DPT, VEC, KIND, CHAN, TOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);       \
      attr_done[cur_device()] = true;                                                                                                     \
    }                                                                                                                                     \
    return scan_launch(linear_state_scan_kernel<DPT, VEC, KIND, CHAN, TOK>, grid, kScanThreads, smem, st, s);                              \
  } while (0)
#define OMC_SCAN_KIND(DPT, VEC, TOK)                                                      \
  do {                                                                                    \
    if (decay_mode == 6) OMC_SCAN_LAUNCH(DPT, VEC, kScanStep, false, TOK);                \
    else if (beta != nullptr && chan) OMC_SCAN_LAUNCH(DPT, VEC, kScanDelta, true, TOK);   \
    else if (beta != nullptr) OMC_SCAN_LAUNCH(DPT, VEC, kScanDelta, false, TOK);          \
    else if (chan) OMC_SCAN_LAUNCH(DPT, VEC, kScanPlain, true, TOK);                      \
    else OMC_SCAN_LAUNCH(DPT, VEC, kScanPlain, false, TOK);                               \
  } while (0)
#define OMC_SCAN_DPT(DPT, TOK)                  \
  do {                                          \
    if (one) OMC_SCAN_KIND(DPT, true, 1);       \
    else if (vec) OMC_SCAN_KIND(DPT, true, TOK); \
    else OMC_SCAN_KIND(DPT, false, TOK);        \
  } while (0)
    if (dpt == 4 && brief) OMC_SCAN_DPT(4, 8);
    else if (dpt == 4) OMC_SCAN_DPT(4, 16);
    else if (dpt == 8 && brief) OMC_SCAN_DPT(8, 8);
    else if (dpt == 8) OMC_SCAN_DPT(8, 16);
    else if (dpt == 16 && (tight || brief)) OMC_SCAN_DPT(16, 8);
    else if (dpt == 16) OMC_SCAN_DPT(16, 16);
    else OMC_SCAN_DPT(32, 8);
#undef OMC_SCAN_DPT
#undef OMC_SCAN_KIND
#undef OMC_SCAN_LAUNCH
  };
  // long portions of the delta rule and with per-channel decays: scan_chunk_kernel; whichever are left, the kernels above. Not decays that are the same in every token: the error of
  // a product of eight of them, always the same too, would add up from stage to stage (1.0 to 1.25 of token by token after 1000 tokens)
  // (every portion has a row at least, so that none can have more than what is left)
  const int long_from = chan ? kScanLongChannel : kScanLongHead;
  if (!several || longest < long_from || rows - portions + 1 < long_from || !(chan || (beta != nullptr && decay_mode == 1))) return tokens();
  if (portions == 1) {   // alone: what row_begin has is this kernel's, however few rows (a padded buffer)
    s.long_from = 1, s.rows = 0x7fffffff;
    return launch_scan_chunk(s, rows, portions, st);
  }
  if (portions == 65535) return tokens();   // no room in the grid for the layer that waits
  s.long_from = long_from;
  // The long chains first, the others beside them. In us, all token by token / one kernel behind the other / beside: 500 + 16 x 1 tokens of 16 heads of 128 x 128 131 / 97 / 90, with
  // decays per channel 195 / 113 / 101 (152 with the short ones first); 65 + 31 x 1 tokens 29 / 36 / 25; 100, 50, 50, 50 33 / 46 / 31. Where no portion is
  // long the first kernel is empty and costs 1.2 on the device (8 x 8 tokens 9.3 / 10.5), so the host says how long they are at most.
  s.beside = 1;
  if (const int rc = launch_scan_chunk(s, rows, portions, st); rc != OMC_OK) return rc;
  s.beside = 2;
  return tokens();
}

extern "C" int omc_gated_rms_rows(const float* x, long long ldx, int rows, int groups, int n, const void* w, int w_dt, float eps,
                                  const float* gate, long long ldg, int gate_act, void* y, int y_dt, long long ldy, void* stream) {
  if (x == nullptr || w == nullptr || y == nullptr || rows < 0 || groups <= 0 || n <= 0 || gate_act < 0 || gate_act > 2)
    return set_error(OMC_ERR_ARG, "omc_gated_rms_rows: bad argument");
  if (rows == 0) return OMC_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int gy = groups > 8 ? (groups + 7) / 8 : 1;
  OMC_DT_SWITCH(w_dt, TW, OMC_DT_SWITCH(y_dt, TY, {
    if (group_rms<false>(x, ldx, rows, groups, n, static_cast<const TW*>(w), eps, gate, ldg, gate_act, static_cast<TY*>(y), ldy, st)) return check_launch("omc_gated_rms_rows");
    gated_rms_kernel<TW, TY><<<dim3(rows, gy > 65535 ? 65535 : gy), 256, 0, st>>>(x, ldx, groups, n, static_cast<const TW*>(w), eps,
                                                                                 gate, ldg, gate_act, static_cast<TY*>(y), ldy);
  }))
  return check_launch("omc_gated_rms_rows");
}

extern "C" int omc_gate_rms_rows(const float* x, long long ldx, int rows, int groups, int n, const void* w, int w_dt, float eps, const void* gate,
                                 int gate_dt, long long ldg, int gate_act, void* y, int y_dt, long long ldy, void* stream) {
  if (x == nullptr || w == nullptr || gate == nullptr || y == nullptr || rows < 0 || groups <= 0 || n <= 0 || gate_act < 0 || gate_act > 2)
    return set_error(OMC_ERR_ARG, "omc_gate_rms_rows: bad argument");
  if (groups > 65535) return set_error(OMC_ERR_SHAPE, "omc_gate_rms_rows: more than 65535 parts");
  if (rows == 0) return OMC_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto al = [](const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; };
  const bool vec = n % 4 == 0 && ldx % 4 == 0 && ldg % 4 == 0 && ldy % 4 == 0 && al(x) && al(gate) && al(y) && al(w);
  const int per = vec ? 4 : 1;
  int threads = 32;   // about one or two pieces per thread up to 256 threads
  while (threads < 256 && threads * per * 2 < n) threads <<= 1;
  const dim3 grid(rows, groups);
  OMC_DT_SWITCH(gate_dt, TG, OMC_DT_SWITCH(w_dt, TW, OMC_DT_SWITCH(y_dt, TY, {
    if (group_rms<true>(x, ldx, rows, groups, n, static_cast<const TW*>(w), eps, static_cast<const TG*>(gate), ldg, gate_act, static_cast<TY*>(y), ldy, st))
      return check_launch("omc_gate_rms_rows");
    if (vec) gate_rms_kernel<TG, TW, TY, true><<<grid, threads, 0, st>>>(x, ldx, n, static_cast<const TW*>(w), eps, static_cast<const TG*>(gate), ldg, gate_act,
                                                                         static_cast<TY*>(y), ldy);
    else gate_rms_kernel<TG, TW, TY, false><<<grid, threads, 0, st>>>(x, ldx, n, static_cast<const TW*>(w), eps, static_cast<const TG*>(gate), ldg, gate_act,
                                                                      static_cast<TY*>(y), ldy);
  })))
  return check_launch("omc_gate_rms_rows");
}

extern "C" int omc_map_rows(float* x, long long ldx, int rows, int cols, int op, const float* A_log, const float* bias, int group,
                            float p_exp, void* stream) {
  if (x == nullptr || rows < 0 || cols <= 0 || op < 1 || op > 3 || (op == 2 && (A_log == nullptr || bias == nullptr || group <= 0)))
    return set_error(OMC_ERR_ARG, "omc_map_rows: bad argument");
  if (rows == 0) return OMC_OK;
  const long long total = (long long)rows * cols;
  map_rows_kernel<<<(unsigned)((total + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(x, ldx, cols, total, op, A_log, bias, group, p_exp);
  return check_launch("omc_map_rows");
}

extern "C" int omc_dyt_conv(const float* x, long long ldx, const float* y1, long long ld1, float a1, const float* y2, long long ld2, float a2,
                            float* x_out, long long ldxo, const float* alpha, const void* nw, const void* nb, const void* cw, int w_dt,
                            int taps, const int32_t* pos, const int32_t* slot, float* state, void* u, int u_dt, long long ldu, int T, int C,
                            int single_rows, void* stream) {
  if (x == nullptr || alpha == nullptr || nw == nullptr || nb == nullptr || cw == nullptr || pos == nullptr || slot == nullptr || u == nullptr ||
      T < 0 || C <= 0 || taps < 1 || taps > kConvMaxTaps || (taps > 1 && state == nullptr) || ((y1 != nullptr || y2 != nullptr) && x_out == nullptr) ||
      (x_out == x && (y1 != nullptr || y2 != nullptr)))
    return set_error(OMC_ERR_ARG, "omc_dyt_conv: bad argument");
  if (T == 0) return OMC_OK;
  const int ch_block = C < 512 ? C : 512;
  const int blocks = (C + ch_block - 1) / ch_block;
  if (blocks > 65535) return set_error(OMC_ERR_SHAPE, "omc_dyt_conv: too many channel blocks");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int rows_per_cta = T >= 256 ? kDytRows : 1;
  const size_t smem = (size_t)ch_block * (rows_per_cta + taps - 1) * sizeof(float);
  const float* xs = (y1 != nullptr || y2 != nullptr) ? x_out : x;   // where the save kernel finds the updated stream
  const long long ldxs = (y1 != nullptr || y2 != nullptr) ? ldxo : ldx;
  OMC_DT_SWITCH(w_dt, TW, OMC_DT_SWITCH(u_dt, TU, {
    if (smem > 48 * 1024) cudaFuncSetAttribute(dyt_conv_kernel<TW, TU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    dyt_conv_kernel<TW, TU><<<dim3((T + rows_per_cta - 1) / rows_per_cta, blocks), 256, smem, st>>>(
        x, ldx, y1, ld1, a1, y2, ld2, a2, x_out, ldxo, alpha, static_cast<const TW*>(nw), static_cast<const TW*>(nb), static_cast<const TW*>(cw),
        taps, pos, slot, state, static_cast<TU*>(u), ldu, T, C, ch_block, rows_per_cta, single_rows ? 1 : 0);
    if (taps > 1 && !single_rows)
      dyt_state_save_kernel<is_bf16_t<TU>::value, TW><<<dim3(T, (C + 1023) / 1024), 256, 0, st>>>(xs, ldxs, alpha, static_cast<const TW*>(nw), static_cast<const TW*>(nb), C,
                                                                           taps - 1, T, pos, slot, state);
  }))
  return check_launch("omc_dyt_conv");
}

extern "C" int omc_selective_scan(const void* x, int x_dt, long long ldx, const float* dt, long long lddt, const float* dt_bias, const float* B,
                                  long long ldb, const float* Cm, long long ldc, const float* A_log, const float* D, const float* z, long long ldz,
                                  float* state, void* y, int y_dt, long long ldy, const int32_t* row_begin, int portions, const int32_t* pos,
                                  const int32_t* slot, int inner, int N, void* stream) {
  if (x == nullptr || dt == nullptr || dt_bias == nullptr || B == nullptr || Cm == nullptr || A_log == nullptr || D == nullptr || state == nullptr ||
      y == nullptr || row_begin == nullptr || pos == nullptr || slot == nullptr || portions < 0 || inner <= 0 || N <= 0)
    return set_error(OMC_ERR_ARG, "omc_selective_scan: bad argument");
  if (portions == 0) return OMC_OK;
  if (N > 256) return set_error(OMC_ERR_SHAPE, "omc_selective_scan: more than 256 states per channel");
  if (portions > 65535) return set_error(OMC_ERR_SHAPE, "omc_selective_scan: more than 65535 portions");
  if (x_dt != y_dt) return set_error(OMC_ERR_ARG, "omc_selective_scan: x and y must have the same dtype");
  SelArgs s{x, ldx, dt, lddt, dt_bias, B, ldb, Cm, ldc, A_log, D, z, ldz, state, y, ldy, row_begin, pos, slot, inner, N};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // two states per lane up to 64 states (many short dependency chains: the loop over tokens is sequential), eight above
  const int per = N <= 64 ? 2 : 8;
  int lanes = 1;
  while (lanes * per < N) lanes <<= 1;
  const int ch = kSelThreads / lanes;
  const size_t smem = sizeof(float) * ((size_t)3 * kSelTok * ch + 2 * (size_t)kSelTok * N);
  dim3 grid((inner + ch - 1) / ch, portions);
#define OMC_SEL_LAUNCH(L, P)                                                        \
  OMC_DT_SWITCH(x_dt, TD, {                                                         \
    selective_scan_kernel<L, P, TD><<<grid, kSelThreads, smem, st>>>(s);            \
  })
  if (per == 2) {
    if (lanes == 1) { OMC_SEL_LAUNCH(1, 2) }
    else if (lanes == 2) { OMC_SEL_LAUNCH(2, 2) }
    else if (lanes == 4) { OMC_SEL_LAUNCH(4, 2) }
    else if (lanes == 8) { OMC_SEL_LAUNCH(8, 2) }
    else if (lanes == 16) { OMC_SEL_LAUNCH(16, 2) }
    else { OMC_SEL_LAUNCH(32, 2) }
  } else {
    if (lanes == 16) { OMC_SEL_LAUNCH(16, 8) }
    else { OMC_SEL_LAUNCH(32, 8) }
  }
#undef OMC_SEL_LAUNCH
  return check_launch("omc_selective_scan");
}

template <typename TD, bool FAST>
static int launch_rglru(const LruArgs& a, int rows, int portions, cudaStream_t st) {
  // how many runs of tokens a CTA works on at once, by the average length of a portion (any choice is right for any length)
  const int avg = (rows + portions - 1) / portions;
  if (avg <= 2) {
    rglru_scan_kernel<TD, FAST, 1><<<dim3((a.width + 127) / 128, portions), dim3(128, 1), 0, st>>>(a);
  } else {
    int W = avg >= 96 ? 16 : (avg >= 24 ? 8 : (avg >= 12 ? 4 : 2));
    if (W == 16 && (long long)((a.width + 31) / 32) * portions > 2 * kLruSms) W = 8;   // 16 runs fit an SM twice: no second wave for a few CTAs
    rglru_scan_kernel<TD, FAST, kLruTok><<<dim3((a.width + 31) / 32, portions), dim3(32, W), (size_t)2 * W * 32 * sizeof(float2), st>>>(a);
  }
  return check_launch("omc_rglru_scan");
}

extern "C" int omc_rglru_scan(const void* u, int dt, long long ldu, const float* g, long long ldg, const float* gb, const float* lam,
                              const float* y, long long ldy, float* state, void* out, long long ldo, const int32_t* row_begin, int portions,
                              const int32_t* pos, const int32_t* slot, int rows, int width, int blocks, float decay_scale, void* stream) {
  if (u == nullptr || g == nullptr || lam == nullptr || state == nullptr || out == nullptr || row_begin == nullptr || pos == nullptr ||
      slot == nullptr || portions < 0 || rows < portions || width <= 0 || blocks <= 0 || width % blocks)
    return set_error(OMC_ERR_ARG, "omc_rglru_scan: bad argument");
  if (portions == 0) return OMC_OK;
  if (portions > 65535) return set_error(OMC_ERR_SHAPE, "omc_rglru_scan: more than 65535 portions");
  if (ldu > INT32_MAX || ldg > INT32_MAX || ldy > INT32_MAX || ldo > INT32_MAX) return set_error(OMC_ERR_SHAPE, "omc_rglru_scan: row stride above 2^31");
  const LruArgs a{u, (int)ldu, g, (int)ldg, gb, lam, y, (int)ldy, state, out, (int)ldo, row_begin, pos, slot, width, width / blocks, decay_scale};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (dt == OMC_DT_F32) return launch_rglru<float, false>(a, rows, portions, st);
  if (dt == OMC_DT_BF16) return launch_rglru<bf16_t, true>(a, rows, portions, st);
  return set_error(OMC_ERR_ARG, "omc_rglru_scan: unknown dtype code");
}
