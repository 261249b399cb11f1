// The delta rule, and recurrences with one decay per key channel, over long portions eight tokens at a time (state_mixers.cu describes the recurrence).
// With S the state in front of a stage of tokens 1..8, G_t the product of the decays up to token t and G_t / G_s always formed as the product (or the
// exponential of the sum) of the decays behind s, never as a quotient:
//     a_t = G_t S^T k_t;   u_t = beta_t (v_t - a_t - sum_{s<t} (G_t / G_s) (k_s . k_t) u_s)   (delta rule; otherwise u_t = v_t)
//     o_t = G_t S^T q_t + sum_{s<=t} (G_t / G_s) (k_s . q_t) u_s;   S <- G_8 S + sum_s (G_8 / G_s) k_s u_s^T
// - the same fp32 sums as token by token in another order, with three fma per state element and token instead of four (two instead of three), one rounding
// of the state by a decay per stage instead of per token, and no chain from token to token but the eight steps of u. A sum for token t holds terms of
// tokens s <= t only, so that an infinity or NaN of a later token reaches no earlier output. The sums of a column do not depend on the other portions
// or the launch: which kernel a portion takes is a matter of its own length alone.
// One half of a CTA has the state (32 elements a thread: 4 columns x 8 channels), the other fetches the inputs and forms what a stage's tokens have among
// themselves, one stage ahead. What bounds it: a stage's chain through some 600 instructions of the one warp that a scheduler has for the state (1.3 us, of which
// the eight-lane sums of the products are a half); with several CTAs per SM shared memory's data path.
// Measured in us (token by token in brackets): delta rule, 16 heads of 128 x 128, portions of 1024, 777, 1024, 301 tokens 250 (351), 4 heads, 1100 tokens 177
// (256), 4 heads of 64 x 64 172 (196), 64 tokens 17 (19) and 15 (15); decays per channel over the same 279 (433), 201 (306), 184 (251), 17 (22) and 15 (19). Error of
// output and state against 64 bits (2-norm) 0.5 to 1.0 of token by token, as what a stage's tokens take out of and add to one another is summed by itself before it meets the larger
// numbers from the state (1.02 to 1.10 for decays per channel with the delta rule otherwise) and a channel's G_8 is two numbers (with one, its rounding in decays that hardly change
// is the same in every stage: 2.5 to 6.5 at decays from 0.99 to 0.9999). Decays that never change stay token by token. With step sizes, or one decay per head and no delta rule, a token's chain is short enough
// that this gains nothing with few CTAs (16 heads of 128 x 64, 1100 tokens: 154, 148), so they stay where they were. The same in mma.sync products of three
// bf16 parts (as exact as fp32 fma where leading products are added in fp32) took 8100 instructions per 16 tokens and 64 columns, most of them splits: 286 (256).
#include <type_traits>

#include "scan_args.cuh"

namespace omc {

constexpr int kScTok = 8, kScThreads = 128, kScWarps = kScThreads / 32;   // tokens of a stage; threads of each of the CTA's two halves
constexpr int kScCpt = 4;                                                 // columns of a thread
constexpr int kScRing = 4;                                                // stages of inputs: one in use, one being prepared, two on their way

template <int DIM, int KIND, bool CHAN>
struct ScanChunkShared {
  static constexpr int CPT = kScCpt, LANES = DIM / 8, GROUPS = kScThreads / LANES, COLS = GROUPS * CPT;
  static constexpr int WC = 32 / LANES * CPT, XP = WC + 4;   // a warp's columns; the pitch keeps the tokens of a quarter warp on different banks
  static constexpr bool DELTA = KIND == kScanDelta;
  struct Stage {
    float k[kScTok * DIM], q[kScTok * DIM], g[CHAN ? kScTok * DIM : 4], v[kScTok * COLS];
  };
  struct Ready {                               // what a stage's tokens have among themselves
    float p[kScTok * 12], kk[DELTA ? kScTok * 12 : 4];   // [t][s]: (G_t / G_s) q_t . k_s, (G_t / G_s) k_t . k_s
    float qh[CHAN ? kScTok * DIM : 4], kh[CHAN && DELTA ? kScTok * DIM : 4], kt[CHAN ? kScTok * DIM : 4];   // G_t q_t, G_t k_t, (G_8 / G_s) k_s
    float gl[CHAN ? DIM : 4], gr[CHAN ? DIM : 4];   // G_8, with minus1 less one, and what its rounding leaves: in decays that stay the same that would be the same in every stage and add up
    float gy[kScTok], r[kScTok], all[4];       // G_t, G_8 / G_s, G_8
  };
  Stage stage[kScRing];
  Ready ready[2];
  float la[64], w[64];                         // tokens of two blocks of 32: log decays, beta
  alignas(16) float r[DELTA ? kScWarps * kScTok * XP : 4], u[DELTA ? kScWarps * kScTok * XP : 4];   // [warp][token][column]
};

__device__ __forceinline__ void cp_async16_or_zero(float* dst, const float* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src), "r"(there ? 16 : 0) : "memory");
}
template <int N>
__device__ __forceinline__ void ld_cols(float (&x)[N], const float* p) {
  if constexpr (N == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    x[0] = t.x, x[1] = t.y;
  } else {
#pragma unroll
    for (int i = 0; i < N; i += 4) {
      const float4 t = *reinterpret_cast<const float4*>(p + i);
      x[i] = t.x, x[i + 1] = t.y, x[i + 2] = t.z, x[i + 3] = t.w;
    }
  }
}
template <int N>
__device__ __forceinline__ void st_cols(float* p, const float (&x)[N]) {
  if constexpr (N == 2) {
    *reinterpret_cast<float2*>(p) = make_float2(x[0], x[1]);
  } else {
#pragma unroll
    for (int i = 0; i < N; i += 4) *reinterpret_cast<float4*>(p + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
  }
}
// Sums of eight numbers over a warp: every lane gets the sum of number lane / 4.
__device__ __forceinline__ float sum8_over_warp(const float (&x)[8], int lane) {
  float y[4], z[2];
#pragma unroll
  for (int j = 0; j < 4; ++j) y[j] = (lane & 16 ? x[j + 4] : x[j]) + __shfl_xor_sync(0xffffffffu, lane & 16 ? x[j] : x[j + 4], 16);
#pragma unroll
  for (int j = 0; j < 2; ++j) z[j] = (lane & 8 ? y[j + 2] : y[j]) + __shfl_xor_sync(0xffffffffu, lane & 8 ? y[j] : y[j + 2], 8);
  float s = (lane & 4 ? z[1] : z[0]) + __shfl_xor_sync(0xffffffffu, lane & 4 ? z[0] : z[1], 4);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

// The z-th portion of at least `least` rows, of any number of portions; -1: they are fewer. scratch: shared memory of nine words, free again behind it.
static __device__ int scan_long_portion(const int32_t* row_begin, int portions, int least, int z, int* scratch) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid / 32;
  for (int p0 = 0; p0 < portions; p0 += 2 * kScThreads) {
    const int p = p0 + tid;
    const bool is = p < portions && row_begin[p + 1] - row_begin[p] >= least;
    const int n = __syncthreads_count(is);
    if (z < n) {
      const unsigned these = __ballot_sync(0xffffffffu, is);
      if (lane == 0) scratch[warp] = __popc(these);
      __syncthreads();
      int before = __popc(these & ((1u << lane) - 1));
      for (int w = 0; w < warp; ++w) before += scratch[w];
      if (is && before == z) scratch[8] = p;
      __syncthreads();
      const int found = scratch[8];
      __syncthreads();
      return found;
    }
    z -= n;
  }
  return -1;
}

template <int DIM, int KIND, bool CHAN>
__global__ void __launch_bounds__(2 * kScThreads, 2) scan_chunk_kernel(ScanArgs a, int portions) {
  typedef ScanChunkShared<DIM, KIND, CHAN> Shared;
  typedef typename Shared::Stage Stage;
  typedef typename Shared::Ready Ready;
  extern __shared__ __align__(16) float sm[];
  Shared& sh = *reinterpret_cast<Shared*>(sm);
  constexpr int CPT = kScCpt, LANES = Shared::LANES, COLS = Shared::COLS, WC = Shared::WC, XP = Shared::XP;
  constexpr bool DELTA = KIND == kScanDelta, HALVES = LANES == 16;

  int portion = 0;
  if (portions > kScThreads) {
    portion = scan_long_portion(a.row_begin, portions, a.long_from, blockIdx.z, reinterpret_cast<int*>(sm));
    if (portion < 0) return;
  } else if (portions > 1) {
    portion = scan_portion(a.row_begin, portions, blockIdx.z, reinterpret_cast<int*>(sm));
  }
  const int r0 = a.row_begin[portion], r1 = a.row_begin[portion + 1], stages = (r1 - r0 + kScTok - 1) / kScTok;
  if (!scan_is_long(a, r1 - r0)) return;
  scan_begin(a);   // not before: CTAs without a portion would still be there when the other kernel's are spread over the SMs (3 x 63 tokens 27 -> 35 us)
  const int h = blockIdx.y, col0 = blockIdx.x * COLS;
  const bool minus1 = CHAN && a.decay_mode == 5;
  auto meet = [] { asm volatile("bar.sync 1, 256;" ::: "memory"); };   // once per stage, both halves

  // Registers go from the half that prepares to the half that has the state: 168 + 88 = the 2 x 128 of the launch
  if (threadIdx.x >= kScThreads) {
    // ---- the half that fetches and prepares: stages i + 2 and i + 3 are on their way and stage i + 1 is prepared while stage i is computed
    asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
    const int tid = threadIdx.x - kScThreads, wl = tid & 31, warp = tid / 32, kvh = h / (a.H / a.G);
    const float A = CHAN ? 0.f : expf(a.A_log[h]), bias = CHAN ? 0.f : a.dt_bias[h];
    constexpr int PIECES = DIM / 4, STEP_T = kScThreads / PIECES, VP = COLS / 4, STEP_V = kScThreads / VP;
    static_assert(kScThreads % VP == 0, "");
    const int piece = tid % PIECES * 4, tok0 = tid / PIECES, vtok = tid / VP, vcol = tid % VP * 4;
    const bool vin = col0 + vcol < a.vdim;
    const float* kp = a.k + (long long)(r0 + tok0) * a.ldk + (long long)kvh * DIM + piece;
    const float* qp = a.q + (long long)(r0 + tok0) * a.ldq + (long long)kvh * DIM + piece;
    const float* gp = CHAN ? a.a + (long long)(r0 + tok0) * a.lda + (long long)h * DIM + piece : nullptr;
    const float* vp = a.v + (vin ? (long long)(r0 + vtok) * a.ldv + (long long)h * a.vdim + col0 + vcol : 0);
    int left = r1 - r0, at4 = 0;               // rows from the next stage to be fetched on, and its place
    auto fetch = [&] {                         // rows behind the portion's end are zeros; behind the last stage nothing
      if (left > 0) {
        Stage& s = sh.stage[at4];
#pragma unroll
        for (int i = 0; i < kScTok; i += STEP_T) {
          const int at = (tok0 + i) * DIM + piece;
          const bool there = tok0 + i < left;
          cp_async16_or_zero(s.k + at, there ? kp + i * a.ldk : a.k, there);
          cp_async16_or_zero(s.q + at, there ? qp + i * a.ldq : a.q, there);
          if (CHAN) cp_async16_or_zero(s.g + at, there ? gp + i * a.lda : a.a, there);
        }
#pragma unroll
        for (int i = 0; i < kScTok; i += STEP_V) {
          const bool there = vin && vtok + i < left;
          if (STEP_V <= kScTok || vtok < kScTok) cp_async16_or_zero(s.v + (vtok + i) * COLS + vcol, there ? vp + i * a.ldv : a.v, there);
        }
        kp += kScTok * a.ldk, qp += kScTok * a.ldq, left -= kScTok;
        if (vin) vp += kScTok * a.ldv;
        if (CHAN) gp += kScTok * a.lda;
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      at4 = at4 + 1 & (kScRing - 1);
    };
    // the numbers that a token has alone, 32 tokens at a time, by the last warp
    float raw_a = 0.f, raw_b = 0.f;
    auto load_raw = [&](int c0) {
      const int t = c0 + wl;
      if (t < r1) {
        if (!CHAN) raw_a = a.a[(long long)t * a.lda + h];
        if (DELTA) raw_b = a.beta[(long long)t * a.ldb + h];
      }
    };
    auto put_raw = [&](int c0, int block) {   // a token behind the end decays nothing (however large A is); its zero rows enter nothing
      const bool there = c0 + wl < r1;
      if (!CHAN) sh.la[(block & 1) * 32 + wl] = there ? -A * softplus_f(raw_a + bias) : 0.f;
      if (DELTA) sh.w[(block & 1) * 32 + wl] = sigmoid_f(raw_b);
    };
    // What the tokens of a stage have among themselves: warp w forms the products of tokens w and 7 - w with those up to them (nine each, the lanes over the channels)
    auto prepare = [&](const Stage& s, Ready& r, int stage, int n) {
      constexpr int V = DIM / 32;
      float aq[9], ak[9], qa[V], qb[V], ka[V], kb[V];
      ld_cols(qa, s.q + warp * DIM + V * wl);
      ld_cols(qb, s.q + (7 - warp) * DIM + V * wl);
      if (DELTA) ld_cols(ka, s.k + warp * DIM + V * wl), ld_cols(kb, s.k + (7 - warp) * DIM + V * wl);
#pragma unroll
      for (int j = 0; j < 9; ++j) {
        const bool first = j <= warp;
        const int from = first ? warp - j : 8 - j;
        float kv[V];
        ld_cols(kv, s.k + from * DIM + V * wl);
        float xq = 0.f, xk = 0.f;
#pragma unroll
        for (int i = 0; i < V; ++i) {
          xq = fmaf(first ? qa[i] : qb[i], kv[i], xq);
          if (DELTA) xk = fmaf(first ? ka[i] : kb[i], kv[i], xk);
        }
        aq[j] = xq, ak[j] = xk;
        if (CHAN) {   // on the way to the token before it the products take in this one's decays
          float g[V];
          ld_cols(g, s.g + from * DIM + V * wl);
          const bool there = from < n;
#pragma unroll
          for (int i = 0; i < V; ++i) {
            const float x = there ? (minus1 ? 1.f + g[i] : g[i]) : 1.f;
            if (first) qa[i] *= x;
            else qb[i] *= x;
            if (DELTA && first) ka[i] *= x;
            if (DELTA && !first) kb[i] *= x;
          }
        }
      }
      float la[kScTok];
      if (!CHAN) ld_cols(la, sh.la + (stage & 7) * kScTok);
      auto between = [&](int lo, int hi) {   // the product of the decays of tokens lo .. hi - 1
        float x = 0.f;
#pragma unroll
        for (int i = 0; i < kScTok; ++i)
          if (i >= lo && i < hi) x += la[i];
        return expf(x);
      };
      float x8q[8], x8k[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) x8q[j] = aq[j], x8k[j] = ak[j];
      const float q8 = sum8_over_warp(x8q, wl), k8 = DELTA ? sum8_over_warp(x8k, wl) : 0.f;
      const float q9 = seq_warp_sum(aq[8]), k9 = DELTA ? seq_warp_sum(ak[8]) : 0.f;
      {   // lane 4 j holds product j of the first eight, lane 1 puts the ninth
        const int j = wl == 1 ? 8 : wl / 4;
        const bool first = j <= warp;
        const int from = first ? warp - j : 8 - j, t = first ? warp : 7 - warp;
        float ratio = 1.f;
        if (!CHAN) ratio = between(from + 1, t + 1);
        if ((wl & 3) == 0 || wl == 1) {
          r.p[t * 12 + from] = (wl == 1 ? q9 : q8) * ratio;
          if (DELTA) r.kk[t * 12 + from] = (wl == 1 ? k9 : k8) * ratio;
        }
      }
      if (!CHAN) {
        if (tid < kScTok) {
          r.gy[tid] = between(0, tid + 1);
          r.r[tid] = between(tid + 1, kScTok);
        } else if (tid == 32) {
          r.all[0] = between(0, kScTok);
        }
      } else {
        // a channel per thread (64 channels: half of the threads go forward, half backward)
        const int i = tid % DIM;
        float x[kScTok], gl, gr;
#pragma unroll
        for (int t = 0; t < kScTok; ++t) x[t] = t < n ? s.g[t * DIM + i] : (minus1 ? 0.f : 1.f);
        if (minus1) {   // (1 + a) (1 + b) - 1
          auto both = [](double a, double b) { return fma(a, b, a) + b; };
          const double all = both(both(both(x[0], x[1]), both(x[2], x[3])), both(both(x[4], x[5]), both(x[6], x[7])));
          gl = (float)all, gr = (float)(all - (double)gl);
#pragma unroll
          for (int t = 0; t < kScTok; ++t) x[t] += 1.f;
        }
        // their products by halves: at most four roundings each instead of seven
        const float x01 = x[0] * x[1], x23 = x[2] * x[3], x45 = x[4] * x[5], x67 = x[6] * x[7], x03 = x01 * x23, x47 = x45 * x67;
        if (!minus1) {   // a product's rounding is an fma's; those of its factors come along
          auto rest = [](float a, float b, float ab, float ra, float rb) { return fmaf(a, b, -ab) + fmaf(a, rb, ra * b); };
          const float r03 = rest(x01, x23, x03, fmaf(x[0], x[1], -x01), fmaf(x[2], x[3], -x23)), r47 = rest(x45, x67, x47, fmaf(x[4], x[5], -x45), fmaf(x[6], x[7], -x67));
          gl = x03 * x47, gr = rest(x03, x47, gl, r03, r47);
        }
        if (DIM == kScThreads || tid < DIM) {
          const float G[kScTok] = {x[0], x01, x01 * x[2], x03, x03 * x[4], x03 * x45, x03 * (x45 * x[6]), x03 * x47};
#pragma unroll
          for (int t = 0; t < kScTok; ++t) {
            r.qh[t * DIM + i] = s.q[t * DIM + i] * G[t];
            if (DELTA) r.kh[t * DIM + i] = s.k[t * DIM + i] * G[t];
          }
          r.gl[i] = gl, r.gr[i] = gr;
        }
        if (DIM == kScThreads || tid >= DIM) {
          const float R[kScTok] = {x[1] * (x23 * x47), x23 * x47, x[3] * x47, x47, x[5] * x67, x67, x[7], 1.f};
#pragma unroll
          for (int t = 0; t < kScTok; ++t) r.kt[t * DIM + i] = s.k[t * DIM + i] * R[t];
        }
      }
    };

    fetch(), fetch(), fetch();
    if (warp == kScWarps - 1) {
      load_raw(r0);
      put_raw(r0, 0);
      load_raw(r0 + 32);
    }
    asm volatile("cp.async.wait_group 2;" ::: "memory");
    asm volatile("bar.sync 2, 128;" ::: "memory");
    prepare(sh.stage[0], sh.ready[0], 0, min(kScTok, r1 - r0));
    for (int i = 0; i < stages; ++i) {
      const int c1 = r0 + (i + 1) * kScTok;
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      meet();   // stage i + 1 is there, stage i prepared, stage i - 1 read by all
      fetch();
      if (warp == kScWarps - 1 && (i & 3) == 0) {
        put_raw(r0 + i * kScTok + 32, i / 4 + 1);
        load_raw(r0 + i * kScTok + 64);
      }
      if (c1 < r1) prepare(sh.stage[i + 1 & (kScRing - 1)], sh.ready[(i + 1) & 1], i + 1, min(kScTok, r1 - c1));
    }
    return;
  }

  // ---- the half that has the state
  asm volatile("setmaxnreg.inc.sync.aligned.u32 168;");
  const int tid = threadIdx.x, wl = tid & 31, warp = tid / 32, lane = tid % LANES, cg = tid / LANES, l7 = lane & 7;
  constexpr int CW = HALVES ? CPT / 2 : CPT;   // columns of a thread once the lanes' sums are formed
  // a thread's columns: slots [0, CPT / 2) from colA, the rest from colB. With 16 lanes to a column group the upper eight hold the halves the other way
  // round, so that what a lane passes on when sums are formed is in the same registers everywhere (as the order of tokens below)
  constexpr int H2 = CPT / 2;
  const int half = HALVES ? (lane >> 3) : 0, base = col0 + CPT * cg;
  const int colA = base + half * H2, colB = base + (half ^ 1) * H2;
  const bool inA = colA < a.vdim, inB = colB < a.vdim;   // widths are multiples of four: halves of four (two) exist or don't as a whole

  // a thread's channels: 4 lane + {0..3} and DIM / 2 + 4 lane + {0..3}, in pairs; the quarter warps read whole runs of a row of k or q
  float* S = a.state + (((long long)a.slot[r0] * a.H + h) * DIM) * a.vdim;
  f32x2 st[CPT][4];
  const bool fresh = a.pos[r0] == 0;
  auto channel = [&](int pair, int j) { return (pair >> 1) * (DIM / 2) + 4 * lane + 2 * (pair & 1) + j; };
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    float e[2][CPT];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float* row = S + (long long)channel(p, j) * a.vdim;
      float x[H2], y[H2];
#pragma unroll
      for (int c = 0; c < H2; ++c) x[c] = y[c] = 0.f;
      if (!fresh && inA) ld_cols(x, row + colA);
      if (!fresh && inB) ld_cols(y, row + colB);
#pragma unroll
      for (int c = 0; c < H2; ++c) e[j][c] = x[c], e[j][H2 + c] = y[c];
    }
#pragma unroll
    for (int c = 0; c < CPT; ++c) st[c][p] = pack2(e[0][c], e[1][c]);
  }

  for (int i = 0; i < stages; ++i) {
    const int c0 = r0 + i * kScTok;
    const Stage& s = sh.stage[i & (kScRing - 1)];
    const Ready& r = sh.ready[i & 1];
    meet();

    // S^T x of the eight tokens over the lanes: lane l goes through the tokens in the order 0 ^ l, 1 ^ l, ..., so at every step of the sum all lanes pass on
    // the same registers; in the end it holds token l % 8 for the columns from colA
    auto dots = [&](const float* x, float (&sum)[CW]) {
      float A1[CPT], A2[CPT], A4[CPT];
#pragma unroll
      for (int j = 0; j < kScTok; ++j) {
        const float* row = x + (j ^ l7) * DIM + 4 * lane;
        const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(row), hi = *reinterpret_cast<const ulonglong2*>(row + DIM / 2);
        float p[CPT];
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          float e, o;
          unpack2(fma2(st[c][3], hi.y, fma2(st[c][2], hi.x, fma2(st[c][1], lo.y, mul2(st[c][0], lo.x)))), e, o);
          p[c] = e + o;
        }
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          if (j & 1) A1[c] += __shfl_xor_sync(0xffffffffu, p[c], 1);
          else A1[c] = p[c];
          if ((j & 3) == 1) A2[c] = A1[c];
          if ((j & 3) == 3) A2[c] += __shfl_xor_sync(0xffffffffu, A1[c], 2);
          if (j == 3) A4[c] = A2[c];
          if (j == 7) A4[c] += __shfl_xor_sync(0xffffffffu, A2[c], 4);
        }
      }
#pragma unroll
      for (int c = 0; c < CW; ++c) sum[c] = HALVES ? A4[c] + __shfl_xor_sync(0xffffffffu, A4[c + CPT - CW], 8) : A4[c];
    };
    float o[CW];
    const float gy = CHAN ? 1.f : r.gy[l7];
    const int wcol = (cg % (32 / LANES)) * CPT;   // of `base` among the warp's columns
    if constexpr (DELTA) {
      const int n = r1 - c0;
      float d[CW], v[CW];
      dots(CHAN ? r.kh : s.k, d);
      ld_cols(v, s.v + l7 * COLS + colA - col0);
#pragma unroll
      for (int c = 0; c < CW; ++c) d[c] = CHAN ? v[c] - d[c] : fmaf(-gy, d[c], v[c]);
      st_cols(sh.r + (warp * kScTok + l7) * XP + wcol + half * H2, d);
      __syncwarp();
      if (wl < WC) {   // a column per lane: u token by token; what earlier ones take out of a token is added up by itself, with the roundings of its own smaller numbers
        const float* rp = sh.r + warp * kScTok * XP + wl;
        float* up = sh.u + warp * kScTok * XP + wl;
        float x[kScTok], w[kScTok], kk[kScTok][kScTok], out_of[kScTok] = {};
#pragma unroll
        for (int t = 0; t < kScTok; ++t) x[t] = rp[t * XP];
        ld_cols(w, sh.w + (i & 7) * kScTok);
#pragma unroll
        for (int t = 1; t < kScTok; ++t)
#pragma unroll
          for (int f = 0; f < t; f += 4) {
            const float4 y = *reinterpret_cast<const float4*>(r.kk + t * 12 + f);
            kk[t][f] = y.x, kk[t][f + 1] = y.y, kk[t][f + 2] = y.z, kk[t][f + 3] = y.w;
          }
#pragma unroll
        for (int t = 0; t < kScTok; ++t) {
          const float u = t < n ? w[t] * (x[t] - out_of[t]) : 0.f;   // nothing of the state comes back through a row behind the end
          up[t * XP] = u;
#pragma unroll
          for (int f = t + 1; f < kScTok; ++f) out_of[f] = fmaf(kk[f][t], u, out_of[f]);
        }
      }
    }
    dots(CHAN ? r.qh : s.q, o);
    if (DELTA) __syncwarp();
    float own[CW] = {};   // what the stage's tokens bring

    // the state and the read-out with what the stage's tokens bring
    if constexpr (CHAN) {
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const ulonglong2 g = *reinterpret_cast<const ulonglong2*>(r.gl + x * (DIM / 2) + 4 * lane), rest = *reinterpret_cast<const ulonglong2*>(r.gr + x * (DIM / 2) + 4 * lane);
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          st[c][2 * x] = fma2(st[c][2 * x], g.x, minus1 ? fma2(st[c][2 * x], rest.x, st[c][2 * x]) : mul2(st[c][2 * x], rest.x));
          st[c][2 * x + 1] = fma2(st[c][2 * x + 1], g.y, minus1 ? fma2(st[c][2 * x + 1], rest.y, st[c][2 * x + 1]) : mul2(st[c][2 * x + 1], rest.y));
        }
      }
    } else {
      const float ga = r.all[0];
      const f32x2 g = pack2(ga, ga);
#pragma unroll
      for (int c = 0; c < CPT; ++c)
#pragma unroll
        for (int p = 0; p < 4; ++p) st[c][p] = mul2(st[c][p], g);
    }
    float pr[kScTok];
    ld_cols(pr, r.p + l7 * 12);
    const float* in = DELTA ? sh.u + warp * kScTok * XP + wcol : s.v + base - col0;
    constexpr int IP = DELTA ? XP : COLS;
#pragma unroll
    for (int f = 0; f < kScTok; ++f) {
      const float* row = (CHAN ? r.kt : s.k) + f * DIM + 4 * lane;
      const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(row), hi = *reinterpret_cast<const ulonglong2*>(row + DIM / 2);
      const float rf = CHAN ? 1.f : r.r[f];
      float xa[H2], xb[H2], x[CPT];
      ld_cols(xa, in + f * IP + half * H2);
      ld_cols(xb, in + f * IP + (half ^ 1) * H2);
#pragma unroll
      for (int c = 0; c < H2; ++c) x[c] = xa[c], x[H2 + c] = xb[c];
#pragma unroll
      for (int c = 0; c < CW; ++c)
        if (f <= l7) own[c] = fmaf(pr[f], x[c], own[c]);
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        const float y = CHAN ? x[c] : x[c] * rf;
        const f32x2 u2 = pack2(y, y);
        st[c][0] = fma2(lo.x, u2, st[c][0]), st[c][1] = fma2(lo.y, u2, st[c][1]);
        st[c][2] = fma2(hi.x, u2, st[c][2]), st[c][3] = fma2(hi.y, u2, st[c][3]);
      }
    }
#pragma unroll
    for (int c = 0; c < CW; ++c) o[c] = (CHAN ? o[c] + own[c] : fmaf(o[c], gy, own[c])) * a.out_scale;
    if (c0 + l7 < r1) {
      float* dst = a.out + (long long)(c0 + l7) * a.ldo + (long long)h * a.vdim + colA;
      if (inA) st_cols(dst, o);
    }
  }
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    float e[2][CPT];
#pragma unroll
    for (int c = 0; c < CPT; ++c) unpack2(st[c][p], e[0][c], e[1][c]);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      float* row = S + (long long)channel(p, j) * a.vdim;
      float x[H2], y[H2];
#pragma unroll
      for (int c = 0; c < H2; ++c) x[c] = e[j][c], y[c] = e[j][H2 + c];
      if (inA) st_cols(row + colA, x);
      if (inB) st_cols(row + colB, y);
    }
  }
}

int launch_scan_chunk(const ScanArgs& a, int rows, int portions, cudaStream_t st) {
  using std::integral_constant;
  const bool chan = a.decay_mode == 3 || a.decay_mode == 5;
  if (a.long_from <= 0 || (!chan && (a.beta == nullptr || a.decay_mode != 1)) || (a.dim != 64 && a.dim != 128)) return set_error(OMC_ERR_SHAPE, "omc_linear_state_scan: not a recurrence of the kernel for long portions");
  const int most = rows / a.long_from < portions ? rows / a.long_from : portions;   // only so many portions can be long ones
  auto go = [&](auto dim_c, auto kind_c, auto chan_c) {
    constexpr int DIM = decltype(dim_c)::value, KIND = decltype(kind_c)::value;
    constexpr bool CHAN = decltype(chan_c)::value;
    typedef ScanChunkShared<DIM, KIND, CHAN> Shared;
    static bool attr_done[kMaxDevices] = {};
    constexpr int smem = (int)sizeof(Shared);
    if (!attr_done[cur_device()]) {
      cudaFuncSetAttribute(scan_chunk_kernel<DIM, KIND, CHAN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      attr_done[cur_device()] = true;
    }
    return scan_launch(scan_chunk_kernel<DIM, KIND, CHAN>, dim3((a.vdim + Shared::COLS - 1) / Shared::COLS, a.H, most), 2 * kScThreads, smem, st, a, portions);
  };
  auto kinds = [&](auto dim_c) {
    if (!chan) return go(dim_c, integral_constant<int, kScanDelta>(), std::false_type());
    if (a.beta != nullptr) return go(dim_c, integral_constant<int, kScanDelta>(), std::true_type());
    return go(dim_c, integral_constant<int, kScanPlain>(), std::true_type());
  };
  return a.dim == 128 ? kinds(integral_constant<int, 128>()) : kinds(integral_constant<int, 64>());
}

}  // namespace omc
