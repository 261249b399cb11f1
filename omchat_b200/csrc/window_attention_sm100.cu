// Windowed and chunked attention of prompt portions on tcgen05 / TMEM (bf16; the work list of omc_window_attn_mma, head widths of 64 or 128 for keys
// and values alike, pages of a multiple of 64 rows, one score map, no kept first keys). Everything else stays with the mma.sync kernel of
// window_attention.cu.
//
// The 128 rows of a CTA are the (token, query head) pairs of one key/value head: one item of the list, or two that follow one another in the same
// request (each takes half of the rows). Rows lie on the 128 lanes of TMEM, so a softmax thread owns one row: no shuffles, and its 64 scores
// of a key tile stay in registers.
//   warps 0..3   Q; softmax, one thread per row: scale, soft cap, distance bias, mask, maximum, probabilities. P goes back to TMEM over its scores as
//                two bf16 numbers (its rounding and what that left), which is the A operand of the output product. The reference maximum of a row
//                moves only when it grew by more than 2^8; O is then rescaled in TMEM.
//   warp 4       MMA issuer (one thread): S = Q K^T of the next tile before O += P V of this one, so scores wait in a second buffer of TMEM
//   warps 5, 6   keys and values by cp.async, two tiles each
// The bias lies in shared memory by head and distance, in base-2 units with the soft cap's constant added: a row walks its tile at fixed offsets
// from one address, and the rows of a warp (consecutive tokens, heads a bank offset apart) meet different banks.
// Two CTAs share an SM and hide each other's waits. What bounds it is the chain of a tile, at two softmax warps per scheduler: with a soft cap (three operations of the
// exponential unit per score, 16 per cycle and SM: 1536 cycles per tile) that unit is busy 42 % of the time, issue slots 43 %, tensor pipe 19 %. Two threads per row were slower without a cap (12 to 27 %: one more barrier per tile) and no
// faster with one. Head fastest and the later items first in the grid: portions end with their items of few keys (103 us with the items fastest).
// Measured, mma.sync kernel in brackets: 32 heads on 8 key/value heads of 128, portions of 1024, 777, 1024 behind 1024 and 301 rows, window 512, cap and
// bias: 89 us (270); 4 x 2048 rows behind 2048, causal: 667 us = 618 TFLOP/s (2880).
// Keys and values come by cp.async and not by TMA: boxes addressed through a block table, every one of them inside the pool, gave illegal accesses with
// a tensor map that claimed more rows than the pool has, and once with one that did not, for no reason that was found.
// A value that is not a finite number reaches every row of a CTA that has its key, also those of earlier tokens (0 x infinity in the output product; on mma.sync the
// rows of one item, here of two).
#include <type_traits>

#include "sm100_step.cuh"

namespace omc {

constexpr int kWsKeys = 64, kWsRows = 128, kWsSoftmax = 128, kWsLoad = 64, kWsThreads = kWsSoftmax + 32 + kWsLoad;
constexpr int kWsBox = kWsKeys * 128;            // bytes of 64 columns x 64 keys

static __device__ unsigned int g_window_failures;   // waits that ran out

struct WinSmArgs {
  const bf16_t* q;
  long long ldq;
  const bf16_t* pool;
  const int32_t* bt;
  const int32_t* items;   // int32[n][4]: first row, tokens, slot, first position
  const float* bias;      // [window][H] or NULL
  const float* sink;
  const float* gate;
  long long ldg;
  int gate_act, gate_heads;
  void* out;
  long long ldo;
  int out_bf16, n_items, max_pages, page_size, H, G, window, chunk, tok, table;   // tok: tokens of a full item; table: bytes of the bias table
  float scale, softcap;
  unsigned int* failed;
};

struct WinSmBars {
  uint64_t q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_ready[2], o_done, mma_done;
  uint32_t tmem, dead;
};
constexpr int kWsTail = 768;                     // bytes behind the bias table: the barriers, and what hidden scores read over its end
static_assert(sizeof(WinSmBars) <= kWsTail, "barriers");

__device__ __forceinline__ float ws_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ws_rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Floats from one head's row of the bias table to the next: rows of the heads of a token start 32 / rep banks apart.
__host__ __device__ constexpr int ws_bias_pitch(int window, int rep) { return (window + 31) / 32 * 32 + (rep > 1 && rep < 32 ? 32 / rep : 0); }

// Whether item b continues item a: the same request, the next row and position, a full item in front, one chunk.
__device__ __forceinline__ bool ws_follows(const int4& a, const int4& b, int tok, int chunk) {
  return a.z == b.z && a.x + a.y == b.x && a.w + a.y == b.w && a.y == tok && b.y > 0 && b.y <= tok && a.w / chunk == b.w / chunk;
}

template <int D, bool CAP, bool BIAS>
__global__ void __launch_bounds__(kWsThreads, 2) window_attn_sm100_kernel(WinSmArgs a) {
  constexpr int kChunks = D / 64, kTile = kChunks * kWsBox, kQChunk = kWsRows * 128;
  constexpr float kLog2e = 1.4426950408889634f;
  // Two items of a run become one CTA. The items of a portion are `tok` tokens apart, so the parity of position / tok alternates along it
  // and says which of two neighbours leads, without a look at more than one item on either side.
  const int kvh = blockIdx.x % a.G, i = a.n_items - 1 - (int)(blockIdx.x / a.G);   // of a portion the later items, which have the most keys, come first
  const int4 it = reinterpret_cast<const int4*>(a.items)[i];
  int4 next = make_int4(0, 0, 0, 0);
  if (it.y <= 0) return;
  if ((it.w / a.tok) & 1) {
    if (i > 0 && ws_follows(reinterpret_cast<const int4*>(a.items)[i - 1], it, a.tok, a.chunk)) return;   // the item in front takes this one
  } else if (i + 1 < a.n_items) {
    next = reinterpret_cast<const int4*>(a.items)[i + 1];
    if (!ws_follows(it, next, a.tok, a.chunk)) next.y = 0;
  }
  extern __shared__ __align__(1024) uint8_t ws_raw[];
  uint8_t* const ks = ws_raw;                              // [2 stages][chunk][64 keys][128 B]
  uint8_t* const vs = ks + 2 * kTile;
  uint8_t* const qs = vs + 2 * kTile;                      // [chunk][128 rows][128 B]
  float* const table = reinterpret_cast<float*>(qs + kChunks * kQChunk);   // hidden scores read up to 190 floats over its ends: Q in front, kWsTail behind
  WinSmBars* const sh = reinterpret_cast<WinSmBars*>(qs + kChunks * kQChunk + a.table);
  const int rep = a.H / a.G, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int first_pos = it.w, n_tok = it.y + next.y;
  const int k_begin = max(max(0, first_pos - a.window + 1), first_pos - first_pos % a.chunk), k_end = first_pos + n_tok;
  const int k0 = k_begin & ~(kWsKeys - 1), n_tiles = (k_end - k0 + kWsKeys - 1) / kWsKeys;

  const WaitReport report{&sh->dead, &g_window_failures, a.failed};
  auto wait = [&](uint64_t* bar, uint32_t parity) { return wait_bounded(bar, parity, report); };
  if (tid == 0) {
    mbar_init(&sh->q_full, kWsSoftmax / 32);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sh->k_full[b], kWsLoad / 32);
      mbar_init(&sh->k_empty[b], 1);
      mbar_init(&sh->v_full[b], kWsLoad / 32);
      mbar_init(&sh->v_empty[b], 1);
      mbar_init(&sh->s_full[b], 1);
      mbar_init(&sh->p_ready[b], kWsSoftmax / 32);
    }
    mbar_init(&sh->o_done, 1);
    mbar_init(&sh->mma_done, 1);
    sh->dead = 0u;
    fence_barrier_init();
  }
  if (warp == 4) {
    tmem_alloc<1>(&sh->tmem, 256);
    tmem_relinquish<1>();
  }
  // loads: eight lanes per 128 bytes of a row, as the 128-byte swizzle has them
  if (tid < kWsSoftmax) {
    const int c = tid & 7;
    for (int r = tid >> 3; r < kWsRows; r += kWsSoftmax / 8) {
      const int4 mine = r < 64 ? it : next;
      const int row = r & 63, token = row / rep, h = row - token * rep;
      const bf16_t* src = a.q + (long long)(mine.x + token) * a.ldq + (long long)(kvh * rep + h) * D + c * 8;
      uint8_t* at = qs + r * 128 + ((c ^ (r & 7)) << 4);
#pragma unroll
      for (int b = 0; b < kChunks; ++b) {
        if (token < mine.y) cp_async16(at + b * kQChunk, src + b * 64, true);
        else *reinterpret_cast<uint4*>(at + b * kQChunk) = make_uint4(0, 0, 0, 0);
      }
    }
    cp_async_commit();
  }
  if constexpr (BIAS) {
    const int pitch = ws_bias_pitch(a.window, rep);
    for (int e = tid; e < a.window * rep; e += kWsThreads) {
      const int dist = e / rep, h = e - dist * rep;
      table[h * pitch + dist] = (a.bias[(long long)dist * a.H + kvh * rep + h] + (CAP ? a.softcap : 0.f)) * kLog2e;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem, tmem_o = tmem + 2 * kWsKeys;   // scores: two buffers of 64 columns

  if (warp == 4) {
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc_bf16_major(kWsRows, kWsKeys, 0, 0), idesc_o = make_idesc_bf16_major(kWsRows, D, 0, 1);
      const uint64_t dq = make_sw128_kmajor_desc(smem_u32(qs)), dk0 = make_sw128_kmajor_desc(smem_u32(ks));
      const uint64_t dv0 = make_sw128_mnmajor_desc(smem_u32(vs), kWsBox, 1024);
      auto scores = [&](int t) {
        const uint64_t dk = dk0 + (uint64_t)((t & 1) * (kTile >> 4));
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
          umma_bf16<1>(tmem + (uint32_t)(t & 1) * kWsKeys, dq + (uint64_t)((k >> 2) * (kQChunk >> 4) + 2 * (k & 3)), dk + (uint64_t)((k >> 2) * (kWsBox >> 4) + 2 * (k & 3)),
                       idesc_s, k != 0 ? 1u : 0u);
        umma_commit(&sh->s_full[t & 1]);
        umma_commit(&sh->k_empty[t & 1]);
      };
      bool go = wait(&sh->q_full, 0) && wait(&sh->k_full[0], 0);
      tc_fence_after();
      if (go) scores(0);
      for (int t = 0; go && t < n_tiles; ++t) {
        const uint32_t phase = (uint32_t)(t >> 1) & 1u;
        if (t + 1 < n_tiles) {
          // over the probabilities of the tile before: the order of products is only promised for one accumulator, so the one that reads them has
          // to be done, not only issued
          go = (t == 0 || wait(&sh->o_done, (uint32_t)(t - 1) & 1u)) && wait(&sh->k_full[(t + 1) & 1], (uint32_t)((t + 1) >> 1) & 1u);
          if (!go) break;
          tc_fence_after();
          scores(t + 1);
        }
        go = wait(&sh->v_full[t & 1], phase) && wait(&sh->p_ready[t & 1], phase);
        if (!go) break;
        tc_fence_after();
        const uint64_t dv = dv0 + (uint64_t)((t & 1) * (kTile >> 4));
        const uint32_t p = tmem + (uint32_t)(t & 1) * kWsKeys;   // columns 0..31: upper numbers, 32..63: lower ones
#pragma unroll
        for (int k = 0; k < kWsKeys / 16; ++k)
#pragma unroll
          for (int low = 0; low < 2; ++low) umma_bf16_ts(tmem_o, p + 32u * low + 8u * k, dv + (uint64_t)(k * 128), idesc_o, (t | k | low) != 0 ? 1u : 0u);
        umma_commit(&sh->o_done);
        umma_commit(&sh->v_empty[t & 1]);
      }
      umma_commit(&sh->mma_done);
      drain_bounded(&sh->mma_done, 0, report);             // every product that was issued is done
    }
  } else if (warp > 4) {
    // keys and values of the tiles in turn, two copies ahead of the one that is waited for
    const int32_t* bt = a.bt + (long long)it.z * a.max_pages;
    const long long W = 2LL * a.G * D;
    const int c = tid & 7, key0 = (tid - kWsSoftmax - 32) >> 3;
    auto arrive = [&](int i, auto ahead) {                 // copy i is there, and visible to the products
      cp_async_wait<decltype(ahead)::value>();
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive((i & 1) ? &sh->v_full[(i >> 1) & 1] : &sh->k_full[(i >> 1) & 1]);
    };
    long long first = 0;                                   // the tile's first row of the pool: a tile starts at a multiple of 64 keys, as pages do
    int i = 0;
    for (; i < 2 * n_tiles; ++i) {
      const int t = i >> 1, j0 = k0 + t * kWsKeys;
      const bool values = i & 1;
      if (!values) first = (long long)bt[j0 / a.page_size] * a.page_size + j0 % a.page_size;
      if (!wait_bounded_warp(values ? &sh->v_empty[t & 1] : &sh->k_empty[t & 1], ((uint32_t)(t >> 1) & 1u) ^ 1u, report)) break;   // the lanes leave together or not at all
      uint8_t* dst = (values ? vs : ks) + (t & 1) * kTile;
      const bf16_t* src = a.pool + first * W + (values ? a.G + kvh : kvh) * D + c * 8;
#pragma unroll
      for (int k = 0; k < kWsKeys; k += kWsLoad / 8) {
        const int key = k + key0;
        uint8_t* at = dst + key * 128 + ((c ^ (key & 7)) << 4);
        // rows that are no keys of this CTA hold whatever the cache holds there: as values they must not meet a product
        const bool is_key = j0 + key >= k_begin && j0 + key < k_end;
#pragma unroll
        for (int b = 0; b < kChunks; ++b) {
          if (is_key) cp_async16(at + b * kWsBox, src + key * W + b * 64, true);
          else *reinterpret_cast<uint4*>(at + b * kWsBox) = make_uint4(0, 0, 0, 0);
        }
      }
      cp_async_commit();
      if (i >= 2) arrive(i - 2, std::integral_constant<int, 2>());
    }
    if (i == 2 * n_tiles) {
      arrive(i - 2, std::integral_constant<int, 1>());
      arrive(i - 1, std::integral_constant<int, 0>());
    }
    cp_async_wait<0>();
  } else {
    const int quarter = warp, row = (quarter & 1) * 32 + lane;   // TMEM lanes go by warp % 4
    const int4 mine = quarter < 2 ? it : next;
    const int n_rows = mine.y * rep, token = row / rep, h = row - token * rep;
    const bool any = (quarter & 1) * 32 < n_rows, is_row = row < n_rows;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    // rows behind the item's last repeat its last token and are not stored
    const int p = mine.w + min(token, mine.y - 1), low = max(p - a.window + 1, p - p % a.chunk);
    const float c1 = CAP ? a.scale / a.softcap * (2.f * kLog2e) : a.scale * kLog2e, c2 = -2.f * a.softcap * kLog2e, cap = a.softcap * kLog2e;
    const float* brow = BIAS ? table + (is_row ? h : 0) * ws_bias_pitch(a.window, rep) + p : nullptr;
    float m_ref = -INFINITY, l = 0.f;
    // the lanes of a warp may leave a wait one by one, and accesses to tensor memory are the warp's as a whole; whether the phase came is not asked
    auto wait_together = [&](uint64_t* bar, uint32_t parity) {
      wait(bar, parity);
      __syncwarp();
    };
    // The output product of the tile before is done. Waited for in front of every arrival that lets the next one start: a wait knows only odd from
    // even, and a warp can be one product behind the others, but never two.
    auto o_before = [&](int t) {
      if (t > 0) wait_together(&sh->o_done, (uint32_t)(t - 1) & 1u);
    };
    cp_async_wait<0>();                                    // this thread's part of Q is there, and visible to the products
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sh->q_full);
    for (int t = 0; t < n_tiles; ++t) {
      const uint32_t ts = tmem + lanes + (uint32_t)(t & 1) * kWsKeys;
      const int j0 = k0 + t * kWsKeys;
      wait_together(&sh->s_full[t & 1], (uint32_t)(t >> 1) & 1u);
      tc_fence_after();
      if (any) {
        float s[kWsKeys];
        {
          uint32_t v[kWsKeys];
          tmem_ld32(ts, v);
          tmem_ld32(ts + 32u, v + 32);
          tmem_ld_wait();
          const float* b = BIAS ? brow - j0 : nullptr;
#pragma unroll
          for (int c = 0; c < kWsKeys; ++c) {
            if constexpr (CAP) s[c] = fmaf(ws_rcp(ws_exp2(__uint_as_float(v[c]) * c1) + 1.f), c2, BIAS ? b[-c] : cap);   // cap * tanh(.) = cap - 2 cap / (e^(2.) + 1)
            else s[c] = BIAS ? fmaf(__uint_as_float(v[c]), c1, b[-c]) : __uint_as_float(v[c]) * c1;
          }
        }
        const int lo = low - j0, hi = p - j0;
        if (!__all_sync(0xffffffffu, lo <= 0 && hi >= kWsKeys - 1)) {
#pragma unroll
          for (int c = 0; c < kWsKeys; ++c) s[c] = c >= lo && c <= hi ? s[c] : -INFINITY;
        }
        float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
        for (int c = 4; c < kWsKeys; c += 4) {
#pragma unroll
          for (int e = 0; e < 4; ++e) mx[e] = fmaxf(mx[e], s[c + e]);
        }
        const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        const bool grow = top > m_ref + 8.f;               // also the first finite maximum of a row
        const bool rescale = __any_sync(0xffffffffu, grow);
        float f = 1.f;
        if (grow) {
          f = ws_exp2(m_ref - top);
          l *= f;
          m_ref = top;
        }
        const float ms = m_ref == -INFINITY ? 0.f : m_ref;   // a row that sees nothing yet
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < kWsKeys; c += 16) {
          uint32_t hi16[8], lo16[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float p0 = ws_exp2(s[c + 2 * e] - ms), p1 = ws_exp2(s[c + 2 * e + 1] - ms);
            const uint32_t up = pack_bf16(p0, p1);
            const float2 u = unpack_bf16(up);
            hi16[e] = up;
            lo16[e] = pack_bf16(p0 - u.x, p1 - u.y);
            sum[e & 1] += p0;
            sum[2 + (e & 1)] += p1;
          }
          tmem_st8(ts + (uint32_t)(c / 2), hi16);
          tmem_st8(ts + 32u + (uint32_t)(c / 2), lo16);
        }
        l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
        if (t > 0 && rescale) {
          o_before(t);
          tc_fence_after();
#pragma unroll 1
          for (int c0 = 0; c0 < D; c0 += 32) {
            uint32_t o[32];
            tmem_ld32(tmem_o + lanes + (uint32_t)c0, o);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 32; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * f);
            tmem_st32(tmem_o + lanes + (uint32_t)c0, o);
          }
        }
        tmem_st_wait();
      }
      o_before(t);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->p_ready[t & 1]);
    }
    wait_together(&sh->o_done, (uint32_t)(n_tiles - 1) & 1u);
    tc_fence_after();
    if (any) {
      const long long tr = mine.x + token;
      const int hd = kvh * rep + h;
      float inv = 1.f;
      if (a.sink != nullptr) {
        const float s0 = a.sink[hd] * kLog2e, r = fmaxf(m_ref, s0);
        inv = exp2f(m_ref - r);
        l = l * inv + exp2f(s0 - r);
      }
      inv /= l;
      auto gact = [&](float z) { return a.gate_act == 1 ? z / (1.f + __expf(-z)) : (a.gate_act == 2 ? 1.f / (1.f + __expf(-z)) : z); };
      if (a.gate != nullptr && a.gate_heads && is_row) inv *= gact(a.gate[tr * a.ldg + hd]);
      const float* gp = a.gate != nullptr && !a.gate_heads ? a.gate + tr * a.ldg + hd * D : nullptr;
#pragma unroll 1
      for (int c0 = 0; c0 < D; c0 += 32) {
        uint32_t v[32];
        tmem_ld32(tmem_o + lanes + (uint32_t)c0, v);
        tmem_ld_wait();
        float o[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) o[c] = __uint_as_float(v[c]) * inv;
        if (is_row) {
          if (gp != nullptr) {
#pragma unroll
            for (int c = 0; c < 32; ++c) o[c] *= gact(gp[c0 + c]);
          }
          if (a.out_bf16) {
            uint4* dst = reinterpret_cast<uint4*>(static_cast<bf16_t*>(a.out) + tr * a.ldo + hd * D + c0);
#pragma unroll
            for (int c = 0; c < 32; c += 8) dst[c / 8] = make_uint4(pack_bf16(o[c], o[c + 1]), pack_bf16(o[c + 2], o[c + 3]), pack_bf16(o[c + 4], o[c + 5]), pack_bf16(o[c + 6], o[c + 7]));
          } else {
            float4* dst = reinterpret_cast<float4*>(static_cast<float*>(a.out) + tr * a.ldo + hd * D + c0);
#pragma unroll
            for (int c = 0; c < 32; c += 4) dst[c / 4] = make_float4(o[c], o[c + 1], o[c + 2], o[c + 3]);
          }
        }
        __syncwarp();   // the next load of tensor memory wants the whole warp
      }
    }
    tc_fence_before();
  }
  __syncwarp();
  __syncthreads();
  if (warp == 4) tmem_dealloc<1>(tmem, 256);
}

static int ws_smem(int d, int table) { return 4 * (d / 64) * kWsBox + (d / 64) * kWsRows * 128 + table + kWsTail; }
static int ws_table(bool bias, int window, int rep) { return bias ? (ws_bias_pitch(window, rep) * rep * 4 + 15) / 16 * 16 : 0; }

// Shapes this kernel takes (the alignment of the output is what its 16-byte accesses want), where it is the faster one. A CTA of it costs some 5 us before
// its first tile, so a row has to see enough keys: at widths of 128 from 64 keys on (64 keys 0.52 to 0.93 of the mma.sync kernel's time, 32 keys up to
// 1.34), at widths of 64, whose tiles are shorter, from 192 on (0.54 to 1.03; 128 keys up to 1.20). Steps of several waves of CTAs would gain from 64 keys on
// there (0.65 to 0.85), but the two kernels round differently, and a request's rows must not depend on what else is in the step.
bool window_sm100_ok(int H, int G, int d, int dv, int maps, int keep_first, int page_size, int n_items, int window, int chunk, const float* bias, const void* out,
                     long long ldo) {
  const int rep = H / G, reach = window < chunk ? window : chunk;
  return (d == 64 || d == 128) && dv == d && maps == 1 && keep_first == 0 && page_size % kWsKeys == 0 && rep <= 64 && ldo % 8 == 0 &&
         reinterpret_cast<uintptr_t>(out) % 16 == 0 && reach >= (d == 128 ? 64 : 192) &&
         (long long)n_items * G < (1ll << 31) && (bias == nullptr || (window <= 16384 && ws_smem(d, ws_table(true, window, rep)) <= 220 * 1024));
}

template <int D, bool CAP, bool BIAS>
static int ws_launch(const WinSmArgs& a, cudaStream_t st) {
  static bool done[kMaxDevices] = {};
  const int dev = cur_device();
  if (!done[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(window_attn_sm100_kernel<D, CAP, BIAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e != cudaSuccess) return set_error(OMC_ERR_CUDA, cudaGetErrorString(e));
    done[dev] = true;
  }
  window_attn_sm100_kernel<D, CAP, BIAS><<<(unsigned)a.n_items * a.G, kWsThreads, ws_smem(D, a.table), st>>>(a);
  return check_launch("omc_window_attn_mma");
}

int window_sm100(const void* q, long long ldq, int T, int H, int G, int d, const void* pool, const int32_t* bt, int max_pages, int page_size, const int32_t* items,
                 int n_items, int window, int chunk, float scale, float softcap, const float* bias, const float* sink, const float* gate, long long ldg, int gate_act,
                 int gate_heads, void* out, int out_dt, long long ldo, cudaStream_t st) {
  const int rep = H / G;
  WinSmArgs a{static_cast<const bf16_t*>(q), ldq, static_cast<const bf16_t*>(pool), bt, items, bias, sink, gate, ldg, gate_act, gate_heads, out, ldo, out_dt == OMC_DT_BF16, n_items, max_pages, page_size, H, G, window, chunk, 64 / rep,
              ws_table(bias != nullptr, window, rep), scale, softcap, nullptr};
  int rc = step_failure_word(&a.failed);
  if (rc != OMC_OK) return rc;
#define OMC_WS(CAP, BIAS) (d == 64 ? ws_launch<64, CAP, BIAS>(a, st) : ws_launch<128, CAP, BIAS>(a, st))
  if (softcap > 0.f) return bias != nullptr ? OMC_WS(true, true) : OMC_WS(true, false);
  return bias != nullptr ? OMC_WS(false, true) : OMC_WS(false, false);
#undef OMC_WS
}

int window_sm100_failures(unsigned int* n) { return cudaMemcpyFromSymbol(n, g_window_failures, sizeof(*n)) == cudaSuccess ? OMC_OK : OMC_ERR_CUDA; }

}  // namespace omc
