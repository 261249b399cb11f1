// Latent attention on tcgen05 / TMEM (bf16; the work list of omc_latent_attn_mma, latent widths that are a multiple of 128 up to 512,
// pages of a multiple of 64 rows). Everything else stays with the mma.sync kernel of latent_attention.cu.
//
// One CTA per item: up to NR = 16 / 32 / 64 rows ((token, head) pairs) against keys in tiles of 128. A key row is 576 numbers wide and its
// first 512 are the value, so an accumulator with the rows on the 128 lanes of TMEM would need all 512 columns for the output alone.
// Here both products are TRANSPOSED: keys and value dimensions lie on the lanes, rows on the columns,
//     S^T [128 keys, NR] = K Q^T          A = the key tile, K-major              B = Q, K-major
//     O^T [r, NR]       += V^T P^T        A = the SAME shared-memory tile read MN-major (r / 128 accumulators)   B = P^T
// which needs (r / 128 + 1) NR columns, lets one staged tile serve both products, and lets a decode step (16 heads of one token) run at
// N = 16 instead of on a mostly empty row tile.
//   warps 0, 10  Q once, by TMA; per tile the 64-column chunks of two boxes of 64 keys, by cp.async: the pages alone say where a row lies, and nobody has to
//                know the rows of the pool (a tensor map of more rows than there are let copies touch what lies behind it). The two chunks (the last
//                time with the rotated one) that hold 128 value dimensions share a barrier, at which each thread's copies arrive by themselves:
//                scores start with the first pair, and a pair is refilled as soon as the output product that reads it is done
//   warp 1       MMA issuer (one thread)
//   warps 2..9   softmax: thread = one key x half the rows. Maxima over keys are maxima over lanes: a transposing butterfly leaves every
//                lane with one row's maximum. The reference maximum of a row only moves when it grew by more than 2^8; the output
//                accumulators are then rescaled in TMEM. Sums stay per thread until the end.
//                P^T goes to shared memory as the B operand, as two bf16 numbers per probability (its rounding and what that left, 2^-18 of it
//                together): with one, tiles of 128 keys and longer key ranges gave 1 to 44 % more error than the mma.sync kernel's tiles of 64. Where
//                Q and the key tile fill shared memory (64 rows, r = 512) half of it takes the places of the rotated chunks, which the scores
//                have consumed.
// What bounds it: shared memory holds one key tile, so a tile of 8000 cycles is a load that only the output products overlap (3100), 100 instructions
// on the tensor pipe (36 for the scores), and one softmax pass over 8192 scores (2200). 16 heads, latents of 512 + 64 (key tiles by TMA / the mma.sync
// kernel in brackets): portions of 1024, 777, 1024 behind 1024 and 301 rows 244 us (260 / 722); 4 x 1024 rows of 32 heads 460 us (495 / 1136); 2048 rows
// 193 us (202 / 653); a decode step of 32 rows over 700 to 2100 keys, merge included, 34 us (33 / 79). By cp.async with a wait and a fence of the load
// warps in front of every pair: 359, 660, 297 and 52 us.
#include "latent_decode.cuh"
#include "sm100_step.cuh"

namespace omc {

constexpr int kKT = 128;                    // keys per tile
constexpr int kChunkBytes = kKT * 128;      // 64 columns of a key tile
constexpr int kLsSoftmax = 256, kLsLoad = 64, kLsThreads = kLsSoftmax + 32 + kLsLoad, kLsMaxRows = 64;

static __device__ unsigned int g_latent_failures;   // waits that ran out

struct LatSmArgs {
  const bf16_t* q;        // q_rows rows; with the pool, for the copies by cp.async
  const bf16_t* pool;
  long long q_rows;
  const int32_t* bt;
  const int32_t* items;   // as LatMmaArgs of latent_attention.cu; NULL: one row per request, at (slot, pos), in `parts` ranges of its keys
  const int32_t* pos;
  const int32_t* slot;
  int parts;
  const float* sink;
  void* out;
  float* ws_o;
  float* ws_ml;
  const float* gate;
  long long ldg;
  int window, max_pages, page_size, H, r, D, nc;   // nc: 64-column chunks of a row
  int p_at[4];                                     // P^T behind Q, in bytes: its upper and its lower numbers, 64 keys each
  bool reload_q;                                   // P^T lies where the last chunk of Q does
  int tmem_cols;
  float scale_log2;
  unsigned int* failed;
};

struct LatSmShared {
  uint64_t q_full, s_full, p_ready, mma_done, full[4], o_done[4];
  uint32_t tmem, dead, rescale[2];
  alignas(16) float mref[kLsMaxRows];
  alignas(16) float fac[kLsMaxRows];
  float part[4][kLsMaxRows];   // reference maxima, rescaling factors, the lane quarters' maxima / sums
};

__device__ __forceinline__ float ls_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Arrives (one of the counted arrivals) once the copies that this thread has issued so far are there.
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) { asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory"); }
__device__ __forceinline__ void ls_softmax_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kLsSoftmax) : "memory"); }

// v[c]: this lane's value of column c. Returns the reduction over the 32 lanes of column lane / (32 / NC) (v is overwritten).
template <int NC, typename Op>
__device__ __forceinline__ float ls_columns(float (&v)[NC], int lane, Op op) {
  int off = 16;
#pragma unroll
  for (int cur = NC; cur > 1; cur >>= 1, off >>= 1) {
    const bool up = lane & off;
#pragma unroll
    for (int i = 0; i < cur / 2; ++i) {
      const float other = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + cur / 2], off);
      v[i] = op(up ? v[i + cur / 2] : v[i], other);
    }
  }
#pragma unroll
  for (; off > 0; off >>= 1) v[0] = op(v[0], __shfl_xor_sync(0xffffffffu, v[0], off));
  return v[0];
}

template <int NC>
__device__ __forceinline__ void ls_tmem_ld(uint32_t addr, uint32_t* v) {
  if constexpr (NC == 32) tmem_ld32(addr, v);
  else if constexpr (NC == 16) tmem_ld16(addr, v);
  else
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(addr)
                 : "memory");
}
template <int NC>
__device__ __forceinline__ void ls_tmem_st(uint32_t addr, const uint32_t* v) {
  if constexpr (NC == 32) tmem_st32(addr, v);
  else if constexpr (NC == 16) tmem_st16(addr, v);
  else tmem_st8(addr, v);
}

template <int NR, typename TO>
__global__ void __launch_bounds__(kLsThreads, 1) latent_attn_sm100_kernel(const __grid_constant__ CUtensorMap tm_q, LatSmArgs a) {
  constexpr int NC = NR / 2;                 // rows per softmax thread
  constexpr int QCHUNK = NR * 128;           // bytes of a 64-column chunk of Q
  extern __shared__ uint8_t ls_raw[];
  __shared__ LatSmShared shared;
  LatSmShared* sh = &shared;
  uint8_t* base = ls_raw + ((1024u - (smem_u32(ls_raw) & 1023u)) & 1023u);
  uint8_t* qs = base;                        // [nc][NR][128 B]
  uint8_t* ks = base + a.nc * QCHUNK;        // [nc][128][128 B]
  if (threadIdx.x == 32) tma_prefetch_desc(&tm_q);
  int first_row, n_tok = 1, slot, first_pos, kb, k_end, part;
  if (a.items != nullptr) {
    const int32_t* it = a.items + blockIdx.x * 8;
    first_row = it[0], n_tok = it[1], slot = it[2], first_pos = it[3], kb = it[4], part = it[6];
    k_end = min(it[5], first_pos + n_tok);
  } else {
    first_row = blockIdx.x / a.parts;
    const int i = blockIdx.x - first_row * a.parts;
    slot = a.slot[first_row], first_pos = a.pos[first_row];
    latent_decode_range(first_pos, a.window, a.parts, i, kb, k_end);
    part = a.parts > 1 ? (int)blockIdx.x : -1;
  }
  const int n_rows = n_tok * a.H;
  const int k0 = kb & ~63;                   // boxes of 64 keys start where pages may
  const int n_tiles = k_end > kb ? (k_end - k0 + kKT - 1) / kKT : 0;
  const int nm = a.r >> 7;                   // 128-dimension tiles of the output
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const WaitReport report{&sh->dead, &g_latent_failures, a.failed};
  auto wait = [&](uint64_t* bar, uint32_t parity) { return wait_bounded(bar, parity, report); };
  auto drain = [&](uint64_t* bar, uint32_t parity) { drain_bounded(bar, parity, report); };
  const int32_t* bt = a.bt + (long long)slot * a.max_pages;
  // The last chunk ends where the row does: its box starts at D - 64 and repeats columns of the chunk before where D is no multiple of 64.
  auto chunk_col = [&](int c) { return c == a.nc - 1 ? a.D - 64 : c * 64; };
  // rows of the pool where the two boxes of tile t start (looked up a tile ahead: a lookup takes as long as 20 KB of the copies)
  auto box_rows = [&](int t, int (&row)[2]) {
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int j = k0 + t * kKT + 64 * b;
      row[b] = j < k_end ? bt[j / a.page_size] * a.page_size + j % a.page_size : -1;
    }
  };
  // The chunks of barrier g by the load warps: eight lanes per 128 bytes of a row, as the 128-byte swizzle has them, eight rows at a time. Rows that are no keys of
  // this item become zeros: what the cache holds there must not meet a product.
  static_assert(kLsLoad == 64, "eight rows at a time");
  const bool loads = warp == 0 || warp == kLsThreads / 32 - 1;
  const int piece = lane & 7, r0 = (warp == 0 ? lane : lane + 32) >> 3, swizzled = r0 * 128 + ((piece ^ r0) << 4);
  auto copy_pair = [&](int t, const int (&row)[2], int g) {
    const int c1 = g == nm - 1 ? a.nc : 2 * g + 2, j = k0 + t * kKT;
    const long long step = 8LL * a.D;
    for (int c = 2 * g; c < c1; ++c) {
      uint8_t* at = ks + c * kChunkBytes + swizzled;
#pragma unroll
      for (int b = 0; b < 2; ++b, at += kChunkBytes / 2) {
        const bf16_t* src = a.pool + (long long)(max(row[b], 0) + r0) * a.D + chunk_col(c) + piece * 8;
        if (j + 64 * b >= kb && j + 64 * b + 64 <= k_end) {
#pragma unroll
          for (int i = 0; i < 8; ++i) cp_async16(at + i * 1024, src + i * step, true);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int key = j + 64 * b + i * 8 + r0;
            cp_async16(at + i * 1024, src + i * step, key >= kb && key < k_end);
          }
        }
      }
    }
    if (t > 0 && a.reload_q && g == nm - 1) {
      const bf16_t* src = a.q + ((long long)first_row * a.H + r0) * a.D + chunk_col(a.nc - 1) + piece * 8;
#pragma unroll
      for (int i = 0; i < NR / 8; ++i) cp_async16(qs + (a.nc - 1) * QCHUNK + swizzled + i * 1024, src + i * step, (long long)first_row * a.H + r0 + i * 8 < a.q_rows);
    }
    cp_async_arrive(&sh->full[g]);           // once this thread's copies so far are there
  };
  if (tid >= 64 && tid < 64 + kLsMaxRows) sh->mref[tid - 64] = -INFINITY;
  if (tid == 0) {
    mbar_init(&sh->q_full, 1);
    mbar_init(&sh->s_full, 1);
    mbar_init(&sh->p_ready, kLsSoftmax / 32);
    mbar_init(&sh->mma_done, 1);
    for (int m = 0; m < 4; ++m) {
      mbar_init(&sh->full[m], kLsLoad);
      mbar_init(&sh->o_done[m], 1);
    }
    sh->dead = 0u;
    sh->rescale[0] = sh->rescale[1] = 0u;
    fence_barrier_init();
    fence_proxy_async();
    if (n_tiles > 0) {
      mbar_arrive_expect_tx(&sh->q_full, a.nc * QCHUNK);
      for (int c = 0; c < a.nc; ++c) tma_load_3d(qs + c * QCHUNK, &tm_q, &sh->q_full, chunk_col(c), first_row * a.H, 0);
    }
  }
  int row[2] = {-1, -1};                     // of the tile that is loaded next
  if (loads && n_tiles > 0) {                // the first tile is on its way while tensor memory is allocated
    box_rows(0, row);
    __syncwarp();
    asm volatile("bar.sync 2, %0;" ::"n"(kLsLoad) : "memory");   // the barriers are there
    for (int g = 0; g < nm; ++g) copy_pair(0, row, g);
  }
  if (warp == 1) {
    __syncwarp();
    tmem_alloc<1>(&sh->tmem, a.tmem_cols);
    tmem_relinquish<1>();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem, tmem_s = tmem + nm * NR;

  if (loads) {
    bool go = true;
    for (int t = 1; go && t < n_tiles; ++t) {
      box_rows(t, row);
      for (int g = 0; g < nm; ++g) {
        go = wait_bounded_warp(&sh->o_done[g], (t - 1) & 1, report);
        if (!go) break;
        copy_pair(t, row, g);
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");   // nothing is on its way any more when these threads leave
    if (tid == 0 && n_tiles > 0) drain(&sh->q_full, 0);
  } else if (warp == 1) {
    if (elect_one() && n_tiles > 0) {
      constexpr uint32_t idesc_s = make_idesc_bf16_major(128, NR, 0, 0);
      constexpr uint32_t idesc_o = make_idesc_bf16_major(128, NR, 1, NR == 64 ? 1 : 0);
      const uint64_t dk0 = make_sw128_kmajor_desc(smem_u32(ks)), dq0 = make_sw128_kmajor_desc(smem_u32(qs));
      const uint64_t dv0 = make_sw128_mnmajor_desc(smem_u32(ks), kChunkBytes, 1024);
      uint64_t dp[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t at = smem_u32(base) + a.p_at[i];
        dp[i] = NR == 64 ? make_sw128_mnmajor_desc(at, 1024, 1024) : make_sw128_kmajor_desc(at);
      }
      const int repeated = (a.nc * 64 - a.D) >> 4;   // steps of 16 that the last chunk has in common with the one before
      bool go = wait(&sh->q_full, 0);
      for (int t = 0; go && t < n_tiles; ++t) {
        for (int g = 0; g < nm; ++g) {
          go = wait(&sh->full[g], t & 1);
          if (!go) break;
          fence_proxy_async();               // what the load warps' copies wrote is seen by the products
          tc_fence_after();
          const int c1 = g == nm - 1 ? a.nc : 2 * g + 2;
          for (int c = 2 * g; c < c1; ++c) {
            const uint64_t dk = dk0 + (uint64_t)(c * (kChunkBytes >> 4)), dq = dq0 + (uint64_t)(c * (QCHUNK >> 4));
            const int first = c == a.nc - 1 ? repeated : 0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (k >= first) umma_bf16<1>(tmem_s, dk + 2 * k, dq + 2 * k, idesc_s, (c | k) != 0 ? 1u : 0u);
          }
        }
        if (!go) break;
        umma_commit(&sh->s_full);            // also: the output products of the tile before are done
        go = wait(&sh->p_ready, t & 1);
        if (!go) break;
        tc_fence_after();
        for (int m = 0; m < nm; ++m) {
          const uint64_t dv = dv0 + (uint64_t)(m * (2 * kChunkBytes >> 4));
#pragma unroll
          for (int k = 0; k < kKT / 16; ++k)
#pragma unroll
            for (int low = 0; low < 2; ++low)
              umma_bf16<1>(tmem + m * NR, dv + (uint64_t)(k * 128), dp[2 * low + (k >> 2)] + (uint64_t)((NR == 64 ? 128 : 2) * (k & 3)), idesc_o,
                           (t | k | low) != 0 ? 1u : 0u);
          umma_commit(&sh->o_done[m]);
        }
      }
      umma_commit(&sh->mma_done);
      drain(&sh->mma_done, 0);        // every product that was issued is done
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2,   // TMEM lanes go by warp % 4
               key_lane = quarter * 32 + lane, c0 = half * NC;
    const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
    const int stid = tid - 64;
    float l[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) l[c] = 0.f;
    // the lanes of a warp may leave a wait one by one, and accesses to tensor memory are the warp's as a whole; whether the phase came is not asked
    auto wait_together = [&](uint64_t* bar, uint32_t parity) {
      wait(bar, parity);
      __syncwarp();
    };
    for (int t = 0; t < n_tiles; ++t) {
      const int j0 = k0 + t * kKT, key = j0 + key_lane;
      wait_together(&sh->s_full, t & 1);
      tc_fence_after();
      // a tile that every row of the item sees in full needs no mask
      const bool whole = j0 >= kb && j0 + kKT <= k_end && j0 + kKT - 1 <= first_pos && (long long)j0 >= (long long)first_pos + n_tok - a.window;
      // the rows that see this thread's key: those of tokens at or behind it, as far as the window reaches
      const bool is_key = key >= kb && key < k_end;
      const int see0 = (is_key ? max(key - first_pos, 0) : kLsMaxRows) * a.H - c0;
      const int see1 = (int)min((long long)kLsMaxRows, (long long)key - first_pos + a.window) * a.H - c0;
      float s[NC];
      auto load_scores = [&] {               // twice per tile: the maxima destroy them, and holding both copies would cost 32 registers
        uint32_t v[NC];
        ls_tmem_ld<NC>(tmem_s + lanes + c0, v);
        tmem_ld_wait();
        if (whole) {
#pragma unroll
          for (int c = 0; c < NC; ++c) s[c] = __uint_as_float(v[c]) * a.scale_log2;
        } else {
#pragma unroll
          for (int c = 0; c < NC; ++c) s[c] = c >= see0 && c < see1 ? __uint_as_float(v[c]) * a.scale_log2 : -INFINITY;
        }
      };
      load_scores();
      const float mx = ls_columns<NC>(s, lane, [](float x, float y) { return fmaxf(x, y); });
      if (lane % (32 / NC) == 0) sh->part[quarter][c0 + lane / (32 / NC)] = mx;
      ls_softmax_sync();
      if (stid < NR) {
        const float now = fmaxf(fmaxf(sh->part[0][stid], sh->part[1][stid]), fmaxf(sh->part[2][stid], sh->part[3][stid]));
        const float old = sh->mref[stid];
        if (now > old + 8.f) {               // also the first finite maximum of a row
          sh->fac[stid] = ls_exp2(old - now);
          sh->mref[stid] = now;
          sh->rescale[t & 1] = 1u;
        } else {
          sh->fac[stid] = 1.f;
        }
      }
      if (stid == kLsSoftmax - 1) sh->rescale[(t + 1) & 1] = 0u;
      ls_softmax_sync();
      if (sh->rescale[t & 1] && t > 0) {
        float f[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) f[c] = sh->fac[c0 + c], l[c] *= f[c];
        for (int m = 0; m < nm; ++m) {
          uint32_t v[NC];
          ls_tmem_ld<NC>(tmem + lanes + m * NR + c0, v);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < NC; ++c) v[c] = __float_as_uint(__uint_as_float(v[c]) * f[c]);
          ls_tmem_st<NC>(tmem + lanes + m * NR + c0, v);
        }
        tmem_st_wait();
      }
      load_scores();
      uint8_t* const hi_at = base + (quarter < 2 ? a.p_at[0] : a.p_at[1]);
      uint8_t* const lo_at = base + (quarter < 2 ? a.p_at[2] : a.p_at[3]);
#pragma unroll
      for (int c = 0; c < NC; c += 8) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int i = 0; i < 8; i += 4) {
          const float4 m4 = *reinterpret_cast<const float4*>(&sh->mref[c0 + c + i]);
          const float m[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
          for (int e = 0; e < 4; e += 2) {
            const float p0 = ls_exp2(s[c + i + e] - (m[e] == -INFINITY ? 0.f : m[e])), p1 = ls_exp2(s[c + i + e + 1] - (m[e + 1] == -INFINITY ? 0.f : m[e + 1]));
            const uint32_t h = pack_bf16(p0, p1);
            const float2 up = unpack_bf16(h);
            hi[(i + e) / 2] = h;
            lo[(i + e) / 2] = pack_bf16(p0 - up.x, p1 - up.y);
            l[c + i + e] += p0;
            l[c + i + e + 1] += p1;
          }
        }
        if constexpr (NR == 64) {            // [key][64 rows]: MN-major
          const int at = (key_lane & 63) * 128 + (((half * (NC / 8) + c / 8) ^ (key_lane & 7)) << 4);
          *reinterpret_cast<uint4*>(hi_at + at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(lo_at + at) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        } else {                             // [row][64 keys] twice: K-major
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int row = c0 + c + i, at = (key_lane & 7) * 2 + row * 128 + ((((key_lane & 63) >> 3) ^ (row & 7)) << 4);
            *reinterpret_cast<uint16_t*>(hi_at + at) = (uint16_t)(hi[i / 2] >> (16 * (i & 1)));
            *reinterpret_cast<uint16_t*>(lo_at + at) = (uint16_t)(lo[i / 2] >> (16 * (i & 1)));
          }
        }
      }
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->p_ready);
    }
    // ---- the sums over all keys, then the output
    const float mine = ls_columns<NC>(l, lane, [](float x, float y) { return x + y; });
    if (lane % (32 / NC) == 0) sh->part[quarter][c0 + lane / (32 / NC)] = mine;
    ls_softmax_sync();
    if (stid < NR) {
      const float sum = (sh->part[0][stid] + sh->part[1][stid]) + (sh->part[2][stid] + sh->part[3][stid]), m = sh->mref[stid];
      if (part >= 0) {
        float* ml = a.ws_ml + ((long long)part * kLsMaxRows + stid) * 2;
        ml[0] = m, ml[1] = sum;
        sh->fac[stid] = 1.f;
      } else if (stid < n_rows) {
        const int h = stid % a.H;
        float f = 1.f / (a.sink != nullptr ? sum + exp2f(a.sink[h] * 1.4426950408889634f - m) : sum);
        if (a.gate != nullptr) f *= 1.f / (1.f + expf(-a.gate[(long long)(first_row + stid / a.H) * a.ldg + h]));
        sh->fac[stid] = f;
      }
    }
    ls_softmax_sync();
    if (n_tiles > 0) wait_together(&sh->o_done[nm - 1], (n_tiles - 1) & 1);
    tc_fence_after();
    for (int m = 0; m < nm; ++m) {
      uint32_t v[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) v[c] = 0u;
      if (n_tiles > 0) {
        ls_tmem_ld<NC>(tmem + lanes + m * NR + c0, v);
        tmem_ld_wait();
      }
      const int dim = m * 128 + key_lane;
      if (part >= 0) {
        float* dst = a.ws_o + ((long long)part * kLsMaxRows + c0) * a.r + dim;
#pragma unroll
        for (int c = 0; c < NC; ++c)
          if (c0 + c < n_rows) dst[(long long)c * a.r] = __uint_as_float(v[c]);
      } else {
        TO* dst = static_cast<TO*>(a.out) + ((long long)first_row * a.H + c0) * a.r + dim;
#pragma unroll
        for (int c = 0; c < NC; ++c)
          if (c0 + c < n_rows) stf(dst + (long long)c * a.r, __uint_as_float(v[c]) * sh->fac[c0 + c]);
      }
    }
    tc_fence_before();
  }
  __syncwarp();
  __syncthreads();
  if (warp == 1) tmem_dealloc<1>(tmem, a.tmem_cols);
}

constexpr int kLsSmemMax = 227 * 1024;
// Shared memory of a launch (0: none fits) and where P^T lies: behind the key tile, or, where that fills it, half of it in the places of the last
// chunks of the key tile and of Q, which only the scores read (Q's is then loaded again with the next tile).
static int ls_smem(int nr, int r, int D, LatSmArgs* a) {
  const int nc = (D + 63) / 64, qc = nr * 128, q = nc * qc, k = nc * kChunkBytes;
  const int slack = 1024 + (int)sizeof(LatSmShared) + 256;
  if (q + k + 4 * qc + slack <= kLsSmemMax) {
    for (int i = 0; i < 4; ++i) a->p_at[i] = q + k + i * qc;
    a->reload_q = false;
    return q + k + 4 * qc + 1024;
  }
  if (D > r && 2 * qc <= kChunkBytes && q + k + qc + slack <= kLsSmemMax) {
    a->p_at[0] = q + k - kChunkBytes, a->p_at[1] = a->p_at[0] + qc, a->p_at[2] = q + k, a->p_at[3] = q - qc;
    a->reload_q = true;
    return q + k + qc + 1024;
  }
  return 0;
}

// Shapes this kernel takes. max_rows: the most rows an item has.
bool latent_sm100_ok(int max_rows, int r, int dr, int page_size, const void* q, const void* pool) {
  LatSmArgs a;
  return max_rows <= kLsMaxRows && r % 128 == 0 && r <= 512 && dr <= 64 && dr % 16 == 0 && page_size % 64 == 0 &&
         reinterpret_cast<uintptr_t>(q) % 16 == 0 && reinterpret_cast<uintptr_t>(pool) % 16 == 0 && ls_smem(max_rows <= 16 ? 16 : (max_rows <= 32 ? 32 : 64), r, r + dr, &a) > 0;
}

template <int NR, typename TO>
static int ls_launch(const CUtensorMap& tq, const LatSmArgs& a, int n_items, int smem, cudaStream_t st) {
  static bool done[kMaxDevices] = {};
  const int dev = cur_device();
  if (!done[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(latent_attn_sm100_kernel<NR, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, kLsSmemMax - (int)sizeof(LatSmShared) - 128);
    if (e != cudaSuccess) return set_error(OMC_ERR_CUDA, cudaGetErrorString(e));
    done[dev] = true;
  }
  latent_attn_sm100_kernel<NR, TO><<<n_items, kLsThreads, smem, st>>>(tq, a);
  return check_launch("omc_latent_attn_mma");
}

int latent_sm100(const void* q, long long q_rows, int H, int r, int dr, const void* pool, const int32_t* bt, int max_pages, int page_size, const int32_t* items,
                 const LatentDecodeRows& rows, int n_items, int max_rows, const float* sink, int window, const float* gate, long long ldg, float scale, void* out, int out_dt, float* ws_o,
                 float* ws_ml, cudaStream_t st) {
  const int D = r + dr, nr = max_rows <= 16 ? 16 : (max_rows <= 32 ? 32 : 64);
  LatSmArgs a{static_cast<const bf16_t*>(q), static_cast<const bf16_t*>(pool), q_rows, bt, items, rows.pos, rows.slot, rows.parts, sink, out, ws_o, ws_ml, gate, ldg, window, max_pages, page_size, H, r, D,
              (D + 63) / 64, {}, false, 0, scale * 1.4426950408889634f, nullptr};
  const int smem = ls_smem(nr, r, D, &a);
  const int cols = (r / 128 + 1) * nr;
  a.tmem_cols = cols <= 32 ? 32 : (cols <= 64 ? 64 : (cols <= 128 ? 128 : (cols <= 256 ? 256 : 512)));
  CUtensorMap tq;
  int rc = step_failure_word(&a.failed);
  if (rc == OMC_OK) rc = step_tensor_map(&tq, q, D, q_rows, D, 1, 0, nr);
  if (rc != OMC_OK) return rc;
  const bool b = out_dt == OMC_DT_BF16;
  if (nr == 16) return b ? ls_launch<16, bf16_t>(tq, a, n_items, smem, st) : ls_launch<16, float>(tq, a, n_items, smem, st);
  if (nr == 32) return b ? ls_launch<32, bf16_t>(tq, a, n_items, smem, st) : ls_launch<32, float>(tq, a, n_items, smem, st);
  return b ? ls_launch<64, bf16_t>(tq, a, n_items, smem, st) : ls_launch<64, float>(tq, a, n_items, smem, st);
}

int latent_sm100_failures(unsigned int* n) { return cudaMemcpyFromSymbol(n, g_latent_failures, sizeof(*n)) == cudaSuccess ? OMC_OK : OMC_ERR_CUDA; }

}  // namespace omc
