// Softmax attention in fp32 over a paged cache for the true-fp32 path (omc_latent_attn, omc_window_attn): the query heads of a token that read the same keys share
// them. The plain kernels of latent_attention.cu and window_attention.cu, a CTA per (row, head) whose warps read every key from global memory for one query, stay for
// bf16 storage, several score maps, kept first keys and the widths and alignments that are not taken here.
//
// A CTA has eight query heads of a token and one key/value head (four where there are no more than four), and a warp per head. Keys (and values) go through shared
// memory in tiles of 32 from the first visible one on, two buffers; the page of a tile is looked up a tile before its copy.
//   scores   a warp has four keys (eight in the smaller CTA) and all heads; its lanes split the key width, 16 bytes each, LD of them to a key, and a transposing
//            butterfly leaves every lane the sum of one (key, head)
//   softmax  a warp has a head, a lane a key: scale, soft cap, distance bias, mask, running maximum
//   values   a thread has four columns of all heads, heads in packed pairs; threads beyond the columns split the keys of a tile, and their partial outputs meet
//            in shared memory at the end
// What bounds it: the shared-memory reads of both products behind three barriers a tile. Half the lanes to a key need 128 registers instead of 177, which lets two CTAs
// share an SM where two fit its shared memory: 376 rows x 8 heads over rows of 256 + 64 50 us (63 by all lanes); where one fits (512 + 64) all lanes, 146 us (159).
// In us, the plain kernels in brackets, all keys / a window of 16: 376 rows of one prompt, latents 8 heads 256 + 64 50 (206) / 10 (24), 16 heads 512 + 64 146 (552) /
// 32 (67); 28 heads over 4 of 128 + 128 101 (318) / 23 (48), 8 over 4 of 64 + 64 46 (92) / 11 (14). 64 rows of 700 keys: 58 (88), 81 (520), 58 (416), 34 (74).
// Few rows have no CTAs to fill the chip, and then a tile's chain of barriers and copies counts: attn_few_rows_kernel.
#include "seq_common.cuh"

namespace omc {

constexpr int kArKeys = 32;   // of a tile

struct AttnRowsArgs {
  const float* q;
  long long ldq;
  const float* pool;
  const int32_t* bt;
  const int32_t* pos;
  const int32_t* slot;
  const float* bias;   // [window][H] or NULL
  const float* sink;
  const float* gate;
  long long ldg;
  int gate_act, gate_heads;
  void* out;
  long long ldo;
  int T, H, G, d, dv, width, voff, max_pages, page_size, window, chunk, head_blocks;   // width: floats per key row of a tile; voff: where the values lie in it
  int koff_g, voff_g, row_w;   // in a cached row: head g's keys at g * koff_g, its values at voff_g + g * dv (voff_g < 0: in the keys); floats of a cached row
  float scale, softcap;
};

typedef unsigned long long ar_f2;
__device__ __forceinline__ void ar_fma(ar_f2& acc, ar_f2 x, ar_f2 y) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(y)); }
__device__ __forceinline__ ar_f2 ar_mul(ar_f2 x, ar_f2 y) {
  ar_f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
  return r;
}
__device__ __forceinline__ ar_f2 ar_both(float x) {
  ar_f2 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void ar_split(ar_f2 v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ void ar_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}

// LD: lanes that share a key (4 ROWS, or half of that where a key is at most 2 * 4 ROWS wide)
template <int ROWS, int LD, typename TY>
__global__ void __launch_bounds__(ROWS * 32) attn_rows_kernel(AttnRowsArgs a) {
  constexpr int kArRows = ROWS, kArThreads = ROWS * 32, COPY = ROWS;   // COPY: threads per key row of a tile
  extern __shared__ __align__(16) float ar_sm[];   // tiles [2][32][width] | Q [ROWS][d] | scores [ROWS][33] | probabilities [32][ROWS] | per row: factor, maximum, sum
  float* const tiles = ar_sm;
  float* const qs = tiles + 2 * kArKeys * a.width;
  float* const ss = qs + kArRows * a.d;
  float* const ps = ss + kArRows * (kArKeys + 1);
  float* const sc = ps + kArKeys * kArRows;
  float* const sm = sc + kArRows;
  float* const sl = sm + kArRows;
  const int t = blockIdx.x, kvh = blockIdx.y / a.head_blocks, hb = blockIdx.y - kvh * a.head_blocks, rep = a.H / a.G;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h0 = kvh * rep + hb * ROWS, heads = min(ROWS, rep - hb * ROWS);   // this CTA's query heads
  const int p = a.pos[t], low = max(max(0, p - a.window + 1), p - p % a.chunk), n_tiles = (p - low + kArKeys) / kArKeys;
  const int32_t* bt = a.bt + (long long)a.slot[t] * a.max_pages;
  int page = -1, at = 0;   // of this thread's row of the next tile, looked up a tile ahead of its copy; -1: no key that the row sees
  auto locate = [&](int i) {
    const int j = low + i * kArKeys + tid / COPY, q = j / a.page_size;
    at = j - q * a.page_size;
    page = j <= p ? bt[q] : -1;
  };
  auto load = [&](int i) {   // rows of the last tile beyond the keys stay as they are: nothing uses their scores, and nobody reads their values
    float* row = tiles + ((i & 1) * kArKeys + tid / COPY) * a.width;
    const int c0 = (tid % COPY) * 4;
    if (page >= 0) {
      const float* src = a.pool + ((long long)page * a.page_size + at) * a.row_w;
      for (int c = c0; c < a.d; c += 4 * COPY) ar_copy16(row + c, src + kvh * a.koff_g + c);
      if (a.voff_g >= 0)
        for (int c = c0; c < a.dv; c += 4 * COPY) ar_copy16(row + a.voff + c, src + a.voff_g + kvh * a.dv + c);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  locate(0);
  for (int e = tid * 4; e < ROWS * a.d; e += kArThreads * 4) {
    if (e < heads * a.d) ar_copy16(qs + e, a.q + (long long)t * a.ldq + (long long)h0 * a.d + e);
    else *reinterpret_cast<float4*>(qs + e) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  load(0);
  if (n_tiles > 1) locate(1);
  // softmax: this warp's row
  const int h = h0 + min(warp, heads - 1);
  const float inv_cap = a.softcap > 0.f ? 1.f / a.softcap : 0.f;
  float m = -INFINITY, l = 0.f;   // l: this lane's keys
  // values: this thread's columns and share of the keys
  const int groups = (a.dv >> 2), g2 = groups <= 8 ? 8 : (groups <= 16 ? 16 : (groups <= 32 ? 32 : (groups <= 64 ? 64 : 128)));   // at most 128 groups: dv <= 512
  const int splits = kArThreads / g2, col = (tid & (g2 - 1)) * 4, split = tid / g2;
  const bool has_cols = col < a.dv;
  ar_f2 acc[kArRows / 2][4];
#pragma unroll
  for (int r = 0; r < kArRows / 2; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0ull;
  constexpr int KP = LD / ROWS, VALS = KP * kArRows, SHARE = 32 / LD;   // keys of a lane; sums of a lane before the butterfly (as many as lanes share them)
  const int sub = lane & (LD - 1), key0 = (warp * SHARE + lane / LD) * KP;

  for (int i = 0; i < n_tiles; ++i) {
    const float* tile = tiles + (i & 1) * kArKeys * a.width;
    const int j0 = low + i * kArKeys, n_keys = min(kArKeys, p - j0 + 1);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();   // this tile is there, and everyone is done with the one before
    if (i + 1 < n_tiles) load(i + 1);
    if (i + 2 < n_tiles) locate(i + 2);
    if (warp * (SHARE * KP) < n_keys) {
      ar_f2 s2[KP][kArRows];
#pragma unroll
      for (int k = 0; k < KP; ++k)
#pragma unroll
        for (int r = 0; r < kArRows; ++r) s2[k][r] = 0ull;
      for (int c = sub * 4; c < a.d; c += LD * 4) {
        ulonglong2 kv[KP];
#pragma unroll
        for (int k = 0; k < KP; ++k) kv[k] = *reinterpret_cast<const ulonglong2*>(tile + (key0 + k) * a.width + c);
#pragma unroll
        for (int r = 0; r < kArRows; ++r) {
          const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(qs + r * a.d + c);
#pragma unroll
          for (int k = 0; k < KP; ++k) {
            ar_fma(s2[k][r], kv[k].x, qv.x);
            ar_fma(s2[k][r], kv[k].y, qv.y);
          }
        }
      }
      float v[VALS];
#pragma unroll
      for (int k = 0; k < KP; ++k)
#pragma unroll
        for (int r = 0; r < kArRows; ++r) {
          float lo, hi;
          ar_split(s2[k][r], lo, hi);
          v[k * kArRows + r] = lo + hi;
        }
      int off = LD / 2;
#pragma unroll
      for (int cur = VALS; cur > 1; cur >>= 1, off >>= 1) {
        const bool up = lane & off;
#pragma unroll
        for (int i = 0; i < cur / 2; ++i) {
          const float other = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + cur / 2], off);
          v[i] = (up ? v[i + cur / 2] : v[i]) + other;
        }
      }
      ss[(sub % kArRows) * (kArKeys + 1) + key0 + sub / kArRows] = v[0];   // value `sub`: key sub / 8, row sub % 8
    }
    __syncthreads();
    {
      float s = ss[warp * (kArKeys + 1) + lane] * a.scale;
      if (a.softcap > 0.f) s = a.softcap * tanhf(s * inv_cap);
      const bool seen = lane < n_keys;
      if (a.bias != nullptr && seen) s += a.bias[(long long)(p - j0 - lane) * a.H + h];
      const float mn = fmaxf(m, seq_warp_max(seen ? s : -INFINITY));
      const float corr = m == -INFINITY ? 0.f : expf(m - mn), pj = seen && s != -INFINITY ? expf(s - mn) : 0.f;
      l = l * corr + pj;
      m = mn;
      ps[lane * kArRows + warp] = pj;
      if (lane == 0) sc[warp] = corr;
    }
    __syncthreads();
    if (has_cols) {
      const ar_f2* f = reinterpret_cast<const ar_f2*>(sc);
      if (i > 0) {
#pragma unroll
        for (int r = 0; r < kArRows / 2; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[r][c] = ar_mul(acc[r][c], f[r]);
      }
      const float* vrow = tile + a.voff + col;
#pragma unroll 4
      for (int k = split; k < n_keys; k += splits) {
        ar_f2 pr[ROWS / 2];
#pragma unroll
        for (int r = 0; r < ROWS / 2; r += 2) {
          const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(ps + k * ROWS + 2 * r);
          pr[r] = x.x, pr[r + 1] = x.y;
        }
        const float4 v = *reinterpret_cast<const float4*>(vrow + k * a.width);
        const ar_f2 vc[4] = {ar_both(v.x), ar_both(v.y), ar_both(v.z), ar_both(v.w)};
#pragma unroll
        for (int r = 0; r < kArRows / 2; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) ar_fma(acc[r][c], pr[r], vc[c]);
      }
    }
  }
  __syncthreads();   // the tiles' place is free
  float* const part = tiles;   // [splits][ROWS][dv]
  if (has_cols) {
#pragma unroll
    for (int r = 0; r < kArRows / 2; ++r) {
      float x[2][4];
#pragma unroll
      for (int c = 0; c < 4; ++c) ar_split(acc[r][c], x[0][c], x[1][c]);
#pragma unroll
      for (int i = 0; i < 2; ++i) *reinterpret_cast<float4*>(part + (split * kArRows + 2 * r + i) * a.dv + col) = make_float4(x[i][0], x[i][1], x[i][2], x[i][3]);
    }
  }
  l = seq_warp_sum(l);
  if (lane == 0) sm[warp] = m, sl[warp] = l;
  __syncthreads();
  for (int e = tid * 4; e < heads * a.dv; e += kArThreads * 4) {
    const int r = e / a.dv, c = e - r * a.dv, hd = h0 + r;
    float4 o = *reinterpret_cast<const float4*>(part + r * a.dv + c);
    for (int s = 1; s < splits; ++s) {
      const float4 x = *reinterpret_cast<const float4*>(part + (s * kArRows + r) * a.dv + c);
      o.x += x.x, o.y += x.y, o.z += x.z, o.w += x.w;
    }
    // the sink: one more term exp(sink) in the denominator, without a key or a value
    const float mt = a.sink != nullptr ? fmaxf(sm[r], a.sink[hd]) : sm[r], f = a.sink != nullptr ? expf(sm[r] - mt) : 1.f;
    float inv = f / (a.sink != nullptr ? sl[r] * f + expf(a.sink[hd] - mt) : sl[r]);
    float y[4] = {o.x, o.y, o.z, o.w};
    auto act = [&](float z) { return a.gate_act == 1 ? z / (1.f + expf(-z)) : (a.gate_act == 2 ? 1.f / (1.f + expf(-z)) : z); };
    if (a.gate != nullptr && a.gate_heads) inv *= act(a.gate[(long long)t * a.ldg + hd]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      y[i] *= inv;
      if (a.gate != nullptr && !a.gate_heads) y[i] *= act(a.gate[(long long)t * a.ldg + (long long)hd * a.dv + c + i]);
    }
    st4(static_cast<TY*>(a.out) + (long long)t * a.ldo + (long long)hd * a.dv + c, y);
  }
}

// Few rows: two heads to a CTA and TILES tiles of keys to a stage, so that a row's heads have CTAs of their own and a chain of copy, scores, softmax and values spans up to
// 128 keys. The same sums in the same order as the kernel above, from LD and the threads (how many of them split the keys of a tile): the same bits, so that
// the number of rows may choose between them. In us, the kernel above / the plain kernels in brackets: 1 row of 4096 keys, 32 heads, latents 128 + 32 133 (242 / 189), 8 heads
// 256 + 64 179 (317 / 333), 16 heads 512 + 64 268 (445 / 1838), 8 heads over 1 of 64 + 64 122 (194 / 180); 3 rows of 130 keys, the same shapes 8.8 (11.8 / 9.8), 9.7 (15 / 13.9),
// 12.2 (19.4 / 65), 8.0 (9.9 / 10.1); 1 row of 16 keys 3.8 (4.4 / 3.7), 3.8 (4.9 / 4.4), 4.2 (6.3 / 10.7), 3.8 (4.2 / 4.3); slowest beside the plain kernels: 4 heads, latents
// 64 + 32 3.9 (3.8 / 3.6).
constexpr int kArFewHeads = 2;
template <int THREADS, int LD, int TILES, typename TY>
__device__ __forceinline__ void attn_few_rows(const AttnRowsArgs& a, int p, int low) {
  constexpr int HEADS = kArFewHeads, WARPS = THREADS / 32, COPY = THREADS / 32, KEYS = kArKeys * TILES, SPITCH = KEYS + 1;   // COPY: threads per key row of a tile
  extern __shared__ __align__(16) float ar_sm[];   // stages [2][KEYS][width] | Q [HEADS][d] | scores [HEADS][KEYS + 1] | probabilities [KEYS][HEADS] | factors [TILES][HEADS] | maxima, sums
  float* const stages = ar_sm;
  float* const qs = stages + 2 * KEYS * a.width;
  float* const ss = qs + HEADS * a.d;
  float* const ps = ss + HEADS * SPITCH;
  float* const sc = ps + KEYS * HEADS;
  float* const sm = sc + TILES * HEADS;
  float* const sl = sm + HEADS;
  const int t = blockIdx.x, kvh = blockIdx.y / a.head_blocks, hb = blockIdx.y - kvh * a.head_blocks, rep = a.H / a.G;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h0 = kvh * rep + hb * HEADS, heads = min(HEADS, rep - hb * HEADS);   // this CTA's query heads
  const int n_stages = (p - low + KEYS) / KEYS;
  const int32_t* bt = a.bt + (long long)a.slot[t] * a.max_pages;
  int page[TILES], at[TILES];   // of this thread's rows of the next stage, looked up a stage ahead of its copy; -1: no key that the row sees
  auto locate = [&](int i) {
#pragma unroll
    for (int b = 0; b < TILES; ++b) {
      page[b] = -1;
      if (b > 0 && low + i * KEYS + b * kArKeys > p) continue;   // a tile without keys
      const int j = low + i * KEYS + b * kArKeys + tid / COPY, q = j / a.page_size;
      at[b] = j - q * a.page_size;
      page[b] = j <= p ? bt[q] : -1;
    }
  };
  auto load = [&](int i) {   // rows of the last stage beyond the keys stay as they are: nothing uses their scores, and nobody reads their values
    const int c0 = (tid % COPY) * 4;
#pragma unroll
    for (int b = 0; b < TILES; ++b) {
      float* row = stages + ((i & 1) * KEYS + b * kArKeys + tid / COPY) * a.width;
      if (page[b] >= 0) {
        const float* src = a.pool + ((long long)page[b] * a.page_size + at[b]) * a.row_w;
        for (int c = c0; c < a.d; c += 4 * COPY) ar_copy16(row + c, src + kvh * a.koff_g + c);
        if (a.voff_g >= 0)
          for (int c = c0; c < a.dv; c += 4 * COPY) ar_copy16(row + a.voff + c, src + a.voff_g + kvh * a.dv + c);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  locate(0);
  for (int e = tid * 4; e < HEADS * a.d; e += THREADS * 4) {
    if (e < heads * a.d) ar_copy16(qs + e, a.q + (long long)t * a.ldq + (long long)h0 * a.d + e);
    else *reinterpret_cast<float4*>(qs + e) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  load(0);
  if (n_stages > 1) locate(1);
  // softmax: this warp's row
  const int h = h0 + min(warp, heads - 1);
  const float inv_cap = a.softcap > 0.f ? 1.f / a.softcap : 0.f;
  float m = -INFINITY, l = 0.f;   // l: this lane's keys
  // values: this thread's columns and share of the keys
  const int groups = (a.dv >> 2), g2 = groups <= 8 ? 8 : (groups <= 16 ? 16 : (groups <= 32 ? 32 : (groups <= 64 ? 64 : 128)));   // at most 128 groups: dv <= 512
  const int splits = THREADS / g2, col = (tid & (g2 - 1)) * 4, split = tid / g2;
  const bool has_cols = col < a.dv;
  ar_f2 acc[4] = {0ull, 0ull, 0ull, 0ull};   // of both heads
  constexpr int SHARE = 32 / LD, OF_LANE = KEYS / (WARPS * SHARE);            // keys that a warp takes at a time, keys of a lane in all
  constexpr int KP = OF_LANE * HEADS > LD ? LD / HEADS : OF_LANE, VALS = KP * HEADS;   // keys of a lane in one pass; its sums before the butterfly, at most as many as lanes share them
  const int sub = lane & (LD - 1), lane_key = warp * (SHARE * OF_LANE) + lane / LD * KP;
  const int mine = sub / (LD / VALS), at_score = (mine % HEADS) * SPITCH + mine / HEADS;   // which of the sums is this lane's: key mine / HEADS, row mine % HEADS

  for (int i = 0; i < n_stages; ++i) {
    const float* stage = stages + (i & 1) * KEYS * a.width;
    const int j0 = low + i * KEYS, n_keys = min(KEYS, p - j0 + 1);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();   // this stage is there, and everyone is done with the one before
    if (i + 1 < n_stages) load(i + 1);
    if (i + 2 < n_stages) locate(i + 2);
    auto scores = [&](int key0) {   // of this lane's KP keys from key0 on
      ar_f2 s2[KP][HEADS];
#pragma unroll
      for (int k = 0; k < KP; ++k)
#pragma unroll
        for (int r = 0; r < HEADS; ++r) s2[k][r] = 0ull;
      for (int c = sub * 4; c < a.d; c += LD * 4) {
        ulonglong2 kv[KP];
#pragma unroll
        for (int k = 0; k < KP; ++k) kv[k] = *reinterpret_cast<const ulonglong2*>(stage + (key0 + k) * a.width + c);
#pragma unroll
        for (int r = 0; r < HEADS; ++r) {
          const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(qs + r * a.d + c);
#pragma unroll
          for (int k = 0; k < KP; ++k) {
            ar_fma(s2[k][r], kv[k].x, qv.x);
            ar_fma(s2[k][r], kv[k].y, qv.y);
          }
        }
      }
      float v[VALS];
#pragma unroll
      for (int k = 0; k < KP; ++k)
#pragma unroll
        for (int r = 0; r < HEADS; ++r) {
          float lo, hi;
          ar_split(s2[k][r], lo, hi);
          v[k * HEADS + r] = lo + hi;
        }
      int off = LD / 2;
#pragma unroll
      for (int cur = VALS; cur > 1; cur >>= 1, off >>= 1) {
        const bool up = lane & off;
#pragma unroll
        for (int i = 0; i < cur / 2; ++i) {
          const float other = __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + cur / 2], off);
          v[i] = (up ? v[i + cur / 2] : v[i]) + other;
        }
      }
#pragma unroll
      for (; off > 0; off >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
      ss[at_score + key0] = v[0];
    };
    if constexpr (OF_LANE == KP) {
      if (warp * (SHARE * KP) < n_keys) scores(lane_key);
    } else {
#pragma unroll 1
      for (int pass = 0; pass < OF_LANE && warp * (SHARE * OF_LANE) + SHARE * pass < n_keys; pass += KP) scores(lane_key + SHARE * pass);
    }
    __syncthreads();
    if (warp < HEADS) {
      float s[TILES], top[TILES];
#pragma unroll
      for (int b = 0; b < TILES; ++b) {
        const int k = b * kArKeys + lane;
        s[b] = top[b] = -INFINITY;
        if (b > 0 && b * kArKeys >= n_keys) continue;
        s[b] = ss[warp * SPITCH + k] * a.scale;
        if (a.softcap > 0.f) s[b] = a.softcap * tanhf(s[b] * inv_cap);
        if (a.bias != nullptr && k < n_keys) s[b] += a.bias[(long long)(p - j0 - k) * a.H + h];
        top[b] = k < n_keys ? s[b] : -INFINITY;
      }
      if (TILES == 1 || n_keys <= kArKeys) {
        top[0] = seq_warp_max(top[0]);
      } else {
#pragma unroll
        for (int b = 0; b < TILES; ++b) top[b] = seq_warp_max(top[b]);
      }
#pragma unroll
      for (int b = 0; b < TILES; ++b) {
        if (b > 0 && b * kArKeys >= n_keys) break;
        const int k = b * kArKeys + lane;
        const float mn = fmaxf(m, top[b]), corr = m == -INFINITY ? 0.f : expf(m - mn), pj = k < n_keys && s[b] != -INFINITY ? expf(s[b] - mn) : 0.f;
        l = l * corr + pj;
        m = mn;
        ps[k * HEADS + warp] = pj;
        if (lane == 0) sc[b * HEADS + warp] = corr;
      }
    }
    __syncthreads();
    auto values = [&](int b, int end) {   // of tile b, whose keys end at `end` of the stage
      if (i + b > 0) {
        const ar_f2 f = *reinterpret_cast<const ar_f2*>(sc + b * HEADS);
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] = ar_mul(acc[c], f);
      }
      const float* vrow = stage + a.voff + col;
#pragma unroll 4
      for (int k = b * kArKeys + split; k < end; k += splits) {
        const ar_f2 pr = *reinterpret_cast<const ar_f2*>(ps + k * HEADS);
        const float4 v = *reinterpret_cast<const float4*>(vrow + k * a.width);
        const ar_f2 vc[4] = {ar_both(v.x), ar_both(v.y), ar_both(v.z), ar_both(v.w)};
#pragma unroll
        for (int c = 0; c < 4; ++c) ar_fma(acc[c], pr, vc[c]);
      }
    };
    if (has_cols) {
      if constexpr (TILES == 1) {
        values(0, n_keys);
      } else {
#pragma unroll 1
        for (int b = 0; b * kArKeys < n_keys; ++b) values(b, min(n_keys, (b + 1) * kArKeys));
      }
    }
  }
  __syncthreads();   // the stages' place is free
  float* const part = stages;   // [splits][HEADS][dv]
  if (has_cols) {
    float x[HEADS][4];
#pragma unroll
    for (int c = 0; c < 4; ++c) ar_split(acc[c], x[0][c], x[1][c]);
#pragma unroll
    for (int r = 0; r < HEADS; ++r) *reinterpret_cast<float4*>(part + (split * HEADS + r) * a.dv + col) = make_float4(x[r][0], x[r][1], x[r][2], x[r][3]);
  }
  l = seq_warp_sum(l);
  if (lane == 0 && warp < HEADS) sm[warp] = m, sl[warp] = l;
  __syncthreads();
  for (int e = tid * 4; e < heads * a.dv; e += THREADS * 4) {
    const int r = e / a.dv, c = e - r * a.dv, hd = h0 + r;
    float4 o = *reinterpret_cast<const float4*>(part + r * a.dv + c);
    for (int s = 1; s < splits; ++s) {
      const float4 x = *reinterpret_cast<const float4*>(part + (s * HEADS + r) * a.dv + c);
      o.x += x.x, o.y += x.y, o.z += x.z, o.w += x.w;
    }
    // the sink: one more term exp(sink) in the denominator, without a key or a value
    const float mt = a.sink != nullptr ? fmaxf(sm[r], a.sink[hd]) : sm[r], f = a.sink != nullptr ? expf(sm[r] - mt) : 1.f;
    float inv = f / (a.sink != nullptr ? sl[r] * f + expf(a.sink[hd] - mt) : sl[r]);
    float y[4] = {o.x, o.y, o.z, o.w};
    auto act = [&](float z) { return a.gate_act == 1 ? z / (1.f + expf(-z)) : (a.gate_act == 2 ? 1.f / (1.f + expf(-z)) : z); };
    if (a.gate != nullptr && a.gate_heads) inv *= act(a.gate[(long long)t * a.ldg + hd]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      y[i] *= inv;
      if (a.gate != nullptr && !a.gate_heads) y[i] *= act(a.gate[(long long)t * a.ldg + (long long)hd * a.dv + c + i]);
    }
    st4(static_cast<TY*>(a.out) + (long long)t * a.ldo + (long long)hd * a.dv + c, y);
  }
}

template <int THREADS, int LD, int TILES, typename TY>
__global__ void __launch_bounds__(THREADS) attn_few_rows_kernel(AttnRowsArgs a) {
  const int p = a.pos[blockIdx.x], low = max(max(0, p - a.window + 1), p - p % a.chunk);
  if (TILES > 1 && p - low < kArKeys) attn_few_rows<THREADS, LD, 1, TY>(a, p, low);   // one tile of keys: less code to fetch
  else attn_few_rows<THREADS, LD, TILES, TY>(a, p, low);
}

static size_t ar_smem(int heads, int tiles, int d, int width) {
  const size_t keys = (size_t)kArKeys * tiles;
  return sizeof(float) * (2 * keys * width + (size_t)heads * d + heads * (keys + 1) + keys * heads + (size_t)tiles * heads + 2 * heads);
}
static int ar_rows(int rep) { return rep > 4 ? 8 : 4; }

// Widths and strides only: whatever the number of rows, a shape is computed with the same sums. One head per key/value head shares nothing and fills a fourth of the
// products; over a reach of 64 keys and more it is still the faster (376 rows, 8 heads of 64 + 64: 29 us against 34, all keys 79 against 98), over 16 keys it is not (20
// against 14).
bool attn_rows_ok(int rep, int d, int dv, bool values_in_keys, long long ldq, long long ldo, int out_dt, const void* q, const void* pool, const void* out, int row_w, int reach) {
  auto al = [](const void* x, int n) { return reinterpret_cast<uintptr_t>(x) % n == 0; };
  const int width = values_in_keys ? d : d + dv;
  return (rep > 1 || reach >= 64) && d % 4 == 0 && dv % 4 == 0 && dv <= 512 && row_w % 4 == 0 && ldq % 4 == 0 && ldo % 4 == 0 && al(q, 16) && al(pool, 16) && al(out, out_dt == OMC_DT_F32 ? 16 : 8) &&
         ar_smem(ar_rows(rep), 1, d, width) <= 220 * 1024 && 2 * kArKeys * width >= ar_rows(rep) * ar_rows(rep) * 128;   // the partial outputs take the tiles' place
}

template <typename Kernel>
static int ar_launch(Kernel kernel, AttnRowsArgs a, int heads, int threads, int tiles, bool (&done)[kMaxDevices], cudaStream_t st) {
  const int dev = cur_device(), rep = a.H / a.G;
  if (!done[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e != cudaSuccess) return set_error(OMC_ERR_CUDA, cudaGetErrorString(e));
    done[dev] = true;
  }
  a.head_blocks = (rep + heads - 1) / heads;
  kernel<<<dim3(a.T, a.G * a.head_blocks), threads, ar_smem(heads, tiles, a.d, a.width), st>>>(a);
  return check_launch("attn_rows");
}

template <int ROWS, int LD, typename TY>
static int ar_go(const AttnRowsArgs& a, cudaStream_t st) {
  // Two heads to a CTA while these CTAs run in one wave: more of them would read the keys of a head group more often than the chip's idle SMs are worth (us, two
  // heads to a CTA / all: 32 rows of 1000 keys, 16 heads over 2 of 128 + 128, 256 CTAs 77 / 58; 1 row of 4096, 32 heads, latents 128 + 32, 16 CTAs 133 / 242).
  static bool done[4][kMaxDevices] = {};
  const int rep = a.H / a.G, reach = min(a.window, a.chunk);
  if ((long long)a.T * a.G * ((rep + kArFewHeads - 1) / kArFewHeads) > 148) return ar_launch(attn_rows_kernel<ROWS, LD, TY>, a, ROWS, ROWS * 32, 1, done[0], st);
  int tiles = reach <= kArKeys ? 1 : (reach <= 2 * kArKeys ? 2 : 4);   // as far as a row sees and shared memory goes
  while (tiles > 1 && ar_smem(kArFewHeads, tiles, a.d, a.width) > 220 * 1024) tiles >>= 1;
  if (tiles == 4) return ar_launch(attn_few_rows_kernel<ROWS * 32, LD, 4, TY>, a, kArFewHeads, ROWS * 32, 4, done[1], st);
  if (tiles == 2) return ar_launch(attn_few_rows_kernel<ROWS * 32, LD, 2, TY>, a, kArFewHeads, ROWS * 32, 2, done[2], st);
  return ar_launch(attn_few_rows_kernel<ROWS * 32, LD, 1, TY>, a, kArFewHeads, ROWS * 32, 1, done[3], st);
}

int attn_rows(const float* q, long long ldq, int T, int H, int G, int d, int dv, bool values_in_keys, const float* pool, const int32_t* bt, int max_pages, int page_size,
              const int32_t* pos, const int32_t* slot, int window, int chunk, float scale, float softcap, const float* bias, const float* sink, const float* gate,
              long long ldg, int gate_act, int gate_heads, void* out, int out_dt, long long ldo, cudaStream_t st) {
  const int rows = ar_rows(H / G), width = values_in_keys ? d : d + dv;
  const AttnRowsArgs a{q, ldq, pool, bt, pos, slot, bias, sink, gate, ldg, gate_act, gate_heads, out, ldo, T, H, G, d, dv, width, values_in_keys ? 0 : d, max_pages, page_size,
                       window, chunk, 0, d, values_in_keys ? -1 : G * d, values_in_keys ? G * d : G * (d + dv), scale, softcap};
  auto of = [&](auto ty) {
    using TY = decltype(ty);
    if (rows == 8) return ar_smem(rows, 1, d, width) <= 113 * 1024 ? ar_go<8, 16, TY>(a, st) : ar_go<8, 32, TY>(a, st);   // two CTAs of 113 KB share an SM
    return d <= 32 ? ar_go<4, 8, TY>(a, st) : ar_go<4, 16, TY>(a, st);
  };
  return out_dt == OMC_DT_F32 ? of(float{}) : of(bf16_t{});
}

}  // namespace omc
