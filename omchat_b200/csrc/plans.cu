// Work lists of prompt portions (latent and windowed attention): built on the host, of which one thread needs a few microseconds, and brought to the device as a
// kernel's parameters - no pinned memory to find, to fill and to keep alive until a copy has read it, and a captured graph has the list in itself.
// Before, array arithmetic in Python, pin_memory and a copy: 300 rows of 16 heads 86 us, a list of windowed attention 22 us.
#include <algorithm>
#include <exception>
#include <vector>

#include "seq_common.cuh"

namespace omc {

template <int N>
struct Words {
  int32_t w[N];
};
template <int N>
__global__ void __launch_bounds__(256) put_words_kernel(const __grid_constant__ Words<N> from, int n, int32_t* __restrict__ to) {
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) to[i] = from.w[i];
}
template <int N>
static void put_words(const int32_t* from, int n, int32_t* to, cudaStream_t st) {
  static thread_local Words<N> words;
  std::copy(from, from + n, words.w);
  put_words_kernel<N><<<(n + 255) / 256, 256, 0, st>>>(words, n, to);
}
// A launch copies all of its parameters, so lists that need few take a kernel of few; 32764 bytes is the most that one may have.
static int put_list(const std::vector<int32_t>& list, int32_t* to, cudaStream_t st) {
  constexpr int kMost = 8000;
  for (size_t at = 0; at < list.size(); at += kMost) {
    const int n = (int)std::min<size_t>(kMost, list.size() - at);
    if (n <= 256) put_words<256>(list.data() + at, n, to + at, st);
    else if (n <= 2048) put_words<2048>(list.data() + at, n, to + at, st);
    else put_words<kMost>(list.data() + at, n, to + at, st);
  }
  return check_launch("a work list");
}

static long long div_up(long long a, long long b) { return (a + b - 1) / b; }

struct LatentItem {
  int32_t v[8];
};
// The lists of LatentAttnPlan (seqlib.py): items of 8 words, those with the most keys first, then merges of 4.
static void latent_lists(const int32_t* portions, int n_portions, int H, int tok, int target_ctas, int min_keys, int max_parts, int row_tile, long long window,
                         std::vector<int32_t>& out, int32_t (&counts)[4]) {
  std::vector<LatentItem> items;
  std::vector<int32_t> merges;
  long long base = 0;
  int most = 1;
  bool any = false;
  for (int p = 0; p < n_portions; ++p) {
    const int n = portions[4 * p + 1];
    base += div_up(n, tok);
    most = any ? std::max(most, std::min(tok, n)) : std::min(tok, n);
    any = true;
  }
  items.reserve((size_t)base);
  int part = 0;
  for (int p = 0; p < n_portions; ++p) {
    const int first_row = portions[4 * p], n = portions[4 * p + 1], slot = portions[4 * p + 2], p0 = portions[4 * p + 3];
    for (int start = 0; start < n; start += tok) {
      const int ntok = std::min(tok, n - start), first = p0 + start;
      const long long low = std::max<long long>(0, first - window + 1), keys = first + ntok - low;   // first key the tile's first row sees, and how many up to its last row's last
      long long want = 1;
      if (base < target_ctas / 2) want = std::max<long long>(1, std::min({div_up(keys, min_keys), div_up(target_ctas, base), (long long)max_parts}));
      if (want == 1) {
        items.push_back({{first_row + start, ntok, slot, first, (int32_t)low, (int32_t)(low + keys), -1, 0}});
        continue;
      }
      const long long span = div_up(div_up(keys, want), row_tile) * row_tile, parts = div_up(keys, span);
      merges.insert(merges.end(), {(first_row + start) * H, ntok * H, part, (int32_t)parts});
      for (long long i = 0; i < parts; ++i)
        items.push_back({{first_row + start, ntok, slot, first, (int32_t)(low + i * span), (int32_t)(low + std::min(keys, (i + 1) * span)), part + (int32_t)i, 0}});
      part += (int32_t)parts;
    }
  }
  // with 148 running at a time a long one at the end would run alone
  std::stable_sort(items.begin(), items.end(), [](const LatentItem& a, const LatentItem& b) { return a.v[5] - a.v[4] > b.v[5] - b.v[4]; });
  out.clear();
  out.reserve(items.size() * 8 + merges.size());
  for (const LatentItem& i : items) out.insert(out.end(), i.v, i.v + 8);
  out.insert(out.end(), merges.begin(), merges.end());
  counts[0] = (int32_t)items.size(), counts[1] = (int32_t)merges.size() / 4, counts[2] = part, counts[3] = most;
}

// The list of window_attn_items (seqlib.py): tiles of `tok` tokens that end where a chunk does, unless a tile of rows is longer than a chunk.
static void window_list(const int32_t* portions, int n_portions, int tok, int row_tile, long long chunk, long long no_chunk, std::vector<int32_t>& out) {
  out.clear();
  const bool cut = row_tile <= chunk && chunk < no_chunk;
  for (int p = 0; p < n_portions; ++p) {
    int first_row = portions[4 * p], n = portions[4 * p + 1], p0 = portions[4 * p + 3];
    const int slot = portions[4 * p + 2];
    while (n > 0) {
      const int m = cut ? (int)std::min<long long>(n, chunk - p0 % chunk) : n;
      for (int s = 0; s < m; s += tok) out.insert(out.end(), {first_row + s, std::min(tok, m - s), slot, p0 + s});
      first_row += m, n -= m, p0 += m;
    }
  }
}

// A list is built when it is counted and kept for the call that fetches it, which follows at once on the same thread.
static thread_local std::vector<int32_t> last_list;

}  // namespace omc

using namespace omc;

extern "C" int omc_latent_plan(const int32_t* portions, int n_portions, int H, int tok, int target_ctas, int min_keys, int max_parts, int row_tile, int window, int32_t* counts) {
  if ((portions == nullptr && n_portions > 0) || counts == nullptr || n_portions < 0 || H <= 0 || tok <= 0 || min_keys <= 0 || max_parts <= 0 || row_tile <= 0 || window <= 0)
    return set_error(OMC_ERR_ARG, "omc_latent_plan: bad argument");
  try {
    int32_t c[4];
    latent_lists(portions, n_portions, H, tok, target_ctas, min_keys, max_parts, row_tile, window, last_list, c);
    std::copy(c, c + 4, counts);
  } catch (const std::exception&) {
    return set_error(OMC_ERR_ARG, "omc_latent_plan: no memory for the list");
  }
  return OMC_OK;
}

extern "C" int omc_window_plan(const int32_t* portions, int n_portions, int tok, int row_tile, int chunk, int no_chunk, int32_t* counts) {
  if ((portions == nullptr && n_portions > 0) || counts == nullptr || n_portions < 0 || tok <= 0 || row_tile <= 0)
    return set_error(OMC_ERR_ARG, "omc_window_plan: bad argument");
  try {
    window_list(portions, n_portions, tok, row_tile, chunk, no_chunk, last_list);
  } catch (const std::exception&) {
    return set_error(OMC_ERR_ARG, "omc_window_plan: no memory for the list");
  }
  counts[0] = (int32_t)(last_list.size() / 4);
  return OMC_OK;
}

extern "C" int omc_plan_words(int32_t* to, int n, int on_device, void* stream) {
  if (n < 0 || (size_t)n != last_list.size() || (to == nullptr && n > 0)) return set_error(OMC_ERR_ARG, "omc_plan_words: not the list that was built last on this thread");
  if (n == 0) return OMC_OK;
  if (on_device) return put_list(last_list, to, static_cast<cudaStream_t>(stream));
  std::copy(last_list.begin(), last_list.end(), to);
  return OMC_OK;
}
