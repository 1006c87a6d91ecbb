// Page top-k selection for sm_100a.
//
// Input scores[H, K, T] (token fastest), output out[T, H, TOPK] int32 ascending, -1 padded.
// The ranking is a strict total order -- (score key desc, page index asc) -- so the result is
// deterministic and bit-exact against a stable sort (the contract the upstream tests pin for
// the bf16 path: tests/smoke/test_sparse_topk_forced.py:266-275).  Score keys follow the
// upstream order-preserving float->uint map (sparse_topk_select.cuh:186-213); pages forced by
// force_begin / force_end rank as FLT_MAX (kForcedOrd there).
//
// Layout of the work for prefill-sized inputs: a CTA owns 32 consecutive tokens of one head; its lanes read 32
// consecutive tokens (one coalesced 128-byte line per page row for fp32), its SL warps share the pages, a thread per
// row and warp.  Two kernels of that layout: topk_threshold_kernel finds the TOPK-th best score of a row with 32-bit
// keys and picks the pages in a second scan; topk_select_kernel (bf16 scores) keeps whole keys, score and page, in one
// 32-bit word and needs one scan.  No transpose workspace (upstream needs one, api.py:1818-1821).
// Decode-sized inputs: topk_row_kernel, a CTA per row.
#include "common.cuh"
#include "nvtx_range.h"

namespace msa {
namespace {

constexpr uint32_t kForcedOrd = 0xFF7FFFFFu;   // key of FLT_MAX

// Order key of a score: the upstream order-preserving float -> uint map with the two cases folded in
// where bit order and value order differ under the stable-sort contract: -0.0 and +0.0 compare equal
// (v + 0.0f turns -0.0 into +0.0), and every NaN ranks above +inf with all NaNs tying (one key).
__device__ __forceinline__ uint32_t ord_key(float v) {
  v += 0.0f;
  const uint32_t bits = __float_as_uint(v);
  const uint32_t key = bits ^ (static_cast<uint32_t>(static_cast<int32_t>(bits) >> 31) | 0x80000000u);
  return v != v ? 0xFFFFFFFFu : key;
}

// Key of topk_select_kernel: bf16 scores only, where the upper half of the order key is exact, so
// (key16 << 16 | ~page16) is one unique 32-bit word (no tie handling anywhere) and a compare-exchange is one max and
// one min.  Not used with forced pages, which rank as the fp32 maximum -- a score bf16 cannot tell from its own largest
// finite value -- nor beyond 65 535 pages.
struct Key1 {
  uint32_t k;
  static __device__ __forceinline__ Key1 none() { return {0u}; }
  static __device__ __forceinline__ Key1 make(uint32_t ord, int page) {
    return {(ord & 0xffff0000u) | (0xffffu - static_cast<uint32_t>(page))};
  }
  __device__ __forceinline__ bool is_none() const { return k == 0u; }
  __device__ __forceinline__ uint32_t page() const { return 0xffffu - (k & 0xffffu); }
};
__device__ __forceinline__ void order(Key1& a, Key1& b) {
  const uint32_t hi = max(a.k, b.k), lo = min(a.k, b.k);
  a.k = hi; b.k = lo;
}
__device__ __forceinline__ Key1 best(const Key1& a, const Key1& b) { return {max(a.k, b.k)}; }
__device__ __forceinline__ void order(uint32_t& a, uint32_t& b) {
  const uint32_t hi = max(a, b), lo = min(a, b);
  a = hi; b = lo;
}
__device__ __forceinline__ uint32_t best(uint32_t a, uint32_t b) { return max(a, b); }

// Descending sort of N keys / merge of a descending list into the sorted top-N list.  Static register indices, no
// data-dependent branch: the 32 rows a warp owns never diverge.  The sort is a bitonic one above 8 keys, an odd-even merge
// sort up to 8: that has fewer exchanges (19 against 24 for 8 keys, 63 against 80 for 16) and is 2 to 5 % faster there, but of
// 16 or 32 keys its code keeps the units waiting (65 536 rows x 256 pages of fp32: 43.5 us against 41.2 for the bitonic one
// with topk 16, 97 against 52 with 32).
template <int N, typename K>
__device__ __forceinline__ void net_sort_desc(K (&v)[N]) {
  if constexpr (N <= 8) {
#pragma unroll
    for (int p = 1; p < N; p <<= 1) {
#pragma unroll
      for (int k = p; k > 0; k >>= 1) {
#pragma unroll
        for (int j = k % p; j + k < N; j += 2 * k) {
#pragma unroll
          for (int i = 0; i < k; ++i) {
            if (i + j + k < N && (i + j) / (2 * p) == (i + j + k) / (2 * p)) order(v[i + j], v[i + j + k]);
          }
        }
      }
    }
  } else {
#pragma unroll
    for (int k = 2; k <= N; k <<= 1) {
#pragma unroll
      for (int j = k >> 1; j > 0; j >>= 1) {
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const int l = i ^ j;
          if (l > i) {
            if ((i & k) == 0) order(v[i], v[l]); else order(v[l], v[i]);
          }
        }
      }
    }
  }
}
template <int N, typename K>
__device__ __forceinline__ void net_merge_desc(K (&key)[N], const K (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) key[i] = best(key[i], v[N - 1 - i]);     // bitonic now
#pragma unroll
  for (int j = N >> 1; j > 0; j >>= 1) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int l = i ^ j;
      if (l > i) order(key[i], key[l]);
    }
  }
}

// Two scans of a row's pages.  The first keeps the TOPK largest order keys -- the scores alone, 32 bits: an exchange
// is a max and a min, where (score, page) in one 64-bit word costs a 64-bit compare and two selects of pairs -- and
// leaves the threshold, the TOPK-th best key.  The second scan, in page order, takes every page above the threshold
// and the first of those at it, as many as fit: exactly the order (key desc, page asc), and the pages come out
// ascending without a sort.  The scores of the second scan come from L2.
// Measured on fp32 scores, kernel alone: 65 536 rows x 256 pages 103 -> 52 us, 32 768 rows x 769 pages 133 -> 65 us
// (64-bit keys in one scan before); 256 tokens x 4 heads x 256 pages 18.5 us (a CTA per row) -> 7.5 us.
// FORCED: some pages rank as FLT_MAX whatever their score.
template <int TOPK, typename T, bool FORCED>
__global__ void __launch_bounds__(512)
topk_threshold_kernel(const T* scores, int32_t* out, int num_heads, int max_k_tiles,
                      int total_q, int nvp, int force_begin, int force_end_start, int slices) {
  chain_begin();
  extern __shared__ uint32_t s_lists[];             // [slices][TOPK][32]: keys of the first scan, pages of the second
  __shared__ uint32_t s_threshold[32], s_count[16 * 32];
  __shared__ int s_quota[32];
  constexpr uint32_t kTie = 0x80000000u;
  constexpr float kMax = 3.402823466e38f;
  const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5;
  const int tok_blocks = (total_q + 31) / 32;
  const int head = blockIdx.x / tok_blocks;
  const int t = (blockIdx.x % tok_blocks) * 32 + lane;
  const bool live = t < total_q;
  // a lane past the last token walks the last one: its loads are valid, its result is not stored
  const T* base = scores + static_cast<size_t>(head) * max_k_tiles * total_q + min(t, total_q - 1);
  uint32_t* mine = s_lists + sl * (TOPK * 32) + lane;
  // a contiguous part of the pages per warp, whole blocks of TOPK
  const int blocks = (nvp + TOPK - 1) / TOPK, per = (blocks + slices - 1) / slices;
  const int p0 = min(nvp, sl * per * TOPK), p1 = min(nvp, p0 + per * TOPK);
  // scores of up to N pages from k0 on, all loads before any use; those past p1 are not read
  auto load = [&](auto& v, int k0) {
    constexpr int N = sizeof(v) / sizeof(float);
    const T* ptr = base + static_cast<size_t>(k0) * total_q;
    if (k0 + N <= p1) {
#pragma unroll
      for (int u = 0; u < N; ++u, ptr += total_q) v[u] = static_cast<float>(*ptr);
    } else {
#pragma unroll
      for (int u = 0; u < N; ++u, ptr += total_q) v[u] = k0 + u < p1 ? static_cast<float>(*ptr) : 0.f;
    }
    if constexpr (FORCED) {
#pragma unroll
      for (int u = 0; u < N; ++u)
        if (k0 + u < force_begin || k0 + u >= force_end_start) v[u] = kMax;
    }
  };

  uint32_t top[TOPK];
#pragma unroll
  for (int i = 0; i < TOPK; ++i) top[i] = 0u;       // below every order key
  for (int k0 = p0; k0 < p1; k0 += TOPK) {
    float v[TOPK];
    load(v, k0);
    uint32_t blk[TOPK];
#pragma unroll
    for (int u = 0; u < TOPK; ++u) blk[u] = ord_key(v[u]);
    if (k0 + TOPK > p1) {
#pragma unroll
      for (int u = 0; u < TOPK; ++u)
        if (k0 + u >= p1) blk[u] = 0u;
    }
    net_sort_desc<TOPK, uint32_t>(blk);
    net_merge_desc<TOPK, uint32_t>(top, blk);
  }
  // tree merge of the slices' lists into slice 0 (slices is a power of two)
  for (int d = 1; d < slices; d <<= 1) {
    if ((sl & (2 * d - 1)) == d) {
#pragma unroll
      for (int i = 0; i < TOPK; ++i) mine[i * 32] = top[i];
    }
    __syncthreads();
    if ((sl & (2 * d - 1)) == 0) {
      uint32_t o[TOPK];
#pragma unroll
      for (int i = 0; i < TOPK; ++i) o[i] = mine[(d * TOPK + i) * 32];
      net_merge_desc<TOPK, uint32_t>(top, o);
    }
  }
  if (sl == 0) {
    int above = 0;
#pragma unroll
    for (int i = 0; i < TOPK; ++i) above += top[i] > top[TOPK - 1] ? 1 : 0;
    s_threshold[lane] = top[TOPK - 1];
    s_quota[lane] = TOPK - above;                   // pages to take among those at the threshold
  }
  __syncthreads();
  // The second scan compares scores: the order key of a number grows with it, -0 and +0 compare equal, and a NaN is
  // above every number (not <=) but ties with a NaN threshold.
  const uint32_t tkey = s_threshold[lane];
  const bool t_nan = tkey == 0xffffffffu;
  const float thr = t_nan ? __int_as_float(0x7fffffff) : __uint_as_float(tkey & 0x80000000u ? tkey ^ 0x80000000u : ~tkey);
  const int quota = s_quota[lane];
  int n = 0, ties = 0;
  for (int k0 = p0; k0 < p1; k0 += 16) {
    float v[16];
    load(v, k0);
    uint32_t above = 0, level = 0;                  // bit u: page k0 + u
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      if (!(v[u] <= thr)) above |= 1u << u;
      if (v[u] == thr || (t_nan && v[u] != v[u])) level |= 1u << u;
    }
    if (t_nan) above = 0;
    uint32_t take = above | level;
    if (k0 + 16 > p1) take &= (1u << (p1 - k0)) - 1u;
    while (take != 0) {
      const int u = __ffs(take) - 1;
      take &= take - 1;
      const bool tie = (level >> u) & 1u;
      if (tie && ties >= quota) continue;           // at most TOPK of a row in all: fewer above than TOPK, quota ties
      mine[n * 32] = static_cast<uint32_t>(k0 + u) | (tie ? kTie : 0u);
      ++n;
      ties += tie ? 1 : 0;
    }
  }
  s_count[sl * 32 + lane] = static_cast<uint32_t>(n - ties) << 16 | static_cast<uint32_t>(ties);
  __syncthreads();
  // slice s of a row puts its pages behind those of the slices before it, whose ties use up the quota first
  int pos = 0, left = quota;
  for (int s2 = 0; s2 < sl; ++s2) {
    const uint32_t c = s_count[s2 * 32 + lane];
    const int use = min(left, static_cast<int>(c & 0xffffu));
    pos += static_cast<int>(c >> 16) + use;
    left -= use;
  }
  if (!live) return;
  int32_t* dst = out + (static_cast<size_t>(t) * num_heads + head) * TOPK;
  for (int i = 0; i < n; ++i) {
    const uint32_t page = mine[i * 32];
    const bool tie = (page & kTie) != 0;
    if (!tie || left > 0) dst[pos++] = static_cast<int32_t>(page & ~kTie);
    if (tie) --left;
  }
}

template <int TOPK, typename T>
__global__ void __launch_bounds__(256)
topk_select_kernel(const T* scores, int32_t* out, int num_heads, int max_k_tiles,
                   int total_q, int nvp, int slices) {
  chain_begin();
  using K = Key1;
  extern __shared__ __align__(8) unsigned char s_raw[];
  K* s_keys = reinterpret_cast<K*>(s_raw);          // [slices][32][TOPK]
  const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5;
  const int tok_blocks = (total_q + 31) / 32;
  const int head = blockIdx.x / tok_blocks;
  const int t = (blockIdx.x % tok_blocks) * 32 + lane;
  const bool live = t < total_q;

  K top[TOPK];
#pragma unroll
  for (int i = 0; i < TOPK; ++i) top[i] = K::none();
  if (live) {
    const T* base = scores + static_cast<size_t>(head) * max_k_tiles * total_q + t;
    // slice sl scans page blocks sl, sl + slices, ... of TOPK consecutive pages each
    for (int k0 = sl * TOPK; k0 < nvp; k0 += slices * TOPK) {
      // all loads of a block before any use; the test of each page only in the last block
      float v[TOPK];
      const T* ptr = base + static_cast<size_t>(k0) * total_q;
      if (k0 + TOPK <= nvp) {
#pragma unroll
        for (int u = 0; u < TOPK; ++u, ptr += total_q) v[u] = static_cast<float>(*ptr);
      } else {
#pragma unroll
        for (int u = 0; u < TOPK; ++u, ptr += total_q) v[u] = k0 + u < nvp ? static_cast<float>(*ptr) : 0.f;
      }
      K blk[TOPK];
#pragma unroll
      for (int u = 0; u < TOPK; ++u) blk[u] = K::make(ord_key(v[u]), k0 + u);
      if (k0 + TOPK > nvp) {
#pragma unroll
        for (int u = 0; u < TOPK; ++u)
          if (k0 + u >= nvp) blk[u] = K::none();
      }
      net_sort_desc<TOPK, K>(blk);
      net_merge_desc<TOPK, K>(top, blk);
    }
  }
  if (slices > 1) {
    K* mine = s_keys + (static_cast<size_t>(sl) * 32 + lane) * TOPK;
#pragma unroll
    for (int i = 0; i < TOPK; ++i) mine[i] = top[i];
    __syncthreads();
    if (sl != 0) return;
    for (int s2 = 1; s2 < slices; ++s2) {
      const K* other = s_keys + (static_cast<size_t>(s2) * 32 + lane) * TOPK;
      K o[TOPK];
#pragma unroll
      for (int i = 0; i < TOPK; ++i) o[i] = other[i];
      net_merge_desc<TOPK, K>(top, o);
    }
  }
  if (!live) return;

  // page indices ascending; empty slots (cannot occur when nvp > TOPK) become -1 and sort last
  uint32_t idx[TOPK];
#pragma unroll
  for (int i = 0; i < TOPK; ++i) idx[i] = top[i].is_none() ? 0xffffffffu : top[i].page();
#pragma unroll
  for (int k = 2; k <= TOPK; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
#pragma unroll
      for (int i = 0; i < TOPK; ++i) {
        const int l = i ^ j;
        if (l > i) {
          const uint32_t a = idx[i], b = idx[l];
          const bool up = (i & k) == 0;
          idx[i] = up ? min(a, b) : max(a, b);
          idx[l] = up ? max(a, b) : min(a, b);
        }
      }
    }
  }
  int32_t* dst = out + (static_cast<size_t>(t) * num_heads + head) * TOPK;
#pragma unroll
  for (int i = 0; i < TOPK; i += 4) {
    int4 v;
    v.x = static_cast<int32_t>(idx[i]); v.y = static_cast<int32_t>(idx[i + 1]);
    v.z = static_cast<int32_t>(idx[i + 2]); v.w = static_cast<int32_t>(idx[i + 3]);
    *reinterpret_cast<int4*>(dst + i) = v;                  // 0xffffffff == -1
  }
}

// Few rows (decode): one CTA per (token, head) row, its 256 threads share the row's pages, NK
// per thread, kept in registers as order keys.  Two levels of the same selection loop, neither
// with a CTA-wide barrier inside: every warp extracts its own TOPK best (each round the lanes offer
// their best key below the previous winner, redux.sync picks the winner, lane r keeps winner r),
// the 8 x TOPK survivors go through shared memory, and warp 0 extracts the final TOPK from them.
// The order is the same strict total order (key desc, page asc), so the result is identical to the
// thread-per-row kernel above.
template <int NKEYS>
__device__ __forceinline__ void warp_select_round(const uint32_t (&ord)[NKEYS], const uint32_t (&page)[NKEYS],
                                                  uint32_t& last_ord, uint32_t& last_page, uint32_t& win_ord,
                                                  uint32_t& win_page) {
  uint32_t bo = 0u, bp = 0xffffffffu;
#pragma unroll
  for (int i = 0; i < NKEYS; ++i) {
    // below the previous winner in (key desc, page asc) order; last_page starts at "before page 0"
    const bool below = ord[i] < last_ord || (ord[i] == last_ord && static_cast<int32_t>(page[i]) > static_cast<int32_t>(last_page));
    const bool better = ord[i] > bo || (ord[i] == bo && page[i] < bp);
    if (below && ord[i] != 0u && better) { bo = ord[i]; bp = page[i]; }
  }
  win_ord = __reduce_max_sync(0xffffffffu, bo);
  win_page = __reduce_min_sync(0xffffffffu, (bo == win_ord && bo != 0u) ? bp : 0xffffffffu);
  if (win_ord != 0u) { last_ord = win_ord; last_page = win_page; }
  else { last_ord = 0u; last_page = 0x7fffffffu; }            // nothing left: later rounds find nothing either
}

template <int TOPK, int NK, typename T>
__global__ void __launch_bounds__(256)
topk_row_kernel(const T* scores, int32_t* out, int num_heads, int max_k_tiles, int total_q,
                int nvp, int force_begin, int force_end_start) {
  chain_begin();
  static_assert(TOPK <= 32, "one winner per lane");
  __shared__ uint32_t s_ord[8 * TOPK], s_page[8 * TOPK];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int t = blockIdx.x % total_q, head = blockIdx.x / total_q;
  const T* base = scores + static_cast<size_t>(head) * max_k_tiles * total_q + t;
  uint32_t ord[NK], page[NK];
  // All loads before any use, four at a time with one test.  (With the load beside its use the compiler only kept several on
  // the way where it could take the scores as constant: 8 192 pages x 496 rows, topk 4: 25 us against 34.)
  T score[NK];
#pragma unroll
  for (int i0 = 0; i0 < NK; i0 += 4) {
    if (256 * (i0 + 4) <= nvp) {
#pragma unroll
      for (int i = i0; i < i0 + 4; ++i) score[i] = base[static_cast<size_t>(tid + 256 * i) * total_q];
    } else {
#pragma unroll
      for (int i = i0; i < i0 + 4; ++i)
        score[i] = tid + 256 * i < nvp ? base[static_cast<size_t>(tid + 256 * i) * total_q] : static_cast<T>(0.f);
    }
  }
#pragma unroll
  for (int i = 0; i < NK; ++i) {
    const int pg = tid + 256 * i;
    page[i] = static_cast<uint32_t>(pg);
    ord[i] = 0u;                                             // 0: not a candidate
    if (pg < nvp) {
      const bool forced = pg < force_begin || pg >= force_end_start;
      ord[i] = forced ? kForcedOrd : ord_key(static_cast<float>(score[i]));
    }
  }
  // level 1: this warp's TOPK best, winner r in lane r
  uint32_t last_ord = 0xffffffffu, last_page = 0xffffffffu;   // (int32) -1: before page 0
  uint32_t my_ord = 0u, my_page = 0xffffffffu;
#pragma unroll
  for (int r = 0; r < TOPK; ++r) {
    uint32_t wo, wp;
    warp_select_round<NK>(ord, page, last_ord, last_page, wo, wp);
    if (lane == r) { my_ord = wo; my_page = wp; }
  }
  if (lane < TOPK) { s_ord[warp * TOPK + lane] = my_ord; s_page[warp * TOPK + lane] = my_page; }
  __syncthreads();
  if (warp != 0) return;
  // level 2: the final TOPK among the 8 * TOPK survivors
  constexpr int NC = 8 * TOPK / 32;
  uint32_t cord[NC], cpage[NC];
#pragma unroll
  for (int i = 0; i < NC; ++i) { cord[i] = s_ord[lane + 32 * i]; cpage[i] = s_page[lane + 32 * i]; }
  last_ord = 0xffffffffu; last_page = 0xffffffffu;
  uint32_t sel = 0xffffffffu;                                 // lane r: the r-th best page, or -1
#pragma unroll
  for (int r = 0; r < TOPK; ++r) {
    uint32_t wo, wp;
    warp_select_round<NC>(cord, cpage, last_ord, last_page, wo, wp);
    if (lane == r) sel = wo != 0u ? wp : 0xffffffffu;
  }
  // ascending page order, -1 (0xffffffff) last: rank = number of smaller entries (ties by lane)
  int rank = 0;
#pragma unroll
  for (int j = 0; j < TOPK; ++j) {
    const uint32_t o = __shfl_sync(0xffffffffu, sel, j);
    rank += (o < sel || (o == sel && j < lane)) ? 1 : 0;
  }
  if (lane < TOPK) out[(static_cast<size_t>(t) * num_heads + head) * TOPK + rank] = static_cast<int32_t>(sel);
}

template <int TOPK>
__global__ void topk_identity_kernel(int32_t* out, size_t rows, int nvp) {
  chain_begin();
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= rows * TOPK) return;
  const int c = static_cast<int>(i % TOPK);
  out[i] = c < nvp ? c : -1;
}

template <int TOPK, typename T>
int launch(const T* scores, int32_t* out, int H, int K, int T_, int nvp, int fb, int fe, cudaStream_t stream) {
  const size_t rows = static_cast<size_t>(H) * T_;
  if (rows == 0) return MSA_OK;
  if (nvp <= TOPK) {
    const size_t n = rows * TOPK;
    launch_chained(topk_identity_kernel<TOPK>, static_cast<unsigned>((n + 255) / 256), 256, 0, stream, out, rows, nvp);
    return cudaGetLastError() == cudaSuccess ? MSA_OK : MSA_ERR_LAUNCH;
  }
  const int fe_start = fe <= nvp ? nvp - fe : 0;
  const bool one_word = sizeof(T) == 2 && fb == 0 && fe == 0 && nvp <= 65535;      // bf16 scores, nothing forced
  // Decode-sized: a CTA per row, its pages in the registers of 256 threads (nk each).  From 32 tokens on a thread per row has
  // its lanes filled.  That one's time grows with the pages alone as long as its CTAs are resident, the other's with rows x
  // nk x topk from a few CTAs per SM on.  The line between them was fitted to both times at 1 456 sizes (32 to 2 048 rows, 33
  // to 8 192 pages, topk 4 to 32, both types): 0.6 % above the faster one on average, at most 1.26 times it but for three
  // sizes (1.7).  fp32, topk 16, CTA per row / thread per row: 32 rows x 1 024 pages 6.5 / 13.0 us, 384 x 2 048 17.6 / 21.9,
  // 384 x 4 096 61 / 39, 1 024 x 256 18.1 / 6.6.
  const int nk = nvp <= 256 * 4 ? 4 : (nvp <= 256 * 8 ? 8 : 32);
  const bool cta_per_row = T_ < 32 || (static_cast<long long>(rows) + 150) * nk * TOPK <= 36LL * (nvp + 128);
  if (cta_per_row && rows <= 2048 && nvp <= 256 * 32) {
    if (nk == 4)
      launch_chained(topk_row_kernel<TOPK, 4, T>, static_cast<unsigned>(rows), 256, 0, stream, scores, out, H, K, T_, nvp, fb, fe_start);
    else if (nk == 8)
      launch_chained(topk_row_kernel<TOPK, 8, T>, static_cast<unsigned>(rows), 256, 0, stream, scores, out, H, K, T_, nvp, fb, fe_start);
    else
      launch_chained(topk_row_kernel<TOPK, 32, T>, static_cast<unsigned>(rows), 256, 0, stream, scores, out, H, K, T_, nvp, fb, fe_start);
    return cudaGetLastError() == cudaSuccess ? MSA_OK : MSA_ERR_LAUNCH;
  }
  const int tok_blocks = (T_ + 31) / 32;
  const long long ctas = static_cast<long long>(tok_blocks) * H;
  if (ctas > 0x7fffffffLL) return MSA_ERR_TOO_LARGE;
  const unsigned grid = static_cast<unsigned>(ctas);
  // enough slices to put ~16 warps on every SM, bounded by the pages there are to scan
  const int most = one_word ? 8 : 16, least_blocks = one_word ? 2 : 1;      // blocks of TOPK pages per slice
  int slices = 1;
  while (slices < most && ctas * slices < 148LL * 16 && nvp / (slices * 2) >= least_blocks * TOPK) slices *= 2;
  const size_t smem = static_cast<size_t>(slices) * 32 * TOPK * 4;
  if (one_word) {
    auto kern = topk_select_kernel<TOPK, T>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    launch_chained(kern, grid, 32 * slices, smem, stream, scores, out, H, K, T_, nvp, slices);
  } else {
    auto kern = fb > 0 || fe_start < nvp ? topk_threshold_kernel<TOPK, T, true> : topk_threshold_kernel<TOPK, T, false>;
    if (smem > 44 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    launch_chained(kern, grid, 32 * slices, smem, stream, scores, out, H, K, T_, nvp, fb, fe_start, slices);
  }
  return cudaGetLastError() == cudaSuccess ? MSA_OK : MSA_ERR_LAUNCH;
}

}  // namespace
}  // namespace msa

extern "C" int msa_topk_select(const void* scores, int32_t score_dtype, int32_t* out, int32_t num_heads,
                               int32_t max_k_tiles, int32_t total_q, int32_t topk, int32_t num_valid_pages,
                               int32_t force_begin, int32_t force_end, msa_stream_t stream_) {
  using namespace msa;
  if (!scores || !out || num_heads < 0 || total_q < 0 || max_k_tiles <= 0) return MSA_ERR_BAD_ARG;
  if (num_valid_pages <= 0 || num_valid_pages > max_k_tiles) return MSA_ERR_BAD_ARG;
  if (force_begin < 0 || force_end < 0 || force_begin + force_end > topk) return MSA_ERR_BAD_ARG;
  msa::NvtxRange range("msa_topk_select");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
#define MSA_TOPK_CASE(KK)                                                                                          \
  case KK:                                                                                                         \
    if (score_dtype == MSA_DT_F32)                                                                                 \
      return launch<KK, float>(static_cast<const float*>(scores), out, num_heads, max_k_tiles, total_q,           \
                               num_valid_pages, force_begin, force_end, stream);                                  \
    if (score_dtype == MSA_DT_BF16)                                                                                \
      return launch<KK, __nv_bfloat16>(static_cast<const __nv_bfloat16*>(scores), out, num_heads, max_k_tiles,    \
                                       total_q, num_valid_pages, force_begin, force_end, stream);                 \
    return MSA_ERR_UNSUPPORTED;
  switch (topk) {
    MSA_TOPK_CASE(4)
    MSA_TOPK_CASE(8)
    MSA_TOPK_CASE(16)
    MSA_TOPK_CASE(32)
    default: return MSA_ERR_UNSUPPORTED;
  }
#undef MSA_TOPK_CASE
}
