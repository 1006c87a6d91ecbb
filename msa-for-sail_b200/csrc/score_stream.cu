// Per-page max score for work items of at most eight rows (the proxy pass of MSA decode: the rows are the
// index heads of one or a few query tokens, upstream sm80_fmha_fwd_mainloop.hpp:427-470 with output_o = false).
//
// HBM-bound: the K cache is read once (32 KB per bf16 page, 16 KB in e4m3), at up to 16 FLOP per byte.  A warp owns one
// 128-key page at a time and streams it, 16 keys a stage, through shared memory of its own, 16 KB (cp.async, whole
// 128-byte lines; nothing wider than a warp to synchronise).  The stages run on from page to page: up to 168 KB in
// flight per SM without a gap.  Lane 4g + t works on pieces t, t + 4, ... (16 bytes each) of keys g and g + 8 of the
// stage, and holds the same pieces of the rows of Q.
//
// Up to four rows: mixed-precision FMAs (fma.rn.f32.f16 / .bf16: fp32 accumulation, no conversion of the products),
// a chain per piece, the pieces added pairwise and the four lanes of a key with two shuffles per row.
// Five to eight rows: warp-level matrix instructions (m16n8k16: 16 keys x 8 rows).  The contraction runs over head_dim
// in whatever order the operands agree on, so a lane's pieces serve as the A fragments of consecutive steps without a
// shuffle.  (Their fp32 accumulation rounds coarser: 1.2e-7 of the score against 64 bits where the FMA chains make
// 4e-8.  So do the tcgen05 instructions, on which these rows ran before.)
// More rows run on the tcgen05 decode kernel: m16n8k16 does 32 rows at a page per ~1 000 clocks and SM, slower than HBM.
// e4m3 is widened to f16 exactly; bf16 queries on an e4m3 cache are rounded to f16.
//
// The pages of all work items are numbered through (a scan of the items' tile counts by every CTA) and dealt to the
// warps in equal runs: ragged lengths and the number of items do not matter for the balance.
//
// Measured, kernel alone on a cold L2: 24 sequences of 1 to 40 960 keys x 4 heads, bf16 (77 MB): 49.5 -> 27.7 us
// (before four rows went in a loop: that took another 2.6 us off the replay of the decode graph it is in); against a
// kernel that loaded to registers, reduced a key over 8 or 16 lanes per row and gave every item the same share of the
// grid.  At 32 x 131 072 keys x 1 head in e4m3 (537 MB) the whole decode pass went from 141 to 135 us.
#include <algorithm>

#include "common.cuh"

namespace msa {
namespace score_stream {
namespace {

constexpr int BN = 128;
constexpr int MAX_ITEMS = 4096;                  // work items numbered at a time
// e4m3, four rows: 64 registers of Q and the conversions leave three warps per scheduler waiting; with four of them (and
// rings of 8 KB, 128 KB in flight per SM) 32 sequences x 320 pages take 67 us instead of 75.
// UNROLL: of the eight stages of a page.  Four rows are 256 multiply-adds a stage and lane: unrolled eight times that is more
// code than the instruction caches hold (10 240 pages: bf16 71 -> 57 us, e4m3 67 -> 52 us with a loop; 2 pages: 8.6 -> 7.1 and
// 9.2 -> 8.0 us).  One or two rows of bf16 are 1 to 2 % better with four stages; in e4m3 they are 5 % better with all eight.
template <bool F8, int R>
struct Cfg {
  static constexpr int NWARPS = F8 && R == 4 ? 16 : 12, NTHREADS = NWARPS * 32;
  static constexpr int RING = (F8 && R == 4 ? 8 : 16) * 1024;         // per warp
  static constexpr int SMEM_BYTES = NWARPS * RING + (MAX_ITEMS + 1) * 4;
  static constexpr int UNROLL = R == 4 ? 1 : (F8 ? 8 : 4);
};

// acc += a.lo * b.lo + a.hi * b.hi, operands packed f16x2 / bf16x2, fp32 accumulate
template <bool F16>
__device__ __forceinline__ void fma2(float& acc, uint32_t a, uint32_t b) {
  if constexpr (!F16) {
    asm("{\n\t.reg .b16 al, ah, bl, bh;\n\t"
        "mov.b32 {al, ah}, %1;\n\tmov.b32 {bl, bh}, %2;\n\t"
        "fma.rn.f32.bf16 %0, al, bl, %0;\n\tfma.rn.f32.bf16 %0, ah, bh, %0;\n\t}"
        : "+f"(acc) : "r"(a), "r"(b));
  } else {
    asm("{\n\t.reg .b16 al, ah, bl, bh;\n\t"
        "mov.b32 {al, ah}, %1;\n\tmov.b32 {bl, bh}, %2;\n\t"
        "fma.rn.f32.f16 %0, al, bl, %0;\n\tfma.rn.f32.f16 %0, ah, bh, %0;\n\t}"
        : "+f"(acc) : "r"(a), "r"(b));
  }
}
__device__ __forceinline__ uint32_t e4m3x2_to_f16x2(uint32_t two_bytes) {
  uint32_t r;
  const unsigned short h = static_cast<unsigned short>(two_bytes);
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(r) : "h"(h));
  return r;
}

// F8: e4m3 cache (q e4m3 or bf16, multiplied as f16); otherwise bf16 cache and bf16 q.  R: most rows of an item.
template <bool F8, int R>
__global__ void __launch_bounds__(Cfg<F8, R>::NTHREADS, 1)
score_stream_kernel(const __grid_constant__ MsaFmhaParams p) {
  using C = Cfg<F8, R>;
  constexpr int NWARPS = C::NWARPS, NTHREADS = C::NTHREADS, RING = C::RING, UNROLL = C::UNROLL;
  constexpr bool MMA = R == 8;
  constexpr int QR = MMA ? 1 : R;                // rows of Q a lane holds (MMA: row g, the B fragments)
  constexpr int MR = MMA ? 2 : R;                // rows whose maximum a lane holds (MMA: rows 2t, 2t + 1)
  constexpr int PIECES = F8 ? 2 : 4;             // 16-byte pieces of a key per lane
  constexpr int STAGE = 2 * PIECES * 512;        // 16 keys: 2 KB in e4m3, 4 KB in bf16
  constexpr int STAGES = RING / STAGE;           // 8 or 4; a page is 8 stages
  static_assert(8 % STAGES == 0, "a page starts at the first stage of the ring");
  extern __shared__ __align__(128) unsigned char s_score[];
  __shared__ int s_warp_sum[NWARPS];
  int* s_pref = reinterpret_cast<int*>(s_score + NWARPS * RING);     // [items + 1] pages before an item
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  // A stage in shared memory: 16 rows of PPR pieces; the halves of every other 64-byte pair are swapped (piece ^ 4 in
  // odd rows), so that the reads of two neighbouring keys use different banks.
  constexpr int PPR = 4 * PIECES, ROW = PPR * 16;
  const int c_row = lane / PPR, c_piece = lane % PPR;                 // what this lane copies: rows c_row + (32 / PPR) u
  const uint32_t copy_dst = smem_u32(s_score + warp * RING) + c_row * ROW + ((c_piece ^ ((c_row & 1) << 2)) << 4);
  const unsigned char* read_row = s_score + warp * RING + g * ROW;    // what it works on: keys g and g + 8
  const int h_r = p.num_qo_heads / p.num_kv_heads, G = p.pack;
  constexpr int e = F8 ? 1 : 2;
  const int64_t tok_bytes = p.k_stride_tok * e;
  chain_begin();

  for (int base = 0; base < p.num_work; base += MAX_ITEMS) {
    const int n = min(MAX_ITEMS, p.num_work - base);
    // ---- number the pages of the items: exclusive scan of the tile counts, a run of items per thread ----
    const int run = (n + NTHREADS - 1) / NTHREADS;
    const int i0 = min(n, tid * run), i1 = min(n, i0 + run);
    int sum = 0;
    for (int i = i0; i < i1; ++i) {
      const MsaWorkItem w = p.work[base + i];
      const int b = chk(w.batch, 0, p.batch, p.status);
      // a batch slot without query tokens (graph-safe padding) has no tiles
      const int cnt = p.qo_start[b + 1] > p.qo_start[b] && w.num_rows > 0 ? max(0, w.kv_tile_end - w.kv_tile_begin) : 0;
      s_pref[i] = cnt;
      sum += cnt;
    }
    int incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += v;
    }
    if (lane == 31) s_warp_sum[warp] = incl;
    __syncthreads();
    int before = incl - sum, total = 0;
#pragma unroll
    for (int k = 0; k < NWARPS; ++k) {
      if (k < warp) before += s_warp_sum[k];
      total += s_warp_sum[k];
    }
    for (int i = i0; i < i1; ++i) {
      const int cnt = s_pref[i];
      s_pref[i] = before;
      before += cnt;
    }
    if (tid == 0) s_pref[n] = total;
    __syncthreads();

    // ---- this warp's run of pages; neighbouring runs go to different CTAs ----
    const int per = (total + static_cast<int>(gridDim.x) * NWARPS - 1) / (static_cast<int>(gridDim.x) * NWARPS);
    const int64_t lo64 = static_cast<int64_t>(warp * gridDim.x + blockIdx.x) * per;
    const int lo = static_cast<int>(min(lo64, static_cast<int64_t>(total))), hi = min(total, lo + per);
    int cur_item = -1;
    int head0 = 0, qo_base = 0, nrows = 0, min_lim = 0;
    uint32_t q[QR][16];
    int lim[MR];
    for (int first = lo; first < hi; first += 32) {
      const int cnt = min(32, hi - first);
      // lane l looks page first + l up: its item, its tile, where it lies
      int l_item = 0, l_tile = 0;
      const unsigned char* l_src = static_cast<const unsigned char*>(p.k);
      if (lane < cnt) {
        const int idx = first + lane;
        int a = 0, z = n;                                    // s_pref[a] <= idx < s_pref[z]
        while (z - a > 1) {
          const int m = (a + z) >> 1;
          if (s_pref[m] <= idx) a = m; else z = m;
        }
        l_item = a;
        const MsaWorkItem w = p.work[base + a];
        l_tile = w.kv_tile_begin + (idx - s_pref[a]);
        const int b = chk(w.batch, 0, p.batch, p.status);
        const int kvh = chk(w.head0, 0, p.num_qo_heads, p.status) / h_r;
        const int phys = chk(p.kv_indices[p.kv_page_indptr[b] + l_tile], 0, static_cast<int>(p.kv_extent), p.status);
        l_src += (static_cast<int64_t>(kvh) * p.k_stride_head + static_cast<int64_t>(phys) * p.k_stride_page) * e;
      }
      const uint64_t l_addr = reinterpret_cast<uint64_t>(l_src);
      // stage s of the run: keys 16 (s % 8) .. + 15 of page s / 8
      auto request = [&](int s, int slot) {
        const int j = s >> 3;
        const uint64_t src0 = __shfl_sync(0xffffffffu, l_addr, j & 31);
        if (j < cnt) {
          const unsigned char* src = reinterpret_cast<const unsigned char*>(src0) + ((s & 7) * 16 + c_row) * tok_bytes + c_piece * 16;
#pragma unroll
          for (int u = 0; u < 2 * PIECES; ++u) cp_async16(copy_dst + slot * STAGE + u * 512, src + u * (32 / PPR) * tok_bytes, true);
        }
        cp_async_commit();
      };
#pragma unroll
      for (int s = 0; s < STAGES - 1; ++s) request(s, s);

      for (int j = 0; j < cnt; ++j) {
        const int item = __shfl_sync(0xffffffffu, l_item, j), tile = __shfl_sync(0xffffffffu, l_tile, j);
        if (item != cur_item) {                              // the rows of this item, under the first stages
          cur_item = item;
          const MsaWorkItem w = p.work[base + item];
          const int b = chk(w.batch, 0, p.batch, p.status);
          head0 = chk(w.head0, 0, p.num_qo_heads, p.status);
          qo_base = p.qo_start[b];
          nrows = min((p.qo_start[b + 1] - qo_base) * G, w.num_rows);
          const int kv_len = p.kv_len[b], off = p.qo_offset[b];
          min_lim = min(off, kv_len - 1);                    // of row 0
#pragma unroll
          for (int m = 0; m < MR; ++m) {
            const int r = MMA ? 2 * t + m : m;
            lim[m] = r < nrows ? min(r / G + off, kv_len - 1) : -1;
          }
#pragma unroll
          for (int qr = 0; qr < QR; ++qr) {
            const int rr = min(MMA ? g : qr, nrows - 1);
            const int gtok = qo_base + rr / G, head = head0 + rr % G;
            const int64_t o = static_cast<int64_t>(gtok) * p.q_stride_tok + static_cast<int64_t>(head) * p.q_stride_head;
            if (F8 && p.q_dtype == MSA_DT_E4M3) {
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                const uint4 v = *reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(p.q) + o + i * 64 + t * 16);
                const uint32_t wv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  q[qr][i * 8 + 2 * k] = e4m3x2_to_f16x2(wv[k] & 0xffffu);
                  q[qr][i * 8 + 2 * k + 1] = e4m3x2_to_f16x2(wv[k] >> 16);
                }
              }
            } else if constexpr (F8) {                       // bf16 q against an e4m3 cache: multiply as f16
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                const uint4* src = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.q) + o + i * 64 + t * 16);
                const uint4 v0 = src[0], v1 = src[1];
                const uint32_t wv[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                  const __half2 h = __floats2half2_rn(bf16_bits_to_float(wv[k] & 0xffffu), bf16_bits_to_float(wv[k] >> 16));
                  q[qr][i * 8 + k] = *reinterpret_cast<const uint32_t*>(&h);
                }
              }
            } else {
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const uint4 v = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.q) + o + i * 32 + t * 8);
                q[qr][i * 4] = v.x; q[qr][i * 4 + 1] = v.y; q[qr][i * 4 + 2] = v.z; q[qr][i * 4 + 3] = v.w;
              }
            }
          }
        }
        float mx[MR];
#pragma unroll
        for (int m = 0; m < MR; ++m) mx[m] = -INFINITY;
        const bool all_visible = tile * BN + BN - 1 <= min_lim;
#pragma unroll UNROLL
        for (int u = 0; u < 8; ++u) {
          cp_async_wait<STAGES - 2>();
          __syncwarp();                                      // every lane's copies of this stage are in, its reads of the last one done
          uint4 v[2 * PIECES];
#pragma unroll
          for (int i = 0; i < PIECES; ++i) {
            const unsigned char* at = read_row + (u % STAGES) * STAGE + (((t + 4 * i) ^ ((g & 1) << 2)) << 4);
            v[i] = *reinterpret_cast<const uint4*>(at);
            v[PIECES + i] = *reinterpret_cast<const uint4*>(at + 8 * ROW);
          }
          float c0[MR], c1[MR];                              // scores of keys g and g + 8
          if constexpr (MMA) {
            float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < PIECES; ++i) {
              const uint32_t k0[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
              const uint32_t k8[4] = {v[PIECES + i].x, v[PIECES + i].y, v[PIECES + i].z, v[PIECES + i].w};
              if constexpr (F8) {
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                  const uint32_t a[4] = {e4m3x2_to_f16x2(k0[s] & 0xffffu), e4m3x2_to_f16x2(k8[s] & 0xffffu),
                                         e4m3x2_to_f16x2(k0[s] >> 16), e4m3x2_to_f16x2(k8[s] >> 16)};
                  mma_16816<true>(c, a, q[0][i * 8 + 2 * s], q[0][i * 8 + 2 * s + 1]);
                }
              } else {
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                  const uint32_t a[4] = {k0[2 * s], k8[2 * s], k0[2 * s + 1], k8[2 * s + 1]};
                  mma_16816<false>(c, a, q[0][i * 4 + 2 * s], q[0][i * 4 + 2 * s + 1]);
                }
              }
            }
            c0[0] = c[0]; c0[1] = c[1]; c1[0] = c[2]; c1[1] = c[3];
          } else {
            auto scores = [&](const uint4* piece, float (&c)[MR]) {
              float acc[PIECES][R];
#pragma unroll
              for (int i = 0; i < PIECES; ++i) {
                const uint32_t k[4] = {piece[i].x, piece[i].y, piece[i].z, piece[i].w};
#pragma unroll
                for (int r = 0; r < R; ++r) acc[i][r] = 0.f;
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                  if constexpr (F8) {
                    const uint32_t klo = e4m3x2_to_f16x2(k[s] & 0xffffu), khi = e4m3x2_to_f16x2(k[s] >> 16);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                      fma2<true>(acc[i][r], q[r][i * 8 + 2 * s], klo);
                      fma2<true>(acc[i][r], q[r][i * 8 + 2 * s + 1], khi);
                    }
                  } else {
#pragma unroll
                    for (int r = 0; r < R; ++r) fma2<false>(acc[i][r], q[r][i * 4 + s], k[s]);
                  }
                }
              }
#pragma unroll
              for (int r = 0; r < R; ++r) {
                float x = PIECES == 4 ? (acc[0][r] + acc[1][r]) + (acc[PIECES - 2][r] + acc[PIECES - 1][r]) : acc[0][r] + acc[1][r];
                x += __shfl_xor_sync(0xffffffffu, x, 1);
                c[r] = x + __shfl_xor_sync(0xffffffffu, x, 2);
              }
            };
            scores(v, c0);
            scores(v + PIECES, c1);
          }
          request(j * 8 + u + STAGES - 1, (u + STAGES - 1) % STAGES);   // the stage read one step ago
          if (all_visible) {
#pragma unroll
            for (int m = 0; m < MR; ++m) mx[m] = max3(mx[m], c0[m], c1[m]);
          } else {
            const int pos = tile * BN + u * 16 + g;
#pragma unroll
            for (int m = 0; m < MR; ++m)
              mx[m] = max3(mx[m], pos <= lim[m] ? c0[m] : -INFINITY, pos + 8 <= lim[m] ? c1[m] : -INFINITY);
          }
        }
#pragma unroll
        for (int m = 0; m < MR; ++m) {
          float x = mx[m];
#pragma unroll
          for (int d = 4; d < 32; d <<= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, d));
          const int r = MMA ? 2 * t + m : m;
          if (g == 0 && (MMA || t == 0) && r < nrows && tile < p.max_k_tiles) {
            const int gtok = qo_base + r / G, head = head0 + r % G;
            const int64_t o = (static_cast<int64_t>(head) * p.max_k_tiles + tile) * p.total_q + gtok;
            if (p.max_score_dtype == MSA_DT_BF16) static_cast<__nv_bfloat16*>(p.max_score)[o] = __float2bfloat16_rn(x);
            else static_cast<float*>(p.max_score)[o] = x;
          }
        }
      }
      cp_async_wait<0>();                                    // the ring starts over with the next 32 pages
      __syncwarp();
    }
    __syncthreads();                                         // s_pref is rewritten for the next items
  }
}

}  // namespace
}  // namespace score_stream

// score-only, dense page list, <= 8 rows per work item, 128-key pages
int score_stream_supported(const MsaFmhaParams& p) {
  if ((p.flags & (MSA_FLAG_OUT_O | MSA_FLAG_OUT_SCORE | MSA_FLAG_SPARSE)) != MSA_FLAG_OUT_SCORE) return 0;
  if (p.page_size != score_stream::BN || p.decode_rows <= 0 || p.decode_rows > 8) return 0;
  if (p.kv_dtype == MSA_DT_BF16 && p.q_dtype != MSA_DT_BF16) return 0;
  if (p.kv_dtype != MSA_DT_BF16 && p.kv_dtype != MSA_DT_E4M3) return 0;
  const int h_r = p.num_qo_heads / p.num_kv_heads;
  if (p.pack != h_r) return 0;
  return 1;
}

int score_stream_launch(const MsaFmhaParams& p, cudaStream_t stream) {
  using namespace score_stream;
  if (p.num_work <= 0) return MSA_OK;
  static int sms[16] = {};
  static bool attr_done[8][16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  int nsm = dev < 16 ? sms[dev] : 0;
  if (nsm == 0) {
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (dev < 16) sms[dev] = nsm;
  }
  using KernelFn = void (*)(const MsaFmhaParams);
  const KernelFn kernels[8] = {score_stream_kernel<false, 1>, score_stream_kernel<false, 2>, score_stream_kernel<false, 4>,
                               score_stream_kernel<false, 8>, score_stream_kernel<true, 1>,  score_stream_kernel<true, 2>,
                               score_stream_kernel<true, 4>,  score_stream_kernel<true, 8>};
  const int threads[8] = {Cfg<false, 1>::NTHREADS, Cfg<false, 2>::NTHREADS, Cfg<false, 4>::NTHREADS, Cfg<false, 8>::NTHREADS,
                          Cfg<true, 1>::NTHREADS,  Cfg<true, 2>::NTHREADS,  Cfg<true, 4>::NTHREADS,  Cfg<true, 8>::NTHREADS};
  const int smem[8] = {Cfg<false, 1>::SMEM_BYTES, Cfg<false, 2>::SMEM_BYTES, Cfg<false, 4>::SMEM_BYTES, Cfg<false, 8>::SMEM_BYTES,
                       Cfg<true, 1>::SMEM_BYTES,  Cfg<true, 2>::SMEM_BYTES,  Cfg<true, 4>::SMEM_BYTES,  Cfg<true, 8>::SMEM_BYTES};
  const int rows = p.decode_rows;
  const int v = (p.kv_dtype == MSA_DT_E4M3 ? 4 : 0) + (rows <= 1 ? 0 : (rows <= 2 ? 1 : (rows <= 4 ? 2 : 3)));
  if (dev >= 16 || !attr_done[v][dev]) {
    if (cudaFuncSetAttribute(kernels[v], cudaFuncAttributeMaxDynamicSharedMemorySize, smem[v]) != cudaSuccess)
      return MSA_ERR_LAUNCH;
    if (dev < 16) attr_done[v][dev] = true;
  }
  // one CTA per SM, fewer only where there cannot be a page for each
  const int64_t most_pages = static_cast<int64_t>(p.num_work) * std::max(1, p.max_k_tiles);
  const int grid = static_cast<int>(std::min<int64_t>(nsm, most_pages));
  return launch_chained(kernels[v], grid, threads[v], smem[v], stream, p) == cudaSuccess ? MSA_OK : MSA_ERR_LAUNCH;
}

}  // namespace msa
