// Top-2 MoE routing and token movement.
//
//   router      softmax(x W_r^T) -> top-2 ids + renormalised gates           jarvis_model.py:218-224
//   metadata    stable partition of assignments m = token*K + k by expert    sparse_model.cu:23-90 (M1)
//   gather      dispatched_x[slot] = x[gather_map[slot]]                     sparse_model.cu:95-112 (M2)
//   combine     out[i] = sum_k gate[i,k] * y[scatter_map[i,k]]  (+ sum, sum^2 of out)
//                                                                            sparse_model.cu:117-165 (M3),
//                                                                            jarvis_model.py:249-250
//   finalize    l_balance, act_mean, act_var                                 jarvis_model.py:244-250
//
// The reference builds the dispatch order with ONE thread walking all N*K assignments; here it
// is a parallel stable counting sort: per-chunk histograms, a scan over (chunk, expert), and a
// ballot-ranked scatter.  The order is a pure function of the ids and is bit-exact.
// All of it is HBM/latency-bound integer and copy work: no tensor cores.
#include <algorithm>

#include "common.cuh"
#include "moe_finalize.cuh"
#include "moe_router.cuh"
#include "launchers.h"

namespace jb {

namespace {

constexpr int MAX_E = 16;
constexpr int ROUTER_THREADS = 256;                 // 8 warps, one token per warp at a time
constexpr int ROUTER_TOKENS_PER_CTA = 32;             // 512 CTAs at 16k tokens: four resident per SM (64 registers)
constexpr int META_CHUNK = 256;                     // assignments per CTA of the metadata kernels
constexpr int DISP_THREADS = 256;

// ---------------------------------------------------------------------------------------------
// router
// ---------------------------------------------------------------------------------------------
template <int E>
__global__ void __launch_bounds__(ROUTER_THREADS)
router_top2_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ w_router, int n_tokens, int C,
                   int tokens_per_cta,
                   int64_t* __restrict__ topk_idx, float* __restrict__ gates, float* __restrict__ probs_out,
                   double* __restrict__ probs_sum, int* __restrict__ top1_hist) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ float w_s[];  // [E][C]
  __shared__ float p_acc[ROUTER_THREADS / 32][E];
  __shared__ int h_acc[E];
  for (int i = threadIdx.x; i < E * C; i += ROUTER_THREADS) w_s[(i / C) * C + router_w_index(i % C)] = __ldg(w_router + i);
  if (threadIdx.x < E) h_acc[threadIdx.x] = 0;
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float p_local[E];
#pragma unroll
  for (int e = 0; e < E; ++e) p_local[e] = 0.f;
  const int tok0 = blockIdx.x * tokens_per_cta;
  for (int tt = warp; tt < tokens_per_cta; tt += ROUTER_THREADS / 32) {
    const int tok = tok0 + tt;
    if (tok >= n_tokens) break;
    const __nv_bfloat16* xr = x + size_t(tok) * C;
    float acc[E];
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] = 0.f;
    for (int c = lane * 8; c < C; c += 256) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(xr + c));
      const float xv[8] = {bf16_lo(v.x), bf16_hi(v.x), bf16_lo(v.y), bf16_hi(v.y),
                           bf16_lo(v.z), bf16_hi(v.z), bf16_lo(v.w), bf16_hi(v.w)};
      router_dot8<E>(xv, w_s, C, c, acc);
    }
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] = warp_sum(acc[e]);
    router_finish<E>(acc, lane, tok, topk_idx, gates, probs_out, h_acc, p_local);
  }
  if (lane == 0) {
#pragma unroll
    for (int e = 0; e < E; ++e) p_acc[warp][e] = p_local[e];
  }
  __syncthreads();
  if (threadIdx.x < E) {
    float s = 0.f;
    for (int w = 0; w < ROUTER_THREADS / 32; ++w) s += p_acc[w][threadIdx.x];
    if (probs_sum) atomicAdd(&probs_sum[threadIdx.x], double(s));
    if (top1_hist && h_acc[threadIdx.x]) atomicAdd(&top1_hist[threadIdx.x], h_acc[threadIdx.x]);
  }
}

// RMSNorm (norm2 of the block, jarvis_model.py:25-26, :431) fused with the router: the normalised row
// is rounded to bf16 and stored for the expert GEMMs, and the SAME rounded values feed the router
// logits in the same summation order as router_top2_kernel, so routing is bit-identical to running
// the two kernels separately while the row is read from HBM once.
template <int E, int PER>
__global__ void __launch_bounds__(ROUTER_THREADS, 2)
rmsnorm_router_kernel(const float* __restrict__ x, const float* __restrict__ w_norm, float eps,
                      __nv_bfloat16* __restrict__ xn, const float* __restrict__ w_router, int n_tokens, int C,
                      int64_t* __restrict__ topk_idx, float* __restrict__ gates,
                      double* __restrict__ probs_sum, int* __restrict__ top1_hist, int* __restrict__ load,
                      unsigned long long* __restrict__ counts8, bool ahead) {
  extern __shared__ __align__(16) float w_s[];  // [E][C], [C]
  __shared__ float p_acc[ROUTER_THREADS / 32][E];
  __shared__ int h_acc[E], l_acc[PER == 1 ? E : 1];           // (the assignments of every expert are counted in a single pass alone)
  auto stage = [&] {
    // the norm's weight, four values a thread, travels with the router's rows (behind them it was a round trip more, 0.5 us)
    const int n4 = 4 * threadIdx.x;
    const float4 wn = n4 < C ? __ldg(reinterpret_cast<const float4*>(w_norm + n4)) : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = threadIdx.x; i < E * C; i += ROUTER_THREADS) w_s[(i / C) * C + router_w_index(i % C)] = __ldg(w_router + i);
    if (n4 < C) *reinterpret_cast<float4*>(w_s + E * C + n4) = wn;
  };
  static_assert(4 * ROUTER_THREADS >= 1024, "d_model is at most 1024");
  if (threadIdx.x < E) {
    h_acc[threadIdx.x] = 0;
    if (PER == 1) l_acc[threadIdx.x] = 0;
  }
  if (ahead) stage();
  pdl_wait();
  pdl_trigger();
  if (!ahead) stage();
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float p_local[E];
#pragma unroll
  for (int e = 0; e < E; ++e) p_local[e] = 0.f;
  // A warp takes PER tokens per pass: with two, their loads are in flight together, the two dependency chains interleave,
  // and the router weights read from shared memory serve both.  The CTAs are persistent (two per SM) and stride
  // over the tokens, so the router matrix is staged once per CTA.  Where one token a warp is a single pass, it is over sooner (24
  // layers and head, 600, 900, 1300 tokens 1667 -> 1637, 1848 -> 1803, 2511 -> 2480 us).  By itself, d_model 1024 and four experts, with the norm's
  // weight staged too and rows loaded side by side: 300, 1184, 2368, 9000, 16,384 tokens 5.4 -> 4.15, 5.5 -> 4.4, 5.7 -> 5.4, 12.4 -> 11.9, 24.4 -> 23.4 us (two a
  // warp and weights from L1 before); 128 channels +2 to +4 % from 1185 tokens on.
  const int n_items = (n_tokens + PER - 1) / PER;
  for (int item = blockIdx.x * (ROUTER_THREADS / 32) + warp; item < n_items; item += gridDim.x * (ROUTER_THREADS / 32)) {
    const int tok = PER * item;
    float v[PER][4][8], ss[PER], r[PER], acc[PER][E];
    const float* xr[PER];                                       // a lone last token is processed twice, stored once
#pragma unroll
    for (int k = 0; k < PER; ++k) xr[k] = x + size_t(tok + k < n_tokens ? tok + k : tok) * C;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = (i * 32 + lane) * 8;
      if (c < C) {
#pragma unroll
        for (int k = 0; k < PER; ++k) {
          const float4 a = __ldg(reinterpret_cast<const float4*>(xr[k] + c)), b = __ldg(reinterpret_cast<const float4*>(xr[k] + c) + 1);
          v[k][i][0] = a.x; v[k][i][1] = a.y; v[k][i][2] = a.z; v[k][i][3] = a.w;
          v[k][i][4] = b.x; v[k][i][5] = b.y; v[k][i][6] = b.z; v[k][i][7] = b.w;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) ss[k] = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if ((i * 32 + lane) * 8 < C) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int k = 0; k < PER; ++k) ss[k] = __fmaf_rn(v[k][i][j], v[k][i][j], ss[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      ss[k] = warp_sum(ss[k]);
      r[k] = rsqrtf(ss[k] / float(C) + eps);
#pragma unroll
      for (int e = 0; e < E; ++e) acc[k][e] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = (i * 32 + lane) * 8;
      if (c < C) {
        const float4 wa = *reinterpret_cast<const float4*>(w_s + E * C + c), wb = *reinterpret_cast<const float4*>(w_s + E * C + c + 4);
#pragma unroll
        for (int k = 0; k < PER; ++k) {
          const uint4 pk = make_uint4(pack_bf16x2(v[k][i][0] * r[k] * wa.x, v[k][i][1] * r[k] * wa.y),
                                      pack_bf16x2(v[k][i][2] * r[k] * wa.z, v[k][i][3] * r[k] * wa.w),
                                      pack_bf16x2(v[k][i][4] * r[k] * wb.x, v[k][i][5] * r[k] * wb.y),
                                      pack_bf16x2(v[k][i][6] * r[k] * wb.z, v[k][i][7] * r[k] * wb.w));
          if (k == 0 || tok + k < n_tokens) *reinterpret_cast<uint4*>(xn + size_t(tok + k) * C + c) = pk;
          const float xv[8] = {bf16_lo(pk.x), bf16_hi(pk.x), bf16_lo(pk.y), bf16_hi(pk.y),
                               bf16_lo(pk.z), bf16_hi(pk.z), bf16_lo(pk.w), bf16_hi(pk.w)};
          router_dot8<E>(xv, w_s, C, c, acc[k]);     // the same shared-memory words for every token: the compiler loads them once
        }
      }
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) {
#pragma unroll
      for (int e = 0; e < E; ++e) acc[k][e] = warp_sum(acc[k][e]);
    }
#pragma unroll
    for (int k = 0; k < PER; ++k)
      if (k == 0 || tok + k < n_tokens) router_finish<E>(acc[k], lane, tok + k, topk_idx, gates, nullptr, h_acc, p_local, PER == 1 && load ? l_acc : nullptr);
  }
  if (lane == 0) {
#pragma unroll
    for (int e = 0; e < E; ++e) p_acc[warp][e] = p_local[e];
  }
  __syncthreads();
  if (threadIdx.x < E) {
    float s = 0.f;
    for (int w = 0; w < ROUTER_THREADS / 32; ++w) s += p_acc[w][threadIdx.x];
    if (probs_sum) atomicAdd(&probs_sum[threadIdx.x], double(s));
    if (top1_hist && h_acc[threadIdx.x]) atomicAdd(&top1_hist[threadIdx.x], h_acc[threadIdx.x]);
    if (PER == 1 && load && l_acc[threadIdx.x]) atomicAdd(&load[threadIdx.x], l_acc[threadIdx.x]);
  }
  if (PER == 1 && counts8 && threadIdx.x == 32) {          // single pass: the CTA's eight tokens, a byte per expert
    unsigned long long c = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) c |= (unsigned long long)(l_acc[e]) << (8 * e);
    counts8[blockIdx.x] = c;
  }
}

// ---------------------------------------------------------------------------------------------
// dispatch metadata: stable counting sort of M = N*K assignments by expert id
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(META_CHUNK)
meta_hist_kernel(const int64_t* __restrict__ flat_idx, int M, int E, int* __restrict__ chunk_counts) {
  pdl_wait();
  pdl_trigger();
  __shared__ int h[MAX_E];
  if (threadIdx.x < MAX_E) h[threadIdx.x] = 0;
  __syncthreads();
  const int m = blockIdx.x * META_CHUNK + threadIdx.x;
  if (m < M) atomicAdd(&h[clamp_expert(flat_idx[m], E)], 1);
  __syncthreads();
  if (threadIdx.x < E) chunk_counts[blockIdx.x * E + threadIdx.x] = h[threadIdx.x];
}

// One CTA, one warp per expert: exclusive scan of the per-chunk counts of that expert, then the
// expert offsets.  chunk_base[c][e] = offsets[e] + sum_{c' < c} counts[c'][e].
__global__ void __launch_bounds__(32 * MAX_E)
meta_scan_kernel(const int* __restrict__ chunk_counts, int n_chunks, int E, int* __restrict__ chunk_base,
                 int* __restrict__ expert_counts, int* __restrict__ expert_offsets) {
  pdl_wait();
  pdl_trigger();
  __shared__ int totals[MAX_E];
  __shared__ int offs[MAX_E + 1];
  const int e = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (e < E) {
    int running = 0;
    for (int c0 = 0; c0 < n_chunks; c0 += 32) {
      const int c = c0 + lane;
      const int v = c < n_chunks ? chunk_counts[c * E + e] : 0;
      int incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      if (c < n_chunks) chunk_base[c * E + e] = running + incl - v;  // offsets[e] added below
      running += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) totals[e] = running;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int i = 0; i < E; ++i) { offs[i] = acc; acc += totals[i]; }
    offs[E] = acc;
    for (int i = 0; i < E; ++i) { expert_counts[i] = totals[i]; expert_offsets[i] = offs[i]; }
    expert_offsets[E] = acc;
  }
  __syncthreads();
  if (e < E) {
    const int add = offs[e];
    for (int c = lane; c < n_chunks; c += 32) chunk_base[c * E + e] += add;
  }
}

__global__ void __launch_bounds__(META_CHUNK)
meta_assign_kernel(const int64_t* __restrict__ flat_idx, int M, int K, int E, const int* __restrict__ chunk_base,
                   int* __restrict__ scatter_map, int* __restrict__ gather_map, int* __restrict__ gate_idx_map) {
  pdl_wait();
  pdl_trigger();
  __shared__ int warp_cnt[META_CHUNK / 32][MAX_E];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m = blockIdx.x * META_CHUNK + threadIdx.x;
  const int e = m < M ? clamp_expert(flat_idx[m], E) : -1;
  int rank = 0;  // assignments of the same expert earlier in this warp
  for (int q = 0; q < E; ++q) {
    const unsigned mask = __ballot_sync(0xffffffffu, e == q);
    if (e == q) rank = __popc(mask & ((1u << lane) - 1u));
    if (lane == 0) warp_cnt[warp][q] = __popc(mask);
  }
  __syncthreads();
  if (m < M) {
    int before = 0;
    for (int w = 0; w < warp; ++w) before += warp_cnt[w][e];
    const int slot = chunk_base[blockIdx.x * E + e] + before + rank;
    scatter_map[m] = slot;
    gather_map[slot] = m / K;
    gate_idx_map[slot] = m % K;
  }
}

// Up to 2048 assignments: the three kernels above in one CTA, ROUNDS of them per thread, all loaded at once.  Same stable
// order: earlier assignments of the same expert come first.  24 layers of 600 tokens 1952 -> 1898 us against the three launches;
// from 2000 tokens on one SM's stores take longer than they do (2331 tokens 3125 -> 3176).
constexpr int META_SMALL_MAX = 2048, META_THREADS = 1024;
template <int ROUNDS>
__global__ void __launch_bounds__(META_THREADS)
meta_small_kernel(const int64_t* __restrict__ flat_idx, int M, int K, int E, int* __restrict__ expert_counts,
                  int* __restrict__ expert_offsets, int* __restrict__ scatter_map, int* __restrict__ gather_map,
                  int* __restrict__ gate_idx_map) {
  pdl_wait();
  pdl_trigger();
  constexpr int SPANS = ROUNDS * META_THREADS / 32, PER_LANE = ROUNDS;     // 32 assignments each; spans of a lane of the scan
  __shared__ int ahead[MAX_E][SPANS];              // assignments of an expert in the span, then in all spans before it
  __shared__ int total[MAX_E];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = int(blockDim.x) >> 5, n_spans = ROUNDS * n_warps;
  int e[ROUNDS], rank[ROUNDS];
#pragma unroll
  for (int i = 0; i < ROUNDS; ++i) {
    const int m = i * int(blockDim.x) + int(threadIdx.x);
    e[i] = m < M ? clamp_expert(flat_idx[m], E) : -1;
    rank[i] = 0;
  }
#pragma unroll
  for (int i = 0; i < ROUNDS; ++i) {
    for (int q = 0; q < E; ++q) {
      const unsigned mask = __ballot_sync(0xffffffffu, e[i] == q);
      if (e[i] == q) rank[i] = __popc(mask & ((1u << lane) - 1u));
      if (lane == 0) ahead[q][i * n_warps + warp] = __popc(mask);
    }
  }
  __syncthreads();
  for (int q = warp; q < E; q += n_warps) {
    int c[PER_LANE], sum = 0;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
      const int k = lane * PER_LANE + j;
      c[j] = k < n_spans ? ahead[q][k] : 0;
      sum += c[j];
    }
    int incl = sum;
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += u;
    }
    int before = incl - sum;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
      const int k = lane * PER_LANE + j;
      if (k < n_spans) ahead[q][k] = before;
      before += c[j];
    }
    if (lane == 31) total[q] = incl;
  }
  __syncthreads();
  if (threadIdx.x <= E) {
    int off = 0;
    for (int q = 0; q < int(threadIdx.x); ++q) off += total[q];
    expert_offsets[threadIdx.x] = off;
    if (threadIdx.x < E) expert_counts[threadIdx.x] = total[threadIdx.x];
  }
#pragma unroll
  for (int i = 0; i < ROUNDS; ++i) {
    if (e[i] >= 0) {
      const int m = i * int(blockDim.x) + int(threadIdx.x);
      int slot = ahead[e[i]][i * n_warps + warp] + rank[i];
      for (int q = 0; q < e[i]; ++q) slot += total[q];
      scatter_map[m] = slot;
      gather_map[slot] = m / K;
      gate_idx_map[slot] = m % K;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// dispatch of top-2 assignments: maps and rows in one launch
// ---------------------------------------------------------------------------------------------
template <int E, int TOK>
__global__ void __launch_bounds__(2 * TOK)
dispatch_hist_kernel(const int64_t* __restrict__ topk_idx, int M, int* __restrict__ chunk_counts) {
  pdl_wait();
  pdl_trigger();
  __shared__ int h[E];
  if (threadIdx.x < E) h[threadIdx.x] = 0;
  __syncthreads();
  const int m = blockIdx.x * (2 * TOK) + threadIdx.x;
  if (m < M) atomicAdd(&h[clamp_expert(topk_idx[m], E)], 1);
  __syncthreads();
  if (threadIdx.x < E) chunk_counts[blockIdx.x * E + threadIdx.x] = h[threadIdx.x];
}

// One CTA per chunk of 32 tokens, or of 64 where that leaves few counts and CTAs enough.  Every CTA adds up the counts of all
// chunks (E integers each, from L2), ranks its assignments with ballots - the order of the kernels above - and copies its rows:
// each is read once and stored at both of its slots, where the gather reads every row twice.  For an MoE layer called by itself;
// sizes and times at one_launch_dispatch.
// Inside the native call the counts are taken from the ids themselves (IDS, up to 512 tokens) or from what the router left for every
// eight tokens (EIGHTS), by every CTA, and the first expert matrix reads the segments off the router's counts while this kernel runs.
// Latency: ids or counts and rows travel together, then one exchange over the CTA.  24 layers and head against metadata (256 tokens:
// by the router's last warp, 3.6 of its 7 us) and gather: 180 tokens 1104 -> 1064 us, 256 1180 -> 1130, steps of 256 sequences 1528 ->
// 1484, all from the ids; then with sums per expert by shared-memory additions instead of a table that every thread adds up, and from the
// router's counts beyond 512: 256 1084 -> 1054, 512 1440 -> 1413, 900 1741 -> 1686, 1300 2436 -> 2381, 3 x 777 2861 -> 2804 (2929 with
// metadata and gather).  Up to 2368 tokens the router is one pass of eight tokens a CTA; from 3000 on, from the ids, it was no faster.
enum DispatchCounts { CHUNKS, IDS, EIGHTS };
template <int E, int TOK, DispatchCounts FROM>
__global__ void __launch_bounds__(DISP_THREADS)
dispatch_kernel(const int64_t* __restrict__ topk_idx, const __nv_bfloat16* __restrict__ x, const void* __restrict__ counted,
                int n_tokens, int C, int* __restrict__ expert_counts, int* __restrict__ expert_offsets, int* __restrict__ scatter_map,
                int* __restrict__ gather_map, int* __restrict__ gate_idx_map, __nv_bfloat16* __restrict__ dispatched) {
  constexpr int WARPS = DISP_THREADS / 32, RANK_WARPS = (2 * TOK + 31) / 32, PER_WARP = TOK / WARPS, ROWS = PER_WARP < 2 ? 1 : 2;
  __shared__ int all_of[E], ahead_of[E], in_warp[RANK_WARPS][E], slots[2 * TOK];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < E) all_of[tid] = ahead_of[tid] = 0;
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  const int tok0 = int(blockIdx.x) * TOK, M = 2 * n_tokens, m = 2 * tok0 + tid;
  // the warp's first two rows and its assignments travel while the counts are added up
  const int first = tok0 + warp * PER_WARP;
  uint4 row[ROWS][4];
  auto load_rows = [&](int t) {
#pragma unroll
    for (int k = 0; k < ROWS; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = (i * 32 + lane) * 8;
        if (first + t + k < n_tokens && c < C) row[k][i] = __ldg(reinterpret_cast<const uint4*>(x + size_t(first + t + k) * C + c));
      }
  };
  load_rows(0);
  const int e = tid < 2 * TOK && m < M ? clamp_expert(topk_idx[m], E) : -1;
  int total[E], before[E];
#pragma unroll
  for (int q = 0; q < E; ++q) total[q] = before[q] = 0;
  if constexpr (FROM != CHUNKS) {
    unsigned long long all = 0, ahead = 0;               // a byte per expert and thread
    if constexpr (FROM == IDS) {
#pragma unroll 2
      for (int t = tid; t < n_tokens; t += DISP_THREADS) {
        const longlong2 id = __ldcg(reinterpret_cast<const longlong2*>(topk_idx) + t);
        const unsigned long long two = (1ull << (8 * clamp_expert(id.x, E))) + (1ull << (8 * clamp_expert(id.y, E)));
        all += two;
        ahead += t < tok0 ? two : 0ull;
      }
    } else {
#pragma unroll 2
      for (int c = tid; 8 * c < n_tokens; c += DISP_THREADS) {
        const unsigned long long v = __ldcg(static_cast<const unsigned long long*>(counted) + c);
        all += v;
        ahead += 8 * c < tok0 ? v : 0ull;
      }
    }
#pragma unroll
    for (int q = 0; q < E; ++q) {
      total[q] = int(all >> (8 * q)) & 0xff;
      before[q] = int(ahead >> (8 * q)) & 0xff;
    }
  } else {
    for (int c = tid; c < int(gridDim.x); c += DISP_THREADS) {
#pragma unroll
      for (int q4 = 0; q4 < E / 4; ++q4) {
        const int4 v = __ldcg(reinterpret_cast<const int4*>(static_cast<const int*>(counted) + size_t(c) * E) + q4);
        const int w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          total[4 * q4 + q] += w[q];
          before[4 * q4 + q] += c < int(blockIdx.x) ? w[q] : 0;
        }
      }
    }
  }
  int mine = 0, before_mine = 0;                           // lane e: the warp's sums of expert e
#pragma unroll
  for (int q = 0; q < E; ++q) {
    const int a = __reduce_add_sync(0xffffffffu, total[q]), b = __reduce_add_sync(0xffffffffu, before[q]);
    if (lane == q) { mine = a; before_mine = b; }
  }
  if (lane < E) {
    atomicAdd(&all_of[lane], mine);
    atomicAdd(&ahead_of[lane], before_mine);
  }
  int rank = 0;
  if (warp < RANK_WARPS) {
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const unsigned mask = __ballot_sync(0xffffffffu, e == q);
      if (e == q) rank = __popc(mask & ((1u << lane) - 1u));
      if (lane == 0) in_warp[warp][q] = __popc(mask);
    }
  }
  __syncthreads();
  if (e >= 0) {
    int slot = rank + ahead_of[e];
    for (int q = 0; q < e; ++q) slot += all_of[q];
    for (int w = 0; w < warp; ++w) slot += in_warp[w][e];
    scatter_map[m] = slot;
    gather_map[slot] = m >> 1;
    gate_idx_map[slot] = m & 1;
    slots[tid] = slot;
  }
  if (blockIdx.x == 0 && tid <= E) {
    int off = 0;
    for (int q = 0; q < tid; ++q) off += all_of[q];
    expert_offsets[tid] = off;
    if (tid < E) expert_counts[tid] = all_of[tid];
  }
  __syncthreads();
  for (int t = 0; t < PER_WARP; t += ROWS) {
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      if (first + t + k >= n_tokens) continue;
      const int at = 2 * (warp * PER_WARP + t + k);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        __nv_bfloat16* dst = dispatched + size_t(min(max(slots[at + h], 0), M - 1)) * C;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int c = (i * 32 + lane) * 8;
          if (c < C) *reinterpret_cast<uint4*>(dst + c) = row[k][i];
        }
      }
    }
    if (t + ROWS < PER_WARP) load_rows(t + ROWS);
  }
}

// ---------------------------------------------------------------------------------------------
// gather / combine
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
dispatch_gather_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ gather_map, int M, int n_tokens,
                       int C, __nv_bfloat16* __restrict__ dispatched) {
  pdl_wait();
  pdl_trigger();
  const int slot = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (slot >= M) return;
  const int lane = threadIdx.x & 31;
  int tok = gather_map[slot];
  tok = tok < 0 ? 0 : (tok >= n_tokens ? n_tokens - 1 : tok);
  const uint4* src = reinterpret_cast<const uint4*>(x + size_t(tok) * C);
  uint4* dst = reinterpret_cast<uint4*>(dispatched + size_t(slot) * C);
  for (int c = lane; c < C / 8; c += 32) dst[c] = __ldg(src + c);
}

template <typename TOut>
__global__ void __launch_bounds__(256)
scatter_combine_kernel(const __nv_bfloat16* __restrict__ y, const float* __restrict__ gates,
                       const int* __restrict__ scatter_map, int n_tokens, int K, int M, int C,
                       TOut* __restrict__ out, double* __restrict__ stats) {
  pdl_wait();
  pdl_trigger();
  __shared__ float red[2][8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tok = blockIdx.x * 8 + warp;
  float s1 = 0.f, s2 = 0.f;
  if (tok < n_tokens) {
    for (int c = lane * 8; c < C; c += 256) {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int k = 0; k < K; ++k) {
        int slot = scatter_map[size_t(tok) * K + k];
        slot = slot < 0 ? 0 : (slot >= M ? M - 1 : slot);
        const float g = gates[size_t(tok) * K + k];
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(y + size_t(slot) * C + c));
        acc[0] += g * bf16_lo(v.x); acc[1] += g * bf16_hi(v.x); acc[2] += g * bf16_lo(v.y); acc[3] += g * bf16_hi(v.y);
        acc[4] += g * bf16_lo(v.z); acc[5] += g * bf16_hi(v.z); acc[6] += g * bf16_lo(v.w); acc[7] += g * bf16_hi(v.w);
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) { s1 += acc[j]; s2 += acc[j] * acc[j]; }
      if constexpr (sizeof(TOut) == 2) {
        *reinterpret_cast<uint4*>(out + size_t(tok) * C + c) =
            make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                       pack_bf16x2(acc[6], acc[7]));
      } else {
        float4* o = reinterpret_cast<float4*>(out + size_t(tok) * C + c);
        o[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
        o[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
      }
    }
  }
  if (stats) {
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if (lane == 0) { red[0][warp] = s1; red[1][warp] = s2; }
    __syncthreads();
    if (threadIdx.x == 0) {
      double a = 0.0, b = 0.0;
      for (int w = 0; w < 8; ++w) { a += double(red[0][w]); b += double(red[1][w]); }
      atomicAdd(&stats[0], a);
      atomicAdd(&stats[1], b);
    }
  }
}

// Top-2 rows of up to 1024 channels: slots and gates before the grid dependency (`ahead`: the kernel before this one made y
// alone), then all of a lane's loads at once; sums and roundings in the order of the kernel above.
// With the router's weights staged ahead of the dependency as well: 24 layers of 256 tokens 1645 -> 1555 us.
template <typename TOut>
__global__ void __launch_bounds__(256)
top2_combine_kernel(const __nv_bfloat16* __restrict__ y, const float* __restrict__ gates, const int* __restrict__ scatter_map,
                    const int64_t* __restrict__ topk_idx, int n_tokens, int C, bool ahead, TOut* __restrict__ out,
                    double* __restrict__ stats) {
  __shared__ float red[2][8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tok = blockIdx.x * 8 + warp, M = 2 * n_tokens;
  int2 sl = make_int2(0, 0);
  float2 g = make_float2(0.f, 0.f);
  auto route = [&] {
    if (tok >= n_tokens) return;
    sl = *(reinterpret_cast<const int2*>(scatter_map) + tok);
    g = *(reinterpret_cast<const float2*>(gates) + tok);
    sl.x = sl.x < 0 ? 0 : (sl.x >= M ? M - 1 : sl.x);
    sl.y = sl.y < 0 ? 0 : (sl.y >= M ? M - 1 : sl.y);
    if (topk_idx && topk_idx[2 * tok + 1] < 0) sl.y = sl.x;
  };
  if (ahead) route();
  __syncwarp();
  pdl_wait();
  pdl_trigger();
  if (!ahead) route();
  float s1 = 0.f, s2 = 0.f;
  if (tok < n_tokens) {
    uint4 v[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = (i * 32 + lane) * 8;
      if (c < C) {
        v[i][0] = __ldg(reinterpret_cast<const uint4*>(y + size_t(sl.x) * C + c));
        v[i][1] = __ldg(reinterpret_cast<const uint4*>(y + size_t(sl.y) * C + c));
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = (i * 32 + lane) * 8;
      if (c < C) {
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float gk = k ? g.y : g.x;
          const uint4 w = v[i][k];
          acc[0] += gk * bf16_lo(w.x); acc[1] += gk * bf16_hi(w.x); acc[2] += gk * bf16_lo(w.y); acc[3] += gk * bf16_hi(w.y);
          acc[4] += gk * bf16_lo(w.z); acc[5] += gk * bf16_hi(w.z); acc[6] += gk * bf16_lo(w.w); acc[7] += gk * bf16_hi(w.w);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) { s1 += acc[j]; s2 += acc[j] * acc[j]; }
        if constexpr (sizeof(TOut) == 2) {
          *reinterpret_cast<uint4*>(out + size_t(tok) * C + c) =
              make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                         pack_bf16x2(acc[6], acc[7]));
        } else {
          float4* o = reinterpret_cast<float4*>(out + size_t(tok) * C + c);
          o[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
          o[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
        }
      }
    }
  }
  if (stats) {
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if (lane == 0) { red[0][warp] = s1; red[1][warp] = s2; }
    __syncthreads();
    if (threadIdx.x == 0) {
      double a = 0.0, b = 0.0;
      for (int w = 0; w < 8; ++w) { a += double(red[0][w]); b += double(red[1][w]); }
      atomicAdd(&stats[0], a);
      atomicAdd(&stats[1], b);
    }
  }
}

// scalars[0] = l_balance, [1] = act_mean, [2] = act_var (unbiased), all f32.
__global__ void moe_finalize_kernel(const double* __restrict__ stats, const double* __restrict__ probs_sum,
                                    const int* __restrict__ top1_hist, int E, long long n_tokens, long long n_elems,
                                    float balance_alpha, float* __restrict__ scalars) {
  pdl_wait();
  pdl_trigger();
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  moe_finalize_scalars(stats, probs_sum, top1_hist, E, n_tokens, n_elems, balance_alpha, scalars);
}

}  // namespace

int launch_router_top2(const void* x_bf16, const float* w_router, int n_tokens, int C, int E, int64_t* topk_idx,
                       float* gates, float* probs_out, double* probs_sum, int* top1_hist, cudaStream_t stream) {
  JB_REQUIRE(n_tokens >= 0 && C > 0, "router_top2: bad shape");
  JB_REQUIRE(E == 4 || E == 8, "router_top2: num_experts (%d) must be 4 or 8", E);
  JB_REQUIRE(C % 8 == 0 && size_t(E) * C * 4 <= 160 * 1024, "router_top2: d_model (%d) must be a multiple of 8 and fit shared memory", C);
  if (n_tokens == 0) return JB200_OK;
  JB_REQUIRE(x_bf16 && w_router && topk_idx && gates, "router_top2: null pointer");
  JB_REQUIRE(aligned16(x_bf16) && aligned16(w_router), "router_top2: pointers must be 16-byte aligned");
  if (n_tokens == 0) return JB200_OK;
  // small batches (decode steps): one token per warp so that more than a handful of CTAs exist
  const int tpc = n_tokens <= 4096 ? ROUTER_THREADS / 32 : ROUTER_TOKENS_PER_CTA;
  const int blocks = (n_tokens + tpc - 1) / tpc;
  const size_t smem = size_t(E) * C * sizeof(float);
  if (E == 4) {
    JB_MAX_SMEM(router_top2_kernel<4>, 160 * 1024);
    launch_dep(router_top2_kernel<4>, blocks, ROUTER_THREADS, smem, stream,
        reinterpret_cast<const __nv_bfloat16*>(x_bf16), w_router, n_tokens, C, tpc, topk_idx, gates, probs_out, probs_sum,
        top1_hist);
  } else {
    JB_MAX_SMEM(router_top2_kernel<8>, 160 * 1024);
    launch_dep(router_top2_kernel<8>, blocks, ROUTER_THREADS, smem, stream,
        reinterpret_cast<const __nv_bfloat16*>(x_bf16), w_router, n_tokens, C, tpc, topk_idx, gates, probs_out, probs_sum,
        top1_hist);
  }
  JB_LAUNCH_CHECK("router_top2_kernel");
  return JB200_OK;
}

int launch_rmsnorm_router(const float* x, const float* w_norm, float eps, void* xn_bf16, const float* w_router,
                          int n_tokens, int C, int E, int64_t* topk_idx, float* gates, double* probs_sum,
                          int* top1_hist, cudaStream_t stream, bool ahead, int* load,
                          unsigned long long* counts8) {
  JB_REQUIRE(n_tokens >= 0 && C > 0, "rmsnorm_router: bad shape");
  JB_REQUIRE(E == 4 || E == 8, "rmsnorm_router: num_experts (%d) must be 4 or 8", E);
  JB_REQUIRE(C % 8 == 0 && C <= 1024, "rmsnorm_router: d_model (%d) must be a multiple of 8 and at most 1024", C);
  if (n_tokens == 0) return JB200_OK;
  JB_REQUIRE(x && w_norm && xn_bf16 && w_router && topk_idx && gates, "rmsnorm_router: null pointer");
  JB_REQUIRE(aligned16(x) && aligned16(w_norm) && aligned16(xn_bf16) && aligned16(w_router),
             "rmsnorm_router: pointers must be 16-byte aligned");
  if (n_tokens == 0) return JB200_OK;
  // persistent CTAs, two per SM, striding over the tokens: two per warp and pass, or one where that leaves a single pass.  By itself only
  // while that is one CTA an SM (d_model 1024, four experts, 1184 and 2368 tokens: 4.4 and 5.95 us with one, 5.4 and 5.4 with two); with counts of
  // eight tokens up to two, for what they save behind it.
  const int sms = sm_count();
  if (sms <= 0) return JB200_ERR_CUDA;
  const int warps = ROUTER_THREADS / 32, per = n_tokens <= (counts8 ? 2 : 1) * sms * warps ? 1 : 2;
  const int blocks = std::min((n_tokens + per * warps - 1) / (per * warps), 2 * sms);
  JB_REQUIRE((!counts8 && !load) || (counts8 && load && per == 1), "rmsnorm_router: counts need a single pass");
  const size_t smem = size_t(E + 1) * C * sizeof(float);      // the router's rows and the norm's
  __nv_bfloat16* xn = reinterpret_cast<__nv_bfloat16*>(xn_bf16);
  auto kernel = per == 1 ? (E == 4 ? rmsnorm_router_kernel<4, 1> : rmsnorm_router_kernel<8, 1>)
                         : (E == 4 ? rmsnorm_router_kernel<4, 2> : rmsnorm_router_kernel<8, 2>);
  launch_dep(kernel, blocks, ROUTER_THREADS, smem, stream, x, w_norm, eps, xn, w_router, n_tokens, C, topk_idx, gates, probs_sum, top1_hist,
             load, counts8, ahead);
  JB_LAUNCH_CHECK("rmsnorm_router_kernel");
  return JB200_OK;
}

size_t moe_metadata_scratch_bytes(int n_tokens, int K, int E) {
  if (n_tokens <= 0 || K <= 0 || E <= 0) return 0;
  const size_t chunks = (size_t(n_tokens) * K + META_CHUNK - 1) / META_CHUNK;
  return 2 * chunks * size_t(E) * sizeof(int);
}

namespace {
// Where the metadata are one CTA's work, metadata and gather are two launches as well, and shorter ones; beyond, they are four, which a
// layer called by itself pays for on the host up to some 8000 tokens (4000 tokens 137 us, 133 with two).  Device time of metadata and
// gather -> histogram and dispatch_kernel: 4 experts, 1024 channels: 300 tokens 3.8 -> 7.4 us, 1024 5.2 -> 7.5, 4096 8.2 -> 8.0, 8192
// 11.3 -> 11.2, 16,384 18.4 -> 18.9, 32,768 43.7 -> 41.1, 65,536 88.5 -> 71.0, 131,072 170 -> 135, 262,144 333 -> 261, 524,288 659 -> 537.
// 8 experts, 512 channels (twice the counts, half the rows): 16,384 12.4 -> 14.5, 32,768 equal, 131,072 102 -> 84, 262,144
// 206 -> 195, 524,288 408 -> 494: every CTA adds up all counts.
constexpr int DISPATCH_MAX = 262144;
bool one_launch_dispatch(int n_tokens) { return 2 * n_tokens > META_SMALL_MAX && n_tokens <= DISPATCH_MAX; }
int dispatch_tokens(int n_tokens) { return n_tokens <= 16384 ? 32 : 64; }      // per CTA: 8000 tokens fill the chip only with the smaller
int dispatch_chunks(int n_tokens) { return (n_tokens + dispatch_tokens(n_tokens) - 1) / dispatch_tokens(n_tokens); }
}  // namespace

size_t moe_dispatch_scratch_bytes(int n_tokens, int E) {
  return one_launch_dispatch(n_tokens) ? size_t(dispatch_chunks(n_tokens)) * E * sizeof(int) : moe_metadata_scratch_bytes(n_tokens, 2, E);
}

int launch_moe_dispatch(const int64_t* topk_idx, const void* x_bf16, int n_tokens, int C, int E, void* scratch, int* expert_counts,
                        int* expert_offsets, int* scatter_map, int* gather_map, int* gate_idx_map, void* dispatched, cudaStream_t stream) {
  JB_REQUIRE(n_tokens >= 1 && n_tokens < (1 << 30) && (E == 4 || E == 8) && C >= 8 && C % 8 == 0 && C <= 1024,
             "moe_dispatch: bad shape (N=%d, C=%d, E=%d)", n_tokens, C, E);
  JB_REQUIRE(topk_idx && x_bf16 && scratch && expert_counts && expert_offsets && scatter_map && gather_map && gate_idx_map && dispatched,
             "moe_dispatch: null pointer");
  JB_REQUIRE(aligned16(x_bf16) && aligned16(dispatched) && aligned16(scratch), "moe_dispatch: pointers must be 16-byte aligned");
  if (!one_launch_dispatch(n_tokens)) {
    const int rc = launch_moe_metadata(topk_idx, n_tokens, 2, E, expert_counts, expert_offsets, scatter_map, gather_map, gate_idx_map,
                                       scratch, stream);
    return rc == JB200_OK ? launch_dispatch_gather(x_bf16, gather_map, 2 * n_tokens, n_tokens, C, dispatched, stream) : rc;
  }
  const int tok = dispatch_tokens(n_tokens), blocks = dispatch_chunks(n_tokens);
  int* chunk_counts = static_cast<int*>(scratch);
  const __nv_bfloat16* x = reinterpret_cast<const __nv_bfloat16*>(x_bf16);
  __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(dispatched);
  auto hist = tok == 32 ? (E == 4 ? dispatch_hist_kernel<4, 32> : dispatch_hist_kernel<8, 32>)
                        : (E == 4 ? dispatch_hist_kernel<4, 64> : dispatch_hist_kernel<8, 64>);
  launch_dep(hist, blocks, 2 * tok, 0, stream, topk_idx, 2 * n_tokens, chunk_counts);
  JB_LAUNCH_CHECK("dispatch_hist_kernel");
  auto kernel = tok == 32 ? (E == 4 ? dispatch_kernel<4, 32, CHUNKS> : dispatch_kernel<8, 32, CHUNKS>)
                          : (E == 4 ? dispatch_kernel<4, 64, CHUNKS> : dispatch_kernel<8, 64, CHUNKS>);
  launch_dep(kernel, blocks, DISP_THREADS, 0, stream, topk_idx, x, chunk_counts, n_tokens, C, expert_counts, expert_offsets, scatter_map,
             gather_map, gate_idx_map, d);
  JB_LAUNCH_CHECK("dispatch_kernel");
  return JB200_OK;
}

int launch_dispatch_chain(const int64_t* topk_idx, const unsigned long long* counts8, const void* x_bf16, int n_tokens, int C, int E,
                          int* expert_counts, int* expert_offsets, int* scatter_map, int* gather_map, int* gate_idx_map, void* dispatched,
                          cudaStream_t stream) {
  JB_REQUIRE(n_tokens >= 1 && n_tokens <= (counts8 ? DISPATCH_EIGHTS_MAX : DISPATCH_IDS_MAX) && (E == 4 || E == 8) && C >= 8 && C % 8 == 0 &&
                 C <= 1024,
             "dispatch_chain: bad shape (N=%d, C=%d, E=%d)", n_tokens, C, E);
  JB_REQUIRE(topk_idx && x_bf16 && expert_counts && expert_offsets && scatter_map && gather_map && gate_idx_map && dispatched,
             "dispatch_chain: null pointer");
  JB_REQUIRE(aligned16(topk_idx) && aligned16(x_bf16) && aligned16(dispatched), "dispatch_chain: pointers must be 16-byte aligned");
  static_assert(DISPATCH_IDS_MAX / DISP_THREADS * 2 < 256 && (DISPATCH_EIGHTS_MAX / 8 + DISP_THREADS - 1) / DISP_THREADS * 16 < 256,
                "a byte per expert and thread");
  const int sms = sm_count();
  if (sms <= 0) return JB200_ERR_CUDA;
  const bool few = n_tokens <= 8 * sms;                    // a wave of CTAs, as small as they go
  auto kernel = counts8 ? (few ? (E == 4 ? dispatch_kernel<4, 8, EIGHTS> : dispatch_kernel<8, 8, EIGHTS>)
                               : (E == 4 ? dispatch_kernel<4, 16, EIGHTS> : dispatch_kernel<8, 16, EIGHTS>))
                        : (E == 4 ? dispatch_kernel<4, 8, IDS> : dispatch_kernel<8, 8, IDS>);
  const int tok = few || !counts8 ? 8 : 16;
  launch_dep(kernel, (n_tokens + tok - 1) / tok, DISP_THREADS, 0, stream, topk_idx, reinterpret_cast<const __nv_bfloat16*>(x_bf16),
             static_cast<const void*>(counts8), n_tokens, C, expert_counts, expert_offsets, scatter_map, gather_map, gate_idx_map,
             reinterpret_cast<__nv_bfloat16*>(dispatched));
  JB_LAUNCH_CHECK("dispatch_kernel");
  return JB200_OK;
}

int launch_moe_metadata(const int64_t* topk_idx, int n_tokens, int K, int E, int* expert_counts, int* expert_offsets,
                        int* scatter_map, int* gather_map, int* gate_idx_map, void* scratch, cudaStream_t stream) {
  JB_REQUIRE(n_tokens >= 0 && K >= 1 && K <= 8, "moe_metadata: bad shape (N=%d, K=%d)", n_tokens, K);
  JB_REQUIRE(E >= 1 && E <= MAX_E, "moe_metadata: num_experts (%d) must be in 1..%d", E, MAX_E);
  JB_REQUIRE(size_t(n_tokens) * K < (size_t(1) << 31), "moe_metadata: too many assignments");
  JB_REQUIRE(expert_counts && expert_offsets, "moe_metadata: null pointer");
  const int M = n_tokens * K;
  const int chunks = (M + META_CHUNK - 1) / META_CHUNK;
  JB_REQUIRE(M == 0 || (topk_idx && scatter_map && gather_map && gate_idx_map && scratch), "moe_metadata: null pointer");
  if (M > 0 && M <= META_SMALL_MAX) {
    const int threads = std::min(META_THREADS, (M + 31) / 32 * 32);
    auto kernel = M <= META_THREADS ? meta_small_kernel<1> : meta_small_kernel<2>;
    launch_dep(kernel, 1, threads, 0, stream, topk_idx, M, K, E, expert_counts, expert_offsets, scatter_map, gather_map,
               gate_idx_map);
    JB_LAUNCH_CHECK("meta_small_kernel");
    return JB200_OK;
  }
  int* chunk_counts = reinterpret_cast<int*>(scratch);
  int* chunk_base = chunk_counts + size_t(chunks) * E;
  if (M > 0) {
    launch_dep(meta_hist_kernel, chunks, META_CHUNK, 0, stream, topk_idx, M, E, chunk_counts);
    JB_LAUNCH_CHECK("meta_hist_kernel");
  }
  launch_dep(meta_scan_kernel, 1, 32 * MAX_E, 0, stream, chunk_counts, chunks, E, chunk_base, expert_counts, expert_offsets);
  JB_LAUNCH_CHECK("meta_scan_kernel");
  if (M > 0) {
    launch_dep(meta_assign_kernel, chunks, META_CHUNK, 0, stream, topk_idx, M, K, E, chunk_base, scatter_map, gather_map,
                                                          gate_idx_map);
    JB_LAUNCH_CHECK("meta_assign_kernel");
  }
  return JB200_OK;
}

// ---------------------------------------------------------------------------------------------
// Allocation-free variant of the dispatch metadata: the two work arrays live in a fixed array
// that is part of the library image, so the caller never has to provide (or allocate) scratch.
// ---------------------------------------------------------------------------------------------
constexpr int STATIC_META_MAX_ASSIGNMENTS = 1 << 18;                                 // N*K <= 262144
constexpr int STATIC_META_MAX_CHUNKS = STATIC_META_MAX_ASSIGNMENTS / META_CHUNK;     // 1024
static __device__ __align__(256) int g_meta_scratch[2 * STATIC_META_MAX_CHUNKS * MAX_E];  // 128 KiB per GPU
static int* g_meta_scratch_ptr[64] = {nullptr};   // device address of the array, one per device ordinal

int moe_metadata_static_max_assignments() { return STATIC_META_MAX_ASSIGNMENTS; }

int launch_moe_metadata_static(const int64_t* topk_idx, int n_tokens, int K, int E, int* expert_counts,
                               int* expert_offsets, int* scatter_map, int* gather_map, int* gate_idx_map,
                               cudaStream_t stream) {
  JB_REQUIRE(n_tokens >= 0 && K >= 1 && K <= 8, "moe_metadata_static: bad shape (N=%d, K=%d)", n_tokens, K);
  JB_REQUIRE(size_t(n_tokens) * size_t(K) <= size_t(STATIC_META_MAX_ASSIGNMENTS),
             "moe_metadata_static: N*K = %zu exceeds the built-in scratch limit of %d assignments; "
             "use jb200_moe_metadata with caller-provided scratch",
             size_t(n_tokens) * size_t(K), STATIC_META_MAX_ASSIGNMENTS);
  int dev = 0;
  JB_CUDA(cudaGetDevice(&dev));
  JB_REQUIRE(dev >= 0 && dev < 64, "moe_metadata_static: device ordinal %d out of range", dev);
  if (!g_meta_scratch_ptr[dev]) {
    // First call on this device: resolve the array's DEVICE address.  In host code the name
    // g_meta_scratch is only a handle for the runtime, not something a kernel may dereference.
    int* ptr = nullptr;
    JB_CUDA(cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_meta_scratch));
    g_meta_scratch_ptr[dev] = ptr;
  }
  // Every entry the scan and assign kernels read is written by the histogram kernel of the same
  // call first, so nothing left over from an earlier call needs clearing.
  return launch_moe_metadata(topk_idx, n_tokens, K, E, expert_counts, expert_offsets, scatter_map, gather_map,
                             gate_idx_map, g_meta_scratch_ptr[dev], stream);
}

int launch_dispatch_gather(const void* x_bf16, const int* gather_map, int M, int n_tokens, int C, void* dispatched,
                           cudaStream_t stream) {
  JB_REQUIRE(M >= 0 && n_tokens >= 0 && C > 0 && C % 8 == 0, "dispatch_gather: bad shape");
  if (M == 0) return JB200_OK;
  JB_REQUIRE(n_tokens > 0 && x_bf16 && gather_map && dispatched, "dispatch_gather: null pointer");
  JB_REQUIRE(aligned16(x_bf16) && aligned16(dispatched), "dispatch_gather: pointers must be 16-byte aligned");
  launch_dep(dispatch_gather_kernel, (M + 7) / 8, 256, 0, stream, reinterpret_cast<const __nv_bfloat16*>(x_bf16), gather_map, M,
                                                          n_tokens, C, reinterpret_cast<__nv_bfloat16*>(dispatched));
  JB_LAUNCH_CHECK("dispatch_gather_kernel");
  return JB200_OK;
}

int launch_scatter_combine(const void* y_bf16, const float* gates, const int* scatter_map, int n_tokens, int K, int C,
                           void* out, int out_dtype, double* stats, cudaStream_t stream, bool ahead, const int64_t* topk_idx) {
  JB_REQUIRE(n_tokens >= 0 && K >= 1 && K <= 8 && C > 0 && C % 8 == 0, "scatter_combine: bad shape");
  JB_REQUIRE(out_dtype == 0 || out_dtype == 1, "scatter_combine: out_dtype must be 0 (f32) or 1 (bf16)");
  if (n_tokens == 0) return JB200_OK;
  JB_REQUIRE(y_bf16 && gates && scatter_map && out, "scatter_combine: null pointer");
  JB_REQUIRE(aligned16(y_bf16) && aligned16(out), "scatter_combine: pointers must be 16-byte aligned");
  const int blocks = (n_tokens + 7) / 8;
  const int M = n_tokens * K;
  if (K == 2 && C <= 1024 && (reinterpret_cast<uintptr_t>(gates) & 7u) == 0 && (reinterpret_cast<uintptr_t>(scatter_map) & 7u) == 0) {
    const __nv_bfloat16* y = reinterpret_cast<const __nv_bfloat16*>(y_bf16);
    if (out_dtype == 1)
      launch_dep(top2_combine_kernel<__nv_bfloat16>, blocks, 256, 0, stream, y, gates, scatter_map, topk_idx, n_tokens, C, ahead,
                 reinterpret_cast<__nv_bfloat16*>(out), stats);
    else
      launch_dep(top2_combine_kernel<float>, blocks, 256, 0, stream, y, gates, scatter_map, topk_idx, n_tokens, C, ahead,
                 reinterpret_cast<float*>(out), stats);
    JB_LAUNCH_CHECK("top2_combine_kernel");
    return JB200_OK;
  }
  if (out_dtype == 1)
    launch_dep(scatter_combine_kernel<__nv_bfloat16>, blocks, 256, 0, stream,
        reinterpret_cast<const __nv_bfloat16*>(y_bf16), gates, scatter_map, n_tokens, K, M, C,
        reinterpret_cast<__nv_bfloat16*>(out), stats);
  else
    launch_dep(scatter_combine_kernel<float>, blocks, 256, 0, stream, reinterpret_cast<const __nv_bfloat16*>(y_bf16), gates,
                                                              scatter_map, n_tokens, K, M, C,
                                                              reinterpret_cast<float*>(out), stats);
  JB_LAUNCH_CHECK("scatter_combine_kernel");
  return JB200_OK;
}

int launch_moe_finalize(const double* stats, const double* probs_sum, const int* top1_hist, int E, long long n_tokens,
                        long long n_elems, float balance_alpha, float* scalars, cudaStream_t stream) {
  JB_REQUIRE(scalars != nullptr, "moe_finalize: null output");
  JB_REQUIRE(n_tokens > 0 && n_elems > 0, "moe_finalize: empty batch");
  launch_dep(moe_finalize_kernel, 1, 32, 0, stream, stats, probs_sum, top1_hist, E, n_tokens, n_elems, balance_alpha, scalars);
  JB_LAUNCH_CHECK("moe_finalize_kernel");
  return JB200_OK;
}

}  // namespace jb
