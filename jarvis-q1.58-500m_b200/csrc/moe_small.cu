// The glue of a block for few tokens (decode steps of small batches, short prompts), where every launch is latency: two
// kernels in the place of five.
//
//   route_small_kernel  norm2 + top-2 router (jarvis_model.py:25-26, :218-224), a warp per token; up to sixteen tokens
//                       the warp that finishes last also makes the dispatch maps (sparse_model.cu:23-90)
//   tail_step_kernel, tail_scan_kernel  combine of the expert rows, MoE statistics, LSF scan, residual add and the RMSNorm
//                       that follows (sparse_model.cu:117-165, jarvis_model.py:244-250, :281-314, :430-436) in one
//                       thread-block cluster: the decay of the scan depends on the variance of ALL combined rows, and
//                       a cluster barrier does what the boundaries of two or three kernels (6 + 9 us, 6 + 8 + 5 us) did.
// Everything a kernel needs that its predecessor on the stream did not make is fetched before the grid dependency is
// waited for.  Every value is rounded and every sum ordered as in the kernels these stand for (rmsnorm_router_kernel,
// meta_small_kernel, scatter_combine_kernel, lsf_step_norm_kernel, lsf_tma_kernel, lsf_short_kernel, rmsnorm_kernel): the
// results are theirs bit for bit, so that a token's experts do not depend on how many others share its call.
#include <algorithm>

#include "common.cuh"
#include "moe_finalize.cuh"
#include "moe_router.cuh"
#include "row_math.cuh"
#include "launchers.h"

namespace jb {

namespace {

struct RouteParams {
  const float* x;              // [N][C]
  const float* w_norm;
  const float* w_router;       // [E][C]
  __nv_bfloat16* xn;           // [N][C] out
  int64_t* idx;                // [N][2]
  float* gates;                // [N][2]
  double* probs_sum;           // [E] accumulated
  int* hist;                   // [E] accumulated
  int* load;                   // [E] accumulated: assignments, first and second ones; null: not wanted
  int* ticket;                 // zero on entry
  int *counts, *offsets, *scatter, *gather, *gate_idx;   // scatter null: no maps
  float eps;
  int N, C;
};

// One warp per token and CTA: with all weights of the lane's channels in registers before the residual row arrives, the
// chain is load - sum - norm - dot - sums - softmax.
// SORT: up to sixteen tokens the warp that finishes last makes the maps; beyond, the sort is 20 to 60 KB of code and up to 3.6 us, and
// the kernels behind work their rows out from the ids.  Up to 512 tokens it beats the persistent router (300 tokens 1274 -> 1230 us
// a forward, 400 1426 -> 1405, 512 1508 -> 1501, 700 1648 -> 1672: every warp reads all weights).
template <int E, bool SORT>
__global__ void __launch_bounds__(32) route_small_kernel(const RouteParams p) {
  __shared__ int h_acc[E];
  // Before the wait: what comes next reads weights alone ahead of its own (the first expert matrix, which decodes them while the
  // out-projection still runs: 17, 37, 64, 128 tokens 714 -> 683, 749 -> 709, 789 -> 763, 894 -> 877 us a forward, steps of 64
  // sequences 846 -> 826) or nothing (the dispatch).  The kernel ahead has triggered behind its wait, so everything before it is complete.
  if (!SORT) pdl_trigger();
  const int lane = threadIdx.x, tok = blockIdx.x;
  constexpr bool AHEAD = E <= 4;                 // eight experts' weights do not fit the registers: read where used
  float wn[GROUPS][8];
  float4 wr[GROUPS][AHEAD ? E : 1][2];
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    const int c = (i * 32 + lane) * 8;
    if (c < p.C) {
      load8(p.w_norm + c, wn[i]);
#pragma unroll
      for (int e = 0; AHEAD && e < E; ++e) {
        wr[i][e][0] = __ldg(reinterpret_cast<const float4*>(p.w_router + size_t(e) * p.C + c));
        wr[i][e][1] = __ldg(reinterpret_cast<const float4*>(p.w_router + size_t(e) * p.C + c) + 1);
      }
    }
  }
  if (lane < E) h_acc[lane] = 0;
  __syncwarp();
  pdl_wait();
  if (SORT) pdl_trigger();

  float v[GROUPS][8], ss = 0.f;
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    const int c = (i * 32 + lane) * 8;
    if (c < p.C) load8(p.x + size_t(tok) * p.C + c, v[i]);
  }
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    if ((i * 32 + lane) * 8 < p.C) {
#pragma unroll
      for (int j = 0; j < 8; ++j) ss = __fmaf_rn(v[i][j], v[i][j], ss);
    }
  }
  ss = warp_sum(ss);
  const float r = rsqrtf(ss / float(p.C) + p.eps);
  float acc[E];
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = 0.f;
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    const int c = (i * 32 + lane) * 8;
    if (c < p.C) {
      const uint4 pk = norm8(v[i], r, make_float4(wn[i][0], wn[i][1], wn[i][2], wn[i][3]),
                             make_float4(wn[i][4], wn[i][5], wn[i][6], wn[i][7]));
      *reinterpret_cast<uint4*>(p.xn + size_t(tok) * p.C + c) = pk;
      const float xv[8] = {bf16_lo(pk.x), bf16_hi(pk.x), bf16_lo(pk.y), bf16_hi(pk.y),
                           bf16_lo(pk.z), bf16_hi(pk.z), bf16_lo(pk.w), bf16_hi(pk.w)};
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const float4* w = reinterpret_cast<const float4*>(p.w_router + size_t(e) * p.C + c);
        acc[e] = AHEAD ? router_dot(acc[e], xv, wr[i][AHEAD ? e : 0][0], wr[i][AHEAD ? e : 0][1])
                       : router_dot(acc[e], xv, __ldg(w), __ldg(w + 1));
      }
    }
  }
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = warp_sum(acc[e]);
  float pr[E];
#pragma unroll
  for (int e = 0; e < E; ++e) pr[e] = 0.f;
  router_finish<E>(acc, lane, tok, p.idx, p.gates, nullptr, h_acc, pr, p.load);       // pr: the probabilities, in lane 0
  int last = 0;
  if (lane == 0) {
    if (SORT && p.scatter) {                     // before the sums: the fence would wait for them too (256 tokens 1366 -> 1358 us a forward)
      __threadfence();
      last = atomicAdd(p.ticket, 1) == p.N - 1;
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
      atomicAdd(p.probs_sum + e, double(pr[e]));
      if (h_acc[e]) atomicAdd(p.hist + e, 1);
    }
  }
  if (!SORT || !__shfl_sync(0xffffffffu, last, 0)) return;
  __threadfence();
  sort_routes<E, 1>(reinterpret_cast<const long long*>(p.idx), p.N, lane, p.counts, p.offsets, p.scatter, p.gather, p.gate_idx);
}

// ---------------------------------------------------------------------------------------------------------------
struct TailParams {
  const __nv_bfloat16* y;      // [2N][C] expert outputs in dispatch order: the only input the kernel before this one made
  const float* gates;          // [N][2]
  const int* scatter;          // [N][2]
  const int64_t* idx;          // [N][2]
  LsfStats st;                 // stats is not read: the sums are made here
  const float* var_scale;
  float alpha_min, alpha_max;
  const float* h_in;           // [B][C] or null
  float* h_out;                // [B][C], may be h_in
  float* x;                    // [N][C] residual stream
  const float* w_norm;         // [C] or null
  float eps;
  __nv_bfloat16* xn;           // [N][C]
  int B, T, N, C;
  unsigned int* status;
};

constexpr int MAX_CTAS = 16;                           // non-portable cluster size: asked for before use (tail_fits)
constexpr int MAX_WARPS = 16;                          // of a CTA; a warp takes one token (tail_max_tokens: how many come)

// Slots of a token's two expert rows.  Without finite logits (idx -1) both are expert 0's, and a GEMM that takes all rows for every
// expert has made the first of them alone.
__device__ __forceinline__ int2 tail_slots(const TailParams& p, int n) {
  int2 s = *reinterpret_cast<const int2*>(p.scatter + 2 * n);
  if (p.idx[2 * n + 1] < 0) s.y = s.x;
  return s;
}

// The combined row of one token: put(i, 8 values rounded to bf16) for every group; the sums of the unrounded ones over the warp.
template <typename F>
__device__ __forceinline__ Combined combine_row(const TailParams& p, int a, int b, float2 g, int lane, F&& put) {
  a = min(max(a, 0), 2 * p.N - 1);
  b = min(max(b, 0), 2 * p.N - 1);
  uint4 ya[GROUPS], yb[GROUPS];
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    const int c = (i * 32 + lane) * 8;
    if (c < p.C) {
      ya[i] = *reinterpret_cast<const uint4*>(p.y + size_t(a) * p.C + c);
      yb[i] = *reinterpret_cast<const uint4*>(p.y + size_t(b) * p.C + c);
    }
  }
  return combine_values(ya, yb, g, lane, p.C, put);
}

// Exchange of the sums: 16 bytes from every CTA, and whatever rows come with them, counted by an mbarrier of the receiver (a cluster
// barrier waits for all stores of all its threads as well: 0.6 us against 0.3).
struct TailShared {
  alignas(16) double part[MAX_WARPS][2], all[MAX_CTAS][2];
  uint64_t bar;
  uint32_t abort_flag;
};
struct Decay {
  float alpha, mean, var;
  bool got;                    // false: this warp has given up waiting for the other CTAs
};
__device__ __noinline__ bool tail_wait_long(uint32_t bar, volatile uint32_t* abort_flag, unsigned int* status) {
  return mbar_wait(bar, 0u, abort_flag, status, JB200_STATUS_LSF_LOAD);
}
// A CTA may leave when what the others send it has landed.  Behind a cluster barrier (threads that have left count as arrived) all of it is
// on its way.
__device__ __noinline__ void tail_landed(uint32_t bar) {
  for (int i = 0; i < 1000; ++i)
    if (mbar_try_wait_parked(bar, 0u, 20000u)) return;
}
// Ahead of everything else; the CTAs of a cluster have all done it behind the cluster_wait() of tail_decay.
__device__ __forceinline__ void tail_begin(TailShared& s, int n_cta, uint32_t row_bytes) {
  if (n_cta == 1) return;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&s.bar), 1);
    s.abort_flag = 0;
    fence_mbar_init();
    mbar_arrive_expect_tx(smem_u32(&s.bar), uint32_t(n_cta) * 16u + row_bytes);
  }
  __syncwarp();
  cluster_arrive();
}

// Sums of the CTA's tokens (one per warp) -> every CTA of the cluster -> the decay of the call, the same bits in every warp.
// Called by all threads; what `push` sends to other CTAs on their `bar` is there when this returns.
template <typename F>
__device__ __forceinline__ Decay tail_decay(const TailParams& p, Combined c, float var_scale, TailShared& s, int rank, int n_cta, F&& push) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
  if (lane == 0) { s.part[warp][0] = double(c.s1); s.part[warp][1] = double(c.s2); }
  if (n_cta > 1) cluster_wait();               // the other CTAs have started: their shared memory may be written
  push();
  __syncthreads();
  if (warp == 0) {
    double a = lane < n_warps ? s.part[lane][0] : 0.0, b = lane < n_warps ? s.part[lane][1] : 0.0;
    for (int o = n_warps > 8 ? 8 : n_warps > 4 ? 4 : n_warps > 2 ? 2 : n_warps >> 1; o > 0; o >>= 1) {        // lanes from n_warps on are zeros
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    a = __shfl_sync(0xffffffffu, a, 0);
    b = __shfl_sync(0xffffffffu, b, 0);
    if (n_cta == 1) {
      if (lane == 0) { s.all[0][0] = a; s.all[0][1] = b; }
    } else if (lane < n_cta) {
      st_async16(cluster_map(smem_u32(&s.all[rank][0]), uint32_t(lane)), cluster_map(smem_u32(&s.bar), uint32_t(lane)),
                 make_uint4(uint32_t(__double2loint(a)), uint32_t(__double2hiint(a)), uint32_t(__double2loint(b)), uint32_t(__double2hiint(b))));
    }
  }
  bool got = true;
  if (n_cta == 1) __syncthreads();
  else if (!mbar_try_wait(smem_u32(&s.bar), 0u)) got = tail_wait_long(smem_u32(&s.bar), &s.abort_flag, p.status);
  got = __all_sync(0xffffffffu, got);
  double sum = lane < n_cta ? s.all[lane][0] : 0.0, sq = lane < n_cta ? s.all[lane][1] : 0.0;
  for (int o = n_cta > 8 ? 8 : 4; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    sq += __shfl_xor_sync(0xffffffffu, sq, o);
  }
  const float2 mv = moe_act_mean_var(__shfl_sync(0xffffffffu, sum, 0), __shfl_sync(0xffffffffu, sq, 0), p.st.n_el, p.st.inv_el, p.st.inv_el1);
  return {lsf_alpha_from_var(p.alpha_min, p.alpha_max, var_scale, mv.y), mv.x, mv.y, got};
}
// The norm's weight, on its way while the kernel ahead runs (what a thread has read into L1 by then is gone behind the grid dependency: read
// from global memory at the end, the weight took 1.9 us).
__device__ __forceinline__ void copy_norm(const TailParams& p, float* s_norm) {
  if (!p.w_norm) return;
  for (int i = threadIdx.x; i < p.C / 4; i += blockDim.x) copy_async_16(smem_u32(s_norm + 4 * i), p.w_norm + 4 * i);
}
// The layer's scalars, by one thread of the cluster that has little else to do.
__device__ __forceinline__ void tail_scalars(const TailParams& p, float l_bal, float mu, Decay d) {
  p.st.scalars[0] = l_bal;
  p.st.scalars[1] = d.mean;
  p.st.scalars[2] = d.var;
  if (p.st.reflect) *p.st.reflect = reflect_penalty(p.st.lam, p.st.tau, mu, d.mean, d.var);
}

// One token per sequence (decode): a warp per token, its row in registers throughout.
__global__ void __launch_bounds__(32 * MAX_WARPS) tail_step_kernel(const TailParams p, const int n_cta) {
  __shared__ TailShared sh;
  __shared__ __align__(16) float s_norm[GROUPS * 256];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = n_cta > 1 ? int(cluster_rank()) : 0;
  const int n = rank + warp * n_cta;
  const bool on = n < p.N;
  tail_begin(sh, n_cta, 0u);
  copy_norm(p, s_norm);
  const float var_scale = __ldg(p.var_scale);
  float x[GROUPS][8], h[GROUPS][8];
  int2 sl = make_int2(0, 0);
  float2 g = make_float2(0.f, 0.f);
  if (on) {
    sl = tail_slots(p, n);
    g = *reinterpret_cast<const float2*>(p.gates + 2 * n);
#pragma unroll
    for (int i = 0; i < GROUPS; ++i) {
      const int c = (i * 32 + lane) * 8;
      if (c < p.C) {
        load8(p.x + size_t(n) * p.C + c, x[i]);
        if (p.h_in) {
          load8(p.h_in + size_t(n) * p.C + c, h[i]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) h[i][j] = 0.f;
        }
      }
    }
  }
  float l_bal = 0.f, mu = 0.f;
  if (rank == 0 && tid == int(blockDim.x) - 1) {
    l_bal = moe_l_balance(p.st.probs_sum, p.st.top1_hist, p.st.E, p.st.inv_tok, p.st.balance_alpha);
    if (p.st.reflect) mu = __ldg(p.st.mu);
  }
  __syncwarp();
  pdl_wait();
  pdl_trigger();

  copy_async_wait();             // visible to all behind the first barrier of tail_decay
  uint4 m[GROUPS];
  Combined c = {0.f, 0.f};
  if (on) c = combine_row(p, sl.x, sl.y, g, lane, [&](int i, uint4 v) { m[i] = v; });
  const Decay d = tail_decay(p, c, var_scale, sh, rank, n_cta, [] {});
  if (!d.got) {                // 2 s late: nobody sends anything behind this
    cluster_arrive();
    cluster_wait();
    tail_landed(smem_u32(&sh.bar));
  }
  const float alpha = d.alpha;
  if (rank == 0 && tid == int(blockDim.x) - 1) tail_scalars(p, l_bal, mu, d);
  if (!on) return;
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    const int ch = (i * 32 + lane) * 8;
    if (ch < p.C) {
      const uint32_t mw[4] = {m[i].x, m[i].y, m[i].z, m[i].w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        h[i][j] = lsf_step(alpha, h[i][j], (j & 1) ? bf16_hi(mw[j >> 1]) : bf16_lo(mw[j >> 1]));
        x[i][j] = x[i][j] + h[i][j];
        ss = __fmaf_rn(x[i][j], x[i][j], ss);
      }
      store8(p.h_out + size_t(n) * p.C + ch, h[i]);
      store8(p.x + size_t(n) * p.C + ch, x[i]);
    }
  }
  if (!p.w_norm) return;
  ss = warp_sum(ss);
  const float r = rsqrtf(ss / float(p.C) + p.eps);
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    const int ch = (i * 32 + lane) * 8;
    if (ch < p.C)
      *reinterpret_cast<uint4*>(p.xn + size_t(n) * p.C + ch) =
          norm8(x[i], r, *reinterpret_cast<const float4*>(s_norm + ch), *reinterpret_cast<const float4*>(s_norm + ch + 4));
  }
}

// Several tokens per sequence.  Rows are combined and normalised by the CTA that owns the token (token n: CTA n % n_cta, a
// warp each), the scan runs where all tokens of a channel are (CTA k: channels [64 k, 64 k + 64)); the rows change
// hands through distributed shared memory.  ms [N][64] bf16: combined rows of the CTA's channels; xs [N][64] f32: their residual rows,
// copied while the kernel ahead runs; hs [B][64]: their membranes; xr [N / n_cta][C] f32: updated residual rows of the CTA's tokens; ends
// [B * runs][64]: what a run of tokens leaves from a zero carry.
// Bound by latency: copies, three exchanges and one chain over a run; a run is worked on by up to four warps, each going along the
// chain but storing four tokens of sixteen.  A launch fetches
// its code anew (34 KB; unrolled over a run, with one for either kind of sequence, 63): the scan took 2.8 us of the 7.2 at 37 tokens, the f64
// divisions 1.0.  24 layers and head 17, 37, 64, 128, 160 tokens 761 -> 713, 775 -> 746, 814 -> 784, 902 -> 891, 1006 -> 996 us.
constexpr int SCAN_CH = 64, RUN = 16;          // channels per CTA, two per lane; tokens per run (lsf_tma_kernel's warp runs)

__global__ void __launch_bounds__(32 * MAX_WARPS) tail_scan_kernel(const TailParams p, const int n_cta) {
  extern __shared__ __align__(16) uint8_t tail_smem[];
  __shared__ TailShared sh;
  __shared__ __align__(16) float s_norm[GROUPS * 256];
  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31, n_warps = blockDim.x >> 5;
  const int N = p.N, B = p.B, T = p.T, C = p.C;
  const int rank = int(cluster_rank());
  // runs of 16 tokens from a zero carry, the carries along the runs, then every token's value, with the roundings of
  // lsf_tma_kernel (T > 8) or lsf_short_kernel
  const int n_runs = T > 8 ? (T + RUN - 1) / RUN : 1, run_len = T > 8 ? RUN : T, items = B * n_runs;
  const int split = T <= 8 ? 1 : 4 * items <= n_warps ? 4 : 2 * items <= n_warps ? 2 : 1;        // warps of a run
  uint8_t* ms = tail_smem;                                                     // [N][128 bytes]
  float* xs = reinterpret_cast<float*>(tail_smem + size_t(N) * SCAN_CH * 2);
  float* hs = xs + size_t(N) * SCAN_CH;                                        // h_out may be h_in
  float* xr = hs + size_t(B) * SCAN_CH;
  float* ends = xr + size_t((N + n_cta - 1) / n_cta) * C;
  const int own = rank + warp * n_cta;                                         // this warp's token
  const bool on = own < N;
  tail_begin(sh, n_cta, uint32_t(N) * (SCAN_CH * 2));
  copy_norm(p, s_norm);
  const float var_scale = __ldg(p.var_scale);
  int2 sl = make_int2(0, 0);
  float2 g = make_float2(0.f, 0.f);
  if (on) {
    sl = tail_slots(p, own);
    g = *reinterpret_cast<const float2*>(p.gates + 2 * own);
  }
  const size_t ch = size_t(rank) * SCAN_CH + lane * 2;
  for (int i = tid; i < N * (SCAN_CH / 4); i += blockDim.x)
    copy_async_16(smem_u32(xs) + uint32_t(i) * 16u, p.x + size_t(i / (SCAN_CH / 4)) * C + rank * SCAN_CH + i % (SCAN_CH / 4) * 4);
  for (int i = tid; i < B * SCAN_CH / 4; i += blockDim.x) {
    const int b = i / (SCAN_CH / 4), q = i % (SCAN_CH / 4);
    reinterpret_cast<float4*>(hs)[i] =
        p.h_in ? *(reinterpret_cast<const float4*>(p.h_in + size_t(b) * C + rank * SCAN_CH) + q) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float l_bal = 0.f, mu = 0.f;
  if (rank == 0 && tid == int(blockDim.x) - 1) {
    l_bal = moe_l_balance(p.st.probs_sum, p.st.top1_hist, p.st.E, p.st.inv_tok, p.st.balance_alpha);
    if (p.st.reflect) mu = __ldg(p.st.mu);
  }
  __syncwarp();
  pdl_wait();
  pdl_trigger();

  uint4 m[GROUPS];
  Combined cm = {0.f, 0.f};
  if (on) cm = combine_row(p, sl.x, sl.y, g, lane, [&](int i, uint4 v) { m[i] = v; });
  const Decay d = tail_decay(p, cm, var_scale, sh, rank, n_cta, [&] {
    if (on) {
#pragma unroll
      for (int i = 0; i < GROUPS; ++i) {
        const int c = (i * 32 + lane) * 8;
        const uint32_t to = uint32_t(c / SCAN_CH);
        if (c < C) st_async16(cluster_map(smem_u32(ms) + uint32_t(own) * (SCAN_CH * 2) + uint32_t(c % SCAN_CH) * 2u, to), cluster_map(smem_u32(&sh.bar), to), m[i]);
      }
    }
  });
  if (rank == 0 && tid == int(blockDim.x) - 1) tail_scalars(p, l_bal, mu, d);

  const float alpha = d.alpha, one_m = 1.0f - alpha;
  float whole = alpha;                                       // alpha to the power of a run's length
#pragma unroll
  for (int i = 1; i < RUN; ++i) whole *= alpha;
  auto m_at = [&](int n) { return *reinterpret_cast<const uint32_t*>(ms + size_t(n) * (SCAN_CH * 2) + lane * 4); };
  auto along = [&](float2& v, uint32_t m) {                  // one token further
    v.x = __fmaf_rn(alpha, v.x, __fmul_rn(one_m, bf16_lo(m)));
    v.y = __fmaf_rn(alpha, v.y, __fmul_rn(one_m, bf16_hi(m)));
  };
  if (n_runs > 1) {
#pragma unroll 1
    for (int w = warp; w < items; w += n_warps) {
      const int b = w / n_runs, run = w - b * n_runs;
      if (run == n_runs - 1) continue;                       // nobody's carry
      float2 e = make_float2(0.f, 0.f);
      uint32_t m[RUN];
#pragma unroll
      for (int j = 0; j < RUN; ++j) m[j] = m_at(b * T + run * RUN + j);
#pragma unroll
      for (int j = 0; j < RUN; ++j) along(e, m[j]);
      *reinterpret_cast<float2*>(ends + w * SCAN_CH + lane * 2) = e;
    }
  }
  copy_async_wait();
  __syncthreads();
#pragma unroll 1
  for (int w = warp; w < items * split; w += n_warps) {      // (sequence, run, part of it)
    const int item = w / split, part = w - item * split, b = item / n_runs, run = item - b * n_runs;
    if (part * (RUN / split) >= T - run * RUN) continue;
    float2 h = *reinterpret_cast<const float2*>(hs + b * SCAN_CH + lane * 2);
    for (int q = 0; q < run; ++q) {                          // the carry into this run
      const float2 e = *reinterpret_cast<const float2*>(ends + (b * n_runs + q) * SCAN_CH + lane * 2);
      h.x = __fmaf_rn(whole, h.x, e.x);
      h.y = __fmaf_rn(whole, h.y, e.y);
    }
    const int left = T - run * RUN, first = b * T + run * RUN, last = min(min(run_len, left), (part + 1) * (RUN / split));
    float2 loc = make_float2(0.f, 0.f), hv = h;
    float pw = alpha;                                        // alpha to the power of the tokens since the carry
#pragma unroll 1
    for (int j0 = 0; j0 < last; j0 += 4) {
      uint32_t m[4];
      float2 x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int n = min(first + j0 + k, N - 1);
        m[k] = m_at(n);
        x[k] = *reinterpret_cast<const float2*>(xs + size_t(n) * SCAN_CH + lane * 2);
      }
      const bool mine = j0 >= part * (RUN / split);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (T > 8) {
          along(loc, m[k]);
          hv.x = __fmaf_rn(pw, h.x, loc.x);
          hv.y = __fmaf_rn(pw, h.y, loc.y);
          pw *= alpha;
        } else {
          const float2 was = hv;
          hv.x = lsf_step(alpha, was.x, bf16_lo(m[k]));
          hv.y = lsf_step(alpha, was.y, bf16_hi(m[k]));
        }
        if (mine && j0 + k < last) {
          const int n = first + j0 + k;
          x[k].x = x[k].x + hv.x;
          x[k].y = x[k].y + hv.y;
          *reinterpret_cast<float2*>(p.x + size_t(n) * C + ch) = x[k];
          cluster_st_64(cluster_map(smem_u32(xr) + (uint32_t(n / n_cta) * uint32_t(C) + uint32_t(ch)) * 4u, uint32_t(n % n_cta)), x[k]);
          if (run * RUN + j0 + k == T - 1) *reinterpret_cast<float2*>(p.h_out + size_t(b) * C + ch) = hv;
        }
      }
    }
  }
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  if (!d.got) tail_landed(smem_u32(&sh.bar));
  if (!p.w_norm || !on) return;

  // ---- the norm of the warp's token ----
  const float* row = xr + size_t(warp) * C;
  float v[GROUPS][8], ss = 0.f;
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    const int c = (i * 32 + lane) * 8;
    if (c < C) {
      load8(row + c, v[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss = __fmaf_rn(v[i][j], v[i][j], ss);
    }
  }
  ss = warp_sum(ss);
  const float r = rsqrtf(ss / float(C) + p.eps);
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    const int c = (i * 32 + lane) * 8;
    if (c < C) *reinterpret_cast<uint4*>(p.xn + size_t(own) * C + c) = norm8(v[i], r, *reinterpret_cast<const float4*>(s_norm + c), *reinterpret_cast<const float4*>(s_norm + c + 4));
  }
}

// [N][64] bf16 and f32, [B][64] f32, [rows][C] f32, [items][64] f32; B and items are at most N / 2 and N / 16 + B.
inline size_t tail_smem_bytes(int N, int B, int rows, int C, int items) {
  return size_t(N) * SCAN_CH * 6 + (size_t(B) * SCAN_CH + size_t(rows) * C + size_t(items) * SCAN_CH) * sizeof(float);
}
constexpr size_t TAIL_SMEM = 200 * 1024;

// Whether clusters of n_cta CTAs can run here, with the shared memory of the largest call; also sets the kernel up for them.  Eight is the
// portable limit; each size beyond it is asked for by itself, since a launch that is refused would come in the middle of a forward.
bool tail_fits(int n_cta) {
  constexpr int MAX_DEVICES = 64, PORTABLE = 8;
  static std::atomic<int> known[MAX_DEVICES][MAX_CTAS + 1];            // 0 not asked yet, 1 yes, -1 no
  if (n_cta <= PORTABLE) return true;
  int dev = 0;
  if (n_cta > MAX_CTAS || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return false;
  int k = known[dev][n_cta].load(std::memory_order_acquire);
  if (k == 0) {
    int n = 0;
    const void* scan = reinterpret_cast<const void*>(tail_scan_kernel);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cfg.gridDim = n_cta; cfg.blockDim = 32 * MAX_WARPS; cfg.dynamicSmemBytes = TAIL_SMEM; cfg.attrs = at; cfg.numAttrs = 1;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = unsigned(n_cta); at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    const bool ok = cudaFuncSetAttribute(reinterpret_cast<const void*>(tail_step_kernel), cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaFuncSetAttribute(scan, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaFuncSetAttribute(scan, cudaFuncAttributeMaxDynamicSharedMemorySize, int(TAIL_SMEM)) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&n, tail_scan_kernel, &cfg) == cudaSuccess && n >= 1;
    if (!ok) (void)cudaGetLastError();
    k = ok ? 1 : -1;
    known[dev][n_cta].store(k, std::memory_order_release);
  }
  return k > 0;
}

// Embedding rows into the f32 residual stream (jarvis_model.py:498) and, while they are in registers, norm1 of the first
// block; clears the chain's accumulators on the way.  One warp per token, C <= 1024.  Without ids the rows are there already.
template <bool IDS>
__global__ void __launch_bounds__(256)
embed_norm_kernel(const int64_t* __restrict__ ids, const float* __restrict__ table, int vocab, const float* __restrict__ w_norm,
                  float eps, float* __restrict__ x, __nv_bfloat16* __restrict__ xn, int n_rows, int C, uint32_t* __restrict__ zero,
                  int n_zero) {
  pdl_wait();
  pdl_trigger();
  const int gtid = blockIdx.x * 256 + threadIdx.x;
  for (int i = gtid; i < n_zero; i += gridDim.x * 256) zero[i] = 0u;
  const int row = gtid >> 5, lane = threadIdx.x & 31;
  if (row >= n_rows) return;
  const float* src = x + size_t(row) * C;
  if constexpr (IDS) {
    long long id = ids[row];
    id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);          // clamp instead of faulting on a bad id
    src = table + size_t(id) * C;
  }
  float v[GROUPS][8], ss = 0.f;
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    const int c = (i * 32 + lane) * 8;
    if (c < C) load8(src + c, v[i]);
  }
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    const int c = (i * 32 + lane) * 8;
    if (c < C) {
      if (IDS) store8(x + size_t(row) * C + c, v[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss = __fmaf_rn(v[i][j], v[i][j], ss);
    }
  }
  ss = warp_sum(ss);
  const float r = rsqrtf(ss / float(C) + eps);
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    const int c = (i * 32 + lane) * 8;
    if (c < C)
      *reinterpret_cast<uint4*>(xn + size_t(row) * C + c) =
          norm8(v[i], r, __ldg(reinterpret_cast<const float4*>(w_norm + c)), __ldg(reinterpret_cast<const float4*>(w_norm + c) + 1));
  }
}

}  // namespace

int launch_embed_norm(const int64_t* ids, const float* table, int vocab, const float* w_norm, float eps, float* x, void* xn_bf16,
                      int n_rows, int C, void* zero, size_t zero_bytes, cudaStream_t stream) {
  JB_REQUIRE((!ids || (table && vocab > 0)) && w_norm && x && xn_bf16 && n_rows > 0, "embed_norm: null pointer or empty");
  JB_REQUIRE(C % 8 == 0 && C <= 1024 && zero_bytes % 4 == 0, "embed_norm: row length %d", C);
  JB_REQUIRE(aligned16(table) && aligned16(x) && aligned16(xn_bf16) && aligned16(w_norm), "embed_norm: pointers must be 16-byte aligned");
  launch_dep(ids ? embed_norm_kernel<true> : embed_norm_kernel<false>, (n_rows + 7) / 8, 256, 0, stream, ids, table, vocab, w_norm, eps, x,
             reinterpret_cast<__nv_bfloat16*>(xn_bf16), n_rows, C, reinterpret_cast<uint32_t*>(zero), int(zero_bytes / 4));
  JB_LAUNCH_CHECK("embed_norm_kernel");
  return JB200_OK;
}

int launch_route_small(const float* x, const float* w_norm, float eps, void* xn_bf16, const float* w_router, int N, int C, int E,
                       int64_t* idx, float* gates, double* probs_sum, int* hist, int* load, int* ticket, int* counts, int* offsets,
                       int* scatter, int* gather, int* gate_idx, cudaStream_t stream) {
  JB_REQUIRE(N >= 1 && N <= ROUTE_SMALL_MAX && C % 8 == 0 && C <= 1024 && (E == 4 || E == 8), "route_small: bad shape (N=%d, C=%d, E=%d)", N, C, E);
  RouteParams p;
  p.x = x; p.w_norm = w_norm; p.w_router = w_router; p.xn = reinterpret_cast<__nv_bfloat16*>(xn_bf16);
  p.idx = idx; p.gates = gates; p.probs_sum = probs_sum; p.hist = hist; p.load = load; p.ticket = ticket;
  p.counts = counts; p.offsets = offsets; p.scatter = scatter; p.gather = gather; p.gate_idx = gate_idx;
  p.eps = eps; p.N = N; p.C = C;
  JB_REQUIRE(!scatter || N <= ROUTE_SORT_MAX, "route_small: no maps of %d tokens", N);
  static_assert(ROUTE_SORT_MAX == 16, "one round of the sort");
  auto kernel = scatter ? (E == 4 ? route_small_kernel<4, true> : route_small_kernel<8, true>)
                        : (E == 4 ? route_small_kernel<4, false> : route_small_kernel<8, false>);
  launch_dep(kernel, N, 32, 0, stream, p);
  JB_LAUNCH_CHECK("route_small_kernel");
  return JB200_OK;
}

int launch_tail(const void* y_bf16, const float* gates, const int* scatter, const int64_t* idx, const LsfStats& st,
                const float* var_scale, float alpha_min, float alpha_max, const float* h_in, float* h_out, float* x,
                const float* w_norm, float eps, void* xn_bf16, int B, int T, int C, cudaStream_t stream) {
  const int N = B * T;
  JB_REQUIRE(N >= 1 && N <= tail_max_tokens(C, T) && C % 128 == 0 && C <= 1024, "tail: bad shape (B=%d, T=%d, C=%d)", B, T, C);
  TailParams p;
  p.y = reinterpret_cast<const __nv_bfloat16*>(y_bf16); p.gates = gates; p.scatter = scatter; p.idx = idx; p.st = st.counted();
  p.var_scale = var_scale; p.alpha_min = alpha_min; p.alpha_max = alpha_max;
  p.h_in = h_in; p.h_out = h_out; p.x = x; p.w_norm = w_norm; p.eps = eps;
  p.xn = reinterpret_cast<__nv_bfloat16*>(xn_bf16);
  p.B = B; p.T = T; p.N = N; p.C = C;
  p.status = device_status_ptr();
  if (!p.status) return JB200_ERR_CUDA;
  if (T == 1) {
    // a lone CTA while its SM can take the rows (4 KB in, 10 KB out each), else sixteen (steps of 64 and 128 sequences, 24 layers
    // and head, in eight 876 and 1127 us, so 848 and 1065), or eight where a cluster cannot have more
    const int n_cta = N <= 4 ? 1 : tail_fits(MAX_CTAS) ? MAX_CTAS : 8;
    const int warps = (N + n_cta - 1) / n_cta;
    if (n_cta == 1) launch_dep(tail_step_kernel, 1, 32 * warps, 0, stream, p, 1);
    else launch_dep_cluster(tail_step_kernel, n_cta, 32 * warps, 0, n_cta, stream, p, n_cta);
    JB_LAUNCH_CHECK("tail_step_kernel");
    return JB200_OK;
  }
  const int n_cta = C / SCAN_CH, rows = (N + n_cta - 1) / n_cta;
  const int items = B * (T > 8 ? (T + RUN - 1) / RUN : 1), warps = std::max(rows, std::min(T > 8 ? 4 * items : items, MAX_WARPS));
  const size_t smem = tail_smem_bytes(N, B, rows, C, items);
  JB_MAX_SMEM(tail_scan_kernel, TAIL_SMEM);
  launch_dep_cluster(tail_scan_kernel, n_cta, 32 * warps, smem, n_cta, stream, p, n_cta);
  JB_LAUNCH_CHECK("tail_scan_kernel");
  return JB200_OK;
}

int tail_max_tokens(int C, int T) {
  // steps: 129 to 256 of them, nine to sixteen a CTA, lose against combine and lsf_step_norm (140 1095 -> 1109 us a step, 192 1334 -> 1376,
  // 256 1527 -> 1605); prompts against combine, scan and norm beyond 192 tokens (200 1158 -> 1139, 4 x 60 1118 -> 1136, 256 1186 -> 1203)
  if (T == 1) return 8 * MAX_WARPS;
  return tail_fits(C / SCAN_CH) ? 12 * (C / SCAN_CH) : 0;
}

}  // namespace jb
