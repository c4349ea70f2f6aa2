// Liquid State Fusion decay scan:  h_t = a_t * h_{t-1} + (1 - a_t) * m_t  per (batch, channel).
//
// Two flavours behind one kernel:
//   * model semantics (LiquidStateFusion.forward, jarvis_engine/jarvis_model.py:281-314): ONE scalar
//     decay per call, alpha = alpha_min + (alpha_max - alpha_min) * sigmoid(-var_scale * act_var),
//     read from device memory so the stream never waits for the host.  The reference evaluates it as
//     a dense T x T decay-matrix product (2*T^2*C flop per sequence); here it is a single streaming
//     pass: 2 bytes read + (optionally) the fused residual update per element.
//   * extension semantics (LiquidStateFusionFunction.forward, liquid_fusion_cuda/liquid_state_fusion.py
//     :49-70; kernel L9 liquid_state_fusion_cuda.cu:412-453): a per-element decay tensor (B, T, D).
//
// Parallel in T inside a CTA: each of the 8 warps scans a run of TPW consecutive tokens with a zero
// carry-in, publishes (product of decays, end value) in shared memory, the carries are combined in
// warp order (the recurrence is an associative affine map), and every thread fixes its values up
// with  h_t = local_t + P_t * carry_in.  A CTA owns 64 channels of one sequence and walks T tile by
// tile.  When B*D/64 CTAs cannot fill the GPU, T is also cut into segments.  A first launch (ENDS_ONLY)
// then computes, with ONE CTA PER TILE of the non-final segments (all tiles in parallel, nothing
// sequential), each tile's end value (and decay product) from a zero carry, reading m once more (it was
// just written by the MoE combine and is normally still in L2); the main launch folds the ends of all
// earlier tiles into its carry-in, which is exact because the recurrence is an affine map.
//
// The two forms the model and the scan sweep run (one scalar decay, bf16 input, and either the fused f32
// residual update or a bf16 output) take lsf_tma_kernel: the same scan, but the [128 tokens x 64 channels] tiles
// travel by TMA (cp.async.bulk.tensor) through a ring of shared-memory stages - loads complete on mbarriers
// (bounded waits), results are written into the tile in place and leave by a TMA store - so the bytes in flight
// no longer depend on how many registers a thread can spare for outstanding loads.
#include <type_traits>

#include "common.cuh"
#include "gemm_shared.cuh"
#include "moe_finalize.cuh"
#include "launchers.h"

namespace jb {

namespace {

constexpr int LSF_WARPS = 8;
constexpr int LSF_THREADS = LSF_WARPS * 32;
constexpr int LSF_CH = 64;  // channels per CTA (2 per lane)

struct LsfParams {
  const void* m;           // [B][T][D]  TM
  const void* alpha_t;     // [B][T][D]  TM   (tensor mode)
  const float* alpha_s;    // scalar decay on the device, or null
  const float* act_var;    // scalar on the device (used when alpha_s is null)
  const float* var_scale;  // scalar on the device
  float alpha_min, alpha_max;
  const float* h0;         // [B][D] f32 or null
  float* resid;            // [B][T][D] f32 in/out or null:  resid += h
  void* out;               // [B][T][D] TOut or null
  float* h_last;           // [B][D] f32 or null
  int B, T, D;
  int seg_len, nseg;       // tokens per segment (multiple of the tile), number of segments (grid.z)
  int n_pre_tiles;         // tiles in the non-final segments = (nseg - 1) * seg_len / tile
  float* seg_end;          // [B][n_pre_tiles][D] end value of each of those tiles from a zero carry
  float* seg_prod;         // [B][n_pre_tiles][D] product of its decays (tensor mode)
};

// Kernels get no more than they use: what these two add, among the parameters of a kernel that does not read it, changed
// its schedule for the worse (per-element decays 32 x 2048: 268 us without, 281 to 304 with; the ends of 8 x 8192: 66, 81).
struct LsfScalarParams : LsfParams {      // one decay per call
  __nv_bfloat16* last16;   // [B][D] or null: the last state in bf16 (h_last is null then)
};
struct LsfChainParams : LsfScalarParams {
  LsfStats st;             // st.stats != null: act_var comes from the MoE layer's accumulators
};
template <bool SCALAR, bool STATS>
using LsfArgs = std::conditional_t<STATS, LsfChainParams, std::conditional_t<SCALAR, LsfScalarParams, LsfParams>>;

template <typename Args>
__device__ __forceinline__ void store_last(const Args& p, size_t at, float2 h) {
  if (p.h_last) *reinterpret_cast<float2*>(p.h_last + at) = h;
  if constexpr (std::is_base_of_v<LsfScalarParams, Args>)
    if (p.last16) *reinterpret_cast<uint32_t*>(p.last16 + at) = pack_bf16x2(h.x, h.y);
}

__device__ __forceinline__ float2 stats_mean_var(const LsfStats& st) {
  return moe_act_mean_var(st.stats[0], st.stats[1], st.n_el, st.inv_el, st.inv_el1);
}

// The scalar decay of a call (model semantics).  With st.stats the variance of the MoE output is derived here, as
// moe_finalize_kernel would have, instead of in a launch of its own between the combine and the scan.
template <typename Args>
__device__ __forceinline__ float lsf_decay(const Args& p) {
  if (p.alpha_s) return __ldg(p.alpha_s);
  float var;
  if constexpr (std::is_same_v<Args, LsfChainParams>) var = p.st.stats ? stats_mean_var(p.st).y : __ldg(p.act_var);
  else var = __ldg(p.act_var);
  return lsf_alpha_from_var(p.alpha_min, p.alpha_max, __ldg(p.var_scale), var);
}
// One thread of the whole grid leaves the MoE layer's scalars: moe_finalize_scalars, quotients from reciprocals (its CTA's others wait for
// it: with divisions here and in the decay 24 layers and head of 256, 512 and 900 tokens took 1137, 1504 and 1829 us, so 1103, 1472 and 1803).
__device__ __forceinline__ void moe_leave_scalars(const LsfStats& st) {
  const float2 mv = stats_mean_var(st);
  if (st.probs_sum && st.top1_hist) {
    double acc = 0.0;
#pragma unroll 1
    for (int e = 0; e < st.E; ++e) acc += div_by(double(st.top1_hist[e]), st.n_tok, st.inv_tok) * div_by(st.probs_sum[e], st.n_tok, st.inv_tok);
    st.scalars[0] = float(double(st.balance_alpha) * double(st.E) * acc);
  }
  st.scalars[1] = mv.x;
  st.scalars[2] = mv.y;
  if (st.reflect) *st.reflect = reflect_penalty(st.lam, st.tau, __ldg(st.mu), mv.x, mv.y);
}
__device__ __forceinline__ void lsf_leave_scalars(const LsfStats& st) {
  if (st.stats && (blockIdx.x | blockIdx.y | blockIdx.z | threadIdx.x) == 0) moe_leave_scalars(st);
}

template <typename T>
__device__ __forceinline__ float2 ld2(const T* p);
template <>
__device__ __forceinline__ float2 ld2<float>(const float* p) { return __ldg(reinterpret_cast<const float2*>(p)); }
template <>
__device__ __forceinline__ float2 ld2<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(p));
  return make_float2(bf16_lo(w), bf16_hi(w));
}
template <typename T>
__device__ __forceinline__ void st2(T* p, float a, float b);
template <>
__device__ __forceinline__ void st2<float>(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
template <>
__device__ __forceinline__ void st2<__nv_bfloat16>(__nv_bfloat16* p, float a, float b) {
  *reinterpret_cast<uint32_t*>(p) = pack_bf16x2(a, b);
}

template <bool TENSOR_ALPHA, typename TM, typename TOut, int TPW, bool ENDS_ONLY, bool STATS>
__global__ void __launch_bounds__(LSF_THREADS, TENSOR_ALPHA ? 1 : 2) lsf_scan_kernel(const LsfArgs<!TENSOR_ALPHA && !ENDS_ONLY, STATS> p) {
  pdl_wait();
  pdl_trigger();
  __shared__ float2 s_end[2][LSF_WARPS][32];   // end value of each warp's run
  __shared__ float2 s_prod[2][LSF_WARPS][32];  // product of decays over the run (tensor mode)
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.y;
  const int ch = blockIdx.x * LSF_CH + lane * 2;
  const bool ch_ok = ch < p.D;
  const size_t seq_base = size_t(b) * p.T * p.D + ch;
  const TM* m = reinterpret_cast<const TM*>(p.m);
  const TM* at = reinterpret_cast<const TM*>(p.alpha_t);
  TOut* out = reinterpret_cast<TOut*>(p.out);

  float alpha = 0.f, pw[TPW];  // scalar mode: pw[i] = alpha^(i+1)
  if constexpr (!TENSOR_ALPHA) {
    alpha = lsf_decay(p);
    float a = alpha;
#pragma unroll
    for (int i = 0; i < TPW; ++i) { pw[i] = a; a *= alpha; }
  }
  constexpr int TILE = LSF_WARPS * TPW;
  const int seg = blockIdx.z;                                    // ENDS_ONLY: the tile's index instead
  const int t_begin = ENDS_ONLY ? seg * TILE : seg * p.seg_len;
  const int t_end = ENDS_ONLY ? t_begin + TILE : min(p.T, t_begin + p.seg_len);
  float2 carry = make_float2(0.f, 0.f);
  float2 pcarry = make_float2(1.f, 1.f);   // running decay product of the segment (ENDS_ONLY, tensor mode)
  if (!ENDS_ONLY) {
    if (p.h0 && ch_ok) carry = __ldg(reinterpret_cast<const float2*>(p.h0 + size_t(b) * p.D + ch));
    if (seg > 0 && ch_ok) {
      const float a_seg = TENSOR_ALPHA ? 0.f : expf(float(TILE) * logf(alpha));   // decay over one tile
      const size_t e0 = (size_t(b) * p.n_pre_tiles) * p.D + ch;
      const int n_before = seg * (p.seg_len / TILE);
      for (int s2 = 0; s2 < n_before; ++s2) {
        const float2 e = __ldg(reinterpret_cast<const float2*>(p.seg_end + e0 + size_t(s2) * p.D));
        if (TENSOR_ALPHA) {
          const float2 q = __ldg(reinterpret_cast<const float2*>(p.seg_prod + e0 + size_t(s2) * p.D));
          carry.x = q.x * carry.x + e.x;
          carry.y = q.y * carry.y + e.y;
        } else {
          carry.x = a_seg * carry.x + e.x;
          carry.y = a_seg * carry.y + e.y;
        }
      }
    }
  }

  int buf = 0;
  for (int tile0 = t_begin; tile0 < t_end; tile0 += LSF_WARPS * TPW, buf ^= 1) {
    const int t0 = tile0 + warp * TPW;
    float2 loc[TPW];
    float2 prod[TENSOR_ALPHA ? TPW : 1];
    float2 mv[TPW], av[TENSOR_ALPHA ? TPW : 1];
#pragma unroll
    for (int i = 0; i < TPW; ++i) {
      const bool ok = ch_ok && (t0 + i) < p.T;
      mv[i] = ok ? ld2<TM>(m + seq_base + size_t(t0 + i) * p.D) : make_float2(0.f, 0.f);
      if (TENSOR_ALPHA) av[i] = ok ? ld2<TM>(at + seq_base + size_t(t0 + i) * p.D) : make_float2(1.f, 1.f);
    }
    // the residual values do not depend on the scan: their loads go out together with those of m, so
    // both streams are in flight at once and the read-modify-write never serialises
    float2 rold[(!ENDS_ONLY) ? TPW : 1];
    if (!ENDS_ONLY && p.resid) {
#pragma unroll
      for (int i = 0; i < TPW; ++i) {
        const int t = t0 + i;
        rold[i] = (ch_ok && t < p.T) ? *reinterpret_cast<const float2*>(p.resid + seq_base + size_t(t) * p.D)
                                     : make_float2(0.f, 0.f);
      }
    }
    float2 h = make_float2(0.f, 0.f), pr = make_float2(1.f, 1.f);
#pragma unroll
    for (int i = 0; i < TPW; ++i) {
      if (TENSOR_ALPHA) {
        // out-of-range tokens carry a = 1, m = 0: the identity map
        h.x = av[i].x * h.x + (1.0f - av[i].x) * mv[i].x;
        h.y = av[i].y * h.y + (1.0f - av[i].y) * mv[i].y;
        pr.x *= av[i].x;
        pr.y *= av[i].y;
        prod[i] = pr;
      } else {
        h.x = alpha * h.x + (1.0f - alpha) * mv[i].x;
        h.y = alpha * h.y + (1.0f - alpha) * mv[i].y;
      }
      loc[i] = h;
    }
    s_end[buf][warp][lane] = h;
    if (TENSOR_ALPHA) s_prod[buf][warp][lane] = pr;
    __syncthreads();
    // carry into this warp's run, and the carry out of the whole tile
    float2 c = carry, cn;
    const float a_run = TENSOR_ALPHA ? 0.f : pw[TPW - 1];
#pragma unroll
    for (int w = 0; w < LSF_WARPS; ++w) {
      if (w == warp) cn = c;
      const float2 e = s_end[buf][w][lane];
      if (TENSOR_ALPHA) {
        const float2 q = s_prod[buf][w][lane];
        c.x = q.x * c.x + e.x;
        c.y = q.y * c.y + e.y;
        if (ENDS_ONLY) { pcarry.x *= q.x; pcarry.y *= q.y; }
      } else {
        c.x = a_run * c.x + e.x;
        c.y = a_run * c.y + e.y;
      }
    }
    carry = c;
    c = cn;
    if (ENDS_ONLY) continue;
#pragma unroll
    for (int i = 0; i < TPW; ++i) {
      const int t = t0 + i;
      if (ch_ok && t < p.T) {
        const float fx = TENSOR_ALPHA ? prod[i].x : pw[i];
        const float fy = TENSOR_ALPHA ? prod[i].y : pw[i];
        const float hx = loc[i].x + fx * c.x;
        const float hy = loc[i].y + fy * c.y;
        const size_t o = seq_base + size_t(t) * p.D;
        if (out) st2<TOut>(out + o, hx, hy);
        if (p.resid) *reinterpret_cast<float2*>(p.resid + o) = make_float2(rold[i].x + hx, rold[i].y + hy);
        if (t == p.T - 1) store_last(p, size_t(b) * p.D + ch, make_float2(hx, hy));
      }
    }
  }
  if (ENDS_ONLY && ch_ok && warp == 0) {
    const size_t e = (size_t(b) * p.n_pre_tiles + seg) * p.D + ch;
    *reinterpret_cast<float2*>(p.seg_end + e) = carry;
    if (TENSOR_ALPHA) *reinterpret_cast<float2*>(p.seg_prod + e) = pcarry;
  }
}

// Short sequences (decode steps): one thread per channel pair walks the few tokens itself.
template <bool TENSOR_ALPHA, typename TM, typename TOut>
__global__ void __launch_bounds__(256) lsf_short_kernel(const LsfArgs<false, !TENSOR_ALPHA> p) {
  pdl_wait();
  pdl_trigger();
  const size_t pair = size_t(blockIdx.x) * 256 + threadIdx.x;
  const int half_d = p.D / 2;
  if (pair >= size_t(p.B) * half_d) return;
  const int b = int(pair / half_d), ch = int(pair % half_d) * 2;
  const TM* m = reinterpret_cast<const TM*>(p.m);
  const TM* at = reinterpret_cast<const TM*>(p.alpha_t);
  TOut* out = reinterpret_cast<TOut*>(p.out);
  float alpha = 0.f;
  if constexpr (!TENSOR_ALPHA) {
    alpha = lsf_decay(p);
    lsf_leave_scalars(p.st);
  }
  float2 h = p.h0 ? *reinterpret_cast<const float2*>(p.h0 + size_t(b) * p.D + ch) : make_float2(0.f, 0.f);
  for (int t = 0; t < p.T; ++t) {
    const size_t o = (size_t(b) * p.T + t) * p.D + ch;
    const float2 mv = ld2<TM>(m + o);
    float2 a = make_float2(alpha, alpha);
    if (TENSOR_ALPHA) a = ld2<TM>(at + o);
    h.x = lsf_step(a.x, h.x, mv.x);
    h.y = lsf_step(a.y, h.y, mv.y);
    if (out) st2<TOut>(out + o, h.x, h.y);
    if (p.resid) {
      float2* r = reinterpret_cast<float2*>(p.resid + o);
      const float2 rv = *r;
      *r = make_float2(rv.x + h.x, rv.y + h.y);
    }
  }
  store_last(p, size_t(b) * p.D + ch, h);
}

// Single-token tail of a block (decode steps), three launches in one: the MoE layer's scalars from its accumulated
// statistics (moe_finalize_kernel), the LSF step with the fused residual (lsf_short_kernel at T = 1: the decay comes
// from act_var, h <- alpha h + (1 - alpha) m, x += h) and the RMSNorm that follows (norm1 of the next block or the
// final norm; rmsnorm_kernel<float, bf16>).  One warp per sequence, lanes on the channels of rmsnorm_kernel with its
// summation order, every rounding as in the three kernels: the results are theirs bit for bit.
struct LsfStepParams {
  const __nv_bfloat16* m;      // [B][C] MoE output
  LsfStats st;                 // accumulators of the MoE layer and where its scalars go
  const float* var_scale;
  float alpha_min, alpha_max;
  const float* h_in;           // [B][C] or null (zero membrane)
  float* h_out;                // [B][C] (may alias h_in)
  float* x;                    // [B][C] residual stream, in/out
  const float* w_norm;         // [C] or null: no norm wanted
  float eps;
  __nv_bfloat16* xn;           // [B][C] out (with w_norm)
  int B, C;
  bool ahead;
};

// The scalars are left by a CTA of their own.  What the kernel before this one did not make (`ahead`: it made m and the
// statistics) is fetched before the grid dependency is waited for.
__global__ void __launch_bounds__(256) lsf_step_norm_kernel(const LsfStepParams p) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const bool scalars = blockIdx.x == gridDim.x - 1, on = !scalars && row < p.B;
  const size_t base = size_t(row) * p.C;
  float4 hq[4][2], xq[4][2], wq[4][2];
  auto fetch = [&] {
    if (!on) return;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = (i * 32 + lane) * 8;
      if (c < p.C) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          hq[i][q] = p.h_in ? *reinterpret_cast<const float4*>(p.h_in + base + c + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
          xq[i][q] = *reinterpret_cast<const float4*>(p.x + base + c + 4 * q);
          if (p.w_norm) wq[i][q] = __ldg(reinterpret_cast<const float4*>(p.w_norm + c) + q);
        }
      }
    }
  };
  if (p.ahead) fetch();
  __syncwarp();
  pdl_wait();
  pdl_trigger();
  if (!p.ahead) fetch();
  if (scalars) {
    if (threadIdx.x == 0) moe_leave_scalars(p.st);
    return;
  }
  if (!on) return;
  const float alpha = lsf_alpha_from_var(p.alpha_min, p.alpha_max, __ldg(p.var_scale), stats_mean_var(p.st).y);
  float v[4][8];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int c = (i * 32 + lane) * 8;
    if (c < p.C) {
      const uint4 mw = __ldg(reinterpret_cast<const uint4*>(p.m + base + c));
      const float mv[8] = {bf16_lo(mw.x), bf16_hi(mw.x), bf16_lo(mw.y), bf16_hi(mw.y),
                           bf16_lo(mw.z), bf16_hi(mw.z), bf16_lo(mw.w), bf16_hi(mw.w)};
      float h[8] = {hq[i][0].x, hq[i][0].y, hq[i][0].z, hq[i][0].w, hq[i][1].x, hq[i][1].y, hq[i][1].z, hq[i][1].w};
      const float xv[8] = {xq[i][0].x, xq[i][0].y, xq[i][0].z, xq[i][0].w, xq[i][1].x, xq[i][1].y, xq[i][1].z, xq[i][1].w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        h[j] = lsf_step(alpha, h[j], mv[j]);
        v[i][j] = xv[j] + h[j];
        ss = __fmaf_rn(v[i][j], v[i][j], ss);
      }
      *reinterpret_cast<float4*>(p.h_out + base + c) = make_float4(h[0], h[1], h[2], h[3]);
      *reinterpret_cast<float4*>(p.h_out + base + c + 4) = make_float4(h[4], h[5], h[6], h[7]);
      *reinterpret_cast<float4*>(p.x + base + c) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
      *reinterpret_cast<float4*>(p.x + base + c + 4) = make_float4(v[i][4], v[i][5], v[i][6], v[i][7]);
    }
  }
  if (!p.w_norm) return;
  ss = warp_sum(ss);
  const float r = rsqrtf(ss / float(p.C) + p.eps);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int c = (i * 32 + lane) * 8;
    if (c < p.C) {
      const float4 wa = wq[i][0], wb = wq[i][1];
      *reinterpret_cast<uint4*>(p.xn + base + c) =
          make_uint4(pack_bf16x2(v[i][0] * r * wa.x, v[i][1] * r * wa.y), pack_bf16x2(v[i][2] * r * wa.z, v[i][3] * r * wa.w),
                     pack_bf16x2(v[i][4] * r * wb.x, v[i][5] * r * wb.y), pack_bf16x2(v[i][6] * r * wb.z, v[i][7] * r * wb.w));
    }
  }
}

constexpr int LSF_TPW = 16;                       // tokens per warp per tile
constexpr int LSF_TILE = LSF_WARPS * LSF_TPW;     // 128 tokens

template <bool TA, typename TM, typename TOut>
int launch_t(const LsfChainParams& p, cudaStream_t stream) {
  if (p.T <= 8) {
    const size_t pairs = size_t(p.B) * (p.D / 2);
    launch_dep(lsf_short_kernel<TA, TM, TOut>, unsigned((pairs + 255) / 256), 256, 0, stream, p);
    JB_LAUNCH_CHECK("lsf_short_kernel");
    return JB200_OK;
  }
  if (p.nseg > 1) {
    dim3 grid_a((p.D + LSF_CH - 1) / LSF_CH, p.B, p.n_pre_tiles);
    launch_dep(lsf_scan_kernel<TA, TM, TOut, LSF_TPW, true, false>, grid_a, LSF_THREADS, 0, stream, p);
    JB_LAUNCH_CHECK("lsf_scan_kernel<ends>");
  }
  dim3 grid((p.D + LSF_CH - 1) / LSF_CH, p.B, p.nseg);
  launch_dep(lsf_scan_kernel<TA, TM, TOut, LSF_TPW, false, false>, grid, LSF_THREADS, 0, stream, p);
  JB_LAUNCH_CHECK("lsf_scan_kernel");
  return JB200_OK;
}


// ------------------------------------------------------------------------------------------------------------
// TMA-staged scan (scalar decay, bf16 m).  FUSED: resid (f32) += h, no other output.  Otherwise: out (bf16) = h.
// Tensor maps are 3-D (channels, tokens, sequences), so tiles are clipped at the end of a sequence: loads past T
// read zeros (m = 0 leaves the recurrence a pure decay), stores past T are dropped.
// ------------------------------------------------------------------------------------------------------------
constexpr int LT_TOK = LSF_WARPS * 16;       // 128 tokens per tile (= LSF_TILE: the ends pre-pass uses the same tiles)
constexpr int LT_M_BYTES = LT_TOK * LSF_CH * 2;    // 16 KiB
constexpr int LT_R_BYTES = LT_TOK * LSF_CH * 4;    // 32 KiB

// CH channels per CTA.  64: a warp takes a run of 16 tokens; 32: two runs, one per half warp, so a tile takes four warps.
template <bool FUSED, int CH>
struct LsfTma {
  static constexpr int RPW = LSF_CH / CH, THREADS = LSF_THREADS / RPW;
  static constexpr int M_BYTES = LT_M_BYTES / RPW;
  static constexpr int STAGE_BYTES = (LT_M_BYTES + (FUSED ? LT_R_BYTES : 0)) / RPW;
  static constexpr size_t CTL_BYTES = 128 + 2 * LSF_WARPS * (CH / 2) * sizeof(float2);   // barriers + flag, run ends
  static constexpr size_t smem_bytes(int stages) { return size_t(stages) * STAGE_BYTES + CTL_BYTES + 128 /* alignment slack */; }
  // Stages: enough CTAs to put two (fused) or three (plain) on every SM -> a short ring each; a grid that leaves
  // SMs with one CTA -> that CTA gets a ring of four stages (and sequences are not cut into segments).
  static constexpr int STAGES_SHARED = FUSED ? 2 : 3;   // plain: four CTAs per SM (64 registers), so 512 CTAs (B=32 x 16 channel tiles) are one wave
  static constexpr int STAGES_ALONE = 4;
};

template <bool FUSED, int CH>
__global__ void __launch_bounds__(LsfTma<FUSED, CH>::THREADS, (FUSED ? 2 : 4) * LsfTma<FUSED, CH>::RPW)
lsf_tma_kernel(const __grid_constant__ CUtensorMap tm_m, const __grid_constant__ CUtensorMap tm_io, const LsfArgs<true, FUSED> p,
               const int n_stages, unsigned int* status) {
  using Cfg = LsfTma<FUSED, CH>;
  constexpr int TPW = LT_TOK / LSF_WARPS;    // 16 (sixteen warps of 8 tokens were measured: slower)
  extern __shared__ uint8_t lsf_smem_raw[];
  const uint32_t raw_addr = smem_u32(lsf_smem_raw);
  const uint32_t base = (raw_addr + 127u) & ~127u;
  uint8_t* tiles = lsf_smem_raw + (base - raw_addr);
  uint8_t* ctl = tiles + size_t(n_stages) * Cfg::STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(ctl);                       // [STAGES]
  uint32_t* abort_flag = reinterpret_cast<uint32_t*>(ctl + 64);
  float2 (*s_end)[LSF_WARPS][CH / 2] = reinterpret_cast<float2 (*)[LSF_WARPS][CH / 2]>(ctl + 128);   // [2][8][channel pairs]

  const int run = threadIdx.x / (CH / 2), lane = threadIdx.x % (CH / 2);   // this thread's run of a tile and channel pair
  const int b = blockIdx.y, seg = blockIdx.z;
  const int ch0 = blockIdx.x * CH;
  const int ch = ch0 + lane * 2;
  const bool ch_ok = ch < p.D;
  const int t_begin = seg * p.seg_len;
  const int t_end = min(p.T, t_begin + p.seg_len);
  const int n_tiles = (t_end - t_begin + LT_TOK - 1) / LT_TOK;

  // in a chain the kernel before this one made m and the statistics alone: residual tiles are fetched ahead of it
  bool ahead = false;
  if constexpr (FUSED) ahead = p.st.stats != nullptr;
  auto issue = [&](int i, bool residual, bool input) {      // thread 0 only
    const int s = i % n_stages;
    const uint32_t bar = smem_u32(&full[s]);
    const uint32_t dst = smem_u32(tiles + size_t(s) * Cfg::STAGE_BYTES);
    if (residual) mbar_arrive_expect_tx(bar, Cfg::STAGE_BYTES);
    if (FUSED && residual) tma_load_3d(dst + Cfg::M_BYTES, &tm_io, ch0, t_begin + i * LT_TOK, b, bar);
    if (input) tma_load_3d(dst, &tm_m, ch0, t_begin + i * LT_TOK, b, bar);
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < n_stages; ++s) mbar_init(smem_u32(&full[s]), 1);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tm_m);
    tma_prefetch_desc(&tm_io);
    if (ahead)
      for (int i = 0; i < n_stages && i < n_tiles; ++i) issue(i, true, false);
  }
  __syncwarp();
  pdl_wait();
  pdl_trigger();
  if (threadIdx.x == 0)
    for (int i = 0; i < n_stages && i < n_tiles; ++i) issue(i, !ahead, true);
  __syncwarp();
  const float alpha = lsf_decay(p);
  if constexpr (FUSED) lsf_leave_scalars(p.st);
  float pw[TPW];   // alpha^(i+1)
  {
    float a = alpha;
#pragma unroll
    for (int i = 0; i < TPW; ++i) { pw[i] = a; a *= alpha; }
  }
  float2 carry = make_float2(0.f, 0.f);
  if (p.h0 && ch_ok) carry = __ldg(reinterpret_cast<const float2*>(p.h0 + size_t(b) * p.D + ch));
  if (seg > 0 && ch_ok) {   // fold the ends of all earlier tiles (left by the ends pre-pass) into the carry-in
    const float a_tile = expf(float(LT_TOK) * logf(alpha));
    const size_t e0 = (size_t(b) * p.n_pre_tiles) * p.D + ch;
    const int n_before = seg * (p.seg_len / LT_TOK);
    for (int s2 = 0; s2 < n_before; ++s2) {
      const float2 e = __ldg(reinterpret_cast<const float2*>(p.seg_end + e0 + size_t(s2) * p.D));
      carry.x = a_tile * carry.x + e.x;
      carry.y = a_tile * carry.y + e.y;
    }
  }

  __syncthreads();

  bool ok = true;
  for (int i = 0; i < n_tiles; ++i) {
    const int s = i % n_stages;
    const int buf = i & 1;
    uint8_t* m_tile = tiles + size_t(s) * Cfg::STAGE_BYTES;
    uint8_t* r_tile = m_tile + Cfg::M_BYTES;
    if (!mbar_wait(smem_u32(&full[s]), uint32_t(i / n_stages) & 1u, abort_flag, status, JB200_STATUS_LSF_LOAD)) ok = false;
    const int tl0 = run * TPW;                           // first token of this run inside the tile
    const int t0 = t_begin + i * LT_TOK + tl0;
    float2 loc[TPW];
    float2 h = make_float2(0.f, 0.f);
    if (ok) {
#pragma unroll
      for (int j = 0; j < TPW; ++j) {
        const uint32_t w = *reinterpret_cast<const uint32_t*>(m_tile + size_t(tl0 + j) * (CH * 2) + lane * 4);
        h.x = alpha * h.x + (1.0f - alpha) * bf16_lo(w);
        h.y = alpha * h.y + (1.0f - alpha) * bf16_hi(w);
        loc[j] = h;
      }
    }
    s_end[buf][run][lane] = h;
    if (__syncthreads_or(!ok)) { ok = false; break; }
    // carry into this run, and the carry out of the whole tile (the recurrence is an affine map)
    float2 c = carry, cn = carry;
#pragma unroll
    for (int w = 0; w < LSF_WARPS; ++w) {
      if (w == run) cn = c;
      const float2 e = s_end[buf][w][lane];
      c.x = pw[TPW - 1] * c.x + e.x;
      c.y = pw[TPW - 1] * c.y + e.y;
    }
    carry = c;
#pragma unroll
    for (int j = 0; j < TPW; ++j) {
      const float hx = loc[j].x + pw[j] * cn.x, hy = loc[j].y + pw[j] * cn.y;
      if (FUSED) {
        float2* r = reinterpret_cast<float2*>(r_tile + size_t(tl0 + j) * (CH * 4) + lane * 8);
        const float2 old = *r;
        *r = make_float2(old.x + hx, old.y + hy);
      } else {
        *reinterpret_cast<uint32_t*>(m_tile + size_t(tl0 + j) * (CH * 2) + lane * 4) = pack_bf16x2(hx, hy);
      }
      if (t0 + j == p.T - 1 && p.h_last && ch_ok)
        *reinterpret_cast<float2*>(p.h_last + size_t(b) * p.D + ch) = make_float2(hx, hy);
    }
    fence_proxy_async_smem();        // the tile's new contents -> visible to the TMA store
    __syncthreads();
    if (threadIdx.x == 0) {
      tma_store_3d(&tm_io, ch0, t_begin + i * LT_TOK, b, smem_u32(FUSED ? r_tile : m_tile));
      bulk_commit_group();
      if (n_stages >= 4) {
        // deep ring: refill the stage of the tile BEFORE this one, whose store has had a whole tile's time to read
        // it, so that this thread does not sit out the latency of the store it has just issued
        if (i >= 1 && i - 1 + n_stages < n_tiles) {
          bulk_wait_group_read<1>();
          issue(i - 1 + n_stages, true, true);
        }
      } else if (i + n_stages < n_tiles) {
        bulk_wait_group_read<0>();   // the store has read the stage: it may be filled again
        issue(i + n_stages, true, true);
      }
    }
  }
  if constexpr (!FUSED) {          // the last row of the output is the last state in bf16 (stored in the loop it cost a spill)
    if (ok && p.last16 && t_end == p.T && run == 0 && ch_ok) {
      const uint8_t* tile = tiles + size_t((n_tiles - 1) % n_stages) * Cfg::STAGE_BYTES;
      *reinterpret_cast<uint32_t*>(p.last16 + size_t(b) * p.D + ch) =
          *reinterpret_cast<const uint32_t*>(tile + size_t((p.T - 1 - t_begin) % LT_TOK) * (CH * 2) + lane * 4);
    }
  }
  if (threadIdx.x == 0) bulk_wait_group<0>();   // every store has landed before the CTA gives up its shared memory
}

// Fused form for sequences of 2 to 8 tiles where a CTA per (sequence, 64 channels) leaves the chip idle: those CTAs work
// through their tiles one after another, ~2 us each (3 x 777 tokens: 15.4 us on 48 CTAs for 8 us worth of bytes), although only
// the carry is sequential.  Here a cluster takes the tiles of a sequence side by side: every CTA scans its runs from zero,
// sends their ends to the CTAs of the later tiles, and after one cluster barrier each works out its own carry along all
// runs before it.  The chain of roundings is lsf_tma_kernel's, so are the results.  In a chain the residual tile and the
// membrane are fetched before the grid dependency is waited for (`ahead`: the kernel before this one made only m).
constexpr int LC_MAX_TILES = 8;
constexpr size_t LC_END_BYTES = LSF_WARPS * 32 * sizeof(float2);      // run ends of one tile
inline size_t lc_smem_bytes(int tiles) { return 128 + LT_M_BYTES + LT_R_BYTES + size_t(tiles) * LC_END_BYTES; }

__global__ void __launch_bounds__(LSF_THREADS, 3)
lsf_cluster_kernel(const __grid_constant__ CUtensorMap tm_m, const __grid_constant__ CUtensorMap tm_io, const LsfChainParams p,
                   const bool ahead, unsigned int* status) {
  constexpr int TPW = LT_TOK / LSF_WARPS;
  extern __shared__ uint8_t lsf_smem_raw[];
  __shared__ uint64_t bar_m, bar_r;
  __shared__ uint32_t abort_flag;
  const uint32_t raw_addr = smem_u32(lsf_smem_raw);
  uint8_t* m_tile = lsf_smem_raw + (((raw_addr + 127u) & ~127u) - raw_addr);
  uint8_t* r_tile = m_tile + LT_M_BYTES;
  float2 (*ends)[LSF_WARPS][32] = reinterpret_cast<float2 (*)[LSF_WARPS][32]>(r_tile + LT_R_BYTES);   // [tile][run][lane]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x, n_tiles = gridDim.x, b = blockIdx.z;       // cluster: the tiles of one sequence
  const int ch0 = blockIdx.y * LSF_CH, ch = ch0 + lane * 2;
  const bool ch_ok = ch < p.D;
  cluster_arrive();
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar_m), 1);
    mbar_init(smem_u32(&bar_r), 1);
    abort_flag = 0;
    fence_mbar_init();
    mbar_arrive_expect_tx(smem_u32(&bar_m), LT_M_BYTES);
    mbar_arrive_expect_tx(smem_u32(&bar_r), LT_R_BYTES);
    if (ahead) tma_load_3d(smem_u32(r_tile), &tm_io, ch0, tile * LT_TOK, b, smem_u32(&bar_r));
    tma_prefetch_desc(&tm_m);
  }
  float2 c = make_float2(0.f, 0.f);
  if (ahead && p.h0 && ch_ok) c = *reinterpret_cast<const float2*>(p.h0 + size_t(b) * p.D + ch);
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  if (threadIdx.x == 0) {
    tma_load_3d(smem_u32(m_tile), &tm_m, ch0, tile * LT_TOK, b, smem_u32(&bar_m));
    if (!ahead) tma_load_3d(smem_u32(r_tile), &tm_io, ch0, tile * LT_TOK, b, smem_u32(&bar_r));
  }
  if (!ahead && p.h0 && ch_ok) c = *reinterpret_cast<const float2*>(p.h0 + size_t(b) * p.D + ch);
  const float alpha = lsf_decay(p);
  const float one_m = 1.0f - alpha;
  float a_run = alpha;                           // alpha^TPW
#pragma unroll
  for (int j = 1; j < TPW; ++j) a_run *= alpha;

  bool ok = mbar_wait(smem_u32(&bar_m), 0u, &abort_flag, status, JB200_STATUS_LSF_LOAD);
  const int tl0 = warp * TPW;
  float2 loc[TPW], h = make_float2(0.f, 0.f);
#pragma unroll
  for (int j = 0; j < TPW; ++j) {
    const uint32_t w = *reinterpret_cast<const uint32_t*>(m_tile + size_t(tl0 + j) * (LSF_CH * 2) + lane * 4);
    h.x = alpha * h.x + one_m * bf16_lo(w);
    h.y = alpha * h.y + one_m * bf16_hi(w);
    loc[j] = h;
  }
  __syncwarp();
  cluster_wait();                                // the other CTAs have started: their shared memory may be written
  ends[tile][warp][lane] = h;
  for (int t = tile + 1; t < n_tiles; ++t) cluster_st_64(cluster_map(smem_u32(&ends[tile][warp][lane]), uint32_t(t)), h);
  __syncwarp();
  cluster_arrive();
  lsf_leave_scalars(p.st);
  __syncwarp();
  cluster_wait();
#pragma unroll 8
  for (int q = 0; q < tile * LSF_WARPS + warp; ++q) {
    const float2 e = (&ends[0][0][0])[q * 32 + lane];
    c.x = a_run * c.x + e.x;
    c.y = a_run * c.y + e.y;
  }
  ok = mbar_wait(smem_u32(&bar_r), 0u, &abort_flag, status, JB200_STATUS_LSF_LOAD) && ok;
  const int t0 = tile * LT_TOK + tl0;
  float a = alpha;
#pragma unroll
  for (int j = 0; j < TPW; ++j, a *= alpha) {
    const float hx = loc[j].x + a * c.x, hy = loc[j].y + a * c.y;
    float2* r = reinterpret_cast<float2*>(r_tile + size_t(tl0 + j) * (LSF_CH * 4) + lane * 8);
    const float2 old = *r;
    *r = make_float2(old.x + hx, old.y + hy);
    if (t0 + j == p.T - 1 && ch_ok && ok)
      store_last(p, size_t(b) * p.D + ch, make_float2(hx, hy));
  }
  fence_proxy_async_smem();
  if (__syncthreads_or(!ok)) return;
  if (threadIdx.x == 0) {
    tma_store_3d(&tm_io, ch0, tile * LT_TOK, b, smem_u32(r_tile));
    bulk_commit_group();
    bulk_wait_group<0>();
  }
}

int make_lsf_map(CUtensorMap* tm, const void* ptr, CUtensorMapDataType dt, int elem, int B, int T, int D, int channels = LSF_CH) {
  const cuuint64_t gdim[3] = {cuuint64_t(D), cuuint64_t(T), cuuint64_t(B)};
  const cuuint64_t gstride[2] = {cuuint64_t(D) * elem, cuuint64_t(T) * D * elem};
  const cuuint32_t box[3] = {cuuint32_t(channels), cuuint32_t(LT_TOK), 1};
  return encode_tiled(tm, dt, 3, ptr, gdim, gstride, box, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                      "lsf_scan");
}

template <bool FUSED>
int launch_tma(LsfChainParams p, cudaStream_t stream) {
  using Cfg = LsfTma<FUSED, LSF_CH>;
  const int sms = sm_count();
  if (sms <= 0) return JB200_ERR_CUDA;
  const long ctas = long((p.D + LSF_CH - 1) / LSF_CH) * p.B;
  int stages = Cfg::STAGES_SHARED;
  if (2 * ctas >= sms && ctas <= 2L * sms) {
    // between half a wave and two CTAs per SM: one uncut CTA per (sequence, 64 channels) with a deep ring keeps
    // the SM's loads in flight by itself; cutting T would cost the ends pre-pass (a second read of m, a launch)
    stages = Cfg::STAGES_ALONE;
    p.nseg = 1;
    p.seg_len = (p.T + LT_TOK - 1) / LT_TOK * LT_TOK;
    p.n_pre_tiles = 0;
  }
  CUtensorMap tm_m, tm_io;
  int rc;
  if ((rc = make_lsf_map(&tm_m, p.m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.B, p.T, p.D)) != JB200_OK) return rc;
  if (FUSED) rc = make_lsf_map(&tm_io, p.resid, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, p.B, p.T, p.D);
  else rc = make_lsf_map(&tm_io, p.out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.B, p.T, p.D);
  if (rc != JB200_OK) return rc;
  unsigned int* status = device_status_ptr();
  if (!status) return JB200_ERR_CUDA;
  if constexpr (!FUSED) {
    // Well beyond three CTAs of 64 channels per SM some SMs hold a fourth and finish last (32 x 2048: 3.46 on average); tiles
    // of half the channels even that out, though they cost 3 % of themselves (30 x 2048 54.7 against 58.9 us, 32 x 2048 57.4
    // against 60.5, but 28 x 2048 52.5 against 51.0 and 24 x 2048 47.2 against 44.5).  Measured at T = 2048; the
    // same unevenness beyond four CTAs per SM is left alone.
    if (ctas > 3L * sms + sms / 8 && ctas <= 4L * sms) {
      using Half = LsfTma<false, LSF_CH / 2>;
      if ((rc = make_lsf_map(&tm_m, p.m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.B, p.T, p.D, LSF_CH / 2)) != JB200_OK) return rc;
      if ((rc = make_lsf_map(&tm_io, p.out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.B, p.T, p.D, LSF_CH / 2)) != JB200_OK) return rc;
      auto kernel = lsf_tma_kernel<false, LSF_CH / 2>;
      JB_MAX_SMEM(kernel, Half::smem_bytes(Half::STAGES_SHARED));
      launch_dep(kernel, dim3((p.D + LSF_CH / 2 - 1) / (LSF_CH / 2), p.B, 1), Half::THREADS, Half::smem_bytes(Half::STAGES_SHARED), stream,
                 tm_m, tm_io, p, Half::STAGES_SHARED, status);
      JB_LAUNCH_CHECK("lsf_tma_kernel<half>");
      return JB200_OK;
    }
  }
  // all tiles at once where a CTA per sequence and channel tile would leave SMs empty (beyond, deep rings overlap as well:
  // 8 x 300 tokens 3.28 against 3.25 ms for 24 layers)
  const int n_tiles = (p.T + LT_TOK - 1) / LT_TOK;
  if (FUSED && p.nseg == 1 && n_tiles >= 2 && n_tiles <= LC_MAX_TILES && 2 * ctas < sms) {
    JB_MAX_SMEM(lsf_cluster_kernel, lc_smem_bytes(LC_MAX_TILES));
    launch_dep_cluster(lsf_cluster_kernel, dim3(n_tiles, (p.D + LSF_CH - 1) / LSF_CH, p.B), LSF_THREADS, lc_smem_bytes(n_tiles),
                       n_tiles, stream, tm_m, tm_io, p, p.st.stats != nullptr, status);
    JB_LAUNCH_CHECK("lsf_cluster_kernel");
    return JB200_OK;
  }
  if (p.nseg > 1) {
    dim3 grid_a((p.D + LSF_CH - 1) / LSF_CH, p.B, p.n_pre_tiles);
    launch_dep(lsf_scan_kernel<false, __nv_bfloat16, __nv_bfloat16, LSF_TPW, true, FUSED>, grid_a, LSF_THREADS, 0, stream, p);
    JB_LAUNCH_CHECK("lsf_scan_kernel<ends>");
  }
  dim3 grid((p.D + LSF_CH - 1) / LSF_CH, p.B, p.nseg);
  auto kernel = lsf_tma_kernel<FUSED, LSF_CH>;
  JB_MAX_SMEM(kernel, Cfg::smem_bytes(Cfg::STAGES_ALONE));
  launch_dep(kernel, grid, LSF_THREADS, Cfg::smem_bytes(stages), stream, tm_m, tm_io, p, stages, status);
  JB_LAUNCH_CHECK("lsf_tma_kernel");
  return JB200_OK;
}

// Segments so that about two CTAs per SM exist, each at least four tiles long.
void pick_lsf_segments(int B, int T, int D, int sms, int* seg_len, int* nseg) {
  const long ctas = long((D + LSF_CH - 1) / LSF_CH) * B;
  long want = (2L * sms) / ctas;   // rounded down: all CTAs resident at once, no partial second wave
  const long max_seg = T / (4 * LSF_TILE);
  if (want > max_seg) want = max_seg;
  if (want < 1) want = 1;
  long len = (T + want - 1) / want;
  len = (len + LSF_TILE - 1) / LSF_TILE * LSF_TILE;
  *seg_len = int(len);
  *nseg = int((T + len - 1) / len);
}

}  // namespace

size_t lsf_scan_scratch_bytes(int B, int T, int D) {
  if (B <= 0 || T <= 0 || D <= 0) return 0;
  const int sms = sm_count();
  int len, ns;
  pick_lsf_segments(B, T, D, sms > 0 ? sms : 148, &len, &ns);
  return size_t(2) * B * size_t(ns - 1) * size_t(len / LSF_TILE) * D * sizeof(float);
}

int launch_lsf_scan(const void* m, int m_dtype, const void* alpha_tensor, const float* alpha_scalar,
                    const float* act_var, const float* var_scale, float alpha_min, float alpha_max, const float* h0,
                    float* resid, void* out, int out_dtype, void* h_last, int last_dtype, void* scratch, int B, int T, int D,
                    cudaStream_t stream, const LsfStats* st) {
  JB_REQUIRE(B >= 0 && T >= 0 && D > 0, "lsf_scan: bad shape (%d, %d, %d)", B, T, D);
  JB_REQUIRE(D % 2 == 0, "lsf_scan: channel count (%d) must be even", D);
  JB_REQUIRE(B <= 65535, "lsf_scan: batch (%d) exceeds 65535", B);
  JB_REQUIRE((m_dtype == 0 || m_dtype == 1) && (out_dtype == 0 || out_dtype == 1) && (last_dtype == 0 || last_dtype == 1), "lsf_scan: dtype must be 0 (f32) or 1 (bf16)");
  if (B == 0 || T == 0) return JB200_OK;
  JB_REQUIRE(m != nullptr, "lsf_scan: null input");
  JB_REQUIRE(alpha_tensor || alpha_scalar || ((act_var || st) && var_scale), "lsf_scan: no decay given");
  JB_REQUIRE(out || resid || h_last, "lsf_scan: no output requested");
  const uintptr_t a8 = 7u, a4 = 3u;
  JB_REQUIRE((reinterpret_cast<uintptr_t>(m) & (m_dtype == 0 ? a8 : a4)) == 0, "lsf_scan: input pointer misaligned");
  JB_REQUIRE(!alpha_tensor || (reinterpret_cast<uintptr_t>(alpha_tensor) & (m_dtype == 0 ? a8 : a4)) == 0, "lsf_scan: alpha pointer misaligned");
  JB_REQUIRE(!out || (reinterpret_cast<uintptr_t>(out) & (out_dtype == 0 ? a8 : a4)) == 0, "lsf_scan: output pointer misaligned");
  JB_REQUIRE(!resid || (reinterpret_cast<uintptr_t>(resid) & a8) == 0, "lsf_scan: residual pointer misaligned");
  JB_REQUIRE((!h0 || (reinterpret_cast<uintptr_t>(h0) & a8) == 0) && (!h_last || (reinterpret_cast<uintptr_t>(h_last) & a8) == 0),
             "lsf_scan: state pointer misaligned");
  LsfChainParams p = {};
  p.m = m; p.alpha_t = alpha_tensor; p.alpha_s = alpha_scalar; p.act_var = act_var; p.var_scale = var_scale;
  p.alpha_min = alpha_min; p.alpha_max = alpha_max; p.h0 = h0; p.resid = resid; p.out = out;
  p.h_last = last_dtype ? nullptr : static_cast<float*>(h_last);
  p.last16 = last_dtype ? static_cast<__nv_bfloat16*>(h_last) : nullptr;
  p.B = B; p.T = T; p.D = D;
  p.seg_len = (T + LSF_TILE - 1) / LSF_TILE * LSF_TILE;
  p.nseg = 1;
  p.n_pre_tiles = 0;
  p.seg_end = p.seg_prod = nullptr;
  if (st) p.st = st->counted();
  if (scratch) {
    JB_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & a8) == 0, "lsf_scan: scratch pointer misaligned");
    const int sms = sm_count();
    if (sms <= 0) return JB200_ERR_CUDA;
    pick_lsf_segments(B, T, D, sms, &p.seg_len, &p.nseg);
    p.n_pre_tiles = (p.nseg - 1) * (p.seg_len / LSF_TILE);
    p.seg_end = reinterpret_cast<float*>(scratch);
    p.seg_prod = p.seg_end + size_t(B) * p.n_pre_tiles * D;
  }
  JB_REQUIRE(p.nseg <= 65535 && p.n_pre_tiles <= 65535, "lsf_scan: too many segments");
  const bool ta = alpha_tensor != nullptr;
  JB_REQUIRE(!ta || last_dtype == 0, "lsf_scan: per-element decays leave an f32 state");
  using bf = __nv_bfloat16;
  // the forms the model and the scan sweep run: tiles by TMA (3-D maps need 16-byte aligned rows)
  if (!ta && m_dtype == 1 && T > 8 && D % 8 == 0 && aligned16(m) && B * long(T) * D < (1L << 40)) {
    if (resid && !out && last_dtype == 0 && aligned16(resid)) return launch_tma<true>(p, stream);
    if (out && !resid && out_dtype == 1 && aligned16(out)) return launch_tma<false>(p, stream);
  }
  JB_REQUIRE(!st || (!ta && T <= 8), "lsf_scan: the decay comes from the accumulators in the fused form alone");
  if (!ta) {
    if (m_dtype == 1 && out_dtype == 1) return launch_t<false, bf, bf>(p, stream);
    if (m_dtype == 1 && out_dtype == 0) return launch_t<false, bf, float>(p, stream);
    if (m_dtype == 0 && out_dtype == 0) return launch_t<false, float, float>(p, stream);
    return launch_t<false, float, bf>(p, stream);
  }
  if (m_dtype == 1 && out_dtype == 1) return launch_t<true, bf, bf>(p, stream);
  if (m_dtype == 1 && out_dtype == 0) return launch_t<true, bf, float>(p, stream);
  if (m_dtype == 0 && out_dtype == 0) return launch_t<true, float, float>(p, stream);
  return launch_t<true, float, bf>(p, stream);
}

int launch_lsf_step_norm(const void* m_bf16, const LsfStats& st, const float* var_scale, float alpha_min, float alpha_max,
                         const float* h_in, float* h_out, float* x, const float* w_norm, float eps, void* xn_bf16, int B,
                         int C, cudaStream_t stream, bool ahead) {
  JB_REQUIRE(B >= 0 && C > 0, "lsf_step_norm: bad shape (%d, %d)", B, C);
  JB_REQUIRE(C % 8 == 0 && C <= 1024, "lsf_step_norm: d_model (%d) must be a multiple of 8 and at most 1024", C);
  JB_REQUIRE(st.E >= 0 && st.E <= 64 && st.n_tokens > 0 && st.n_elems > 0, "lsf_step_norm: bad counts");
  if (B == 0) return JB200_OK;
  JB_REQUIRE(m_bf16 && st.stats && st.scalars && var_scale && h_out && x, "lsf_step_norm: null pointer");
  JB_REQUIRE((w_norm == nullptr) == (xn_bf16 == nullptr), "lsf_step_norm: norm weight and normalised output come together");
  JB_REQUIRE(aligned16(m_bf16) && aligned16(h_out) && aligned16(x) && (!h_in || aligned16(h_in)) &&
                 (!w_norm || (aligned16(w_norm) && aligned16(xn_bf16))),
             "lsf_step_norm: pointers must be 16-byte aligned");
  LsfStepParams p;
  p.m = reinterpret_cast<const __nv_bfloat16*>(m_bf16);
  p.st = st.counted();
  p.var_scale = var_scale; p.alpha_min = alpha_min; p.alpha_max = alpha_max;
  p.h_in = h_in; p.h_out = h_out; p.x = x; p.w_norm = w_norm; p.eps = eps;
  p.xn = reinterpret_cast<__nv_bfloat16*>(xn_bf16);
  p.B = B; p.C = C;
  p.ahead = ahead;
  launch_dep(lsf_step_norm_kernel, (B + 7) / 8 + 1, 256, 0, stream, p);
  JB_LAUNCH_CHECK("lsf_step_norm_kernel");
  return JB200_OK;
}

}  // namespace jb
