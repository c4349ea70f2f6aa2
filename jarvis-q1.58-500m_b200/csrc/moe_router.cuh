// Device pieces of the top-2 router (jarvis_engine/jarvis_model.py:218-224) shared by its kernels.
#pragma once
#include "common.cuh"

namespace jb {

#if defined(__CUDACC__)

// The expert an assignment is sorted under: router_finish leaves -1 where logits are NaN.
__device__ __forceinline__ int clamp_expert(long long e, int E) { return e < 0 ? 0 : (e >= E ? E - 1 : int(e)); }

// logits of one token (already warp-reduced, identical in every lane) -> softmax, top-2 with ties going
// to the lower expert id, gates, and the per-warp accumulators of P and the top-1 histogram.
template <int E>
__device__ __forceinline__ void router_finish(const float (&acc)[E], int lane, int tok, int64_t* topk_idx,
                                              float* gates, float* probs_out, int* h_acc, float (&p_local)[E],
                                              int* load_acc = nullptr) {
  float mx = acc[0];
#pragma unroll
  for (int e = 1; e < E; ++e) mx = fmaxf(mx, acc[e]);
  float p[E], den = 0.f;
#pragma unroll
  for (int e = 0; e < E; ++e) { p[e] = expf(acc[e] - mx); den += p[e]; }
  const float inv = 1.0f / den;
  int i0 = 0, i1 = -1;
  float p0 = -1.f, p1 = -1.f;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    p[e] *= inv;
    if (p[e] > p0) { p1 = p0; i1 = i0; p0 = p[e]; i0 = e; }
    else if (p[e] > p1) { p1 = p[e]; i1 = e; }
  }
  if (lane == 0) {
    topk_idx[size_t(tok) * 2 + 0] = i0;
    topk_idx[size_t(tok) * 2 + 1] = i1;
    const float g = p0 + p1 + 1e-8f;
    gates[size_t(tok) * 2 + 0] = p0 / g;
    gates[size_t(tok) * 2 + 1] = p1 / g;
    if (probs_out) {
#pragma unroll
      for (int e = 0; e < E; ++e) probs_out[size_t(tok) * E + e] = p[e];
    }
    atomicAdd(&h_acc[i0], 1);
    if (load_acc) {                // assignments, first and second ones, as clamp_expert sorts them
      atomicAdd(&load_acc[i0], 1);
      atomicAdd(&load_acc[i1 < 0 ? 0 : i1], 1);
    }
#pragma unroll
    for (int e = 0; e < E; ++e) p_local[e] += p[e];
  }
}

// Router weights in shared memory: [E][C] with the 4-float groups of every row swizzled (group g of a row
// sits at g ^ ((g >> 3) & 1)).  A lane reads the two groups of its 8 consecutive channels, so lanes are
// 32 bytes apart and, unswizzled, lanes l and l + 4 of each 8-lane phase would hit the same banks.
__device__ __forceinline__ int router_w_index(int c) {   // c: channel, any value; returns the swizzled column
  const int g = c >> 2;
  return ((g ^ ((g >> 3) & 1)) << 2) | (c & 3);
}

// acc + the products of 8 consecutive channels: the one form every router kernel uses, so that their logits have the same bits
__device__ __forceinline__ float router_dot(float acc, const float (&xv)[8], float4 wa, float4 wb) {
  return acc + (xv[0] * wa.x + xv[1] * wa.y + xv[2] * wa.z + xv[3] * wa.w + xv[4] * wb.x + xv[5] * wb.y + xv[6] * wb.z +
                xv[7] * wb.w);
}

// 8 consecutive activations times the matching router weights of every expert
template <int E>
__device__ __forceinline__ void router_dot8(const float (&xv)[8], const float* w_s, int C, int c, float (&acc)[E]) {
  const int ca = router_w_index(c), cb = router_w_index(c + 4);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const float4 wa = *reinterpret_cast<const float4*>(w_s + e * C + ca);
    const float4 wb = *reinterpret_cast<const float4*>(w_s + e * C + cb);
    acc[e] = router_dot(acc[e], xv, wa, wb);
  }
}

#endif

}  // namespace jb
