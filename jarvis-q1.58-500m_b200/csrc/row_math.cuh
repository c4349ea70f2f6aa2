// Pieces of the row kernels for few tokens (moe_small.cu, step_cluster.cu): a warp holds a row of up to 1024 channels in its
// registers.  One definition of each, so that all forms give the same bits.
#pragma once
#include "common.cuh"

namespace jb {

#if defined(__CUDACC__)

// Channel of element j of group i of a lane in the row kernels: (32 i + lane) * 8 + j, four groups for C = 1024.
constexpr int GROUPS = 4;

__device__ __forceinline__ void load8(const float* src, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(src), b = *reinterpret_cast<const float4*>(src + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void store8(float* dst, const float (&v)[8]) {
  *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(dst + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ uint4 norm8(const float (&v)[8], float r, float4 wa, float4 wb) {
  return make_uint4(pack_bf16x2(v[0] * r * wa.x, v[1] * r * wa.y), pack_bf16x2(v[2] * r * wa.z, v[3] * r * wa.w),
                    pack_bf16x2(v[4] * r * wb.x, v[5] * r * wb.y), pack_bf16x2(v[6] * r * wb.z, v[7] * r * wb.w));
}

// One token's row from its two expert rows (sparse_model.cu:117-165): put(i, 8 values rounded to bf16) for every group; the sums
// of the unrounded values over the warp.
struct Combined { float s1, s2; };
template <typename F>
__device__ __forceinline__ Combined combine_values(const uint4 (&ya)[GROUPS], const uint4 (&yb)[GROUPS], float2 g, int lane, int C,
                                                   F&& put) {
  float s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int i = 0; i < GROUPS; ++i) {
    if ((i * 32 + lane) * 8 < C) {
      const uint32_t wa[4] = {ya[i].x, ya[i].y, ya[i].z, ya[i].w}, wb[4] = {yb[i].x, yb[i].y, yb[i].z, yb[i].w};
      float acc[8];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[2 * j] = __fmaf_rn(g.y, bf16_lo(wb[j]), __fmul_rn(g.x, bf16_lo(wa[j])));
        acc[2 * j + 1] = __fmaf_rn(g.y, bf16_hi(wb[j]), __fmul_rn(g.x, bf16_hi(wa[j])));
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) { s1 += acc[j]; s2 = __fmaf_rn(acc[j], acc[j], s2); }
      put(i, make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]), pack_bf16x2(acc[4], acc[5]),
                        pack_bf16x2(acc[6], acc[7])));
    }
  }
  return {warp_sum(s1), warp_sum(s2)};
}

// Stable counting sort of the 2 N assignments by expert by one warp, 32 at a time and all loaded at once
// (sparse_model.cu:23-90).  A negative id (NaN logits) is sorted under expert 0.
template <int E, int ROUNDS>
__device__ __forceinline__ void sort_routes(const long long* ids, int N, int lane, int* counts, int* offsets, int* scatter,
                                            int* gather, int* gate_idx) {
  const int M = 2 * N;
  int n_of = 0;                                  // lane e < E: assignments of expert e
  int ex[ROUNDS];
#pragma unroll
  for (int i = 0; i < ROUNDS; ++i) ex[i] = i * 32 + lane < M ? max(int(__ldcg(ids + i * 32 + lane)), 0) : -1;
#pragma unroll
  for (int i = 0; i < ROUNDS; ++i) {
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const unsigned b = __ballot_sync(0xffffffffu, ex[i] == q);
      if (lane == q) n_of += __popc(b);
    }
  }
  int incl = n_of;
#pragma unroll
  for (int o = 1; o < E; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  int at = incl - n_of;                          // lane e: next free slot of expert e
  if (lane < E) {
    counts[lane] = n_of;
    offsets[lane] = at;
    if (lane == E - 1) offsets[E] = incl;
  }
#pragma unroll
  for (int i = 0; i < ROUNDS; ++i) {
    const int m = i * 32 + lane, e = ex[i];
    int slot = 0;
#pragma unroll
    for (int q = 0; q < E; ++q) {
      const unsigned b = __ballot_sync(0xffffffffu, e == q);
      const int base = __shfl_sync(0xffffffffu, at, q);
      if (e == q) slot = base + __popc(b & ((1u << lane) - 1u));
      if (lane == q) at += __popc(b);
    }
    if (m < M) {
      scatter[m] = slot;
      gather[slot] = m >> 1;
      gate_idx[slot] = m & 1;
    }
  }
}

#endif

}  // namespace jb
