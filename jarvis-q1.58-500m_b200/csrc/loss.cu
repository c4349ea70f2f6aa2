// Evaluation loss from bf16 logits (Jarvis.forward with targets, jarvis_engine/jarvis_model.py:536-545): per-row cross
// entropy in one pass over the row, then one small launch for the mean and the auxiliary terms.  Replaces a float32
// copy of the logits (12 bytes of traffic per logit with its softmax) and ~150 scalar tensor operations.
#include "common.cuh"
#include "launchers.h"

namespace jb {

namespace {

constexpr int CE_THREADS = 512;
constexpr float LOG2E = 1.44269504088896340736f;

// One CTA per row.  Bound by HBM: 2 bytes per logit, 100 KB per row at the model's vocabulary; every thread keeps a
// running maximum and the sum of exponentials relative to it, rescaled once per eight values that raise the maximum.
__global__ void __launch_bounds__(CE_THREADS)
ce_rows_kernel(const __nv_bfloat16* __restrict__ logits, int ld, int V, const int64_t* __restrict__ targets,
               float* __restrict__ row_loss) {
  pdl_wait();
  pdl_trigger();
  __shared__ float s_m[CE_THREADS / 32], s_s[CE_THREADS / 32];
  const int row = blockIdx.x, t = threadIdx.x;
  const __nv_bfloat16* lr = logits + size_t(row) * ld;
  float m = -INFINITY, s = 0.f;
  auto take = [&](const float (&v)[8]) {
    float mx = v[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) mx = fmaxf(mx, v[j]);
    if (mx > m) { s *= exp2f((m - mx) * LOG2E); m = mx; }
    if (m == -INFINITY) {                  // no finite value yet: fmaxf passes NaN over, and -inf counts as nothing
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (v[j] != v[j]) s = v[j];
      return;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) s += exp2f((v[j] - m) * LOG2E);
  };
  const int nv = V >> 3;
#pragma unroll 4
  for (int c = t; c < nv; c += CE_THREADS) {
    const uint4 w = __ldg(reinterpret_cast<const uint4*>(lr) + c);
    const float v[8] = {bf16_lo(w.x), bf16_hi(w.x), bf16_lo(w.y), bf16_hi(w.y), bf16_lo(w.z), bf16_hi(w.z), bf16_lo(w.w), bf16_hi(w.w)};
    take(v);
  }
  if (8 * nv + t < V) {                    // fewer than eight left over
    float v[8];
    v[0] = __bfloat162float(lr[8 * nv + t]);
#pragma unroll
    for (int j = 1; j < 8; ++j) v[j] = -INFINITY;
    take(v);
  }
  auto merge = [&](float m2, float s2) {
    const float mx = fmaxf(m, m2);
    s = mx == -INFINITY ? s + s2 : s * exp2f((m - mx) * LOG2E) + s2 * exp2f((m2 - mx) * LOG2E);
    m = mx;
  };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) merge(__shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, s, o));
  if ((t & 31) == 0) { s_m[t >> 5] = m; s_s[t >> 5] = s; }
  __syncthreads();
  if (t == 0) {
    for (int w = 1; w < CE_THREADS / 32; ++w) merge(s_m[w], s_s[w]);
    const long long y = targets[row];
    float loss = __int_as_float(0x7fc00000);
    if (y >= 0 && y < V) loss = m + logf(s) - __bfloat162float(lr[y]);
    row_loss[row] = y == -100 ? 0.f : loss;
  }
}

__global__ void __launch_bounds__(1024)
ce_mean_kernel(const float* __restrict__ row_loss, const int64_t* __restrict__ targets, int n_rows,
               const float* __restrict__ aux_a, int stride_a, const float* __restrict__ aux_b, int n_aux,
               float* __restrict__ loss) {
  pdl_wait();
  pdl_trigger();
  __shared__ double s_sum[32];
  __shared__ int s_cnt[32];
  double sum = 0.0;
  int cnt = 0;
  for (int r = threadIdx.x; r < n_rows; r += 1024) {
    sum += double(row_loss[r]);
    cnt += targets[r] != -100;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  }
  if ((threadIdx.x & 31) == 0) { s_sum[threadIdx.x >> 5] = sum; s_cnt[threadIdx.x >> 5] = cnt; }
  __syncthreads();
  if (threadIdx.x == 0) {
    sum = 0.0; cnt = 0;
    for (int w = 0; w < 32; ++w) { sum += s_sum[w]; cnt += s_cnt[w]; }
    float extra_a = 0.f, extra_b = 0.f;
    for (int i = 0; i < n_aux; ++i) {
      if (aux_a) extra_a += aux_a[size_t(i) * stride_a];
      if (aux_b) extra_b += aux_b[i];
    }
    *loss = float(sum / double(cnt)) + extra_a + extra_b;       // no row with a target: 0 / 0 = NaN, as torch gives
  }
}

}  // namespace

int launch_cross_entropy(const void* logits, int ld, int n_rows, int V, const int64_t* targets, float* row_loss,
                         const float* aux_a, int stride_a, const float* aux_b, int n_aux, float* loss, cudaStream_t stream) {
  JB_REQUIRE(n_rows >= 0 && V >= 1 && ld >= V && ld % 8 == 0 && n_aux >= 0, "cross_entropy: bad shape (%d rows, V=%d, ld=%d)", n_rows, V, ld);
  JB_REQUIRE(loss && (n_rows == 0 || (logits && targets && row_loss)), "cross_entropy: null pointer");
  JB_REQUIRE(aligned16(logits), "cross_entropy: logits must be 16-byte aligned");
  if (n_rows > 0) {
    launch_dep(ce_rows_kernel, n_rows, CE_THREADS, 0, stream, reinterpret_cast<const __nv_bfloat16*>(logits), ld, V, targets, row_loss);
    JB_LAUNCH_CHECK("ce_rows_kernel");
  }
  launch_dep(ce_mean_kernel, 1, 1024, 0, stream, row_loss, targets, n_rows, aux_a, stride_a, aux_b, n_aux, loss);
  JB_LAUNCH_CHECK("ce_mean_kernel");
  return JB200_OK;
}

}  // namespace jb
