// Ternary linear layers for a few tokens (decode steps of small batches, short prompts) on mma.sync.
//
// At 1..16 tokens a layer's four products are under 1 us of arithmetic and 5 MB of 2-bit weights; ternary_gemm_kernel
// spends 11-18 us on each of them (set-up of TMEM, barriers and tensor maps, then a ring whose every stage waits for a
// decode through shared memory, on as few as 8 of the 148 SMs).  Here a CTA takes 64 out-features and copies their codes
// and the token rows - one contiguous block each - to shared memory with asynchronous 16-byte copies, all in flight at
// once (one bulk copy per row measured 1-3 us slower); a warp then walks all of K for 16 out-features x 8 or 16 tokens.
// The weights do not depend on the kernel before this one: in a chain they are requested before the grid dependency is
// waited for.  The first
// expert matrix takes every token for every expert and stores only the routed ones (fetching rows through the gather map put one
// more memory latency and most of the instructions of a call in front of its first MMA).
//
// Results are those of ternary_gemm_kernel bit for bit: the f32 accumulator is one chain over K in steps of 16, and
// mma.sync.m16n8k16 rounds a step as tcgen05.mma does (measured: no differing bit for K = 16..2048, normal and
// log-normal data).  Splitting K over warps would be ~0.6 us faster per call, but reordered sums make calls of different
// sizes differ in the last bit, which a router's near-ties turn into different experts.
//
// ldmatrix delivers the activations in natural K order; the four lanes of a quad read the same weight words and shift
// out their own two pairs (a shift and a mask per bf16 pair).  Rows g and g + 8 of a fragment are out-features 2g and
// 2g + 1, so that a lane ends up with neighbours.  Loops are kept short: every instruction runs a few times per launch,
// so the time to fetch code is part of the latency.
// The legacy tensor path is on purpose: tcgen05 would need the decoded weights in shared or tensor memory first, and at
// these sizes the MMA rate is not what bounds the call - latency is.
#include "common.cuh"
#include "gemm_shared.cuh"
#include "launchers.h"

namespace jb {

namespace {

constexpr int ROW_WARPS = 4;           // 16-feature tiles of a CTA, a warp each: they share the copy of the token rows

struct SmallGemmParams {
  const __nv_bfloat16* x;      // [M][K]
  const uint8_t* w;            // prepared [G][N][K/4]
  const float* alpha;          // [G][N / alpha_rows]
  const int32_t* seg;          // device [G+1] or null (one segment [0, M))
  const int64_t* idx;          // every group takes all M rows of x and row n goes to out row scatter[2n + k] where
  const int32_t* scatter;      //   idx[2n + k] is the group ([M][2] both); or null: group g takes rows [seg[g], seg[g + 1])
  void* out;                   // [M][N], or [2M][N] with idx
  int M, N, K, alpha_rows, epilogue;
};

__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// Two neighbouring out-features of one token, alpha applied.
__device__ __forceinline__ void store_pair(const SmallGemmParams& p, size_t o, float a, float b) {
  if (p.epilogue == JB200_EPI_RESID_F32) {
    // one addition per element, done by the memory system: nothing waits for the old value
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(reinterpret_cast<float*>(p.out) + o), "f"(a), "f"(b) : "memory");
  } else {
    if (p.epilogue == JB200_EPI_GELU_BF16) { a = gelu_erf(a); b = gelu_erf(b); }
    *reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(p.out) + o) = pack_bf16x2(a, b);
  }
}

// Operands of a double step (32 in-features): code words of out-features 2g and 2g + 1, activations of TT token tiles.
template <int TT>
struct Step {
  uint32_t lo[2], hi[2], b[TT][4];
  __device__ __forceinline__ void load(uint32_t wa, uint32_t w_stride, uint32_t xa, uint32_t x_stride, int s) {
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(lo[0]), "=r"(lo[1]) : "r"(wa + uint32_t(s) * 4u));
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(hi[0]), "=r"(hi[1]) : "r"(wa + w_stride + uint32_t(s) * 4u));
#pragma unroll
    for (int i = 0; i < TT; ++i)
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                   : "=r"(b[i][0]), "=r"(b[i][1]), "=r"(b[i][2]), "=r"(b[i][3])
                   : "r"(xa + uint32_t(i) * 8u * x_stride + uint32_t(s) * 32u));
  }
  __device__ __forceinline__ void mma(float (&acc)[TT][4], int t) const {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t a[4] = {(lo[h] << (14 - 2 * t)) & 0xC000C000u, (hi[h] << (14 - 2 * t)) & 0xC000C000u,   // in-features 2t, 2t + 1
                             (lo[h] << (6 - 2 * t)) & 0xC000C000u, (hi[h] << (6 - 2 * t)) & 0xC000C000u};    // 8 + 2t, 9 + 2t
#pragma unroll
      for (int i = 0; i < TT; ++i) mma_16816(acc[i], a, b[i][2 * h], b[i][2 * h + 1]);
    }
  }
};

// TT: 8-token tiles of a pass over a segment; every warp takes all of them for its 16 out-features.
template <int TT>
__global__ void __launch_bounds__(32 * ROW_WARPS) small_gemm_kernel(const SmallGemmParams p) {
  extern __shared__ __align__(128) uint8_t small_smem[];
  constexpr int THREADS = 32 * ROW_WARPS, ROWS = 16 * ROW_WARPS, TOK = 8 * TT;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int f0 = blockIdx.x * ROWS, grp = blockIdx.y;
  const uint32_t w_stride = uint32_t(p.K / 4) + 16u, x_stride = uint32_t(p.K) * 2u + 16u;   // padded: no bank conflicts
  const uint32_t wgt = smem_u32(small_smem), act = wgt + uint32_t(ROWS) * w_stride;

  // `n_rows` rows of `pieces` 16-byte pieces, contiguous in memory, to rows padded by one piece
  auto copy_rows = [&](uint32_t dst, const void* from, int n_rows, int pieces) {
    const uint8_t* src = static_cast<const uint8_t*>(from) + size_t(tid) * 16;
    const int total = n_rows * pieces, dq = THREADS % pieces, dr = THREADS / pieces;
    int r = tid / pieces, q = tid - r * pieces;
    uint32_t d = dst + uint32_t(tid + r) * 16u;
#pragma unroll 4
    for (int i = tid; i < total; i += THREADS, src += size_t(THREADS) * 16) {
      cp_async16(d, src);
      q += dq;
      const int wrap = q >= pieces ? 1 : 0;
      q -= wrap ? pieces : 0;
      d += uint32_t(THREADS + dr + wrap) * 16u;
    }
    cp_async_commit();
  };
  // weights and segments were complete before the kernel ahead of this one started
  int beg = 0, end = p.M;
  copy_rows(wgt, p.w + (size_t(grp) * p.N + f0) * size_t(p.K / 4), ROWS, p.K / 64);
  if (p.seg) {
    beg = min(max(__ldg(p.seg + grp), 0), p.M);
    end = min(max(__ldg(p.seg + grp + 1), 0), p.M);
  }
  const float alpha = 0.5f * __ldg(p.alpha + size_t(grp) * (p.N / p.alpha_rows) + f0 / p.alpha_rows);   // codes decode to +-2
  __syncwarp();
  pdl_wait();
  pdl_trigger();

#pragma unroll 1
  for (int tb = beg; tb < end; tb += TOK) {
    const int n = min(TOK, end - tb);
    copy_rows(act, p.x + size_t(tb) * p.K, n, p.K / 8);
    int dst[TT][2];                              // output rows of this lane's tokens, -1: not stored
#pragma unroll
    for (int i = 0; i < TT; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int tk = i * 8 + 2 * t + h, row = tb + tk;
        dst[i][h] = tk < n ? row : -1;
        if (p.idx && tk < n) {
          const longlong2 e = *reinterpret_cast<const longlong2*>(p.idx + 2 * row);
          const int2 s = *reinterpret_cast<const int2*>(p.scatter + 2 * row);
          dst[i][h] = e.x == grp ? s.x : (e.y == grp ? s.y : -1);
          if (dst[i][h] >= 2 * p.M) dst[i][h] = -1;
        }
      }
    float acc[TT][4];
#pragma unroll
    for (int i = 0; i < TT; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // rows of the tile past the segment's end hold whatever was there: their columns are never stored
    const uint32_t xa = act + uint32_t(lane & 7) * x_stride + uint32_t(lane >> 3) * 16u;
    const uint32_t wa = wgt + uint32_t(warp * 16 + 2 * g) * w_stride;
    const int s_end = p.K / 16;
    Step<TT> cur, nxt;                           // the next double step's operands are fetched under this one's MMAs
    cur.load(wa, w_stride, xa, x_stride, 0);
#pragma unroll 4
    for (int s = 0; s < s_end; s += 2) {
      nxt.load(wa, w_stride, xa, x_stride, s + 2 < s_end ? s + 2 : s);
      cur.mma(acc, t);
      cur = nxt;
    }
    const int feat = f0 + warp * 16 + 2 * g;
#pragma unroll
    for (int i = 0; i < TT; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (dst[i][h] >= 0) store_pair(p, size_t(dst[i][h]) * p.N + feat, alpha * acc[i][h], alpha * acc[i][2 + h]);
    if (tb + TOK < end) __syncthreads();         // this pass has used its rows
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

constexpr size_t SMEM_MAX = 226 * 1024;
// All codes of a CTA's out-features and the token rows of a tile, each row padded by 16 bytes.
inline size_t smem_need(int tile, int K) { return size_t(16 * ROW_WARPS) * (K / 4 + 16) + size_t(tile) * (size_t(K) * 2 + 16); }

}  // namespace

bool small_gemm_fits(int tile, int K) { return smem_need(tile, K) <= SMEM_MAX; }

int launch_small_gemm(const void* x_bf16, int M, int K, const uint8_t* w_prepared, const float* alpha, int alpha_rows, int N,
                      int G, const int32_t* seg, const int64_t* idx, const int32_t* scatter, int epilogue, void* out,
                      int tile, cudaStream_t stream) {
  JB_REQUIRE(epilogue == JB200_EPI_BF16 || epilogue == JB200_EPI_GELU_BF16 || epilogue == JB200_EPI_RESID_F32, "small_gemm: epilogue %d", epilogue);
  JB_REQUIRE(M >= 1 && K % 128 == 0 && N % 64 == 0 && alpha_rows % 64 == 0, "small_gemm: bad shape (M=%d, N=%d, K=%d)", M, N, K);
  SmallGemmParams p;
  p.x = reinterpret_cast<const __nv_bfloat16*>(x_bf16);
  p.w = w_prepared; p.alpha = alpha; p.seg = seg; p.idx = idx; p.scatter = scatter; p.out = out;
  p.M = M; p.N = N; p.K = K; p.alpha_rows = alpha_rows; p.epilogue = epilogue;
  const size_t smem = smem_need(tile, K);
  JB_REQUIRE(tile == 8 || tile == 16, "small_gemm: tiles of %d tokens", tile);
  JB_REQUIRE(smem <= SMEM_MAX, "small_gemm: in_features (%d) too large", K);
  const dim3 grid(N / (16 * ROW_WARPS), G);
  if (tile == 8) {
    JB_MAX_SMEM(small_gemm_kernel<1>, SMEM_MAX);
    launch_dep(small_gemm_kernel<1>, grid, 32 * ROW_WARPS, smem, stream, p);
  } else {
    JB_MAX_SMEM(small_gemm_kernel<2>, SMEM_MAX);
    launch_dep(small_gemm_kernel<2>, grid, 32 * ROW_WARPS, smem, stream, p);
  }
  JB_LAUNCH_CHECK("small_gemm_kernel");
  return JB200_OK;
}

}  // namespace jb
