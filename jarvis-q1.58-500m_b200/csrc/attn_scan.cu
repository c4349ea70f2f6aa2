// Scalar-decay associative linear-attention causal scan on the 5th-generation tensor cores, fused with its prologue.
//
//   q <- (ELU(q)+1)/sqrt(D),  k <- ELU(k)+1,  half-split RoPE on both   (jarvis_model.py:124-128, :29-71;
//                                                                      fused kernel A1, associative_attention_cuda.cu:28-112)
//   S_t = gamma*S_{t-1} + v_t (x) k_t,   o_t = S_t q_t                  (jarvis_model.py:131-190)
//   optional initial state S_in and final state S_out (B, H, D_v, D_k)  (associative_attention.py:126-152, :273-308;
//                                                                      kernel A3, associative_attention_cuda.cu:218-265)
//
// The reference's chunk-parallel path does the four chunk products as batched library GEMMs over materialised
// per-chunk states (associative_attention.py:242-266).  Here a CTA walks (sequence, head, segment)s in 128-token
// chunks and issues the same four products as tcgen05.mma (bf16 operands from shared
// memory, fp32 accumulators in tensor memory); the state S never leaves the SM (fp32 master copy in registers,
// bf16 copy in shared memory as an MMA operand), so HBM traffic is q, k, v in / o out (512 B per token-head)
// plus one optional state load / store per (sequence, head).  Chunk length is free: the chunked form equals
// the recurrence for any length, only rounding differs.
//
// Per chunk of c <= 128 tokens (i, j: query / key token inside the chunk; g = gamma):
//   TMA (128B-swizzled [128 tokens][64] boxes)                        ->  q, k, v tiles in shared memory
//   feature map + RoPE in place on q and k;  kw[j] = k'[j] * g^(c-1-j)
//   MMA  A:  scores = Q' K'^T       (M=128 i, N=128 j, K=64; both operands K-major)
//            O2     = Q' S^T        (M=128 i, N=64 dv, K=64; S bf16 [dv][dk] is K-major)
//   MMA  S:  dS     = V^T Kw        (M=dv, N=dk, K=128 j; both operands are the [token][64] tiles read
//                                    MN-major; M is padded to 128 by reading the 64 dv twice)
//   P[i][j] = scores * g^(i-j) / 8 for j <= i, else 0                   (TMEM -> registers -> TMEM, bf16)
//   MMA  B:  O1     = P V           (M=128 i, N=64 dv, K=128 j; V read MN-major from its raw tile)
//   S = g^c S + dS (registers; bf16 copy to smem);   o[i] = O1 + g^(i+1)/8 * O2  -> global
// Every wait (TMA arrival, MMA completion) is an mbarrier wait bounded in time.
//
// Sequence segments: when B*H alone cannot fill the GPU (prefill of a few long sequences), T is cut into
// segments.  A first launch (STATE_ONLY) runs only the k/v half of the work for every non-final segment from a
// zero state and stores its contribution D_s; the main launch starts segment s from
// S = fold_{s' < s}(gamma^L S + D_s'), which is exact because the recurrence is linear in S.
// Extra HBM traffic: k and v of the non-final segments are read twice (the second time mostly from L2).
#include <type_traits>

#include "attn_step.cuh"
#include "common.cuh"
#include "launchers.h"

namespace jb {

namespace {

constexpr int D = 64;             // head dim (fixed by the path: 16 heads x 64)
constexpr int CH = 128;           // tokens per chunk = rows of one MMA tile
constexpr int TILE_BYTES = CH * D * 2;          // 16 KiB: [128 tokens][64 bf16], 128B-swizzled
constexpr int S_BYTES = D * D * 2;              // 8 KiB: bf16 state [dv][dk]

struct AttnParams {
  const float* gamma;      // [H] decay in (0,1)
  const float* cos_tab;    // [n_pos][32]
  const float* sin_tab;    // [n_pos][32]
  const int32_t* pos0;     // [B] first position of each sequence, or null (use pos0_scalar)
  int pos0_scalar;
  int n_pos;
  const float* s_in;       // [B][H][64][64] or null
  float* s_out;            // [B][H][64][64] or null
  __nv_bfloat16* o;        // [B*T][ld_o], head h at columns h*64
  int ld_o;
  int B, T, H;
  int seg_chunks;          // chunks per sequence segment (grid.z walks the segments)
  int nseg;
  float* seg_state;        // [B][H][n_pieces][64][64]: state contribution of each piece
  int n_pieces;            // pieces stored per (sequence, head): nseg - 1, or nseg in a state-only call
  int qk_prepared;         // q, k already hold phi(.) + RoPE with the head dim interleaved (d, d+32 adjacent)
  int wide_tab;            // RoPE tables are 32-byte aligned: 256-bit loads
  // Several sequence-heads per CTA (as many CTAs as SMs): with split, equal shares of all chunks, cut wherever they end.  CTAs
  // take tickets from ctrl[0]; the CTA with ticket t leaves the state after its first part of a cut sequence-head in handoff[t],
  // counts its state warps in ctrl[1 + t], and ticket t + 1 goes on from there.
  int split;
  int per_cta, spare;      // sequence-heads, or with split chunks, of every CTA; the first `spare` take one more
  float* handoff;          // [CTAs][64][64] f32
  int* ctrl;               // [1 + CTAs], zeroed before the launch
  unsigned int* status;
  int settled;             // decays, angles and positions (single-token step: the state too) were complete before the kernel ahead of this one started
};

__device__ __forceinline__ uint32_t swz(int row, int chunk16) {  // byte offset inside a swizzled [rows][128 B] tile
  return uint32_t(row) * 128u + (uint32_t(chunk16 ^ (row & 7)) << 4);
}

// Shared-memory matrix descriptor, 128-byte swizzle.  K-major operands (rows of 64 K-elements): lbo is unused
// (16), sbo = 1024 is the distance between 8-row groups.  MN-major operands (a [K rows][64 MN-elements] tile):
// sbo = 1024 is the distance between groups of 8 K rows, lbo the distance between blocks of 64 MN-elements.
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16;
  d |= static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}
// kind::f16 instruction descriptor: bf16 operands, fp32 accumulator; a_mn / b_mn = 1 reads that operand MN-major.
__host__ __device__ constexpr uint32_t umma_idesc(int m, int n, int a_mn, int b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(a_mn) << 15) | (uint32_t(b_mn) << 16) |
         (uint32_t(n >> 3) << 17) | (uint32_t(m >> 4) << 24);
}

__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// Eight angles of a row of a RoPE table: 32 bytes at a 32-byte step from the table's start, in one load where that is aligned.
__device__ __forceinline__ void load_angles8(const float* src, bool wide, float (&a)[8]) {
  if (wide) {
    asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a[0]), "=f"(a[1]), "=f"(a[2]), "=f"(a[3]), "=f"(a[4]), "=f"(a[5]), "=f"(a[6]), "=f"(a[7])
        : "l"(src));
  } else {
    const float4 lo = __ldg(reinterpret_cast<const float4*>(src)), hi = __ldg(reinterpret_cast<const float4*>(src) + 1);
    a[0] = lo.x; a[1] = lo.y; a[2] = lo.z; a[3] = lo.w; a[4] = hi.x; a[5] = hi.y; a[6] = hi.z; a[7] = hi.w;
  }
}

// ------------------------------------------------------------------------------------------------------------
// k/v-only pass: the state contribution of one piece of a sequence from a zero state (pieces = the non-final
// segments of a full call, or all pieces of a state-only call).  One CTA per (sequence, head, piece), 256 threads,
// two CTAs per SM.  Per chunk: TMA k, v (two stages) -> kw = phi(k) with RoPE, times gamma^(c-1-j) ->
// dS = V^T Kw as tcgen05.mma (accumulator in TMEM) -> S = gamma^c S + dS in registers.  The feature map, the
// angles and the rounding of kw are instruction for instruction those of the pipeline kernel's prologue, so a
// segmented call and an unsegmented one see the same bf16 operands.
// ------------------------------------------------------------------------------------------------------------
constexpr int STATE_THREADS = 256;
constexpr uint32_t STATE_TMEM_COLS = 64;

struct StateSmem {
  uint8_t k[2][TILE_BYTES];
  uint8_t v[2][TILE_BYTES];
  uint8_t kw[TILE_BYTES];
  float pw[CH + 1];            // gamma^n
  uint64_t full[2], bar_s;
  uint32_t tmem_base;
  uint32_t abort_flag;
};
constexpr size_t STATE_SMEM_BYTES = sizeof(StateSmem) + 1024;

__global__ void __launch_bounds__(STATE_THREADS, 2)
attn_state_pass_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                       const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  StateSmem* sm = reinterpret_cast<StateSmem*>(smem_raw + (base - raw_addr));

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int qd = warp & 3;          // TMEM lane quarter this warp may access
  const int hf = warp >> 2;
  const int h = blockIdx.x, b = blockIdx.y, seg = blockIdx.z;
  const int T = p.T;
  const int n_chunks = (T + CH - 1) / CH;
  const int ck_begin = seg * p.seg_chunks;
  const int ck_end = min(n_chunks, ck_begin + p.seg_chunks);
  const int row0 = b * T;

  if (tid == 0) {
    mbar_init(smem_u32(&sm->full[0]), 1);
    mbar_init(smem_u32(&sm->full[1]), 1);
    mbar_init(smem_u32(&sm->bar_s), 1);
    sm->abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  if (warp == 0) {
    __syncwarp();                 // tcgen05.alloc is warp-collective: lane 0 rejoins from the barrier set-up first
    tmem_alloc(smem_u32(&sm->tmem_base), STATE_TMEM_COLS);
    tmem_relinquish();
  }
  // What the kernel before this one did not make (`settled`) is read while it runs, and the first tiles are asked for as soon as
  // they are there (behind the decay table they came 1.3 us later).
  const int cg = tid & 3;
  float c64[8], s64[8];
  int pos_base = 0;
  auto tables = [&] {
    pos_base = p.pos0 ? p.pos0[b] : p.pos0_scalar;
    const float log_g = logf(__ldg(p.gamma + h));
    for (int n = tid; n <= CH; n += STATE_THREADS) sm->pw[n] = expf(log_g * float(n));
    const int stp = 64 < p.n_pos ? 64 : p.n_pos - 1;
    const float4* cq = reinterpret_cast<const float4*>(p.cos_tab + size_t(stp) * 32 + cg * 8);
    const float4* sq = reinterpret_cast<const float4*>(p.sin_tab + size_t(stp) * 32 + cg * 8);
    const float4 d0 = __ldg(cq), d1 = __ldg(cq + 1), e0 = __ldg(sq), e1 = __ldg(sq + 1);
    c64[0] = d0.x; c64[1] = d0.y; c64[2] = d0.z; c64[3] = d0.w; c64[4] = d1.x; c64[5] = d1.y; c64[6] = d1.z; c64[7] = d1.w;
    s64[0] = e0.x; s64[1] = e0.y; s64[2] = e0.z; s64[3] = e0.w; s64[4] = e1.x; s64[5] = e1.y; s64[6] = e1.z; s64[7] = e1.w;
  };
  auto issue = [&](int ck) {      // thread 0 only
    const int st = (ck - ck_begin) & 1;
    const uint32_t bar = smem_u32(&sm->full[st]);
    mbar_arrive_expect_tx(bar, 2 * TILE_BYTES);
    tma_load_2d(smem_u32(sm->k[st]), &tm_k, h * D, row0 + ck * CH, bar);
    tma_load_2d(smem_u32(sm->v[st]), &tm_v, h * D, row0 + ck * CH, bar);
  };
  if (p.settled) tables();
  __syncwarp();
  pdl_wait();
  pdl_trigger();
  if (tid == 0) {
    for (int ck = ck_begin; ck < ck_begin + 2 && ck < ck_end; ++ck) issue(ck);
  }
  if (!p.settled) tables();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = sm->tmem_base;
  const uint32_t tm_lane = tm + (uint32_t(32 * qd) << 16);

  // the thread's share of the state: row dv = 32*(qd&1) + lane, columns 16*cg .. 16*cg+15 (see the pipeline kernel)
  const int s_row = 32 * (qd & 1) + lane;
  const int s_cg = 2 * (qd >> 1) + hf;
  float S[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) S[e] = 0.f;

  const int r_lo = (tid >> 5) * 8 + ((tid >> 2) & 1) * 4 + ((tid >> 3) & 3);

  bool ok = true;
  for (int ck = ck_begin; ck < ck_end; ++ck) {
    const int lc = ck - ck_begin;
    const int st = lc & 1;
    const int c_len = min(CH, T - ck * CH);
    const uint8_t* k_p = sm->k[st];
    float cs[8], sn[8];
    if (!p.qk_prepared) {         // angles of the thread's first row (in flight during the wait below)
      int pos = pos_base + ck * CH + r_lo;
      pos = pos < 0 ? 0 : (pos >= p.n_pos ? p.n_pos - 1 : pos);
      const float4* cp = reinterpret_cast<const float4*>(p.cos_tab + size_t(pos) * 32 + cg * 8);
      const float4* sp = reinterpret_cast<const float4*>(p.sin_tab + size_t(pos) * 32 + cg * 8);
      const float4 a0 = __ldg(cp), a1 = __ldg(cp + 1), b0 = __ldg(sp), b1 = __ldg(sp + 1);
      cs[0] = a0.x; cs[1] = a0.y; cs[2] = a0.z; cs[3] = a0.w; cs[4] = a1.x; cs[5] = a1.y; cs[6] = a1.z; cs[7] = a1.w;
      sn[0] = b0.x; sn[1] = b0.y; sn[2] = b0.z; sn[3] = b0.w; sn[4] = b1.x; sn[5] = b1.y; sn[6] = b1.z; sn[7] = b1.w;
    }
    if (!mbar_wait(smem_u32(&sm->full[st]), uint32_t(lc >> 1) & 1u, &sm->abort_flag, p.status, JB200_STATUS_ATTN_LOAD)) ok = false;
    if (ok) {
#pragma unroll
      for (int it = 0; it < 2; ++it) {
        const int r = r_lo + 64 * it;
        const float w = r < c_len ? sm->pw[c_len - 1 - r] : 0.f;   // rows past the end contribute nothing
        const uint4 lo = *reinterpret_cast<const uint4*>(k_p + swz(r, cg));
        const uint4 hi = *reinterpret_cast<const uint4*>(k_p + swz(r, cg + 4));
        const uint32_t lw[4] = {lo.x, lo.y, lo.z, lo.w}, hw[4] = {hi.x, hi.y, hi.z, hi.w};
        uint32_t wl[4], wh[4];
        if (p.qk_prepared) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            wl[j] = pack_bf16x2(bf16_lo(lw[j]) * w, bf16_hi(lw[j]) * w);
            wh[j] = pack_bf16x2(bf16_lo(hw[j]) * w, bf16_hi(hw[j]) * w);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float a0 = elu1(bf16_lo(lw[j])), a1 = elu1(bf16_hi(lw[j]));   // d
            const float b0 = elu1(bf16_lo(hw[j])), b1 = elu1(bf16_hi(hw[j]));   // d + 32
            const float l0 = a0 * cs[2 * j] - b0 * sn[2 * j], l1 = a1 * cs[2 * j + 1] - b1 * sn[2 * j + 1];
            const float h0 = b0 * cs[2 * j] + a0 * sn[2 * j], h1 = b1 * cs[2 * j + 1] + a1 * sn[2 * j + 1];
            wl[j] = pack_bf16x2(l0 * w, l1 * w);
            wh[j] = pack_bf16x2(h0 * w, h1 * w);
          }
          if (it == 0) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float cn = cs[e] * c64[e] - sn[e] * s64[e];
              sn[e] = sn[e] * c64[e] + cs[e] * s64[e];
              cs[e] = cn;
            }
          }
        }
        *reinterpret_cast<uint4*>(sm->kw + swz(r, cg)) = make_uint4(wl[0], wl[1], wl[2], wl[3]);
        *reinterpret_cast<uint4*>(sm->kw + swz(r, cg + 4)) = make_uint4(wh[0], wh[1], wh[2], wh[3]);
      }
    }
    fence_proxy_async_smem();   // kw -> visible to the tensor core; orders the reads of k before the next TMA write
    tc_fence_before_sync();
    if (__syncthreads_or(!ok)) { ok = false; break; }
    tc_fence_after_sync();
    if (tid == 0) {
      constexpr uint32_t id_ds = umma_idesc(128, 64, 1, 1);
      const uint32_t v_a = smem_u32(sm->v[st]), kw_a = smem_u32(sm->kw);
#pragma unroll
      for (int ks = 0; ks < 8; ++ks)
        umma_bf16_ss(tm, umma_desc(v_a + ks * 2048, 0, 1024), umma_desc(kw_a + ks * 2048, 1024, 1024), id_ds, ks != 0);
      umma_commit(smem_u32(&sm->bar_s));
    }
    if (!mbar_wait(smem_u32(&sm->bar_s), uint32_t(lc) & 1u, &sm->abort_flag, p.status, JB200_STATUS_ATTN_MMA)) ok = false;
    tc_fence_after_sync();
    if (tid == 0 && ok && ck + 2 < ck_end) issue(ck + 2);     // this chunk's k and v buffers are free again
    __syncwarp();
    if (ok) {
      uint32_t r[16];
      tmem_ld_32x16(tm_lane + 16 * s_cg, r);
      tmem_ld_wait();
      const float gc = sm->pw[c_len];
#pragma unroll
      for (int e = 0; e < 16; ++e) S[e] = gc * S[e] + __uint_as_float(r[e]);
    }
  }

  if (ok) {       // pieces stay in the kernel's own column order (interleaved when q/k were prepared)
    float* sp = p.seg_state + ((size_t(b) * p.H + h) * p.n_pieces + seg) * D * D + s_row * D + 16 * s_cg;
#pragma unroll
    for (int e4 = 0; e4 < 4; ++e4)
      *reinterpret_cast<float4*>(sp + 4 * e4) = make_float4(S[4 * e4], S[4 * e4 + 1], S[4 * e4 + 2], S[4 * e4 + 3]);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tm, STATE_TMEM_COLS);
  }
}

// ------------------------------------------------------------------------------------------------------------
// The full pass as a warp-specialised pipeline: one CTA per SM, 24 warps, several chunks in flight.
//   warp 0       TMA producer: q, k, v tiles of a chunk as soon as the MMAs that read its stage have retired
//   warp 1       MMA issuer, per chunk c:  A1(c) scores = Q' K'^T -> TMEM SC[c%2];  S(c) dS = V^T Kw -> TMEM DS[c%2];
//                A2(c) O2 = Q' S^T -> TMEM O2[c%2] (needs the state before chunk c in smem)
//   warp 2       MMA issuer, B(c): O1 = P V -> TMEM SC[c%2] columns 0-63 (needs P of c), on its own so that it never
//                waits behind the next chunk's prologue
//   warp 3       idle (registers are handed out to groups of four warps)
//   warps 4-11   prologue: feature map + RoPE in place on q and k of a stage, kw = k' * gamma^(c-1-j)
//   warps 12-15  state: S = gamma^c S + dS in registers, its bf16 copy in smem; decay tables of the heads to come
//   warps 16-19, 20-23  consumers of the even and of the odd chunks: decay mask scores -> P, output rows (by TMA through the v
//                tile of the chunk, which P V was the last to read)
// What bounds it now: the prologue, 3700 of the ~4100 cycles of a chunk (two warps per scheduler; sixteen warps, or more registers,
// were 3 to 8 % slower, its two rows unrolled 20 %: the roles' loops share the instruction caches, at 67 KB of code a chunk took 5000
// cycles when all SMs ran and 3700 on one alone).  With one group of consumers (eight warps, half the columns each) for every
// chunk the period was the serial chain scores -> mask -> P V -> output rows, 5500 cycles.  Two groups of four warps overlap the chains of
// two chunks, the state has warps of its own, one lane of a warp arrives on a barrier (256 arrivals took 300-400 cycles, four a chunk), a
// CTA walks several sequence-heads without draining (filling and draining took ~12 us each), output rows go by TMA (stored
// directly they took 512 of 3000 wavefronts of a chunk), angles come 32 bytes a load.  B x T of 16 heads, before -> after: 32 x 2048 158 -> 125 us,
// 32 x 512 55.5 -> 43, 8 x 2048 43.1 -> 36.6, 32 x 64 24.3 -> 15.5, 1 x 16384 in segments 77 -> 71, 1 x 37 and 1 x 128 5.9 -> 6.2 and
// 6.4 -> 6.8 (the chain of a lone chunk); up to nine sequences of one or two chunks 0.2 to 0.5 us more, with a carried state 1.1 to 1.7 less
// (1 x 37 7.9 -> 6.7, 9 x 200 11.0 -> 9.7).
// P (bf16 pairs, 64 columns) overlays score columns 64-127: a warp owns its lanes, and walks the 16-key blocks downwards, so
// what it overwrites it has read.
// ------------------------------------------------------------------------------------------------------------
constexpr int PRO_WARP0 = 4, STATE_WARP0 = 12, CON_WARP0 = 16, PIPE_THREADS = 24 * 32;
constexpr int PRO_WARPS = 8, STATE_WARPS = 4, CON_WARPS = 4;  // consumers: of each group
// Registers a thread: the CTA is launched with 80 for each of its six groups of four warps; the issuers give up what the
// others take.
constexpr int LAUNCH_REGS = 80, ISSUE_REGS = 48, PRO_REGS = 88, STATE_REGS = 80, CON_REGS = 88;
static_assert(ISSUE_REGS + 2 * PRO_REGS + STATE_REGS + 2 * CON_REGS <= 6 * LAUNCH_REGS, "no more registers than the CTA was launched with");
template <int N> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
constexpr int NST = 3;                                       // stages of the q / k / kw / v tiles
constexpr uint32_t PIPE_TMEM_COLS = 512;
constexpr uint32_t PT_SC = 0, PT_O2 = 256, PT_DS = 384;      // SC[2] x 128, O2[2] x 64, DS[2] x 64
constexpr uint32_t PT_P = 64;                                // P inside SC

// Powers of a head's decay.  NTAB: the state warps fill the tables of the sequence-head after next while the consumers
// may still be two chunks, so at most two sequence-heads, behind.
struct DecayTab {
  float pwm[2 * CH];           // pwm[x + CH] = gamma^x / 8 for x >= 0, 0 for x < 0: the decay mask by (i - j)
  float pw[CH + 4];            // gamma^n, n <= CH
};
constexpr int NTAB = 6;

struct PipeSmem {
  uint8_t q[NST][TILE_BYTES];
  uint8_t k[NST][TILE_BYTES];
  uint8_t kw[NST][TILE_BYTES];
  uint8_t v[NST][TILE_BYTES];
  uint8_t s[2][S_BYTES];       // bf16 state copy, [c & 1] = state before chunk c of this CTA
  DecayTab tab[NTAB];
  uint64_t full_qk[NST], full_v[NST], empty_qk[NST], empty_v[NST], pro_done[NST];
  uint64_t bar_sc[2], bar_s[2], bar_o2[2], bar_b[2], s_done[2], p_done[2], o_done[2];
  uint64_t tab_full[NTAB];
  uint32_t tmem_base;
  uint32_t abort_flag;
  int ticket;
};
constexpr size_t PIPE_SMEM_BYTES = sizeof(PipeSmem) + 1024;
static_assert(PIPE_SMEM_BYTES <= 227 * 1024, "shared memory of a CTA");

__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

// The sequence-heads of a CTA, and of those that are not whole the chunks.  One segment of one sequence-head where sequences
// are cut into segments; else a share of all chunks in order of (sequence, head, chunk): from chunk c0 of unit u0 to before
// chunk c1 of unit u1.  The first part of the last unit is scanned first and the second part of the first unit last: a second
// part needs the state that the CTA before this one leaves behind its first item.
struct Item {
  int unit, begin, end;
  int piece;                   // 0 a whole sequence-head or a segment, 1 a first part (leaves its end state in handoff), 2 a second part
};
struct Share {
  int u0, c0, u1, c1, begin, end, n_items, n_chunks;
  __device__ __forceinline__ Share(const AttnParams& p, int cta, int n_chunks_) : n_chunks(n_chunks_) {
    begin = 0;
    end = n_chunks;
    c0 = c1 = 0;
    const int U = p.B * p.H;
    if (p.nseg > 1) {
      const int seg = cta / U;
      u0 = cta - seg * U;
      u1 = u0 + 1;
      begin = seg * p.seg_chunks;
      end = min(n_chunks, begin + p.seg_chunks);
    } else {
      const int a = cta * p.per_cta + min(cta, p.spare), e = a + p.per_cta + (cta < p.spare);
      u0 = a;
      u1 = e;
      if (p.split) {
        u0 = a / n_chunks;
        c0 = a - u0 * n_chunks;
        u1 = e / n_chunks;
        c1 = e - u1 * n_chunks;
      }
    }
    n_items = u1 - u0 + (c1 > 0);
  }
  __device__ __forceinline__ int chunks() const { return (u1 - u0) * (end - begin) - c0 + c1; }
  __device__ __forceinline__ Item at(int k) const {
    const int first = c1 > 0, whole = c0 > 0;
    if (k < first) return {u1, 0, c1, 1};
    if (whole && k == n_items - 1) return {u0, c0, n_chunks, 2};
    return {u0 + whole + k - first, begin, end, 0};
  }
};

__device__ __forceinline__ void fill_tab(DecayTab& t, float log_g, int tid, int threads) {
  for (int n = tid; n <= CH; n += threads) t.pw[n] = expf(log_g * float(n));
  for (int n = tid; n < 2 * CH; n += threads) {
    // gamma^(i-j) / sqrt(D): the 1/8 of the query feature map is a power of two, so applying it to the scores
    // (and to the cross-chunk factor) instead of to every element of q gives the same bits
    const int x = n - CH;
    t.pwm[n] = x >= 0 ? 0.125f * expf(log_g * float(x)) : 0.f;
  }
}

template <bool PREPARED>
__global__ void __launch_bounds__(PIPE_THREADS, 1)
attn_scan_pipe_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                      const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o, const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  PipeSmem* sm = reinterpret_cast<PipeSmem*>(smem_raw + (base - raw_addr));

  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int T = p.T;
  const int n_chunks = (T + CH - 1) / CH;

  if (tid == 0) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(smem_u32(&sm->full_qk[s]), 1);
      mbar_init(smem_u32(&sm->full_v[s]), 1);
      mbar_init(smem_u32(&sm->empty_qk[s]), 1);
      mbar_init(smem_u32(&sm->empty_v[s]), CON_WARPS);
      mbar_init(smem_u32(&sm->pro_done[s]), PRO_WARPS);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&sm->bar_sc[s]), 1);
      mbar_init(smem_u32(&sm->bar_s[s]), 1);
      mbar_init(smem_u32(&sm->bar_o2[s]), 1);
      mbar_init(smem_u32(&sm->bar_b[s]), 1);
      mbar_init(smem_u32(&sm->s_done[s]), STATE_WARPS);
      mbar_init(smem_u32(&sm->p_done[s]), CON_WARPS);
      mbar_init(smem_u32(&sm->o_done[s]), CON_WARPS);
    }
    for (int s = 0; s < NTAB; ++s) mbar_init(smem_u32(&sm->tab_full[s]), STATE_WARPS);
    sm->abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
    tma_prefetch_desc(&tm_o);
  }
  if (warp == 0) {
    __syncwarp();                 // tcgen05.alloc is warp-collective: lane 0 rejoins from the barrier set-up first
    tmem_alloc(smem_u32(&sm->tmem_base), PIPE_TMEM_COLS);
    tmem_relinquish();
  }
  // `settled`: the decay tables too are made while the kernel before this one runs, unless the head is not known before the
  // ticket is.
  const bool tables_first = p.settled && !p.split;
  if (!tables_first) {
    pdl_wait();
    pdl_trigger();
  }
  int cta = blockIdx.x;
  if (p.split) {
    // a ticket instead of the block index: whoever holds a second part started after the first part was taken
    if (tid == 0) sm->ticket = atomicAdd(p.ctrl, 1);
    __syncthreads();
    cta = sm->ticket;
  }
  const Share share(p, cta, n_chunks);
  fill_tab(sm->tab[0], logf(__ldg(p.gamma + share.at(0).unit % p.H)), tid, PIPE_THREADS);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = sm->tmem_base;
  volatile uint32_t* abort_flag = &sm->abort_flag;
  // Then the roles that read what it made (tiles; states of segments) wait for it; angles are on their way before, and rows leave
  // behind the tiles they come from.

  // Chunks are counted over all items (g): stages, accumulators and barrier phases follow that count.
  if (warp < PRO_WARP0) {
    regs_dec<ISSUE_REGS>();
    if (warp == 0) {
      // ---------------- TMA producer ----------------
      if (tables_first) {
        pdl_wait();
        pdl_trigger();
      }
      int s = 0, g = 0;
      uint32_t prev = 1u;                         // parity of the PREVIOUS use of the stage
      bool ok = true;
      for (int k = 0; ok && k < share.n_items; ++k) {
        const Item it = share.at(k);
        const int b = it.unit / p.H, col = (it.unit - b * p.H) * D;
        for (int ck = it.begin; ck < it.end; ++ck, ++g) {
          const int r = b * T + ck * CH;
          if (g >= NST && !mbar_wait(smem_u32(&sm->empty_qk[s]), prev, abort_flag, p.status, JB200_STATUS_ATTN_LOAD)) { ok = false; break; }
          if (elect_one()) {
            mbar_arrive_expect_tx(smem_u32(&sm->full_qk[s]), 2 * TILE_BYTES);
            tma_load_2d(smem_u32(sm->k[s]), &tm_k, col, r, smem_u32(&sm->full_qk[s]));
            tma_load_2d(smem_u32(sm->q[s]), &tm_q, col, r, smem_u32(&sm->full_qk[s]));
          }
          __syncwarp();
          if (g >= NST && !mbar_wait(smem_u32(&sm->empty_v[s]), prev, abort_flag, p.status, JB200_STATUS_ATTN_LOAD)) { ok = false; break; }
          if (elect_one()) {
            mbar_arrive_expect_tx(smem_u32(&sm->full_v[s]), TILE_BYTES);
            tma_load_2d(smem_u32(sm->v[s]), &tm_v, col, r, smem_u32(&sm->full_v[s]));
          }
          __syncwarp();
          if (++s == NST) { s = 0; prev ^= 1u; }
        }
      }
    } else if (warp == 1) {
      // ---------------- MMA issuer: scores, dS, O2 ----------------
      constexpr uint32_t id_sc = umma_idesc(128, 128, 0, 0), id_o2 = umma_idesc(128, 64, 0, 0), id_ds = umma_idesc(128, 64, 1, 1);
      // Operand descriptors of stage 0; stage s is +s*TILE_BYTES (+1024 in the address field).  A K-step of 16
      // elements is +32 bytes (+2) inside a K-major row, +2048 bytes (+128: two 8-row groups) in the MN-major
      // [token][64] tiles.
      constexpr uint64_t STG = TILE_BYTES >> 4;
      const uint64_t d_q0 = umma_desc(smem_u32(sm->q[0]), 16, 1024), d_k0 = umma_desc(smem_u32(sm->k[0]), 16, 1024);
      const uint64_t d_kw0 = umma_desc(smem_u32(sm->kw[0]), 1024, 1024);
      const uint64_t d_v0 = umma_desc(smem_u32(sm->v[0]), 0, 1024);       // as the M operand of dS: the 64 dv read twice
      const uint64_t d_s0 = umma_desc(smem_u32(sm->s[0]), 16, 1024);
      const int n_tot = share.chunks();
      int s = 0;                                   // stage of chunk g
      uint32_t sp = 0u;                            // parity of this use of the stage
      for (int g = 0; g < n_tot; ++g) {
        const int buf = g & 1;                     // accumulators and the state copy alternate
        const uint32_t u = uint32_t(g >> 1) & 1u;
        const uint64_t dq = d_q0 + uint64_t(s) * STG, dk = d_k0 + uint64_t(s) * STG, dkw = d_kw0 + uint64_t(s) * STG;
        const uint64_t dv = d_v0 + uint64_t(s) * STG, ds = d_s0 + uint64_t(buf) * (S_BYTES >> 4);
        if (!mbar_wait(smem_u32(&sm->pro_done[s]), sp, abort_flag, p.status, JB200_STATUS_ATTN_MMA)) break;
        // the output rows of chunk g - 2 have left SC[buf] and O2[buf]
        if (g >= 2 && !mbar_wait(smem_u32(&sm->o_done[buf]), u ^ 1u, abort_flag, p.status, JB200_STATUS_ATTN_MMA)) break;
        tc_fence_after_sync();
        if (elect_one()) {
  #pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma_bf16_ss(tm + PT_SC + 128 * buf, dq + uint64_t(ks * 2), dk + uint64_t(ks * 2), id_sc, ks != 0);
          umma_commit(smem_u32(&sm->bar_sc[buf]));
        }
        __syncwarp();
        if (!mbar_wait(smem_u32(&sm->full_v[s]), sp, abort_flag, p.status, JB200_STATUS_ATTN_LOAD)) break;
        // DS[buf] was read before the state before chunk g - 1 was published, which A2(g - 1) waited for
        if (elect_one()) {
  #pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            umma_bf16_ss(tm + PT_DS + 64 * buf, dv + uint64_t(ks * 128), dkw + uint64_t(ks * 128), id_ds, ks != 0);
          umma_commit(smem_u32(&sm->bar_s[buf]));
        }
        __syncwarp();
        if (!mbar_wait(smem_u32(&sm->s_done[buf]), u, abort_flag, p.status, JB200_STATUS_ATTN_MMA)) break;
        tc_fence_after_sync();
        if (elect_one()) {
  #pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma_bf16_ss(tm + PT_O2 + 64 * buf, dq + uint64_t(ks * 2), ds + uint64_t(ks * 2), id_o2, ks != 0);
          umma_commit(smem_u32(&sm->bar_o2[buf]));
          umma_commit(smem_u32(&sm->empty_qk[s]));       // q, k, kw of this stage, and v but for B(g)
        }
        __syncwarp();
        if (++s == NST) { s = 0; sp ^= 1u; }
      }
    } else if (warp == 2) {
      // ---------------- MMA issuer: O1 = P V into the score columns the mask has read; P is read from TMEM ----------------
      constexpr uint32_t id_o1 = umma_idesc(128, 64, 0, 1);
      const uint64_t d_v0 = umma_desc(smem_u32(sm->v[0]), 1024, 1024);    // as the N operand
      const int n_tot = share.chunks();
      int s = 0;
      uint32_t sp = 0u;
      for (int g = 0; g < n_tot; ++g) {
        const int buf = g & 1;
        const uint64_t dv = d_v0 + uint64_t(s) * (TILE_BYTES >> 4);
        if (!mbar_wait(smem_u32(&sm->full_v[s]), sp, abort_flag, p.status, JB200_STATUS_ATTN_LOAD)) break;
        if (!mbar_wait(smem_u32(&sm->p_done[buf]), uint32_t(g >> 1) & 1u, abort_flag, p.status, JB200_STATUS_ATTN_MMA)) break;
        if (n_tot == 1 && !mbar_wait(smem_u32(&sm->p_done[1]), 0u, abort_flag, p.status, JB200_STATUS_ATTN_MMA)) break;
        tc_fence_after_sync();
        const uint32_t tm_p = tm + PT_SC + PT_P + (n_tot == 1 ? 128 : 128 * buf);
        if (elect_one()) {
  #pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            umma_bf16_ts(tm + PT_SC + 128 * buf, tm_p + ks * 8, dv + uint64_t(ks * 128), id_o1, ks != 0);
          umma_commit(smem_u32(&sm->bar_b[buf]));
        }
        __syncwarp();
        if (++s == NST) { s = 0; sp ^= 1u; }
      }
    }
  } else if (warp < STATE_WARP0) {
    regs_inc<PRO_REGS>();
    // ---------------- prologue warps ----------------
    const int ptid = tid - PRO_WARP0 * 32;
    // 128 rows x 4 column groups of 8 rotary pairs = 512 items per chunk, two per thread: (row r, group cg) and
    // (row r + 64, group cg).  Eight consecutive lanes take 4 groups of two rows that are 4 apart, so that their
    // 16-byte accesses to the swizzled tiles fall into different banks.
    const int cg = ptid & 3;
    const int r_lo = (ptid >> 5) * 8 + ((ptid >> 2) & 1) * 4 + ((ptid >> 3) & 3);
    // RoPE angles: the thread's 8 frequencies are fixed.  The angles of its first row come from the table (the
    // loads for the NEXT chunk are issued when a chunk is finished, so their latency passes during the wait for
    // that chunk's tiles); its second row is 64 positions further, one fixed rotation by (cos, sin)(64 theta_i)
    // away (angle addition in f32: error ~1e-7 against the 4e-3 of the bf16 result).  Every chunk starts from
    // the table again, so results do not depend on how a sequence is cut into segments or calls.
    float cs[8], sn[8], c64[8], s64[8];
    auto load_angles = [&](int unit, int ck) {
      int pos = (p.pos0 ? p.pos0[unit / p.H] : p.pos0_scalar) + ck * CH + r_lo;
      pos = pos < 0 ? 0 : (pos >= p.n_pos ? p.n_pos - 1 : pos);
      load_angles8(p.cos_tab + size_t(pos) * 32 + cg * 8, p.wide_tab, cs);
      load_angles8(p.sin_tab + size_t(pos) * 32 + cg * 8, p.wide_tab, sn);
    };
    {
      const int stp = 64 < p.n_pos ? 64 : p.n_pos - 1;     // tables shorter than 65 rows: rows >= 64 are past the end anyway
      load_angles8(p.cos_tab + size_t(stp) * 32 + cg * 8, p.wide_tab, c64);
      load_angles8(p.sin_tab + size_t(stp) * 32 + cg * 8, p.wide_tab, s64);
    }
    int s = 0;
    uint32_t sp = 0u;
    bool ok = true;
    for (int k = 0; ok && k < share.n_items; ++k) {
      const Item itm = share.at(k);
      const float* pw = sm->tab[k % NTAB].pw;
      if (k == 0 && !PREPARED) load_angles(itm.unit, itm.begin);
      if (k > 0 && !mbar_wait(smem_u32(&sm->tab_full[k % NTAB]), uint32_t(k / NTAB) & 1u, abort_flag, p.status, JB200_STATUS_ATTN_LOAD)) break;
      for (int ck = itm.begin; ck < itm.end; ++ck) {
        const int c_len = min(CH, T - ck * CH);
        uint8_t* q_p = sm->q[s];
        uint8_t* k_p = sm->k[s];
        uint8_t* kw_p = sm->kw[s];
        if (!mbar_wait(smem_u32(&sm->full_qk[s]), sp, abort_flag, p.status, JB200_STATUS_ATTN_LOAD)) { ok = false; break; }
#pragma unroll 1
        for (int it = 0; it < 2; ++it) {
          const int r = r_lo + 64 * it;
          const float w = r < c_len ? pw[c_len - 1 - r] : 0.f;   // rows past the end contribute nothing
          if (PREPARED) {
            // q', k' came out of the projection's epilogue: only the decay-weighted copy of k is made here
            const uint4 lo = *reinterpret_cast<const uint4*>(k_p + swz(r, cg));
            const uint4 hi = *reinterpret_cast<const uint4*>(k_p + swz(r, cg + 4));
            *reinterpret_cast<uint4*>(kw_p + swz(r, cg)) =
                make_uint4(pack_bf16x2(bf16_lo(lo.x) * w, bf16_hi(lo.x) * w), pack_bf16x2(bf16_lo(lo.y) * w, bf16_hi(lo.y) * w),
                           pack_bf16x2(bf16_lo(lo.z) * w, bf16_hi(lo.z) * w), pack_bf16x2(bf16_lo(lo.w) * w, bf16_hi(lo.w) * w));
            *reinterpret_cast<uint4*>(kw_p + swz(r, cg + 4)) =
                make_uint4(pack_bf16x2(bf16_lo(hi.x) * w, bf16_hi(hi.x) * w), pack_bf16x2(bf16_lo(hi.y) * w, bf16_hi(hi.y) * w),
                           pack_bf16x2(bf16_lo(hi.z) * w, bf16_hi(hi.z) * w), pack_bf16x2(bf16_lo(hi.w) * w, bf16_hi(hi.w) * w));
            continue;
          }
          // all four 16-byte pieces of the row pair first, so that their latencies overlap
          uint4* ql_p = reinterpret_cast<uint4*>(q_p + swz(r, cg));
          uint4* qh_p = reinterpret_cast<uint4*>(q_p + swz(r, cg + 4));
          uint4* kl_p = reinterpret_cast<uint4*>(k_p + swz(r, cg));
          uint4* kh_p = reinterpret_cast<uint4*>(k_p + swz(r, cg + 4));
          const uint4 ql = *ql_p, qh = *qh_p, kl = *kl_p, kh = *kh_p;
#pragma unroll
          for (int which = 0; which < 2; ++which) {  // 0: q, 1: k
            const uint4 lo = which == 0 ? ql : kl, hi = which == 0 ? qh : kh;
            const uint32_t lw[4] = {lo.x, lo.y, lo.z, lo.w}, hw[4] = {hi.x, hi.y, hi.z, hi.w};
            uint32_t ol[4], oh[4], wl[4], wh[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float a0 = elu1(bf16_lo(lw[j])), a1 = elu1(bf16_hi(lw[j]));   // d
              const float b0 = elu1(bf16_lo(hw[j])), b1 = elu1(bf16_hi(hw[j]));   // d + 32
              // x*cos + rotate_half(x)*sin:  out[d] = x[d]cos - x[d+32]sin,  out[d+32] = x[d+32]cos + x[d]sin
              const float l0 = a0 * cs[2 * j] - b0 * sn[2 * j], l1 = a1 * cs[2 * j + 1] - b1 * sn[2 * j + 1];
              const float h0 = b0 * cs[2 * j] + a0 * sn[2 * j], h1 = b1 * cs[2 * j + 1] + a1 * sn[2 * j + 1];
              ol[j] = pack_bf16x2(l0, l1);
              oh[j] = pack_bf16x2(h0, h1);
              if (which == 1) {
                wl[j] = pack_bf16x2(l0 * w, l1 * w);
                wh[j] = pack_bf16x2(h0 * w, h1 * w);
              }
            }
            *(which == 0 ? ql_p : kl_p) = make_uint4(ol[0], ol[1], ol[2], ol[3]);
            *(which == 0 ? qh_p : kh_p) = make_uint4(oh[0], oh[1], oh[2], oh[3]);
            if (which == 1) {
              *reinterpret_cast<uint4*>(kw_p + swz(r, cg)) = make_uint4(wl[0], wl[1], wl[2], wl[3]);
              *reinterpret_cast<uint4*>(kw_p + swz(r, cg + 4)) = make_uint4(wh[0], wh[1], wh[2], wh[3]);
            }
          }
          if (it == 0) {             // advance the angles by 64 positions: to the thread's second row
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float cn = cs[e] * c64[e] - sn[e] * s64[e];
              sn[e] = sn[e] * c64[e] + cs[e] * s64[e];
              cs[e] = cn;
            }
          }
        }
        if (!PREPARED) {
          if (ck + 1 < itm.end) {
            load_angles(itm.unit, ck + 1);
          } else if (k + 1 < share.n_items) {
            const Item nx = share.at(k + 1);
            load_angles(nx.unit, nx.begin);
          }
        }
        fence_proxy_async_smem();                          // generic-proxy writes -> visible to the tensor core
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm->pro_done[s]));
        if (++s == NST) { s = 0; sp ^= 1u; }
      }
    }
  } else if (warp < CON_WARP0) {
    // ---------------- state ----------------
    // f32 state: row dv = 32*(qd&1) + lane, columns dk = 32*half .. +31 (the accumulator of MMA S holds the 64 dv rows
    // twice, lanes 0-63 and 64-127, so every warp finds its share in its own lane quarter)
    if (tables_first) pdl_wait();
    const int qd = warp & 3, half = qd >> 1, s_row = 32 * (qd & 1) + lane;
    const int stid = tid - STATE_WARP0 * 32;
    const uint32_t tm_ds = tm + (uint32_t(32 * qd) << 16) + PT_DS + 32 * half;
    float S[32];
    auto add4 = [&](const float* src, float f, bool coherent) {        // S = f * S + src, 16 bytes at a time
#pragma unroll
      for (int e4 = 0; e4 < 8; ++e4) {
        const float4 v4 = coherent ? __ldcg(reinterpret_cast<const float4*>(src) + e4) : __ldg(reinterpret_cast<const float4*>(src) + e4);
        S[4 * e4 + 0] = f * S[4 * e4 + 0] + v4.x; S[4 * e4 + 1] = f * S[4 * e4 + 1] + v4.y;
        S[4 * e4 + 2] = f * S[4 * e4 + 2] + v4.z; S[4 * e4 + 3] = f * S[4 * e4 + 3] + v4.w;
      }
    };
    auto publish_state = [&](int buf) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        *reinterpret_cast<uint4*>(sm->s[buf] + swz(s_row, 4 * half + c)) =
            make_uint4(pack_bf16x2(S[8 * c], S[8 * c + 1]), pack_bf16x2(S[8 * c + 2], S[8 * c + 3]),
                       pack_bf16x2(S[8 * c + 4], S[8 * c + 5]), pack_bf16x2(S[8 * c + 6], S[8 * c + 7]));
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm->s_done[buf]));
    };
    bool ok = true;
    int g = 0;
    for (int k = 0; ok && k < share.n_items; ++k) {
      const Item it = share.at(k);
      const int h = it.unit % p.H;
      const size_t bh = size_t(it.unit);
      const float* pw = sm->tab[k % NTAB].pw;
#pragma unroll
      for (int e = 0; e < 32; ++e) S[e] = 0.f;
      if (it.piece == 2) {
        // second part of a cut sequence-head: the state after the first part, written by the state warps of the CTA that
        // scanned it (in this kernel's own element order).  Bounded wait on their count.
        if (lane == 0) {
          int* flag = p.ctrl + cta;                      // 1 + (the ticket before this one)
          const unsigned long long t0 = globaltimer_ns();
          int seen;
          for (;;) {
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(flag) : "memory");
            if (seen >= STATE_WARPS || *abort_flag) break;
            if (globaltimer_ns() - t0 > JB_WAIT_LIMIT_NS) {
              *abort_flag = 1u;
              atomicCAS(p.status, 0u, JB200_STATUS_ATTN_HANDOFF);
              break;
            }
            __nanosleep(200);
          }
        }
        __syncwarp();
        __threadfence();
        add4(p.handoff + size_t(cta - 1) * D * D + s_row * D + 32 * half, 0.f, true);
      } else {
        if (p.s_in) {
          const float* sp = p.s_in + bh * D * D + s_row * D;
          if (PREPARED) {      // prepared q/k: the dk axis is interleaved
#pragma unroll
            for (int e = 0; e < 32; ++e) S[e] = __ldg(sp + (16 * half + (e >> 1)) + 32 * (e & 1));
          } else {
            add4(sp + 32 * half, 0.f, false);
          }
        }
        if (it.begin > 0) {   // state entering this segment: fold the earlier segments' contributions, oldest first
          const float gL = expf(logf(__ldg(p.gamma + h)) * float(p.seg_chunks * CH));
          const float* dp = p.seg_state + bh * p.n_pieces * D * D + s_row * D + 32 * half;
          for (int s2 = it.begin / p.seg_chunks; s2 > 0; --s2, dp += D * D) add4(dp, gL, false);
        }
      }
      publish_state(g & 1);
      // decay tables, two sequence-heads ahead (the first one's are there)
      for (int n = k == 0 ? 0 : k + 2; n <= k + 2 && n < share.n_items; ++n) {
        if (n > 0) fill_tab(sm->tab[n % NTAB], logf(__ldg(p.gamma + share.at(n).unit % p.H)), stid, 32 * STATE_WARPS);
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm->tab_full[n % NTAB]));
      }
      if (k > 0 && !mbar_wait(smem_u32(&sm->tab_full[k % NTAB]), uint32_t(k / NTAB) & 1u, abort_flag, p.status, JB200_STATUS_ATTN_LOAD)) { ok = false; break; }
      for (int ck = it.begin; ck < it.end; ++ck, ++g) {
        const float gc = pw[min(CH, T - ck * CH)];
        if (!mbar_wait(smem_u32(&sm->bar_s[g & 1]), uint32_t(g >> 1) & 1u, abort_flag, p.status, JB200_STATUS_ATTN_MMA)) { ok = false; break; }
        tc_fence_after_sync();
        __syncwarp();               // tcgen05.ld / st are warp-collective: rejoin after the per-thread wait
        uint32_t r[32];
        tmem_ld_32x32(tm_ds + 64 * (g & 1), r);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 32; ++e) S[e] = gc * S[e] + __uint_as_float(r[e]);
        if (ck + 1 < it.end) publish_state((g + 1) & 1);
      }
      if (!ok) break;
      if (it.piece == 1) {
        // first part of a cut sequence-head: its end state for the CTA that takes the second part
        float* hp = p.handoff + size_t(cta) * D * D + s_row * D + 32 * half;
#pragma unroll
        for (int e4 = 0; e4 < 8; ++e4)
          __stcg(reinterpret_cast<float4*>(hp) + e4, make_float4(S[4 * e4], S[4 * e4 + 1], S[4 * e4 + 2], S[4 * e4 + 3]));
        __threadfence();
        __syncwarp();
        if (lane == 0) atomicAdd(p.ctrl + 1 + cta, 1);
      } else if (p.s_out && it.end == n_chunks) {
        float* sp = p.s_out + bh * D * D + s_row * D;
        if (PREPARED) {
#pragma unroll
          for (int e = 0; e < 32; ++e) sp[(16 * half + (e >> 1)) + 32 * (e & 1)] = S[e];
        } else {
#pragma unroll
          for (int e4 = 0; e4 < 8; ++e4)
            *reinterpret_cast<float4*>(sp + 32 * half + 4 * e4) = make_float4(S[4 * e4], S[4 * e4 + 1], S[4 * e4 + 2], S[4 * e4 + 3]);
        }
      }
    }
  } else {
    // ---------------- consumers ----------------
    regs_inc<CON_REGS>();
    const int qd = warp & 3;                             // TMEM lane quarter of this warp
    const int grp = (warp - CON_WARP0) / CON_WARPS;      // takes the chunks with this parity
    const int i = 32 * qd + lane;                        // query row = TMEM lane
    const uint32_t tm_sc = tm + (uint32_t(32 * qd) << 16) + PT_SC + 128 * grp;
    const uint32_t tm_o2 = tm + (uint32_t(32 * qd) << 16) + PT_O2 + 64 * grp;
    uint32_t u = 0u;                                     // phase of the group's barriers
    bool ok = true;
    int g = 0, s = 0, pending = -1;                      // stage of chunk g; the one whose v tile this warp's rows are leaving through
    auto release = [&](int stage) {
      if (lane == 0) {
        bulk_wait_group_read<0>();
        mbar_arrive(smem_u32(&sm->empty_v[stage]));
      }
      __syncwarp();
    };
    if (share.chunks() == 1) {
      // A lone chunk: both groups work on it, the upper and the lower key blocks of a row (P goes to the other accumulator, since
      // what one group writes the other may not have read), then half of the output columns each, stored directly (one
      // sequence of 37 and 128 tokens 6.9 -> 6.2 and 7.2 -> 6.8 us).
      const Item it = share.at(0);
      const int b = it.unit / p.H, col = (it.unit - b * p.H) * D + 32 * grp;
      const DecayTab& tab = sm->tab[0];
      const uint32_t tm_lane = tm + (uint32_t(32 * qd) << 16);
      if (mbar_wait(smem_u32(&sm->bar_sc[0]), 0u, abort_flag, p.status, JB200_STATUS_ATTN_MMA)) {
        tc_fence_after_sync();
        __syncwarp();
        uint32_t r[16], w[8];
#pragma unroll 1
        for (int n = 0; n <= qd; ++n) {
          const int jb = n + (grp ? qd + 1 : 0);             // 16-key block
          tmem_ld_32x16(tm_lane + PT_SC + 16 * jb, r);
          tmem_ld_wait();
          const float* f = tab.pwm + (i - 16 * jb + CH);
#pragma unroll
          for (int c2 = 0; c2 < 8; ++c2) w[c2] = pack_bf16x2(__uint_as_float(r[2 * c2]) * f[-2 * c2], __uint_as_float(r[2 * c2 + 1]) * f[-2 * c2 - 1]);
          tmem_st_32x8(tm_lane + PT_SC + 128 + PT_P + 8 * jb, w);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = 0u;
        for (int jb = 2 * qd + 2 + grp; jb < 8; jb += 2) tmem_st_32x8(tm_lane + PT_SC + 128 + PT_P + 8 * jb, w);   // above the diagonal
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm->p_done[grp]));
      }
      const float gi = 0.125f * tab.pw[i + 1];
      const int t = it.begin * CH + i;
      __nv_bfloat16* op = p.o + size_t(b * T + t) * p.ld_o + col;
      if (mbar_wait(smem_u32(&sm->bar_o2[0]), 0u, abort_flag, p.status, JB200_STATUS_ATTN_MMA) &&
          mbar_wait(smem_u32(&sm->bar_b[0]), 0u, abort_flag, p.status, JB200_STATUS_ATTN_MMA)) {
        tc_fence_after_sync();
        __syncwarp();
        uint32_t a[32], c2[32];
        tmem_ld_32x32(tm_lane + PT_SC + 32 * grp, a);
        tmem_ld_32x32(tm_lane + PT_O2 + 32 * grp, c2);
        tmem_ld_wait();
        if (t < T) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              w[e] = pack_bf16x2(fmaf(gi, __uint_as_float(c2[8 * c + 2 * e]), __uint_as_float(a[8 * c + 2 * e])),
                                 fmaf(gi, __uint_as_float(c2[8 * c + 2 * e + 1]), __uint_as_float(a[8 * c + 2 * e + 1])));
            *reinterpret_cast<uint4*>(op + 8 * c) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        __syncwarp();
      }
      ok = false;                                          // nothing left for the loop
    }
    for (int k = 0; ok && k < share.n_items; ++k) {
      const Item it = share.at(k);
      const int b = it.unit / p.H, col = (it.unit - b * p.H) * D;
      const DecayTab& tab = sm->tab[k % NTAB];
      for (int ck = it.begin; ck < it.end; ++ck, ++g, s = s + 1 == NST ? 0 : s + 1) {
        if ((g & 1) != grp) continue;
        if (pending >= 0) release(pending);
        // ---- decay mask: scores -> P (lane = query row, column c = keys 2c, 2c+1) ----
        if (k > 0 && !mbar_wait(smem_u32(&sm->tab_full[k % NTAB]), uint32_t(k / NTAB) & 1u, abort_flag, p.status, JB200_STATUS_ATTN_LOAD)) { ok = false; break; }
        if (!mbar_wait(smem_u32(&sm->bar_sc[grp]), u, abort_flag, p.status, JB200_STATUS_ATTN_MMA)) { ok = false; break; }
        tc_fence_after_sync();
        __syncwarp();
        {
          uint32_t r[2][16];
          tmem_ld_32x16(tm_sc + 32 * qd + 16, r[0]);
          {
            uint32_t z[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) z[e] = 0u;
#pragma unroll
            for (int jb = 1; jb < 4; ++jb)
              if (jb > qd) tmem_st_32x16(tm_sc + PT_P + 16 * jb, z);     // above the diagonal for all rows of this warp
          }
          const float* f = tab.pwm + (i - 32 * qd - 16 + CH);   // f[-c]: factor of key 16*jb + c
#pragma unroll 1
          for (int jb = 2 * qd + 1; jb > 0; jb -= 2) {         // 16-key blocks jb and jb - 1
#pragma unroll
            for (int n = 0; n < 2; ++n) {
              tmem_ld_wait();
              if (n == 0) tmem_ld_32x16(tm_sc + 16 * (jb - 1), r[1]);
              else if (jb > 1) tmem_ld_32x16(tm_sc + 16 * (jb - 2), r[0]);
              uint32_t w[8];
#pragma unroll
              for (int c2 = 0; c2 < 8; ++c2)
                w[c2] = pack_bf16x2(__uint_as_float(r[n][2 * c2]) * f[16 * n - 2 * c2], __uint_as_float(r[n][2 * c2 + 1]) * f[16 * n - 2 * c2 - 1]);
              tmem_st_32x8(tm_sc + PT_P + 8 * (jb - n), w);
            }
            f += 32;
          }
          tmem_st_wait();
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm->p_done[grp]));
        // ---- output rows: o[i] = O1 + gamma^(i+1)/8 * O2 ----
        const float gi = 0.125f * tab.pw[i + 1];
        if (!mbar_wait(smem_u32(&sm->bar_o2[grp]), u, abort_flag, p.status, JB200_STATUS_ATTN_MMA)) { ok = false; break; }
        if (!mbar_wait(smem_u32(&sm->bar_b[grp]), u, abort_flag, p.status, JB200_STATUS_ATTN_MMA)) { ok = false; break; }
        u ^= 1u;
        tc_fence_after_sync();
        __syncwarp();
        uint8_t* o_p = sm->v[s];                           // P V has read the chunk's v tile: the rows leave through it
#pragma unroll 1
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t a[32], c2[32];
          tmem_ld_32x32(tm_sc + 32 * hf, a);
          tmem_ld_32x32(tm_o2 + 32 * hf, c2);
          tmem_ld_wait();
          if (hf == 1) {                                   // both accumulators are in registers now
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&sm->o_done[grp]));
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
              w[e] = pack_bf16x2(fmaf(gi, __uint_as_float(c2[8 * c + 2 * e]), __uint_as_float(a[8 * c + 2 * e])),
                                 fmaf(gi, __uint_as_float(c2[8 * c + 2 * e + 1]), __uint_as_float(a[8 * c + 2 * e + 1])));
            *reinterpret_cast<uint4*>(o_p + swz(i, 4 * hf + c)) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          if (32 * qd < T - ck * CH) tma_store_3d(&tm_o, col, ck * CH + 32 * qd, b, smem_u32(o_p) + 32 * 128 * qd);
          bulk_commit_group();
        }
        pending = s;
      }
    }
    if (lane == 0) bulk_wait_group<0>();
    __syncwarp();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tm, PIPE_TMEM_COLS);
  }
}

// State-only calls (no output rows wanted): every piece of the sequence has left its contribution D_s, scanned
// from a zero state, in seg_state; the state after the whole sequence is
//   S = gamma^T S_in + sum_s gamma^(T - end_s) D_s,      end_s = last token of piece s + 1.
// One CTA per (head, sequence), 16 elements per thread.  The pieces are in the kernel's own column order
// (interleaved when q/k were prepared); s_in / s_out use the natural one.
__global__ void __launch_bounds__(256) attn_fold_states_kernel(const AttnParams p) {
  pdl_wait();
  pdl_trigger();
  const int h = blockIdx.x, b = blockIdx.y;
  const float log_g = logf(__ldg(p.gamma + h));
  const int L = p.seg_chunks * CH;
  const size_t bh = size_t(b) * p.H + h;
  for (int e = threadIdx.x; e < D * D; e += 256) {
    const int r = e >> 6, d = e & 63;
    const int col = p.qk_prepared ? (2 * (d & 31) + (d >> 5)) : d;
    float acc = p.s_in ? expf(log_g * float(p.T)) * __ldg(p.s_in + bh * D * D + e) : 0.f;
    for (int s2 = 0; s2 < p.n_pieces; ++s2) {
      const int end = min((s2 + 1) * L, p.T);
      acc += expf(log_g * float(p.T - end)) * __ldg(p.seg_state + (bh * p.n_pieces + s2) * D * D + r * D + col);
    }
    p.s_out[bh * D * D + e] = acc;
  }
}

// One-token step (decode): S <- gamma*S + v (x) k', o = S q' for every (sequence, head).  Pure state
// streaming: 2 x 16 KiB of fp32 state per (sequence, head) against 384 B of q, k, v, so the kernel is a
// coalesced read-modify-write of S with the feature map + RoPE of the single token done in shared memory.
// Thread t owns state row t/4, columns 16*(t%4)..+15; s_out may alias s_in.
__global__ void __launch_bounds__(256)
attn_decode_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                   const __nv_bfloat16* __restrict__ v, int ld_qkv, const AttnParams p) {
  __shared__ __align__(16) float sv[D], rq[D], rk[D];
  const int h = blockIdx.x, b = blockIdx.y, t = threadIdx.x;
  // What the token does not decide first: the thread's 64 bytes of state, the position and its angles.  In a chain they
  // were written long before and are fetched while the projection still runs.
  const int row = t >> 2, c0 = (t & 3) * 16;
  const size_t so = (size_t(b) * p.H + h) * D * D + size_t(row) * D + c0;
  float4 st[4];
  float cs = 0.f, sn = 0.f, gamma = 0.f;
  auto fetch = [&]() {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      st[i] = p.s_in ? *reinterpret_cast<const float4*>(p.s_in + so + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
    gamma = __ldg(p.gamma + h);
    if (t < D / 2) {
      int pos = p.pos0 ? p.pos0[b] : p.pos0_scalar;
      pos = pos < 0 ? 0 : (pos >= p.n_pos ? p.n_pos - 1 : pos);
      cs = __ldg(p.cos_tab + size_t(pos) * 32 + t);
      sn = __ldg(p.sin_tab + size_t(pos) * 32 + t);
    }
  };
  if (p.settled) fetch();
  __syncwarp();
  pdl_wait();
  pdl_trigger();
  if (!p.settled) fetch();
  const size_t off = size_t(b) * ld_qkv + h * D;
  if (t < D / 2) {
    const float q0 = elu1(__bfloat162float(q[off + t])) * 0.125f, q1 = elu1(__bfloat162float(q[off + t + 32])) * 0.125f;
    const float k0 = elu1(__bfloat162float(k[off + t])), k1 = elu1(__bfloat162float(k[off + t + 32]));
    rq[t] = rope_lo(q0, q1, cs, sn);  rq[t + 32] = rope_hi(q0, q1, cs, sn);
    rk[t] = rope_lo(k0, k1, cs, sn);  rk[t + 32] = rope_hi(k0, k1, cs, sn);
  } else if (t < D / 2 + D) {
    sv[t - 32] = __bfloat162float(v[off + t - 32]);
  }
  __syncthreads();
  const float vr = sv[row];
  float acc = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int c = c0 + 4 * i;
    st[i].x = decode_update(gamma, st[i].x, vr, rk[c]);      st[i].y = decode_update(gamma, st[i].y, vr, rk[c + 1]);
    st[i].z = decode_update(gamma, st[i].z, vr, rk[c + 2]);  st[i].w = decode_update(gamma, st[i].w, vr, rk[c + 3]);
    acc += decode_dot4(st[i], *reinterpret_cast<const float4*>(rq + c));
  }
  if (p.s_out) {
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(p.s_out + so + 4 * i) = st[i];
  }
  acc += __shfl_xor_sync(0xffffffffu, acc, 1);
  acc += __shfl_xor_sync(0xffffffffu, acc, 2);
  if ((t & 3) == 0) p.o[size_t(b) * p.ld_o + h * D + row] = __float2bfloat16_rn(acc);
}

// The same step as a stream of 16 KiB state tiles through shared memory: a fixed grid of CTAs (two per SM), each
// walking its share of the (sequence, head) pairs with four tiles in flight as untiled bulk copies (global -> shared
// on an mbarrier, shared -> global as a bulk group), the update done in place in the tile.  Bytes in flight do not
// depend on registers or on CTA turnover, which is what holds attn_decode_kernel at ~0.6 of the HBM peak.  Needs
// both s_in and s_out (they may be the same buffer); the feature map of the NEXT pair's token is computed while the
// current tile is awaited.  Thread t of 256: columns 32*((t>>3)&1) + 4*(t&7) .. +3 of rows 16*i + (t>>4), i = 0..3, so
// a quarter-warp always touches 128 contiguous bytes of the tile (no bank conflicts).
constexpr int DEC_STAGES = 4;
constexpr int DEC_TILE_BYTES = D * D * 4;
struct DecodeSmem {
  float tile[DEC_STAGES][D * D];
  uint64_t full[DEC_STAGES];
  float rq[2][D], rk[2][D], sv[2][D];
  uint32_t abort_flag;
};
constexpr size_t DEC_SMEM_BYTES = sizeof(DecodeSmem) + 128;

__global__ void __launch_bounds__(256, 2)
attn_decode_stream_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k,
                          const __nv_bfloat16* __restrict__ v, int ld_qkv, const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  DecodeSmem* sm = reinterpret_cast<DecodeSmem*>(smem_raw + (((raw_addr + 127u) & ~127u) - raw_addr));
  const int t = threadIdx.x, lane = t & 31;
  if (t == 0) {
    for (int s = 0; s < DEC_STAGES; ++s) mbar_init(smem_u32(&sm->full[s]), 1);
    sm->abort_flag = 0;
    fence_mbar_init();
  }
  const int n_units = p.B * p.H;
  const int n_my = (n_units - int(blockIdx.x) + int(gridDim.x) - 1) / int(gridDim.x);   // units u = blockIdx.x + i * gridDim.x
  auto unit_of = [&](int i) { return int(blockIdx.x) + i * int(gridDim.x); };
  auto issue_load = [&](int i) {      // thread 0 only
    const int s = i % DEC_STAGES;
    mbar_arrive_expect_tx(smem_u32(&sm->full[s]), DEC_TILE_BYTES);
    bulk_load_1d(smem_u32(sm->tile[s]), p.s_in + size_t(unit_of(i)) * D * D, DEC_TILE_BYTES, smem_u32(&sm->full[s]));
  };
  auto issue_first = [&]() {
    if (t == 0) {
      for (int i = 0; i < DEC_STAGES && i < n_my; ++i) issue_load(i);
    }
  };
  if (p.settled) issue_first();      // the first state tiles travel while the projection still runs
  __syncwarp();
  pdl_wait();
  pdl_trigger();
  if (!p.settled) issue_first();
  __syncthreads();
  volatile uint32_t* abort_flag = &sm->abort_flag;
  // feature map + RoPE of the token of unit i into buffer i & 1: threads 0..31 the q / k pairs (d, d + 32), 32..95 v
  auto token_features = [&](int i) {
    if (t >= 96) return;
    const int u = unit_of(i), b = u / p.H, h = u - b * p.H, buf = i & 1;
    const size_t off = size_t(b) * ld_qkv + h * D;
    if (t < 32) {
      const float q0 = elu1(__bfloat162float(q[off + t])) * 0.125f, q1 = elu1(__bfloat162float(q[off + t + 32])) * 0.125f;
      const float k0 = elu1(__bfloat162float(k[off + t])), k1 = elu1(__bfloat162float(k[off + t + 32]));
      int pos = p.pos0 ? p.pos0[b] : p.pos0_scalar;
      pos = pos < 0 ? 0 : (pos >= p.n_pos ? p.n_pos - 1 : pos);
      const float c = __ldg(p.cos_tab + size_t(pos) * 32 + t), sn = __ldg(p.sin_tab + size_t(pos) * 32 + t);
      sm->rq[buf][t] = rope_lo(q0, q1, c, sn);  sm->rq[buf][t + 32] = rope_hi(q0, q1, c, sn);
      sm->rk[buf][t] = rope_lo(k0, k1, c, sn);  sm->rk[buf][t + 32] = rope_hi(k0, k1, c, sn);
    } else {
      sm->sv[buf][t - 32] = __bfloat162float(v[off + t - 32]);
    }
  };
  if (n_my > 0) token_features(0);
  __syncthreads();
  const int col0 = 32 * ((t >> 3) & 1) + 4 * (t & 7), r0 = t >> 4;
  for (int i = 0; i < n_my; ++i) {
    const int s = i % DEC_STAGES, buf = i & 1;
    const int u = unit_of(i), b = u / p.H, h = u - b * p.H;
    if (i + 1 < n_my) token_features(i + 1);          // its loads overlap the wait for this unit's tile
    const float gamma = __ldg(p.gamma + h);
    const float4 kq = *reinterpret_cast<const float4*>(&sm->rk[buf][col0]);
    const float4 qq = *reinterpret_cast<const float4*>(&sm->rq[buf][col0]);
    if (!mbar_wait(smem_u32(&sm->full[s]), uint32_t(i / DEC_STAGES) & 1u, abort_flag, p.status, JB200_STATUS_ATTN_LOAD)) break;
    float acc[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int row = 16 * j + r0;
      float4* cell = reinterpret_cast<float4*>(&sm->tile[s][row * D + col0]);
      const float vr = sm->sv[buf][row];
      float4 st = *cell;
      st.x = decode_update(gamma, st.x, vr, kq.x);  st.y = decode_update(gamma, st.y, vr, kq.y);
      st.z = decode_update(gamma, st.z, vr, kq.z);  st.w = decode_update(gamma, st.w, vr, kq.w);
      *cell = st;
      acc[j] = decode_dot4(st, qq);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
    }
    if ((lane & 15) == 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j) p.o[size_t(b) * p.ld_o + h * D + 16 * j + r0] = __float2bfloat16_rn(acc[j]);
    }
    fence_proxy_async_smem();      // the updated tile goes out through the async proxy
    __syncthreads();               // tile complete; also orders this iteration's reads of rq/rk/sv before their reuse
    if (t == 0) {
      bulk_store_1d(p.s_out + size_t(u) * D * D, smem_u32(sm->tile[s]), DEC_TILE_BYTES);
      bulk_commit_group();
      if (i >= 1 && i - 1 + DEC_STAGES < n_my) {
        bulk_wait_group_read<1>();   // the store of unit i - 1 has read its tile: the stage takes unit i - 1 + DEC_STAGES
        issue_load(i - 1 + DEC_STAGES);
      }
    }
  }
  if (t == 0) bulk_wait_group<0>();
}

int make_map(CUtensorMap* tm, const void* ptr, int rows, int cols, int ld) {
  const cuuint64_t gdim[2] = {cuuint64_t(cols), cuuint64_t(rows)};
  const cuuint64_t gstride[1] = {cuuint64_t(ld) * 2};
  const cuuint32_t box[2] = {cuuint32_t(D), cuuint32_t(CH)};
  return encode_tiled(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, ptr, gdim, gstride, box, CU_TENSOR_MAP_SWIZZLE_128B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_128B, "attn_scan");
}

}  // namespace

// From so many chunks on a cut is worth the ticket, the hand-off and the clearing of their words (16 x 512, four chunks: 26.4 us
// before and now; eight: 32 x 1024 in equal shares 3.5 sequence-heads per SM instead of four).
static constexpr int SPLIT_CHUNKS = 4;

// Segments: the pipeline kernel runs one CTA per SM, so sequences are cut only when B*H leaves SMs idle;
// each segment is at least two chunks long.
static void pick_segments(int B, int T, int H, int sms, int* seg_chunks, int* nseg) {
  const int n_chunks = (T + CH - 1) / CH;
  long want = long(sms) / (long(B) * H);
  if (want < 1) want = 1;
  if (want > n_chunks / 2) want = n_chunks / 2 > 0 ? n_chunks / 2 : 1;
  int sc = int((n_chunks + want - 1) / want);
  *seg_chunks = sc;
  *nseg = (n_chunks + sc - 1) / sc;
}

// More sequence-heads than SMs: as many CTAs as SMs walk them, and where they do not come out even, shares are cut inside a
// sequence-head.
static bool pick_split(int B, int T, int H, int sms) {
  const long U = long(B) * H;
  const long n_chunks = (T + CH - 1) / CH;
  return U > sms && U % sms != 0 && n_chunks >= SPLIT_CHUNKS && U * n_chunks < (1l << 31);
}

size_t attn_scan_scratch_bytes(int B, int T, int H) {
  if (B <= 0 || T <= 0 || H <= 0) return 0;
  int sms = sm_count();
  if (sms <= 0) sms = 148;
  int sc, ns;
  pick_segments(B, T, H, sms, &sc, &ns);
  const size_t seg_bytes = size_t(B) * H * size_t(ns) * D * D * sizeof(float);   // ns - 1 pieces for a full call, ns for a state-only one
  const size_t split_bytes = pick_split(B, T, H, sms) ? size_t(sms) * D * D * sizeof(float) + (size_t(sms) + 1) * sizeof(int) : 0;
  return seg_bytes > split_bytes ? seg_bytes : split_bytes;
}

int launch_attn_scan(const void* q, const void* k, const void* v, int ld_qkv, const float* gamma,
                     const float* cos_tab, const float* sin_tab, int n_pos, const int32_t* pos0, int pos0_scalar,
                     const float* s_in, void* o, int ld_o, float* s_out, void* scratch, int B, int T, int H,
                     int head_dim, int flags, cudaStream_t stream, bool settled) {
  JB_REQUIRE((flags & ~JB200_ATTN_QK_PREPARED) == 0, "attn_scan: unknown flags %d", flags);
  JB_REQUIRE(!(flags & JB200_ATTN_QK_PREPARED) || T > 1, "attn_scan: prepared q/k is for T > 1 (single-token steps take raw q, k)");
  JB_REQUIRE(head_dim == D, "attn_scan: head_dim (%d) must be %d", head_dim, D);
  JB_REQUIRE(B >= 0 && T >= 0 && H > 0, "attn_scan: bad shape (B=%d, T=%d, H=%d)", B, T, H);
  JB_REQUIRE(B <= 65535, "attn_scan: batch (%d) exceeds 65535", B);
  if (B == 0 || T == 0) return JB200_OK;
  JB_REQUIRE(k && v && gamma && cos_tab && sin_tab, "attn_scan: null pointer");
  JB_REQUIRE(o ? (q != nullptr) : (s_out && scratch && T > 1),
             "attn_scan: a call without output rows (state only) needs s_out, scratch and T > 1; any other call needs q and o");
  if (!q) q = k;     // state only: the tensor map of q is built but never used
  JB_REQUIRE(ld_qkv >= H * D && ld_qkv % 8 == 0 && (!o || (ld_o >= H * D && ld_o % 8 == 0)),
             "attn_scan: row strides must cover H*64 columns and be multiples of 8 elements");
  JB_REQUIRE(aligned16(q) && aligned16(k) && aligned16(v) && (!o || aligned16(o)) && aligned16(cos_tab) && aligned16(sin_tab),
             "attn_scan: pointers must be 16-byte aligned");
  JB_REQUIRE(size_t(B) * T < (size_t(1) << 31), "attn_scan: too many rows");
  JB_REQUIRE(n_pos >= 1, "attn_scan: empty RoPE table");
  if (!pos0) JB_REQUIRE(pos0_scalar >= 0 && pos0_scalar + T <= n_pos, "attn_scan: RoPE table (%d rows) too short for positions %d..%d", n_pos, pos0_scalar, pos0_scalar + T - 1);
  JB_REQUIRE(!s_in || aligned16(s_in), "attn_scan: state pointers must be 16-byte aligned");
  JB_REQUIRE(!s_out || aligned16(s_out), "attn_scan: state pointers must be 16-byte aligned");
  if (T == 1) {
    AttnParams dp;
    dp.gamma = gamma; dp.cos_tab = cos_tab; dp.sin_tab = sin_tab; dp.pos0 = pos0; dp.pos0_scalar = pos0_scalar;
    dp.n_pos = n_pos; dp.s_in = s_in; dp.s_out = s_out; dp.o = reinterpret_cast<__nv_bfloat16*>(o); dp.ld_o = ld_o;
    dp.B = B; dp.T = 1; dp.H = H; dp.seg_chunks = 1; dp.nseg = 1; dp.seg_state = nullptr; dp.n_pieces = 0; dp.qk_prepared = 0;
    dp.wide_tab = 0; dp.settled = settled ? 1 : 0; dp.status = device_status_ptr();
    if (!dp.status) return JB200_ERR_CUDA;
    if (s_in && s_out && B * H >= 64) {
      // the state streams through shared memory as bulk copies: two CTAs per SM walk the (sequence, head) pairs
      const int sms = sm_count();
      if (sms <= 0) return JB200_ERR_CUDA;
      JB_MAX_SMEM(attn_decode_stream_kernel, DEC_SMEM_BYTES);
      const int grid = B * H < 2 * sms ? B * H : 2 * sms;
      launch_dep(attn_decode_stream_kernel, grid, 256, DEC_SMEM_BYTES, stream, reinterpret_cast<const __nv_bfloat16*>(q),
                 reinterpret_cast<const __nv_bfloat16*>(k), reinterpret_cast<const __nv_bfloat16*>(v), ld_qkv, dp);
      JB_LAUNCH_CHECK("attn_decode_stream_kernel");
      return JB200_OK;
    }
    launch_dep(attn_decode_kernel, dim3(H, B), 256, 0, stream, reinterpret_cast<const __nv_bfloat16*>(q),
                                                        reinterpret_cast<const __nv_bfloat16*>(k),
                                                        reinterpret_cast<const __nv_bfloat16*>(v), ld_qkv, dp);
    JB_LAUNCH_CHECK("attn_decode_kernel");
    return JB200_OK;
  }
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_map(&tq, q, B * T, H * D, ld_qkv)) != JB200_OK) return rc;
  if ((rc = make_map(&tk, k, B * T, H * D, ld_qkv)) != JB200_OK) return rc;
  if ((rc = make_map(&tv, v, B * T, H * D, ld_qkv)) != JB200_OK) return rc;
  AttnParams p;
  p.gamma = gamma; p.cos_tab = cos_tab; p.sin_tab = sin_tab; p.pos0 = pos0; p.pos0_scalar = pos0_scalar;
  p.n_pos = n_pos; p.s_in = s_in; p.s_out = s_out; p.o = reinterpret_cast<__nv_bfloat16*>(o); p.ld_o = ld_o;
  p.B = B; p.T = T; p.H = H;
  p.qk_prepared = (flags & JB200_ATTN_QK_PREPARED) ? 1 : 0;
  p.wide_tab = ((reinterpret_cast<uintptr_t>(cos_tab) | reinterpret_cast<uintptr_t>(sin_tab)) & 31u) == 0 ? 1 : 0;
  p.n_pieces = 0;
  p.status = device_status_ptr();
  if (!p.status) return JB200_ERR_CUDA;
  const int sms = sm_count();
  if (sms <= 0) return JB200_ERR_CUDA;
  p.seg_chunks = (T + CH - 1) / CH;
  p.nseg = 1;
  p.seg_state = reinterpret_cast<float*>(scratch);
  if (scratch) pick_segments(B, T, H, sms, &p.seg_chunks, &p.nseg);   // without scratch: one segment per sequence
  JB_REQUIRE(p.nseg <= 65535, "attn_scan: too many segments");
  p.settled = settled || p.nseg > 1;      // the pass over the segments waited for whatever made gamma
  JB_REQUIRE(!scratch || aligned16(scratch), "attn_scan: scratch pointer must be 16-byte aligned");
  p.n_pieces = o ? p.nseg - 1 : p.nseg;
  p.split = 0; p.handoff = nullptr; p.ctrl = nullptr;
  if (!o) {
    // state only: the k/v pass over every piece, then the fold
    JB_MAX_SMEM(attn_state_pass_kernel, STATE_SMEM_BYTES);
    AttnParams ps = p;
    ps.settled = settled ? 1 : 0;
    launch_dep(attn_state_pass_kernel, dim3(H, B, p.nseg), STATE_THREADS, STATE_SMEM_BYTES, stream, tk, tv, ps);
    JB_LAUNCH_CHECK("attn_state_pass_kernel");
    launch_dep(attn_fold_states_kernel, dim3(H, B), 256, 0, stream, p);
    JB_LAUNCH_CHECK("attn_fold_states_kernel");
    return JB200_OK;
  }
  if (p.qk_prepared) JB_MAX_SMEM(attn_scan_pipe_kernel<true>, PIPE_SMEM_BYTES);
  else JB_MAX_SMEM(attn_scan_pipe_kernel<false>, PIPE_SMEM_BYTES);
  if (p.nseg > 1) {
    JB_MAX_SMEM(attn_state_pass_kernel, STATE_SMEM_BYTES);
    AttnParams ps = p;
    ps.settled = settled ? 1 : 0;
    launch_dep(attn_state_pass_kernel, dim3(H, B, p.nseg - 1), STATE_THREADS, STATE_SMEM_BYTES, stream, tk, tv, ps);
    JB_LAUNCH_CHECK("attn_state_pass_kernel");
  }
  // output rows leave 32 at a time, clipped at the end of their sequence
  CUtensorMap to;
  const cuuint64_t odim[3] = {cuuint64_t(H) * D, cuuint64_t(T), cuuint64_t(B)};
  const cuuint64_t ostride[2] = {cuuint64_t(ld_o) * 2, cuuint64_t(T) * ld_o * 2};
  const cuuint32_t obox[3] = {cuuint32_t(D), 32, 1};
  if ((rc = encode_tiled(&to, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, o, odim, ostride, obox, CU_TENSOR_MAP_SWIZZLE_128B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, "attn_scan")) != JB200_OK)
    return rc;
  const long units = long(B) * H * p.nseg;
  const unsigned grid = unsigned(p.nseg > 1 || units < sms ? units : sms);
  if (scratch && p.nseg == 1 && pick_split(B, T, H, sms)) {
    p.split = 1;
    p.handoff = reinterpret_cast<float*>(scratch);
    p.ctrl = reinterpret_cast<int*>(p.handoff + size_t(grid) * D * D);
    JB_CUDA(cudaMemsetAsync(p.ctrl, 0, (size_t(grid) + 1) * sizeof(int), stream));
  }
  const long total = p.split ? long(B) * H * p.seg_chunks : long(B) * H;
  p.per_cta = int(total / grid);
  p.spare = int(total % grid);
  launch_dep(p.qk_prepared ? attn_scan_pipe_kernel<true> : attn_scan_pipe_kernel<false>, dim3(grid), PIPE_THREADS, PIPE_SMEM_BYTES, stream, tq,
             tk, tv, to, p);
  JB_LAUNCH_CHECK("attn_scan_pipe_kernel");
  return JB200_OK;
}

}  // namespace jb
