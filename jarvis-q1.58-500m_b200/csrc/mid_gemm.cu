// Ternary linear layers for up to a few hundred tokens on the 5th-generation tensor cores: the latency form of
// ternary_gemm_kernel.
//
// With one or two tiles per SM nothing amortises a pipeline's fill: ternary_gemm_kernel takes 11-18 us for products whose
// arithmetic is ~1 us, because every K-block of its four-stage ring waits for a code load from L2, the decode, the MMA
// and the stage's release one after another (~550 cycles), after TMEM, barriers and tensor maps have been set up.  Here
//   - the work is a list of (token tile, out-feature tile) items that every CTA reads off the segment offsets; those were
//     complete before the kernel ahead on the stream began, so a CTA knows its weights at once and decodes them into every
//     stage there is before the grid dependency is waited for;
//   - K-blocks travel in chunks of CK: one TMA copy, one barrier wait and one commit per chunk (issued singly they cost
//     ~290, ~95 and ~100 cycles next to 4 x 40-48 cycles for a K-block's MMAs), with as many chunks in flight as fit
//     (a smaller ring that lets two CTAs share an SM and prologues overlap measured 5-15 % slower);
//   - code loads run four chunks ahead in registers that are never moved (a move waits for the load);
//   - the eight decoder warps become the epilogue; the residual is added by reductions, nothing waits for old values.
// What is left is the chain itself: 4 x 40-48 cycles per K-block.  Accumulation is the same chain of K = 16 steps as in
// ternary_gemm_kernel: results are its bit for bit.
#include <algorithm>

#include "common.cuh"
#include "gemm_shared.cuh"
#include "launchers.h"
#include "row_math.cuh"

namespace jb {

namespace {

constexpr int BK = 64;
constexpr int CK = 2;                          // K-blocks per chunk (four: 1-3 % slower, the ring gets too coarse)
constexpr int MAX_CHUNKS = 8, DEC_WARP0 = 2, THREADS = 320, MAP_WARP = 10;
constexpr int SLOTS = 4;                       // chunks whose codes are in registers

struct MidParams {
  const uint8_t* w;            // prepared [G][N][K/4]
  const float* alpha;          // [G][N / alpha_rows]
  const int32_t* seg;          // device [G+1] or null (every group takes rows [0, M), or the segments are counted from routes)
  MidRoutes routes;
  void* out;
  int M, N, K, G, n_ft, alpha_rows, epilogue;
  int bn[3], chunks[3];        // token tiles and their rings: the first whose items are one wave, else the last
  uint32_t tmem_cols;
  unsigned int* status;
};

struct Maps {
  CUtensorMap x[3];            // one box per token tile
};

struct Ctl {
  uint64_t full[MAX_CHUNKS], empty[MAX_CHUNKS], acc_full, acc_empty;
  uint32_t tmem_base, abort_flag;
  int pick;
  int32_t beg[MAX_GROUPS], end[MAX_GROUPS], first[MAX_GROUPS + 1];   // a group's rows and its first token tile
};

// The items of a CTA: a token tile (rows [tok0, end) of group grp, at most bn of them) and an out-feature tile, the latter
// varying fastest.  The first one is worked out before the grid dependency is waited for; after it, only a CTA that has
// another item pays for the division.
struct Items {
  int i, grp, tok0, end, ft;
  __device__ __forceinline__ bool at(const MidParams& p, const Ctl& ctl, int bn) {
    if (i >= ctl.first[p.G] * p.n_ft) return false;
    const int t = i / p.n_ft;
    ft = i - t * p.n_ft;
    grp = 0;
    while (t >= ctl.first[grp + 1]) ++grp;
    tok0 = ctl.beg[grp] + (t - ctl.first[grp]) * bn;
    end = ctl.end[grp];
    return true;
  }
  __device__ __forceinline__ bool first(const MidParams& p, const Ctl& ctl, int bn) {
    i = blockIdx.x;
    return at(p, ctl, bn);
  }
  __device__ __forceinline__ bool next(const MidParams& p, const Ctl& ctl, int bn) {
    i += gridDim.x;
    return at(p, ctl, bn);
  }
};

// Accumulator of a tile of 64 out-features: 16 in each quarter of the lanes.  32 columns of the lower 16 lanes; thread (g, c) of
// 8 x 4 receives of rows g (v[4j], v[4j + 1]) and g + 8 (v[4j + 2], v[4j + 3]) the columns 8j + 2c and 8j + 2c + 1.
__device__ __forceinline__ void tmem_ld_16x256b_x4(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// BM: out-features of a tile.  128 is the MMA's full rate; but up to ~100 tokens a step is bound by the shared memory that its
// operands are read from (BM + bn rows of 32 bytes, 128 bytes a cycle, and the same again for the decoded weights and
// the copied rows), so tiles of 64, on twice as many SMs, take less time each: half the codes to fetch and decode, half the epilogue.
// ROUTE: 0 rows or segments as given, 1 rows stored in dispatch order and the maps left by a warp of their own, 2 segments counted from
// the ids, 3 rows stored at the slots of the maps (kernels of their own: the code of the others costs a plain call 1 %).
// One CTA per SM, since its ring fills the shared memory: with routes 1 and 2 kept to the registers of two, 24 layers and head took 967 us where
// they take 957 at 72 tokens, 1037 and 1032 at 100, as long from 128 on, and steps of 100 and 160 sequences 1144 and 1133, 1349 and 1340.
template <int BM, int ROUTE>
__global__ void __launch_bounds__(ROUTE == 1 ? THREADS + 32 : THREADS, 1)
mid_gemm_kernel(const __grid_constant__ Maps maps, const MidParams p) {
  constexpr int A_BYTES = BM * BK * 2;
  extern __shared__ uint8_t smem_raw[];
  __shared__ Ctl ctl;
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const int warp = warp_index(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_CHUNKS; ++s) {
      mbar_init(smem_u32(&ctl.full[s]), 1 + 8);      // the producer's expectation and the eight decoder warps
      mbar_init(smem_u32(&ctl.empty[s]), 1);
    }
    mbar_init(smem_u32(&ctl.acc_full), 1);
    mbar_init(smem_u32(&ctl.acc_empty), 8);
    ctl.abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&maps.x[0]);
  }
  if (warp == 0) {
    __syncwarp();                 // tcgen05.alloc is warp-collective: lane 0 rejoins from the barrier set-up first
    tmem_alloc(smem_u32(&ctl.tmem_base), p.tmem_cols);
    tmem_relinquish();
  }
  // Weights and segments were complete before the kernel ahead of this one started: every role waits for the grid dependency
  // where it first needs the rows.
  if (warp == 1) {
    static_assert(MAX_GROUPS <= 32, "one lane per group");
    int beg = 0, end = 0;
    if (lane < p.G) {
      beg = p.seg ? min(max(__ldg(p.seg + lane), 0), p.M) : 0;
      end = p.seg ? min(max(__ldg(p.seg + lane + 1), 0), p.M) : p.M;
    }
    if constexpr (ROUTE == 2) {                // the kernel ahead makes the offsets; the ids are older
      constexpr int ROUNDS = 2 * MID_ROUTE_TOKENS / 32;
      int ex[ROUNDS], n_of = 0;
#pragma unroll
      for (int i = 0; i < ROUNDS; ++i) ex[i] = i * 32 + lane < p.M ? max(int(p.routes.ids[i * 32 + lane]), 0) : -1;
      for (int q = 0; q < p.G; ++q) {
        int n = 0;
#pragma unroll
        for (int i = 0; i < ROUNDS; ++i) n += __popc(__ballot_sync(0xffffffffu, ex[i] == q));
        if (lane == q) n_of = n;
      }
      end = n_of;
      for (int d = 1; d < MAX_GROUPS; d *= 2) {
        const int u = __shfl_up_sync(0xffffffffu, end, d);
        if (lane >= d) end += u;
      }
      beg = end - n_of;
    }
    auto tiles_of = [&](int bn) {              // token tiles of groups 0..lane
      int t = end > beg ? (end - beg + bn - 1) / bn : 0;
      for (int d = 1; d < MAX_GROUPS; d *= 2) {
        const int u = __shfl_up_sync(0xffffffffu, t, d);
        if (lane >= d) t += u;
      }
      return t;
    };
    int pick = 0, tiles = tiles_of(p.bn[0]);
    while (pick < 2 && p.bn[2] != p.bn[0] && __shfl_sync(0xffffffffu, tiles, p.G - 1) * p.n_ft > int(gridDim.x)) {
      ++pick;
      tiles = tiles_of(pick == 1 ? p.bn[1] : p.bn[2]);
    }
    if (lane < p.G) {
      ctl.beg[lane] = beg;
      ctl.end[lane] = end;
      ctl.first[lane + 1] = tiles;
    }
    if (lane == 0) {
      ctl.first[0] = 0;
      ctl.pick = pick;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = ctl.tmem_base;
  volatile uint32_t* abort_flag = &ctl.abort_flag;
  // votes: their results are in uniform registers, which copies and MMAs are issued from (a value read from shared memory
  // there cost 1.8 us a launch)
  const bool t1 = __any_sync(0xffffffffu, ctl.pick == 1), t2 = __any_sync(0xffffffffu, ctl.pick == 2);
  const int bn = t2 ? p.bn[2] : t1 ? p.bn[1] : p.bn[0], n_ch = p.K / (BK * CK);
  const int S = t2 ? p.chunks[2] : t1 ? p.chunks[1] : p.chunks[0];
  const uint32_t kb_bytes = uint32_t(bn) * BK * 2, b_bytes = kb_bytes * CK;
  const uint32_t b_base = base + uint32_t(S) * (CK * A_BYTES);
  const CUtensorMap* tmap_x = t2 ? &maps.x[2] : t1 ? &maps.x[1] : &maps.x[0];
  if (warp == 0) {
    // ---------------- TMA producer ----------------
    Items it;
    bool more = it.first(p, ctl, bn);
    pdl_wait();
    pdl_trigger();
    int s = 0;
    uint32_t ph = 1u;
    bool ok = true;
    for (; ok && more; more = it.next(p, ctl, bn)) {
#pragma unroll 1
      for (int c = 0; c < n_ch; ++c) {
        const uint32_t full = smem_u32(&ctl.full[s]);
        if (!mbar_wait(smem_u32(&ctl.empty[s]), ph, abort_flag, p.status, JB200_STATUS_GEMM_PRODUCER)) { ok = false; break; }
        if (elect_one()) {
          mbar_arrive_expect_tx(full, b_bytes);
          tma_load_3d(b_base + uint32_t(s) * b_bytes, tmap_x, 0, it.tok0, c * CK, full);
        }
        __syncwarp();
        if (++s == S) { s = 0; ph ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    Items it;
    bool more = it.first(p, ctl, bn);
    pdl_wait();
    pdl_trigger();
    const uint32_t idesc = umma_idesc_bf16(BM, bn);
    const uint64_t adesc0 = umma_desc_k_sw128(base), bdesc0 = umma_desc_k_sw128(b_base);
    uint64_t ad = adesc0, bd = bdesc0;
    int s = 0;
    uint32_t ph = 0u, tile = 0u;
    bool ok = true;
    for (; ok && more; more = it.next(p, ctl, bn), ++tile) {
      if (!mbar_wait(smem_u32(&ctl.acc_empty), (tile & 1u) ^ 1u, abort_flag, p.status, JB200_STATUS_GEMM_MMA)) break;
      tc_fence_after_sync();
#pragma unroll 1
      for (int c = 0; c < n_ch; ++c) {
        if (!mbar_wait(smem_u32(&ctl.full[s]), ph, abort_flag, p.status, JB200_STATUS_GEMM_MMA)) { ok = false; break; }
        tc_fence_after_sync();
        if (elect_one()) {
#pragma unroll
          for (int j = 0; j < CK; ++j) {
            const uint64_t aj = ad + uint64_t(j) * (A_BYTES >> 4), bj = bd + uint64_t(j) * (kb_bytes >> 4);
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk)
              umma_bf16_ss(tmem, aj + uint64_t(kk * 2), bj + uint64_t(kk * 2), idesc, (c | j | kk) != 0 ? 1u : 0u);
          }
          umma_commit(smem_u32(&ctl.empty[s]));
          if (c + 1 == n_ch) umma_commit(smem_u32(&ctl.acc_full));
        }
        __syncwarp();
        ad += (CK * A_BYTES) >> 4;
        bd += b_bytes >> 4;
        if (++s == S) { s = 0; ph ^= 1u; ad = adesc0; bd = bdesc0; }
      }
    }
  } else if (ROUTE == 1 && warp == MAP_WARP) {
    // ---------------- dispatch maps, beside everything else ----------------
    pdl_wait();
    pdl_trigger();
    if (blockIdx.x == 0) {
      const long long* ids = reinterpret_cast<const long long*>(p.routes.ids);
      const MidRoutes& r = p.routes;
      constexpr int ROUNDS = 2 * MID_ROUTE_TOKENS / 32;
      if (p.G == 4) sort_routes<4, ROUNDS>(ids, p.M, lane, r.counts, r.offsets, r.scatter, r.gather, r.gate_idx);
      else sort_routes<8, ROUNDS>(ids, p.M, lane, r.counts, r.offsets, r.scatter, r.gather, r.gate_idx);
    }
  } else {
    // ---------------- decoders, then epilogue ----------------
    // This thread decodes, of K-block `par` of every chunk, row r of the tile: all 64 codes with 128 rows, half `hh` of them with 64.
    // Rows g and g + 8 of 16 are out-features 2g and 2g + 1 there, so that the epilogue's threads end up with neighbours.
    constexpr int WORDS = BM / 32;                                 // words of 16 codes
    const int par = (warp - DEC_WARP0) >> 2, idx = ((warp - DEC_WARP0) & 3) * 32 + lane;
    const int r = idx % BM, hh = idx / BM;
    const int feat = BM == 128 ? r : (r & ~15) + 2 * (r & 7) + ((r >> 3) & 1);
    const uint8_t* wrow = nullptr;
    float alpha = 0.f;
    auto weights_of = [&](const Items& it) {
      wrow = p.w + (size_t(it.grp) * p.N + size_t(it.ft) * BM + feat) * (size_t(p.K) / 4) + par * 16 + hh * 8;
      alpha = 0.5f * __ldg(p.alpha + size_t(it.grp) * (p.N / p.alpha_rows) + (it.ft * BM) / p.alpha_rows);   // codes decode to +-2
    };
    const uint32_t swz = uint32_t(r & 7);
    struct Codes { uint32_t w[WORDS]; };
    Codes code[SLOTS];
    auto load_codes = [&](int u, int c) {
      const uint8_t* src = wrow + size_t(c * CK) * 16;
      if constexpr (WORDS == 4) {
        const uint4 v = c < n_ch ? __ldg(reinterpret_cast<const uint4*>(src)) : make_uint4(0u, 0u, 0u, 0u);
        code[u].w[0] = v.x; code[u].w[1] = v.y; code[u].w[2] = v.z; code[u].w[3] = v.w;
      } else {
        const uint2 v = c < n_ch ? __ldg(reinterpret_cast<const uint2*>(src)) : make_uint2(0u, 0u);
        code[u].w[0] = v.x; code[u].w[1] = v.y;
      }
    };
    auto put = [&](const Codes& cw, uint8_t* arow) {       // codes -> (its half of) a swizzled 128-byte row
#pragma unroll
      for (int wi = 0; wi < WORDS; ++wi) {
        uint32_t v[8];
        decode16_prepared(cw.w[wi], v);
        const uint32_t piece = uint32_t(2 * (wi + WORDS * hh));
        *reinterpret_cast<uint4*>(arow + ((piece ^ swz) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<uint4*>(arow + (((piece + 1) ^ swz) << 4)) = make_uint4(v[4], v[5], v[6], v[7]);
      }
    };
    // Chunk c of a tile goes to ring slot and phase of the running count over all tiles; code[c % SLOTS] is its codes.
    int c = 0, s = 0;
    uint32_t ph = 1u;
    bool ok = true;
    auto start_codes = [&]() {
#pragma unroll
      for (int u = 0; u < SLOTS; ++u) load_codes(u, u);
    };
    auto decode_to = [&](int limit, bool fresh) {
#pragma unroll 1
      while (c < limit) {
#pragma unroll
        for (int u = 0; u < SLOTS; ++u) {            // c % SLOTS == u: entered in the middle after an earlier call
          if ((c & (SLOTS - 1)) != u || c >= limit) continue;
          if (!fresh && !mbar_wait(smem_u32(&ctl.empty[s]), ph, abort_flag, p.status, JB200_STATUS_GEMM_DECODE)) { ok = false; c = limit; break; }
          put(code[u], smem + size_t(s) * (CK * A_BYTES) + size_t(par) * A_BYTES + size_t(r) * 128);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&ctl.full[s]));
          load_codes(u, c + SLOTS);
          ++c;
          if (++s == S) { s = 0; ph ^= 1u; }
        }
      }
    };
    const int fresh = S < n_ch ? S : n_ch;           // chunks that go into unused slots
    Items it;
    bool more = it.first(p, ctl, bn);
    if (more) {
      weights_of(it);
      start_codes();
      decode_to(fresh, true);
    }
    __syncwarp();
    pdl_wait();
    pdl_trigger();
    const int q4 = warp & 3;                         // TMEM lane quadrant of this warp
    uint32_t tile = 0u;
    for (; ok && more; more = it.next(p, ctl, bn), ++tile) {
      if (tile > 0) {
        c = 0;
        weights_of(it);
        start_codes();
      }
      decode_to(n_ch, false);
      if (!ok) break;
      const int n = min(bn, it.end - it.tok0), f0 = it.ft * BM + q4 * (BM / 4);
      // The slots of the group's rows in dispatch order, while the last MMAs run: those of all lower groups come first, then rank
      // by token (a token has at most one assignment of a group; without finite logits both are group 0's, and the first is stored).
      constexpr int BLOCKS = MID_ROUTE_TOKENS / 32;
      unsigned first[BLOCKS], second[BLOCKS];          // tokens whose first / second assignment is the group's
      int slot0 = 0;
      if constexpr (ROUTE == 1) {
        int a[BLOCKS], b[BLOCKS];
#pragma unroll
        for (int k = 0; k < BLOCKS; ++k) {
          const int t = 32 * k + lane;
          const longlong2 e = t < p.M ? *reinterpret_cast<const longlong2*>(p.routes.ids + 2 * t) : make_longlong2(MAX_GROUPS, MAX_GROUPS);
          a[k] = max(int(e.x), 0);
          b[k] = max(int(e.y), 0);
        }
#pragma unroll
        for (int k = 0; k < BLOCKS; ++k) {
          if (32 * k >= p.M) { first[k] = second[k] = 0u; continue; }
          first[k] = __ballot_sync(0xffffffffu, a[k] == it.grp);
          second[k] = __ballot_sync(0xffffffffu, b[k] == it.grp);
          slot0 += __popc(__ballot_sync(0xffffffffu, a[k] < it.grp)) + __popc(__ballot_sync(0xffffffffu, b[k] < it.grp));
        }
      }
      if (!mbar_wait(smem_u32(&ctl.acc_full), tile & 1u, abort_flag, p.status, JB200_STATUS_GEMM_EPILOGUE)) break;
      tc_fence_after_sync();
      __syncwarp();
#pragma unroll 1
      for (int c0 = par * 32; c0 < n; c0 += 64) {
        // output row of token c0 + lane; -1: not stored
        int row = c0 + lane < n ? it.tok0 + c0 + lane : -1;
        if (ROUTE == 3 && row >= 0) {
          const longlong2 e = *reinterpret_cast<const longlong2*>(p.routes.ids + 2 * row);
          const int2 sc = *reinterpret_cast<const int2*>(p.routes.scatter + 2 * row);
          row = e.x == it.grp ? sc.x : (e.y == it.grp ? sc.y : -1);
          if (row >= 2 * p.M) row = -1;
        }
        if constexpr (ROUTE == 1) {
          const int t = it.tok0 + c0 + lane;
          int slot = slot0;
          bool mine = false;
#pragma unroll
          for (int k = 0; k < BLOCKS; ++k) {
            const int d = t - 32 * k;
            const unsigned before = d <= 0 ? 0u : d >= 32 ? 0xffffffffu : (1u << d) - 1u;
            slot += __popc(first[k] & before) + __popc(second[k] & before);
            if (d >= 0 && d < 32) mine = ((first[k] | second[k]) >> d) & 1u;
          }
          row = row >= 0 && mine && slot < 2 * p.M ? slot : -1;
        }
        __syncwarp();
        if constexpr (BM == 128) {
          uint32_t v[32];
          tmem_ld_32x32(tmem + (uint32_t(q4 * 32) << 16) + uint32_t(c0), v);
          tmem_ld_wait();
          if (p.epilogue == JB200_EPI_RESID_F32) {
            // lane = feature: a warp instruction covers 128 bytes of one token's row
            float* o = reinterpret_cast<float*>(p.out) + f0 + lane;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const int rj = __shfl_sync(0xffffffffu, row, j);
              const float val = alpha * __uint_as_float(v[j]);
              if (rj >= 0) asm volatile("red.global.add.f32 [%0], %1;" ::"l"(o + size_t(rj) * p.N), "f"(val) : "memory");
            }
          } else {
            const bool gelu = p.epilogue == JB200_EPI_GELU_BF16;
            const int odd = lane & 1;
            __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(p.out) + f0 + (lane & ~1);
#pragma unroll
            for (int jj = 0; jj < 16; ++jj) {
              float a = alpha * __uint_as_float(v[2 * jj]), b = alpha * __uint_as_float(v[2 * jj + 1]);
              if (gelu) { a = gelu_erf(a); b = gelu_erf(b); }
              const float got = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
              const uint32_t w2 = odd ? pack_bf16x2(got, b) : pack_bf16x2(a, got);   // features (f & ~1, f | 1)
              const int rj = __shfl_sync(0xffffffffu, row, 2 * jj + odd);            // token 2jj (even lanes) / 2jj + 1 (odd)
              if (rj >= 0) *reinterpret_cast<uint32_t*>(o + size_t(rj) * p.N) = w2;
            }
          }
        } else {
          const int feat = f0 + (lane >> 2) * 2, c = lane & 3;
          uint32_t v[16];
          tmem_ld_16x256b_x4(tmem + (uint32_t(q4 * 32) << 16) + uint32_t(c0), v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) {                    // token 8 (j / 2) + 2c + j % 2
            const int rj = __shfl_sync(0xffffffffu, row, 8 * (j >> 1) + 2 * c + (j & 1));
            float a = alpha * __uint_as_float(v[4 * (j >> 1) + (j & 1)]), b = alpha * __uint_as_float(v[4 * (j >> 1) + 2 + (j & 1)]);
            if (p.epilogue == JB200_EPI_RESID_F32) {
              if (rj >= 0)
                asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(reinterpret_cast<float*>(p.out) + size_t(rj) * p.N + feat),
                             "f"(a), "f"(b) : "memory");
            } else {
              if (p.epilogue == JB200_EPI_GELU_BF16) { a = gelu_erf(a); b = gelu_erf(b); }
              if (rj >= 0) *reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(p.out) + size_t(rj) * p.N + feat) = pack_bf16x2(a, b);
            }
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctl.acc_empty));
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, p.tmem_cols);
  }
}

inline int chunk_bytes(int bm, int bn) { return CK * (bm + bn) * BK * 2; }

}  // namespace

int mid_gemm_chunks(int bm, int bn, int K) { return std::min({(224 * 1024) / chunk_bytes(bm, bn), MAX_CHUNKS, K / (BK * CK)}); }

int launch_mid_gemm(const void* x_bf16, int M, int K, const uint8_t* w_prepared, const float* alpha, int alpha_rows, int N, int G,
                    const int32_t* seg, const MidRoutes* routes, int epilogue, void* out, int bm, int bn,
                    int bn_max, cudaStream_t stream) {
  JB_REQUIRE(epilogue == JB200_EPI_BF16 || epilogue == JB200_EPI_GELU_BF16 || epilogue == JB200_EPI_RESID_F32, "mid_gemm: epilogue %d", epilogue);
  JB_REQUIRE(M >= 1 && (bm == 64 || bm == 128) && N % bm == 0 && K % (BK * CK) == 0 && alpha_rows % bm == 0 && bn >= 16 && bn % 16 == 0 &&
                 bn_max >= bn && bn_max <= 256 && bn_max % 16 == 0 &&
                 G >= 1 && G <= MAX_GROUPS,
             "mid_gemm: bad shape (M=%d, N=%d, K=%d, bn=%d)", M, N, K, bn);
  MidParams p;
  p.w = w_prepared; p.alpha = alpha; p.seg = seg; p.routes = routes ? *routes : MidRoutes{}; p.out = out;
  p.M = M; p.N = N; p.K = K; p.G = G; p.n_ft = N / bm; p.alpha_rows = alpha_rows; p.epilogue = epilogue;
  const bool cut = seg || p.routes.segments, given = routes && routes->given;
  JB_REQUIRE(!routes || given || (!seg && (G == 4 || G == 8) && M <= (cut ? 2 : 1) * MID_ROUTE_TOKENS && (p.routes.scatter == nullptr) == cut),
             "mid_gemm: %d rows by %d groups cannot be routed here", M, G);
  p.tmem_cols = bn_max <= 32 ? 32u : bn_max <= 64 ? 64u : bn_max <= 128 ? 128u : 256u;
  p.status = device_status_ptr();
  if (!p.status) return JB200_ERR_CUDA;
  const int n_kb = K / BK;
  Maps maps;                                   // [K-block][token][64]: one copy takes the same rows of CK K-blocks
  const cuuint64_t gdim[3] = {cuuint64_t(BK), cuuint64_t(M), cuuint64_t(n_kb)};
  const cuuint64_t gstride[2] = {cuuint64_t(K) * 2, cuuint64_t(BK) * 2};
  size_t smem = 0;
  for (int i = 0; i < 3; ++i) {
    p.bn[i] = i == 0 ? bn : i == 1 ? (bn + bn_max) / 32 * 16 : bn_max;
    p.chunks[i] = mid_gemm_chunks(bm, p.bn[i], K);
    smem = std::max(smem, size_t(p.chunks[i]) * chunk_bytes(bm, p.bn[i]) + 1024);
    const cuuint32_t box[3] = {cuuint32_t(BK), cuuint32_t(p.bn[i]), cuuint32_t(CK)};
    const int rc = encode_tiled(&maps.x[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, x_bf16, gdim, gstride, box,
                                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, "mid_gemm");
    if (rc != JB200_OK) return rc;
  }
  const int sms = sm_count();
  if (sms <= 0) return JB200_ERR_CUDA;
  const long tiles = cut ? (M + bn - 1) / bn + G - 1 : long(G) * ((M + bn - 1) / bn), items = tiles * p.n_ft;   // at most
  const dim3 grid(unsigned(items < sms ? items : sms));
  const int route = !routes ? 0 : given ? 3 : cut ? 2 : 1;
  auto launch = [&](auto kernel, std::atomic<unsigned long long>* set_up) {
    const int rc = set_max_smem(reinterpret_cast<const void*>(kernel), 225 * 1024, set_up);
    if (rc == JB200_OK) launch_dep(kernel, grid, route == 1 ? THREADS + 32 : THREADS, smem, stream, maps, p);
    return rc;
  };
  static std::atomic<unsigned long long> set_up[8];
  int rc;
  if (bm == 64)
    rc = route == 0   ? launch(mid_gemm_kernel<64, 0>, set_up)
         : route == 1 ? launch(mid_gemm_kernel<64, 1>, set_up + 1)
         : route == 2 ? launch(mid_gemm_kernel<64, 2>, set_up + 2)
                      : launch(mid_gemm_kernel<64, 3>, set_up + 3);
  else
    rc = route == 0   ? launch(mid_gemm_kernel<128, 0>, set_up + 4)
         : route == 1 ? launch(mid_gemm_kernel<128, 1>, set_up + 5)
         : route == 2 ? launch(mid_gemm_kernel<128, 2>, set_up + 6)
                      : launch(mid_gemm_kernel<128, 3>, set_up + 7);
  if (rc != JB200_OK) return rc;
  JB_LAUNCH_CHECK("mid_gemm_kernel");
  return JB200_OK;
}

}  // namespace jb
