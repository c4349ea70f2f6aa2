// Ternary linear layers for up to a few hundred tokens on the 5th-generation tensor cores: the latency form of
// ternary_gemm_kernel.
//
// With one or two tiles per SM nothing amortises a pipeline's fill: ternary_gemm_kernel takes 11-18 us for products whose
// arithmetic is ~1 us, because every K-block of its four-stage ring waits for a code load from L2, the decode, the MMA
// and the stage's release one after another (~550 cycles), after TMEM, barriers and tensor maps have been set up.  Here
//   - the work is a list of (token tile, out-feature tile) items that every CTA reads off the segment offsets; those were
//     complete before the kernel ahead on the stream began, so a CTA knows its weights at once and decodes them into every
//     stage there is before the grid dependency is waited for;
//   - the weights are the MMA's A operand in TENSOR memory: a K = 16 step of N tokens takes 10 + N / 2 cycles, where 128 rows read from
//     shared memory cost 43 + N / 2 and 64 rows 27 + N / 2 (48 tokens: 34 against 67 and 51).  What the accumulator leaves of the
//     512 columns and the rows of shared memory hold fourteen K-blocks of up to 64 rows, of 128, 160 and 256 rows (K = 1024) ten, eight and
//     four (mid_gemm_ring): of K = 1024 and small tiles nearly all is decoded ahead, when no MMA is in the way of the stores;
//   - K-blocks travel in chunks of CK: one TMA copy, one barrier wait and one commit per chunk (~290, ~85 and ~45 cycles,
//     none of which hides behind MMAs: issuing them takes as long as they do), with as many chunks in flight as fit: four K-blocks a
//     chunk where three of them do, else two (24 layers and head with two -> four: 17, 37, 64, 128, 256 tokens 677 -> 654, 697 -> 675,
//     745 -> 712, 866 -> 841, 1062 -> 1030 us; with a ring of two or one 900 tokens 1694 -> 1784; counted at run time +1.5 %);
//   - codes come by TMA, all at once up to K = 2048, in rows of 128 bytes;
//   - the eight decoder warps become the epilogue; the residual is added by reductions, nothing waits for old values.  Weight
//     rows are dealt to lanes so that a thread finds four neighbouring out-features of a token: 8- and 16-byte stores, no shuffles.
// Weights from shared memory, in tiles of 64 or 128 out-features and with codes in registers -> in tensor memory, in chunks of two, and
// nothing else changed: 24 layers and head as a graph 881 -> 779 us at 37 tokens, 1096 -> 904 at 128, 1360 -> 1181 at 256, 2068 -> 1849 at 900, steps
// of 64 and 256 sequences 958 -> 878 and 1699 -> 1533.  (The chunks of four above were measured after router, dispatch and tails had become shorter.)
// What is left: the first copy's way (0.5 us after the dependency), 0.17-0.2 us for two K-blocks, epilogue and the end of the grid (0.6 and
// 0.6-0.9 us), and where the kernel ahead is short, decoding (0.14 us a K-block).  Not kept: sixteen decoder warps (180 to 512 tokens 2-3 %
// slower: their registers are not free while the kernel ahead runs), one look at all barriers in place of a wait each, commits left out, a pass
// through MMA loop and epilogue before the dependency (each +1-3 %), a box of codes stored in one go (+2 %).
// Accumulation is the same chain of K = 16 steps as in ternary_gemm_kernel: results are its bit for bit.
#include <algorithm>

#include "common.cuh"
#include "gemm_shared.cuh"
#include "launchers.h"
#include "row_math.cuh"

namespace jb {

namespace {

constexpr int BM = 128, BK = 64;               // out-features of a tile, K of a block
constexpr int CK_MOST = 4;                     // K-blocks per chunk: four, or two where the ring would be too coarse
constexpr int MAX_CHUNKS = 8, DEC_WARP0 = 2, CODE_WARP = 10, MAP_WARP = 11, THREADS = 32 * (CODE_WARP + 1);
constexpr int BOX_KB = 8, BOX_BYTES = BM * BOX_KB * 16, MAX_BOXES = 4;      // codes of eight K-blocks a copy, 128 bytes a row
constexpr uint32_t TMEM_COLS = 512, KB_COLS = BK / 2;                       // a K-block of weights: a bf16 pair per column

struct MidParams {
  const float* alpha;          // [G][N / alpha_rows]
  const int32_t* seg;          // device [G+1] or null (every group takes rows [0, M), or the segments are given by counts or routes)
  const int32_t* counts;       // device [G] or null: their lengths, where the kernel ahead makes the offsets
  MidRoutes routes;
  void* out;
  int M, N, K, G, n_ft, alpha_rows, epilogue;
  int bn[3], chunks[3];        // token tiles and their rings: the first whose items are one wave, else the last
  int boxes;                   // of the ring of codes
  unsigned int* status;
};

struct Maps {
  CUtensorMap x[3];            // one box per token tile
  CUtensorMap w;               // the packed codes
};

// A launch fetches its code anew, and a few microseconds long it feels every kilobyte of it: what is rarely run is a call.
__device__ __noinline__ bool wait_long(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, unsigned int* status, unsigned int code) {
  return mbar_wait(bar, parity, abort_flag, status, code);
}
__device__ __forceinline__ bool wait_for(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, unsigned int* status, unsigned int code) {
  return mbar_try_wait(bar, parity) || wait_long(bar, parity, abort_flag, status, code);
}

struct Ctl {
  uint64_t full[MAX_CHUNKS], empty[MAX_CHUNKS], acc_full, acc_empty, code_full[MAX_BOXES], code_empty[MAX_BOXES];
  uint32_t tmem_base, abort_flag;
  int pick;
  int32_t beg[MAX_GROUPS], end[MAX_GROUPS], first[MAX_GROUPS + 1];   // a group's rows and its first token tile
};

// The items of a CTA: a token tile (rows [tok0, end) of group grp, at most bn of them) and an out-feature tile, the latter
// varying fastest.  The first one is worked out before the grid dependency is waited for.
struct Items {
  int i, grp, tok0, end, ft;
};
// Group, out-feature tile (16 bits) and first row of item i, packed; all bits where there is none.
__device__ __noinline__ unsigned long long item_at(int i, const Ctl* ctl, int G, int n_ft, int bn) {
  if (i >= ctl->first[G] * n_ft) return ~0ull;
  const int t = i / n_ft, ft = i - t * n_ft;
  int g = 0;
  while (t >= ctl->first[g + 1]) ++g;
  return (unsigned long long)(ctl->beg[g] + (t - ctl->first[g]) * bn) << 32 | unsigned(g << 16 | ft);
}

// 32 columns of a warp's 32 lanes from registers; and 16 columns into them.
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
// 16 lanes x 16 columns: thread (g, c) of 8 x 4 receives of lanes g (v[4j], v[4j + 1]) and g + 8 (v[4j + 2], v[4j + 3]) the columns
// 8j + 2c and 8j + 2c + 1.
__device__ __forceinline__ void tmem_ld_16x256b_x2(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}

__host__ __device__ constexpr int acc_cols(int bn) { return (bn + 63) / 64 * 64; }      // the ring of weights begins there

// ROUTE: 0 rows or segments as given, 1 rows stored in dispatch order and the maps left by a warp of their own, 2 segments counted from
// the ids (kernels of their own: the code of the others costs a plain call 1 %).
template <int ROUTE, int CK>
__global__ void __launch_bounds__(ROUTE == 1 ? THREADS + 32 : THREADS, 1)
mid_gemm_kernel(const __grid_constant__ Maps maps, const MidParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ Ctl ctl;
  __shared__ int s_rows[ROUTE == 1 ? 8 : 1][MID_ROUTE_TOKENS / 2];     // an epilogue warp's output rows
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  const int warp = warp_index(), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < MAX_CHUNKS; ++s) {
      mbar_init(smem_u32(&ctl.full[s]), 1 + 8);      // the producer's expectation and the eight decoder warps
      mbar_init(smem_u32(&ctl.empty[s]), 1);
    }
    mbar_init(smem_u32(&ctl.acc_full), 1);
    mbar_init(smem_u32(&ctl.acc_empty), 8);
    for (int b = 0; b < MAX_BOXES; ++b) {
      mbar_init(smem_u32(&ctl.code_full[b]), 1);
      mbar_init(smem_u32(&ctl.code_empty[b]), 8);
    }
    ctl.abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&maps.w);
    tma_prefetch_desc(&maps.x[0]);
  }
  if (warp == 0) {
    __syncwarp();                 // tcgen05.alloc is warp-collective: lane 0 rejoins from the barrier set-up first
    tmem_alloc(smem_u32(&ctl.tmem_base), TMEM_COLS);
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
    if (ROUTE == 2 || p.counts) {              // the kernel ahead makes the offsets; ids and counts are older
      int n_of = 0;
      if constexpr (ROUTE == 2) {
        constexpr int ROUNDS = 2 * MID_ROUTE_TOKENS / 32;
        int ex[ROUNDS];
#pragma unroll
        for (int i = 0; i < ROUNDS; ++i) ex[i] = i * 32 + lane < p.M ? max(int(p.routes.ids[i * 32 + lane]), 0) : -1;
        for (int q = 0; q < p.G; ++q) {
          int n = 0;
#pragma unroll
          for (int i = 0; i < ROUNDS; ++i) n += __popc(__ballot_sync(0xffffffffu, ex[i] == q));
          if (lane == q) n_of = n;
        }
      } else if (lane < p.G) {
        n_of = max(__ldg(p.counts + lane), 0);
      }
      end = n_of;
      for (int d = 1; d < MAX_GROUPS; d *= 2) {
        const int u = __shfl_up_sync(0xffffffffu, end, d);
        if (lane >= d) end += u;
      }
      beg = min(end - n_of, p.M);
      end = min(end, p.M);
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
  const uint32_t tmem = __shfl_sync(0xffffffffu, ctl.tmem_base, 0);       // in uniform registers, as the votes below
  volatile uint32_t* abort_flag = &ctl.abort_flag;
  // votes: their results are in uniform registers, which copies and MMAs are issued from (a value read from shared memory
  // there cost 1.8 us a launch)
  const bool t1 = __any_sync(0xffffffffu, ctl.pick == 1), t2 = __any_sync(0xffffffffu, ctl.pick == 2);
  const int bn = t2 ? p.bn[2] : t1 ? p.bn[1] : p.bn[0], n_ch = p.K / (BK * CK);
  const int S = t2 ? p.chunks[2] : t1 ? p.chunks[1] : p.chunks[0];
  const uint32_t kb_bytes = uint32_t(bn) * BK * 2, b_bytes = kb_bytes * uint32_t(CK);
  const uint32_t b_base = base + uint32_t(p.boxes) * BOX_BYTES, a_tmem = tmem + uint32_t(acc_cols(bn));
  const CUtensorMap* tmap_x = t2 ? &maps.x[2] : t1 ? &maps.x[1] : &maps.x[0];
  auto item = [&](Items& it, int i) {
    const unsigned long long r = item_at(i, &ctl, p.G, p.n_ft, bn);
    if (r == ~0ull) return false;
    it.i = i;
    it.grp = int(r >> 16) & 0xffff;
    it.ft = int(r) & 0xffff;
    it.tok0 = int(r >> 32);
    it.end = ctl.end[it.grp];
    return true;
  };
  if (warp == 0) {
    // ---------------- TMA producer ----------------
    Items it;
    bool more = item(it, blockIdx.x);
    pdl_wait();
    pdl_trigger();
    int s = 0;
    uint32_t ph = 1u;
    bool ok = true;
    for (; ok && more; more = item(it, it.i + gridDim.x)) {
#pragma unroll 1
      for (int c = 0; c < n_ch; ++c) {
        const uint32_t full = smem_u32(&ctl.full[s]);
        if (!wait_for(smem_u32(&ctl.empty[s]), ph, abort_flag, p.status, JB200_STATUS_GEMM_PRODUCER)) { ok = false; break; }
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
    bool more = item(it, blockIdx.x);
    pdl_wait();
    pdl_trigger();
    const uint32_t idesc = umma_idesc_bf16(BM, bn);
    const uint64_t bdesc0 = umma_desc_k_sw128(b_base);
    uint64_t bd = bdesc0;
    uint32_t at = a_tmem;
    int s = 0;
    uint32_t ph = 0u, tile = 0u;
    bool ok = true;
    for (; ok && more; more = item(it, it.i + gridDim.x), ++tile) {
      if (!wait_for(smem_u32(&ctl.acc_empty), (tile & 1u) ^ 1u, abort_flag, p.status, JB200_STATUS_GEMM_MMA)) break;
      tc_fence_after_sync();
#pragma unroll 1
      for (int c = 0; c < n_ch; ++c) {
        if (!wait_for(smem_u32(&ctl.full[s]), ph, abort_flag, p.status, JB200_STATUS_GEMM_MMA)) { ok = false; break; }
        tc_fence_after_sync();
        if (elect_one()) {
#pragma unroll
          for (int j = 0; j < CK; ++j) {
            const uint64_t bj = bd + uint64_t(j) * (kb_bytes >> 4);
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk)
              umma_bf16_ts(tmem, at + uint32_t(j * KB_COLS + kk * 8), bj + uint64_t(kk * 2), idesc, (c | j | kk) != 0 ? 1u : 0u);
          }
          umma_commit(smem_u32(&ctl.empty[s]));
          if (c + 1 == n_ch) umma_commit(smem_u32(&ctl.acc_full));
        }
        __syncwarp();
        at += CK * KB_COLS;
        bd += b_bytes >> 4;
        if (++s == S) { s = 0; ph ^= 1u; at = a_tmem; bd = bdesc0; }
      }
    }
  } else if (warp == CODE_WARP) {
    // ---------------- codes, as far ahead of the decoders as their ring holds ----------------
    Items it;
    int s = 0;
    uint32_t ph = 1u;
    bool ok = true;
    for (bool more = item(it, blockIdx.x); ok && more; more = item(it, it.i + gridDim.x)) {
#pragma unroll 1
      for (int k = 0; k < p.K / 4; k += BOX_KB * 16) {
        const uint32_t full = smem_u32(&ctl.code_full[s]);
        if (!wait_for(smem_u32(&ctl.code_empty[s]), ph, abort_flag, p.status, JB200_STATUS_GEMM_PRODUCER)) { ok = false; break; }
        if (elect_one()) {
          mbar_arrive_expect_tx(full, BOX_BYTES);
          tma_load_2d(base + uint32_t(s) * BOX_BYTES, &maps.w, k, it.grp * p.N + it.ft * BM, full);
        }
        __syncwarp();
        if (++s == p.boxes) { s = 0; ph ^= 1u; }
      }
    }
    pdl_wait();
    pdl_trigger();
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
    // This thread decodes, of every other K-block from `par` on, the 64 codes of the out-feature that its lane of tensor memory holds.
    // Lanes g, g + 8, g + 16 and g + 24 of a warp's 32 are four neighbours, so that a thread of the epilogue has them together; which
    // of the four is turned by g / 2, for eight lanes' codes in eight different bank groups.
    const int par = (warp - DEC_WARP0) >> 2, q4 = warp & 3;                          // q4: the lanes this warp can reach
    const int r = q4 * 32 + 4 * (lane & 7) + ((lane >> 3) ^ ((lane & 7) >> 1));
    const uint32_t code_row = base + uint32_t(r) * (BOX_KB * 16), a_lane = a_tmem + (uint32_t(q4) << 21) + uint32_t(par) * KB_COLS;
    // Chunk c of a tile goes to ring slot and phase of the running count over all tiles.
    int c = 0, s = 0, box = 0;
    uint32_t ph = 1u, box_ph = 0u;
    bool ok = true;
    constexpr int BOX_CHUNKS = BOX_KB / CK;
    auto decode_to = [&](int limit, bool fresh) {
#pragma unroll 1
      for (; c < limit; ++c) {
        const int in_box = c & (BOX_CHUNKS - 1);
        if (in_box == 0 && !wait_for(smem_u32(&ctl.code_full[box]), box_ph, abort_flag, p.status, JB200_STATUS_GEMM_DECODE)) { ok = false; return; }
        if (!fresh) {
          if (!wait_for(smem_u32(&ctl.empty[s]), ph, abort_flag, p.status, JB200_STATUS_GEMM_DECODE)) { ok = false; return; }
          tc_fence_after_sync();
          __syncwarp();
        }
#pragma unroll 1
        for (int h = 0; h < CK; h += 2) {
          uint32_t w[4], v[32];
          const uint32_t piece = uint32_t(in_box * CK + h + par) ^ uint32_t(r & 7);       // 128-byte swizzle: no bank conflicts
          asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(code_row + uint32_t(box) * BOX_BYTES + (piece << 4)) : "memory");
#pragma unroll
          for (int i = 0; i < 4; ++i) decode16_prepared(w[i], v + 8 * i);
          tmem_st_32x32(a_lane + uint32_t(s * CK + h) * KB_COLS, v);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctl.full[s]));
        if (++s == S) { s = 0; ph ^= 1u; }
        if (in_box == BOX_CHUNKS - 1 || c + 1 == n_ch) {          // the box has been read
          if (lane == 0) mbar_arrive(smem_u32(&ctl.code_empty[box]));
          if (++box == p.boxes) { box = 0; box_ph ^= 1u; }
        }
      }
    };
    float alpha = 0.f;
    auto scale_of = [&](const Items& it) {         // codes decode to +-2
      alpha = 0.5f * __ldg(p.alpha + size_t(it.grp) * (p.N / p.alpha_rows) + (it.ft * BM) / p.alpha_rows);
    };
    const int fresh = S < n_ch ? S : n_ch;           // chunks that go into unused slots
    Items it;
    bool more = item(it, blockIdx.x);
    if (more) {
      scale_of(it);
      decode_to(fresh, true);
    }
    __syncwarp();
    pdl_wait();
    pdl_trigger();
    uint32_t tile = 0u;
    for (; ok && more; more = item(it, it.i + gridDim.x), ++tile) {
      if (tile > 0) {
        c = 0;
        scale_of(it);
      }
      decode_to(n_ch, false);
      if (!ok) break;
      const int n = min(bn, it.end - it.tok0), f0 = it.ft * BM + q4 * 32;
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
      // Of 32 tokens, 16 are this warp's (those of its K-block's parity): lane % 16 holds the output row of one of them, -1 for none.
      const int t0 = 16 * par + (lane & 15);
      if constexpr (ROUTE == 1) {
        int* rows = s_rows[warp - DEC_WARP0];
#pragma unroll 1
        for (int b = 0; 32 * b < n; ++b) {
          const int t = it.tok0 + 32 * b + t0;
          int slot = slot0;
          bool mine = false;
#pragma unroll
          for (int k = 0; k < BLOCKS; ++k) {
            const int d = t - 32 * k;
            const unsigned before = d <= 0 ? 0u : d >= 32 ? 0xffffffffu : (1u << d) - 1u;
            slot += __popc(first[k] & before) + __popc(second[k] & before);
            if (d >= 0 && d < 32) mine = ((first[k] | second[k]) >> d) & 1u;
          }
          if (lane < 16) rows[16 * b + lane] = 32 * b + t0 < n && mine && slot < 2 * p.M ? slot : -1;
        }
        __syncwarp();
      }
      if (!wait_for(smem_u32(&ctl.acc_full), tile & 1u, abort_flag, p.status, JB200_STATUS_GEMM_EPILOGUE)) break;
      tc_fence_after_sync();
      __syncwarp();
      const int g = lane >> 2, turn = g >> 1, feat = f0 + 4 * g;
      const uint32_t halves = (turn & 1) ? 0x1032u : 0x3210u;
#pragma unroll 1
      for (int b = 0; 32 * b + 16 * par < n; ++b) {
        uint32_t v[2][8];
        const uint32_t at = tmem + (uint32_t(q4) << 21) + uint32_t(32 * b + 16 * par);
        tmem_ld_16x256b_x2(at, v[0]);
        tmem_ld_16x256b_x2(at + (16u << 16), v[1]);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 4; ++q) {                              // token 8 (q / 2) + 2 (lane % 4) + q % 2 of the 16
          const int t = 8 * (q >> 1) + 2 * (lane & 3) + (q & 1);
          int row = 32 * b + 16 * par + t < n ? it.tok0 + 32 * b + 16 * par + t : -1;
          if constexpr (ROUTE == 1) row = s_rows[warp - DEC_WARP0][16 * b + t];
          const int k = 4 * (q >> 1) + (q & 1);
          uint64_t y0 = mul_f32x2(f32x2(__uint_as_float(v[0][k]), __uint_as_float(v[0][k + 2])), f32x2(alpha, alpha));
          uint64_t y1 = mul_f32x2(f32x2(__uint_as_float(v[1][k]), __uint_as_float(v[1][k + 2])), f32x2(alpha, alpha));
          float x0, x1, x2, x3;
          if (p.epilogue == JB200_EPI_RESID_F32) {
            const uint64_t lo = (turn & 2) ? y1 : y0, hi = (turn & 2) ? y0 : y1;
            f32x2_split(lo, x0, x1);
            f32x2_split(hi, x2, x3);
            const bool sw = turn & 1;
            if (row >= 0)          // (addends and sums below 2^-126 become zero, as in small_gemm.cu; TMA's reduction keeps them)
              asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                           ::"l"(reinterpret_cast<float*>(p.out) + size_t(row) * p.N + feat), "f"(sw ? x1 : x0), "f"(sw ? x0 : x1),
                             "f"(sw ? x3 : x2), "f"(sw ? x2 : x3) : "memory");
          } else {
            if (p.epilogue == JB200_EPI_GELU_BF16) {
              y0 = gelu_erf_x2(y0);
              y1 = gelu_erf_x2(y1);
            }
            f32x2_split(y0, x0, x1);
            f32x2_split(y1, x2, x3);
            const uint32_t w0 = __byte_perm(pack_bf16x2(x0, x1), 0u, halves), w1 = __byte_perm(pack_bf16x2(x2, x3), 0u, halves);
            if (row >= 0)
              *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.out) + size_t(row) * p.N + feat) =
                  (turn & 2) ? make_uint2(w1, w0) : make_uint2(w0, w1);
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
    tmem_dealloc(tmem, TMEM_COLS);
  }
}

constexpr int RING_SMEM = 222 * 1024, RING_LEAST = 3;
inline int chunk_bytes(int bn, int ck) { return ck * bn * BK * 2; }
inline int code_boxes(int K) { return std::min((K + BOX_KB * BK - 1) / (BOX_KB * BK), MAX_BOXES); }
constexpr size_t LEAST_SMEM = 116 * 1024;      // two CTAs of an SM would only wait for each other's tensor memory

}  // namespace

// Chunks in flight: weights in what the accumulator leaves of tensor memory, rows in what the codes leave of shared memory.
MidRing mid_gemm_ring(int bn, int K, bool coarse) {
  const int ck = coarse ? CK_MOST : 2;
  MidRing r = {0, ck, 0, 0};
  if (K % (BK * ck) != 0) return r;
  r.chunks = std::min({(int(TMEM_COLS) - acc_cols(bn)) / int(ck * KB_COLS), (RING_SMEM - code_boxes(K) * BOX_BYTES) / chunk_bytes(bn, ck),
                       MAX_CHUNKS, K / (BK * ck)});
  r.tmem_cols = acc_cols(bn) + r.chunks * ck * int(KB_COLS);
  r.smem = code_boxes(K) * BOX_BYTES + r.chunks * chunk_bytes(bn, ck) + 1024;       // the base is rounded up to 1024
  return r;
}

bool mid_gemm_coarse_fits(int bn, int K) { return mid_gemm_ring(bn, K, true).chunks >= RING_LEAST; }

int launch_mid_gemm(const void* x_bf16, int M, int K, const uint8_t* w_prepared, const float* alpha, int alpha_rows, int N, int G,
                    const int32_t* seg, const int32_t* counts, const MidRoutes* routes, int epilogue, void* out, int bn, int bn_max,
                    bool coarse, cudaStream_t stream) {
  JB_REQUIRE(epilogue == JB200_EPI_BF16 || epilogue == JB200_EPI_GELU_BF16 || epilogue == JB200_EPI_RESID_F32, "mid_gemm: epilogue %d", epilogue);
  JB_REQUIRE(M >= 1 && N % BM == 0 && K % (BK * 2) == 0 && alpha_rows % BM == 0 && bn >= 16 && bn % 16 == 0 &&
                 bn_max >= bn && bn_max <= 256 && bn_max % 16 == 0 &&
                 G >= 1 && G <= MAX_GROUPS && (!coarse || mid_gemm_coarse_fits(bn_max, K)),
             "mid_gemm: bad shape (M=%d, N=%d, K=%d, bn=%d)", M, N, K, bn);
  MidParams p;
  p.alpha = alpha; p.seg = seg; p.counts = counts; p.routes = routes ? *routes : MidRoutes{}; p.out = out;
  p.M = M; p.N = N; p.K = K; p.G = G; p.n_ft = N / BM; p.alpha_rows = alpha_rows; p.epilogue = epilogue;
  const bool cut = seg || counts || p.routes.segments;
  JB_REQUIRE(!routes || (!seg && (G == 4 || G == 8) && M <= (cut ? 2 : 1) * MID_ROUTE_TOKENS && (p.routes.scatter == nullptr) == cut),
             "mid_gemm: %d rows by %d groups cannot be routed here", M, G);
  p.boxes = code_boxes(K);
  p.status = device_status_ptr();
  if (!p.status) return JB200_ERR_CUDA;
  const int n_kb = K / BK;
  int ck = 2;
  Maps maps;                                   // [K-block][token][64]: one copy takes the same rows of ck K-blocks
  const cuuint64_t gdim[3] = {cuuint64_t(BK), cuuint64_t(M), cuuint64_t(n_kb)};
  const cuuint64_t gstride[2] = {cuuint64_t(K) * 2, cuuint64_t(BK) * 2};
  size_t smem = LEAST_SMEM;
  for (int i = 0; i < 3; ++i) {
    p.bn[i] = i == 0 ? bn : i == 1 ? (bn + bn_max) / 32 * 16 : bn_max;
    const MidRing ring = mid_gemm_ring(p.bn[i], K, coarse);
    ck = ring.kb;
    p.chunks[i] = ring.chunks;
    smem = std::max(smem, size_t(ring.smem));
    if (i > 0 && p.bn[i] == p.bn[i - 1]) {
      maps.x[i] = maps.x[i - 1];
      continue;
    }
    const cuuint32_t box[3] = {cuuint32_t(BK), cuuint32_t(p.bn[i]), cuuint32_t(ck)};
    const int rc = encode_tiled(&maps.x[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, x_bf16, gdim, gstride, box,
                                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, "mid_gemm");
    if (rc != JB200_OK) return rc;
  }
  const cuuint64_t wdim[2] = {cuuint64_t(K) / 4, cuuint64_t(G) * N}, wstride[1] = {cuuint64_t(K) / 4};
  const cuuint32_t wbox[2] = {BOX_KB * 16, BM};
  const int rcw = encode_tiled(&maps.w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, w_prepared, wdim, wstride, wbox, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, "mid_gemm (weights)");
  if (rcw != JB200_OK) return rcw;
  const int sms = sm_count();
  if (sms <= 0) return JB200_ERR_CUDA;
  const long tiles = cut ? (M + bn - 1) / bn + G - 1 : long(G) * ((M + bn - 1) / bn), items = tiles * p.n_ft;   // at most
  const dim3 grid(unsigned(items < sms ? items : sms));
  const int route = !routes ? 0 : cut ? 2 : 1;
  auto launch = [&](auto kernel, std::atomic<unsigned long long>* set_up) {
    const int rc = set_max_smem(reinterpret_cast<const void*>(kernel), RING_SMEM + 1024, set_up);
    if (rc == JB200_OK) launch_dep(kernel, grid, route == 1 ? THREADS + 32 : THREADS, smem, stream, maps, p);
    return rc;
  };
  static std::atomic<unsigned long long> set_up[6];
  auto pick = [&](auto two, auto four, std::atomic<unsigned long long>* done) { return ck == 2 ? launch(two, done) : launch(four, done + 1); };
  const int rc = route == 0   ? pick(mid_gemm_kernel<0, 2>, mid_gemm_kernel<0, 4>, set_up)
                 : route == 1 ? pick(mid_gemm_kernel<1, 2>, mid_gemm_kernel<1, 4>, set_up + 2)
                              : pick(mid_gemm_kernel<2, 2>, mid_gemm_kernel<2, 4>, set_up + 4);
  if (rc != JB200_OK) return rc;
  JB_LAUNCH_CHECK("mid_gemm_kernel");
  return JB200_OK;
}

}  // namespace jb
