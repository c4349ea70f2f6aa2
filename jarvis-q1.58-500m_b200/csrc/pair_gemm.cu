// Ternary linear layers for many tokens: CTA pairs on the 5th-generation tensor cores.
//
// ternary_gemm_kernel's SM moves, per 64-wide K-block of a 128 x 256 tile, 16 KiB of decoded weights and 32 KiB of
// activations into shared memory and reads them back for the MMAs: about 850 cycles of shared-memory pipe for 512 cycles
// of tensor pipe.  Here two SMs work on one tile of 256 tokens x 256 out-features (tcgen05.mma.cta_group::2): each holds
// 128 tokens, decodes half of the weights and accumulates its tokens' rows, 64 KiB through each SM's shared memory per
// K-block instead of 96, and L2 delivers every operand once per pair.
//
// The activations are the M operand, so a TMEM lane is a token and an epilogue thread finds 32 consecutive out-features of
// its token in registers: they leave as 32-byte stores without any exchange between lanes (weights as the M operand cost
// ~200 instructions per 32 x 32 chunk against ~40, and the decoders wait for the same issue slots).  A last wave that is at
// most half (a quarter) full is cut into tiles of half (a quarter of) the width.
//
// The pair's leader (cluster rank 0) issues every MMA.  Its `full` barriers count its own and the peer's decoder warps
// (remote arrivals) and the bytes of both CTAs' TMA loads; `empty` and `acc_full` are committed to both CTAs; `acc_empty`
// counts both CTAs' epilogue warps.  Loops that issue copies or MMAs are run by a whole warp (elect_one).
// Accumulation is the same chain of K = 16 steps as in the one-CTA kernels: results are theirs bit for bit.
#include "common.cuh"
#include "gemm_shared.cuh"
#include "launchers.h"

namespace jb {

namespace {

constexpr int BM = 128, BK = 64, BN = 256;             // tokens per CTA (256 per pair), K per stage, out-features per tile
constexpr int A_BYTES = BM * BK * 2;                   // 16 KiB: this CTA's tokens
constexpr int B_BYTES = (BN / 2) * BK * 2;             // 16 KiB: this CTA's half of the weights
constexpr int CODE_SLOTS = 3, CODE_KB = 4, CODE_BYTES = (BN / 2) * CODE_KB * 16;   // ring of codes: four K-blocks, 8 KiB a slot
constexpr int DEC_GROUPS = 2;                          // of four warps, on alternate K-blocks (three or four: 3-8 % slower)
constexpr int CODE_WARP = 2, DEC_WARP0 = 3, EPI_WARP0 = DEC_WARP0 + 4 * DEC_GROUPS, THREADS = 32 * (EPI_WARP0 + 8);
constexpr uint32_t TMEM_COLS = 512;

// The residual form trades one ring stage for a 4 KiB tile per epilogue warp, from which the memory system adds to x.
constexpr int stages(bool resid) { return resid ? 5 : 6; }
constexpr int OUT_BYTES = 32 * 32 * 4;

struct PairCtl {
  uint64_t full[6], empty[6], acc_full[2], acc_empty[2], code_full[CODE_SLOTS], code_empty[CODE_SLOTS];
  uint32_t tmem_base, abort_flag;
  int32_t seg[MAX_GROUPS + 1];
};
constexpr size_t CTL_BYTES = (sizeof(PairCtl) + 127) / 128 * 128;
constexpr size_t smem_bytes(bool resid) {
  return 1024 + size_t(stages(resid)) * (A_BYTES + B_BYTES) + size_t(CODE_SLOTS) * CODE_BYTES + (resid ? 8 * OUT_BYTES : 0) + CTL_BYTES;
}
static_assert(smem_bytes(false) <= 227 * 1024 && smem_bytes(true) <= 227 * 1024, "shared memory of one CTA");

// ---- cta_group::2 forms of the wrappers in common.cuh ----
__device__ __forceinline__ void pair_tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
}
__device__ __forceinline__ void pair_tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void pair_umma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on the barrier at this offset in both CTAs once all previously issued MMAs of this thread retire.
__device__ __forceinline__ void pair_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(uint16_t(3)) : "memory");
}
// Tile load into this CTA whose bytes are counted by a barrier of the pair's leader.
__device__ __forceinline__ void pair_tma_load_2d(uint32_t dst_smem, const void* tmap, int c0, int c1, uint32_t leader_bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst_smem), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(leader_bar) : "memory");
}
// (with .release.cluster every arrival waits for the warp's outstanding memory operations: 1400 cycles per K-block)
__device__ __forceinline__ void cluster_mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait that also orders what the other CTA did before its arrival.
__device__ __forceinline__ bool cluster_mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}"
      : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
__device__ __forceinline__ bool cluster_mbar_wait(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, unsigned int* status,
                                                  unsigned int code) {
  if (cluster_mbar_try(bar, parity)) return true;
  const unsigned long long t0 = globaltimer_ns();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 32; ++i)
      if (cluster_mbar_try(bar, parity)) return true;
    if (*abort_flag) return false;
    if (globaltimer_ns() - t0 > JB_WAIT_LIMIT_NS) {
      *abort_flag = 1u;
      atomicCAS(status, 0u, code);
      return false;
    }
  }
}

__device__ __forceinline__ void st_global_256(void* p, const uint32_t* w) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}
// 32 consecutive out-features of one token: alpha, epilogue, 32-byte accesses.  `o`: element offset of the first.
__device__ __forceinline__ void store_row_chunk(const GemmParams& p, uint32_t (&v)[32], float alpha, size_t o) {
  if (p.epilogue == JB200_EPI_BF16 || p.epilogue == JB200_EPI_GELU_BF16) {
    uint32_t w[16];
    const bool gelu = p.epilogue == JB200_EPI_GELU_BF16;
    const uint64_t al = f32x2(alpha, alpha);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      uint64_t x = mul_f32x2(f32x2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), al);
      if (gelu) x = gelu_erf_x2(x);
      float a, b;
      f32x2_split(x, a, b);
      w[j] = pack_bf16x2(a, b);
    }
    __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(p.out) + o;
    st_global_256(d, w);
    st_global_256(d + 16, w + 8);
    return;
  }
  float* d = reinterpret_cast<float*>(p.out) + o;
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(alpha * __uint_as_float(v[j]));
  if (p.epilogue == JB200_EPI_RESID_F32) {
    // calls with segments (their tiles end inside the matrix, where a tile reduction would not be clipped)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                   ::"l"(d + 4 * j), "f"(__uint_as_float(v[4 * j])), "f"(__uint_as_float(v[4 * j + 1])),
                     "f"(__uint_as_float(v[4 * j + 2])), "f"(__uint_as_float(v[4 * j + 3])) : "memory");
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) st_global_256(d + 8 * j, v + 8 * j);
  }
}

struct PairTile {
  int group, tok0, tok_end, f0, width;      // segment, token rows, out-features [f0, f0 + width)
};
// The tiles of a call: `whole` of full width, then the rest cut into `parts` each.  Out-features vary fastest, so CTAs running
// together share activation tiles through L2.
struct PairPlan {
  int whole, parts, total;
};
__device__ __forceinline__ PairPlan pair_plan(const PairCtl* ctl, int G, int n_fp, int n_pairs) {
  int n = 0;
  for (int g = 0; g < G; ++g) n += (ctl->seg[g + 1] - ctl->seg[g] + 2 * BM - 1) / (2 * BM);
  n *= n_fp;
  const int rest = n % n_pairs;
  const int parts = 4 * rest <= n_pairs ? 4 : 2 * rest <= n_pairs ? 2 : 1;
  return {n - rest, parts, n - rest + rest * parts};
}
__device__ __forceinline__ bool pair_tile(const PairCtl* ctl, const PairPlan& plan, int t, int n_fp, int G, PairTile* c) {
  int part = 0;
  c->width = BN;
  if (t >= plan.whole) {
    const int q = t - plan.whole;
    t = plan.whole + q / plan.parts;
    part = q % plan.parts;
    c->width = BN / plan.parts;
  }
  int tt = t / n_fp;
  c->f0 = (t - tt * n_fp) * BN + part * c->width;
  for (int g = 0; g < G; ++g) {
    const int beg = ctl->seg[g], end = ctl->seg[g + 1];
    const int tiles = (end - beg + 2 * BM - 1) / (2 * BM);
    if (tt < tiles) {
      c->group = g;
      c->tok0 = beg + tt * 2 * BM;
      c->tok_end = end;
      return true;
    }
    tt -= tiles;
  }
  return false;
}

template <bool RESID>
__global__ void __launch_bounds__(THREADS, 1)
pair_gemm_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                 const __grid_constant__ CUtensorMap tmap_out, const __grid_constant__ GemmParams p) {
  constexpr int STAGES = stages(RESID);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t base = (raw_addr + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (base - raw_addr);
  const uint32_t a_base = base, b_base = base + STAGES * A_BYTES;
  const uint32_t code_base = b_base + STAGES * B_BYTES;
  const uint32_t out_base = code_base + CODE_SLOTS * CODE_BYTES;
  PairCtl* ctl = reinterpret_cast<PairCtl*>(smem + (out_base - base) + (RESID ? 8 * OUT_BYTES : 0));

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int rank = int(cluster_rank());
  const int n_kb = p.K / BK, n_fp = (p.N + BN - 1) / BN;
  const bool dense_w = p.w_layout == 2;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&ctl->full[s]), dense_w ? 1 : 1 + 8);     // the leader's expectation, four decoder warps per CTA
      mbar_init(smem_u32(&ctl->empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&ctl->acc_full[a]), 1);
      mbar_init(smem_u32(&ctl->acc_empty[a]), 16);                 // eight epilogue warps per CTA
    }
    for (int c = 0; c < CODE_SLOTS; ++c) {
      mbar_init(smem_u32(&ctl->code_full[c]), 1);
      mbar_init(smem_u32(&ctl->code_empty[c]), 4 * DEC_GROUPS);
    }
    ctl->abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap_x);
    tma_prefetch_desc(&tmap_w);
  }
  if (warp == 0) {
    __syncwarp();                 // tcgen05.alloc is warp-collective: lane 0 rejoins from the barrier set-up first
    pair_tmem_alloc(smem_u32(&ctl->tmem_base), TMEM_COLS);
    pair_tmem_relinquish();
  }
  __syncwarp();
  // In a chain (`settled`) only the activations are the work of the kernel before this one: the warp that loads them waits
  // for it, while codes are loaded and decoded into every stage there is.  All else follows from its loads.
  if (!p.settled) {
    pdl_wait();
    pdl_trigger();
  }
  if (threadIdx.x == 0) {
    if (p.seg_counts) {
      int at = 0;
      for (int g = 0; g < p.G; ++g) {
        ctl->seg[g] = at;
        at = min(at + max(p.seg_counts[g], 0), p.M);
      }
      ctl->seg[p.G] = at;
    } else if (p.seg_offsets) {
      for (int g = 0; g <= p.G; ++g) ctl->seg[g] = min(max(p.seg_offsets[g], 0), p.M);
    } else {
      ctl->seg[0] = 0;
      ctl->seg[1] = p.M;
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  cluster_arrive();               // both CTAs' barriers are initialised before either arrives on the other's
  cluster_wait();
  tc_fence_after_sync();
  const uint32_t tmem = ctl->tmem_base;
  volatile uint32_t* abort_flag = &ctl->abort_flag;
  const int pair = int(blockIdx.x >> 1), n_pairs = int(gridDim.x >> 1);

  const PairPlan plan = pair_plan(ctl, p.G, n_fp, n_pairs);
  const int total = plan.total;

  if (warp == 0) {
    // ---------------- TMA producer: this CTA's tokens (and, dense, its weight rows) ----------------
    if (p.settled) {
      pdl_wait();
      pdl_trigger();
    }
    int s = 0;
    uint32_t ph = 1u;
    bool ok = true;
    PairTile tc;
    for (int t = pair; ok && t < total; t += n_pairs) {
      if (!pair_tile(ctl, plan, t, n_fp, p.G, &tc)) break;
      const int row = tc.tok0 + rank * BM, w_rows = tc.width / 2, wrow = tc.group * p.N + tc.f0 + rank * w_rows;
      const uint32_t bytes = 2u * (uint32_t(A_BYTES) + (dense_w ? uint32_t(w_rows) * BK * 2 : 0u));     // of both CTAs
#pragma unroll 1
      for (int kb = 0; kb < n_kb; ++kb) {
        if (!mbar_wait(smem_u32(&ctl->empty[s]), ph, abort_flag, p.status, JB200_STATUS_GEMM_PRODUCER)) { ok = false; break; }
        const uint32_t full = cluster_map(smem_u32(&ctl->full[s]), 0u);
        if (elect_one()) {
          if (rank == 0) mbar_arrive_expect_tx(smem_u32(&ctl->full[s]), bytes);
          pair_tma_load_2d(a_base + uint32_t(s) * A_BYTES, &tmap_x, kb * BK, row, full);
          if (dense_w) {
            for (int r = 0; r < w_rows; r += 32)
              pair_tma_load_2d(b_base + uint32_t(s) * B_BYTES + uint32_t(r) * BK * 2, &tmap_w, kb * BK, wrow + r, full);
          }
        }
        __syncwarp();
        if (++s == STAGES) { s = 0; ph ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer: the leader's, for both CTAs ----------------
    if (rank == 0) {
      const uint64_t ad0 = umma_desc_k_sw128(a_base), bd0 = umma_desc_k_sw128(b_base);
      uint64_t ad = ad0, bd = bd0;
      int s = 0;
      uint32_t ph = 0u, tile = 0u;
      bool ok = true;
      for (int t = pair; ok && t < total; t += n_pairs, ++tile) {
        const uint32_t acc = tile & 1u;
        const uint32_t idesc = umma_idesc_bf16(2 * BM, t < plan.whole ? BN : BN / plan.parts);
        if (!cluster_mbar_wait(smem_u32(&ctl->acc_empty[acc]), ((tile >> 1) & 1u) ^ 1u, abort_flag, p.status, JB200_STATUS_GEMM_MMA)) break;
        tc_fence_after_sync();
        const uint32_t d = tmem + acc * BN;
#pragma unroll 1
        for (int kb = 0; kb < n_kb; ++kb) {
          if (!cluster_mbar_wait(smem_u32(&ctl->full[s]), ph, abort_flag, p.status, JB200_STATUS_GEMM_MMA)) { ok = false; break; }
          tc_fence_after_sync();
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < BK / 16; ++kk)
              pair_umma(d, ad + uint64_t(kk * 2), bd + uint64_t(kk * 2), idesc, (kb | kk) != 0 ? 1u : 0u);
            pair_commit(smem_u32(&ctl->empty[s]));
            if (kb + 1 == n_kb) pair_commit(smem_u32(&ctl->acc_full[acc]));
          }
          __syncwarp();
          ad += A_BYTES >> 4;
          bd += B_BYTES >> 4;
          if (++s == STAGES) { s = 0; ph ^= 1u; ad = ad0; bd = bd0; }
        }
      }
    }
  } else if (warp == CODE_WARP) {
    // ---------------- code producer: the packed weights of four K-blocks a time, by TMA ----------------
    // (loaded by the decoders themselves, 16 bytes from each of 32 rows per instruction, they take as long in the load/store
    // unit as the decoded tile's stores do, and the decoders stop keeping up)
    if (!dense_w) {
      int c = 0;
      uint32_t ph = 1u;
      bool ok = true;
      PairTile tc;
      for (int t = pair; ok && t < total; t += n_pairs) {
        if (!pair_tile(ctl, plan, t, n_fp, p.G, &tc)) break;
        const int w_rows = tc.width / 2, wrow = tc.group * p.N + tc.f0 + rank * w_rows;
#pragma unroll 1
        for (int kb = 0; kb < n_kb; kb += CODE_KB) {
          if (!mbar_wait(smem_u32(&ctl->code_empty[c]), ph, abort_flag, p.status, JB200_STATUS_GEMM_PRODUCER)) { ok = false; break; }
          if (elect_one()) {
            const uint32_t bar = smem_u32(&ctl->code_full[c]);
            mbar_arrive_expect_tx(bar, uint32_t(w_rows) * CODE_KB * 16);
            for (int r = 0; r < w_rows; r += 32)
              tma_load_2d(code_base + uint32_t(c) * CODE_BYTES + uint32_t(r) * CODE_KB * 16, &tmap_w, kb * 16, wrow + r, bar);
          }
          __syncwarp();
          if (++c == CODE_SLOTS) { c = 0; ph ^= 1u; }
        }
      }
    }
  } else if (warp < EPI_WARP0) {
    // ---------------- weight decoders: group g takes K-blocks g, g + 2 of every slot of codes ----------------
    if (!dense_w) {
      const int g = (warp - DEC_WARP0) >> 2;
      const int r = ((warp - DEC_WARP0) & 3) * 32 + lane;          // weight row inside the CTA's half of the tile
      const uint32_t swz = uint32_t(r & 7), code_row = uint32_t(r) * (CODE_KB * 16), code_swz = uint32_t((r >> 1) & 3);
      const int slots = total > pair ? ((total - pair - 1) / n_pairs + 1) * (n_kb / CODE_KB) : 0;
      int s = g, c = 0;
      uint32_t ph = 1u, c_ph = 0u;
      bool ok = true;
      // (narrow tiles: rows past theirs are decoded from whatever the slot holds and never read)
#pragma unroll 1
      for (int i = 0; ok && i < slots; ++i) {
        if (!mbar_wait(smem_u32(&ctl->code_full[c]), c_ph, abort_flag, p.status, JB200_STATUS_GEMM_DECODE)) break;
        uint32_t words[2][4];
#pragma unroll
        for (int u = 0; u < 2; ++u)                                // 64-byte rows in the 64-byte swizzle: no bank conflicts
          asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(words[u][0]), "=r"(words[u][1]), "=r"(words[u][2]), "=r"(words[u][3])
                       : "r"(code_base + uint32_t(c) * CODE_BYTES + code_row + ((uint32_t(g + 2 * u) ^ code_swz) << 4)) : "memory");
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (!mbar_wait(smem_u32(&ctl->empty[s]), ph, abort_flag, p.status, JB200_STATUS_GEMM_DECODE)) { ok = false; break; }
          uint8_t* brow = smem + size_t(STAGES) * A_BYTES + size_t(s) * B_BYTES + size_t(r) * 128;
#pragma unroll
          for (int wi = 0; wi < 4; ++wi) {
            uint32_t v[8];
            if (p.w_layout == 1) decode16_prepared(words[u][wi], v); else decode16(words[u][wi], v);
            *reinterpret_cast<uint4*>(brow + ((uint32_t(2 * wi) ^ swz) << 4)) = make_uint4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<uint4*>(brow + ((uint32_t(2 * wi + 1) ^ swz) << 4)) = make_uint4(v[4], v[5], v[6], v[7]);
          }
          fence_proxy_async_smem();  // generic-proxy writes -> visible to the tensor core's async proxy
          __syncwarp();
          if (lane == 0) cluster_mbar_arrive(cluster_map(smem_u32(&ctl->full[s]), 0u));
          s += DEC_GROUPS;
          if (s >= STAGES) { s -= STAGES; ph ^= 1u; }
        }
        // only now: the loads above are known to have delivered, their values are in the stores that the fences waited for
        if (lane == 0) mbar_arrive(smem_u32(&ctl->code_empty[c]));
        if (++c == CODE_SLOTS) { c = 0; c_ph ^= 1u; }
      }
    }
  } else {
    // ---------------- epilogue: a lane is a token, its registers are out-features ----------------
    const int q = warp & 3;                     // TMEM lane quadrant this warp may read
    const int half = (warp - EPI_WARP0) >> 2;   // which of the alternating 32-feature chunks
    uint32_t tile = 0u;
    PairTile tc;
    for (int t = pair; t < total; t += n_pairs, ++tile) {
      if (!pair_tile(ctl, plan, t, n_fp, p.G, &tc)) break;
      const uint32_t acc = tile & 1u;
      const int tok = tc.tok0 + rank * BM + q * 32 + lane;
      const bool on = tok < tc.tok_end;
      if (!mbar_wait(smem_u32(&ctl->acc_full[acc]), (tile >> 1) & 1u, abort_flag, p.status, JB200_STATUS_GEMM_EPILOGUE)) break;
      tc_fence_after_sync();
      __syncwarp();
      const uint32_t t_lane = tmem + (uint32_t(q * 32) << 16) + acc * BN;
      for (int c0 = half * 32; c0 < tc.width; c0 += 64) {
        const int f = tc.f0 + c0;
        if (f >= p.N) break;                    // the last tile of an odd multiple of 128
        const float alpha = dense_w ? 1.0f
                                    : __ldg(p.alpha + size_t(tc.group) * (p.N / p.alpha_rows) + f / p.alpha_rows) *
                                          (p.w_layout ? 0.5f : 1.0f);   // prepared weights decode to +-2
        uint32_t v[32];
        tmem_ld_32x32(t_lane + c0, v);
        tmem_ld_wait();
        if (RESID) {
          // x[token][feature] += alpha * acc by the memory system: the tile leaves as one TMA reduction, which clips rows past
          // the matrix.  Rows of 128 bytes in the 128-byte swizzle: every 16-byte store of eight lanes covers all banks.
          if (lane == 0) bulk_wait_group_read<0>();     // the previous reduction has read this warp's tile
          __syncwarp();
          const uint32_t stage = out_base + uint32_t(warp - EPI_WARP0) * OUT_BYTES, dst = stage + uint32_t(lane) * 128u;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};"
                         ::"r"(dst + (uint32_t(j ^ (lane & 7)) << 4)), "f"(alpha * __uint_as_float(v[4 * j])),
                           "f"(alpha * __uint_as_float(v[4 * j + 1])), "f"(alpha * __uint_as_float(v[4 * j + 2])),
                           "f"(alpha * __uint_as_float(v[4 * j + 3])) : "memory");
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_reduce_add_2d(&tmap_out, f, tc.tok0 + rank * BM + q * 32, stage);
            bulk_commit_group();
          }
          continue;
        }
        if (on) store_row_chunk(p, v, alpha, size_t(tok) * p.N + f);
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) cluster_mbar_arrive(cluster_map(smem_u32(&ctl->acc_empty[acc]), 0u));
    }
    if (RESID && lane == 0) bulk_wait_group<0>();       // every reduction has landed before the CTA ends
  }

  __syncwarp();
  tc_fence_before_sync();
  cluster_arrive();               // neither CTA leaves while the other's MMAs, commits or arrivals may still reach it
  cluster_wait();
  if (warp == 0) {
    tc_fence_after_sync();
    pair_tmem_dealloc(tmem, TMEM_COLS);
  }
}

}  // namespace

int launch_pair_gemm(const GemmParams& p, const void* x_bf16, int sms, cudaStream_t stream) {
  const int pairs = sms / 2;
  CUtensorMap tmap;
  const cuuint64_t gdim[2] = {cuuint64_t(p.K), cuuint64_t(p.M)};
  const cuuint64_t gstride[1] = {cuuint64_t(p.K) * 2};
  const cuuint32_t box[2] = {cuuint32_t(BK), cuuint32_t(BM)};
  int rc = encode_tiled(&tmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, x_bf16, gdim, gstride, box, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, "ternary_linear");
  if (rc != JB200_OK) return rc;
  CUtensorMap tmap_w;
  if (p.w_layout == 2) {
    const cuuint64_t wdim[2] = {cuuint64_t(p.K), cuuint64_t(p.N)};
    const cuuint32_t wbox[2] = {cuuint32_t(BK), 32};
    rc = encode_tiled(&tmap_w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, p.w_packed, wdim, gstride, wbox, CU_TENSOR_MAP_SWIZZLE_128B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, "dense_linear (weights)");
  } else {
    const cuuint64_t wdim[2] = {cuuint64_t(p.K) / 4, cuuint64_t(p.G) * p.N};
    const cuuint64_t wstride[1] = {cuuint64_t(p.K) / 4};
    const cuuint32_t wbox[2] = {cuuint32_t(CODE_KB) * 16, 32};
    rc = encode_tiled(&tmap_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, p.w_packed, wdim, wstride, wbox, CU_TENSOR_MAP_SWIZZLE_64B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_128B, "ternary_linear (weights)");
  }
  if (rc != JB200_OK) return rc;
  const long tiles = (long((p.M + 2 * BM - 1) / (2 * BM)) + (p.G - 1)) * ((p.N + BN - 1) / BN) * 4;   // at most, with cut tiles
  const dim3 grid(2 * unsigned(tiles < pairs ? tiles : pairs));
  CUtensorMap tmap_out = tmap;
  if (p.epilogue == JB200_EPI_RESID_F32 && !p.seg_offsets) {
    const cuuint64_t odim[2] = {cuuint64_t(p.N), cuuint64_t(p.M)};
    const cuuint64_t ostride[1] = {cuuint64_t(p.N) * 4};
    const cuuint32_t obox[2] = {32, 32};
    rc = encode_tiled(&tmap_out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, p.out, odim, ostride, obox, CU_TENSOR_MAP_SWIZZLE_128B,
                      CU_TENSOR_MAP_L2_PROMOTION_L2_128B, "ternary_linear (residual stream)");
    if (rc != JB200_OK) return rc;
    JB_MAX_SMEM(pair_gemm_kernel<true>, smem_bytes(true));
    launch_dep_cluster(pair_gemm_kernel<true>, grid, dim3(THREADS), smem_bytes(true), 2, stream, tmap, tmap_w, tmap_out, p);
  } else {
    JB_MAX_SMEM(pair_gemm_kernel<false>, smem_bytes(false));
    launch_dep_cluster(pair_gemm_kernel<false>, grid, dim3(THREADS), smem_bytes(false), 2, stream, tmap, tmap_w, tmap_out, p);
  }
  JB_LAUNCH_CHECK("pair_gemm_kernel");
  return JB200_OK;
}

}  // namespace jb
