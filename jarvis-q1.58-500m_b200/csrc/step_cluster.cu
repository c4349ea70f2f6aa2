// A whole single-token step of up to a few dozen sequences in ONE launch: every layer of the model in thread-block clusters of
// sixteen CTAs.
//
// Kernel by kernel a layer of a decode step is seven to ten dependent launches, 25 us at one sequence and 44 us at 64, of which
// the arithmetic is a few: each launch pays for its predecessor's last block, the grid dependency, a round trip for the rows it
// starts from and an epilogue.  What no form can avoid is the chain of MMAs over K (one f32 accumulator per output, kept so that
// a token's experts do not depend on the form that ran): 5 x 64 steps of 23 cycles = 4 us a layer.  Here
//   - a cluster carries its sequences through all layers: CTA c holds head c (its q, k, v rows, its attention states), 64 rows
//     of the output projection and a sixteenth of the expert matrices; the token rows live in shared memory, replicated;
//   - rows change hands by st.async into the other CTAs' shared memory, counted by an mbarrier there (about 1000 cycles for a
//     few hundred bytes, 16 bytes a cycle and CTA beyond; a grid barrier in global memory measured 2000 + the loads): attention
//     rows, residual rows, expert hidden rows and expert outputs, four exchanges a layer.  Norms, router and the block's tail
//     are computed by every CTA for all its cluster's tokens: cheaper than an exchange each;
//   - weights, states and membranes are 4 KB units - what one warp needs for one job - that a producer warp brings into a ring of
//     shared memory in the order of use, as far ahead as the ring is deep, across layers: no stage waits for memory unless the
//     ring has run dry.  Ternary weights are laid out once in MMA fragment order: a lane's 16 bytes are its A operands
//     of eight steps (the prepared layout cost 16 wavefronts of shared memory per eight steps, this one 4);
//   - sequences meet only in the variance that sets the LSF decay: with several clusters their sums travel as tagged
//     words through global memory, one exchange a layer.  Those clusters wait for one another, so they are one cooperative launch.
// With one token in a cluster (FULL) every CTA takes a sixteenth of every expert (few experts are used, each by one token);
// beyond, an expert belongs to four CTAs, which exchange its hidden rows among themselves.
// Measured (24 layers and the vocabulary head, replayed as a graph, kernel by kernel -> here): 1 sequence 621 -> 494 us, 2 675 -> 517,
// 4 710 -> 504, 7 715 -> 511, 8 718 -> 630, 16 810 -> 655, 32 937 -> 751, 56 1049 -> 928.  With more tokens a cluster the form
// loses: every cluster decodes all weights for itself, and shared memory holds eight.  The kernels have become faster since, those for more than
// sixteen tokens above all: kernel by kernel 1 sequence 572, 2 609, 4 643, 8 657, 12 711, 16 769, 17 602, 20 609, 24 612, 32 637, 40 663, 48 684, 56 713 us, here
// 492, 508, 503, 633, 633, 656, 657, 662, 690, 743, 788, 844, 927.  So from 17 sequences on the kernels would be the faster form; the line below has not been
// drawn again.
// Every value is rounded and every f32 sum ordered as in the kernels this one stands for.  The f64 sums over tokens behind mean and
// variance, and those of the router's probabilities, are added in another order and rounded to f32 after that: the tests find the
// results equal bit for bit, and a last bit of those scalars is what could differ.
#include "attn_step.cuh"
#include "common.cuh"
#include "gemm_shared.cuh"
#include "launchers.h"
#include "moe_finalize.cuh"
#include "moe_router.cuh"
#include "row_math.cuh"

namespace jb {

namespace {

constexpr int CTAS = 16, C = 1024, D = 64, E = 4, HID = 2048;      // cluster; d_model = 16 heads x 64, experts of 2048
constexpr int WARPS = 16, THREADS = 32 * (WARPS + 2);              // sixteen that compute, the producer, the one of settle()
constexpr int UNIT = 4096, MAX_UNITS = 48;
constexpr int ROW_C = 2 * C + 16, ROW_H = 2 * HID + 16;            // bf16 rows that ldmatrix reads, padded against bank conflicts
constexpr int MAX_TOKENS = 8;                                     // of a cluster
constexpr int MAX_CLUSTERS = 8, MAX_LAYERS = 32;                   // layers of one launch
constexpr int SCRATCH = 512;                                       // bytes per warp

// A layer's weights: 16-row x 1024-in-feature tiles of q|k|v, out-projection, w1, w2 (two halves each), then scalars.  Only what is
// derived from parameters by quantising or by the decays' sigmoid; norms, router and var_scale are read where the caller has them, so
// that a captured step follows an edit of those as the kernels do.
constexpr int T_OUT = 3 * C / 16, T_W1 = T_OUT + C / 16, T_W2 = T_W1 + E * HID / 16, T_END = T_W2 + 2 * E * C / 16;
constexpr int SC_GAMMA = 0, SC_AQKV = 16, SC_AOUT = 19, SC_A1 = 20, SC_A2 = 24, SC_FLOATS = 32;
constexpr size_t LAYER_BYTES = size_t(T_END) * UNIT + 256;

struct StepLayer {
  const uint8_t* tiles;
  const float *w_norm1, *w_norm2, *w_router, *var_scale, *s_in, *h_in, *mu;
  float *s_out, *h_out;
  float eps1, eps2, alpha_min, alpha_max, balance_alpha, lam, tau;
};

struct StepParams {
  StepLayer layer[MAX_LAYERS];
  const int64_t* ids;
  const float* table;
  float* x;
  const float *cos_tab, *sin_tab;
  const int32_t* pos0;
  const float* w_final;
  __nv_bfloat16* hidden_out;
  uint8_t *acc, *routing;
  float *scalars, *reflect;
  unsigned int* status;
  size_t acc_stride, routing_stride;
  uint32_t r_idx, r_gates, r_counts, r_offsets, r_scatter, r_gather, r_gate_idx;       // within a layer's routing block
  uint32_t o_p1, o_p2, o_sc, o_rx, o_ry, o_xn, o_rh, o_qkv, o_ho, o_cs, o_scr, o_ring;      // within dynamic shared memory
  double n_elems, n_inv, n1_inv;       // of the MoE output, and the reciprocals of n and n - 1
  uint32_t units_inv;                  // ceil(2^32 / units)
  int vocab, n_pos, pos0_scalar, N, n_layers, n_clusters, units;
  float eps_final;
};

struct Ctl {
  uint64_t full[MAX_UNITS], empty[MAX_UNITS], p1_full, p1_empty, p2_there, p2_full, p2_empty;
  uint64_t got_o, got_x, got_h, got_y;               // rows that have arrived
  double part[MAX_TOKENS][2];
  alignas(8) float gates2[MAX_TOKENS][2];
  alignas(8) uint32_t word[32];
  int expert[MAX_TOKENS][2];                         // two different ones
  uint32_t second[MAX_TOKENS];                       // where the second assignment's row is, after the first one's
  float alpha, var_scale[2];
  uint32_t abort_flag;
  int last;
  uint8_t list[WARPS][2 * MAX_TOKENS];
};
static_assert(sizeof(Ctl) <= 2048, "static shared memory");
constexpr size_t DYN_MAX = 227 * 1024 - 2048;

// ---- the pieces ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void ldsm4(uint32_t (&b)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(a));
}
__device__ __forceinline__ void bar_compute() { asm volatile("bar.sync 1, 512;" ::: "memory"); }
static_assert(WARPS * 32 == 512, "the barrier's count");

// Bounded wait for a phase of an mbarrier (one that other CTAs complete, or a copy).  A wait that gave up lets every later one of
// the CTA pass at once: the kernel runs to its end on whatever is there (indexes are clamped), so no barrier is left short of
// a warp.  The loop is a function of its own: inlined at every wait it would push the layer's code out of the instruction cache.
__device__ __forceinline__ bool phase_done(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}"
      : "=r"(done) : "r"(bar), "r"(parity), "r"(20000u) : "memory");
  return done != 0;
}
__device__ __noinline__ bool wait_long(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, unsigned int* status) {
  const unsigned long long t0 = globaltimer_ns();
  for (;;) {
    if (*abort_flag) return false;
#pragma unroll 1
    for (int i = 0; i < 32; ++i)
      if (phase_done(bar, parity)) return true;
    if (globaltimer_ns() - t0 > JB_WAIT_LIMIT_NS) {
      *abort_flag = 1u;
      atomicCAS(status, 0u, JB200_STATUS_STEP_CLUSTER);
      return false;
    }
  }
}
__device__ __forceinline__ bool wait_phase(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, unsigned int* status) {
  return phase_done(bar, parity) || wait_long(bar, parity, abort_flag, status);
}

// 16 out-features x 8 tokens x 1024 in-features: `a` is this lane's place in a weight unit, xa its ldmatrix row.  Activations are
// fetched a double step ahead, weights eight steps: 26 cycles a step with four warps on the SM, 38, 53, 68 with 8, 12, 16 (the MMAs
// alone 23, 25, 29, 39; the rest is the codes' shifts and masks).  Called in one place: see Step.
__device__ __forceinline__ void gemm_unit(float (&acc)[4], uint32_t a, uint32_t xa) {
  uint4 w = lds128(a);
  uint32_t b[4], bn[4];
  ldsm4(b, xa);
#pragma unroll 1
  for (int ch = 0; ch < 8; ++ch) {
    const uint4 wn = lds128(a + uint32_t(ch < 7 ? ch + 1 : 7) * 512u);
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      const int next = ch * 4 + d + 1 < 32 ? ch * 4 + d + 1 : 31;
      ldsm4(bn, xa + uint32_t(next) * 64u);
      const uint32_t lo = d < 2 ? w.x : w.y, hi = d < 2 ? w.z : w.w;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int j = 4 * (d & 1) + 2 * h;
        const uint32_t f[4] = {(lo << (14 - 2 * j)) & 0xC000C000u, (hi << (14 - 2 * j)) & 0xC000C000u,
                               (lo << (12 - 2 * j)) & 0xC000C000u, (hi << (12 - 2 * j)) & 0xC000C000u};
        mma_16816(acc, f, b[2 * h], b[2 * h + 1]);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) b[e] = bn[e];
    }
    w = wn;
  }
}

// ---- the kernel ------------------------------------------------------------------------------------------------
// Every instruction runs once or a few times a layer, so the layer's code has to stay in the instruction cache (32 KB run at full
// rate, 32 to 128 KB at three cycles an instruction, more at six): the four products share one loop over phases, long waits are
// calls, row loops are left rolled.  Written out stage by stage the kernel was 140 KB and a step of one sequence took 543 us.
template <bool FULL, bool STREAM>
struct Step {
  const StepParams& p;
  Ctl& ctl;
  uint8_t* smem;
  uint32_t base;                 // of dynamic shared memory
  int warp, lane, c, cluster, n0, NT;
  volatile uint32_t* abort_flag;

  __device__ __forceinline__ uint32_t bar(const uint64_t& b) const { return smem_u32(&b); }
  __device__ __forceinline__ bool wait(const uint64_t& b, uint32_t parity) const {
    const bool ok = wait_phase(bar(b), parity & 1u, abort_flag, p.status);
    __syncwarp();
    return ok;
  }
  __device__ __forceinline__ int state_units() const { return FULL ? 0 : 4 * NT; }
  __device__ __forceinline__ int layer_units(int l) const { return 80 + state_units() + (p.layer[l].h_in ? NT : 0); }

  // ---------------- producer ----------------
  __device__ __forceinline__ void produce() const {
    int slot = 0, issued = 0, norms = 0, routers = 0;
    uint32_t ph = 1u;
    bool ok = true;
    // `n` units from src, `stride` bytes apart
    auto units = [&](const void* src, size_t stride, int n) {
#pragma unroll 1
      for (int i = 0; i < n && ok; ++i) {
        ok = wait(ctl.empty[slot], ph);
        if (!ok) break;
        if (elect_one()) {
          mbar_arrive_expect_tx(bar(ctl.full[slot]), UNIT);
          bulk_load_1d(base + p.o_ring + uint32_t(slot) * UNIT, static_cast<const uint8_t*>(src) + i * stride, UNIT, bar(ctl.full[slot]));
        }
        __syncwarp();
        ++issued;
        if (++slot == p.units) { slot = 0; ph ^= 1u; }
      }
    };
    // norm weights and scalars number i: those of layer i, after the last the final norm's
    auto norm1 = [&](int i) {
      const bool lay = i < p.n_layers;
      const float* w = lay ? p.layer[i].w_norm1 : p.w_final;
      if (!ok || !w) return;
      ok = wait(ctl.p1_empty, uint32_t(i) ^ 1u);
      if (!ok) return;
      ++norms;
      if (elect_one()) {
        mbar_arrive_expect_tx(bar(ctl.p1_full), C * 4 + (lay ? SC_FLOATS * 4 : 0));
        bulk_load_1d(base + p.o_p1, w, C * 4, bar(ctl.p1_full));
        if (lay)
          bulk_load_1d(base + p.o_sc + uint32_t(i & 1) * (SC_FLOATS * 4), p.layer[i].tiles + size_t(T_END) * UNIT, SC_FLOATS * 4,
                       bar(ctl.p1_full));
      }
      __syncwarp();
    };
    // A layer's units in the order of use, a run of them per lane: q, k, v; states; out-projection; w1; the halves of w2; membranes
    enum { WEIGHTS, STATE, OUT, DOWN, MEMBRANE };
    const int states = FULL ? 0 : NT, runs = 17 + states, q = lane < 3 ? lane : lane - states;
    static_assert(17 + MAX_TOKENS <= 32, "a lane per run");
    int r_kind = WEIGHTS, r_n = 4, r_off = 0;
    if (lane >= 3 && q < 3) {
      r_kind = STATE;
      r_off = ((n0 + lane - 3) * CTAS + c) * 4;
    } else if (q < 3) {
      r_off = q * (C / 16) + c * 4;
    } else if (q == 3) {
      r_kind = OUT;
      r_off = T_OUT + c * 4;
    } else if (q < 8) {
      r_n = 8;
      r_off = T_W1 + (FULL ? (q - 4) * (HID / 16) + c * 8 : (c & 3) * (HID / 16) + (c >> 2) * 32 + 8 * (q - 4));
    } else if (q < 16) {
      const int j = q & 3;
      r_kind = DOWN;
      r_off = T_W2 + 2 * (FULL ? j * (C / 16) + c * 4 : (c & 3) * (C / 16) + (c >> 2) * 16 + 4 * j) + ((q - 8) >> 2);
    } else {
      r_kind = MEMBRANE;
      r_off = n0;
      r_n = NT;
    }
#pragma unroll 1
    for (int l = -1; l < p.n_layers && ok; ++l) {
      const StepLayer& y = p.layer[l < 0 ? 0 : l];
      const uint8_t* w = y.tiles;
      // The ring is shallower than a layer: the next layer's states and this cluster's share of its weights come into L2 meanwhile.
      if (l + 1 < p.n_layers) {
        const StepLayer& z = p.layer[l + 1];
        if (z.s_in && lane < NT) l2_prefetch(z.s_in + (size_t(n0 + lane) * CTAS + c) * (D * D), D * D * 4);
#pragma unroll 1
        for (int i = cluster * CTAS + c + p.n_clusters * CTAS * lane; i < T_END / 4; i += p.n_clusters * CTAS * 32)
          l2_prefetch(z.tiles + size_t(i) * (4 * UNIT), 4 * UNIT);
        __syncwarp();
      }
#pragma unroll 1
      for (int i = 0; i < (l < 0 ? 0 : runs) && ok; ++i) {
        const int kind = __shfl_sync(0xffffffffu, r_kind, i), off = __shfl_sync(0xffffffffu, r_off, i);
        const int n = __shfl_sync(0xffffffffu, r_n, i);
        if (kind == OUT) {
          ok = wait(ctl.p2_empty, uint32_t(l) ^ 1u);
          routers += ok ? 1 : 0;
          if (ok && elect_one()) {
            mbar_arrive_expect_tx(bar(ctl.p2_there), C * 4 + E * UNIT);
            bulk_load_1d(base + p.o_p2, y.w_norm2, C * 4, bar(ctl.p2_there));
            bulk_load_1d(base + p.o_p2 + C * 4, y.w_router, E * UNIT, bar(ctl.p2_there));
          }
          __syncwarp();
        }
        const uint8_t* src = kind == STATE      ? reinterpret_cast<const uint8_t*>(y.s_in)
                             : kind == MEMBRANE ? reinterpret_cast<const uint8_t*>(y.h_in)
                                                : w;
        if (src) units(src + size_t(off) * UNIT, kind == DOWN ? 2 * UNIT : UNIT, n);
      }
      norm1(l + 1);
    }
    if (!ok) {           // given up: copies in flight land before this CTA's shared memory goes
      auto landed = [&](const uint64_t& b, int n) {           // n phases of it, the last of which may be open
#pragma unroll 1
        for (int i = 0; n > 0 && i < 2000 && !phase_done(bar(b), uint32_t(n - 1) & 1u); ++i) {}
      };
      landed(ctl.p1_full, norms);
      landed(ctl.p2_there, routers);
#pragma unroll 1
      for (int u = issued > p.units ? issued - p.units : 0; u < issued; ++u) landed(ctl.full[u % p.units], u / p.units + 1);
    }
  }

  // ---------------- what a layer reads from the parameters themselves, by a warp of its own ----------------
  // The router's rows in the order in which route() reads them without bank conflicts: 16 bytes (group i, half, lane) hold channels
  // (32 i + lane) 8 + 4 half; in their own order every read is a two-way conflict.  And var_scale.  By the producer, as copies of 16 bytes,
  // this cost a step 1 % at one sequence and 5 % at 32; by warps that have no part in q, k, v the layer's code grew from 47 to 61 KB
  // (592 us for 498).
  __device__ __forceinline__ void settle() const {
    const uint32_t router = base + p.o_p2 + C * 4, to = router + uint32_t(lane & 1) * 512u + uint32_t(lane >> 1) * 16u;
#pragma unroll 1
    for (int l = 0; l < p.n_layers; ++l) {
      const float var_scale = *p.layer[l].var_scale;
      if (!wait(ctl.p2_there, uint32_t(l))) return;
#pragma unroll 4
      for (uint32_t i = 0; i < E * UNIT; i += 1024) {        // a group's 1 KB stays where it is
        const uint4 a = lds128(router + i + uint32_t(lane) * 16u), b = lds128(router + i + 512u + uint32_t(lane) * 16u);
        __syncwarp();
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(to + i), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w) : "memory");
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(to + i + 256u), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the next layer's bulk copy comes after these stores
      ctl.var_scale[l & 1] = var_scale;       // two: the next one may be here before decay() has run
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(ctl.p2_full));
    }
  }
  static __device__ __forceinline__ void l2_prefetch(const void* src, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
  }

  // ---------------- what the sixteen other warps share ----------------
  // Slot of unit number u (u below 2^16: the multiplication is exact), waiting until it is there.  Copies do not land in order, so the
  // unit that had the slot before may still be on its way to another warp; a wait by parity would take its barrier, a phase short, for
  // done.  Hence first that unit's release.
  __device__ __forceinline__ int unit_wait(int u) const {
    const int turn = int(__umulhi(uint32_t(u), p.units_inv)), slot = u - turn * p.units;
    wait(ctl.empty[slot], uint32_t(turn) ^ 1u);
    wait(ctl.full[slot], uint32_t(turn));
    return slot;
  }
  __device__ __forceinline__ void unit_done(int slot) const {
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(ctl.empty[slot]));
  }
  __device__ __forceinline__ uint32_t unit_at(int slot) const { return base + p.o_ring + uint32_t(slot) * UNIT; }
  __device__ __forceinline__ uint32_t scratch() const { return base + p.o_scr + uint32_t(warp) * SCRATCH; }
  // tokens of this cluster that expert e serves, as 2 n + k in this warp's list; their number
  __device__ __forceinline__ int tokens_of(int e) const {
    const bool k1 = lane < NT && ctl.expert[lane][1] == e, on = k1 || (lane < NT && ctl.expert[lane][0] == e);
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (on) ctl.list[warp][__popc(m & ((1u << lane) - 1u))] = uint8_t(2 * lane + (k1 ? 1 : 0));
    __syncwarp();
    return __popc(m);
  }
  // The first / second / ... used expert's tiles go to the warps in turn, an expert nobody wants only gives its units back.  FULL: the
  // warp's tile of expert e among `tiles` (or >= tiles: none).
  __device__ __forceinline__ int tile_of(unsigned used, int e, int tiles) const {
    const int before = (used >> e) & 1u ? __popc(used & ((1u << e) - 1u)) : e;
    return (warp - tiles * before) & 15;
  }

  // Attention step of a few value rows of one sequence's state in this CTA's head.  FULL: eight rows whose states are in registers; else
  // sixteen rows, unit u.  STREAM: attn_decode_stream_kernel's sums (four columns a lane), else attn_decode_kernel's (sixteen).
  __device__ __forceinline__ void attend(int u, float4 (&st)[4], int n, int row0, float gamma, float* s_out) const {
    const __nv_bfloat16* qkv = reinterpret_cast<const __nv_bfloat16*>(smem + p.o_qkv + n * 384);
    float* rq = reinterpret_cast<float*>(smem + p.o_scr + warp * SCRATCH);
    float* rk = rq + D;
    {
      const float* cs = reinterpret_cast<const float*>(smem + p.o_cs + n * 256);
      const float q0 = elu1(__bfloat162float(qkv[lane])) * 0.125f, q1 = elu1(__bfloat162float(qkv[lane + 32])) * 0.125f;
      const float k0 = elu1(__bfloat162float(qkv[D + lane])), k1 = elu1(__bfloat162float(qkv[D + lane + 32]));
      rq[lane] = rope_lo(q0, q1, cs[lane], cs[32 + lane]);  rq[lane + 32] = rope_hi(q0, q1, cs[lane], cs[32 + lane]);
      rk[lane] = rope_lo(k0, k1, cs[lane], cs[32 + lane]);  rk[lane + 32] = rope_hi(k0, k1, cs[lane], cs[32 + lane]);
    }
    __syncwarp();
    float* out = s_out ? s_out + (size_t(n0 + n) * CTAS + c) * (D * D) + row0 * D : nullptr;
    const __nv_bfloat16* v = qkv + 2 * D + row0;
    __nv_bfloat16* o16 = reinterpret_cast<__nv_bfloat16*>(rq);         // the outputs take the place of rq, rk once those have been read
    if (FULL && !STREAM) {
      const int row = lane >> 2, c0 = 16 * (lane & 3);
      const float vr = __bfloat162float(v[row]);
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int col = c0 + 4 * i;
        const float4 kq = *reinterpret_cast<const float4*>(rk + col);
        st[i].x = decode_update(gamma, st[i].x, vr, kq.x);  st[i].y = decode_update(gamma, st[i].y, vr, kq.y);
        st[i].z = decode_update(gamma, st[i].z, vr, kq.z);  st[i].w = decode_update(gamma, st[i].w, vr, kq.w);
        if (out) *reinterpret_cast<float4*>(out + row * D + col) = st[i];
        acc += decode_dot4(st[i], *reinterpret_cast<const float4*>(rq + col));
      }
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      __syncwarp();
      if ((lane & 3) == 0) o16[row] = __float2bfloat16_rn(acc);
    } else if (FULL) {
      const int col = 4 * (lane & 15), half = lane >> 4;
      const float4 kq = *reinterpret_cast<const float4*>(rk + col), qq = *reinterpret_cast<const float4*>(rq + col);
      float o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int row = 2 * i + half;
        const float vr = __bfloat162float(v[row]);
        st[i].x = decode_update(gamma, st[i].x, vr, kq.x);  st[i].y = decode_update(gamma, st[i].y, vr, kq.y);
        st[i].z = decode_update(gamma, st[i].z, vr, kq.z);  st[i].w = decode_update(gamma, st[i].w, vr, kq.w);
        *reinterpret_cast<float4*>(out + row * D + col) = st[i];
        o[i] = decode_dot4(st[i], qq);
      }
#pragma unroll
      for (int m = 1; m < 16; m <<= 1)
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] += __shfl_xor_sync(0xffffffffu, o[i], m);
      __syncwarp();
      if ((lane & 15) == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) o16[2 * i + half] = __float2bfloat16_rn(o[i]);
      }
    } else {
      const int col = 4 * (lane & 15), half = lane >> 4;
      const float4 kq = *reinterpret_cast<const float4*>(rk + col), qq = *reinterpret_cast<const float4*>(rq + col);
      const int slot = unit_wait(u);
      const uint32_t tile = unit_at(slot) + uint32_t(half * D + col) * 4u;
      float mine = 0.f;            // lane 2 (or 18) + i: output row 2 i (2 i + 1)
#pragma unroll 2
      for (int i = 0; i < 8; ++i) {
        const int row = 2 * i + half;
        const float vr = __bfloat162float(v[row]);
        const uint4 w = lds128(tile + uint32_t(i) * (2 * D * 4));
        float4 s = make_float4(__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z), __uint_as_float(w.w));
        s.x = decode_update(gamma, s.x, vr, kq.x);  s.y = decode_update(gamma, s.y, vr, kq.y);
        s.z = decode_update(gamma, s.z, vr, kq.z);  s.w = decode_update(gamma, s.w, vr, kq.w);
        *reinterpret_cast<float4*>(out + row * D + col) = s;
        float o = decode_dot4(s, qq);
#pragma unroll
        for (int m = 1; m < 16; m <<= 1) o += __shfl_xor_sync(0xffffffffu, o, m);
        if ((lane & 15) == i) mine = o;
      }
      unit_done(slot);
      if ((lane & 15) < 8) o16[2 * (lane & 15) + half] = __float2bfloat16_rn(mine);
    }
    __syncwarp();
    if ((!FULL || lane < 16) && !*abort_flag) {
      const int part = lane >> 4;
      const uint32_t to = base + p.o_rh + uint32_t(n) * ROW_C + uint32_t(c * D + row0) * 2u + uint32_t(part) * 16u;
      st_async16(cluster_map(to, uint32_t(lane & 15)), cluster_map(bar(ctl.got_o), uint32_t(lane & 15)),
                 lds128(scratch() + uint32_t(part) * 16u));
    }
    __syncwarp();
  }

  // The CTA's 64 channels of token `warp`'s membrane after layer l.  h_out may be h_in, which every CTA of the cluster reads whole:
  // written only when all of them are past that layer's tail.
  __device__ __forceinline__ void membrane_out(int l) const {
    if (lane < 16)
      reinterpret_cast<float4*>(p.layer[l].h_out + size_t(n0 + warp) * C + c * D)[lane] =
          reinterpret_cast<const float4*>(smem + p.o_ho + warp * (D * 4))[lane];
  }

  // ---- a token's row in shared memory, eight channels a lane in four groups (loops are left rolled: a quarter of the code) ----
  static __device__ __forceinline__ void copy8(float* dst, const uint64_t (&v)[4]) {
    reinterpret_cast<ulonglong2*>(dst)[0] = make_ulonglong2(v[0], v[1]);
    reinterpret_cast<ulonglong2*>(dst)[1] = make_ulonglong2(v[2], v[3]);
  }
  static __device__ __forceinline__ void read8(uint64_t (&v)[4], const float* src) {
    const ulonglong2 a = reinterpret_cast<const ulonglong2*>(src)[0], b = reinterpret_cast<const ulonglong2*>(src)[1];
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
  static __device__ __forceinline__ void add_squares(float& ss, const uint64_t (&v)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float a, b;
      f32x2_split(v[j], a, b);
      ss = __fmaf_rn(a, a, ss);
      ss = __fmaf_rn(b, b, ss);
    }
  }
  __device__ __forceinline__ float* x_row() const { return reinterpret_cast<float*>(smem + p.o_rx + warp * (C * 4)) + lane * 8; }
  // RMSNorm of token `warp`'s residual row -> bf16 row of the activations, and every group to `also`.  The roundings are norm8's.
  template <typename F>
  __device__ __forceinline__ void norm_row(float ss, float eps, uint32_t weights, F&& also) const {
    const float r = rsqrtf(warp_sum(ss) / float(C) + eps);
    const uint64_t rr = f32x2(r, r);
    const float* w = reinterpret_cast<const float*>(smem + weights) + lane * 8;
#pragma unroll 1
    for (int i = 0; i < GROUPS; ++i) {
      uint64_t x[4], wt[4];
      read8(x, x_row() + i * 256);
      read8(wt, w + i * 256);
      uint32_t v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float a, b;
        f32x2_split(mul_f32x2(mul_f32x2(x[j], rr), wt[j]), a, b);
        v[j] = pack_bf16x2(a, b);
      }
      *reinterpret_cast<uint4*>(smem + p.o_xn + warp * ROW_C + (i * 32 + lane) * 16) = make_uint4(v[0], v[1], v[2], v[3]);
      also(i, v);
    }
  }
  // group i of this lane is in the CTA's 64 channels
  __device__ __forceinline__ bool own(int i) const { return i == (c >> 2) && (lane >> 3) == (c & 3); }

  // norm2 and router of token `warp`: router_finish's values with an expert per lane
  __device__ __forceinline__ void route(int l) const {
    const StepLayer& y = p.layer[l];
    wait(ctl.p2_full, uint32_t(l));
    wait(ctl.got_x, uint32_t(l));
    if (l > 0) membrane_out(l - 1);        // rows of this layer have come from everybody
    float ss = 0.f;
#pragma unroll 1
    for (int i = 0; i < GROUPS; ++i) {
      uint64_t x[4];
      read8(x, x_row() + i * 256);
      add_squares(ss, x);
    }
    float acc[E] = {};
    norm_row(ss, y.eps2, p.o_p2, [&](int i, const uint32_t (&v)[4]) {
      const float xv[8] = {bf16_lo(v[0]), bf16_hi(v[0]), bf16_lo(v[1]), bf16_hi(v[1]),
                           bf16_lo(v[2]), bf16_hi(v[2]), bf16_lo(v[3]), bf16_hi(v[3])};
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const float4* w = reinterpret_cast<const float4*>(smem + p.o_p2 + C * 4 + e * UNIT) + i * 64 + lane;
        acc[e] = router_dot(acc[e], xv, w[0], w[32]);
      }
    });
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] = warp_sum(acc[e]);
    float mx = acc[0];
#pragma unroll
    for (int e = 1; e < E; ++e) mx = fmaxf(mx, acc[e]);
    float mine = acc[0];                   // lane e: expert e's logit
#pragma unroll
    for (int e = 1; e < E; ++e) mine = lane == e ? acc[e] : mine;
    mine = expf(mine - mx);
    float pr[E], den = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) { pr[e] = __shfl_sync(0xffffffffu, mine, e); den += pr[e]; }
    const float inv = 1.0f / den;
    int i0 = 0, i1 = -1;
    float p0 = -1.f, p1 = -1.f;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      pr[e] *= inv;
      if (pr[e] > p0) { p1 = p0; i1 = i0; p0 = pr[e]; i0 = e; }
      else if (pr[e] > p1) { p1 = pr[e]; i1 = e; }
    }
    if (lane < 2) {                        // the token's two assignments
      const float gate = (lane ? p1 : p0) / (p0 + p1 + 1e-8f);
      const int id = lane ? i1 : i0;
      ctl.gates2[warp][lane] = gate;
      // NaN logits: both assignments are expert i0's, as in the maps.  Two different ones run all the same, which the exchanges count on;
      // the other one's row is not read.
      ctl.expert[warp][lane] = id < 0 ? (i0 + 1) % E : id;
      if (lane) ctl.second[warp] = id < 0 ? 0u : 2u * C;
      if (c == 0) {
        uint8_t* r = p.routing + l * p.routing_stride;
        const size_t at = size_t(n0 + warp) * 2 + lane;
        reinterpret_cast<int64_t*>(r + p.r_idx)[at] = id;
        reinterpret_cast<float*>(r + p.r_gates)[at] = gate;
      }
    }
    if (c == 0 && lane < E) {
      mine *= inv;                         // lane e: expert e's probability
      double* a = reinterpret_cast<double*>(p.acc + l * p.acc_stride) + 2;
      atomicAdd(a + lane, double(mine));
      if (lane == i0) atomicAdd(reinterpret_cast<int*>(a + E) + lane, 1);
    }
  }

  // Sum of token `warp`'s two expert rows, in the place of the first, and its statistics
  __device__ __forceinline__ void combine() const {
    uint8_t* row = smem + p.o_ry + warp * (C * 4) + lane * 16;
    const float2 gate = *reinterpret_cast<const float2*>(ctl.gates2[warp]);
    const uint64_t ga = f32x2(gate.x, gate.x), gb = f32x2(gate.y, gate.y);
    const uint8_t* row_b = row + ctl.second[warp];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll 1
    for (int i = 0; i < GROUPS; ++i) {
      const uint4 a = *reinterpret_cast<const uint4*>(row + i * 512), b = *reinterpret_cast<const uint4*>(row_b + i * 512);
      auto one = [&](uint32_t wa, uint32_t wb) {
        float lo, hi;
        f32x2_split(fma_f32x2(gb, f32x2(bf16_lo(wb), bf16_hi(wb)), mul_f32x2(ga, f32x2(bf16_lo(wa), bf16_hi(wa)))), lo, hi);
        s1 += lo;
        s1 += hi;
        s2 = __fmaf_rn(lo, lo, s2);
        s2 = __fmaf_rn(hi, hi, s2);
        return pack_bf16x2(lo, hi);
      };
      uint4 m;
      m.x = one(a.x, b.x);
      m.y = one(a.y, b.y);
      m.z = one(a.z, b.z);
      m.w = one(a.w, b.w);
      *reinterpret_cast<uint4*>(row + i * 512) = m;
    }
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if (lane == 0) { ctl.part[warp][0] = double(s1); ctl.part[warp][1] = double(s2); }
    __syncwarp();
  }

  // The decay of layer l from the sums over all tokens, by one warp; -> ctl.alpha
  __device__ __forceinline__ void decay(int l) const {
    const StepLayer& y = p.layer[l];
    double s[2] = {0.0, 0.0};
#pragma unroll 1
    for (int n = 0; n < NT; ++n) { s[0] += ctl.part[n][0]; s[1] += ctl.part[n][1]; }
    if (p.n_clusters > 1) {
      // the halves of both sums, each next to a tag that nothing else writes since the words were cleared
      unsigned long long* words = reinterpret_cast<unsigned long long*>(p.acc + l * p.acc_stride + p.acc_stride - MAX_CLUSTERS * 32);
      if (c == 0 && lane < 4) {
        const unsigned long long v = __double_as_longlong(lane < 2 ? s[0] : s[1]);
        const unsigned long long half = (lane & 1) ? v >> 32 : v & 0xffffffffull;
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(words + cluster * 4 + lane), "l"(half | (1ull << 32)) : "memory");
      }
      unsigned long long w = 0, t0 = 0;
#pragma unroll 1
      for (int i = 0; lane < 4 * p.n_clusters; ++i) {
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(words + lane) : "memory");
        if ((w >> 32) || *abort_flag) break;
        if ((i & 31) == 31) {
          if (!t0) t0 = globaltimer_ns();
          else if (globaltimer_ns() - t0 > JB_WAIT_LIMIT_NS) {
            *abort_flag = 1u;
            atomicCAS(p.status, 0u, JB200_STATUS_STEP_CLUSTER);
            break;
          }
        }
      }
      __syncwarp();
      ctl.word[lane] = uint32_t(w);
      __syncwarp();
      const double* v = reinterpret_cast<const double*>(ctl.word);      // little endian: the two halves are the sum
      s[0] = s[1] = 0.0;
#pragma unroll 1
      for (int k = 0; k < p.n_clusters; ++k) { s[0] += v[2 * k]; s[1] += v[2 * k + 1]; }
    }
    // moe_act_mean, moe_act_var
    const double mean64 = div_by(s[0], p.n_elems, p.n_inv), var64 = div_by(s[1] - s[0] * mean64, p.n_elems - 1.0, p.n1_inv);
    const float mean = float(mean64), var = float(var64 > 0.0 ? var64 : 0.0);
    if (lane == 0) {
      ctl.alpha = lsf_alpha_from_var(y.alpha_min, y.alpha_max, ctl.var_scale[l & 1], var);
      if (cluster == 0 && c == 0) {
        p.scalars[size_t(l) * 3 + 1] = mean;
        p.scalars[size_t(l) * 3 + 2] = var;
        if (p.reflect && y.mu) p.reflect[l] = reflect_penalty(y.lam, y.tau, __ldg(y.mu), mean, var);
      }
    }
  }

  __device__ __forceinline__ void compute() const {
    // ---- the rows the step starts from, angles ----
    if (warp < NT) {
      const int n = n0 + warp;
      const float* src = p.x + size_t(n) * C;
      if (p.ids) {
        long long id = p.ids[n];
        id = id < 0 ? 0 : (id >= p.vocab ? p.vocab - 1 : id);
        src = p.table + size_t(id) * C;
      }
      int pos = p.pos0 ? p.pos0[n] : p.pos0_scalar;
      pos = pos < 0 ? 0 : (pos >= p.n_pos ? p.n_pos - 1 : pos);
      float* cs = reinterpret_cast<float*>(smem + p.o_cs + warp * 256);
      cs[lane] = __ldg(p.cos_tab + size_t(pos) * 32 + lane);
      cs[32 + lane] = __ldg(p.sin_tab + size_t(pos) * 32 + lane);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        reinterpret_cast<float4*>(smem + p.o_rx + warp * (C * 4))[i * 32 + lane] = reinterpret_cast<const float4*>(src)[i * 32 + lane];
      __syncwarp();
    }
    if (p.n_clusters == 1 && c == 0 && warp == WARPS - 1) {
#pragma unroll 1
      for (int i = lane; i < p.n_layers; i += 32) {
        double* acc = reinterpret_cast<double*>(p.acc + i * p.acc_stride);
        for (int e = 0; e < E; ++e) { acc[2 + e] = 0.0; reinterpret_cast<int*>(acc + 2 + E)[e] = 0; }
      }
    }

    int u0 = 0;
    uint32_t h_parity = 0u;
    // l = -1: only the norm in front of the first layer
#pragma unroll 1
    for (int l = -1; l < p.n_layers; ++l) {
      const StepLayer& y = p.layer[l < 0 ? 0 : l];
      const uint32_t par = uint32_t(l) & 1u;
      const float* sc = reinterpret_cast<const float*>(smem + p.o_sc) + par * SC_FLOATS;
      const bool last = l + 1 == p.n_layers, follow = !last || p.w_final;
      if (l >= 0) {
        const int u_out = u0 + 12 + state_units();
        // not before: blocks of the next kernel would sit on the other SMs, waiting, for as long as this one runs
        if (last) pdl_trigger();
        if (warp == WARPS - 1 && lane == 0 && !*abort_flag) {      // (a phase that did not end cannot be armed again)
          mbar_arrive_expect_tx(bar(ctl.got_o), uint32_t(NT) * (C * 2));
          mbar_arrive_expect_tx(bar(ctl.got_x), uint32_t(NT) * (C * 4));
          mbar_arrive_expect_tx(bar(ctl.got_y), uint32_t(NT) * (C * 4));
        }
        // FULL: the states of this warp's eight rows travel while q, k, v are made, in attn_decode_kernel's lanes (sixteen columns of
        // a row) or attn_decode_stream_kernel's (four columns of every other row)
        float4 st[4];
        if (FULL) {
          const size_t at = (size_t(n0) * CTAS + c) * (D * D) + (warp & 7) * (8 * D) + (STREAM ? 4 * lane : 16 * lane);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            st[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (y.s_in && warp < 8) st[i] = *reinterpret_cast<const float4*>(y.s_in + at + (STREAM ? 2 * D : 4) * i);
          }
        }
        unsigned used = 0;
        int n_e = 0;
        // ---- the four products: q, k, v of head c; output projection; first and second expert matrix ----
#pragma unroll 1
        for (int ph = 0; ph < 4; ++ph) {
          if (ph == 1) {
            bar_compute();
            const float gamma = sc[SC_GAMMA + c];
#pragma unroll 1
            for (int j = warp; j < (FULL ? 8 : 4 * NT); j += WARPS)
              attend(u0 + 12 + j, st, FULL ? 0 : j >> 2, FULL ? j * 8 : (j & 3) * 16, gamma, y.s_out);
          } else if (ph == 2) {
            if (warp < NT) route(l);
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(ctl.p2_empty));
            bar_compute();
            if (FULL) {
              used = __reduce_or_sync(0xffffffffu, lane < NT ? (1u << ctl.expert[lane][0]) | (1u << ctl.expert[lane][1]) : 0u);
              if (warp == WARPS - 1 && lane == 0 && !*abort_flag) mbar_arrive_expect_tx(bar(ctl.got_h), uint32_t(NT) * (4 * HID));
            } else {
              n_e = tokens_of(c & 3);
              if (n_e > 0 && warp == WARPS - 1 && lane == 0 && !*abort_flag)
                mbar_arrive_expect_tx(bar(ctl.got_h), uint32_t(n_e) * (2 * HID));
            }
          }
          const int jobs = ph < 2 ? (warp < (ph ? 4 : 12) ? 1 : 0) : FULL ? E : ph == 2 ? 2 : 1;
#pragma unroll 1
          for (int k = 0; k < jobs; ++k) {
            int u, f0, n = NT, e = FULL ? k : c & 3;
            bool on = true;
            if (ph < 2) {
              u = (ph ? u_out : u0) + warp;
              f0 = warp * 16;
            } else if (FULL) {
              const int tiles = ph == 2 ? 8 : 4, q = tile_of(used, e, tiles);
              if (q >= tiles) continue;
              on = (used >> e) & 1u;
              u = u_out + (ph == 2 ? 4 : 36) + e * tiles + q;
              f0 = (c * tiles + q) * 16;
              if (on) n = tokens_of(e);
            } else {
              u = u_out + (ph == 2 ? 4 : 36) + k * WARPS + warp;
              f0 = (c >> 2) * (ph == 2 ? 512 : 256) + (k * WARPS + warp) * 16;
              n = n_e;
              on = n > 0;
            }
            const uint8_t* list = ctl.list[warp];
            const int halves = ph == 3 ? 2 : 1;
            float acc[4] = {};
            const int s = min(lane & 7, n - 1), row = !on ? 0 : ph < 2 ? s : ph == 2 ? list[s] >> 1 : FULL ? list[s] : s;
            uint32_t xa = base + ((ph & 1) ? p.o_rh : p.o_xn) + uint32_t(row) * uint32_t(ph == 3 ? ROW_H : ROW_C) +
                          uint32_t(lane >> 3) * 16u;
#pragma unroll 1
            for (int h = 0; h < halves; ++h) {
              const int slot = unit_wait(u + 16 * h);
              if (on) {
                if (h == 0 && (ph & 1)) wait(ph == 1 ? ctl.got_o : ctl.got_h, ph == 1 ? par : h_parity);
                gemm_unit(acc, unit_at(slot) + uint32_t(lane) * 16u, xa);
              }
              unit_done(slot);
              xa += 2 * 1024;
            }
            if (!on) continue;
            // ---- epilogue: a row of 16 features per token, then in pieces of 16 bytes to whoever needs it ----
            // codes decode to +-2
            const float alpha = 0.5f * sc[ph == 0 ? SC_AQKV + (warp >> 2) : ph == 1 ? SC_AOUT : ph == 2 ? SC_A1 + e : SC_A2 + e];
            const int g = lane >> 2, t = lane & 3;
            const uint32_t rows = ph == 0 ? base + p.o_qkv + uint32_t(f0) * 2u : scratch();
            const uint32_t row_bytes = ph == 0 ? 3 * D * 2 : ph == 1 ? 64 : 32;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int tok = 2 * t + h;
              float a = __fmul_rn(alpha, acc[h]), b = __fmul_rn(alpha, acc[2 + h]);
              if (tok >= n) continue;
              const uint32_t at = rows + uint32_t(tok) * row_bytes;
              if (ph == 1) {
                const float2 r = *reinterpret_cast<const float2*>(smem + p.o_rx + tok * (C * 4) + (c * D + f0 + 2 * g) * 4);
                asm volatile("st.shared.v2.f32 [%0], {%1, %2};"
                             ::"r"(at + uint32_t(g) * 8u), "f"(__fadd_rn(r.x, a)), "f"(__fadd_rn(r.y, b)) : "memory");
              } else {
                if (ph == 2) { a = gelu_erf(a); b = gelu_erf(b); }
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(at + uint32_t(g) * 4u), "r"(pack_bf16x2(a, b)) : "memory");
              }
            }
            if (ph == 0) continue;
            __syncwarp();
            const int lp = ph == 1 ? 2 : 1;               // pieces of a row: 2^lp
            const int ld = !FULL && ph == 2 ? 2 : 4;      // CTAs: 2^ld
            const uint64_t& b = ph == 1 ? ctl.got_x : ph == 2 ? ctl.got_h : ctl.got_y;
            const uint32_t to0 = base + (ph == 1 ? p.o_rx + uint32_t(c * D + f0) * 4u : (ph == 2 ? p.o_rh : p.o_ry) + uint32_t(f0) * 2u);
            const uint32_t to_bytes = ph == 1 ? C * 4 : ph == 2 ? ROW_H : 2 * C;
#pragma unroll 1
            for (int i = *abort_flag ? 1 << 30 : lane; i < n << (lp + ld); i += 32) {      // a CTA that has given up sends nothing more
              const int d = i & ((1 << ld) - 1), q = i >> ld, tok = q >> lp, r = q & ((1 << lp) - 1);
              const uint32_t rank = uint32_t(ld == 2 ? e + 4 * d : d);
              const int to = ph == 1 || (!FULL && ph == 2) ? tok : list[tok];
              st_async16(cluster_map(to0 + uint32_t(to) * to_bytes + uint32_t(r) * 16u, rank), cluster_map(bar(b), rank),
                         lds128(rows + uint32_t(tok) * row_bytes + uint32_t(r) * 16u));
            }
            __syncwarp();
          }
        }
        if (FULL || n_e > 0) h_parity ^= 1u;

        // ---- combine, statistics, decay ----
        if (warp < NT) {
          wait(ctl.got_y, par);
          combine();
        }
        // One token's warp would need neither barrier; without any, the compiler threads the tail's branches into copies of its code.
        if (!FULL) bar_compute();
        if (warp == (FULL ? 0 : WARPS - 1)) decay(l);
        bar_compute();
      }
      // ---- LSF, residual, the norm that follows ----
      if (warp < NT) {
        const float alpha = ctl.alpha;
        const uint64_t al = f32x2(alpha, alpha), one_m = f32x2(1.0f - alpha, 1.0f - alpha);
        const int slot = l >= 0 && y.h_in ? unit_wait(u0 + 80 + state_units() + warp) : -1;
        float ss = 0.f;
#pragma unroll 1
        for (int i = 0; i < GROUPS; ++i) {
          uint64_t x[4];
          read8(x, x_row() + i * 256);
          if (l >= 0) {
            uint64_t h[4] = {0ull, 0ull, 0ull, 0ull};
            if (slot >= 0) read8(h, reinterpret_cast<const float*>(smem + p.o_ring + slot * UNIT) + (i * 32 + lane) * 8);
            const uint4 m = *reinterpret_cast<const uint4*>(smem + p.o_ry + warp * (C * 4) + (i * 32 + lane) * 16);
            const uint32_t mw[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {        // lsf_step
              h[j] = fma_f32x2(al, h[j], mul_f32x2(one_m, f32x2(bf16_lo(mw[j]), bf16_hi(mw[j]))));
              asm("add.rn.f32x2 %0, %0, %1;" : "+l"(x[j]) : "l"(h[j]));
            }
            copy8(x_row() + i * 256, x);
            if (own(i)) {
              copy8(reinterpret_cast<float*>(smem + p.o_ho + warp * (D * 4)) + (lane & 7) * 8, h);
              if (last) copy8(p.x + size_t(n0 + warp) * C + (i * 32 + lane) * 8, x);
            }
          }
          add_squares(ss, x);
        }
        if (slot >= 0) unit_done(slot);
        if (follow) {
          wait(ctl.p1_full, par ^ 1u);
          norm_row(ss, last ? p.eps_final : p.layer[last ? 0 : l + 1].eps1, p.o_p1, [&](int i, const uint32_t (&v)[4]) {
            if (last && own(i))
              *reinterpret_cast<uint4*>(p.hidden_out + size_t(n0 + warp) * C + (i * 32 + lane) * 8) = make_uint4(v[0], v[1], v[2], v[3]);
          });
        }
      }
      if (follow) wait(ctl.p1_full, par ^ 1u);
      bar_compute();
      if (lane == 0) mbar_arrive(bar(ctl.p1_empty));
      if (l >= 0) u0 += layer_units(l);
    }

    // ---- side outputs: dispatch maps and l_balance of every layer, by the CTA that finishes last of one per cluster ----
    if (c != 0) return;
    if (p.n_clusters > 1) {
      if (warp == 0 && lane == 0) {
        __threadfence();
        int* done = reinterpret_cast<int*>(p.acc + (2 + E) * 8 + E * 4);
        ctl.last = atomicAdd(done, 1) == p.n_clusters - 1;
        __threadfence();
      }
      bar_compute();
      if (!ctl.last) return;
    }
    const double inv_tokens = 1.0 / double(p.N);
#pragma unroll 1
    for (int l = warp; l < p.n_layers; l += WARPS) {
      uint8_t* r = p.routing + l * p.routing_stride;
      constexpr int ROUNDS = (2 * MAX_CLUSTERS * (FULL ? 1 : MAX_TOKENS) + 31) / 32;
      sort_routes<E, ROUNDS>(reinterpret_cast<const long long*>(r + p.r_idx), p.N, lane, reinterpret_cast<int*>(r + p.r_counts),
                             reinterpret_cast<int*>(r + p.r_offsets), reinterpret_cast<int*>(r + p.r_scatter),
                             reinterpret_cast<int*>(r + p.r_gather), reinterpret_cast<int*>(r + p.r_gate_idx));
      if (lane == 0) {
        const double* a = reinterpret_cast<const double*>(p.acc + l * p.acc_stride) + 2;
        double pe[E];
        int hist[E];
        for (int e = 0; e < E; ++e) { pe[e] = __ldcg(a + e); hist[e] = __ldcg(reinterpret_cast<const int*>(a + E) + e); }
        p.scalars[size_t(l) * 3] = moe_l_balance(pe, hist, E, inv_tokens, p.layer[l].balance_alpha);
      }
    }
  }
};

template <bool FULL, bool STREAM>
__global__ void __launch_bounds__(THREADS, 1) step_cluster_kernel(const __grid_constant__ StepParams p) {
  extern __shared__ __align__(128) uint8_t step_smem[];
  __shared__ Ctl ctl;
  if (threadIdx.x == 0) {
#pragma unroll 1
    for (int i = 0; i < p.units; ++i) {
      mbar_init(smem_u32(&ctl.full[i]), 1);
      mbar_init(smem_u32(&ctl.empty[i]), 1);
    }
    mbar_init(smem_u32(&ctl.p1_full), 1);
    mbar_init(smem_u32(&ctl.p1_empty), WARPS);
    mbar_init(smem_u32(&ctl.p2_there), 1);
    mbar_init(smem_u32(&ctl.p2_full), 1);
    mbar_init(smem_u32(&ctl.p2_empty), WARPS);
    mbar_init(smem_u32(&ctl.got_o), 1);
    mbar_init(smem_u32(&ctl.got_x), 1);
    mbar_init(smem_u32(&ctl.got_h), 1);
    mbar_init(smem_u32(&ctl.got_y), 1);
    ctl.abort_flag = 0;
    fence_mbar_init();
  }
  __syncthreads();
  cluster_arrive();              // nobody writes into a CTA that has not set up its barriers, or that has left
  cluster_wait();
  pdl_wait();
  const int cluster = int(blockIdx.x) / CTAS, n0 = cluster * p.N / p.n_clusters;
  const Step<FULL, STREAM> s{p, ctl, step_smem, smem_u32(step_smem), warp_index(), int(threadIdx.x & 31), int(cluster_rank()), cluster, n0,
                     FULL ? 1 : (cluster + 1) * p.N / p.n_clusters - n0, &ctl.abort_flag};
  if (s.warp == WARPS) s.produce();
  else if (s.warp == WARPS + 1) s.settle();
  else s.compute();
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  if (s.warp < s.NT) s.membrane_out(p.n_layers - 1);
}

// ---- weights in fragment order: a block per 4 KB unit, a thread per 16 bytes -----------------------------------
// Chunk ch (128 in-features, eight steps of 16) of a tile: lane (g, t) has the codes of its A operands, row 2g steps 0-3 and 4-7, then
// row 2g + 1.  Word: pair j = 2 step + half (in-features 16 step + 8 half + 2t, + 1) at bits 2j and 16 + 2j, as
// (sign << 1) | nonzero, so that a shift and a mask give a bf16 pair of {0, +-2}.
__global__ void __launch_bounds__(256)
step_weights_kernel(const uint8_t* __restrict__ w_qkv, const uint8_t* __restrict__ w_out, const uint8_t* __restrict__ w1,
                    const uint8_t* __restrict__ w2, const float* __restrict__ gamma, const float* __restrict__ a_qkv,
                    const float* __restrict__ a_out, const float* __restrict__ a1, const float* __restrict__ a2,
                    uint8_t* __restrict__ out) {
  const int u = blockIdx.x, lane = threadIdx.x & 31, ch = threadIdx.x >> 5;
  uint4* dst = reinterpret_cast<uint4*>(out + size_t(u) * UNIT) + threadIdx.x;
  if (u >= T_END) {
    const int i = threadIdx.x;
    if (i >= SC_FLOATS) return;
    reinterpret_cast<float*>(out + size_t(u) * UNIT)[i] =
        i < SC_AQKV ? gamma[i] : i < SC_AOUT ? a_qkv[i - SC_AQKV] : i < SC_A1 ? a_out[0] : i < SC_A2 ? a1[i - SC_A1]
        : i < SC_A2 + E ? a2[i - SC_A2] : 0.f;
    return;
  }
  const uint8_t* rows;
  int tile, K = C, half = 0;
  if (u < T_OUT) { rows = w_qkv; tile = u; }
  else if (u < T_W1) { rows = w_out; tile = u - T_OUT; }
  else if (u < T_W2) { rows = w1; tile = u - T_W1; }
  else { rows = w2; tile = (u - T_W2) >> 1; half = (u - T_W2) & 1; K = HID; }
  const int g = lane >> 2, t = lane & 3;
  uint32_t v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {    // row 2g + (i >> 1), steps 4 (i & 1) ..
    const uint32_t* src = reinterpret_cast<const uint32_t*>(rows + size_t(tile * 16 + 2 * g + (i >> 1)) * (K / 4)) + half * 64 + ch * 8 +
                          4 * (i & 1);
    uint32_t o = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const uint32_t w = src[s];
      o |= ((w >> (2 * t)) & 0x00030003u) << (4 * s);
      o |= ((w >> (2 * (t + 4))) & 0x00030003u) << (4 * s + 2);
    }
    v[i] = o;
  }
  *dst = make_uint4(v[0], v[1], v[2], v[3]);
}

struct Plan {
  int units;
  uint32_t o_p1, o_p2, o_sc, o_rx, o_ry, o_xn, o_rh, o_qkv, o_ho, o_cs, o_scr, o_ring;
  size_t smem;
};
constexpr Plan plan_of(int tokens, bool full) {
  Plan s = {};
  uint32_t at = 0;
  auto take = [&](size_t n) { const uint32_t o = at; at += uint32_t((n + 127) / 128 * 128); return o; };
  s.o_p1 = take(C * 4);
  s.o_p2 = take(C * 4 + E * UNIT);
  s.o_sc = take(2 * SC_FLOATS * 4);
  s.o_rx = take(size_t(tokens) * C * 4);                                   // residual rows
  s.o_ry = take(size_t(tokens) * C * 4);                                   // the two expert outputs of a token, then their sum
  s.o_xn = take(size_t(tokens) * ROW_C);
  s.o_rh = take(size_t(tokens) * (full ? 2 * ROW_H : ROW_H));              // attention rows, then expert hidden rows
  s.o_qkv = take(size_t(tokens) * 3 * D * 2);
  s.o_ho = take(size_t(tokens) * D * 4);
  s.o_cs = take(size_t(tokens) * D * 4);
  s.o_scr = take(WARPS * SCRATCH);
  s.o_ring = at;
  s.units = int((DYN_MAX - at) / UNIT);
  if (s.units > MAX_UNITS) s.units = MAX_UNITS;
  s.smem = at + size_t(s.units) * UNIT;
  return s;
}
// unit_wait goes by parity, so the unit two turns before the awaited one must have been given back.  The producer works in order: what is a
// ring before the warp's last unit has been.  The two are at most sixteen units apart (32 with a token per cluster, where a
// warp may have no tile of a used expert; block barriers between them only help), hence rings of no fewer.
static_assert(plan_of(MAX_TOKENS, false).units >= 16 && plan_of(1, true).units >= 32, "the ring is too short for waits by parity");

bool stream_sums(int N) { return N * CTAS >= 64; }      // launch_attn_scan's choice

// Clusters of sixteen that are resident at once on the current device (0: none); asked once per device.
int max_clusters() {
  static std::atomic<int> known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int n = known[dev].load(std::memory_order_acquire);
  if (n == 0) {
    for (const void* k : {reinterpret_cast<const void*>(step_cluster_kernel<true, false>),
                          reinterpret_cast<const void*>(step_cluster_kernel<true, true>),
                          reinterpret_cast<const void*>(step_cluster_kernel<false, true>)}) {
      if (cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
          cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, int(DYN_MAX)) != cudaSuccess) {
        (void)cudaGetLastError();
        known[dev].store(-1, std::memory_order_release);
        return 0;
      }
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cfg.gridDim = CTAS; cfg.blockDim = THREADS; cfg.dynamicSmemBytes = DYN_MAX; cfg.attrs = at; cfg.numAttrs = 1;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CTAS; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    if (cudaOccupancyMaxActiveClusters(&n, step_cluster_kernel<false, true>, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      n = 0;
    }
    n = n < 1 ? -1 : n > MAX_CLUSTERS ? MAX_CLUSTERS : n;
    known[dev].store(n, std::memory_order_release);
  }
  return n > 0 ? n : 0;
}

}  // namespace

size_t step_weight_bytes(int c, int h, int e, int hidden) { return c == C && h == CTAS && e == E && hidden == HID ? LAYER_BYTES : 0; }
int step_max_sequences() { return max_clusters() * MAX_TOKENS; }

// Clusters that a step of N sequences runs in where `most` are resident at once; 0: kernel by kernel.  carried: every layer takes an
// attention state and leaves one.
//
// A sequence per cluster while there are clusters (two sequences in one cluster 591 us, in two 516), then two in each (8 sequences in two,
// three, four clusters 694, 657, 641 us), then as many as it takes.  From launch_attn_scan's limit on sums are attn_decode_stream_kernel's,
// which knows no call without states; several sequences in a cluster exist with these sums alone, so two or three sequences
// that do not get a cluster each (a device with room for one or two) are left to the kernels.
int step_clusters(int N, int most, bool carried) {
  if (most > MAX_CLUSTERS) most = MAX_CLUSTERS;
  if (N < 1 || N > most * MAX_TOKENS || (stream_sums(N) && !carried)) return 0;
  int n_cl = N <= most ? N : (N + 1) / 2;
  if (n_cl > most) n_cl = most;
  return n_cl < N && !stream_sums(N) ? 0 : n_cl;
}

int launch_step_weights(const jb200_layer* y, int c, int h, int e, int hidden, void* out, cudaStream_t stream) {
  JB_REQUIRE(y && out && y->w_qkv && y->w_out && y->w1 && y->w2 && y->gamma && y->a_qkv && y->a_out && y->a1 && y->a2,
             "step_weights: null pointer");
  JB_REQUIRE(step_weight_bytes(c, h, e, hidden) != 0, "step_weights: d_model %d / heads %d / experts %d x %d have no such form", c, h, e,
             hidden);
  JB_REQUIRE(aligned16(out) && aligned16(y->w_qkv) && aligned16(y->w_out) && aligned16(y->w1) && aligned16(y->w2),
             "step_weights: pointers must be 16-byte aligned");
  step_weights_kernel<<<T_END + 1, 256, 0, stream>>>(y->w_qkv, y->w_out, y->w1, y->w2, y->gamma, y->a_qkv, y->a_out, y->a1, y->a2,
                                                     static_cast<uint8_t*>(out));
  JB_LAUNCH_CHECK("step_weights_kernel");
  return JB200_OK;
}

int launch_step_cluster(const jb200_layer* layers, int n_layers, const jb200_forward* f, const void* const* weights, cudaStream_t stream,
                        bool* taken) {
  *taken = false;
  const int N = f->B;
  if (f->T != 1 || !weights || step_weight_bytes(f->C, f->H, f->E, f->hidden) == 0) return JB200_OK;
  bool carried = true;
  for (int l = 0; l < n_layers; ++l) {
    carried = carried && f->s_in && f->s_in[l] && f->s_out && f->s_out[l];
    if (!weights[l] || !aligned16(weights[l]) || !aligned16(f->h_out[l]) || (f->h_in && !aligned16(f->h_in[l]))) return JB200_OK;
  }
  const int n_cl = step_clusters(N, max_clusters(), carried);
  if (n_cl == 0) return JB200_OK;
  // States and membranes are fetched layers ahead: what one layer writes must not be what another one reads, nor its own input
  // except in place.
  for (int l = 0; l < n_layers; ++l)
    for (int k = 0; k < n_layers; ++k) {
      auto meet = [&](const float* a, const float* b, size_t n) { return a && b && !(k == l && a == b) && a < b + n && b < a + n; };
      if (meet(f->h_in ? f->h_in[l] : nullptr, f->h_out[k], size_t(N) * C) ||
          meet(f->s_in ? f->s_in[l] : nullptr, f->s_out ? f->s_out[k] : nullptr, size_t(N) * C * D)) return JB200_OK;
    }
  const int tokens = (N + n_cl - 1) / n_cl;
  const bool full = tokens == 1;
  const Plan s = plan_of(tokens, full);
  size_t off[7];
  StepParams p = {};
  // A layer's accumulators, and the words in which the sums of several clusters meet, lie in the workspace: the rest of it is not
  // used here.
  p.acc_stride = accumulator_bytes(E) + MAX_CLUSTERS * 32;
  if (forward_workspace_bytes(N, 1, C, CTAS, E, HID) < n_layers * p.acc_stride) return JB200_OK;
  p.routing_stride = routing_layout(N, E, off);
  p.r_idx = uint32_t(off[0]); p.r_gates = uint32_t(off[1]); p.r_counts = uint32_t(off[2]); p.r_offsets = uint32_t(off[3]);
  p.r_scatter = uint32_t(off[4]); p.r_gather = uint32_t(off[5]); p.r_gate_idx = uint32_t(off[6]);
  p.o_p1 = s.o_p1; p.o_p2 = s.o_p2; p.o_sc = s.o_sc; p.o_rx = s.o_rx; p.o_xn = s.o_xn; p.o_rh = s.o_rh; p.o_qkv = s.o_qkv;
  p.o_ho = s.o_ho; p.o_ry = s.o_ry; p.o_cs = s.o_cs; p.o_scr = s.o_scr; p.o_ring = s.o_ring; p.units = s.units;
  p.x = f->x; p.cos_tab = f->cos_tab; p.sin_tab = f->sin_tab; p.pos0 = f->pos0; p.pos0_scalar = f->pos0_scalar; p.n_pos = f->n_pos;
  p.N = N; p.n_clusters = n_cl; p.vocab = f->vocab;
  p.n_elems = double(N) * C; p.n_inv = 1.0 / p.n_elems; p.n1_inv = 1.0 / (p.n_elems - 1.0);
  p.units_inv = uint32_t(0xffffffffu / uint32_t(s.units)) + 1u;
  p.status = device_status_ptr();
  if (!p.status) return JB200_ERR_CUDA;
  if (n_cl > 1) JB_CUDA(cudaMemsetAsync(f->workspace, 0, n_layers * p.acc_stride, stream));
  for (int l0 = 0; l0 < n_layers; l0 += MAX_LAYERS) {
    const int n = n_layers - l0 < MAX_LAYERS ? n_layers - l0 : MAX_LAYERS;
    const bool end = l0 + n == n_layers;
    p.n_layers = n;
    p.ids = l0 == 0 ? f->ids : nullptr;
    p.table = f->table;
    p.w_final = end ? f->w_final : nullptr;
    p.eps_final = f->eps_final;
    p.hidden_out = reinterpret_cast<__nv_bfloat16*>(f->hidden_out);
    p.acc = static_cast<uint8_t*>(f->workspace) + l0 * p.acc_stride;
    p.routing = static_cast<uint8_t*>(f->routing) + l0 * p.routing_stride;
    p.scalars = f->scalars + size_t(l0) * 3;
    p.reflect = f->reflect ? f->reflect + l0 : nullptr;
    for (int i = 0; i < n; ++i) {
      const jb200_layer& y = layers[l0 + i];
      StepLayer& d = p.layer[i];
      d.tiles = static_cast<const uint8_t*>(weights[l0 + i]);
      d.w_norm1 = y.w_norm1; d.w_norm2 = y.w_norm2; d.w_router = y.w_router; d.var_scale = y.var_scale; d.mu = y.mu;
      d.s_in = f->s_in ? f->s_in[l0 + i] : nullptr; d.s_out = f->s_out ? f->s_out[l0 + i] : nullptr;
      d.h_in = f->h_in ? f->h_in[l0 + i] : nullptr; d.h_out = f->h_out[l0 + i];
      d.eps1 = y.eps1; d.eps2 = y.eps2; d.alpha_min = y.alpha_min; d.alpha_max = y.alpha_max; d.balance_alpha = y.balance_alpha;
      d.lam = y.reflect_lam; d.tau = y.reflect_tau;
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    cfg.gridDim = unsigned(n_cl * CTAS); cfg.blockDim = THREADS; cfg.dynamicSmemBytes = s.smem; cfg.stream = stream;
    cfg.attrs = at; cfg.numAttrs = 2;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CTAS; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    if (n_cl > 1) {
      at[1].id = cudaLaunchAttributeCooperative;
      at[1].val.cooperative = 1;
    } else {
      at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      at[1].val.programmaticStreamSerializationAllowed = dependent_launch_enabled() ? 1 : 0;
    }
    const cudaError_t e = !full ? cudaLaunchKernelEx(&cfg, step_cluster_kernel<false, true>, p)
                          : stream_sums(N) ? cudaLaunchKernelEx(&cfg, step_cluster_kernel<true, true>, p)
                                           : cudaLaunchKernelEx(&cfg, step_cluster_kernel<true, false>, p);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      if (l0 == 0 && e == cudaErrorCooperativeLaunchTooLarge) return JB200_OK;      // fewer SMs than the device has: kernel by kernel
      return cuda_fail(e, "step_cluster_kernel");
    }
    count_launch();
  }
  *taken = true;
  return JB200_OK;
}

}  // namespace jb
