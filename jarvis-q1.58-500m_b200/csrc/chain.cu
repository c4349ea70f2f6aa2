// Whole layers in one host call: the launch sequence of JarvisBlock.forward (jarvis_engine/jarvis_model.py:428-441) and
// of the model's loop around it (:498-516), issued from C++ over one caller-owned workspace.  A forward is a few
// hundred launches; issued one by one from Python they cost ~15 us each (5 ms for 24 layers), more than the GPU
// needs for anything below a few thousand tokens, issued here ~2 us each.
#include <algorithm>

#include "common.cuh"
#include "launchers.h"

namespace jb {

namespace {

inline size_t up(size_t n, size_t a) { return (n + a - 1) / a * a; }

struct Routing {
  size_t idx, gates, counts, offsets, scatter, gather, gate_idx, bytes;
  Routing(int N, int E) {
    size_t o = 0;
    auto take = [&](size_t n) { const size_t at = o; o += up(n, 16); return at; };
    idx = take(size_t(N) * 2 * 8);
    gates = take(size_t(N) * 2 * 4);
    counts = take(size_t(E) * 4);
    offsets = take(size_t(E + 1) * 4);
    scatter = take(size_t(N) * 2 * 4);
    gather = take(size_t(N) * 2 * 4);
    gate_idx = take(size_t(N) * 2 * 4);
    bytes = o;
  }
};

// Buffers of one layer, reused by the next: a kernel only ever overlaps its immediate predecessor, and nothing below
// writes what its predecessor still reads.
struct Workspace {
  size_t xn, qkv, o, hid, y, out, attn, lsf, meta, bytes;
  Workspace(int B, int T, int C, int H, int E, int hidden) {
    const size_t N = size_t(B) * T;
    size_t p = 0;
    auto take = [&](size_t n) { const size_t at = p; p += up(n, 256); return at; };
    xn = take(N * C * 2);
    qkv = take(N * 3 * C * 2);          // later the dispatched rows [2N][C]
    o = take(N * C * 2);                // later the MoE output
    hid = take(N * 2 * hidden * 2);
    y = take(N * 2 * C * 2);
    out = o;
    attn = take(T > 1 ? attn_scan_scratch_bytes(B, T, H) : 0);
    lsf = take(T > 1 ? lsf_scan_scratch_bytes(B, T, C) : 0);
    meta = take(std::max(moe_metadata_scratch_bytes(int(N), 2, E), (N + 7) / 8 * sizeof(unsigned long long)));
    bytes = p;
  }
};

// Which form of the ternary product a call of so many tokens runs (their results are the same bits): up to 16 tokens
// mma.sync straight from the codes (24 layers of single-token steps 0.62 against 0.86 ms at 1 sequence, equal at 16), up to
// MID_TOKENS the tcgen05 form that is built for latency, beyond that the persistent pipeline (when the line was drawn: 640 tokens 1.96
// against 2.08 ms with the pipeline, 900 2.20 against 2.29, 1000 equal, 1152 2.81 against 2.74).
constexpr int SMALL_TOKENS = 16, MID_TOKENS = 960;
// Up to here the first expert GEMM takes all rows for every expert and stores the routed ones: more MMAs, no dispatch.  A token without
// finite router logits is stored once, for expert 0, and its second hidden row holds whatever was there: combine and tail
// take the first one's output for both assignments (stored twice by the GEMM, 64 sequences were 1.5 % slower).  24 layers and head as a graph
// with the dispatch -> without: 80 tokens 1141 -> 1060 us, 128 1188 -> 1133, 5 x 30 1227 -> 1200, 180 1310 -> 1298, steps of 128 sequences
// 1360 -> 1326, 192 equal, 256 tokens 1375 -> 1423.  The same line for eight experts, though their MMAs are four times the routed ones, and
// for wide ones (d_model 1024, us a layer, 65, 100 and 160 tokens): 8 x 2048 48.8 -> 44.7, 52.5 -> 48.1, 58.0 -> 55.3; 4 x 4096 51.1 -> 47.9,
// 53.5 -> 50.4, 61.4 -> 58.5; 8 x 4096 61.2 -> 60.9, 67.1 -> 65.6, 76.8 -> 73.6; steps of 160 sequences 67.2 -> 65.5, 67.3 -> 65.4, 86.5 -> 80.2.
constexpr int ALL_ROWS_TOKENS = MID_ROUTE_TOKENS;
// Tiles of the latency form.  Tokens: the smallest multiple of 16 from r.least on that leaves a launch of so many rows in each group on
// r.most SMs; with tiles of 64 it may take `room` SMs, and from there on the tile grows until it does; where even one tile for all rows
// does not, that one.  (A larger one would be MMAs, copies and shared memory for rows that are not there: 256 rows where the first expert matrix has more than
// EXPERT_MOST tiles, us a layer at d_model 1024, 17, 37 and 128 tokens: 8 x 2048 49.4 -> 42.6, 50.5 -> 43.8, 51.4 -> 49.6; 4 x 4096 51.1 -> 44.0,
// 52.0 -> 45.3, 55.1 -> 53.6; 8 x 4096 74.6 -> 55.4, 74.7 -> 59.5, 70.8 -> 67.7.)
struct MidRule {
  int least, most;
};
inline int mid_tile(int rows, int groups, int n_ft, MidRule r, int room) {
  const int all = rows < 256 ? (rows + 15) / 16 * 16 : 256, usual = all < 64 ? all : 64;
  auto ctas = [&](int bn) { return long(n_ft) * groups * ((rows + bn - 1) / bn); };
  for (int bn = r.least; bn < usual; bn += 16)
    if (ctas(bn) <= r.most) return bn;
  int bn = usual;
  while (bn < all && ctas(bn) > room) bn += 16;
  return bn;
}
// Small tiles shorten chain and epilogue, but SMs that a launch takes are not there for the next one to begin on (barriers, codes
// fetched and decoded).  24 layers and head as a graph, tiles from 64 on -> these: 37 tokens 821 -> 780 us, 64 864 -> 836, 80 883 -> 850, 128 967 -> 902,
// 160 1049 -> 997, 256 1193 -> 1179, steps of 64, 128, 192 sequences 899 -> 875, 1166 -> 1120, 1342 -> 1328.  With other lines: q|k|v up to
// 124 SMs steps of 192 1341; out-projection up to 130 SMs 512 tokens 1522 -> 1551, from 32 tokens on 128 898 -> 927; second expert matrix up to
// 112 SMs 80 and 160 tokens 850 -> 868 and 997 -> 1016, the first one from 32 on up to 130 SMs 37 tokens 786 -> 816.
constexpr MidRule QKV_TILES = {16, 74}, OUT_TILES = {16, 100}, W1_TILES = {64, 0}, W2_TILES = {16, 74};
constexpr int EXPERT_MOST = 74;
struct MidTile {
  int bn, bn_max;
};
// Tiles of a launch: every group takes all M rows, or (cut) M rows are cut into segments that are known on the device alone: a
// tile for rows that are spread evenly, with an eighth to spare, and one for whatever they are (M / bn_max tiles and one cut short in
// every other group), up to one for all of them.
inline MidTile mid_plan(int M, int groups, int n_out, bool cut, MidRule r, int sms) {
  const int n_ft = n_out / MID_FEATURES, even = (M + groups - 1) / groups;
  if (!cut) {
    const int bn = mid_tile(M, groups, n_ft, r, groups > 1 ? EXPERT_MOST : sms);
    return {bn, bn};
  }
  MidTile t;
  t.bn = t.bn_max = mid_tile(even + (even + 7) / 8, groups, n_ft, r, sms);
  while (t.bn_max < 256 && t.bn_max < M && long(n_ft) * ((M + t.bn_max - 1) / t.bn_max + groups - 1) > sms) t.bn_max += 16;
  return t;
}

// Beyond MID_TOKENS the attention's products stay with the latency form while they are one wave of its largest tiles: a pair's 256 x 256
// tiles leave half of the SMs idle there, and its first tile is stored 10 us after the dependency.  24 layers and head with pairs ->
// out-projection in tiles of up to 256 rows: 1000 tokens 2178 -> 2101 us, 1800 2622 -> 2534, 3 x 777 3063 -> 2943, 4000 4140 -> 4047, 4600
// 4425 -> 4383; q|k|v as well: 1000 2101 -> 2054, 1300 2618 -> 2562, 1536 2553 -> 2526.  The same line for narrow models and other experts (us a
// layer, 4 x 2 d_model): 128 channels 961, 2368, 9000, 37,000 tokens 49.3 -> 43.4, 67.0 -> 60.3, 99.7 -> 94.2, 219.9 -> 214.9; 256, 9000 111.4 -> 109.8; 512, 9000
// 149.6 -> 146.0; 768, 4600 139.5 -> 135.6; nowhere slower, nor with eight experts or experts of four times d_model.
inline bool mid_wave(int N, int n_out, int sms) { return long(n_out / MID_FEATURES) * ((N + 255) / 256) <= sms; }

// The first expert matrix takes every token's row, or the assignments in segments; the second one always segments.
inline MidTile expert_plan(int tokens, bool second, int C, int E, int hidden, int sms) {
  const bool cut = second || tokens > ALL_ROWS_TOKENS;
  return mid_plan(cut ? 2 * tokens : tokens, E, second ? C : hidden, cut, second ? W2_TILES : W1_TILES, sms);
}

// Forms and tiles of a call's products.  Chunks of four K-blocks, where the rings of all products that run the same kernel hold them: each
// finds its code in the instruction cache after the one before, two kernels in turn do not (900 tokens, the out-projection alone in chunks of
// four: 1694 -> 1728 us).  Up to ALL_ROWS_TOKENS the expert matrices run kernels of their own.
struct Products {
  bool mid, mid_qkv, mid_out, coarse, w1_coarse, w2_coarse;
  MidTile qkv, out, w1, w2;
  Products(int N, bool small, int C, int E, int hidden, int sms)
      : mid(!small && N <= MID_TOKENS), mid_qkv(mid || (!small && mid_wave(N, 3 * C, sms))), mid_out(mid || (!small && mid_wave(N, C, sms))),
        qkv(mid_plan(N, 1, 3 * C, false, QKV_TILES, sms)), out(mid_plan(N, 1, C, false, OUT_TILES, sms)),
        w1(expert_plan(N, false, C, E, hidden, sms)), w2(expert_plan(N, true, C, E, hidden, sms)) {
    const bool all_rows = N <= ALL_ROWS_TOKENS;
    w1_coarse = mid && mid_gemm_coarse_fits(w1.bn_max, C);
    w2_coarse = mid && mid_gemm_coarse_fits(w2.bn_max, hidden);
    coarse = (!mid_qkv || mid_gemm_coarse_fits(qkv.bn_max, C)) && (!mid_out || mid_gemm_coarse_fits(out.bn_max, C)) &&
             (!mid || all_rows || (w1_coarse && w2_coarse));
    if (!all_rows) w1_coarse = w2_coarse = coarse;
  }
};

// What makes the dispatch maps of a call (counts, offsets, slots), and whether the router also leaves the assignments of every expert
// (`load`), from which the first expert matrix takes its segments while maps and rows are made; without them it takes the maps' offsets.  Up
// to ALL_ROWS_TOKENS there is no dispatch.  Beyond, maps and rows in one launch: from the ids on any device, or, where the router is a single
// pass of eight tokens a CTA, two CTAs an SM, from the counts that it leaves.  Times of the forms: dispatch_kernel.
struct Dispatch {
  enum Maker { ROUTER, EXPERT_GEMM, FROM_IDS, FROM_EIGHTS, METADATA } maps;
  bool load;
};
inline bool small_form(int N, int C, int hidden) { return N <= SMALL_TOKENS && small_gemm_fits(N <= 8 ? 8 : 16, std::max(C, hidden)); }
inline Dispatch dispatch_plan(int N, bool small, int sms) {
  static_assert(ROUTE_SMALL_MAX <= DISPATCH_IDS_MAX, "the router of few tokens leaves no counts of eight");
  if (N <= ALL_ROWS_TOKENS) return {small ? Dispatch::ROUTER : Dispatch::EXPERT_GEMM, false};
  if (N <= ROUTE_SMALL_MAX) return {Dispatch::FROM_IDS, true};
  if (N <= std::min(DISPATCH_EIGHTS_MAX, 16 * sms)) return {Dispatch::FROM_EIGHTS, true};
  return {Dispatch::METADATA, false};
}

#define JB_TRY(call)                    \
  do {                                  \
    const int rc__ = (call);            \
    if (rc__ != JB200_OK) return rc__;  \
  } while (0)

}  // namespace

int expert_tiles_host(int tokens, int second, int C, int E, int hidden, int sms, int32_t* out) {
  if (tokens < 1 || tokens > MID_TOKENS || C < 128 || E < 1 || hidden < 128 || sms < 1 || !out) return 0;
  const Products g(tokens, false, C, E, hidden, sms);
  const MidTile& t = second ? g.w2 : g.w1;
  const int K = second ? hidden : C;
  const bool coarse = second ? g.w2_coarse : g.w1_coarse;
  out[0] = !second && tokens <= ALL_ROWS_TOKENS;
  out[1] = MID_FEATURES; out[2] = t.bn; out[3] = t.bn_max;
  out[4] = mid_gemm_ring(t.bn, K, coarse).chunks; out[5] = mid_gemm_ring(t.bn_max, K, coarse).chunks;
  return 1;
}

int mid_ring_host(int bn, int K, int coarse, int32_t* out) {
  if (bn < 16 || bn > 256 || bn % 16 != 0 || K < 128 || !out) return 0;
  const MidRing r = mid_gemm_ring(bn, K, coarse != 0);
  out[0] = r.chunks; out[1] = r.kb; out[2] = r.tmem_cols; out[3] = r.smem;
  return r.chunks >= 1;
}

int dispatch_plan_host(int tokens, int C, int hidden, int sms, int32_t* out) {
  if (tokens < 1 || C < 128 || hidden < 128 || sms < 1 || !out) return 0;
  const Dispatch d = dispatch_plan(tokens, small_form(tokens, C, hidden), sms);
  out[0] = d.maps; out[1] = d.load;
  return 1;
}

size_t accumulator_bytes(int E) { return (size_t(2 + E) * 8 + size_t(2 * E + 1) * 4 + 7) / 8 * 8; }

size_t routing_layout(int N, int E, size_t* offsets) {
  const Routing r(N > 0 ? N : 0, E > 0 ? E : 0);
  if (offsets) {
    const size_t all[7] = {r.idx, r.gates, r.counts, r.offsets, r.scatter, r.gather, r.gate_idx};
    for (int i = 0; i < 7; ++i) offsets[i] = all[i];
  }
  return r.bytes;
}

size_t forward_workspace_bytes(int B, int T, int C, int H, int E, int hidden) {
  if (B <= 0 || T <= 0 || C <= 0 || H <= 0 || E <= 0 || hidden <= 0) return 0;
  return Workspace(B, T, C, H, E, hidden).bytes;
}

int forward_layers(const jb200_layer* layers, int n_layers, const jb200_forward* f, const void* const* step_weights, cudaStream_t st) {
  JB_REQUIRE(layers && f && n_layers >= 1, "forward_layers: null pointer or no layers");
  const int B = f->B, T = f->T, C = f->C, H = f->H, E = f->E, hidden = f->hidden;
  JB_REQUIRE(B >= 1 && T >= 1 && size_t(B) * T < (size_t(1) << 30), "forward_layers: bad shape (B=%d, T=%d)", B, T);
  JB_REQUIRE(C % 128 == 0 && C <= 1024 && C == 64 * H && hidden % 128 == 0 && (E == 4 || E == 8),
             "forward_layers: d_model %d / heads %d / hidden %d / experts %d not supported", C, H, hidden, E);
  JB_REQUIRE(f->x && f->cos_tab && f->sin_tab && f->h_out && f->accumulators && f->scalars && f->routing && f->workspace,
             "forward_layers: null pointer");
  JB_REQUIRE((f->w_final == nullptr) == (f->hidden_out == nullptr), "forward_layers: w_final and hidden_out come together");
  JB_REQUIRE(!f->ids || (f->table && f->vocab > 0), "forward_layers: ids without an embedding table");
  // Everything is looked at before the first launch: an error leaves x and the states as they were.
  const uintptr_t a8 = 7u, a256 = 255u;
  JB_REQUIRE(aligned16(f->x) && aligned16(f->cos_tab) && aligned16(f->sin_tab) && aligned16(f->routing) && aligned16(f->table) &&
                 aligned16(f->w_final) && aligned16(f->hidden_out) && (reinterpret_cast<uintptr_t>(f->accumulators) & a8) == 0 &&
                 (reinterpret_cast<uintptr_t>(f->workspace) & a256) == 0,
             "forward_layers: pointers must be 16-byte aligned (accumulators 8, workspace 256)");
  for (int l = 0; l < n_layers; ++l) {
    const jb200_layer& p = layers[l];
    JB_REQUIRE(p.w_norm1 && p.w_norm2 && p.w_router && p.gamma && p.var_scale && p.w_qkv && p.a_qkv && p.w_out && p.a_out &&
                   p.w1 && p.a1 && p.w2 && p.a2 && f->h_out[l],
               "forward_layers: a pointer of layer %d is missing", l);
    JB_REQUIRE(aligned16(p.w_norm1) && aligned16(p.w_norm2) && aligned16(p.w_router) && aligned16(p.w_qkv) &&
                   aligned16(p.w_out) && aligned16(p.w1) && aligned16(p.w2),
               "forward_layers: weights must be 16-byte aligned (layer %d)", l);
    const uintptr_t hs = reinterpret_cast<uintptr_t>(f->h_out[l]) | reinterpret_cast<uintptr_t>(f->h_in ? f->h_in[l] : nullptr);
    JB_REQUIRE((hs & a8) == 0 && aligned16(f->s_in ? f->s_in[l] : nullptr) && aligned16(f->s_out ? f->s_out[l] : nullptr),
               "forward_layers: attention states must be 16-byte aligned, membranes 8 (layer %d)", l);
  }
  if (T == 1 && step_weights) {
    bool taken = false;
    JB_TRY(launch_step_cluster(layers, n_layers, f, step_weights, st, &taken));
    if (taken) return JB200_OK;
  }
  const int N = B * T;
  const Workspace ws(B, T, C, H, E, hidden);
  const Routing rl(N, E);
  uint8_t* w = static_cast<uint8_t*>(f->workspace);
  uint16_t *xn = reinterpret_cast<uint16_t*>(w + ws.xn), *qkv = reinterpret_cast<uint16_t*>(w + ws.qkv);
  uint16_t *o = reinterpret_cast<uint16_t*>(w + ws.o), *hid = reinterpret_cast<uint16_t*>(w + ws.hid);
  uint16_t *y = reinterpret_cast<uint16_t*>(w + ws.y), *out = reinterpret_cast<uint16_t*>(w + ws.out);
  uint16_t* disp = qkv;
  float* x = f->x;
  const int small_tile = N <= 8 ? 8 : 16;
  const bool small = small_form(N, C, hidden);                  // beyond, the tcgen05 form streams K
  const bool all_rows = N <= ALL_ROWS_TOKENS;
  const int sms = sm_count();
  if (sms <= 0) return JB200_ERR_CUDA;
  const Dispatch by = dispatch_plan(N, small, sms);
  const Products g(N, small, C, E, hidden, sms);
  const bool mid = g.mid, mid_qkv = g.mid_qkv, mid_out = g.mid_out;
  auto mid_gemm = [&](const void* in, int M, int K, const uint8_t* wt, const float* al, int al_rows, int n_out, int G, const int32_t* seg,
                      const int32_t* counts, const MidRoutes* routes, int epi, void* dst, const MidTile& t, bool coarse) {
    return launch_mid_gemm(in, M, K, wt, al, al_rows, n_out, G, seg, counts, routes, epi, dst, t.bn, t.bn_max, coarse, st);
  };

  // the accumulators and the router's work counters are one block: cleared by the first kernel
  uint8_t* acc0 = static_cast<uint8_t*>(f->accumulators);
  const size_t acc_stride = accumulator_bytes(E);
  JB_TRY(launch_embed_norm(f->ids, f->table, f->vocab, layers[0].w_norm1, layers[0].eps1, x, xn, N, C, acc0, n_layers * acc_stride, st));

  for (int l = 0; l < n_layers; ++l) {
    const jb200_layer& p = layers[l];
    const bool last = l + 1 == n_layers;
    const float* s_in = f->s_in ? f->s_in[l] : nullptr;
    float* s_out = f->s_out ? f->s_out[l] : nullptr;
    const float* h_in = f->h_in ? f->h_in[l] : nullptr;
    float* h_out = f->h_out[l];
    const bool h16 = aligned16(h_in) && aligned16(h_out);      // the fused tails read 16 bytes at a time, the scan 8
    double* acc = reinterpret_cast<double*>(acc0 + l * acc_stride);            // sum, sum of squares, P_e
    int32_t* hist = reinterpret_cast<int32_t*>(acc + 2 + E);                   // top-1 counts
    int32_t* load = hist + E;                                                  // assignments
    int32_t* ticket = load + E;
    float* scalars = f->scalars + size_t(l) * 3;
    uint8_t* r = static_cast<uint8_t*>(f->routing) + size_t(l) * rl.bytes;
    int64_t* idx = reinterpret_cast<int64_t*>(r + rl.idx);
    float* gates = reinterpret_cast<float*>(r + rl.gates);
    int *counts = reinterpret_cast<int*>(r + rl.counts), *offs = reinterpret_cast<int*>(r + rl.offsets);
    int *scatter = reinterpret_cast<int*>(r + rl.scatter), *gather = reinterpret_cast<int*>(r + rl.gather);
    int* gate_idx = reinterpret_cast<int*>(r + rl.gate_idx);

    // x += attn(norm1(x))
    if (small)
      JB_TRY(launch_small_gemm(xn, N, C, p.w_qkv, p.a_qkv, C, 3 * C, 1, nullptr, nullptr, nullptr, JB200_EPI_BF16, qkv, small_tile, st));
    else if (mid_qkv)
      JB_TRY(mid_gemm(xn, N, C, p.w_qkv, p.a_qkv, C, 3 * C, 1, nullptr, nullptr, nullptr, JB200_EPI_BF16, qkv, g.qkv, g.coarse));
    else
      JB_TRY(launch_ternary_gemm(xn, N, C, p.w_qkv, p.a_qkv, C, 3 * C, 1, nullptr, JB200_EPI_BF16, qkv, 0, 1, st, nullptr, true));
    // a state updated in place needs one segment per sequence: later segments would read what the last one writes
    void* attn_scratch = (T > 1 && !(s_in && s_in == s_out)) ? w + ws.attn : nullptr;
    if (attn_scratch && ws.attn == ws.lsf) attn_scratch = nullptr;            // no scratch wanted at this shape
    JB_TRY(launch_attn_scan(qkv, qkv + C, qkv + 2 * C, 3 * C, p.gamma, f->cos_tab, f->sin_tab, f->n_pos, f->pos0, f->pos0_scalar,
                            s_in, o, C, s_out, attn_scratch, B, T, H, 64, 0, st, true));
    if (small)
      JB_TRY(launch_small_gemm(o, N, C, p.w_out, p.a_out, C, C, 1, nullptr, nullptr, nullptr, JB200_EPI_RESID_F32, x, small_tile, st));
    else if (mid_out)
      JB_TRY(mid_gemm(o, N, C, p.w_out, p.a_out, C, C, 1, nullptr, nullptr, nullptr, JB200_EPI_RESID_F32, x, g.out, g.coarse));
    else
      JB_TRY(launch_ternary_gemm(o, N, C, p.w_out, p.a_out, C, C, 1, nullptr, JB200_EPI_RESID_F32, x, 0, 1, st, nullptr, true));

    // moe(norm2(x)).  late_maps: the first expert GEMM makes the dispatch maps in a warp of its own, beside its MMAs; in the router
    // they are behind a fence, a ticket and a second reading of the ids.  24 layers and head as a graph so 80 tokens 1061 -> 1005 us, 128
    // 1139 -> 1098, 5 x 30 1199 -> 1157, steps of 100 sequences 1187 -> 1158; since its epilogue has its rows before the last MMA also
    // 17, 37, 64 tokens 766 -> 759, 780 -> 774, 836 -> 816 and steps of 57 840 -> 835.
    const bool late_maps = by.maps == Dispatch::EXPERT_GEMM;
    const MidRoutes store = {idx, false, counts, offs, scatter, gather, gate_idx};
    const MidRoutes rows_of = {idx, true, nullptr, nullptr, nullptr, nullptr, nullptr};
    int32_t* router_load = by.load ? load : nullptr;
    unsigned long long* counts8 = by.maps == Dispatch::FROM_EIGHTS ? reinterpret_cast<unsigned long long*>(w + ws.meta) : nullptr;
    if (N <= ROUTE_SMALL_MAX) {
      JB_TRY(launch_route_small(x, p.w_norm2, p.eps2, xn, p.w_router, N, C, E, idx, gates, acc + 2, hist, router_load, ticket,
                                counts, offs, by.maps == Dispatch::ROUTER ? scatter : nullptr, gather, gate_idx, st));
    } else {
      JB_TRY(launch_rmsnorm_router(x, p.w_norm2, p.eps2, xn, p.w_router, N, C, E, idx, gates, acc + 2, hist, st, true,
                                   router_load, counts8));
    }
    if (by.maps == Dispatch::METADATA)
      JB_TRY(launch_moe_metadata(idx, N, 2, E, counts, offs, scatter, gather, gate_idx, w + ws.meta, st));
    if (all_rows) {
      // every expert takes all rows where they are and stores the routed ones: no dispatch
      if (small)
        JB_TRY(launch_small_gemm(xn, N, C, p.w1, p.a1, hidden, hidden, E, nullptr, idx, scatter, JB200_EPI_GELU_BF16, hid, small_tile, st));
      else
        JB_TRY(mid_gemm(xn, N, C, p.w1, p.a1, hidden, hidden, E, nullptr, nullptr, &store, JB200_EPI_GELU_BF16, hid, g.w1, g.w1_coarse));
    } else {
      if (by.maps != Dispatch::METADATA) JB_TRY(launch_dispatch_chain(idx, counts8, xn, N, C, E, counts, offs, scatter, gather, gate_idx, disp, st));
      else JB_TRY(launch_dispatch_gather(xn, gather, 2 * N, N, C, disp, st));
      if (mid)
        JB_TRY(mid_gemm(disp, 2 * N, C, p.w1, p.a1, hidden, hidden, E, by.load ? nullptr : offs, router_load, nullptr, JB200_EPI_GELU_BF16, hid, g.w1, g.w1_coarse));
      else
        JB_TRY(launch_ternary_gemm(disp, 2 * N, C, p.w1, p.a1, hidden, hidden, E, offs, JB200_EPI_GELU_BF16, hid, 0, 1, st, nullptr, true, router_load));
    }
    if (small)
      JB_TRY(launch_small_gemm(hid, 2 * N, hidden, p.w2, p.a2, C, C, E, offs, nullptr, nullptr, JB200_EPI_BF16, y, small_tile, st));
    else if (mid)
      JB_TRY(mid_gemm(hid, 2 * N, hidden, p.w2, p.a2, C, C, E, late_maps ? nullptr : offs, nullptr, late_maps ? &rows_of : nullptr, JB200_EPI_BF16, y, g.w2, g.w2_coarse));
    else
      JB_TRY(launch_ternary_gemm(hid, 2 * N, hidden, p.w2, p.a2, C, C, E, offs, JB200_EPI_BF16, y, 0, 1, st, nullptr, true));

    // combine, x += lsf(moe), and the norm of what follows
    const float* w_next = last ? f->w_final : layers[l + 1].w_norm1;
    const float eps_next = last ? f->eps_final : layers[l + 1].eps1;
    void* xn_next = last ? f->hidden_out : static_cast<void*>(xn);
    const LsfStats stats = {acc, acc + 2, hist, E, N, (long long)N * C, p.balance_alpha, scalars,
                            p.mu, p.reflect_lam, p.reflect_tau, (f->reflect && p.mu) ? f->reflect + l : nullptr};
    if (h16 && N <= tail_max_tokens(C, T)) {
      JB_TRY(launch_tail(y, gates, scatter, idx, stats, p.var_scale, p.alpha_min, p.alpha_max, h_in, h_out, x, w_next, eps_next,
                         w_next ? xn_next : nullptr, B, T, C, st));
      continue;
    }
    JB_TRY(launch_scatter_combine(y, gates, scatter, N, 2, C, out, 1, acc, st, true, all_rows ? idx : nullptr));
    if (h16 && T == 1) {
      JB_TRY(launch_lsf_step_norm(out, stats, p.var_scale, p.alpha_min, p.alpha_max, h_in, h_out, x, w_next, eps_next,
                                  w_next ? xn_next : nullptr, B, C, st, true));
    } else {
      void* lsf_scratch = (h_in && h_in == h_out) || ws.lsf == ws.meta ? nullptr : w + ws.lsf;
      JB_TRY(launch_lsf_scan(out, 1, nullptr, nullptr, nullptr, p.var_scale, p.alpha_min, p.alpha_max, h_in, x, nullptr, 0,
                             h_out, 0, lsf_scratch, B, T, C, st, &stats));
      if (w_next) JB_TRY(launch_rmsnorm(x, 0, w_next, eps_next, xn_next, 1, N, C, st, true));
    }
  }
  return JB200_OK;
}

}  // namespace jb
