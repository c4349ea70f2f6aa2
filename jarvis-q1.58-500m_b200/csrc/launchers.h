// Host-side launch functions implemented by the kernel translation units and called by the
// extern "C" layer in api.cu.  All return JB200_OK / JB200_ERR_ARG / JB200_ERR_CUDA.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "jarvis_b200.h"

namespace jb {

size_t pack_ternary_scratch_bytes(int out_features, int in_features);
int launch_pack_ternary(const float* w, int out_features, int in_features, const float* alpha_in, uint8_t* packed,
                        float* alpha_out, void* scratch, cudaStream_t stream);
int launch_pack_codes(const float* w_ternary, size_t n_elems, uint8_t* packed, cudaStream_t stream);
int launch_unpack_ternary(const uint8_t* packed, size_t n_bytes, int out_dtype, void* out, cudaStream_t stream);

// Extra arguments of the JB200_EPI_QK_ROPE_BF16 epilogue (q/k/v projection fused with the attention prologue).
struct GemmRope {
  const float* cos_tab;   // [n_pos][32]
  const float* sin_tab;
  const int32_t* pos0;    // [M / T] or null
  int pos0_scalar, n_pos, T, rope_feats;
};
int launch_ternary_gemm(const void* x_bf16, int M, int K, const uint8_t* w_packed, const float* alpha,
                        int alpha_rows, int N, int G, const int32_t* seg_offsets, int epilogue, void* out,
                        int bn_override, int w_layout, cudaStream_t stream, const GemmRope* rope = nullptr, bool settled = false,
                        const int32_t* seg_counts = nullptr);
// The same product for a few tokens (small_gemm.cu), bit for bit; bf16, GELU and residual epilogues.  idx / scatter ([M][2]):
// all M rows go through every group's matrix and row n is stored at scatter[2n + k] where idx[2n + k] is the group; else seg
// as above.  tile: rows a CTA takes at a time, 8 or 16.  Within a chain only: weights
// and seg were complete before the kernel ahead of this one on the stream began, and are read while it runs.
int launch_small_gemm(const void* x_bf16, int M, int K, const uint8_t* w_prepared, const float* alpha, int alpha_rows, int N,
                      int G, const int32_t* seg, const int64_t* idx, const int32_t* scatter, int epilogue, void* out,
                      int tile, cudaStream_t stream);
// It keeps whole rows of codes and activations in shared memory: in-features it can take with such tiles (about 7200 with 8
// rows, 4800 with 16).
bool small_gemm_fits(int tile, int K);
// The same product again, latency form on tcgen05 (mid_gemm.cu) with tiles of bn rows, or of bn_max rows where the segments
// need more tiles of bn than there are SMs.  Arguments as launch_small_gemm, but for routes
// (top-2 assignments of at most MID_ROUTE_TOKENS tokens).  Every group takes all M rows, the routed ones are stored in dispatch order, and
// the maps are left in scatter and the others.  With segments (no maps) the M rows
// are the assignments in that order.
constexpr int MID_ROUTE_TOKENS = 160;
struct MidRoutes {
  const int64_t* ids;          // [tokens][2]
  bool segments;
  int *counts, *offsets, *scatter, *gather, *gate_idx;
};
int launch_mid_gemm(const void* x_bf16, int M, int K, const uint8_t* w_prepared, const float* alpha, int alpha_rows, int N, int G,
                    const int32_t* seg, const int32_t* counts, const MidRoutes* routes, int epilogue, void* out, int bn, int bn_max,
                    bool coarse, cudaStream_t stream);
constexpr int MID_FEATURES = 128;              // out-features of its tiles
struct MidRing {
  int chunks, kb, tmem_cols, smem;             // chunks in flight, K-blocks of one, tensor-memory columns and shared memory in use
};
MidRing mid_gemm_ring(int bn, int K, bool coarse);      // its ring with token tiles of bn rows; no chunks where K is not a multiple of one
bool mid_gemm_coarse_fits(int bn, int K);      // `coarse`, chunks of four K-blocks in place of two: where its ring still holds three
int launch_prepare_weights(const uint8_t* packed, size_t n_bytes, uint8_t* prepared, cudaStream_t stream);
void decode16_host(uint32_t w, uint32_t* out8);
void decode16_prepared_host(uint32_t w_canonical, uint32_t* out8);

// ahead (here and below): the weights were complete before the kernel ahead of this one on the stream began, so they may be
// fetched before it ends.  True within jb200_forward_layers; a caller of a single stage may have just written them.
int launch_rmsnorm(const void* x, int x_dtype, const float* w, float eps, void* y, int y_dtype, int n_rows, int C,
                   cudaStream_t stream, bool ahead = false);
int launch_embedding(const int64_t* idx, const float* table, int vocab, float* out, int n_rows, int C,
                     cudaStream_t stream);

int launch_router_top2(const void* x_bf16, const float* w_router, int n_tokens, int C, int E, int64_t* topk_idx,
                       float* gates, float* probs_out, double* probs_sum, int* top1_hist, cudaStream_t stream);
int launch_rmsnorm_router(const float* x, const float* w_norm, float eps, void* xn_bf16, const float* w_router,
                          int n_tokens, int C, int E, int64_t* topk_idx, float* gates, double* probs_sum,
                          int* top1_hist, cudaStream_t stream, bool ahead = false, int* load = nullptr,
                          unsigned long long* counts8 = nullptr);
size_t moe_metadata_scratch_bytes(int n_tokens, int K, int E);
// Maps and rows of top-2 assignments at once.  scratch: moe_dispatch_scratch_bytes.
size_t moe_dispatch_scratch_bytes(int n_tokens, int E);
int launch_moe_dispatch(const int64_t* topk_idx, const void* x_bf16, int n_tokens, int C, int E, void* scratch, int* expert_counts,
                        int* expert_offsets, int* scatter_map, int* gather_map, int* gate_idx_map, void* dispatched, cudaStream_t stream);
// The same in one launch, inside a chain.  counts8: what launch_rmsnorm_router left, the assignments of every eight tokens, a byte per
// expert; null: counted from the ids.  Bounds: as far as each was measured to be the faster one (148 SMs, where a single pass of the router ends
// at 2368 tokens); a thread adds up to 255 assignments of an expert in a byte.
constexpr int DISPATCH_IDS_MAX = 512, DISPATCH_EIGHTS_MAX = 2368;
int launch_dispatch_chain(const int64_t* topk_idx, const unsigned long long* counts8, const void* x_bf16, int n_tokens, int C, int E,
                          int* expert_counts, int* expert_offsets, int* scatter_map, int* gather_map, int* gate_idx_map, void* dispatched,
                          cudaStream_t stream);
int launch_moe_metadata(const int64_t* topk_idx, int n_tokens, int K, int E, int* expert_counts, int* expert_offsets,
                        int* scatter_map, int* gather_map, int* gate_idx_map, void* scratch, cudaStream_t stream);
int moe_metadata_static_max_assignments();
int launch_moe_metadata_static(const int64_t* topk_idx, int n_tokens, int K, int E, int* expert_counts,
                               int* expert_offsets, int* scatter_map, int* gather_map, int* gate_idx_map,
                               cudaStream_t stream);
int launch_dispatch_gather(const void* x_bf16, const int* gather_map, int M, int n_tokens, int C, void* dispatched,
                           cudaStream_t stream);
// topk_idx (top-2 of a chain only, or null): a token whose second id is -1 takes its first row twice.
int launch_scatter_combine(const void* y_bf16, const float* gates, const int* scatter_map, int n_tokens, int K, int C,
                           void* out, int out_dtype, double* stats, cudaStream_t stream, bool ahead = false,
                           const int64_t* topk_idx = nullptr);
int launch_moe_finalize(const double* stats, const double* probs_sum, const int* top1_hist, int E, long long n_tokens,
                        long long n_elems, float balance_alpha, float* scalars, cudaStream_t stream);

// Accumulators of the MoE layer whose output an LSF call scans: the scan derives act_var from them and leaves the
// layer's scalars (l_balance, act_mean, act_var), so that no launch of its own is needed for those.
struct LsfStats {
  const double* stats;       // [2] sum, sum of squares; null: not used
  const double* probs_sum;   // [E]
  const int* top1_hist;      // [E]
  int E;
  long long n_tokens, n_elems;
  float balance_alpha;
  float* scalars;            // [3] out
  const float* mu;           // with reflect: the layer's reflective penalty is left there
  float lam, tau;
  float* reflect;            // [1] out or null
  // the counts as doubles with their reciprocals, for the quotients on the device: filled by the launch functions
  double n_tok, inv_tok, n_el, inv_el, inv_el1;
  LsfStats counted() const {
    LsfStats s = *this;
    s.n_tok = double(n_tokens); s.inv_tok = 1.0 / s.n_tok;
    s.n_el = double(n_elems); s.inv_el = 1.0 / s.n_el; s.inv_el1 = 1.0 / (s.n_el - 1.0);
    return s;
  }
};
int launch_lsf_scan(const void* m, int m_dtype, const void* alpha_tensor, const float* alpha_scalar,
                    const float* act_var, const float* var_scale, float alpha_min, float alpha_max, const float* h0,
                    float* resid, void* out, int out_dtype, void* h_last, int last_dtype, void* scratch, int B, int T, int D,
                    cudaStream_t stream, const LsfStats* st = nullptr);
size_t lsf_scan_scratch_bytes(int B, int T, int D);
int launch_lsf_step_norm(const void* m_bf16, const LsfStats& st, const float* var_scale, float alpha_min, float alpha_max,
                         const float* h_in, float* h_out, float* x, const float* w_norm, float eps, void* xn_bf16, int B,
                         int C, cudaStream_t stream, bool ahead = false);

// settled: gamma, angle tables, pos0 and, at T == 1, s_in were complete before the kernel ahead of this one on the stream began.
int launch_attn_scan(const void* q, const void* k, const void* v, int ld_qkv, const float* gamma,
                     const float* cos_tab, const float* sin_tab, int n_pos, const int32_t* pos0, int pos0_scalar,
                     const float* s_in, void* o, int ld_o, float* s_out, void* scratch, int B, int T, int H,
                     int head_dim, int flags, cudaStream_t stream, bool settled = false);
size_t attn_scan_scratch_bytes(int B, int T, int H);

// Few tokens (moe_small.cu).
constexpr int ROUTE_SMALL_MAX = 512, ROUTE_SORT_MAX = 16;   // tokens; tokens with maps
int tail_max_tokens(int C, int T);     // most tokens that launch_tail takes: 128 of single-token steps, 12 for every 64 channels of prompts
int launch_embed_norm(const int64_t* ids, const float* table, int vocab, const float* w_norm, float eps, float* x, void* xn_bf16,
                      int n_rows, int C, void* zero, size_t zero_bytes, cudaStream_t stream);
// scatter null: the assignments alone, no maps.  load: how many of them every expert has, or null.
int launch_route_small(const float* x, const float* w_norm, float eps, void* xn_bf16, const float* w_router, int N, int C, int E,
                       int64_t* idx, float* gates, double* probs_sum, int* hist, int* load, int* ticket, int* counts, int* offsets,
                       int* scatter, int* gather, int* gate_idx, cudaStream_t stream);
int launch_tail(const void* y_bf16, const float* gates, const int* scatter, const int64_t* idx, const LsfStats& st,
                const float* var_scale, float alpha_min, float alpha_max, const float* h_in, float* h_out, float* x,
                const float* w_norm, float eps, void* xn_bf16, int B, int T, int C, cudaStream_t stream);
// A single-token step of all layers in one launch (step_cluster.cu).  weights[l]: launch_step_weights' layout of layer l
// (step_weight_bytes, 0 where there is no such form).  taken: false where the call is not one of its kind and nothing was done.
size_t step_weight_bytes(int C, int H, int E, int hidden);
int step_max_sequences();
int step_clusters(int N, int most, bool carried);
int launch_step_weights(const jb200_layer* layer, int C, int H, int E, int hidden, void* out, cudaStream_t stream);
int launch_step_cluster(const jb200_layer* layers, int n_layers, const jb200_forward* f, const void* const* weights,
                        cudaStream_t stream, bool* taken);
int launch_cross_entropy(const void* logits, int ld, int n_rows, int V, const int64_t* targets, float* row_loss,
                         const float* aux_a, int stride_a, const float* aux_b, int n_aux, float* loss, cudaStream_t stream);
int mid_ring_host(int bn, int K, int coarse, int32_t* out);
int dispatch_plan_host(int tokens, int C, int hidden, int sms, int32_t* out);
int expert_tiles_host(int tokens, int second, int C, int E, int hidden, int sms, int32_t* out);
size_t accumulator_bytes(int E);
size_t routing_layout(int N, int E, size_t* offsets);
size_t forward_workspace_bytes(int B, int T, int C, int H, int E, int hidden);
int forward_layers(const jb200_layer* layers, int n_layers, const jb200_forward* f, const void* const* step_weights, cudaStream_t stream);

int launch_peer_barrier(const void* const* peer_flags, int world, int rank, cudaStream_t stream);
int launch_ep_pull_gather(const void* const* peer_offs, const void* const* peer_gmap, const void* const* peer_xn,
                          int world, int rank, int E, int C, int K, int n_max, int max_rows, void* dispatched,
                          int32_t* seg_offsets, int32_t* meta, cudaStream_t stream);
int launch_ep_pull_combine(const void* const* peer_y, const void* const* peer_meta, const int32_t* offs_local,
                           const int64_t* topk_idx, const float* gates, const int32_t* scatter_map, int world, int rank,
                           int E, int C, int K, int n_tokens, int max_rows, void* out, int out_dtype, double* stats,
                           cudaStream_t stream);
int launch_sample(const void* logits, int logits_dtype, int ld, int n_rows, int V, float temperature, int top_k,
                  float top_p, const float* u, int64_t* out_token, float* out_prob, cudaStream_t stream);

}  // namespace jb
