// Host-callable launchers of the MoE kernels; every one only enqueues on `stream`.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

struct gevva_moe;
struct gevva_dense;

namespace gv {

// gevva_moe_launch_stages and gevva_dense_launch on at most `sm_count` SMs (their persistent kernels
// take one CTA per SM): what lets the two sides of a feed-forward layer run beside each other.
int moe_launch_stages_on(gevva_moe* runner, const void* in, const int* ids, const float* route_weights, void* out,
                         int tokens, unsigned stages, cudaStream_t stream, int sm_count);
// (`status`: the word into which the dense kernels report a wait that ran out.)
int dense_launch_on(gevva_dense* dense, const void* in, void* out_unscaled, int tokens, cudaStream_t stream,
                    int sm_count, int* status);
int moe_sm_count(const gevva_moe* runner);
int moe_max_tokens(const gevva_moe* runner);
int current_sm_count();  // of the current device; 0 if the runtime does not say
// Whether the runner's expert GEMMs of a batch of this size are one launch that streams the weights.
bool moe_streams(const gevva_moe* runner, int tokens);

// Device-resident description of one launch's routing, written by the route sort
// and read by every later stage without a host round trip.
struct RoutePlan {
  int* sorted_experts;     // [R]   expert of sorted row
  int* sorted_routes;      // [R]   original route (8*token+k) of sorted row
  int* inverse_routes;     // [R]   sorted row of original route
  int* expert_offsets;     // [129] first sorted row of each expert, [128] = R
  int* scale_row_offsets;  // [129] first scale-factor row (128-row padded) of each expert
  int* tile_expert;        // [R/128 + 128] expert of each 128-row tile
  int* num_m_tiles;        // [1]
  int* pair_tile;          // optional [R/128 + 128]: 2 * (first tile of a pair) + (1 if the pair has two
                           // tiles); a pair = two consecutive 128-row tiles of one expert, or its last odd one
  int* num_pairs;          // optional [1]
  int* tile_ready;         // optional [R/128 + 128], zero on entry and on exit: per expert, w13 items that have
                           // stored their share of the w2 operand (streaming kernel)
  const int* tile_first;   // optional [1]: a GEMM launch covers tiles [tile_first, tile_first + num_m_tiles)
  int* chunk_hist;         // [ceil(R/1024) * 128] scratch of the multi-block sort
  int* status;             // [1]   device status word (gv::Status)
  const int* remap;        // optional [128]: sort key = remap[expert id] (expert-parallel placement)
  int* sync;               // optional [2], zero on entry: arrival/departure counters of the one-launch sort
  int* stream_sync;        // optional [kStreamSyncInts], zero on entry and on exit: counters of the streaming
                           // kernel (gv_stream_schedule.h)
};

// Weights that the kernel behind a launch begins with, asked into L2 by that launch (two arrays; empty: nothing is asked).
struct WeightsAhead {
  const uint8_t* base[2];
  uint32_t bytes[2];  // multiples of 16
};

void launch_route(const void* logits_bf16, int ld, const void* expert_scale_bf16, float* weights,
                  int* ids, int tokens, const float* activation_scales,
                  const float* projection_weight_scale, cudaStream_t stream);

// Router projection fused with routing: x [tokens, 2816] (bf16, or E4M3 with per-row scales) times
// router_w [128, 2816]^T, optional f32 bias, bf16 rounding, top-8 + softmax.  Returns a cudaError_t value.
int launch_route_project(const void* x, const void* router_w, bool fp8, const float* bias,
                         const void* expert_scale_bf16, float* weights, int* ids, void* logits_out,
                         const float* activation_scales, const float* weight_scale, int tokens, int* status,
                         cudaStream_t stream);

void launch_route_sort(const int* expert_ids, int routes, const RoutePlan& plan,
                       cudaStream_t stream);

// Route sort and input quantiser in one launch; at most 128 tokens (1024 routes).
constexpr int kFusedSortQuantizeMaxTokens = 128;
void launch_route_sort_quantize_small(const void* input_bf16, const int* expert_ids, const float* in_scale_q,
                                      const RoutePlan& plan, int tokens, uint8_t* packed, uint8_t* scales,
                                      cudaStream_t stream);

// bf16 [tokens, 2816] -> codes [R, 1408] (sorted order) + swizzled scale bytes.  behind_sort: the
// stream's previous kernel is the route sort of this batch.
void launch_quantize_input(const void* input_bf16, const int* expert_ids, const float* in_scale_q,
                           const RoutePlan& plan, int tokens, uint8_t* packed, uint8_t* scales, bool behind_sort,
                           const WeightsAhead& ahead, cudaStream_t stream);

// bf16 [R, 1408] ([up;gate]) -> codes [R, 352] + swizzled scale bytes.
void launch_geglu_quantize(const void* fused_bf16, const float* in_scale_q, const RoutePlan& plan,
                           int routes, uint8_t* packed, uint8_t* scales, cudaStream_t stream);

void launch_reduce_routes(const void* routed_bf16, const float* route_weights,
                          const int* inverse_routes, int tokens, void* output_bf16, bool behind_gemm,
                          cudaStream_t stream);

// Grouped NVFP4 GEMM: out[r, n] = bf16(alpha[e] * sum_k A[r,k] B[e,n,k]).
struct GemmOperands {
  CUtensorMap map_a;        // [row capacity, K/2] bytes, box 128 x 128 B, 128B swizzle
  CUtensorMap map_a32;      // same matrix through a 32-row box (groups of at most 32 rows)
  CUtensorMap map_b;        // [128*N, K/2] bytes, same box
  CUtensorMap map_b64;      // CTA-pair fused w13 form: the same matrix through a 64-row box
  CUtensorMap map_b_units;  // fused w13 form: [experts * 2 halves, 704 rows, 1408 bytes], box 2 x 64 rows x 128 B
  CUtensorMap map_b_down;   // w2: the weights in the column order of grouped_gemm_down.cu
  CUtensorMap map_down_pieces;  // grouped_gemm_down_pair.cu, dense_gemm_pair.cu: 32 weight rows in that order
  CUtensorMap map_down_a_sf, map_down_b_sf;  // grouped_gemm_down_pair.cu: the scales
  CUtensorMap map_a_sf;     // CTA-pair form: a_scales as [atoms of 512 B][128 x u32], box of four atoms
  CUtensorMap map_b_sf;     // CTA-pair form: b_scales likewise; box of eight atoms (fused w13) or four (w2)
  const uint8_t* a_scales;  // activation scale regions
  const uint8_t* b_scales;  // [128, N, K/16] swizzled per expert
  const float* alpha;       // [128]
  void* out;                // bf16 [row capacity, N]
  const unsigned long long* row_dest;  // optional: per-row output address instead of `out`
  int n_out;                // N: 1408 or 2816
  int k_in;                 // K: 2816 or 704
  // Fused w13 form (GeGLU + requantise in the epilogue, no bf16 output): weights through map_b_units
  // with unit_scales, results to the w2 operand buffers below.  (As CTA pairs: map_b, map_b64 and
  // the copy made by launch_retile_w13_scales in b_scales.)
  bool fused_geglu;
  const uint8_t* unit_scales;  // launch_retile_w13_unit_scales
  const uint8_t* down_scales;  // w2: launch_retile_w2_scales
  bool early_weights;         // the stream's previous kernel is one of this library's that lets its dependents go
                              // only after its own wait: the weights need not wait for it
  bool serial_launch;         // launch the ordinary way: no start before the stream's previous kernel ends
  bool use_pairs;             // NVFP4 forms with 256 weight rows per item: run as CTA pairs (tcgen05 cta_group::2)
                              // when the plan carries a pair list
  bool fp8;                   // dense E4M3 x E4M3 (no block scales); k_in counts bytes = elements
  bool wide;                  // fp8: 256 weight rows per item instead of 128
  uint8_t* next_codes;        // [row capacity, 352]
  uint8_t* next_scales;       // scale regions of the w2 operand
  const float* next_scale_q;  // g2.input_scale_quant [128]
};

void launch_grouped_gemm(const GemmOperands& op, const RoutePlan& plan, int sm_count,
                         cudaStream_t stream);

// w13 block scales [128,1408,176] (sidecar layout) -> per-item atoms for the fused form.
size_t retiled_w13_scale_bytes(int experts);
void launch_retile_w13_scales(const uint8_t* sidecar_scales, uint8_t* tiled, int experts,
                              cudaStream_t stream);

// Byte matrix [rows, row_bytes] seen through a box of box_rows x 128 bytes with the 128-byte
// swizzle; bytes out of range read as zero.  False if the driver entry point is missing.
bool make_operand_tensor_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes,
                             int box_rows);

// w13 codes [experts, 2 halves, 704 rows, 1408 bytes] through a box of both halves x 64 rows x 128 bytes.
bool make_w13_unit_tensor_map(CUtensorMap* map, const void* base, uint64_t experts);

// w2 codes [experts * 2816 rows, 352 bytes] as [64-row groups][8][4][2] rows with strides of 64, 2, 16 and 1
// rows, through a box of 192 rows x 128 bytes: the column order of grouped_gemm_down.cu.
bool make_piece_tensor_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes);  // 32 rows in that order
bool make_w2_down_tensor_map(CUtensorMap* map, const void* base, uint64_t experts);

// The w2 GEMM of prefill-sized batches (grouped_gemm_down.cu): op.map_a, map_b_down, down_scales.
size_t retiled_w2_scale_bytes(int experts);
void launch_retile_w2_scales(const uint8_t* sidecar_scales, uint8_t* tiled, int experts, cudaStream_t stream);
// The dense MLP of a few tokens (dense_few_rows.cu): rows of the caller's tensors aligned to 16 bytes.
constexpr int kDenseFewTokens = 2;
constexpr int kDenseFewUpRows = 48, kDenseFewDownRows = 32;  // weight rows of a CTA: of the gate and as many of the up projection, and of the down projection
struct DenseFewOperands {
  const void* input;               // bf16 [tokens, 2816]
  const CUtensorMap* map_gate_up;  // weights [2 (gate, up), 2112, 2816], boxes of kDenseFewUpRows rows of both
  const CUtensorMap* map_down;     // weights [2816, 2112], boxes of kDenseFewDownRows rows
  float gate_scale, up_scale;
  uint8_t *act_codes, *prod_codes;
  float *act_scales, *prod_scales;
  void* gate_up;                   // bf16 [tokens, 4224], unscaled
  void* products;                  // bf16 [kDenseFewTokens, 2112]
  void* out;                       // bf16 [tokens, 2816], unscaled
  int* status;
  bool serial_launch;              // the second launch does not begin before the first one has ended
};
// Weights [2, rows, row_bytes] through boxes of `box_rows` rows of both halves, 128-byte swizzle.
bool make_halves_tensor_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes, int box_rows);
int prepare_dense_few();
void launch_dense_few(const DenseFewOperands& op, int tokens, cudaStream_t stream);
// The dense projections by CTA pairs (dense_gemm_pair.cu): op.map_a, map_down_pieces, out, n_out, k_in.
int prepare_dense_pairs();
void launch_dense_pairs(const GemmOperands& op, int tokens, int* status, int sm_count, cudaStream_t stream);
// w2 by CTA pairs (grouped_gemm_down_pair.cu): op.map_a, map_down_pieces, map_down_a_sf, map_down_b_sf; all row tiles, no row_dest.
int prepare_grouped_down_pairs();
void launch_grouped_down_pairs(const GemmOperands& op, const RoutePlan& plan, int sm_count, cudaStream_t stream);
void launch_grouped_down(const GemmOperands& op, const RoutePlan& plan, int sm_count, cudaStream_t stream);
int prepare_grouped_down();

// Scale-factor bytes seen as rows of one 512-byte atom each (128 x u32), through a box of
// `box_atoms` consecutive atoms; no swizzle.
bool make_scale_tensor_map(CUtensorMap* map, const void* base, uint64_t bytes, int box_atoms);

// The CTA-pair form (grouped_gemm_pair.cu): fused w13 (op.fused_geglu) or plain w2 (n_out % 256 == 0).
void launch_grouped_gemm_pairs(const GemmOperands& op, const RoutePlan& plan, int sm_count, cudaStream_t stream);
int prepare_grouped_gemm_pairs();

// Fused w13 + GeGLU + requantise run by CTA pairs with the weights on the MMA's M side and up to
// 256 rows of one expert on its N side (grouped_gemm_w13_pair.cu).
constexpr int kW13PairBoxes = 16;
struct W13PairOperands {
  CUtensorMap map_x[kW13PairBoxes];  // activation codes [row capacity, 1408] bytes through boxes of 8, 16, ... 128 rows x 128 B
  CUtensorMap map_w;      // w13 codes in the row order of its MMAs, a unit of 64 columns (up and gate rows) a copy
  CUtensorMap map_x_sf;   // activation scale regions as [128-row blocks, 44 atoms, 512 B], box of one block x 4 atoms: a
                          // second copy where a chunk has rows in two blocks
  CUtensorMap map_w_sf;   // unit-tiled weight scales (launch_retile_w13_unit_scales), box of four atoms
  const float* alpha;           // [experts]
  uint8_t* next_codes;          // [row capacity, 352]
  uint8_t* next_scales;         // scale regions of the w2 operand
  const float* next_scale_q;    // [experts]
  bool serial_launch;
  bool early_weights;           // as in GemmOperands; the route plan too comes from before the previous kernel
};
size_t w13_unit_scale_bytes(int experts);
void launch_retile_w13_unit_scales(const uint8_t* sidecar_scales, uint8_t* tiled, int experts, bool fragments,
                                   cudaStream_t stream);
void launch_w13_pairs(const W13PairOperands& op, const RoutePlan& plan, int sm_count, cudaStream_t stream);
int prepare_w13_pairs();

// Both expert GEMMs of a batch with few rows an expert in one persistent launch with the weights on the
// MMA's M side (experts_stream.cu).
constexpr int kStreamBoxes = 8;         // activation boxes of 8, 16, ... 64 rows
constexpr int kStreamMaxTokens = 1024;  // the kernel's chunk list; where the launch pays is the caller's rule
struct StreamOperands {
  CUtensorMap map_w13;                 // make_w13_unit_tensor_map
  CUtensorMap map_w2;                  // [128 * 2816, 352] bytes, box 128 x 128 B
  CUtensorMap map_up[kStreamBoxes];    // input codes [row capacity, 1408] through boxes of 8(i+1) rows x 128 B
  CUtensorMap map_down[kStreamBoxes];  // w2 operand codes [row capacity, 352] likewise
  const uint8_t* w13_scales;           // launch_retile_w13_unit_scales
  const uint8_t* w2_scales;            // sidecar layout
  const uint8_t* input_scales;
  uint8_t* inter_codes;
  uint8_t* inter_scales;
  void* routed;                        // bf16 [row capacity, 2816]
  const float *alpha1, *alpha2, *in_scale_q2;
};
// On a sorted plan and a quantised input; plan.tile_ready (by expert here) and plan.stream_sync zero on
// entry and on exit.
void launch_stream_experts(const StreamOperands& op, const RoutePlan& plan, int sm_count, cudaStream_t stream);
// With the route sort and the input quantiser inside, where stream_layer_fits.
bool stream_layer_fits(int tokens, int sm_count);
void launch_stream_layer(const StreamOperands& op, const RoutePlan& plan, const void* input_bf16, const int* expert_ids,
                         const float* in_scale_q1, uint8_t* packed, uint8_t* scales, int tokens, int sm_count,
                         cudaStream_t stream);
int prepare_stream_experts();

// Must be called once per device before launch_grouped_gemm (sets the dynamic
// shared-memory limit).  Returns a cudaError_t value.
int prepare_grouped_gemm();

// Synthetic-expert packer: fp32 [experts, N, K] -> NVFP4 codes, swizzled scale
// bytes and the per-expert global scale amax/(6*448).
void launch_pack_weights(const float* weights, int experts, int n_out, int k_in, uint8_t* codes,
                         uint8_t* scales, float* global_scales, cudaStream_t stream);

// ---- feed-forward steps around the expert path and the dense FP8 MLP (dense_ff.cu) ------
void launch_ff_prepare(const void* input, const void* dense_weight, const void* expert_weight,
                       const void* router_scale, void* dense_out, void* expert_out, void* router_out,
                       int rows, cudaStream_t stream);
// Also writes the plan of the dense projections seen as grouped GEMMs with one group.
void launch_fp8_quantize_rows(const void* input, uint8_t* out, float* scales, int rows, bool weights_ahead, const RoutePlan& plan,
                              cudaStream_t stream);
void launch_gelu_quantize_fp8(const void* gate_up, const float* activation_scales, float gate_w_scale,
                              float up_w_scale, const float* gelu_table, uint8_t* out, float* scales, int rows,
                              int sm_count, bool serial_launch, cudaStream_t stream);
void launch_ff_finalize(const void* dense, const void* dense_weight, const void* expert_routes,
                        const float* route_weights, const int* inverse_routes, const void* expert_weight,
                        const void* combined_weight, const void* residual, const void* layer_scalar,
                        void* output, int rows, const float* dense_activation_scales,
                        const float* dense_projection_scale, cudaStream_t stream);
void launch_pack_fp8(const float* w, size_t count, uint8_t* out, float* scale_out, cudaStream_t stream);

}  // namespace gv
