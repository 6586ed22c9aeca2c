// C ABI of the dense FP8 GeGLU MLP and of the feed-forward steps before and after the
// expert path (declared in include/gevva_moe.h).  The reference runs the three dense
// projections through cuBLASLt (Fp8LinearRunner::launch_unscaled,
// src/cuda/runtime/fp8_linear.cuh:215-473, called at src/cuda/runtime/prefill.cuh:1211-1230);
// here they are the tcgen05 kernels of dense_gemm_pair.cu or, beside the experts, of grouped_gemm.cu in its FP8 form; dense_few_rows.cu for
// one or two tokens.
#include <cuda.h>
#include <cuda_runtime.h>

#include <new>

#include "../../include/gevva_moe.h"
#include "gv_common.cuh"
#include "gv_exact.h"
#include "gv_launchers.h"

namespace {
constexpr int kDense = 2112;
}

struct gevva_dense {
  gevva_dense_weights weights{};
  int max_tokens = 0;
  int sm_count = 0;
  gv::RoutePlan plan{};
  gv::GemmOperands gate_up{}, down{};
  CUtensorMap map_few_gate_up{}, map_few_down{};  // of the weights, for up to kDenseFewTokens tokens
  uint8_t* act_fp8 = nullptr;     // [T, 2816]
  float* act_scales = nullptr;    // [T]
  void* gate_up_out = nullptr;    // bf16 [T, 4224], unscaled
  uint8_t* prod_fp8 = nullptr;    // [T, 2112]
  float* prod_scales = nullptr;   // [T]
  void* few_products = nullptr;   // bf16 [kDenseFewTokens, 2112]
  float* ones = nullptr;          // [128]
  float* gelu_table = nullptr;    // [GV_GELU_FLOATS]
  float* down_scale = nullptr;    // [1]: weights.down_scale on the device, for gevva_ff_finalize
  int* ints = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;  // gevva_ff_layer_launch: to the second stream and back
};

// Whether a GEMM of the dense MLP takes 256 weight rows an item instead of 128.  The launch lasts as many items
// as its busiest CTA has, and a wide item takes about one and a half times a narrow one (48 KB of operands a K
// block against 32 KB): wide where that is no longer.  Alone on 148 SMs (where pairs of CTAs run now, but for outputs that they cannot store)
// the MLP took (us, narrow -> wide)
// 31.9 -> 35.4 at 301 tokens, where one wave of narrow items is enough, 39.0 -> 35.5 at 600, 74.8 -> 62.6 at 2048
// and 131.9 -> 108.4 at 4096.  On the few SMs that it gets beside the experts of a decode batch (whole layers in a graph):
// 57.5 -> 53.7 at 8 tokens, 71.6 -> 71.8 at 16, 91.4 -> 91.9 at 40, 95.9 -> 95.7 at 64, 104.1 -> 103.2 at 128.
static bool wide_items(int tokens, int n_out, int sms) {
  const int row_tiles = (tokens + gv::kTileM - 1) / gv::kTileM;
  const int narrow = (row_tiles * ((n_out + 127) / 128) + sms - 1) / sms;
  const int wide = (row_tiles * ((n_out + 255) / 256) + sms - 1) / sms;
  return 3 * wide <= 2 * narrow;
}

int gv::dense_launch_on(gevva_dense* d, const void* in, void* out_unscaled, int tokens, cudaStream_t stream,
                        int sm_count, int* status) {
  if (tokens <= gv::kDenseFewTokens) {
    // (these need no plan)
    gv::DenseFewOperands op{};
    op.input = in;
    op.map_gate_up = &d->map_few_gate_up;
    op.map_down = &d->map_few_down;
    op.gate_scale = d->weights.gate_scale;
    op.up_scale = d->weights.up_scale;
    op.act_codes = d->act_fp8;
    op.prod_codes = d->prod_fp8;
    op.act_scales = d->act_scales;
    op.prod_scales = d->prod_scales;
    op.gate_up = d->gate_up_out;
    op.products = d->few_products;
    op.out = out_unscaled;
    op.status = status;
    op.serial_launch = sm_count < d->sm_count;
    gv::launch_dense_few(op, tokens, stream);
    return cudaGetLastError() == cudaSuccess ? GEVVA_MOE_OK : GEVVA_MOE_CUDA_ERROR;
  }
  gv::RoutePlan plan = d->plan;
  plan.status = status;
  // By CTA pairs where the MLP has all SMs (figures in dense_gemm_pair.cu).  On the few that it gets beside the experts, whose weight
  // stream bounds the layer, the one-CTA kernels are as fast or faster: whole layers in a graph 16 tokens 264.8 and 266.6 us by pairs, 40 tokens
  // 337 and 343, 301 tokens 321 and 322, 640 tokens 363.5 and 366.
  // The pair kernel stores 32 bytes at a time; rows are whole multiples of that, so an output that is aligned to 16 only, as the
  // one-CTA kernel takes it, goes there (same bits; the MLP takes 54.4 us instead of 46.5 then at 2048 tokens, 27.4 instead of 24.6 at 301).
  const bool pairs = sm_count >= 2 && sm_count == d->sm_count;
  gv::launch_fp8_quantize_rows(in, d->act_fp8, d->act_scales, tokens, pairs, plan, stream);
  const auto project = [&](gv::GemmOperands op) {
    if (pairs && (reinterpret_cast<uintptr_t>(op.out) & 31) == 0) {
      gv::launch_dense_pairs(op, tokens, status, sm_count, stream);
    } else {
      op.wide = wide_items(tokens, op.n_out, sm_count);
      gv::launch_grouped_gemm(op, plan, sm_count, stream);
    }
  };
  project(d->gate_up);
  // Beside the experts this kernel is launched the ordinary way: its CTAs, one a token, would otherwise wait out the first
  // projection on SMs that the streaming launch's last CTAs need (296 tokens with 16 dense SMs: 373 -> 2000 us for three layers,
  // because tokens of CTAs that are not running are then quantised by the others one by one).  Whole layers in a graph, us, chained and
  // ordinary: 16 tokens 271 and 268 (four layers), 100 tokens 371 and 368, 128 tokens 390 and 380.  A dozen CTAs fit anywhere.
  const bool beside = sm_count < d->sm_count;
  gv::launch_gelu_quantize_fp8(d->gate_up_out, d->act_scales, d->weights.gate_scale, d->weights.up_scale,
                               d->gelu_table, d->prod_fp8, d->prod_scales, tokens, sm_count, beside && tokens > 12, stream);
  gv::GemmOperands down = d->down;
  down.out = out_unscaled;
  project(down);
  return cudaGetLastError() == cudaSuccess ? GEVVA_MOE_OK : GEVVA_MOE_CUDA_ERROR;
}

extern "C" {

void gevva_dense_destroy(gevva_dense* d) {
  if (!d) return;
  cudaFree(d->act_fp8);
  cudaFree(d->act_scales);
  cudaFree(d->gate_up_out);
  cudaFree(d->prod_fp8);
  cudaFree(d->prod_scales);
  cudaFree(d->few_products);
  cudaFree(d->ones);
  cudaFree(d->gelu_table);
  cudaFree(d->down_scale);
  cudaFree(d->ints);
  if (d->fork) cudaEventDestroy(d->fork);
  if (d->join) cudaEventDestroy(d->join);
  delete d;
}

int gevva_dense_create(gevva_dense** out, const gevva_dense_weights* weights, int max_tokens) {
  if (!out || !weights || !weights->gate_up || !weights->down || max_tokens < 1) return GEVVA_MOE_BAD_ARGUMENT;
  if (max_tokens > 131072) return GEVVA_MOE_TOO_LARGE;
  int major = 0, sms = 0;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
    return GEVVA_MOE_CUDA_ERROR;
  if (major != 10) return GEVVA_MOE_NO_DEVICE;
  if (gv::prepare_grouped_gemm() != 0) return GEVVA_MOE_CUDA_ERROR;
  gevva_dense* d = new (std::nothrow) gevva_dense;
  if (!d) return GEVVA_MOE_CUDA_ERROR;
  d->weights = *weights;
  d->max_tokens = max_tokens;
  d->sm_count = sms;
  const size_t t = static_cast<size_t>(max_tokens);
  const size_t tiles = t / gv::kTileM + gv::kExperts + 1;
  const size_t int_count = 2 * (gv::kExperts + 1) + tiles + 2;
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&d->act_fp8), t * gv::kHidden);
  if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&d->act_scales), t * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&d->gate_up_out, t * 2 * kDense * 2);
  if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&d->prod_fp8), t * kDense);
  if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&d->prod_scales), t * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&d->few_products, gv::kDenseFewTokens * kDense * 2);
  if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&d->ones), gv::kExperts * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&d->down_scale), sizeof(float));
  if (e == cudaSuccess)
    e = cudaMemcpy(d->down_scale, &weights->down_scale, sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&d->ints), int_count * sizeof(int));
  if (e == cudaSuccess) e = cudaMemset(d->ints, 0, int_count * sizeof(int));
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&d->fork, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&d->join, cudaEventDisableTiming);
  if (e == cudaSuccess) {
    float host_ones[gv::kExperts];
    for (float& v : host_ones) v = 1.0f;
    e = cudaMemcpy(d->ones, host_ones, sizeof(host_ones), cudaMemcpyHostToDevice);
  }
  if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&d->gelu_table), GV_GELU_FLOATS * sizeof(float));
  if (e == cudaSuccess) {
    float host_table[GV_GELU_FLOATS];
    for (uint32_t i = 0; i < GV_GELU_FLOATS; ++i) host_table[i] = gv_gelu_entry(i);
    e = cudaMemcpy(d->gelu_table, host_table, sizeof(host_table), cudaMemcpyHostToDevice);
  }
  if (e != cudaSuccess) {
    gevva_dense_destroy(d);
    return GEVVA_MOE_CUDA_ERROR;
  }
  int* cursor = d->ints;
  auto carve = [&](size_t n) { int* p = cursor; cursor += n; return p; };
  d->plan.expert_offsets = carve(gv::kExperts + 1);
  d->plan.scale_row_offsets = carve(gv::kExperts + 1);
  d->plan.tile_expert = carve(tiles);
  d->plan.num_m_tiles = carve(1);
  d->plan.status = carve(1);
  bool ok = true;
  ok = ok && gv::make_operand_tensor_map(&d->gate_up.map_a, d->act_fp8, t, gv::kHidden, gv::kTileM);
  ok = ok && gv::make_operand_tensor_map(&d->gate_up.map_a32, d->act_fp8, t, gv::kHidden, 32);
  ok = ok && gv::make_operand_tensor_map(&d->down.map_a32, d->prod_fp8, t, kDense, 32);
  ok = ok && gv::make_operand_tensor_map(&d->gate_up.map_b, weights->gate_up, 2 * kDense, gv::kHidden, gv::kTileM);
  ok = ok && gv::make_operand_tensor_map(&d->down.map_a, d->prod_fp8, t, kDense, gv::kTileM);
  ok = ok && gv::make_operand_tensor_map(&d->down.map_b, weights->down, gv::kHidden, kDense, gv::kTileM);
  ok = ok && gv::make_piece_tensor_map(&d->gate_up.map_down_pieces, weights->gate_up, 2 * kDense, gv::kHidden);
  ok = ok && gv::make_piece_tensor_map(&d->down.map_down_pieces, weights->down, gv::kHidden, kDense);
  ok = ok && gv::make_halves_tensor_map(&d->map_few_gate_up, weights->gate_up, kDense, gv::kHidden, gv::kDenseFewUpRows);
  ok = ok && gv::make_operand_tensor_map(&d->map_few_down, weights->down, gv::kHidden, kDense, gv::kDenseFewDownRows);
  ok = ok && gv::prepare_dense_pairs() == 0 && gv::prepare_dense_few() == 0;
  if (!ok) {
    gevva_dense_destroy(d);
    return GEVVA_MOE_CUDA_ERROR;
  }
  d->gate_up.alpha = d->ones;
  d->gate_up.out = d->gate_up_out;
  d->gate_up.n_out = 2 * kDense;
  d->gate_up.k_in = gv::kHidden;
  d->gate_up.fp8 = true;
  d->down.alpha = d->ones;
  d->down.n_out = gv::kHidden;
  d->down.k_in = kDense;
  d->down.fp8 = true;
  *out = d;
  return GEVVA_MOE_OK;
}

int gevva_dense_launch(gevva_dense* d, const void* in, void* out_unscaled, int tokens,
                       gevva_stream_t stream) {
  if (!d || !in || !out_unscaled || tokens < 1 || tokens > d->max_tokens ||
      ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out_unscaled)) & 15))
    return GEVVA_MOE_BAD_ARGUMENT;  // (rows are read and written 16 bytes at a time at least)
  return gv::dense_launch_on(d, in, out_unscaled, tokens, stream, d->sm_count, d->plan.status);
}

int* gevva_dense_status_word(gevva_dense* d) { return d ? d->plan.status : nullptr; }

int gevva_dense_last_status(gevva_dense* d) {
  if (!d) return GEVVA_MOE_BAD_ARGUMENT;
  int status = 0;
  if (cudaDeviceSynchronize() != cudaSuccess ||
      cudaMemcpy(&status, d->plan.status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess ||
      (status != 0 && cudaMemset(d->plan.status, 0, sizeof(int)) != cudaSuccess))
    return GEVVA_MOE_CUDA_ERROR;
  return -status;
}

const float* gevva_dense_output_scales(const gevva_dense* d) { return d ? d->prod_scales : nullptr; }

const float* gevva_dense_projection_scale(const gevva_dense* d) { return d ? d->down_scale : nullptr; }

int gevva_dense_buffer(const gevva_dense* d, int which, void** ptr, size_t* bytes) {
  if (!d || !ptr || !bytes) return GEVVA_MOE_BAD_ARGUMENT;
  const size_t t = static_cast<size_t>(d->max_tokens);
  switch (which) {
    case 0: *ptr = d->act_fp8; *bytes = t * gv::kHidden; break;
    case 1: *ptr = d->act_scales; *bytes = t * 4; break;
    case 2: *ptr = d->gate_up_out; *bytes = t * 2 * kDense * 2; break;
    case 3: *ptr = d->prod_fp8; *bytes = t * kDense; break;
    case 4: *ptr = d->prod_scales; *bytes = t * 4; break;
    default: return GEVVA_MOE_BAD_ARGUMENT;
  }
  return GEVVA_MOE_OK;
}

int gevva_ff_prepare(const void* input, const void* dense_weight, const void* expert_weight,
                     const void* router_scale, void* dense_out, void* expert_out, void* router_out,
                     int rows, gevva_stream_t stream) {
  if (!input || !dense_weight || !expert_weight || !router_scale || !dense_out || !expert_out ||
      !router_out || rows < 0)
    return GEVVA_MOE_BAD_ARGUMENT;
  if (rows == 0) return GEVVA_MOE_OK;
  gv::launch_ff_prepare(input, dense_weight, expert_weight, router_scale, dense_out, expert_out, router_out,
                        rows, stream);
  return cudaGetLastError() == cudaSuccess ? GEVVA_MOE_OK : GEVVA_MOE_CUDA_ERROR;
}

int gevva_ff_finalize(const void* dense, const void* dense_weight, const void* expert_routes,
                      const float* route_weights, const int* inverse_routes, const void* expert_weight,
                      const void* combined_weight, const void* residual, const void* layer_scalar,
                      void* output, int rows, const float* dense_activation_scales,
                      const float* dense_projection_scale, gevva_stream_t stream) {
  if (!dense || !dense_weight || !expert_routes || !route_weights || !expert_weight || !combined_weight ||
      !residual || !layer_scalar || !output || rows < 0 ||
      (dense_activation_scales != nullptr && dense_projection_scale == nullptr))
    return GEVVA_MOE_BAD_ARGUMENT;
  if (rows == 0) return GEVVA_MOE_OK;
  gv::launch_ff_finalize(dense, dense_weight, expert_routes, route_weights, inverse_routes, expert_weight,
                         combined_weight, residual, layer_scalar, output, rows, dense_activation_scales,
                         dense_projection_scale, stream);
  return cudaGetLastError() == cudaSuccess ? GEVVA_MOE_OK : GEVVA_MOE_CUDA_ERROR;
}

// The intermediates of one layer call, carved from the caller's workspace.
namespace {
struct LayerWorkspace {
  uint8_t* dense_in;
  uint8_t* expert_in;
  uint8_t* router_in;
  uint8_t* dense_out;
  float* route_weights;
  int* ids;
  size_t bytes;
  LayerWorkspace(void* base, int tokens) {
    uint8_t* cursor = static_cast<uint8_t*>(base);
    size_t used = 0;
    auto carve = [&](size_t n) {
      uint8_t* p = cursor ? cursor + used : nullptr;
      used += (n + 255) & ~static_cast<size_t>(255);
      return p;
    };
    const size_t t = static_cast<size_t>(tokens);
    const size_t rows = t * gv::kHidden * 2;
    dense_in = carve(rows);
    expert_in = carve(rows);
    router_in = carve(rows);
    dense_out = carve(rows);
    route_weights = reinterpret_cast<float*>(carve(t * gv::kTopK * sizeof(float)));
    ids = reinterpret_cast<int*>(carve(t * gv::kTopK * sizeof(int)));
    bytes = used;
  }
};
// SMs that the dense MLP of a layer whose experts stream gets beside them.  An expert launch of this size
// holds its SMs from the router to its end, and its time is that of its weights' way through HBM, which 132
// SMs fill as well as 148; the 18 MB of dense weights pass meanwhile.  With a few tokens the experts are
// few and the dense side is the longer chain, so it gets more; 33 SMs hold the first projection's items of 128
// weight rows in one wave, 17 those of 256 (whole layers in a graph, us, at 16 / 17 / 33 / 48 SMs: 1 token 46.4 / 38.9 / 34.4 /
// 32.3, 4 tokens 52.8 / 45.0 / 44.2 / 43.4, 5 tokens 55.5 / 47.7 / 44.9 / 47.2, 8 tokens 60.5 / 52.1 / 54.2 / 57.4, 12 tokens
// 62.7 / 62.3 / 64.2 / 68.1, 40 tokens 93.6 / 94.6 / 99.6 / -, 128 tokens 107.4 / 108.4 / 109.9 / -).
// (With one or two tokens the dense side is dense_few_rows.cu now, 44 CTAs of an SM each: at 48 / 44 / 40 / 32 / 16 SMs 1 token 24.5 / 24.6 / 27.2 / 27.5 / 33.3,
// 2 tokens 27.7 / 27.8 / 29.7 / 30.3 / 35.3.)
// Three layers at 0 (both sides take all SMs) / 20 / 24 / 28 / 33 / 40 / 48: 130 tokens 333 / 284 / 285 / 290 / 289 / 292 / 299,
// 200 tokens 344 / 296 / 297 / 302 / 301 / 305 / 312, 256 tokens - / 306 / 305 / - / - / - / -, 296 tokens 363 / 333 / 325 / 316 / 313 / 317 / 324,
// 400 tokens 355 / 364 / 331 / 335 / 333 / 333 / 338, 512 tokens 368 / - / 348 / - / 350 / 350 / 354, 640 tokens 390 / - / 403 / - / 376 / 379 / 385.
// Where the experts do not stream, above 640 tokens or under an option, sharing gains nothing (700 tokens 425 at 0, 422 at 40, 1024 479 and 488,
// 2048 448 and 469; three layers at 0 and the table's share: runners with GEVVA_MOE_OPTION_W13_PAIRS 130 tokens 317 and 323, 400 345 and 388,
// with GEVVA_MOE_OPTION_PAIRS 484 and 532, 550 and 641, with GEVVA_MOE_DECODE_MERGED=0 319 and 331, 363 and 374).
// Loads other than even ones, three layers in a graph at 0 / 20 / 22 / 24 / 33 SMs: bias of deviation 0.5 on the router logits, 130 tokens 290 / 257 / 258 / 256 / 263,
// 256 tokens 324 / 292 / 293 / 295 / 298; Zipf(1.1), 130 tokens 235 / 215 / 203 / 198 / 192, 256 tokens 279 / 257 / 231 / 233 / 236 (even 340 / 304 / 305 / 306 / 308, 250
// and 253 tokens, on both sides of the last batch whose sort 126 SMs take in, 301 / 304 at 22).  At 0 / 28 / 33 / 40: bias 0.5, 400 tokens 336 / 329 / 330 / 342, 640 tokens
// 405 / 407 / 412 / 430, the one place where sharing gains nothing; Zipf 288 / 280 / 285 / 289 and 379 / 368 / 376 / 386.
// (48, 22 and 16 SMs are the table's, not a matter of waves.)
int dense_sms_beside(int tokens, int sms) {
  const int wanted = tokens <= 4 ? 48 : tokens <= 6 ? 33 : tokens <= 12 ? 17 : tokens <= 128 ? 16 : tokens <= 256 ? 22 : 33;
  return wanted * 2 < sms ? wanted : sms / 2;
}
}  // namespace

size_t gevva_ff_layer_workspace_bytes(int tokens) { return tokens < 1 ? 0 : LayerWorkspace(nullptr, tokens).bytes; }

int gevva_ff_layer_launch(const gevva_ff_layer* layer, const void* hidden, void* out, void* workspace, int tokens,
                          gevva_stream_t stream, gevva_stream_t aux_stream) {
  if (!layer || !layer->dense_pre || !layer->expert_pre || !layer->router_scale || !layer->router_weight ||
      !layer->expert_scale || !layer->dense_post || !layer->expert_post || !layer->combined_post ||
      !layer->layer_scalar || !layer->experts || !layer->dense || !hidden || !out || !workspace ||
      (reinterpret_cast<uintptr_t>(workspace) & 255) || (reinterpret_cast<uintptr_t>(layer->router_weight) & 15) ||
      tokens < 1 || tokens > layer->dense->max_tokens || tokens > gv::moe_max_tokens(layer->experts))
    return GEVVA_MOE_BAD_ARGUMENT;  // (what the parts would refuse, before the first of them is launched)
  const LayerWorkspace w(workspace, tokens);
  gevva_dense* dense = layer->dense;
  const bool beside = aux_stream != stream;
  // The dense MLP starts as soon as its input exists, on SMs that the router leaves idle; beside a
  // decode-sized expert launch on SMs of its own.
  const int sms = gv::moe_sm_count(layer->experts);
  const bool split = beside && sms > 1 && (tokens <= gv::kFusedSortQuantizeMaxTokens || gv::moe_streams(layer->experts, tokens));
  const int dense_sms = split ? dense_sms_beside(tokens, sms) : sms;
  const int expert_sms = split ? sms - dense_sms : sms;
  gv::launch_ff_prepare(hidden, layer->dense_pre, layer->expert_pre, layer->router_scale, w.dense_in, w.expert_in,
                        w.router_in, tokens, stream);
  if (beside) {
    if (cudaEventRecord(dense->fork, stream) != cudaSuccess ||
        cudaStreamWaitEvent(aux_stream, dense->fork, 0) != cudaSuccess)
      return GEVVA_MOE_CUDA_ERROR;
  }
  // One word for the whole layer: what gevva_moe_last_status of its experts reads.
  int* const status_word = gevva_moe_status_word(layer->experts);
  int status = gv::dense_launch_on(dense, w.dense_in, w.dense_out, tokens, beside ? aux_stream : stream, dense_sms, status_word);
  if (beside && cudaEventRecord(dense->join, aux_stream) != cudaSuccess) return GEVVA_MOE_CUDA_ERROR;
  if (status == GEVVA_MOE_OK)
    status = gevva_moe_route_project(w.router_in, layer->router_weight, nullptr, layer->expert_scale, w.route_weights,
                                     w.ids, nullptr, tokens, status_word, stream);
  if (status == GEVVA_MOE_OK)
    status = gv::moe_launch_stages_on(layer->experts, w.expert_in, w.ids, nullptr, nullptr, tokens,
                                      GEVVA_MOE_STAGE_ALL & ~static_cast<unsigned>(GEVVA_MOE_STAGE_REDUCE), stream,
                                      expert_sms);
  // joined in every case: a caller that captures `stream` must get its second stream back
  if (beside && cudaStreamWaitEvent(stream, dense->join, 0) != cudaSuccess) return GEVVA_MOE_CUDA_ERROR;
  if (status != GEVVA_MOE_OK) return status;
  gv::launch_ff_finalize(w.dense_out, layer->dense_post, gevva_moe_routed_output(layer->experts), w.route_weights,
                         gevva_moe_inverse_routes(layer->experts), layer->expert_post, layer->combined_post, hidden,
                         layer->layer_scalar, out, tokens, dense->prod_scales, dense->down_scale, stream);
  return cudaGetLastError() == cudaSuccess ? GEVVA_MOE_OK : GEVVA_MOE_CUDA_ERROR;
}

int gevva_pack_fp8(const float* weights, size_t count, void* out, float* scale, gevva_stream_t stream) {
  if (!weights || !out || !scale || count == 0) return GEVVA_MOE_BAD_ARGUMENT;
  gv::launch_pack_fp8(weights, count, static_cast<uint8_t*>(out), scale, stream);
  return cudaGetLastError() == cudaSuccess ? GEVVA_MOE_OK : GEVVA_MOE_CUDA_ERROR;
}

}  // extern "C"
