// Host side of the C ABI declared in include/gevva_moe.h: owns scratch, builds
// the TMA tensor maps once, and enqueues the stages of one MoE layer in the order
// of the reference's Impl::launch (src/nvfp4_cutlass.cu:1827-1886).  No
// allocation, synchronisation or host-dependent branch on device data happens on
// the launch path, so a launch can be captured into a CUDA graph like the
// reference's (src/cuda/runtime/verifier.cuh:1058-1078).
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>

#include "../../include/gevva_moe.h"
#include <nvtx3/nvToolsExt.h>

#include "gv_common.cuh"
#include "gv_launchers.h"
#include "gv_scratch.h"
#include "gv_stream_schedule.h"

namespace {

using namespace gv;

constexpr int kMaxTokens = 131072;
constexpr int kStreamTokens = 640;  // see moe_streams
// The quantiser of a call that goes on to the experts asks for the first weights of w13, which such batches need (nearly every expert has
// rows, and they are taken in order; where no route goes to those sixteen it costs up to 1.1 us: 400 tokens on the last eight experts 44.5 -> 45.6 a layer, 613 56.8 -> 57.9,
// 300 to 613 on the last sixty-four as before, 82.4 instead of 85.4 and 87.4 instead of 90.9 on all): HBM has little else to do while the sort and the quantiser run.  16 experts are the first
// item of every SM and a little more (8 and 80 MB instead of 36 gain less).  Where the experts stream, us of the listed number of layers without / with: 300 tokens
// 361.8 / 358.9 (four), 400 187.8 / 184.7, 613 191.3 / 189.2, 640 205.1 / 202.3 (two), Zipf(1.1) 500 the same; feed-forward layers of 301 tokens 314.2 / 312.7, 400
// 330.0 / 326.9 (three), 640 248.9 / 248.1 (two).  By pairs: 700 228.9 / 227.0, 1000 244.8 / 241.9, 1400 280.3 / 277.7 (two), 2048 nothing, and feed-forward layers, whose
// dense MLP runs between, lose by it (1000 tokens 311 / 319, 2048 442 / 447), as others' that take their rows unreduced would.
constexpr int kAheadExperts = 16, kAheadTokens = 1536;
// w2 by CTA pairs that share weights between two row tiles of an expert: from 160 rows an expert on average, where most experts
// have two tiles.  One CTA a tile and pairs, us a layer of two in a graph, pauses between (spread 0.3): even loads 2048 tokens 144.8 and 148.0, 2304 158.4 and 156.0,
// 2560 164.2 and 161.3, 3072 176.0 and 172.0, 4096 221.8 and 214.4, 8192 381.6 and 369.6; router bias of deviation 0.5 2048 147.2 and 152.9, 2560 166.7 and 169.3,
// 3072 184.1 and 187.4, 3584 202.4 and 203.3, 4096 221.9 and 221.2, 8192 384.7 and 370.5; Zipf(1.1) 2560 175.3 and 182.1, 3072 196.3 and 198.6, 4096 231.3 and
// 234.3, 5000 270.8 and 269.6, 8192 395.3 and 389.7.  So the sides cross between 2048 and 2304 tokens of even loads and only at some 4000 and 4500 of uneven ones, which lose
// up to 2 and 4 % in between; the host does not know the routes, and the line lies between.
constexpr int kDownPairTokens = 2560;
static_assert(kStreamTokens <= gv::kStreamMaxTokens, "the streaming kernel's chunk list");

// The CUDA face of the allocator that gv_scratch.h takes as a parameter.
struct CudaScratchRuntime {
  static inline cudaError_t last_error = cudaSuccess;
  static bool allocate(void** pointer, size_t bytes) {
    last_error = cudaMalloc(pointer, bytes);
    return last_error == cudaSuccess;
  }
  static bool zero(void* pointer, size_t bytes) {
    last_error = cudaMemset(pointer, 0, bytes);
    return last_error == cudaSuccess;
  }
  static void release(void* pointer) noexcept { cudaFree(pointer); }
};

struct Scratch {
  int references = 1;
  int max_tokens = 0;
  int routes = 0;
  uint8_t* input_codes = nullptr;
  uint8_t* input_sf = nullptr;
  void* w13_out = nullptr;
  uint8_t* inter_codes = nullptr;
  uint8_t* inter_sf = nullptr;
  void* w2_out = nullptr;
  int* ints = nullptr;  // one allocation carved into the RoutePlan arrays
  gv::ScratchMemory<CudaScratchRuntime> memory;
  RoutePlan plan{};
  size_t input_sf_bytes = 0, inter_sf_bytes = 0, tile_capacity = 0;
};

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult result;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &result) !=
            cudaSuccess ||
        result != cudaDriverEntryPointSuccess)
      ptr = nullptr;
    return reinterpret_cast<EncodeTiledFn>(ptr);
  }();
  return fn;
}

// Byte matrix [rows, row_bytes] viewed through a 128-row x 128-byte box with the
// 128-byte swizzle the MMA descriptors expect.  Out-of-range bytes read as zero.
bool make_operand_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes,
                      int box_rows = kTileM) {
  const cuuint64_t dims[2] = {row_bytes, rows};
  const cuuint64_t strides[1] = {row_bytes};
  const cuuint32_t box[2] = {static_cast<cuuint32_t>(kTileKBytes), static_cast<cuuint32_t>(box_rows)};
  const cuuint32_t element_strides[2] = {1, 1};
  EncodeTiledFn fn = encode_tiled();
  if (!fn) return false;
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box,
            element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool make_scale_map(CUtensorMap* map, const void* base, uint64_t bytes, int box_atoms) {
  const cuuint64_t dims[2] = {128, bytes / 512};
  const cuuint64_t strides[1] = {512};
  const cuuint32_t box[2] = {128, static_cast<cuuint32_t>(box_atoms)};
  const cuuint32_t element_strides[2] = {1, 1};
  EncodeTiledFn fn = encode_tiled();
  if (!fn || dims[1] == 0) return false;
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(base), dims, strides, box,
            element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Bytes [halves, rows, row_bytes] through a box of two halves x box_rows rows x 128 bytes (128-byte swizzle).
bool make_halves_map(CUtensorMap* map, const void* base, uint64_t halves, uint64_t rows, uint64_t row_bytes, int box_rows) {
  const cuuint64_t dims[3] = {row_bytes, rows, halves};
  const cuuint64_t strides[2] = {row_bytes, rows * row_bytes};
  const cuuint32_t box[3] = {static_cast<cuuint32_t>(kTileKBytes), static_cast<cuuint32_t>(box_rows), 2};
  const cuuint32_t element_strides[3] = {1, 1, 1};
  EncodeTiledFn fn = encode_tiled();
  if (!fn) return false;
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box,
            element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// w13 codes [experts, 2 halves (up, gate), 704 rows, 1408 bytes] through a box of both halves x
// 64 rows: one copy brings a unit's up rows and gate rows.
bool make_w13_unit_map(CUtensorMap* map, const void* base, uint64_t experts) {
  return make_halves_map(map, base, experts * 2, kInter, kHidden / 2, 64);
}

// w13 codes [experts, up and gate halves of 704 rows, 1408 bytes] in the row order of grouped_gemm_w13_pair.cu:
// row 32b + 16o + 8h + i of a 128-row box is row 16b + 2i + o of half h, b counting blocks of 16 rows.
bool make_w13_fragment_map(CUtensorMap* map, const void* base, uint64_t experts) {
  constexpr cuuint64_t row = kHidden / 2;
  // the last dimension starts in an up half; its extent keeps the gate half, 704 rows on, inside the matrix
  const cuuint64_t dims[5] = {row, 8, 2, 2, (experts * kW13Out - kInter) / 16};
  const cuuint64_t strides[4] = {2 * row, kInter * row, row, 16 * row};
  const cuuint32_t box[5] = {static_cast<cuuint32_t>(kTileKBytes), 8, 2, 2, 4};
  const cuuint32_t element_strides[5] = {1, 1, 1, 1, 1};
  EncodeTiledFn fn = encode_tiled();
  if (!fn) return false;
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, const_cast<void*>(base), dims, strides, box, element_strides,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Weight rows in the order of grouped_gemm_down.cu, row 8g + 2t + i of a 64-row group being row 16t + 2g + i: a box of `groups` groups,
// or of half a one (0).
bool make_column_order_map(CUtensorMap* map, const void* base, uint64_t rows, cuuint64_t row, int groups) {
  const cuuint64_t dims[5] = {row, 2, 4, 8, rows / 64};
  const cuuint64_t strides[4] = {row, 16 * row, 2 * row, 64 * row};
  const cuuint32_t box[5] = {static_cast<cuuint32_t>(kTileKBytes), 2, 4, groups ? 8u : 4u, groups ? static_cast<cuuint32_t>(groups) : 1u};
  const cuuint32_t element_strides[5] = {1, 1, 1, 1, 1};
  EncodeTiledFn fn = encode_tiled();
  if (!fn) return false;
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, const_cast<void*>(base), dims, strides, box, element_strides,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool make_w2_down_map(CUtensorMap* map, const void* base, uint64_t experts) {
  return make_column_order_map(map, base, experts * kHidden, kInter / 2, 3);
}

// Scale bytes of an activation operand as [128-row blocks, atoms per block, 128 x u32] through a
// box of one block x four atoms: the scales of one K block of up to 128 rows.
bool make_block_scale_map(CUtensorMap* map, const void* base, uint64_t bytes, int atoms_per_block) {
  const uint64_t block_bytes = static_cast<uint64_t>(atoms_per_block) * 512;
  const cuuint64_t dims[3] = {128, static_cast<cuuint64_t>(atoms_per_block), bytes / block_bytes};
  const cuuint64_t strides[2] = {512, block_bytes};
  const cuuint32_t box[3] = {128, 4, 1};
  const cuuint32_t element_strides[3] = {1, 1, 1};
  EncodeTiledFn fn = encode_tiled();
  if (!fn || dims[2] == 0) return false;
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<void*>(base), dims, strides, box,
            element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

thread_local char g_error_text[256] = "";

int cuda_failure(cudaError_t error, const char* what) {
  std::snprintf(g_error_text, sizeof(g_error_text), "%s: %s", what, cudaGetErrorString(error));
  return GEVVA_MOE_CUDA_ERROR;
}

#define GV_CUDA(call, what)                                  \
  do {                                                       \
    const cudaError_t gv_error_ = (call);                    \
    if (gv_error_ != cudaSuccess) return cuda_failure(gv_error_, what); \
  } while (0)

void free_scratch(Scratch* s) {
  if (!s) return;
  s->memory.release();
  delete s;
}

int make_scratch(int tokens, Scratch** out) {
  Scratch* s = new (std::nothrow) Scratch;
  if (!s) return GEVVA_MOE_CUDA_ERROR;
  const gv::ScratchSizes sizes = gv::scratch_sizes(tokens);
  s->max_tokens = tokens;
  s->routes = static_cast<int>(sizes.routes);
  s->input_sf_bytes = sizes.bytes[1];
  s->inter_sf_bytes = sizes.bytes[4];
  s->tile_capacity = sizes.tile_capacity;
  const size_t routes = sizes.routes;
  const size_t chunks = sizes.chunks;
  if (!s->memory.acquire(sizes)) {
    delete s;
    return cuda_failure(CudaScratchRuntime::last_error, "scratch allocation");
  }
  s->input_codes = static_cast<uint8_t*>(s->memory.buffers[0]);
  s->input_sf = static_cast<uint8_t*>(s->memory.buffers[1]);
  s->w13_out = s->memory.buffers[2];
  s->inter_codes = static_cast<uint8_t*>(s->memory.buffers[3]);
  s->inter_sf = static_cast<uint8_t*>(s->memory.buffers[4]);
  s->w2_out = s->memory.buffers[5];
  s->ints = static_cast<int*>(s->memory.buffers[6]);
  int* cursor = s->ints;
  auto carve = [&](size_t count) {
    int* p = cursor;
    cursor += count;
    return p;
  };
  s->plan.sorted_experts = carve(routes);
  s->plan.sorted_routes = carve(routes);
  s->plan.inverse_routes = carve(routes);
  s->plan.expert_offsets = carve(kExperts + 1);
  s->plan.scale_row_offsets = carve(kExperts + 1);
  s->plan.tile_expert = carve(s->tile_capacity);
  s->plan.num_m_tiles = carve(1);
  s->plan.pair_tile = carve(s->tile_capacity);
  s->plan.num_pairs = carve(1);
  s->plan.tile_ready = carve(s->tile_capacity + 1);
  s->plan.chunk_hist = carve(chunks * kExperts);
  s->plan.status = carve(1);
  s->plan.sync = carve(2);  // taken from the 64 spare ints; zero like everything else here
  s->plan.stream_sync = carve(gv::kStreamSyncInts);
  *out = s;
  return GEVVA_MOE_OK;
}

}  // namespace

namespace gv {
bool make_w13_unit_tensor_map(CUtensorMap* map, const void* base, uint64_t experts) {
  return make_w13_unit_map(map, base, experts);
}
bool make_halves_tensor_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes, int box_rows) {
  return make_halves_map(map, base, 2, rows, row_bytes, box_rows);
}
bool make_w2_down_tensor_map(CUtensorMap* map, const void* base, uint64_t experts) {
  return make_w2_down_map(map, base, experts);
}
bool make_piece_tensor_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes) {
  return make_column_order_map(map, base, rows, row_bytes, 0);
}
bool make_operand_tensor_map(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes,
                             int box_rows) {
  return make_operand_map(map, base, rows, row_bytes, box_rows);
}
bool make_scale_tensor_map(CUtensorMap* map, const void* base, uint64_t bytes, int box_atoms) {
  return make_scale_map(map, base, bytes, box_atoms);
}
}  // namespace gv

namespace {
// The bounded-wait primitive of the GEMM kernels, exercised on its own: one thread waits on
// a local mbarrier that nothing will ever complete, gives up after `limit_cycles`, records
// kWaitTimeout in the status word and returns normally.
__global__ void bounded_wait_probe_kernel(int* status, long long limit_cycles) {
  __shared__ uint64_t barrier;
  if (threadIdx.x == 0) {
    gv::mbar_init(&barrier, 1);
    gv::fence_barrier_init();
    if (!gv::mbar_wait_bounded(&barrier, 0, limit_cycles))
      atomicExch(status, static_cast<int>(gv::kWaitTimeout));
  }
}
}  // namespace

struct gevva_moe {
  Scratch* scratch = nullptr;
  gevva_moe_weights weights{};
  gv::GemmOperands w13{};        // bf16 output (stage access, debugging)
  gv::GemmOperands w13_fused{};  // GeGLU + requantise in the epilogue (the production path)
  gv::GemmOperands w2{};
  uint8_t* w13_sf_tiled = nullptr;  // runner-owned re-tiling of weights.w13_sf for the CTA-pair tile kernels
  gv::W13PairOperands w13_pairs{};  // the CTA-pair form of the fused w13 stage
  uint8_t* w13_sf_units = nullptr;  // runner-owned re-tiling of weights.w13_sf by unit of 64 columns (and its allocation,
                                    // which the next two share)
  uint8_t* w13_sf_fragments = nullptr;  // the same in the row order of grouped_gemm_w13_pair.cu
  uint8_t* w2_sf_down = nullptr;    // re-tiling of weights.w2_sf in the column order of grouped_gemm_down.cu
  gv::StreamOperands stream_experts{};  // few rows an expert: both GEMMs in one launch, weights on the MMA's M side
  bool w13_pair_form = false;       // GEVVA_MOE_OPTION_W13_PAIRS, or GEVVA_MOE_W13_PAIRS=1 for a whole process
  bool w13_single = false;          // GEVVA_MOE_W13_PAIRS=0: the fused w13 of large batches by the one-CTA kernel, which
                                    // expert-parallel ranks use (to compare the two)
  int sm_count = 0;
  bool pairs = false;               // GEVVA_MOE_OPTION_PAIRS: prefill-sized launches run the expert GEMMs as CTA pairs
  bool decode_front = true;         // ... and the route sort and the input quantiser in the same launch (GEVVA_MOE_DECODE_FRONT=0: a launch of their own)
  bool merged_decode = true;        // batches of at most kStreamTokens: w13 and w2 in one launch (GEVVA_MOE_DECODE_MERGED=0: two)
  bool nvtx = false;                // GEVVA_MOE_OPTION_NVTX: one range per stage around its launches
};

namespace {
// A named NVTX range around the launches of one stage, when the runner was created with the
// option (the ranges cost nothing unless a tool is attached, but are off by default).
struct StageRange {
  bool on;
  StageRange(bool enabled, const char* name) : on(enabled) {
    if (on) nvtxRangePushA(name);
  }
  ~StageRange() {
    if (on) nvtxRangePop();
  }
};
}  // namespace

int gv::moe_sm_count(const gevva_moe* runner) { return runner->sm_count; }
int gv::moe_max_tokens(const gevva_moe* runner) { return runner->scratch->max_tokens; }

// Few rows an expert: the layer streams weights, and one launch with the weights on the MMA's M side does both GEMMs.
// Against the launches of larger batches (w13 by CTA pairs, then w2), us a layer of four distinct ones in a graph, pauses between, one B200 (spread 0.2):
// router logits without bias, 300 tokens 86.1 against 94.1, 400 87.3 / 96.3, 500 90.1 / 99.5, 640 95.4 / 104.6 (up to 296
// tokens it also takes in the sort and the quantiser); with a bias of deviation 0.5 85.4 / 93.9, 88.0 / 96.4, 91.7 / 100.1,
// 98.4 / 105.5; with a Zipf(1.1) bias 72.9 / 79.5, 78.0 / 84.0, 84.8 / 88.9, 95.7 / 99.6: a heavy expert has many 64-row
// chunks, each with the whole of its weights.  The launch pays all the way to the line, least for the heaviest experts.
// (The pair options leave batches of at most 128 tokens alone.)
bool gv::moe_streams(const gevva_moe* runner, int tokens) {
  const bool pair_options = (runner->pairs || runner->w13_pair_form) && tokens > gv::kFusedSortQuantizeMaxTokens;
  return runner->merged_decode && !pair_options && tokens <= kStreamTokens;
}

int gv::moe_launch_stages_on(gevva_moe* runner, const void* in, const int* ids, const float* route_weights, void* out,
                             int tokens, unsigned stages, cudaStream_t stream, int sm_count) {
  Scratch* s = runner->scratch;
  // "expert runner token count exceeds its plan", src/nvfp4_cutlass.cu:1830-1832
  if (tokens < 1 || tokens > s->max_tokens) return GEVVA_MOE_BAD_ARGUMENT;
  if ((stages & (GEVVA_MOE_STAGE_SORT | GEVVA_MOE_STAGE_QUANTIZE)) && !ids) return GEVVA_MOE_BAD_ARGUMENT;
  if ((stages & GEVVA_MOE_STAGE_QUANTIZE) && !in) return GEVVA_MOE_BAD_ARGUMENT;
  if ((stages & GEVVA_MOE_STAGE_REDUCE) && (!out || !route_weights)) return GEVVA_MOE_BAD_ARGUMENT;
  const int routes = tokens * kTopK;
  // Decode-sized batches (at most a few rows per expert) stream weights and gain nothing from
  // pairing two row tiles of an expert; they keep the one-CTA-per-tile kernel.
  const bool use_pairs = runner->pairs && tokens > gv::kFusedSortQuantizeMaxTokens;
  const unsigned front = GEVVA_MOE_STAGE_SORT | GEVVA_MOE_STAGE_QUANTIZE;
  const unsigned both = GEVVA_MOE_STAGE_W13 | GEVVA_MOE_STAGE_GEGLU;
  const unsigned gemms = both | GEVVA_MOE_STAGE_W2;
  // Weights on the MMA's M side, by CTA pairs: faster than (2048 tokens on) or as fast as the one-CTA tile kernel
  // wherever a batch does not stream (figures in grouped_gemm_w13_pair.cu).
  const bool w13_by_pairs = !use_pairs && sm_count >= 2 && !runner->w13_single &&
                            (tokens > kStreamTokens || (runner->w13_pair_form && tokens > gv::kFusedSortQuantizeMaxTokens));
  const unsigned layer_body = front | GEVVA_MOE_STAGE_W13 | GEVVA_MOE_STAGE_GEGLU | GEVVA_MOE_STAGE_W2;
  const bool streams = !(stages & GEVVA_MOE_STAGE_UNFUSED) && gv::moe_streams(runner, tokens);
  if ((stages & layer_body) == layer_body && streams && runner->decode_front && gv::stream_layer_fits(tokens, sm_count)) {
    // ... and the route sort and the quantiser; the weights stream while the input is being quantised
    StageRange range(runner->nvtx, "gevva_moe.sort+quantize+w13+geglu+w2");
    gv::launch_stream_layer(runner->stream_experts, s->plan, in, ids, runner->weights.in_scale_q1, s->input_codes,
                            s->input_sf, tokens, sm_count, stream);
    stages &= ~layer_body;
  }
  if ((stages & front) == front && tokens <= gv::kFusedSortQuantizeMaxTokens) {
    // decode-sized batch: one launch does both
    StageRange range(runner->nvtx, "gevva_moe.sort+quantize");
    gv::launch_route_sort_quantize_small(in, ids, runner->weights.in_scale_q1, s->plan, tokens, s->input_codes,
                                         s->input_sf, stream);
  } else {
    if (stages & GEVVA_MOE_STAGE_SORT) {
      StageRange range(runner->nvtx, "gevva_moe.sort");
      gv::launch_route_sort(ids, routes, s->plan, stream);
    }
    StageRange range(runner->nvtx && (stages & GEVVA_MOE_STAGE_QUANTIZE), "gevva_moe.quantize");
    if (stages & GEVVA_MOE_STAGE_QUANTIZE) {
      gv::WeightsAhead ahead{};
      if ((stages & gemms) == gemms && (streams || (w13_by_pairs && tokens <= kAheadTokens && (stages & GEVVA_MOE_STAGE_REDUCE)))) {
        ahead.base[0] = static_cast<const uint8_t*>(runner->weights.w13);
        ahead.bytes[0] = kAheadExperts * gv::kW13Out * (gv::kHidden / 2);
        ahead.base[1] = streams ? runner->w13_sf_units : runner->w13_sf_fragments;
        ahead.bytes[1] = static_cast<uint32_t>(gv::w13_unit_scale_bytes(kAheadExperts));
      }
      gv::launch_quantize_input(in, ids, runner->weights.in_scale_q1, s->plan, tokens, s->input_codes,
                                s->input_sf, (stages & GEVVA_MOE_STAGE_SORT) != 0, ahead, stream);
    }
  }
  if ((stages & gemms) == gemms && streams) {
    StageRange range(runner->nvtx, "gevva_moe.w13+geglu+w2");
    gv::launch_stream_experts(runner->stream_experts, s->plan, sm_count, stream);
    stages &= ~gemms;
  }
  if ((stages & both) == both && !(stages & GEVVA_MOE_STAGE_UNFUSED)) {
    // production path: GeGLU + requantise inside the w13 epilogue, no bf16 w13 output
    StageRange range(runner->nvtx, "gevva_moe.w13+geglu");
    if (w13_by_pairs) {
      gv::W13PairOperands w13 = runner->w13_pairs;
      w13.early_weights = (stages & front) == front;
      gv::launch_w13_pairs(w13, s->plan, sm_count, stream);
    } else {
      gv::GemmOperands w13 = runner->w13_fused;
      w13.use_pairs = use_pairs;
      w13.early_weights = (stages & front) == front && tokens > gv::kFusedSortQuantizeMaxTokens;
      gv::launch_grouped_gemm(w13, s->plan, sm_count, stream);
    }
  } else {
    if (stages & GEVVA_MOE_STAGE_W13)
      gv::launch_grouped_gemm(runner->w13, s->plan, sm_count, stream);
    if (stages & GEVVA_MOE_STAGE_GEGLU)
      gv::launch_geglu_quantize(s->w13_out, runner->weights.in_scale_q2, s->plan, routes,
                                s->inter_codes, s->inter_sf, stream);
  }
  // the fused w13 launch of this call is w2's predecessor, and w2 the reduce's
  const bool behind_w13 = (stages & both) == both && !(stages & GEVVA_MOE_STAGE_UNFUSED) && !use_pairs;
  const bool behind_w2 = (stages & GEVVA_MOE_STAGE_W2) && !use_pairs && behind_w13;
  if (stages & GEVVA_MOE_STAGE_W2) {
    StageRange range(runner->nvtx, "gevva_moe.w2");
    gv::GemmOperands w2 = runner->w2;
    w2.use_pairs = use_pairs;
    w2.early_weights = behind_w13;
    if (!use_pairs && sm_count >= 2 && tokens >= kDownPairTokens) gv::launch_grouped_down_pairs(w2, s->plan, sm_count, stream);
    else gv::launch_grouped_gemm(w2, s->plan, sm_count, stream);
  }
  StageRange reduce_range(runner->nvtx && (stages & GEVVA_MOE_STAGE_REDUCE), "gevva_moe.reduce");
  if (stages & GEVVA_MOE_STAGE_REDUCE)
    gv::launch_reduce_routes(s->w2_out, route_weights, s->plan.inverse_routes, tokens, out, behind_w2, stream);
  GV_CUDA(cudaGetLastError(), "moe launch");
  return GEVVA_MOE_OK;
}

extern "C" {

const char* gevva_moe_strerror(int status) {
  switch (status) {
    case GEVVA_MOE_OK: return "ok";
    case GEVVA_MOE_BAD_EXPERT_ID: return "expert id outside [0,128)";
    case GEVVA_MOE_WAIT_TIMEOUT: return "bounded device wait expired";
    case GEVVA_MOE_BAD_ARGUMENT: return "bad argument";
    case GEVVA_MOE_CUDA_ERROR: return g_error_text[0] ? g_error_text : "CUDA error";
    case GEVVA_MOE_NO_DEVICE: return "no sm_100 device or driver entry point";
    case GEVVA_MOE_TOO_LARGE: return "size beyond the supported maximum";
    default: return "unknown status";
  }
}

int gevva_moe_create(gevva_moe** out, const gevva_moe_weights* weights, int max_tokens,
                     gevva_moe* share_scratch_with, const gevva_moe_options* options) {
  if (options && (options->flags & ~static_cast<uint32_t>(GEVVA_MOE_OPTION_NVTX | GEVVA_MOE_OPTION_PAIRS | GEVVA_MOE_OPTION_W13_PAIRS)))
    return GEVVA_MOE_BAD_ARGUMENT;
  if (!out || !weights || !weights->w13 || !weights->w13_sf || !weights->w2 || !weights->w2_sf ||
      !weights->alpha1 || !weights->alpha2 || !weights->in_scale_q1 || !weights->in_scale_q2)
    return GEVVA_MOE_BAD_ARGUMENT;
  if (max_tokens < 1) return GEVVA_MOE_BAD_ARGUMENT;
  if (max_tokens > kMaxTokens) return GEVVA_MOE_TOO_LARGE;
  if (share_scratch_with && share_scratch_with->scratch->max_tokens != max_tokens)
    return GEVVA_MOE_BAD_ARGUMENT;  // "shared expert capacity mismatch", src/nvfp4_cutlass.cu:1788
  int device = 0;
  GV_CUDA(cudaGetDevice(&device), "cudaGetDevice");
  int major = 0, sms = 0;  // (all properties of a device take 3 ms to ask for)
  GV_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device), "cudaDeviceGetAttribute");
  GV_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device), "cudaDeviceGetAttribute");
  if (major != 10 || !encode_tiled()) return GEVVA_MOE_NO_DEVICE;
  GV_CUDA(static_cast<cudaError_t>(gv::prepare_grouped_gemm()), "cudaFuncSetAttribute");

  gevva_moe* m = new (std::nothrow) gevva_moe;
  if (!m) return GEVVA_MOE_CUDA_ERROR;
  m->weights = *weights;
  m->nvtx = options && (options->flags & GEVVA_MOE_OPTION_NVTX);
  // The CTA-pair form (tcgen05 cta_group::2) is bit-identical but measured slower than one CTA per
  // tile on this part (175 against 102 us for w13 at 4096 tokens), so it is opt-in: by option, or
  // for a whole process by GEVVA_MOE_PAIRS=1.
  const char* merged_env = std::getenv("GEVVA_MOE_DECODE_MERGED");
  m->merged_decode = !(merged_env && merged_env[0] == '0');
  const char* front_env = getenv("GEVVA_MOE_DECODE_FRONT");
  m->decode_front = !(front_env && front_env[0] == '0');
  const char* pairs_env = std::getenv("GEVVA_MOE_PAIRS");
  m->pairs = (options && (options->flags & GEVVA_MOE_OPTION_PAIRS)) || (pairs_env && pairs_env[0] == '1');
  m->sm_count = sms;
  if (share_scratch_with) {
    m->scratch = share_scratch_with->scratch;
    ++m->scratch->references;
  } else {
    const int status = make_scratch(max_tokens, &m->scratch);
    if (status != GEVVA_MOE_OK) {
      delete m;
      return status;
    }
  }
  Scratch* s = m->scratch;
  const uint64_t rows = static_cast<uint64_t>(s->routes);
  bool ok = true;
  ok = ok && make_operand_map(&m->w13.map_a, s->input_codes, rows, kHidden / 2);
  ok = ok && make_operand_map(&m->w13.map_a32, s->input_codes, rows, kHidden / 2, 32);
  ok = ok && make_operand_map(&m->w2.map_a32, s->inter_codes, rows, kInter / 2, 32);
  ok = ok && make_operand_map(&m->w13.map_b, weights->w13, static_cast<uint64_t>(kExperts) * kW13Out,
                              kHidden / 2);
  ok = ok && make_operand_map(&m->w2.map_a, s->inter_codes, rows, kInter / 2);
  ok = ok && make_operand_map(&m->w2.map_b, weights->w2, static_cast<uint64_t>(kExperts) * kHidden,
                              kInter / 2);
  if (!ok) {
    gevva_moe_destroy(m);
    std::snprintf(g_error_text, sizeof(g_error_text), "cuTensorMapEncodeTiled failed");
    return GEVVA_MOE_CUDA_ERROR;
  }
  // The fused w13 epilogues pair up rows with gate rows inside one MMA tile; their weight scales are a
  // one-off re-tiling of the caller's tensor (the caller's memory is not touched).
  {
    // one allocation for the three: of a runner's creation most goes into allocations
    const size_t unit_bytes = gv::w13_unit_scale_bytes(kExperts);  // a multiple of 2 KiB
    cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&m->w13_sf_units), 2 * unit_bytes + gv::retiled_w2_scale_bytes(kExperts));
    if (e == cudaSuccess) {
      m->w13_sf_fragments = m->w13_sf_units + unit_bytes;
      m->w2_sf_down = m->w13_sf_fragments + unit_bytes;
      gv::launch_retile_w13_unit_scales(static_cast<const uint8_t*>(weights->w13_sf), m->w13_sf_units, kExperts, false, nullptr);
      gv::launch_retile_w13_unit_scales(static_cast<const uint8_t*>(weights->w13_sf), m->w13_sf_fragments, kExperts, true, nullptr);
      gv::launch_retile_w2_scales(static_cast<const uint8_t*>(weights->w2_sf), m->w2_sf_down, kExperts, nullptr);
      e = cudaGetLastError();
    }
    if (e == cudaSuccess && m->pairs) {
      // the opt-in CTA-pair form of the tile kernels has a tiling of its own
      e = cudaMalloc(reinterpret_cast<void**>(&m->w13_sf_tiled), gv::retiled_w13_scale_bytes(kExperts));
      if (e == cudaSuccess) {
        gv::launch_retile_w13_scales(static_cast<const uint8_t*>(weights->w13_sf), m->w13_sf_tiled, kExperts, nullptr);
        e = cudaGetLastError();
      }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
    if (e != cudaSuccess) {
      gevva_moe_destroy(m);
      return cuda_failure(e, "weight scale re-tiling");
    }
    if (m->pairs) {
      ok = make_scale_map(&m->w13.map_a_sf, s->input_sf, s->input_sf_bytes, 4) &&
           make_scale_map(&m->w13.map_b_sf, m->w13_sf_tiled, gv::retiled_w13_scale_bytes(kExperts), 8) &&
           make_scale_map(&m->w2.map_a_sf, s->inter_sf, s->inter_sf_bytes, 4) &&
           make_scale_map(&m->w2.map_b_sf, weights->w2_sf, static_cast<uint64_t>(kExperts) * kHidden * (kInter / 16), 4) &&
           make_operand_map(&m->w13.map_b64, weights->w13, static_cast<uint64_t>(kExperts) * kW13Out, kHidden / 2, 64);
      if (!ok) {
        gevva_moe_destroy(m);
        std::snprintf(g_error_text, sizeof(g_error_text), "cuTensorMapEncodeTiled failed (pair maps)");
        return GEVVA_MOE_CUDA_ERROR;
      }
    }
    gv::StreamOperands& st = m->stream_experts;
    ok = make_w13_unit_map(&st.map_w13, weights->w13, kExperts) &&
         make_w2_down_map(&m->w2.map_b_down, weights->w2, kExperts) && gv::make_piece_tensor_map(&m->w2.map_down_pieces, weights->w2, static_cast<uint64_t>(kExperts) * kHidden, kInter / 2) &&
         make_scale_map(&m->w2.map_down_a_sf, s->inter_sf, s->inter_sf_bytes, 4) &&
         make_scale_map(&m->w2.map_down_b_sf, m->w2_sf_down, gv::retiled_w2_scale_bytes(kExperts), 8);
    for (int i = 0; i < gv::kStreamBoxes; ++i)
      ok = ok && make_operand_map(&st.map_up[i], s->input_codes, rows, kHidden / 2, 8 * (i + 1)) &&
           make_operand_map(&st.map_down[i], s->inter_codes, rows, kInter / 2, 8 * (i + 1));
    if (!ok) {
      gevva_moe_destroy(m);
      std::snprintf(g_error_text, sizeof(g_error_text), "cuTensorMapEncodeTiled failed (streaming form)");
      return GEVVA_MOE_CUDA_ERROR;
    }
    st.map_w2 = m->w2.map_b;
    st.w13_scales = m->w13_sf_units;
    st.w2_scales = static_cast<const uint8_t*>(weights->w2_sf);
    st.input_scales = s->input_sf;
    st.inter_codes = s->inter_codes;
    st.inter_scales = s->inter_sf;
    st.routed = s->w2_out;
    st.alpha1 = weights->alpha1;
    st.alpha2 = weights->alpha2;
    st.in_scale_q2 = weights->in_scale_q2;
  }
  const char* w13_pairs_env = std::getenv("GEVVA_MOE_W13_PAIRS");
  m->w13_pair_form = (options && (options->flags & GEVVA_MOE_OPTION_W13_PAIRS)) || (w13_pairs_env && w13_pairs_env[0] == '1');
  m->w13_single = !m->w13_pair_form && w13_pairs_env && w13_pairs_env[0] == '0';
  {
    cudaError_t e = static_cast<cudaError_t>(gv::prepare_w13_pairs());
    if (e == cudaSuccess) e = static_cast<cudaError_t>(gv::prepare_grouped_down_pairs());
    if (e != cudaSuccess) {
      gevva_moe_destroy(m);
      return cuda_failure(e, "CTA-pair forms");
    }
    gv::W13PairOperands& wp = m->w13_pairs;
    ok = true;
    for (int i = 0; i < gv::kW13PairBoxes; ++i)
      ok = ok && make_operand_map(&wp.map_x[i], s->input_codes, rows, kHidden / 2, 8 * (i + 1));
    ok = ok && make_w13_fragment_map(&wp.map_w, weights->w13, kExperts) &&
         make_block_scale_map(&wp.map_x_sf, s->input_sf, s->input_sf_bytes, kHidden / 64) &&
         make_scale_map(&wp.map_w_sf, m->w13_sf_fragments, gv::w13_unit_scale_bytes(kExperts), 4);
    if (!ok) {
      gevva_moe_destroy(m);
      std::snprintf(g_error_text, sizeof(g_error_text), "cuTensorMapEncodeTiled failed (w13 pair maps)");
      return GEVVA_MOE_CUDA_ERROR;
    }
    wp.alpha = weights->alpha1;
    wp.next_codes = s->inter_codes;
    wp.next_scales = s->inter_sf;
    wp.next_scale_q = weights->in_scale_q2;
    wp.serial_launch = false;
  }
  m->w13.a_scales = s->input_sf;
  m->w13.b_scales = static_cast<const uint8_t*>(weights->w13_sf);
  m->w13.alpha = weights->alpha1;
  m->w13.out = s->w13_out;
  m->w13.n_out = kW13Out;
  m->w13.k_in = kHidden;
  m->w13_fused = m->w13;
  m->w13_fused.b_scales = m->w13_sf_tiled;  // pairs only
  m->w13_fused.map_b_units = m->stream_experts.map_w13;
  m->w13_fused.unit_scales = m->w13_sf_units;
  m->w13_fused.out = nullptr;
  m->w13_fused.fused_geglu = true;
  m->w13_fused.next_codes = s->inter_codes;
  m->w13_fused.next_scales = s->inter_sf;
  m->w13_fused.next_scale_q = weights->in_scale_q2;
  m->w2.a_scales = s->inter_sf;
  m->w2.b_scales = static_cast<const uint8_t*>(weights->w2_sf);
  m->w2.alpha = weights->alpha2;
  m->w2.out = s->w2_out;
  m->w2.down_scales = m->w2_sf_down;
  m->w2.n_out = kHidden;
  m->w2.k_in = kInter;
  *out = m;
  return GEVVA_MOE_OK;
}

void gevva_moe_destroy(gevva_moe* runner) {
  if (!runner) return;
  if (runner->scratch && --runner->scratch->references == 0) free_scratch(runner->scratch);
  cudaFree(runner->w13_sf_tiled);
  cudaFree(runner->w13_sf_units);
  delete runner;
}

int gevva_moe_route(const void* logits_bf16, int ld, const void* expert_scale_bf16, float* weights,
                    int* ids, int tokens, const float* act_scales, const float* w_scale,
                    gevva_stream_t stream) {
  if (!logits_bf16 || !expert_scale_bf16 || !weights || !ids || ld < kExperts || tokens < 0 ||
      (act_scales != nullptr) != (w_scale != nullptr))
    return GEVVA_MOE_BAD_ARGUMENT;
  if (tokens == 0) return GEVVA_MOE_OK;
  gv::launch_route(logits_bf16, ld, expert_scale_bf16, weights, ids, tokens, act_scales, w_scale,
                   stream);
  GV_CUDA(cudaGetLastError(), "route_128_top8");
  return GEVVA_MOE_OK;
}

int gevva_moe_route_project(const void* router_input_bf16, const void* router_weight_bf16, const float* bias,
                            const void* expert_scale_bf16, float* weights, int* ids, void* logits_out,
                            int tokens, int* device_status, gevva_stream_t stream) {
  if (!router_input_bf16 || !router_weight_bf16 || !expert_scale_bf16 || !weights || !ids || tokens < 0 ||
      (reinterpret_cast<uintptr_t>(router_input_bf16) & 15) || (reinterpret_cast<uintptr_t>(router_weight_bf16) & 15) ||
      (reinterpret_cast<uintptr_t>(bias) & 15))
    return GEVVA_MOE_BAD_ARGUMENT;
  if (tokens == 0) return GEVVA_MOE_OK;
  if (!encode_tiled()) return GEVVA_MOE_NO_DEVICE;
  GV_CUDA(static_cast<cudaError_t>(gv::launch_route_project(router_input_bf16, router_weight_bf16, false, bias,
                                                            expert_scale_bf16, weights, ids, logits_out, nullptr,
                                                            nullptr, tokens, device_status, stream)),
          "route_project");
  return GEVVA_MOE_OK;
}

int gevva_moe_route_project_fp8(const void* router_input_e4m3, const float* activation_scales,
                                const void* router_weight_e4m3, const float* weight_scale,
                                const void* expert_scale_bf16, float* weights, int* ids, void* logits_out,
                                int tokens, int* device_status, gevva_stream_t stream) {
  if (!router_input_e4m3 || !activation_scales || !router_weight_e4m3 || !weight_scale || !expert_scale_bf16 ||
      !weights || !ids || tokens < 0 || (reinterpret_cast<uintptr_t>(router_input_e4m3) & 15) ||
      (reinterpret_cast<uintptr_t>(router_weight_e4m3) & 15))
    return GEVVA_MOE_BAD_ARGUMENT;
  if (tokens == 0) return GEVVA_MOE_OK;
  if (!encode_tiled()) return GEVVA_MOE_NO_DEVICE;
  GV_CUDA(static_cast<cudaError_t>(gv::launch_route_project(router_input_e4m3, router_weight_e4m3, true, nullptr,
                                                            expert_scale_bf16, weights, ids, logits_out,
                                                            activation_scales, weight_scale, tokens, device_status,
                                                            stream)),
          "route_project_fp8");
  return GEVVA_MOE_OK;
}

int* gevva_moe_status_word(gevva_moe* runner) { return runner ? runner->scratch->plan.status : nullptr; }

int gevva_moe_launch_stages(gevva_moe* runner, const void* in, const int* ids,
                            const float* route_weights, void* out, int tokens, unsigned stages,
                            gevva_stream_t stream) {
  if (!runner) return GEVVA_MOE_BAD_ARGUMENT;
  return gv::moe_launch_stages_on(runner, in, ids, route_weights, out, tokens, stages, stream, runner->sm_count);
}

int gevva_moe_launch(gevva_moe* runner, const void* in, const int* ids, const float* route_weights,
                     void* out, int tokens, gevva_stream_t stream) {
  if (!in || !ids) return GEVVA_MOE_BAD_ARGUMENT;
  unsigned stages = GEVVA_MOE_STAGE_ALL;
  if (!out) stages &= ~static_cast<unsigned>(GEVVA_MOE_STAGE_REDUCE);
  return gevva_moe_launch_stages(runner, in, ids, route_weights, out, tokens, stages, stream);
}

const void* gevva_moe_routed_output(const gevva_moe* runner) {
  return runner ? runner->scratch->w2_out : nullptr;
}

const int* gevva_moe_inverse_routes(const gevva_moe* runner) {
  return runner ? runner->scratch->plan.inverse_routes : nullptr;
}

int gevva_moe_last_status(gevva_moe* runner) {
  if (!runner) return GEVVA_MOE_BAD_ARGUMENT;
  int status = 0;
  GV_CUDA(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
  GV_CUDA(cudaMemcpy(&status, runner->scratch->plan.status, sizeof(int), cudaMemcpyDeviceToHost),
          "status read");
  if (status != 0) GV_CUDA(cudaMemset(runner->scratch->plan.status, 0, sizeof(int)), "status clear");
  return -status;
}

int gevva_moe_probe_bounded_wait(gevva_moe* runner, long long limit_cycles, gevva_stream_t stream) {
  if (!runner || limit_cycles < 1 || limit_cycles > 2000000000ll) return GEVVA_MOE_BAD_ARGUMENT;
  bounded_wait_probe_kernel<<<1, 32, 0, stream>>>(runner->scratch->plan.status, limit_cycles);
  GV_CUDA(cudaGetLastError(), "bounded wait probe");
  return GEVVA_MOE_OK;
}

int gevva_moe_buffer(const gevva_moe* runner, int buffer_id, void** device_ptr, size_t* bytes) {
  if (!runner || !device_ptr || !bytes) return GEVVA_MOE_BAD_ARGUMENT;
  const Scratch* s = runner->scratch;
  const size_t routes = static_cast<size_t>(s->routes);
  switch (buffer_id) {
    case GEVVA_MOE_BUF_INPUT_CODES: *device_ptr = s->input_codes; *bytes = routes * (kHidden / 2); break;
    case GEVVA_MOE_BUF_INPUT_SF: *device_ptr = s->input_sf; *bytes = s->input_sf_bytes; break;
    case GEVVA_MOE_BUF_W13_OUT: *device_ptr = s->w13_out; *bytes = routes * kW13Out * 2; break;
    case GEVVA_MOE_BUF_INTER_CODES: *device_ptr = s->inter_codes; *bytes = routes * (kInter / 2); break;
    case GEVVA_MOE_BUF_INTER_SF: *device_ptr = s->inter_sf; *bytes = s->inter_sf_bytes; break;
    case GEVVA_MOE_BUF_W2_OUT: *device_ptr = s->w2_out; *bytes = routes * kHidden * 2; break;
    case GEVVA_MOE_BUF_SORTED_EXPERTS: *device_ptr = s->plan.sorted_experts; *bytes = routes * 4; break;
    case GEVVA_MOE_BUF_SORTED_ROUTES: *device_ptr = s->plan.sorted_routes; *bytes = routes * 4; break;
    case GEVVA_MOE_BUF_INVERSE_ROUTES: *device_ptr = s->plan.inverse_routes; *bytes = routes * 4; break;
    case GEVVA_MOE_BUF_EXPERT_OFFSETS: *device_ptr = s->plan.expert_offsets; *bytes = (kExperts + 1) * 4; break;
    case GEVVA_MOE_BUF_SCALE_ROW_OFFSETS: *device_ptr = s->plan.scale_row_offsets; *bytes = (kExperts + 1) * 4; break;
    case GEVVA_MOE_BUF_TILE_EXPERT: *device_ptr = s->plan.tile_expert; *bytes = s->tile_capacity * 4; break;
    case GEVVA_MOE_BUF_NUM_TILES: *device_ptr = s->plan.num_m_tiles; *bytes = 4; break;
    default: return GEVVA_MOE_BAD_ARGUMENT;
  }
  return GEVVA_MOE_OK;
}

int gevva_moe_pack_experts(const float* weights, int experts, int n_out, int k_in, void* codes,
                           void* scales, float* global_scales, gevva_stream_t stream) {
  if (!weights || !codes || !scales || !global_scales || experts < 1 || n_out < 128 ||
      n_out % 128 != 0 || k_in < 64 || k_in % 64 != 0)
    return GEVVA_MOE_BAD_ARGUMENT;
  gv::launch_pack_weights(weights, experts, n_out, k_in, static_cast<uint8_t*>(codes),
                          static_cast<uint8_t*>(scales), global_scales, stream);
  GV_CUDA(cudaGetLastError(), "pack experts");
  return GEVVA_MOE_OK;
}

}  // extern "C"
