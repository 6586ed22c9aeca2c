// Both expert GEMMs of a batch with few rows an expert, in one persistent launch that streams weights.
//
// What bounds it.  Every routed expert's 3.3 MB come from HBM once: 65 us of it when all 128 experts are
// hit, whatever the batch; with a handful of tokens the time is the chain sort -> quantise -> w13 ->
// GeGLU -> w2.  So the weights sit on MMA-M (128 rows a tile, all of them real) and the rows of an
// expert on MMA-N, in multiples of 16.  What that buys is not tensor time (an MMA takes 40 to 64 cycles at N up to
// 128, and the pipe is 4 to 8 % busy) but finer steps: a pipeline stage carries 18 KB of weights instead of 34, and
// a w13 item is 64 intermediate columns (11 an expert, 180 KB), so one token's eight experts keep 88 SMs busy
// instead of 48.  A chunk ends at 64 rows because four accumulators of 64 columns and seven stages' scales fill tensor
// memory, and seven stages with 8 KB of rows each shared memory; an expert with more rows reads its weights once a chunk.
// Alone and from a cold L2: 64 tokens 75.8 us for 430 MB of DRAM traffic, 400 tokens (kFront false) 72.2 us for 440 MB,
// 5.7 and 6.1 TB/s over the whole launch.
//
//   w13 item   (chunk of at most 64 rows of an expert) x (unit of 64 intermediate columns): MMA rows 0..63
//              are the unit's up rows, 64..127 its gate rows (one 3-D box brings both; their scales come
//              from a copy re-tiled by unit, made at runner creation)
//   w2 item    (chunk) x (128 output columns)
// One list per launch, all w13 items chunk by chunk, then all w2 items.  A CTA's first w13 item is given by its number,
// further ones are claimed one by one, a little ahead; the w2 items are dealt in the order in which the CTAs run out of
// w13 items, so that those that are one short (180 KB) get four w2 items (48 KB each) first, and the last three of each share lie in
// a pool.  SMs get through their weights at different rates, and the CTAs on SMs that the router held start 1.7 us late: with fixed
// shares the CTAs of 64 tokens ended between 60.4 and 67.5 us (median 62.7).
// A CTA's items are worked out by the claim warp, ahead of their use, and the other roles read them as words from a ring.  Worked out
// from numbers by each role for itself, and with fixed shares, us a layer: 1 token 21.05 (now 20.75), 5 33.6 (33.9), 16 55.1 (53.3), 37 72.0 (69.3), 64 77.3
// (74.9), 200 83.5 (81.4), 613 95.9 (95.6), Zipf(1.1) 64 tokens 45.8 (45.7), 200 62.5 (60.9).  (The pool without the ring: 1 token 21.3, 5 33.5, 16 54.3,
// 37 71.4, 64 77.9, 200 85.3 against 21.0, 33.2, 55.2, 73.2, 79.0, 86.4 in that comparison; two or six items of a share in it: the same.)
//
// Roles (14 warps): 0 fetches weights, 1 copies scale factors to tensor memory and issues MMAs, 2 fetches activations
// (one thread each), 3 only takes part in the sort and the quantiser, 4..11 are the epilogue (two warps per 32-lane quarter, alternating
// groups of eight rows), 12 publishes finished w13 items, 13 works out the next ones.  Seven stages of one K block (256 elements); four accumulators of 64 columns,
// so nothing waits for a drain.  How fast a CTA gets through K blocks is a matter of how those three threads are written, not of
// bytes: with a warp of its own for the scale copies (a commit and a barrier more a stage), waits by whole warps and rolled K
// loops a w13 item whose weights lay in L2 took 3.8 us, with one thread a role and the K loops unrolled by two and four
// 2.6 (unrolled by eleven 3.4: its code no longer stays in the instruction cache).  64 tokens 86.2 -> 83.6 us a layer, 1 token 22.7 -> 21.9.  In the w13 epilogue a thread holds one weight row for eight tokens, so
// bf16(alpha * acc), which is what the reference's GEMM stores, changes hands through shared memory and a
// thread then owns one column of four tokens: GeGLU, block maxima over sixteen lanes, codes.  (One token at a
// time, with the scale worked out in all sixteen lanes, this took 87000 of 165000 cycles at 613 tokens and
// bounded the launch; now 48000, a layer 113.6 -> 110.9 us.)  The w2
// epilogue pairs two columns by one shuffle per two tokens and stores 64-byte pieces of a row.
//
// A w2 item needs the w2 operand rows of its expert: when the epilogue warps have stored an item, a
// publisher warp adds one to the expert's counter (release); the activation side of a w2 item waits for
// 11 x chunks of them (bounded acquire spin), crosses to the async proxy and loads.  The weight side
// waits for nothing, so weight bytes keep arriving across the boundary.
//
// What other streams run may keep a part of the grid from starting for any time, and another such grid that waits for
// SMs that this one holds must not be waited for.  So no wait depends on a CTA that is not running: of what is
// waited for, w13 items lie with CTAs that run (gv_stream_schedule.h), and tokens that are not quantised
// after 20 us are quantised by the CTAs that wait (stream_rescue_tokens).  Items dealt in advance to CTAs that were
// assumed to run, with a cooperative launch to have that, cost 2 us a layer in a graph and 4 us eagerly (64
// tokens, 87.7 -> 90 and 91 us), because such a launch starts only once all SMs are free.
//
// In its kFront form the kernel also sorts the routes and quantises the input: every CTA ranks the whole
// batch's routes for itself, with a bit per expert and token (a route's rank is the number of bits before its own; a token that names
// an expert twice is seen when its bit is set already, and the routes are then counted one by one) and derives the group geometry;
// CTA c quantises tokens c and c + CTAs with ten warps, a K block each, then adds one to a counter that
// the activation side waits for.  At 200 tokens that saves 4 us of a layer against launches of their own; with
// five tokens a CTA it would lose five (613 tokens: 119.5 against 114.1 us).
// Until that counter is full, all that moves is the weights that fit the ring, and its chain (stores, their
// release to the GPU, the poll, the copies) takes 5 to 8 us while they do.  So a CTA's first w13 item does not wait: if it has
// at most eight rows, eleven warps quantise these into the pipeline stages, and the counter is full by the
// time that the second item needs it.  24.5 -> 22.9 us a layer at 1 token, 36.1 -> 34.1 at 5, 53.7 -> 52.2 at 16, 70.2 -> 69.7
// at 37, nothing from 64 on, where more rows take as long as the counter (with 24 rows allowed, 5 us slower at 200).
// Time stamps at 64 tokens, from the end of the dependency wait: geometry 2.8 us with counts by match.any and three scans, 1.5
// with bits and one scan of packed words (200 tokens 3.8 and 1.9); the grid's own tokens 4.7 and 3.6.  Those come before the
// first item's rows wherever some CTA has a second item, and the MMA warp leaves its share of them to warp 3.
// 1 token 177 -> 172 us a pass of eight layers, 64 tokens 656 -> 646, 200 tokens (four layers) 360 -> 356.
// The code in front of the roles runs once a launch, and while the weights keep the way to L2 busy an instruction
// line that has to be fetched costs up to a microsecond: it is kept small, loops are not unrolled, and the two quantisers
// are run once on nothing in front of the dependency wait (37 tokens 615 -> 611, 40-token feed-forward layers 343 -> 338).
// Weights are asked for with an L2 policy that lets them give way first.  A launch passes 400 MB through L2, and without
// the policy that pushes out what the next launches start with: their code, the router's matrix, tokens, rows and counters.
// Us a layer (eight in a graph, one GPU): 1 token 21.5 -> 21.0, 5 34.2 -> 33.0, 16 57.1 -> 55.1, 37 75.2 -> 73.0, 64 80.9 -> 77.5, 200 87.2 -> 83.6,
// 400 92.6 -> 89.5, 613 99.7 -> 95.4.  Experts with several chunks, whose weights are read once a chunk, gain as much (Zipf(1.1), 200 tokens
// 65.1 -> 62.5, 613 96.7 -> 94; bias of deviation 0.5, 613 tokens 102.3 -> 98.7; theirs left without the policy: 64.0, 97.0, 103).
#include "gv_common.cuh"
#include "gv_gemm_parts.cuh"
#include "gv_launchers.h"
#include "gv_quantize.cuh"
#include "gv_stream_schedule.h"

namespace gv {

namespace {

constexpr int kStStages = 7;
constexpr int kStRows = 64;                               // rows of a chunk at most (MMA-N)
constexpr int kStAccStages = 4;
constexpr int kStWeightWarp = 0, kStMmaWarp = 1, kStTokenWarp = 2, kStSpareWarp = 3, kStEpilogueWarp = 4;
constexpr int kStEpilogueWarps = 8;
constexpr int kStPublishWarp = kStEpilogueWarp + kStEpilogueWarps;     // 12
constexpr int kStClaimWarp = kStPublishWarp + 1;                       // 13
constexpr int kStThreads = (kStClaimWarp + 1) * 32;                    // 448
constexpr uint32_t kStTmemColumns = 512;
constexpr uint32_t kStSfColumn = kStAccStages * kStRows;  // 256
constexpr uint32_t kStSfColumnsPerStage = 32;             // 16 for the weights, 16 for the rows
static_assert(kStSfColumn + kStSfColumnsPerStage * kStStages <= kStTmemColumns, "tensor memory budget");
constexpr int kStWeightBytes = kTileM * kTileKBytes;      // 16 KiB
constexpr int kStTokenBytes = kStRows * kTileKBytes;      // 8 KiB
static_assert(kStreamUpItems == kUnits && kStreamDownItems == kHidden / 128, "items of a chunk");
constexpr int kStUpKBlocks = kHidden / kTileK;            // 11
static_assert(kStMmaWarp == 1 && kStPublishWarp - 1 == kStUpKBlocks, "warps 1..11 quantise a K block of the first item each; of the CTA's own tokens warps 2..11, warp 3 two");
static_assert(kStWeightWarp == 0 && kExperts == 128, "threads 0..127 scan the experts");
constexpr int kStLoadUnroll = 2, kStMmaUnroll = 4;        // K blocks of w13 items
constexpr int kStDownKBlocks = 3;                         // 704 = 256 + 256 + 192
constexpr int kStDownLastMmas = 3;
constexpr int kStMaxChunks = 256;
constexpr int kStExchangeRows = 32;
constexpr int kStOwnTokens = 2;                           // kFront: tokens a CTA quantises, at most
constexpr int kStFrontRoutes = 6;                         // kFront: routes a thread looks at, at most
constexpr int kStFrontTokens = kStFrontRoutes * kStThreads / kTopK;  // 336
constexpr int kStFrontWords = (kStFrontTokens + 31) / 32; // 11, odd: an expert's words lie in banks of their own
constexpr uint32_t kStNoRow = 0xffffffffu;
constexpr int kStSelfRows = 8;                            // kFront: rows of a first item that the CTA quantises itself, at most
constexpr int kStItems = 32;                              // items on their way from the claim warp to the others, at most
constexpr int kStItemsAhead = 2;                          // item i is worked out once this many before it are still to be begun
constexpr uint32_t kStItemDown = 1u << 21, kStItemEnd = 1u << 22;
constexpr int kStAllPublished = 1 << 20;
constexpr long long kStRescueCycles = 40000;              // 20 us without progress

struct alignas(1024) StreamSmem {
  uint8_t a[kStStages][kStWeightBytes];
  uint8_t b[kStStages][kStTokenBytes];
  uint8_t sfa[kStStages][kSfStageBytes];
  uint8_t sfb[kStStages][kSfStageBytes];
  union {
    __nv_bfloat16 exchange[2][kStExchangeRows][128];  // [token][MMA row]
    uint32_t tokens_of[kExperts][kStFrontWords];      // the sort's, before: a bit per token
  };
  uint64_t full[kStStages], empty[kStStages];
  uint64_t acc_full[kStAccStages], acc_empty[kStAccStages];
  volatile int progress[kStEpilogueWarps];  // w13 items whose rows each epilogue warp has stored
  volatile int published;                   // w13 items that the publisher has counted; kStAllPublished at its end
  volatile int first_mine;                  // whether the CTA's first w13 item is its to count; -1: not known yet
  volatile int begun;                       // items that the weight warp has begun
  volatile uint32_t items[kStItems];        // the CTA's items: see stream_word
  uint32_t tmem_base;
  volatile int abort;
  volatile int left;  // an epilogue warp gave up waiting
  int last;           // this CTA is the last one to finish
  int chunks;
  int offsets[kExperts + 1];
  int scale_rows[kExperts + 1];
  int chunks_of[kExperts];
  short chunk_expert[kStMaxChunks];
  short chunk_index[kStMaxChunks];  // which chunk of its expert
  uint32_t scan[kExperts / 32];
  // kFront
  volatile int repeats;                // a token names an expert twice: tokens_of does not count its routes
  int histogram[kExperts];             // ... which these two do
  int own_rank[kStOwnTokens * kTopK];
  // the routes of this CTA's tokens
  alignas(16) uint2 route_at[kStOwnTokens * kTopK];  // where the row's codes and its scale bytes begin
  alignas(16) float route_multiplier[kStOwnTokens * kTopK];
  float scale_q1[kExperts];
  GegluTables tables;
};
constexpr size_t kStSmemBytes = sizeof(StreamSmem) + 1024;
static_assert(kStSmemBytes <= 232448, "shared memory budget of one sm_100 CTA");

struct StreamMaps {
  CUtensorMap w13;                 // [256 halves, 704 rows, 1408 bytes], box 2 x 64 rows x 128 bytes
  CUtensorMap w2;                  // [128 * 2816 rows, 352 bytes], box 128 rows x 128 bytes
  CUtensorMap up[kStRows / 8];     // input codes through boxes of 8, 16, ... 64 rows x 128 bytes
  CUtensorMap down[kStRows / 8];   // w2 operand codes likewise
};

struct StreamParams {
  RoutePlan plan;
  const uint8_t* w13_scales;  // re-tiled by unit
  const uint8_t* w2_scales;   // sidecar layout
  const uint8_t* input_scales;
  uint8_t* inter_codes;
  uint8_t* inter_scales;
  __nv_bfloat16* routed;
  const float *alpha1, *alpha2, *in_scale_q2;
  // kFront only
  const __nv_bfloat16* input;
  const int* expert_ids;
  const float* in_scale_q1;
  uint8_t* packed;
  uint8_t* scales;
  int tokens;
};

struct StreamItem {
  bool down;
  int expert;
  int chunk;   // of the expert
  int n_tile;  // unit of 64 intermediate columns, or tile of 128 output columns
};

// An item as a word: expert, n_tile << 7, chunk << 12, kStItemDown; or kStItemEnd behind the last one.
__device__ __forceinline__ uint32_t stream_word(int expert, int chunk, int n_tile) {
  return static_cast<uint32_t>(expert) | static_cast<uint32_t>(n_tile) << 7 | static_cast<uint32_t>(chunk) << 12;
}
__device__ __forceinline__ StreamItem stream_unpack(uint32_t word) {
  StreamItem it;
  it.down = word & kStItemDown;
  it.expert = word & 127u;
  it.n_tile = word >> 7 & 31u;
  it.chunk = word >> 12 & 511u;
  return it;
}
static_assert(kExperts == 128 && kStreamDownItems <= 32 && kStreamUpItems <= 32 && kStMaxChunks <= 512, "fields of an item's word");

// The word of item `i` of this CTA, w13 items first, with the turn of its place in the ring above it.  The claim warp works the items out and
// announces one after the other, the end also when it gives up; its own waits are bounded, so the wait below ends.
__device__ __forceinline__ uint32_t stream_turn(int i) { return static_cast<uint32_t>(i / kStItems + 1) << 24; }
__device__ __forceinline__ bool stream_announced(uint32_t word, int i) { return (word & 0xff000000u) == stream_turn(i); }
__device__ __forceinline__ bool stream_next(const StreamSmem* smem, int& taken, StreamItem& it) {
  uint32_t word = smem->items[taken % kStItems];
  while (!stream_announced(word, taken)) {
    __nanosleep(32);
    word = smem->items[taken % kStItems];
  }
  if (word & kStItemEnd) return false;
  it = stream_unpack(word);
  ++taken;
  return true;
}

// By one thread of the claim warp, which is never more than three items ahead of the weight warp.  No other reader is further than nine
// items behind that one (pipeline and accumulators), but for the publisher, which reads the w13 items.
__device__ __forceinline__ void stream_announce(StreamSmem* smem, int i, uint32_t word) {
  const long long start = clock64();
  while (smem->published + kStItems <= i && !smem->abort && clock64() - start < kWaitLimitCycles) __nanosleep(64);
  __threadfence_block();
  smem->items[i % kStItems] = stream_turn(i) | word;
}

// The lane's view of the CTAs' first items: one that is not taken, or `firsts`.
__device__ __forceinline__ int stream_open_first(const int* sync, int firsts, int lane) {
  int taken[kStreamMaxCtas / 32], open = firsts;
#pragma unroll
  for (int j = 0; j < kStreamMaxCtas / 32; ++j)
    taken[j] = lane + 32 * j < firsts ? *reinterpret_cast<const volatile int*>(sync + kStreamFirsts + lane + 32 * j) : 1;
#pragma unroll
  for (int j = 0; j < kStreamMaxCtas / 32; ++j)
    if (taken[j] == 0) open = lane + 32 * j;
  return open;
}

// Item `index` of the list of w13 items, or of that of w2 items.
__device__ __forceinline__ uint32_t stream_word_of(int index, bool down, const StreamSmem* smem) {
  const int per_chunk = down ? kStreamDownItems : kStreamUpItems;
  const int chunk = index / per_chunk;
  return stream_word(smem->chunk_expert[chunk], smem->chunk_index[chunk], index - chunk * per_chunk) | (down ? kStItemDown : 0u);
}

// Nothing unless `wanted`, which is the same in the whole warp; the registers are undefined then.
__device__ __forceinline__ void tmem_load_32x8(bool wanted, uint32_t tmem_address, uint32_t (&r)[8]) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %9, 0;\n\t"
      "@p tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t}"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(tmem_address), "r"(static_cast<uint32_t>(wanted))
      : "memory");
}

// A number of MMAs as a type.
template <int kCount>
struct MmaCount {
  __device__ constexpr int operator()() const { return kCount; }
};

// The MMAs of one K block (K = 64 each) with a runtime instruction descriptor (its N field).  Scale
// columns of the stage: weights of MMA j at +4j; rows at +16 + 4j, plus two where the chunk is the second
// half of its 128-row scale atom.
template <int kMmas>
__device__ __forceinline__ void stream_mmas(uint32_t tmem_acc, uint32_t tmem_sfa, uint32_t tmem_sfb, uint32_t a_lo,
                                            uint32_t b_lo, uint32_t descriptor, uint32_t accumulate) {
  constexpr uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);  // 8 rows x 128 B groups, 128B swizzle
#pragma unroll
  for (int j = 0; j < kMmas; ++j) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 d0, d1;\n\t"
        "setp.ne.b32 p, %7, 0;\n\t"
        "mov.b64 d0, {%1, %3};\n\t"
        "mov.b64 d1, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], d0, d1, %4, [%5], [%6], p;\n\t}" ::"r"(tmem_acc),
        "r"(a_lo + 2 * j), "r"(b_lo + 2 * j), "r"(hi), "r"(descriptor), "r"(tmem_sfa + 4 * j), "r"(tmem_sfb + 4 * j),
        "r"(j == 0 ? accumulate : 1u)
        : "memory");
  }
}

// A load that is issued here; the compiler puts an ordinary one where its value is used, a trip to memory later.
__device__ __forceinline__ uint4 stream_load_now(const uint4* address) {
  uint4 v;
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(address) : "memory");
  return v;
}

__device__ __forceinline__ int stream_load_acquire(const int* address) {
  int value;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(value) : "l"(address) : "memory");
  return value;
}

// Adds one, after everything that happened before in this thread and in those it has synchronised with; it has arrived when this returns (one in
// flight could come behind the zeros of the CTA that finishes last).
__device__ __forceinline__ void stream_count_release(int* address, StreamSmem* smem) {
  int before;
  asm volatile("atom.release.gpu.global.add.s32 %0, [%1], 1;" : "=r"(before) : "l"(address) : "memory");
  if (before < 0) smem->abort = 1;  // never: what waits for the answer
}

// Of the claim warp: until the weight warp has begun `items` of the CTA's.
__device__ __forceinline__ bool stream_wait_begun(StreamSmem* smem, int items, int* status) {
  return stream_wait(
      2 * kWaitLimitCycles, [&] { return smem->begun >= items; }, [&] { return smem->abort != 0; }, [] { return clock64(); },
      [] { __nanosleep(64); },
      [&] {
        smem->abort = 1;
        atomicExch(status, static_cast<int>(kWaitTimeout));
      });
}

// Bounded acquire spin of one thread on a counter in global memory; or, where one is given, on a second one.
__device__ __forceinline__ bool stream_wait_counter(const int* counter, int target, StreamSmem* smem, int* status,
                                                    const int* other = nullptr, int other_target = 0) {
  const long long start = clock64();
  bool ready = false;
  for (uint32_t spin = 1; !ready; ++spin) {
    ready = stream_load_acquire(counter) >= target;
    if (!ready && (spin & 63u) == 0) {
      if (other && stream_load_acquire(other) >= other_target) {
        ready = true;
        break;
      }
      if (smem->abort) break;
      if (clock64() - start > kWaitLimitCycles) {
        smem->abort = 1;
        atomicExch(status, static_cast<int>(kWaitTimeout));
        break;
      }
    }
  }
  return ready;
}

// Eight columns a lane (two lanes a 16-value block): code bytes and scale of the block.  The arithmetic of
// quantize_routes_of_token.
__device__ __forceinline__ uint32_t stream_quantise(const float (&values)[8], float maximum, float multiplier,
                                                    const float* reciprocals, uint32_t& codes) {
  const uint32_t scale = encode_e4m3(gv_sixth(__fmul_rn(multiplier, maximum)));
  const float inverse = gv_scale_inverse_exact(multiplier) ? gv_scale_inverse(multiplier, scale, reciprocals)
                                                           : scale_inverse_divided(multiplier, scale);
  codes = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    codes |= encode_e2m1x2(__fmul_rn(values[2 * i], inverse), __fmul_rn(values[2 * i + 1], inverse)) << (8 * i);
  return scale;
}

__device__ __forceinline__ float stream_block_maximum(const uint4& raw, float (&values)[8]) {
  unpack_bf16x8(raw, values);
  float maximum = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) maximum = fmaxf(maximum, fabsf(values[i]));
  return fmaxf(maximum, __shfl_xor_sync(0xffffffffu, maximum, 1));
}

// K block `kb` of one token by a warp: the codes and scale bytes of its eight routes (entries first..first+7 of
// the route arrays) go to their sorted rows.  (Arguments by value: a kernel parameter's fields read through a reference
// come from memory, a microsecond away.)
__device__ __noinline__ void stream_quantise_token(uint8_t* packed, uint8_t* scales, const StreamSmem* smem, int first, int kb,
                                                   int lane, uint4 raw, bool dry) {
  float values[8];
  const float maximum = stream_block_maximum(raw, values);
  packed += kb * kTileKBytes + 4 * lane;
  // scale groups of a row go four to an aligned word of the swizzled layout: eight lanes a word
  scales += static_cast<uint32_t>(4 * kb + (lane >> 3)) * kSfAtomBytes;
  uint4 at[kTopK / 2];  // code offset and scale offset of two routes each
#pragma unroll
  for (int i = 0; i < kTopK / 2; ++i) at[i] = reinterpret_cast<const uint4*>(smem->route_at + first)[i];
  const float4 m0 = *reinterpret_cast<const float4*>(smem->route_multiplier + first);
  const float4 m1 = *reinterpret_cast<const float4*>(smem->route_multiplier + first + 4);
  const float multipliers[kTopK] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
  uint32_t codes = 0, scale_word = 0;
#pragma unroll 1
  for (int done = 0; done < kTopK;) {
    // the routes from `done` on that share a static scale share the result
    float multiplier = 0.0f;
#pragma unroll
    for (int k = 0; k < kTopK; ++k)
      if (k == done) multiplier = multipliers[k];
    const uint32_t scale = stream_quantise(values, maximum, multiplier, smem->tables.reciprocals, codes);
    scale_word = scale | (__shfl_down_sync(0xffffffffu, scale, 2) << 8) | (__shfl_down_sync(0xffffffffu, scale, 4) << 16) |
                 (__shfl_down_sync(0xffffffffu, scale, 6) << 24);
    const int from = done;
    bool same = true;
#pragma unroll
    for (int k = 0; k < kTopK; ++k) {
      const uint32_t code_at = k & 1 ? at[k / 2].z : at[k / 2].x, scale_at = k & 1 ? at[k / 2].w : at[k / 2].y;
      same = same && (k < from || __float_as_uint(multipliers[k]) == __float_as_uint(multiplier));
      const bool store = same && k >= from && code_at != kStNoRow && !dry;
      if (store) *reinterpret_cast<uint32_t*>(packed + code_at) = codes;
      if (store && (lane & 7) == 0) *reinterpret_cast<uint32_t*>(scales + scale_at) = scale_word;
      done = same && k >= from ? k + 1 : done;
    }
  }
}

// The token of row `target` of an expert (rows in the order of the sort).
__device__ __forceinline__ int stream_token_of_row(const StreamSmem* smem, int expert, int target, int words) {
#pragma unroll 1
  for (int w = 0; w < words; ++w) {
    uint32_t bits = smem->tokens_of[expert][w];
    const int count = __popc(bits);
    if (target < count) {
      for (; target > 0; --target) bits &= bits - 1;
      return 32 * w + __ffs(static_cast<int>(bits)) - 1;
    }
    target -= count;
  }
  return 0;
}

// The same from the ids, by a warp, for rows first + lane; and a route's rank among those of its expert: where a token
// names an expert twice.
__device__ __noinline__ int stream_token_of_row_repeated(const int* expert_ids, int routes, int expert, int first, int lane) {
  int before = 0, token = 0;
#pragma unroll 4
  for (int base = 0; base < routes; base += 32) {
    uint32_t all = __ballot_sync(0xffffffffu, base + lane < routes && expert_ids[base + lane] == expert);
    const int count = __popc(all);
    int target = first + lane - before;
    if (target >= 0 && target < count) {
      for (; target > 0; --target) all &= all - 1;
      token = (base + __ffs(static_cast<int>(all)) - 1) / kTopK;
    }
    before += count;
  }
  return token;
}
__device__ __noinline__ int stream_rank_repeated(const int* expert_ids, int route, int lane) {
  const int expert = expert_ids[route];
  int rank = 0;
#pragma unroll 4
  for (int base = 0; base < route; base += 32)
    rank += __popc(__ballot_sync(0xffffffffu, base + lane < route && expert_ids[base + lane] == expert));
  return rank;
}

// K block `kb` of an item's `rows` tokens (lane r holds the one of row r) by a warp, straight into a pipeline stage: codes in
// the 128B-swizzled layout of the row side, scale bytes at rows scale_row.. of the stage's four atoms.  The tokens
// are fetched into the stage first, 512 bytes each from its byte 2048 on, where the codes that replace them
// never reach a token that is still to be read; or, in a batch of a few, they lie there already, in their own order.
// Everything here runs once a launch, while the weights keep the way to L2 busy, and an instruction line that has to
// be fetched takes about a microsecond: hence one copy of the code and no unrolling.
constexpr int kStTokensAt = 2048;
__device__ __forceinline__ void stream_fetch_token(uint8_t* stage_rows, int slot, const uint4* input, int token, int kb, int lane) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(stage_rows + kStTokensAt + slot * 512 + lane * 16)),
               "l"(input + static_cast<size_t>(token) * (kHidden / 8) + kb * (kTileK / 8) + lane)
               : "memory");
}
static_assert(kStTokensAt + kStSelfRows * 512 <= kStTokenBytes && kStSelfRows * kTileKBytes <= kStTokensAt, "codes and tokens in one stage");
__device__ __noinline__ void stream_quantise_stage(const uint4* input, StreamSmem* smem, int stage, int kb, int rows, int tokens,
                                                   bool fetched, int scale_row, float multiplier, int lane, bool dry) {
  uint8_t* const b = smem->b[stage];
  uint8_t* const sf = smem->sfb[stage] + (lane >> 3) * kSfAtomBytes + ((lane >> 1) & 3);
  if (!fetched) {
#pragma unroll 1
    for (int r = 0; r < rows; ++r) stream_fetch_token(b, r, input, __shfl_sync(0xffffffffu, tokens, r), kb, lane);
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
#pragma unroll 1
  for (int r = 0; r < rows; ++r) {
    const int slot = fetched ? __shfl_sync(0xffffffffu, tokens, r) : r;
    float values[8];
    const float maximum = stream_block_maximum(*reinterpret_cast<const uint4*>(b + kStTokensAt + slot * 512 + lane * 16), values);
    uint32_t codes;
    const uint32_t scale = stream_quantise(values, maximum, multiplier, smem->tables.reciprocals, codes);
    *reinterpret_cast<uint32_t*>(b + r * kTileKBytes + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4) = codes;
    const int n = scale_row + r;
    if ((lane & 1) == 0) sf[(n & 31) * 16 + ((n >> 5) & 3) * 4] = static_cast<uint8_t>(scale);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (lane == 0 && !dry) mbar_arrive(&smem->full[stage]);
}

// Offsets of the codes and the scale bytes of an expert's row (below 4 MB in batches of this size).
__device__ __forceinline__ uint2 stream_route_at(const StreamSmem* smem, int expert, int rank) {
  return make_uint2(static_cast<uint32_t>(smem->offsets[expert] + rank) * (kHidden / 2),
                    static_cast<uint32_t>(smem->scale_rows[expert]) * (kHidden / 16) +
                        static_cast<uint32_t>(sf_offset(rank, 0, kHidden / 16)));
}

// By the publisher warp of a CTA that has had nothing to do for a while: the grid's CTAs quantise two tokens each at most,
// and some may not be running.  The ones that are go over all tokens, token by token; a CTA that starts after all writes the
// same bytes again.  (Their ranks are counted anew: the sort's tables have given way to the exchange tile.)
__device__ __noinline__ void stream_rescue_tokens(const StreamParams& p, StreamSmem* smem, int lane) {
  int* const sync = p.plan.stream_sync;
  const int owners = p.tokens < static_cast<int>(gridDim.x) ? p.tokens : static_cast<int>(gridDim.x);
  if (stream_load_acquire(sync + kStreamQuantised) >= owners) return;
#pragma unroll 1
  for (;;) {
    int token = 0;
    if (lane == 0) token = atomicAdd(sync + kStreamRescueClaims, 1);
    token = __shfl_sync(0xffffffffu, token, 0);
    if (token >= p.tokens || smem->abort) return;
#pragma unroll 1
    for (int k = 0; k < kTopK; ++k) {
      const int route = token * kTopK + k;
      const int expert = p.expert_ids[route];
      int rank = 0;
#pragma unroll 1
      for (int base = 0; base < route; base += 32)
        rank += __popc(__ballot_sync(0xffffffffu, base + lane < route && p.expert_ids[base + lane] == expert));
      if (lane == 0) {
        const bool valid = expert >= 0 && expert < kExperts;
        smem->route_at[k] = valid ? stream_route_at(smem, expert, rank) : make_uint2(kStNoRow, 0);
        smem->route_multiplier[k] = valid ? smem->scale_q1[expert] : 0.0f;
      }
    }
    __syncwarp();
    const uint4* const input = reinterpret_cast<const uint4*>(p.input) + static_cast<size_t>(token) * (kHidden / 8) + lane;
#pragma unroll 1
    for (int kb = 0; kb < kStUpKBlocks; ++kb) stream_quantise_token(p.packed, p.scales, smem, 0, kb, lane, __ldg(input + kb * (kTileK / 8)), false);
    __syncwarp();
    if (lane == 0) stream_count_release(sync + kStreamRescued, smem);
  }
}

template <bool kFront>
__global__ void __launch_bounds__(kStThreads, 1)
stream_experts_kernel(const __grid_constant__ StreamMaps maps, const __grid_constant__ StreamParams p) {
  extern __shared__ uint8_t smem_raw[];
  StreamSmem* smem =
      reinterpret_cast<StreamSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int cta = blockIdx.x;
  int* const status = p.plan.status;

  if (tid == 0) {
    for (int s = 0; s < kStStages; ++s) {
      mbar_init(&smem->full[s], 2);  // one arrival (with its byte count) per producer warp
      mbar_init(&smem->empty[s], 1);
    }
    for (int s = 0; s < kStAccStages; ++s) {
      mbar_init(&smem->acc_full[s], 1);
      mbar_init(&smem->acc_empty[s], kStEpilogueWarps);
    }
    for (int w = 0; w < kStEpilogueWarps; ++w) smem->progress[w] = 0;
    smem->published = 0;
    smem->first_mine = -1;
    smem->begun = 0;
    smem->repeats = 0;
    smem->abort = 0;
    smem->left = 0;
    fence_barrier_init();
    prefetch_tensor_map(&maps.w13);
    prefetch_tensor_map(&maps.w2);
    prefetch_tensor_map(&maps.up[0]);
    prefetch_tensor_map(&maps.down[0]);
  }
  if (tid < kStItems) smem->items[tid] = 0;
  if (kFront && tid < kTopK) {
    smem->route_at[tid] = make_uint2(kStNoRow, 0);
    smem->route_multiplier[tid] = 1.0f;
  }
  if (warp == kStMmaWarp) {
    tmem_alloc(&smem->tmem_base, kStTmemColumns);
    tmem_relinquish();
  }
  load_geglu_tables(&smem->tables);
  __syncthreads();
  fill_geglu_tables(&smem->tables);
  if (kFront)
    for (int i = tid; i < kExperts * kStFrontWords; i += kStThreads) (&smem->tokens_of[0][0])[i] = 0;
  grid_launch_dependents();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = smem->tmem_base;
  if (kFront && p.tokens > kStSelfRows && warp >= 4 && warp < 8) {
    // the quantisers' code is brought in while the CTA has nothing else to do
    stream_quantise_token(p.packed, p.scales, smem, 0, 0, lane, make_uint4(0, 0, 0, 0), true);
    stream_quantise_stage(nullptr, smem, warp - 4, 0, 1, 0, true, 0, 1.0f, lane, true);
  }
  const int first_chunk = cta / kStreamUpItems, first_unit = cta - first_chunk * kStreamUpItems;  // the CTA's first w13 item
  grid_dependency_wait();  // what earlier kernels of the stream wrote is visible from here on
  int* const sync = p.plan.stream_sync;
  int first_taken = 0;
  if (tid == kStClaimWarp * 32) first_taken = atomicExch(sync + kStreamFirsts + cta, 1);

  // ---------------- group geometry ----------------
  const bool has_token = kFront && cta < p.tokens;
  const int ctas = gridDim.x;
  const int routes = kFront ? p.tokens * kTopK : 0;
  const int words = (p.tokens + 31) >> 5;
  const int own = has_token ? (p.tokens - 1 - cta) / ctas + 1 : 0;
  const int kb = warp - kStMmaWarp;  // 0..10: the K block that the warp quantises
  // in a batch this small every token may be in the CTA's first item
  const bool fetched = kFront && p.tokens <= kStSelfRows && kb < kStStages;
  // Of the CTA's own tokens, that goes for warps 2..11; warp 3, which has no role later, takes the MMA warp's K block, too.
  uint4 own_raw[kStOwnTokens], mma_raw[kStOwnTokens];
  int own_expert = -1;  // publisher warp, a lane each of the CTA's own routes
  int count = 0;  // threads 0..127: rows of expert tid
  if constexpr (kFront) {
    const float scale_q1 = tid < kExperts ? p.in_scale_q1[tid] : 0.0f;
    int ids[kStFrontRoutes];
#pragma unroll
    for (int k = 0; k < kStFrontRoutes; ++k) ids[k] = tid + k * kStThreads < routes ? p.expert_ids[tid + k * kStThreads] : -1;
    const int own_route = (cta + lane / kTopK * ctas) * kTopK + lane % kTopK;
    if (warp == kStPublishWarp && lane < own * kTopK) own_expert = p.expert_ids[own_route];
    // what the warp will quantise (see below) is on its way meanwhile
    const uint4* const input = reinterpret_cast<const uint4*>(p.input);
    if (fetched && kb >= 0)
      for (int t = 0; t < p.tokens; ++t) stream_fetch_token(smem->b[kb], t, input, t, kb, lane);
    if (kb > 0 && kb < kStUpKBlocks) {
#pragma unroll
      for (int t = 0; t < kStOwnTokens; ++t)
        if (t < own) {
          const uint4* const token = input + static_cast<size_t>(cta + t * ctas) * (kHidden / 8) + lane;
          own_raw[t] = stream_load_now(token + kb * (kTileK / 8));
          if (warp == kStSpareWarp) mma_raw[t] = stream_load_now(token);
        }
    }
    // Every expert's tokens as bits; a bit found set is a token that names its expert twice.
    uint32_t repeated = 0;
#pragma unroll
    for (int k = 0; k < kStFrontRoutes; ++k) {
      const int route = tid + k * kStThreads;
      if (route < routes) {
        const uint32_t bit = 1u << ((route / kTopK) & 31);
        if (ids[k] >= 0 && ids[k] < kExperts) repeated |= atomicOr(&smem->tokens_of[ids[k]][route / (32 * kTopK)], bit) & bit;
        else if (cta == 0) atomicExch(status, static_cast<int>(kBadExpertId));
      }
    }
    if (repeated) smem->repeats = 1;
    if (tid < kExperts) {
      smem->scale_q1[tid] = scale_q1;
      smem->histogram[tid] = 0;
    }
    __syncthreads();
    if (smem->repeats) {
      // not what a router gives: counted one by one
#pragma unroll
      for (int k = 0; k < kStFrontRoutes; ++k)
        if (ids[k] >= 0 && ids[k] < kExperts) atomicAdd(&smem->histogram[ids[k]], 1);
      for (int q = warp; q < own * kTopK; q += kStThreads / 32) {
        const int rank = stream_rank_repeated(p.expert_ids, (cta + q / kTopK * ctas) * kTopK + q % kTopK, lane);
        if (lane == 0) smem->own_rank[q] = rank;
      }
      __syncthreads();
      if (tid < kExperts) count = smem->histogram[tid];
    } else if (tid < kExperts) {
#pragma unroll
      for (int w = 0; w < kStFrontWords; ++w)
        if (w < words) count += __popc(smem->tokens_of[tid][w]);
    }
  } else {
    if (tid < kExperts) count = p.plan.expert_offsets[tid + 1] - p.plan.expert_offsets[tid];
  }
  if (tid < kExperts) {
    // rows, 128-row scale tiles and chunks of the experts before this one, in one word
    static_assert(kStreamMaxTokens * kTopK < (1 << 14) && kExperts + kStreamMaxTokens * kTopK / kTileM < (1 << 9) && kStMaxChunks < (1 << 9), "scan in one word");
    const int tiles = (count + kTileM - 1) / kTileM, chunks = (count + kStRows - 1) / kStRows;
    const uint32_t packed = static_cast<uint32_t>(count) | static_cast<uint32_t>(tiles) << 14 | static_cast<uint32_t>(chunks) << 23;
    uint32_t inclusive = packed;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
      const uint32_t other = __shfl_up_sync(0xffffffffu, inclusive, offset);
      if (lane >= offset) inclusive += other;
    }
    if (lane == 31) smem->scan[warp] = inclusive;
    named_barrier(4, kExperts);
#pragma unroll
    for (int w = 0; w < kExperts / 32 - 1; ++w)
      if (w < warp) inclusive += smem->scan[w];
    const uint32_t before = inclusive - packed;
    const int row = before & 0x3fffu, tile = before >> 14 & 0x1ffu, chunk = before >> 23;
    smem->offsets[tid] = row;
    smem->scale_rows[tid] = tile * kTileM;
    smem->chunks_of[tid] = chunks;
#pragma unroll 1
    for (int c = 0; c < chunks; ++c) {
      smem->chunk_expert[chunk + c] = static_cast<short>(tid);
      smem->chunk_index[chunk + c] = static_cast<short>(c);
      if (chunk + c == first_chunk) smem->items[0] = stream_turn(0) | stream_word(tid, c, first_unit);
    }
    if (tid == kExperts - 1) {
      const int all_chunks = chunk + chunks;
      smem->offsets[kExperts] = row + count;
      smem->scale_rows[kExperts] = (tile + tiles) * kTileM;
      smem->chunks = all_chunks;
    }
    if (kFront && cta == 0) {
      p.plan.expert_offsets[tid] = row;
      p.plan.scale_row_offsets[tid] = tile * kTileM;
      for (int t = 0; t < tiles; ++t) p.plan.tile_expert[tile + t] = tid;
      if (tid == kExperts - 1) {
        p.plan.expert_offsets[kExperts] = row + count;
        p.plan.scale_row_offsets[kExperts] = (tile + tiles) * kTileM;
        p.plan.num_m_tiles[0] = tile + tiles;
      }
    }
  }
  if (fetched) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    fence_proxy_async_smem();  // a stage whose tokens are not used after all is filled by a tensor-map copy
  }
  __syncthreads();
  const int ups = smem->chunks * kStreamUpItems;  // w13 items of the launch
  int taken = 0;                                  // items that this thread's role has walked past
  StreamItem it{};
  bool ok = true;

  // kFront: the CTA's first w13 item does not wait for the grid's quantised rows: its own warps put them into
  // the pipeline stages (not the concern of the weight and claim warps, which leave it out)
  bool self_first = kFront && cta < ups;
  if (kFront && warp != kStWeightWarp && warp != kStClaimWarp) {  // the weights are under way meanwhile
    const uint4* const input = reinterpret_cast<const uint4*>(p.input);
    int first = 0, first_rows = 0;
    if (self_first) {
      it = stream_unpack(smem->items[0]);
      first = it.chunk * kStRows;
      first_rows = smem->offsets[it.expert + 1] - smem->offsets[it.expert] - first;
      first_rows = first_rows > kStRows ? kStRows : first_rows;
      self_first = first_rows <= kStSelfRows;  // with more, the grid's rows are there as early
    }
    float multiplier = 0.0f;
    int tokens = 0;  // lane r: the token of row r of that item
    if (self_first && warp != kStPublishWarp) {
      multiplier = smem->scale_q1[it.expert];
      if (smem->repeats) tokens = stream_token_of_row_repeated(p.expert_ids, routes, it.expert, first, lane);
      else if (lane < first_rows) tokens = stream_token_of_row(smem, it.expert, first + lane, words);
      __syncwarp();
    }
    // The CTA's own tokens come first where some CTA has a second item, which needs the grid's.
    const bool own_first = ups > ctas;
#pragma unroll 1
    for (int step = 0; step < 2; ++step) {
      if ((step == 0) != own_first) {
        if (self_first && warp != kStPublishWarp && kb < kStStages)
          stream_quantise_stage(input, smem, kb, kb, first_rows, tokens, fetched, first % kTileM, multiplier, lane, false);
      } else if (has_token && warp != kStMmaWarp) {
        constexpr int kOwnThreads = kStUpKBlocks * 32;  // warps 2..12
        if (warp == kStPublishWarp) {
          // where this CTA's tokens' routes go
          if (lane < own * kTopK) {
            const int route = (cta + lane / kTopK * ctas) * kTopK + lane % kTopK;
            const int expert = own_expert;
            const bool valid = expert >= 0 && expert < kExperts;  // others are flagged above
            if (valid) {
              int rank = 0;
              if (smem->repeats) {
                rank = smem->own_rank[lane];
              } else {
                const int token = route / kTopK;
#pragma unroll 1
                for (int w = 0; w < token >> 5; ++w) rank += __popc(smem->tokens_of[expert][w]);
                rank += __popc(smem->tokens_of[expert][token >> 5] & ((1u << (token & 31)) - 1u));
              }
              const int dst = smem->offsets[expert] + rank;
              p.plan.sorted_experts[dst] = expert;
              p.plan.sorted_routes[dst] = route;
              p.plan.inverse_routes[route] = dst;
              smem->route_at[lane] = stream_route_at(smem, expert, rank);
            } else {
              smem->route_at[lane] = make_uint2(kStNoRow, 0);
            }
            smem->route_multiplier[lane] = valid ? smem->scale_q1[expert] : 0.0f;
          }
          named_barrier(3, kOwnThreads);
          named_barrier(1, kOwnThreads);
          if (lane == 0) stream_count_release(sync + kStreamQuantised, smem);
        } else {
          named_barrier(3, kOwnThreads);
#pragma unroll 1
          for (int t = 0; t < own; ++t) {
            stream_quantise_token(p.packed, p.scales, smem, t * kTopK, kb, lane, own_raw[t ? 1 : 0], false);
            if (warp == kStSpareWarp) stream_quantise_token(p.packed, p.scales, smem, t * kTopK, 0, lane, mma_raw[t ? 1 : 0], false);
          }
          asm volatile("bar.arrive 1, %0;" ::"n"(kOwnThreads) : "memory");
        }
      }
    }
    if (self_first && kb >= kStStages && kb < kStUpKBlocks) {
      // the stage's second use
      if (__all_sync(0xffffffffu, wait_or_abort(&smem->empty[kb - kStStages], 0u, smem, status)))
        stream_quantise_stage(input, smem, kb - kStStages, kb, first_rows, tokens, false, first % kTileM, multiplier, lane, false);
    }
  }

  if (warp == kStWeightWarp || warp == kStTokenWarp) {
    // ---------------- producers, a thread each ----------------
    const bool weight_side = warp == kStWeightWarp;
    const uint64_t read_once = read_once_policy();
    int stage = 0, issued = 0;
    uint32_t phase = 0;
    bool rows_pending = kFront && !weight_side;
    if (self_first && !weight_side) {
      (void)stream_next(smem, taken, it);
      stage = kStUpKBlocks % kStStages;
      phase = kStUpKBlocks / kStStages & 1;
    }
    if (elect_one()) {
      while (ok && stream_next(smem, taken, it)) {
        if (weight_side) smem->begun = taken;
        const int first = it.chunk * kStRows;
        const int rows = smem->offsets[it.expert + 1] - smem->offsets[it.expert] - first;
        const int boxes = rows >= kStRows ? kStRows / 8 : (rows + 7) / 8;
        const int row = smem->offsets[it.expert] + first;
        const uint8_t* sf;
        if (weight_side) {
          sf = it.down ? p.w2_scales + static_cast<size_t>(it.expert * kHidden + it.n_tile * 128) * (kInter / 16)
                       : p.w13_scales + static_cast<size_t>(it.expert * kUnitSlots + it.n_tile) * kStUpKBlocks * kSfStageBytes;
        } else {
          const size_t scale_row = smem->scale_rows[it.expert] + first / kTileM * kTileM;
          if (rows_pending && !it.down) {
            // the w13 operand exists once every CTA with tokens has quantised them and counted itself
            ok = stream_wait_counter(sync + kStreamQuantised, p.tokens < ctas ? p.tokens : ctas, smem, status,
                                     sync + kStreamRescued, p.tokens);
            if (!ok) break;
            rows_pending = false;
            asm volatile("fence.proxy.async.global;" ::: "memory");
          }
          sf = it.down ? p.inter_scales + scale_row * (kInter / 16) : p.input_scales + scale_row * (kHidden / 16);
          if (it.down) {
            // the rows exist once every w13 item of the expert has been counted; they were written by ordinary stores of other SMs and are read through the async proxy
            ok = stream_wait_counter(p.plan.tile_ready + it.expert, kUnits * smem->chunks_of[it.expert], smem, status);
            if (!ok) break;
            asm volatile("fence.proxy.async.global;" ::: "memory");
          }
        }
        // One K block.  The loops around it are unrolled because a trip of a rolled one takes 320 cycles, whatever it loads (the
        // back edge waits until the copy has read its operands); unrolled it is as fast as 128 rows arrive from L2, 226 cycles.
        const auto load = [&](int kb, uint32_t sf_bytes) {
          ok = wait_or_abort(&smem->empty[stage], phase ^ 1u, smem, status);
          if (!ok) return false;
          const int x = kb * kTileKBytes;
          uint64_t* bar = &smem->full[stage];
          if (weight_side) {
            mbar_arrive_expect_tx(bar, kStWeightBytes + sf_bytes);
            if (it.down) tma_load_2d(smem->a[stage], &maps.w2, bar, x, it.expert * kHidden + it.n_tile * 128, read_once);
            else tma_load_3d(smem->a[stage], &maps.w13, bar, x, it.n_tile * 64, 2 * it.expert, read_once);
            bulk_load_1d(smem->sfa[stage], sf + static_cast<size_t>(kb) * kSfStageBytes, sf_bytes, bar, read_once);
          } else {
            mbar_arrive_expect_tx(bar, static_cast<uint32_t>(boxes * 8 * kTileKBytes) + sf_bytes);
            tma_load_2d(smem->b[stage], it.down ? &maps.down[boxes - 1] : &maps.up[boxes - 1], bar, x, row);
            bulk_load_1d(smem->sfb[stage], sf + static_cast<size_t>(kb) * kSfStageBytes, sf_bytes, bar);
          }
          ++issued;
          if (++stage == kStStages) {
            stage = 0;
            phase ^= 1u;
          }
          return true;
        };
        if (it.down) {
#pragma unroll
          for (int kb = 0; kb < kStDownKBlocks; ++kb)
            if (!load(kb, (kb + 1 == kStDownKBlocks ? kStDownLastMmas : 4) * kSfAtomBytes)) break;
        } else {
#pragma unroll kStLoadUnroll
          for (int kb = 0; kb < kStUpKBlocks; ++kb)
            if (!load(kb, kSfStageBytes)) break;
        }
      }
      if (!ok || smem->abort) {
        // unwinding: the copies already issued land before shared memory is given up
        const int pending = issued < kStStages ? issued : kStStages;
        for (int i = 0; i < pending; ++i) {
          if (--stage < 0) {
            stage = kStStages - 1;
            phase ^= 1u;
          }
          mbar_wait_bounded(&smem->full[stage], phase, 40000000ll);
        }
      }
    }
    __syncwarp();
  } else if (kFront && warp == kStSpareWarp) {
    // ---------------- what does not fit the ring ----------------
    // A CTA whose first item waits for the grid's quantised rows has its ring full of weights meanwhile, and nothing moves.  So
    // the rest of the item's weights and the start of the next item's are asked into L2: 100 tokens 502.6 -> 501.6 us a pass of six
    // layers, 150 tokens 346.9 -> 344.4 (four), 200 tokens 356.5 -> 352.5, 290 tokens 368.8 -> 364.  (From every CTA: 1 token 171 -> 177,
    // 64 tokens 647 -> 651, because there the ring is at work all the time; the whole next item: no better at 200, 657 at 64.)
    if (!self_first && cta < ups && elect_one()) {
#pragma unroll 1
      for (int n = 0; n < 2; ++n) {
        uint32_t word = smem->items[n];
        for (int spin = 0; !stream_announced(word, n) && spin < 200 && !smem->abort; ++spin) {
          __nanosleep(32);
          word = smem->items[n];
        }
        if (!stream_announced(word, n) || (word & (kStItemDown | kStItemEnd))) break;
        const StreamItem ahead = stream_unpack(word);
        const uint8_t* sf = p.w13_scales + static_cast<size_t>(ahead.expert * kUnitSlots + ahead.n_tile) * kStUpKBlocks * kSfStageBytes;
#pragma unroll 2
        for (int k = n ? 0 : kStStages; k < (n ? kStUpKBlocks - kStStages : kStUpKBlocks); ++k) {
          asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];" ::"l"(&maps.w13), "r"(k * kTileKBytes),
                       "r"(ahead.n_tile * 64), "r"(2 * ahead.expert)
                       : "memory");
          asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(sf + k * kSfStageBytes), "r"(kSfStageBytes) : "memory");
        }
      }
    }
    __syncwarp();
  } else if (warp == kStMmaWarp) {
    // ---------------- scale copies and MMAs, in one thread ----------------
    if (elect_one()) {
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      const uint32_t a_lo0 = (smem_u32(smem->a[0]) & 0x3ffffu) >> 4;
      const uint32_t b_lo0 = (smem_u32(smem->b[0]) & 0x3ffffu) >> 4;
      const uint32_t sfa_lo0 = (smem_u32(smem->sfa[0]) & 0x3ffffu) >> 4;
      const uint32_t sfb_lo0 = (smem_u32(smem->sfb[0]) & 0x3ffffu) >> 4;
      constexpr uint32_t hi_sf = (128u >> 4) | (1u << 14);  // 8 rows x 16 B, no swizzle
      bool landed = false;  // the next stage's bytes have been seen
      while (ok && stream_next(smem, taken, it)) {
        const int first = it.chunk * kStRows;
        int rows = smem->offsets[it.expert + 1] - smem->offsets[it.expert] - first;
        rows = rows > kStRows ? kStRows : rows;
        // E2M1 x E2M1, both K-major, UE4M3 scales, M = 128; N = the rows in multiples of 16
        const uint32_t descriptor = (1u << 7) | (1u << 10) | (static_cast<uint32_t>((rows + 15) / 16 * 2) << 17) |
                                    (static_cast<uint32_t>(kTileM >> 4) << 24);
        const uint32_t half = (first % kTileM) / 32;
        if (!wait_or_abort(&smem->acc_empty[acc], acc_phase ^ 1u, smem, status)) break;
        const uint32_t d = tmem_base + static_cast<uint32_t>(acc) * kStRows;
        // One K block, unrolled for the producers' reason.
        const auto multiply = [&](int kb, auto mmas, bool last) {
          if (!landed) ok = wait_or_abort(&smem->full[stage], phase, smem, status);
          if (!ok) return false;
          tc_fence_after_sync();
          const uint32_t sf = tmem_base + kStSfColumn + kStSfColumnsPerStage * stage;
          const uint32_t a_lo = a_lo0 + static_cast<uint32_t>(stage) * (kStWeightBytes >> 4);
          const uint32_t b_lo = b_lo0 + static_cast<uint32_t>(stage) * (kStTokenBytes >> 4);
          const uint32_t sf_offset = static_cast<uint32_t>(stage) * (kSfStageBytes >> 4);
          uint64_t* const empty = &smem->empty[stage];
          if (++stage == kStStages) {
            stage = 0;
            phase ^= 1u;
          }
          issue_sf_copies<mmas(), 128>(sf, sfa_lo0 + sf_offset, sfb_lo0 + sf_offset, hi_sf);
          stream_mmas<mmas()>(d, sf, sf + 16 + half, a_lo, b_lo, descriptor, kb != 0);
          landed = mbar_try_wait(&smem->full[stage], phase);
          tc_commit(empty);
          if (last) tc_commit(&smem->acc_full[acc]);
          return true;
        };
        if (it.down) {
#pragma unroll
          for (int kb = 0; kb < kStDownKBlocks - 1; ++kb)
            if (!multiply(kb, MmaCount<4>(), false)) break;
          if (ok) (void)multiply(kStDownKBlocks - 1, MmaCount<kStDownLastMmas>(), true);
        } else {
#pragma unroll kStMmaUnroll
          for (int kb = 0; kb < kStUpKBlocks; ++kb)
            if (!multiply(kb, MmaCount<4>(), kb + 1 == kStUpKBlocks)) break;
        }
        if (++acc == kStAccStages) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
    }
    __syncwarp();
  } else if (warp == kStClaimWarp) {
    // ---------------- claims ----------------
    // Two items ahead of the weight warp, which is busy with one for four microseconds: a claim takes one to two under
    // load, and weights that are asked for that much later are lost time (by the weight warp itself, 37 tokens took 3.4 us a
    // layer more).
    if (lane == 0) smem->first_mine = first_taken == 0;
    const StreamShares shares(smem->chunks, ctas);
    int turn = shares.fixed_turn(cta);
    bool exhausted = shares.up <= ctas, all_started = false, gave_up = false;
    int i = cta < shares.up ? 1 : 0;
#pragma unroll 1
    for (;; ++i) {
      if (!all_started) all_started = __all_sync(0xffffffffu, stream_open_first(sync, shares.firsts, lane) == shares.firsts);
      const long long start = clock64();
      gave_up = !__all_sync(0xffffffffu, i <= kStItemsAhead || stream_wait_begun(smem, i - kStItemsAhead + 1, status));
      int index = -1;  // the claimed item, if any
      if (!gave_up) {
        if (!exhausted) {
          if (lane == 0) index = shares.firsts + atomicAdd(sync + kStreamItemClaims, 1);
          index = __shfl_sync(0xffffffffu, index, 0);
          exhausted = index >= shares.up;
          turn = index - shares.up;
          if (exhausted) index = -1;
        }
        while (exhausted) {
          // the end, unless a CTA has not started: after a while its first item is this one's
          const int open = all_started ? shares.firsts : stream_open_first(sync, shares.firsts, lane);
          const uint32_t any = __ballot_sync(0xffffffffu, open < shares.firsts);
          if (any == 0) break;
          gave_up = __any_sync(0xffffffffu, smem->abort);
          if (gave_up) break;
          if (__any_sync(0xffffffffu, clock64() - start > kStRescueCycles)) {
            const int source = __ffs(static_cast<int>(any)) - 1;
            int was_taken = 1;
            if (lane == source) was_taken = atomicExch(sync + kStreamFirsts + open, 1);
            index = __shfl_sync(0xffffffffu, open, source);
            if (__shfl_sync(0xffffffffu, was_taken, source) == 0) break;
            index = -1;
          }
          __nanosleep(64);
        }
      }
      if (index < 0) break;
      if (lane == 0) stream_announce(smem, i, stream_word_of(index, false, smem));
      __syncwarp();
    }
    // The CTA's share of the w2 items but for its last ones; those of all shares lie in a pool.  SMs get through their weights at
    // different rates, and the CTAs that waited for the router's SMs start late.
    if (lane == 0) {
      StreamDownWalk<int> walk(shares, turn);
#pragma unroll 1
      for (; !gave_up; ++i) {
        gave_up = !stream_wait_begun(smem, i - kStItemsAhead, status);
        if (walk.asks()) {
          walk.next = atomicAdd(sync + kStreamDownClaims, 1);
          walk.after = atomicAdd(sync + kStreamDownClaims, 1);
        }
        const int item = walk.item();
        if (gave_up || item < 0) break;
        stream_announce(smem, i, stream_word_of(item, true, smem));
        if (walk.advance()) walk.after = atomicAdd(sync + kStreamDownClaims, 1);
      }
      if (!walk.answered()) smem->abort = 1;  // never: what waits for the answers
      stream_announce(smem, i, kStItemEnd);
    }
    __syncwarp();
  } else if (warp == kStPublishWarp) {
    // ---------------- publisher ----------------
    // Making an item's stores visible to the grid takes one to two microseconds under load.  The epilogue
    // warps leave that to this warp (their progress is a release to the CTA, the additions here extend it to
    // the GPU) and go on.
    int published = 0;
    bool rescue = kFront;
    long long start = clock64();
    for (;;) {
      int done = __reduce_min_sync(0xffffffffu, smem->progress[lane & (kStEpilogueWarps - 1)]);
      const int first_mine = __shfl_sync(0xffffffffu, smem->first_mine, 0);
      if (first_mine < 0) done = published;
      if (done == published) {
        const uint32_t next = smem->items[published % kStItems];
        const bool over = stream_announced(next, published) && (next & (kStItemDown | kStItemEnd));
        const long long idle = clock64() - start;
        if (__any_sync(0xffffffffu, over || smem->abort || idle > 2 * kWaitLimitCycles)) break;
        if (kFront && rescue && __any_sync(0xffffffffu, idle > kStRescueCycles)) {
          stream_rescue_tokens(p, smem, lane);
          rescue = false;
        }
        __nanosleep(64);
        continue;
      }
      __threadfence_block();
      __syncwarp();
      for (int i = published + lane; i < done; i += 32) {
        const uint32_t word = smem->items[i % kStItems];
        // (overwritten only where the claim warp gave up waiting; a first item that another CTA took is that CTA's to count)
        if (stream_announced(word, i) && (i > 0 || first_mine > 0))
          stream_count_release(p.plan.tile_ready + stream_unpack(word).expert, smem);
      }
      __syncwarp();
      published = done;
      if (lane == 0) smem->published = done;
      start = clock64();
    }
    if (lane == 0) smem->published = kStAllPublished;
  } else if (warp >= kStEpilogueWarp) {
    // ---------------- epilogue ----------------
    const int quarter = warp & 3;                        // the tensor-memory lanes this warp may read
    const int side = (warp - kStEpilogueWarp) >> 2;      // groups side, side + 2, ... of eight rows
    const int et = tid - kStEpilogueWarp * 32;
    int acc = 0, buffer = 0;
    uint32_t acc_phase = 0;
    while (stream_next(smem, taken, it)) {
      const int first = it.chunk * kStRows;
      const int row0 = smem->offsets[it.expert] + first;
      int rows = smem->offsets[it.expert + 1] - row0;
      rows = rows > kStRows ? kStRows : rows;
      const float alpha = it.down ? p.alpha2[it.expert] : p.alpha1[it.expert];
      const float multiplier = it.down ? 0.0f : p.in_scale_q2[it.expert];
      const bool ready = __all_sync(0xffffffffu, wait_or_abort(&smem->acc_full[acc], acc_phase, smem, status));
      uint32_t r[4][8];
      if (ready) {
        tc_fence_after_sync();
        const uint32_t source = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(acc) * kStRows;
#pragma unroll
        for (int g = 0; g < 4; ++g)
          tmem_load_32x8((side + 2 * g) * 8 < rows, source + (side + 2 * g) * 8, r[g]);
        tmem_load_wait(r);
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&smem->acc_empty[acc]);
      }
      if (++acc == kStAccStages) {
        acc = 0;
        acc_phase ^= 1u;
      }
      if (it.down) {
        if (!ready) break;
        __nv_bfloat16* out = p.routed + static_cast<size_t>(row0) * kHidden + it.n_tile * 128 + quarter * 32 + (lane & ~1);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int token0 = (side + 2 * g) * 8;
          if (token0 >= rows) break;
#pragma unroll
          for (int pair = 0; pair < 4; ++pair) {
            // even lanes finish token 2*pair, odd lanes token 2*pair + 1, two columns each
            const uint32_t keep = (lane & 1) ? r[g][2 * pair + 1] : r[g][2 * pair];
            const uint32_t other = __shfl_xor_sync(0xffffffffu, (lane & 1) ? r[g][2 * pair] : r[g][2 * pair + 1], 1);
            const float lo = __fmul_rn(alpha, __uint_as_float((lane & 1) ? other : keep));
            const float hi = __fmul_rn(alpha, __uint_as_float((lane & 1) ? keep : other));
            const int token = token0 + 2 * pair + (lane & 1);
            if (token < rows) *reinterpret_cast<uint32_t*>(out + static_cast<size_t>(token) * kHidden) = pack_bf16x2(lo, hi);
          }
        }
        continue;
      }
      // w13: 32 tokens at a time through the exchange tile
      const int column = et & 63;
      bool stop = false;
#pragma unroll
      for (int part = 0; part < kStRows / kStExchangeRows; ++part) {
        const int base = part * kStExchangeRows;
        if (base >= rows) break;
        if (ready) {
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            const int token0 = (side + 2 * g) * 8;  // within the part
            if (base + token0 < rows) {
#pragma unroll
              for (int t = 0; t < 8; ++t)
                smem->exchange[buffer][token0 + t][quarter * 32 + lane] =
                    __float2bfloat16_rn(__fmul_rn(alpha, __uint_as_float(r[2 * part + g][t])));
            }
          }
        } else {
          smem->left = 1;
        }
        // All eight warps meet here also when one of them gave up, and then leave together.
        named_barrier(2, kStEpilogueWarps * 32);
        if (smem->left) {
          stop = true;
          break;
        }
        // four tokens a thread (of 16 a round): their chains overlap, and the block's scale is worked out once
        // for every four lanes instead of in all sixteen
        for (int token = (et >> 6) * 4; token < kStExchangeRows; token += 16) {
          if (base + token >= rows) break;
          float v[4], maximum[4];
          bool in_table = true;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float up = __bfloat162float(smem->exchange[buffer][token + j][column]);
            const float gate = __bfloat162float(smem->exchange[buffer][token + j][64 + column]);
            const int index = erf_index((__float_as_uint(gate) >> 16) & 0x7fffu);
            in_table &= index >= 0 || base + token + j >= rows;  // rows past the end hold anything
            v[j] = __fmul_rn(gelu_from_erf(gate, smem->tables.erf_of[max(index, 0)]), up);
          }
          if (!in_table) {
#pragma unroll 1
            for (int j = 0; j < 4; ++j) {
              const float exact = __fmul_rn(gelu_of_bf16(__bfloat162float(smem->exchange[buffer][token + j][64 + column]), &smem->tables),
                                            __bfloat162float(smem->exchange[buffer][token + j][column]));
              if (j == 0) v[0] = exact;
              else if (j == 1) v[1] = exact;
              else if (j == 2) v[2] = exact;
              else v[3] = exact;
            }
          }
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 4; ++j) maximum[j] = fabsf(v[j]);
          // maxima over the block's sixteen lanes; lane 8a + 4b + c of the block is left with token 2a + b's
          const bool a = lane & 8, b = lane & 4;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const float received = __shfl_xor_sync(0xffffffffu, a ? maximum[j] : maximum[j + 2], 8);
            maximum[j] = fmaxf(a ? maximum[j + 2] : maximum[j], received);
          }
          float most = fmaxf(b ? maximum[1] : maximum[0], __shfl_xor_sync(0xffffffffu, b ? maximum[0] : maximum[1], 4));
          most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 2));
          most = fmaxf(fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 1)), 0.0f);  // (a block of NaN has scale zero)
          const uint32_t scale = encode_e4m3(gv_sixth(__fmul_rn(multiplier, most)));
          const float inverse = gv_scale_inverse_exact(multiplier) ? gv_scale_inverse(multiplier, scale, smem->tables.reciprocals)
                                                                   : scale_inverse_divided(multiplier, scale);
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = __fmul_rn(v[j], __shfl_sync(0xffffffffu, inverse, (lane & 16) | (4 * j)));
          // Columns 2c and 2c + 1 make byte c of a block's eight code bytes.  Even lanes go on with tokens 0 and 1, odd
          // ones with 2 and 3; then lane bit 1 picks one of the two, and lanes 0..3 of a block end with a token each.
          const bool odd = lane & 1, second = lane & 2;
          const float r0 = __shfl_xor_sync(0xffffffffu, odd ? v[0] : v[2], 1);
          const float r1 = __shfl_xor_sync(0xffffffffu, odd ? v[1] : v[3], 1);
          const uint32_t byte0 = odd ? encode_e2m1x2(r0, v[2]) : encode_e2m1x2(v[0], r0);
          const uint32_t byte1 = odd ? encode_e2m1x2(r1, v[3]) : encode_e2m1x2(v[1], r1);
          const uint32_t neighbour = __shfl_xor_sync(0xffffffffu, second ? byte0 : byte1, 2);
          uint32_t word = second ? neighbour | (byte1 << 8) : byte0 | (neighbour << 8);
          word |= __shfl_down_sync(0xffffffffu, word, 4) << 16;
          const uint32_t high = __shfl_down_sync(0xffffffffu, word, 8);
          const int block = it.n_tile * 4 + (column >> 4);
          const int coded = base + token + 2 * (lane & 1) + ((lane >> 1) & 1);
          if ((column & 15) < 4 && coded < rows)
            *reinterpret_cast<uint2*>(p.inter_codes + static_cast<size_t>(row0 + coded) * (kInter / 2) + block * 8) =
                make_uint2(word, high);
          const int scaled_token = base + token + 2 * ((lane >> 3) & 1) + ((lane >> 2) & 1);
          if ((lane & 3) == 0 && scaled_token < rows)
            p.inter_scales[static_cast<size_t>(smem->scale_rows[it.expert]) * (kInter / 16) +
                           sf_offset(first + scaled_token, block, kInter / 16)] = static_cast<uint8_t>(scale);
        }
        buffer ^= 1;
      }
      if (stop) break;
      __syncwarp();
      if (lane == 0) {
        __threadfence_block();
        smem->progress[warp - kStEpilogueWarp] = taken;
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == kStMmaWarp) {
    tc_fence_after_sync();
    __syncwarp();
    tmem_dealloc(tmem_base, kStTmemColumns);
  }
  // The CTA that finishes last puts the counters back for the next launch.  No fence is needed in front of this: all waits of the CTA lie before
  // it, and whatever the CTA has added to a counter has arrived, also where a wait ran out: the answer of every claim and every count has been
  // looked at.  (With a fence, which waits for the CTA's last rows to arrive, 0.5 us a layer more: 1 token 20.75 and 20.2, 64 tokens 74.9 and 74.3.)
  if (tid == 0) smem->last = atomicAdd(sync + kStreamFinished, 1) == ctas - 1;
  __syncthreads();
  if (smem->last) {
    if (tid < kExperts) p.plan.tile_ready[tid] = 0;
    for (int i = tid; i < kStreamSyncInts; i += kStThreads) sync[i] = 0;
  }
}

StreamParams make_params(const StreamOperands& op, const RoutePlan& plan) {
  StreamParams p{};
  p.plan = plan;
  p.w13_scales = op.w13_scales;
  p.w2_scales = op.w2_scales;
  p.input_scales = op.input_scales;
  p.inter_codes = op.inter_codes;
  p.inter_scales = op.inter_scales;
  p.routed = static_cast<__nv_bfloat16*>(op.routed);
  p.alpha1 = op.alpha1;
  p.alpha2 = op.alpha2;
  p.in_scale_q2 = op.in_scale_q2;
  return p;
}

StreamMaps make_maps(const StreamOperands& op) {
  StreamMaps maps;
  maps.w13 = op.map_w13;
  maps.w2 = op.map_w2;
  for (int i = 0; i < kStRows / 8; ++i) {
    maps.up[i] = op.map_up[i];
    maps.down[i] = op.map_down[i];
  }
  return maps;
}

}  // namespace

static_assert(kStOwnTokens == 2 && kExperts <= 255, "the front's indexes");
static_assert(kStRows / 8 == kStreamBoxes, "one map per box height");
static_assert(kExperts + kStreamMaxTokens * kTopK / kStRows <= kStMaxChunks, "chunk list");

bool stream_layer_fits(int tokens, int sm_count) {
  return tokens <= kStFrontTokens && tokens <= sm_count * kStOwnTokens;
}


int prepare_stream_experts() {
  cudaError_t e = cudaFuncSetAttribute(stream_experts_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(kStSmemBytes));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(stream_experts_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(kStSmemBytes));
  return static_cast<int>(e);
}

void launch_stream_experts(const StreamOperands& op, const RoutePlan& plan, int sm_count, cudaStream_t stream) {
  launch_chained(stream_experts_kernel<false>, dim3(sm_count < kStreamMaxCtas ? sm_count : kStreamMaxCtas), dim3(kStThreads), kStSmemBytes, stream, make_maps(op),
                 make_params(op, plan));
}

void launch_stream_layer(const StreamOperands& op, const RoutePlan& plan, const void* input_bf16, const int* expert_ids,
                         const float* in_scale_q1, uint8_t* packed, uint8_t* scales, int tokens, int sm_count,
                         cudaStream_t stream) {
  StreamParams p = make_params(op, plan);
  p.input = static_cast<const __nv_bfloat16*>(input_bf16);
  p.expert_ids = expert_ids;
  p.in_scale_q1 = in_scale_q1;
  p.packed = packed;
  p.scales = scales;
  p.tokens = tokens;
  launch_chained(stream_experts_kernel<true>, dim3(sm_count < kStreamMaxCtas ? sm_count : kStreamMaxCtas), dim3(kStThreads), kStSmemBytes, stream, make_maps(op), p);
}

}  // namespace gv
