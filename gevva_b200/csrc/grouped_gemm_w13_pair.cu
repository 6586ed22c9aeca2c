// Fused w13 GEMM + GeGLU + NVFP4 requantisation run by CTA pairs, weights on the MMA's M side.
//
// What bounds it.  One K block of 256 elements of a 128 x 256 tile costs 512 tensor-pipe cycles, but in the
// one-CTA kernel (grouped_gemm.cu) shared memory has to take in 54 KiB and give the MMAs 48 KiB for it: 800
// cycles.  Here a CTA pair (tcgen05 cta_group::2, M = 256) holds 256 weight rows, 128 per CTA, against up to 256
// token rows of one expert on the N side, half of them loaded by each CTA: at most 38 KiB in and 38 out, scales included.  And because
// the tokens sit on N, which may be any multiple of 16, a group of 200 rows is one item and not two 128-row tiles.
// An item is 11 K blocks, each of four MMAs of N / 2 tensor cycles (39 at least) and eight or twelve scale copies.  Issuing those takes one
// thread some 300 cycles a K block, and beside the epilogue's warps on its scheduler more, so a narrow item costs nearly what one of
// 170 rows does: chunks are as wide as the MMA allows.  (That is not the whole of it: 4096 tokens' 1176 items come to 35 us so, and their operands to 54 us of
// HBM and 40 of L2 time, but the kernel takes 77 to 85; an item of 256 rows takes some 9300 cycles, 5632 of them the tensor pipe's.  What the
// issuing thread waits for in the others has not been counted.)  Chunks of 208 rows and a loop of the whole warp -> this (us, alone): 4096 tokens 96.5 -> 88.2,
// of uneven loads 94.2 -> 87.4, 16384 290 -> 269; a whole layer of 700 tokens 109.5 -> 108.5, 4096 254 -> 245, 16384 795 -> 770.
// Beside large batches the clock drops to 1.35 GHz under the power limit (this kernel repeated for seconds at 4096 tokens).
// Alone (us, one-CTA kernel -> the first form of this one; uniform routing): 53.1 -> 53.2 at 1024 tokens, 63.9 -> 58.9 at 2048,
// 83.5 -> 70 at 3000, 97 -> 95 at 4096, 172 -> 151 at 8192, 330 -> 293 at 16384.
//
// Work.  A chunk is up to 256 consecutive rows of an expert; one with more is cut into as few chunks as that takes, of 192 or 256 rows but for the last, so that a
// chunk's scales start at a 64-row boundary of their 128-row blocks.  The intermediate width 704 is cut into 11 units
// of 64 columns; a CTA computes one unit as 128 MMA rows, the unit's up and gate rows interleaved so that a thread
// of the epilogue finds both of a column in its registers (see there; the order costs nothing: it is a
// five-dimensional view of the same weights, and the scales have a re-tiled copy made at runner creation).  A work
// item is (chunk, two units); the second CTA of the sixth item has no unit (its weight scales are zero and its
// results are dropped).
//
// Protocol.  Two TMA producers in each CTA (weight side, token side) fill a ring of six stages (where some chunk has more than 208 rows,
// the tokens' has five: 227 KB of shared memory hold no more),
// all loads of both CTAs complete on the `full` barrier of the first CTA (tensor-map loads in
// their cta_group::2 form, no multicast; the scale atoms travel through tensor maps too).  There
// the MMA thread copies the scale atoms of a landed stage into tensor memory, issues four MMAs
// (copies and MMAs of one thread execute in order) and commits to `empty` of both CTAs.  Two accumulators, so that the
// eight epilogue warps of each CTA work on one item while the next is computed; two of 256 columns do not fit beside the scales, so such two have 48 in common,
// which the epilogue reads first and releases by themselves (an item waits for that where the two would meet).  The items of a pair are worked out once, by all threads.  A step of the
// epilogue (32 tokens, 1800 cycles) took 3500 more when a gate was zero or tiny, which 3 to 25 % of the steps have: such gates now take the
// polynomial's first interval in line (of the accumulators' columns that no row owns, too).  With that, pairs of values to an instruction and the next
// accumulators fetched ahead: 700 tokens 53.2 -> 51.6 us, 4096 88.2 -> 85.2, 16384 269 -> 263; a layer of 700 tokens 108.5 -> 107.4,
// of 4096 245 -> 240.  (With the accumulator transposed
// through shared memory by sixteen warps that traffic bounded the kernel, 107 us at 4096 tokens; with this epilogue
// twelve warps are as fast as eight and sixteen 10 % slower.)  Every wait is bounded.
#include "gv_common.cuh"
#include "gv_cta_pair.cuh"
#include "gv_gemm_parts.cuh"
#include "gv_launchers.h"

namespace gv {

namespace {

constexpr int kWpStages = 6;                   // K blocks of weights in flight
constexpr int kWpParts = 2;                    // epilogue warps a block of 16 columns
constexpr int kWpTokenWarp = 0, kWpMmaWarp = 1, kWpEpilogueWarp = 2, kWpWeightWarp = kWpEpilogueWarp + 4 * kWpParts;
constexpr int kWpThreads = (kWpWeightWarp + 1) * 32;
constexpr uint32_t kWpTmemColumns = 512;
constexpr int kWpRows = 256;                   // rows of a chunk at most (MMA N)
constexpr int kWpAccStages = 2;
// Tensor memory: two accumulators, the first from column 0 on, the second up to where the scales begin, so that two of more than
// kWpSfColumn columns together have their inner ends in common; then one K block's scales, per MMA j: weights at +12j, the chunk's two
// 128-row blocks at +12j+4 and +12j+8.
constexpr uint32_t kWpSfColumn = kWpTmemColumns - 48;
static_assert(2 * kWpRows - kWpSfColumn <= 2 * 32 - 16, "shared columns: in the first step of the two parts of the epilogue");
// Token rows in flight: six K blocks of chunks of up to kWpNarrow rows or, where some chunk of the batch has more, five of up to kWpRows.
constexpr int kWpNarrow = 208;
constexpr int kWpTokenBytes = kWpNarrow / 2 * kTileKBytes;     // 13 KiB
constexpr int kWpWideTokenBytes = kWpRows / 2 * kTileKBytes;   // 16 KiB
constexpr int kWpWideStages = 5;
constexpr int kWpTokenRing = kWpWideStages * kWpWideTokenBytes;
static_assert(kWpStages * kWpTokenBytes <= kWpTokenRing, "token ring");
constexpr int kWpTileBytes = 128 * kTileKBytes;  // 16 KiB
constexpr int kWpUnits = kInter / 64;            // 11
constexpr int kWpUnitSlots = 12;                 // the re-tiled scales carry a twelfth, all-zero unit
constexpr int kWpItemsPerChunk = kWpUnitSlots / 2;
constexpr int kWpTable = 512;                    // rounds whose items are worked out once (131072 tokens on 148 SMs have 343)

struct alignas(1024) WpSmem {
  uint8_t w[kWpStages][kWpTileBytes];          // this CTA's 64 up + 64 gate weight rows
  uint8_t x[kWpTokenRing];                     // this CTA's half of the chunk's token rows
  uint8_t sfw[kWpStages][kSfStageBytes];       // scales of this CTA's weight rows
  uint8_t sfx[kWpStages][2 * kSfStageBytes];   // scales of the chunk's one or two 128-row blocks
  uint64_t full[kWpStages];    // leader: the stage's bytes have landed in both CTAs
  uint64_t empty[kWpStages];   // both CTAs: the MMAs that read the stage have completed
  uint64_t acc_full[kWpAccStages];   // both CTAs: the item's accumulator is complete
  uint64_t acc_empty[kWpAccStages];  // leader: both CTAs' epilogues have copied the accumulator out
  uint64_t acc_shared[kWpAccStages]; // leader: ... or the columns of it that the other accumulator may have in common
  uint64_t table;                    // `items` is there
  uint32_t tmem_base;
  volatile int abort;
  // group geometry, by expert: first row, first scale row, chunks before it
  int offsets[kExperts + 1], scale_rows[kExperts + 1], chunks[kExperts + 1], scan[4];
  uint32_t items[kWpTable];    // this pair's items but the first, see wp_pack
  GegluTables tables;
};

constexpr size_t kWpSmemBytes = sizeof(WpSmem) + 1024;
static_assert(kWpSmemBytes <= 232448, "shared memory budget");

// The 128 weight rows of a unit in the kernel's order: see make_w13_fragment_map (moe_abi.cu).
__device__ __forceinline__ void wp_load_weights(void* smem_dst, const void* tensor_map, uint32_t barrier, int x, int block) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2"
      " [%0], [%1, {%2, %3, %3, %3, %4}], [%5];" ::"r"(smem_u32(smem_dst)),
      "l"(tensor_map), "r"(x), "r"(0), "r"(block), "r"(barrier)
      : "memory");
}

// Scale copies of one K block (four MMAs of K = 64) for both CTAs: per MMA j the atom of the
// weight rows and the atoms of the chunk's one or two 128-row blocks of tokens.
__device__ __forceinline__ void wp_issue_sf_copies(uint32_t tmem_sf, uint32_t sfw_lo, uint32_t sfx_lo, bool two_blocks) {
  constexpr uint32_t hi_sf = (128u >> 4) | (1u << 14);                // 8 rows x 16 B, no swizzle
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j) {
    pair_copy_sf(tmem_sf + 12 * j, hi_sf, sfw_lo + 32 * j);
    pair_copy_sf(tmem_sf + 12 * j + 4, hi_sf, sfx_lo + 32 * j);
  }
  if (two_blocks)
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j) pair_copy_sf(tmem_sf + 12 * j + 8, hi_sf, sfx_lo + 128 + 32 * j);
}

__device__ __forceinline__ void wp_issue_mmas(uint32_t tmem_acc, uint32_t tmem_sf, uint32_t shift, uint32_t w_lo, uint32_t x_lo,
                                              uint32_t idesc, uint32_t accumulate) {
  constexpr uint32_t hi_ab = (1024u >> 4) | (1u << 14) | (2u << 29);  // 8 rows x 128 B, 128B swizzle
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j)
    pair_mma(tmem_acc, hi_ab, w_lo + 2 * j, x_lo + 2 * j, idesc, tmem_sf + 12 * j, tmem_sf + 12 * j + 4 + shift,
           j == 0 ? accumulate : 1u);
}

// 16 lanes x 32 columns: register 4g + i holds columns 8g + 2t + (i & 1) of row lane/4 + 8 * (i / 2).  Nothing unless `wanted`,
// which is the same in the whole warp; the registers are undefined then.
__device__ __forceinline__ void wp_load_16x32(bool wanted, uint32_t tmem_address, uint32_t (&r)[16]) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %17, 0;\n\t"
      "@p tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t}"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(tmem_address), "r"(static_cast<uint32_t>(wanted))
      : "memory");
}

__device__ __forceinline__ void wp_arrive(uint64_t* bar, bool is_leader) {
  if (is_leader) mbar_arrive(bar);
  else pair_arrive_remote(bar, 0);
}

struct WpItem {
  int expert;
  int first;     // first 128-row scale tile of the chunk
  int shift;     // tensor-memory columns (of 32 rows) by which the chunk starts inside that tile: 0 or 2
  int local;     // first row of the chunk within the expert
  int row0;      // first sorted row of the chunk
  int valid;     // rows of the chunk, 1..256
  int n;         // MMA N: valid rounded up to 16
  int unit_pair; // 0..5
};

// Chunks of an expert: as few as cover its rows, and all but the last of the same multiple of 64 (192 or 256), so that a chunk's scales
// start at a column of its first scale tile's atom and end within the next tile's.
__host__ __device__ __forceinline__ int wp_chunks_of(int rows) { return (rows + kWpRows - 1) / kWpRows; }
__host__ __device__ __forceinline__ int wp_chunk_rows(int rows) {
  const int chunks = wp_chunks_of(rows);
  return chunks <= 1 ? rows : (rows + 64 * chunks - 1) / (64 * chunks) * 64;
}

// An item in a word: expert, unit pair, N / 16 (never zero), first row / 64; zero: none.
__device__ __noinline__ uint32_t wp_pack(const WpSmem* smem, int round) {
  // Snake order over the pairs of the grid: the unit pairs of a chunk go to neighbouring
  // clusters, which then read the same token rows from L2 at about the same time.
  const int slots = static_cast<int>(gridDim.x) >> 1;
  const int mine = static_cast<int>(blockIdx.x) >> 1;
  const int slot = (round & 1) ? slots - 1 - mine : mine;
  const int index = round * slots + slot;
  const int chunk = index / kWpItemsPerChunk;
  if (chunk >= smem->chunks[kExperts]) return 0;
  int expert = 0;  // the last expert with chunks[expert] <= chunk
#pragma unroll
  for (int step = kExperts / 2; step; step >>= 1)
    if (smem->chunks[expert + step] <= chunk) expert += step;
  const int rows = smem->offsets[expert + 1] - smem->offsets[expert];
  const int chunk_rows = wp_chunk_rows(rows);
  const int local = (chunk - smem->chunks[expert]) * chunk_rows;
  const int valid = rows - local < chunk_rows ? rows - local : chunk_rows;
  return static_cast<uint32_t>(expert) | static_cast<uint32_t>(index - chunk * kWpItemsPerChunk) << 7 |
         static_cast<uint32_t>((valid + 15) >> 4) << 10 | static_cast<uint32_t>(local >> 6) << 15;
}

// Behind a wait for `table` but for the first round, whose loads do not wait for it.  (Rounds past the table are those of the largest batches on a
// few SMs.)
__device__ __forceinline__ uint32_t wp_word(const WpSmem* smem, int round) {
  return round != 0 && round < kWpTable ? smem->items[round] : wp_pack(smem, round);
}

// False if there is none; then there is none in any later round either.
__device__ __forceinline__ bool wp_item(const WpSmem* smem, int round, WpItem& item) {
  const uint32_t word = wp_word(smem, round);
  if (word == 0) return false;
  item.expert = static_cast<int>(word & 127u);
  item.unit_pair = static_cast<int>((word >> 7) & 7u);
  item.n = static_cast<int>((word >> 10) & 31u) << 4;
  item.local = static_cast<int>(word >> 15) << 6;
  item.row0 = smem->offsets[item.expert] + item.local;
  item.first = (smem->scale_rows[item.expert] + item.local) / kTileM;
  item.shift = (item.local & (kTileM - 1)) >> 5;
  item.valid = min(item.n, smem->offsets[item.expert + 1] - item.row0);
  return true;
}

__device__ __forceinline__ bool wp_two_blocks(const WpItem& item) { return item.shift * 32 + item.n > kTileM; }

struct WpTokenMaps {
  CUtensorMap rows[kW13PairBoxes];   // boxes of 8, 16, ... 128 token rows x 128 bytes
};

constexpr int kWpKBlocks = kHidden / 2 / kTileKBytes;   // 11

struct WpParams {
  const float* alpha;          // [experts] g1 output scale
  uint8_t* next_codes;         // [row capacity, 352] w2 operand codes
  uint8_t* next_scales;        // scale regions of the w2 operand
  const float* next_scale_q;   // [experts] g2.input_scale_quant
  const int* expert_offsets;
  const int* scale_row_offsets;
  int* status;
  bool early_weights;
};

// The leader's MMA thread.  In one thread, with running addresses and a look at the next stage's barrier ahead of the issue; not unrolled over the stages,
// which takes 20 to 80 cycles off a K block when the code is there, but every launch of a layer fetches its code anew: 34 KB more of it
// cost layers of 700 to 2500 tokens 3 us.
__device__ __forceinline__ void wp_issue(WpSmem* smem, uint32_t tmem_base, bool wide, int* status) {
  const uint32_t w_lo0 = (smem_u32(smem->w[0]) & 0x3ffffu) >> 4, x_lo0 = (smem_u32(smem->x) & 0x3ffffu) >> 4;
  const uint32_t sfw_lo0 = (smem_u32(smem->sfw[0]) & 0x3ffffu) >> 4, sfx_lo0 = (smem_u32(smem->sfx[0]) & 0x3ffffu) >> 4;
  const uint32_t token_step = (wide ? kWpWideTokenBytes : kWpTokenBytes) >> 4;
  const uint32_t x_end = x_lo0 + (wide ? kWpWideStages : kWpStages) * token_step;
  const uint32_t tmem_sf = tmem_base + kWpSfColumn;
  uint32_t phase = 0, acc_phase = 0, acc = 0, word = wp_word(smem, 0), next = 0;
  uint32_t x_lo = x_lo0, stage = 0;
  uint32_t before = 0;   // N / 16 of the item before
  bool landed = false;   // the next stage's bytes have been seen
  for (int round = 0; word != 0; ++round, word = next) {
    if (round == 0 && !wait_or_abort(&smem->table, 0, smem, status)) return;
    next = wp_word(smem, round + 1);
    const uint32_t n16 = (word >> 10) & 31u;
    const uint32_t shift = (word >> 14) & 2u;  // an odd multiple of 64 rows into the expert: two columns of 32 rows into its scale tile
    const bool two_blocks = shift * 2 + n16 > 8;
    // E2M1 x E2M1, both K-major, UE4M3 scales; N at [17,23) in units of 8, M = 256 at [24,29) in units of 16
    const uint32_t idesc = (1u << 7) | (1u << 10) | (n16 << 18) | (static_cast<uint32_t>(256 >> 4) << 24);
    const uint32_t tmem_acc = tmem_base + (acc == 0 ? 0 : kWpSfColumn - 16 * n16);
    if (!wait_or_abort(&smem->acc_empty[acc], acc_phase ^ 1u, smem, status)) return;
    if (before + n16 > kWpSfColumn / 16 && !wait_or_abort(&smem->acc_shared[acc ^ 1u], acc == 0 ? acc_phase ^ 1u : acc_phase, smem, status)) return;
    before = n16;
#pragma unroll 1
    for (uint32_t kb = 0; kb < kWpKBlocks; ++kb) {
      if (!landed && !wait_or_abort(&smem->full[stage], phase, smem, status)) return;
      tc_fence_after_sync();
      const uint32_t w_lo = w_lo0 + stage * (kWpTileBytes >> 4);
      const uint32_t sfw_lo = sfw_lo0 + stage * (kSfStageBytes >> 4), sfx_lo = sfx_lo0 + stage * (2 * kSfStageBytes >> 4);
      uint64_t* const empty = &smem->empty[stage];
      if (++stage == kWpStages) {
        stage = 0;
        phase ^= 1u;
      }
      landed = mbar_try_wait(&smem->full[stage], phase);
      // copies and MMAs of one thread execute in order in the tensor pipe, so one set of scale
      // columns serves every K block
      wp_issue_sf_copies(tmem_sf, sfw_lo, sfx_lo, two_blocks);
      wp_issue_mmas(tmem_acc, tmem_sf, shift, w_lo, x_lo, idesc, kb);
      pair_commit_both(empty);   // both CTAs may refill the stage
      x_lo += token_step;
      if (x_lo == x_end) x_lo = x_lo0;
    }
    pair_commit_both(&smem->acc_full[acc]);
    if (++acc == kWpAccStages) {
      acc = 0;
      acc_phase ^= 1u;
    }
  }
}

__global__ void __launch_bounds__(kWpThreads, 1)
w13_geglu_pair_kernel(const __grid_constant__ WpTokenMaps map_x, const __grid_constant__ CUtensorMap map_w,
                      const __grid_constant__ CUtensorMap map_x_sf, const __grid_constant__ CUtensorMap map_w_sf,
                      const WpParams p) {
  extern __shared__ uint8_t smem_raw[];
  WpSmem* smem = reinterpret_cast<WpSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_cta_rank();   // 0 = leader
  const bool is_leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kWpStages; ++s) {
      mbar_init(&smem->full[s], 2);   // the leader's two producers each announce both CTAs' byte count
      mbar_init(&smem->empty[s], 1);
    }
    for (int b = 0; b < kWpAccStages; ++b) {
      mbar_init(&smem->acc_full[b], 1);
      mbar_init(&smem->acc_empty[b], 2 * 4 * kWpParts);  // the epilogue warps of both CTAs
      mbar_init(&smem->acc_shared[b], 2 * 4 * kWpParts);
    }
    mbar_init(&smem->table, 4 * kWpParts);
    smem->abort = 0;
    fence_barrier_init();
    prefetch_tensor_map(&map_w);
    prefetch_tensor_map(&map_x_sf);
    prefetch_tensor_map(&map_w_sf);
  }
  // Both CTAs run and their barriers exist before either touches the other's tensor memory or arrives there.
  __syncwarp();
  cluster_sync_all();
  if (warp == kWpMmaWarp) pair_tmem_alloc(&smem->tmem_base, kWpTmemColumns);  // the whole tensor memory
  load_geglu_tables(&smem->tables);
  __syncthreads();
  fill_geglu_tables(&smem->tables);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = smem->tmem_base;
  // The plan and the weights may come from before the previous kernel: see W13PairOperands::early_weights.
  if (!p.early_weights) grid_dependency_wait();

  bool wide = false;  // some chunk has more than kWpNarrow rows
  if (warp < 4) {
    // thread = expert: chunks before it
    const int e = threadIdx.x;
    const int row = p.expert_offsets[e], next_row = p.expert_offsets[e + 1];
    const int own = wp_chunks_of(next_row - row);
    wide = wp_chunk_rows(next_row - row) > kWpNarrow;
    int inclusive = own;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
      const int other = __shfl_up_sync(0xffffffffu, inclusive, offset);
      if (lane >= offset) inclusive += other;
    }
    if (lane == 31) smem->scan[warp] = inclusive;
    smem->offsets[e] = row;
    smem->scale_rows[e] = p.scale_row_offsets[e];
    if (e == kExperts - 1) smem->offsets[kExperts] = next_row;
    named_barrier(5, 128);
    for (int w = 0; w < warp; ++w) inclusive += smem->scan[w];
    smem->chunks[e] = inclusive - own;
    if (e == kExperts - 1) smem->chunks[kExperts] = inclusive;
  }
  wide = __syncthreads_or(wide);
  if (warp != kWpWeightWarp) {
    grid_dependency_wait();
    grid_launch_dependents();  // after the wait: whoever starts now may read what came before this kernel
  }

  if (warp == kWpTokenWarp || warp == kWpWeightWarp) {
    // ---------------- TMA producers (one warp for each side in each CTA) ----------------
    const bool weight_side = warp == kWpWeightWarp;
    int stage = 0;
    uint32_t phase = 0;
    int issued = 0;
    bool ok = true;
    // The token side may be fewer K blocks ahead; what it waits for is then a younger stage's MMAs.
    const int token_stages = wide ? kWpWideStages : kWpStages, token_bytes = wide ? kWpWideTokenBytes : kWpTokenBytes;
    int wait_stage = weight_side ? 0 : kWpStages - token_stages, slot = 0;
    uint32_t wait_phase = 1;
    WpItem item;
    for (int round = 0; ok && wp_item(smem, round, item); ++round) {
      const int unit = 2 * item.unit_pair + static_cast<int>(rank);
      const bool unit_exists = unit < kWpUnits;
      const int half = item.n >> 1;                            // token rows per CTA, a multiple of 8
      const int token_row = item.row0 + static_cast<int>(rank) * half;
      const bool second_exists = 2 * item.unit_pair + 1 < kWpUnits;
      // Per K block and CTA: the unit's weight rows and their scales (2 KiB), or the token rows and the scales (2 KiB each) of the
      // one or two 128-row blocks that the chunk has rows in.
      const bool two_blocks = wp_two_blocks(item);
      const uint32_t both_bytes = weight_side ? 2 * kSfStageBytes + kWpTileBytes + (second_exists ? kWpTileBytes : 0)
                                              : 2 * ((two_blocks ? 2 : 1) * kSfStageBytes + static_cast<uint32_t>(half) * kTileKBytes);
      const CUtensorMap* token_map = &map_x.rows[(half >> 3) - 1];
      const int w_sf_row = ((item.expert * kWpUnitSlots + unit) * kWpKBlocks) * 4;
      for (int kb = 0; kb < kWpKBlocks; ++kb) {
        ok = __all_sync(0xffffffffu, wait_or_abort(&smem->empty[wait_stage], wait_phase, smem, p.status));
        if (!ok) break;
        if (elect_one()) {
          const int x = kb * kTileKBytes;
          const uint32_t bar = is_leader ? smem_u32(&smem->full[stage])
                                         : cluster_map_shared(smem_u32(&smem->full[stage]), 0);
          if (is_leader) mbar_arrive_expect_tx(&smem->full[stage], both_bytes);
          if (weight_side) {
            if (unit_exists) wp_load_weights(smem->w[stage], &map_w, bar, x, item.expert * (kW13Out / 16) + unit * 4);
            pair_load(smem->sfw[stage], &map_w_sf, bar, 0, w_sf_row + 4 * kb);
          } else {
            pair_load(smem->x + slot * token_bytes, token_map, bar, x, token_row);
            pair_load_3d(smem->sfx[stage], &map_x_sf, bar, 0, 4 * kb, item.first);
            if (two_blocks) pair_load_3d(smem->sfx[stage] + kSfStageBytes, &map_x_sf, bar, 0, 4 * kb, item.first + 1);
          }
        }
        __syncwarp();
        ++issued;
        if (++stage == kWpStages) {
          stage = 0;
          phase ^= 1u;
        }
        if (++wait_stage == kWpStages) {
          wait_stage = 0;
          wait_phase ^= 1u;
        }
        if (++slot == token_stages) slot = 0;
      }
      if (round == 0 && ok) ok = __all_sync(0xffffffffu, wait_or_abort(&smem->table, 0, smem, p.status));
    }
    if (!ok && lane == 0 && is_leader) {
      // Unwinding: let the copies already issued (by either CTA) land before shared memory is
      // given up; the second CTA stays resident until the cluster barrier at the end.
      const int pending = issued < kWpStages ? issued : kWpStages;
      int s = stage;
      uint32_t ph = phase;
      for (int i = 0; i < pending; ++i) {
        if (--s < 0) {
          s = kWpStages - 1;
          ph ^= 1u;
        }
        mbar_wait_bounded(&smem->full[s], ph, 40000000ll);
      }
    }
  } else if (warp == kWpMmaWarp) {
    // ---------------- leader: scale copies and MMAs for both CTAs, in one thread ----------------
    if (is_leader && elect_one()) {
      wp_issue(smem, tmem_base, wide, p.status);
    }
    __syncwarp();
  } else {
    // ---------------- epilogue: eight warps in each CTA ----------------
    // A warp may touch only the tensor-memory lanes 32*(warp%4)..+31: one block of 16 intermediate columns,
    // 16b + 2i + o being the up row of lane 16o + i and the gate row of lane 16o + 8 + i.  In the 16x256b layout a
    // thread holds rows lane/4 and lane/4 + 8, so up and gate of columns 2i and 2i + 1 (i = lane / 4), for eight of
    // 32 tokens: GeGLU needs no exchange, a block's maximum is one over the eight lanes of equal lane % 4, and the
    // thread's two codes are byte i of the block's eight.  Three steps of exchange leave lane i with the maximum,
    // and then the code bytes, of the i-th of its eight tokens.
    const int block = warp & 3;
    const int part = (warp - kWpEpilogueWarp) >> 2;
    const bool a = lane & 16, b = lane & 8, c = lane & 4;
    const uint32_t keep_b = b ? 0x7632u : 0x5410u, send_b = b ? 0x5410u : 0x7632u;
    const uint32_t keep_c = c ? 0x7531u : 0x6420u, send_c = c ? 0x6420u : 0x7531u;
    const uint32_t low_word = b ? 0x4062u : 0x6240u, high_word = b ? 0x5173u : 0x7351u;
    const int own_token = 8 * (lane >> 3) + 2 * (lane & 3) + ((lane >> 2) & 1);  // of the 32: the (lane / 4)-th of the thread's
    constexpr int groups = kInter / 16;
    for (int round = threadIdx.x - 32 * kWpEpilogueWarp; round < kWpTable; round += 32 * 4 * kWpParts) smem->items[round] = wp_pack(smem, round);
    __syncwarp();
    if (lane == 0) mbar_arrive(&smem->table);
    const bool there = __all_sync(0xffffffffu, wait_or_abort(&smem->table, 0, smem, p.status));
    int acc = 0;
    uint32_t acc_phase = 0;
    uint32_t even[16], odd[16];
    WpItem item;
    for (int round = 0; there && wp_item(smem, round, item); ++round) {
      const int unit = 2 * item.unit_pair + static_cast<int>(rank);
      const int steps = unit < kWpUnits ? (item.valid + 31) >> 5 : 0;  // of 32 tokens, dealt to the two warps of a block
      const float alpha = p.alpha[item.expert];
      const unsigned long long alphas = two(alpha, alpha);
      const float multiplier = p.next_scale_q[item.expert];
      if (!__all_sync(0xffffffffu, wait_or_abort(&smem->acc_full[acc], acc_phase, smem, p.status))) break;
      tc_fence_after_sync();
      const uint32_t tmem_rows = tmem_base + (static_cast<uint32_t>(block * 32) << 16) + (acc == 0 ? 0u : kWpSfColumn - static_cast<uint32_t>(item.n));
      uint8_t* const scales = p.next_scales + static_cast<size_t>(smem->scale_rows[item.expert]) * groups;
      // from the end that the two accumulators share; the next step's accumulators are fetched under a step's arithmetic
      int turn = (part + round) % kWpParts;
      bool first = true;
      const auto load = [&](bool wanted, int turn_of_load) {
        const int step = acc == 0 ? steps - 1 - turn_of_load : turn_of_load;
        wp_load_16x32(wanted, tmem_rows + 32 * step, even);
        wp_load_16x32(wanted, tmem_rows + (16u << 16) + 32 * step, odd);
      };
      load(turn < steps, turn);
      tmem_load_wait(even, odd);
#pragma unroll 1
      for (;;) {
        const bool last = turn + kWpParts >= steps;
        if (first || last) {
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) {
            if (first) wp_arrive(&smem->acc_shared[acc], is_leader);
            if (last) wp_arrive(&smem->acc_empty[acc], is_leader);
          }
          first = false;
        }
        if (turn >= steps) break;
        const int token = 32 * (acc == 0 ? steps - 1 - turn : turn) + own_token;
        // bf16(alpha * acc), columns 2i and 2i + 1 of token k = 2g + s (8g + 2 (lane % 4) + s of the 32)
        uint32_t up[8], gate[8];
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          const int r = 2 * k;
          const unsigned long long u0 = mul2(alphas, two(__uint_as_float(even[r]), __uint_as_float(even[r + 1])));
          const unsigned long long u1 = mul2(alphas, two(__uint_as_float(odd[r]), __uint_as_float(odd[r + 1])));
          const unsigned long long g0 = mul2(alphas, two(__uint_as_float(even[r + 2]), __uint_as_float(even[r + 3])));
          const unsigned long long g1 = mul2(alphas, two(__uint_as_float(odd[r + 2]), __uint_as_float(odd[r + 3])));
          up[k] = pack_bf16x2(low_of(u0), low_of(u1));
          up[k + 1] = pack_bf16x2(high_of(u0), high_of(u1));
          gate[k] = pack_bf16x2(low_of(g0), low_of(g1));
          gate[k + 1] = pack_bf16x2(high_of(g0), high_of(g1));
        }
        load(!last, turn + kWpParts);  // under this step's arithmetic; waited for at its end
        // erf of the magnitudes from the table, two indices to a word
        constexpr uint32_t kFirst = kErfFirst * 0x10001u, kLast = (kErfFirst + kErfEntries - 1) * 0x10001u;
        float erf0[8], erf1[8];
        uint32_t smallest = 0xffffffffu;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t magnitudes = gate[k] & 0x7fff7fffu;
          smallest = __vminu2(smallest, magnitudes);
          const uint32_t offsets = 4u * __vminu2(__vmaxu2(magnitudes, kFirst), kLast) - 4u * kFirst;
          const char* const table = reinterpret_cast<const char*>(smem->tables.erf_of);
          erf0[k] = *reinterpret_cast<const float*>(table + (offsets & 0xffffu));
          erf1[k] = *reinterpret_cast<const float*>(table + (offsets >> 16));
        }
        if (__vminu2(smallest, kFirst) != kFirst) {  // one gate in 20000 of unit variance, and the zeros of rows that do not exist
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const uint32_t low = gate[k] & 0x7fffu, high = (gate[k] >> 16) & 0x7fffu;
            if (low < kErfFirst) erf0[k] = erf_below_table(__uint_as_float(low << 16));
            if (high < kErfFirst) erf1[k] = erf_below_table(__uint_as_float(high << 16));
          }
        }
        __syncwarp();
        // gelu_from_erf of the gates times up
        float v0[8], v1[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float gate0 = __uint_as_float(gate[k] << 16), gate1 = __uint_as_float(gate[k] & 0xffff0000u);
          const unsigned long long half = mul2(two(0.5f, 0.5f), two(gate0, gate1));
          const unsigned long long one_plus = add2(two(1.0f, 1.0f), two(copysignf(erf0[k], gate0), copysignf(erf1[k], gate1)));
          const unsigned long long v = mul2(mul2(half, one_plus), two(__uint_as_float(up[k] << 16), __uint_as_float(up[k] & 0xffff0000u)));
          v0[k] = low_of(v);
          v1[k] = high_of(v);
        }
        float most[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) most[k] = fmaxf(fabsf(v0[k]), fabsf(v1[k]));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float received = __shfl_xor_sync(0xffffffffu, a ? most[k] : most[k + 4], 16);
          most[k] = fmaxf(a ? most[k + 4] : most[k], received);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float received = __shfl_xor_sync(0xffffffffu, b ? most[k] : most[k + 2], 8);
          most[k] = fmaxf(b ? most[k + 2] : most[k], received);
        }
        // (a block of NaN has scale zero)
        const float maximum = fmaxf(fmaxf(c ? most[1] : most[0], __shfl_xor_sync(0xffffffffu, c ? most[0] : most[1], 4)), 0.0f);
        const uint32_t scale = encode_e4m3(gv_sixth(__fmul_rn(multiplier, maximum)));
        const float inverse = gv_scale_inverse_exact(multiplier) ? gv_scale_inverse(multiplier, scale, smem->tables.reciprocals)
                                                                 : scale_inverse_divided(multiplier, scale);
        uint32_t words[2];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          float inverses[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) inverses[k] = __shfl_sync(0xffffffffu, inverse, (lane & 3) | (16 * half + 4 * k));
          float x0[4], x1[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const unsigned long long x = mul2(two(v0[4 * half + k], v1[4 * half + k]), two(inverses[k], inverses[k]));
            x0[k] = low_of(x);
            x1[k] = high_of(x);
          }
          asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
              "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\t"
              "cvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
              "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\t"
              "cvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
              "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
              : "=r"(words[half])
              : "f"(x0[0]), "f"(x1[0]), "f"(x0[1]), "f"(x1[1]), "f"(x0[2]), "f"(x1[2]), "f"(x0[3]), "f"(x1[3]));
        }
        // 8 x 8 bytes over the eight lanes, transposed: bits 2, 1 and 0 of the lane number in turn
        const uint32_t received_a = __shfl_xor_sync(0xffffffffu, a ? words[0] : words[1], 16);
        const uint32_t lo = a ? received_a : words[0], hi = a ? words[1] : received_a;
        const uint32_t received_b = __shfl_xor_sync(0xffffffffu, __byte_perm(lo, hi, send_b), 8);
        const uint32_t kept_b = __byte_perm(lo, hi, keep_b);
        const uint32_t received_c = __shfl_xor_sync(0xffffffffu, __byte_perm(kept_b, received_b, send_c), 4);
        const uint32_t kept_c = __byte_perm(kept_b, received_b, keep_c);
        const uint32_t first = c ? received_c : kept_c, second = c ? kept_c : received_c;
        if (token < item.valid) {
          *reinterpret_cast<uint2*>(p.next_codes + static_cast<size_t>(item.row0 + token) * (kInter / 2) + unit * 32 + block * 8) =
              make_uint2(__byte_perm(first, second, low_word), __byte_perm(first, second, high_word));
          scales[sf_offset(item.local + token, 4 * unit + block, groups)] = static_cast<uint8_t>(scale);
        }
        if (last) break;
        turn += kWpParts;
        tmem_load_wait(even, odd);
      }
      if (++acc == kWpAccStages) {
        acc = 0;
        acc_phase ^= 1u;
      }
    }
  }

  tc_fence_before_sync();
  // Both CTAs stay until neither can still receive a remote arrive, a copy or a multicast commit.
  cluster_sync_all();
  if (warp == kWpMmaWarp) {
    tc_fence_after_sync();
    __syncwarp();
    pair_tmem_dealloc(tmem_base, kWpTmemColumns);
  }
}

// Re-tiles the w13 block scales by unit of 64 intermediate columns, twelve slots an expert of which the last is
// all zero: [expert][unit][K block of 256][MMA 0..3][512-byte atom], the atom being (n%32)*16 + (n/32)*4 + k over
// the unit's 128 MMA rows n.  kFragments: in this file's row order; else the 64 up rows, then the 64 gate rows.
// One thread per byte.
template <bool kFragments>
__global__ void retile_w13_unit_scales_kernel(const uint8_t* __restrict__ sidecar, uint8_t* __restrict__ tiled,
                                              int experts) {
  constexpr int groups = kHidden / 16;          // 176
  constexpr int k_blocks = kHidden / 256;       // 11
  const size_t index = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const size_t total = static_cast<size_t>(experts) * kWpUnitSlots * k_blocks * 4 * kSfAtomBytes;
  if (index >= total) return;
  const int byte = static_cast<int>(index % kSfAtomBytes);
  size_t rest = index / kSfAtomBytes;
  const int mma = static_cast<int>(rest % 4);
  rest /= 4;
  const int k_block = static_cast<int>(rest % k_blocks);
  rest /= k_blocks;
  const int unit = static_cast<int>(rest % kWpUnitSlots);
  const int expert = static_cast<int>(rest / kWpUnitSlots);
  const int n = ((byte & 15) >> 2) * 32 + (byte >> 4);  // MMA row of this byte
  const int k = byte & 3;
  uint8_t value = 0;
  if (unit < kWpUnits) {
    const bool gate = kFragments ? (n & 8) != 0 : n >= 64;
    const int column = kFragments ? 16 * (n >> 5) + 2 * (n & 7) + ((n >> 4) & 1) : n & 63;
    const int source_row = (gate ? kInter : 0) + unit * 64 + column;
    value = sidecar[static_cast<size_t>(expert) * kW13Out * groups +
                    sf_offset(source_row, (k_block * 4 + mma) * 4 + k, groups)];
  }
  tiled[index] = value;
}

}  // namespace

size_t w13_unit_scale_bytes(int experts) {
  return static_cast<size_t>(experts) * kWpUnitSlots * (kHidden / 256) * 4 * kSfAtomBytes;
}

void launch_retile_w13_unit_scales(const uint8_t* sidecar_scales, uint8_t* tiled, int experts, bool fragments,
                                   cudaStream_t stream) {
  const unsigned blocks = static_cast<unsigned>((w13_unit_scale_bytes(experts) + 255) / 256);
  if (fragments) retile_w13_unit_scales_kernel<true><<<blocks, 256, 0, stream>>>(sidecar_scales, tiled, experts);
  else retile_w13_unit_scales_kernel<false><<<blocks, 256, 0, stream>>>(sidecar_scales, tiled, experts);
}

int prepare_w13_pairs() {
  return static_cast<int>(cudaFuncSetAttribute(w13_geglu_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(kWpSmemBytes)));
}

void launch_w13_pairs(const W13PairOperands& op, const RoutePlan& plan, int sm_count, cudaStream_t stream) {
  WpParams p{};
  p.alpha = op.alpha;
  p.next_codes = op.next_codes;
  p.next_scales = op.next_scales;
  p.next_scale_q = op.next_scale_q;
  p.expert_offsets = plan.expert_offsets;
  p.scale_row_offsets = plan.scale_row_offsets;
  p.status = plan.status;
  p.early_weights = op.early_weights;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(sm_count & ~1));
  config.blockDim = dim3(kWpThreads);
  config.dynamicSmemBytes = kWpSmemBytes;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = 2;
  attributes[0].val.clusterDim.y = 1;
  attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = op.serial_launch ? 1 : 2;
  WpTokenMaps token_maps;
  for (int i = 0; i < kW13PairBoxes; ++i) token_maps.rows[i] = op.map_x[i];
  cudaLaunchKernelEx(&config, w13_geglu_pair_kernel, token_maps, op.map_w, op.map_x_sf, op.map_w_sf, p);
}

}  // namespace gv
