// The grouped w2 GEMM of the largest batches by CTA pairs: two 128-row tiles of an expert against the same output columns.
//
// What bounds it.  Operands in and rows out share the way between an SM and L2: 100 KB in take 0.72 us an item there, 48 KB out 0.84 to
// 1.0 us, both 1.4 to 2.1.  One CTA a tile (grouped_gemm_down.cu) fetches 103 KB for 128 rows x 192 columns and takes 2 us; a pair
// (tcgen05 cta_group::2, M = 256) needs the weights once for two row tiles, each CTA half of them: 66 KB an item and CTA.  With few tokens most
// experts have a single tile, whose pair fetches 132 KB where one CTA fetches 103; where the line lies is said at kDownPairTokens (moe_abi.cu).
// Without its stores the form before the next paragraph took 44 us of 68 at 4096 tokens, 115 of 203 at 16384.  Eight epilogue warps and stores without a cache
// hint make no difference.
// Two pairs of an expert share the weights, too: each weight stage is used by both, one after the other, and an item fetches 42 KB instead of 59.  (Loads and
// stores share the fabric: 48 KB stored and 64 KB loaded an item and SM take 1.45 us with everything in L2, either alone 1.0; the kernel took 1.6 at 16384
// tokens.)  And what does not fill a round of units is dealt out in thirds of them.  Alone, us, without both -> with: 2600 tokens 53.0 -> 50.4, 4096 67.3 -> 64.0, 8192
// 109.6 -> 108.8, 16384 197.5 -> 191.5; without the thirds 53.2, 65.0, 109.8 and 195; 4096 of uneven loads 69.7 -> 68.6 (without thirds 72.4), Zipf(1.1) 77.2 -> 77.3.
// Everything else is as in that file, whose column order, re-tiled scales and schedule this one shares: items of 192 columns, a unit
// five of one pair (three there: 2 % more at 16384 tokens) or three of two, a tile's activations fetched once a unit, two accumulators, results stored from registers.  The last tile of an expert
// with an odd number has no partner: its pair's second CTA fetches its half of the weights and stores nothing.
//
// Roles of each CTA (8 warps): 0 fetches weights, 1 copies scale factors and issues MMAs (in the first CTA, for both), 2 fetches
// activations, 4..7 the epilogue; one thread each but for the last.  Loads of both CTAs complete on the first one's barriers, MMAs on
// both's.  Every wait is bounded.
#include "gv_common.cuh"
#include "gv_cta_pair.cuh"
#include "gv_gemm_parts.cuh"
#include "gv_launchers.h"

namespace gv {

namespace {

constexpr int kDpStages = 7;                    // weight stages: one K block of this CTA's half of 192 output columns
constexpr int kDpSlots = 6;                     // K blocks of row tiles: the unit at work and the next
constexpr int kDpKBlocks = 3;                   // 704 = 256 + 256 + 192
constexpr int kDpLastMmas = 3;
constexpr int kDpAtoms = kInter / 64;           // 11 scale atoms a row tile
constexpr int kDpColumns = 192;                 // output columns of an item (MMA N)
constexpr int kDpTiles = (kHidden + kDpColumns - 1) / kDpColumns;       // 15
constexpr int kDpLastColumns = kHidden - (kDpTiles - 1) * kDpColumns;   // 128
constexpr int kDpUnitTiles = 5, kDpDoubleTiles = 3;   // column tiles of a unit of one pair of row tiles (5 items), and of two (6 items)
constexpr int kDpPairUnits = kDpTiles / kDpUnitTiles, kDpDoubleUnits = kDpTiles / kDpDoubleTiles;
static_assert(kDpTiles % kDpUnitTiles == 0 && kDpTiles % kDpDoubleTiles == 0 && kDpLastColumns == 128, "units of whole items, the last one of N = 128");
constexpr int kDpPieceRows = 32;                // weight rows of a copy: half a 64-column group
// Tensor memory: two accumulators, the scales of the unit's one or two row tiles (four columns an MMA), a K block's
// weight scales (eight columns an MMA; copies and MMAs execute in order, so one buffer is enough).
constexpr int kDpAccStages = 2;
constexpr uint32_t kDpSfaColumn = kDpAccStages * kDpColumns;
constexpr uint32_t kDpSfaColumns = kDpAtoms * 4;
constexpr uint32_t kDpSfbColumn = kDpSfaColumn + 2 * kDpSfaColumns;
constexpr uint32_t kDpTmemColumns = 512;
static_assert(kDpSfbColumn + 32 <= kDpTmemColumns, "tensor memory budget");
constexpr int kDpTokenBytes = 128 * kTileKBytes;            // 16 KiB
constexpr int kDpPieceBytes = kDpPieceRows * kTileKBytes;   // 4 KiB
constexpr int kDpWeightBytes = kDpColumns / 2 * kTileKBytes;  // 12 KiB
constexpr int kDpWeightSfBytes = 2 * kSfStageBytes;
constexpr int kDpWeightWarp = 0, kDpMmaWarp = 1, kDpTokenWarp = 2, kDpEpilogueWarp = 4;
constexpr int kDpEpilogueWarps = 4;
constexpr int kDpThreads = (kDpEpilogueWarp + kDpEpilogueWarps) * 32;

struct alignas(1024) DownPairSmem {
  uint8_t a[kDpSlots][kDpTokenBytes];
  uint8_t b[kDpStages][kDpWeightBytes];
  uint8_t sfa[kDpSlots][kSfStageBytes];
  uint8_t sfb[kDpStages][kDpWeightSfBytes];
  uint64_t a_full[kDpSlots], b_full[kDpStages];    // first CTA: the bytes have landed in both
  uint64_t a_empty[kDpSlots], b_empty[kDpStages];  // both CTAs: the MMAs that read them have completed
  uint64_t acc_full[kDpAccStages];                 // both CTAs
  uint64_t acc_empty[kDpAccStages];                // first CTA: both CTAs' epilogues have copied the accumulator out
  uint32_t tmem_base;
  volatile int abort;
  // by expert: first row, first row tile, units before it
  int offsets[kExperts + 1], tiles[kExperts], units[kExperts + 1], scan[kExperts / 32];
};
constexpr size_t kDpSmemBytes = sizeof(DownPairSmem) + 1024;
static_assert(kDpSmemBytes <= 232448, "shared memory budget of one sm_100 CTA");

struct DownPairParams {
  const float* alpha;
  __nv_bfloat16* out;
  const int* expert_offsets;
  const int* scale_row_offsets;
  int* status;
  bool early_weights;
};

// One or two pairs of row tiles of an expert, of each of which this CTA has one tile, and column tiles [begin, end).
struct DownPairUnit {
  int expert, begin, end;
  int pairs;
  int first;       // row tile of the expert that the first pair begins with
  int rows;        // of the expert
};
struct DownPairTile {
  int tile;        // this CTA's row tile of the pair
  int row0, rows;  // its first sorted row, and how many it has (none: an odd tile's partner)
  bool both;       // the pair's second tile exists
};
__device__ __forceinline__ int down_pairs_of(int rows) { return (rows + 2 * kTileM - 1) / (2 * kTileM); }
__device__ __forceinline__ DownPairTile down_pair_tile(const DownPairSmem* smem, const DownPairUnit& unit, int pair, uint32_t rank) {
  const int index = unit.first + 2 * pair + static_cast<int>(rank), local = index * kTileM;
  DownPairTile t;
  t.tile = smem->tiles[unit.expert] + index;
  t.row0 = smem->offsets[unit.expert] + local;
  t.rows = unit.rows - local < kTileM ? unit.rows - local : kTileM;
  t.both = unit.rows > (unit.first + 2 * pair + 1) * kTileM;
  return t;
}

// An expert's units are those of its pairs two by two, then those of a pair left over; they are numbered expert by expert and dealt to the
// clusters in snake order, so that at any time the grid works on neighbouring row tiles and an expert's weights are fetched from HBM once.
struct DownPairSchedule {
  const DownPairSmem* smem;
  int round = 0;
  __device__ explicit DownPairSchedule(const DownPairSmem* s) : smem(s) {}
  __device__ bool next(DownPairUnit& unit) {
    const int clusters = static_cast<int>(gridDim.x) >> 1, mine = static_cast<int>(blockIdx.x) >> 1;
    const int index = round * clusters + ((round & 1) ? clusters - 1 - mine : mine);
    ++round;
    // What does not fill a round is dealt out in thirds of a unit where that makes the last clusters' way shorter.
    const int units = smem->units[kExperts], whole = units / clusters * clusters;
    const int over = 3 * (units - whole) <= 2 * clusters ? index - whole : -1, third = over % 3, number = over < 0 ? index : whole + over / 3;
    if (number >= units) return false;  // only the last round is incomplete
    int expert = 0;  // the last one with units[expert] <= number
#pragma unroll
    for (int step = kExperts / 2; step; step >>= 1)
      if (smem->units[expert + step] <= number) expert += step;
    unit.expert = expert;
    unit.rows = smem->offsets[expert + 1] - smem->offsets[expert];
    const int own = number - smem->units[expert], doubles = down_pairs_of(unit.rows) / 2;
    unit.pairs = own < doubles * kDpDoubleUnits ? 2 : 1;
    const int part = unit.pairs == 2 ? own % kDpDoubleUnits : own - doubles * kDpDoubleUnits;
    const int columns = unit.pairs == 2 ? kDpDoubleTiles : kDpUnitTiles;
    unit.first = 4 * (unit.pairs == 2 ? own / kDpDoubleUnits : doubles);
    unit.begin = part * columns;
    unit.end = unit.begin + columns;
    if (over >= 0) {
      const int step = (columns + 2) / 3;
      unit.begin += third * step;
      unit.end = min(unit.end, unit.begin + step);
    }
    return true;
  }
};

__global__ void __launch_bounds__(kDpThreads, 1)
grouped_down_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_a_sf,
                         const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_b_sf,
                         const DownPairParams p) {
  extern __shared__ uint8_t smem_raw[];
  DownPairSmem* smem = reinterpret_cast<DownPairSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_cta_rank();
  const bool is_leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kDpSlots; ++s) {
      mbar_init(&smem->a_full[s], 1);   // the first CTA's producer announces both CTAs' byte count
      mbar_init(&smem->a_empty[s], 1);
    }
    for (int s = 0; s < kDpStages; ++s) {
      mbar_init(&smem->b_full[s], 1);
      mbar_init(&smem->b_empty[s], 1);
    }
    for (int s = 0; s < kDpAccStages; ++s) {
      mbar_init(&smem->acc_full[s], 1);
      mbar_init(&smem->acc_empty[s], 2 * kDpEpilogueWarps);
    }
    smem->abort = 0;
    fence_barrier_init();
    prefetch_tensor_map(&map_a);
    prefetch_tensor_map(&map_a_sf);
    prefetch_tensor_map(&map_b);
    prefetch_tensor_map(&map_b_sf);
  }
  // Both CTAs run and their barriers exist before either touches the other's tensor memory or arrives there.
  __syncwarp();
  cluster_sync_all();
  if (warp == kDpMmaWarp) pair_tmem_alloc(&smem->tmem_base, kDpTmemColumns);  // the whole tensor memory
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = smem->tmem_base;
  // The weights and the plan come from before the previous kernel, which let this one start after its own wait.
  if (!p.early_weights) grid_dependency_wait();
  if (warp < kExperts / 32) {
    // thread = expert: units before it
    const int e = threadIdx.x;
    const int row = p.expert_offsets[e], next_row = p.expert_offsets[e + 1];
    const int pairs = down_pairs_of(next_row - row);
    const int own = pairs / 2 * kDpDoubleUnits + pairs % 2 * kDpPairUnits;
    int inclusive = own;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1) {
      const int other = __shfl_up_sync(0xffffffffu, inclusive, offset);
      if (lane >= offset) inclusive += other;
    }
    if (lane == 31) smem->scan[warp] = inclusive;
    smem->offsets[e] = row;
    smem->tiles[e] = p.scale_row_offsets[e] / kTileM;
    if (e == kExperts - 1) smem->offsets[kExperts] = next_row;
    named_barrier(1, kExperts);
    for (int w = 0; w < warp; ++w) inclusive += smem->scan[w];
    smem->units[e] = inclusive - own;
    if (e == kExperts - 1) smem->units[kExperts] = inclusive;
  }
  __syncthreads();
  if (warp != kDpWeightWarp) {
    grid_dependency_wait();
    grid_launch_dependents();  // after the wait: whoever starts now may read what came before this kernel
  }

  DownPairSchedule schedule(smem);
  DownPairUnit unit;
  bool ok = true;

  if (warp == kDpWeightWarp) {
    // ---------------- weights: this CTA's half of every column tile of every unit, three K blocks each ----------------
    if (elect_one()) {
      const uint32_t full0 = is_leader ? smem_u32(&smem->b_full[0]) : cluster_map_shared(smem_u32(&smem->b_full[0]), 0);
      int stage = 0, issued = 0;
      uint32_t phase = 0;
      while (ok && schedule.next(unit)) {
        for (int n = unit.begin; ok && n < unit.end; ++n) {
          const int pieces = n + 1 == kDpTiles ? kDpLastColumns / 2 / kDpPieceRows : kDpColumns / 2 / kDpPieceRows;
          const int group0 = unit.expert * (kHidden / 64) + (kDpColumns / 64) * n;
          const int sf_row = (unit.expert * kDpTiles + n) * kDpKBlocks * 8;
#pragma unroll
          for (int kb = 0; kb < kDpKBlocks; ++kb) {
            ok = wait_or_abort(&smem->b_empty[stage], phase ^ 1u, smem, p.status);
            if (!ok) break;
            const uint32_t bar = full0 + 8 * stage;
            if (is_leader)
              mbar_arrive_expect_tx(&smem->b_full[stage], 2u * (static_cast<uint32_t>(pieces) * kDpPieceBytes + kDpWeightSfBytes));
#pragma unroll
            for (int j = 0; j < kDpColumns / 2 / kDpPieceRows; ++j) {
              const int piece = static_cast<int>(rank) * pieces + j;
              if (j < pieces)
                pair_load_piece(smem->b[stage] + j * kDpPieceBytes, &map_b, bar, kb * kTileKBytes, piece & 1, group0 + (piece >> 1));
            }
            pair_load(smem->sfb[stage], &map_b_sf, bar, 0, sf_row + 8 * kb);
            ++issued;
            if (++stage == kDpStages) {
              stage = 0;
              phase ^= 1u;
            }
          }
        }
      }
      if (!ok && is_leader) {
        // Unwinding: the copies already issued (by either CTA) land before shared memory is given up; the second CTA stays
        // resident until the cluster barrier at the end.
        const int pending = issued < kDpStages ? issued : kDpStages;
        for (int i = 0; i < pending; ++i) {
          if (--stage < 0) {
            stage = kDpStages - 1;
            phase ^= 1u;
          }
          mbar_wait_bounded(&smem->b_full[stage], phase, 40000000ll);
        }
      }
    }
    __syncwarp();
  } else if (warp == kDpTokenWarp) {
    // ---------------- activations: this CTA's row tiles of every unit once ----------------
    if (elect_one()) {
      const uint32_t full0 = is_leader ? smem_u32(&smem->a_full[0]) : cluster_map_shared(smem_u32(&smem->a_full[0]), 0);
      int slot = 0, issued = 0;
      uint32_t phase = 0;
      while (ok && schedule.next(unit)) {
        for (int pair = 0; ok && pair < unit.pairs; ++pair) {
          const DownPairTile tile = down_pair_tile(smem, unit, pair, rank);
#pragma unroll
          for (int kb = 0; kb < kDpKBlocks; ++kb) {
            ok = wait_or_abort(&smem->a_empty[slot], phase ^ 1u, smem, p.status);
            if (!ok) break;
            const uint32_t bar = full0 + 8 * slot;
            if (is_leader) mbar_arrive_expect_tx(&smem->a_full[slot], (tile.both ? 2u : 1u) * (kDpTokenBytes + kSfStageBytes));
            if (is_leader || tile.both) {
              // (the last K block's fourth atom is the next tile's first; nothing reads it)
              pair_load(smem->a[slot], &map_a, bar, kb * kTileKBytes, tile.row0);
              pair_load(smem->sfa[slot], &map_a_sf, bar, 0, tile.tile * kDpAtoms + 4 * kb);
            }
            ++issued;
            if (++slot == kDpSlots) {
              slot = 0;
              phase ^= 1u;
            }
          }
        }
      }
      if (!ok && is_leader) {
        const int pending = issued < kDpSlots ? issued : kDpSlots;
        for (int i = 0; i < pending; ++i) {
          if (--slot < 0) {
            slot = kDpSlots - 1;
            phase ^= 1u;
          }
          mbar_wait_bounded(&smem->a_full[slot], phase, 40000000ll);
        }
      }
    }
    __syncwarp();
  } else if (warp == kDpMmaWarp) {
    // ---------------- first CTA: scale copies and MMAs for both, in one thread ----------------
    // They execute in order.  The scales of a row tile are copied once a unit; a weight stage is released by the unit's last pair.
    if (is_leader && elect_one()) {
      constexpr uint32_t hi_sf = (128u >> 4) | (1u << 14);                // 8 rows x 16 B, no swizzle
      constexpr uint32_t hi_ab = (1024u >> 4) | (1u << 14) | (2u << 29);  // 8 rows x 128 B, 128B swizzle
      const uint32_t a_lo0 = (smem_u32(smem->a[0]) & 0x3ffffu) >> 4, b_lo0 = (smem_u32(smem->b[0]) & 0x3ffffu) >> 4;
      const uint32_t sfa_lo0 = (smem_u32(smem->sfa[0]) & 0x3ffffu) >> 4, sfb_lo0 = (smem_u32(smem->sfb[0]) & 0x3ffffu) >> 4;
      const uint32_t tmem_sfb = tmem_base + kDpSfbColumn;
      int stage0 = 0, acc = 0;                // stage0: where the column tile's first K block is
      uint32_t phase0 = 0, acc_phase = 0;
      uint32_t uses = 0;                      // pairs of the units before: a pair's K blocks are in slots 0..2 or 3..5 by turns
      bool landed = false;                    // the next column tile's first stage has been seen
      while (ok && schedule.next(unit)) {
        for (int n = unit.begin; ok && n < unit.end; ++n) {
          // E2M1 x E2M1, both K-major, UE4M3 scales; N at [17,23) in units of 8, M = 256 at [24,29) in units of 16
          const uint32_t columns = n + 1 == kDpTiles ? kDpLastColumns : kDpColumns;
          const uint32_t descriptor = (1u << 7) | (1u << 10) | ((columns >> 3) << 17) | (static_cast<uint32_t>(256 >> 4) << 24);
          int stage = stage0;
          uint32_t phase = phase0;
#pragma unroll 1
          for (int pair = 0; ok && pair < unit.pairs; ++pair) {
            const bool last_pair = pair + 1 == unit.pairs;
            const uint32_t use = uses + static_cast<uint32_t>(pair), slot0 = (use & 1u) * kDpKBlocks;
            const uint32_t tmem_acc = tmem_base + static_cast<uint32_t>(acc) * kDpColumns;
            ok = wait_or_abort(&smem->acc_empty[acc], acc_phase ^ 1u, smem, p.status);
            if (!ok) break;
            tc_fence_after_sync();
            stage = stage0;
            phase = phase0;
#pragma unroll
            for (int kb = 0; kb < kDpKBlocks; ++kb) {
              constexpr int kMmas[kDpKBlocks] = {4, 4, kDpLastMmas};
              const uint32_t slot = slot0 + kb;
              if (n == unit.begin) ok = wait_or_abort(&smem->a_full[slot], (use >> 1) & 1u, smem, p.status);
              if (ok && pair == 0 && !landed) ok = wait_or_abort(&smem->b_full[stage], phase, smem, p.status);
              if (!ok) break;
              tc_fence_after_sync();
              const uint32_t tmem_sfa = tmem_base + kDpSfaColumn + static_cast<uint32_t>(pair) * kDpSfaColumns + static_cast<uint32_t>(16 * kb);
              if (n == unit.begin) {
                const uint32_t sfa = sfa_lo0 + slot * (kSfStageBytes >> 4);
#pragma unroll
                for (int j = 0; j < kMmas[kb]; ++j) pair_copy_sf(tmem_sfa + 4 * j, hi_sf, sfa + 32 * j);
              }
              const uint32_t sfb = sfb_lo0 + static_cast<uint32_t>(stage) * (kDpWeightSfBytes >> 4);
              const uint32_t a = a_lo0 + slot * (kDpTokenBytes >> 4);
              const uint32_t b = b_lo0 + static_cast<uint32_t>(stage) * (kDpWeightBytes >> 4);
              uint64_t* const empty = &smem->b_empty[stage];
              if (++stage == kDpStages) {
                stage = 0;
                phase ^= 1u;
              }
#pragma unroll
              for (int j = 0; j < kMmas[kb]; ++j) {
                pair_copy_sf(tmem_sfb + 8 * j, hi_sf, sfb + 32 * j);
                pair_copy_sf(tmem_sfb + 8 * j + 4, hi_sf, sfb + 128 + 32 * j);
              }
#pragma unroll
              for (int j = 0; j < kMmas[kb]; ++j)
                pair_mma(tmem_acc, hi_ab, a + 2 * j, b + 2 * j, descriptor, tmem_sfa + 4 * j, tmem_sfb + 8 * j, (kb | j) != 0 ? 1u : 0u);
              if (pair == 0) landed = mbar_try_wait(&smem->b_full[stage], phase);
              if (last_pair) pair_commit_both(empty);
              if (n + 1 == unit.end) pair_commit_both(&smem->a_empty[slot]);
              if (kb + 1 == kDpKBlocks) pair_commit_both(&smem->acc_full[acc]);
            }
            if (++acc == kDpAccStages) {
              acc = 0;
              acc_phase ^= 1u;
            }
          }
          stage0 = stage;
          phase0 = phase;
        }
        uses += static_cast<uint32_t>(unit.pairs);
      }
    }
    __syncwarp();
  } else if (warp >= kDpEpilogueWarp) {
    // ---------------- epilogue: 64 columns of 16 rows at a time ----------------
    static_assert(kDpEpilogueWarps == 4 && kDpSlots == 2 * kDpKBlocks, "a quarter of the rows each; a pair's K blocks are in slots 0 to 2 or 3 to 5");
    const int quarter = warp & 3;                        // the tensor-memory lanes this warp may read
    constexpr int kParts = 2;                            // 16-row parts of the quarter
    const int row_in_tile = quarter * 32 + (lane >> 2);  // and 8, 16 and 24 further down
    const uint32_t tmem_rows = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    unsigned long long keep_in_l2;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(keep_in_l2));
    int acc = 0;
    uint32_t acc_phase = 0;
    while (ok && schedule.next(unit)) {
      const float alpha = p.alpha[unit.expert];
      for (int item = unit.begin * unit.pairs; item < unit.end * unit.pairs; ++item) {
        const int n = unit.pairs == 2 ? item >> 1 : item;
        const DownPairTile tile = down_pair_tile(smem, unit, unit.pairs == 2 ? item & 1 : 0, rank);
        const int warp_rows = tile.rows - quarter * 32;  // of this warp's quarter that exist
        ok = __all_sync(0xffffffffu, wait_or_abort(&smem->acc_full[acc], acc_phase, smem, p.status));
        if (!ok) break;
        tc_fence_after_sync();
        const int groups = n + 1 == kDpTiles ? kDpLastColumns / 64 : kDpColumns / 64;
        const int steps = warp_rows <= 0 ? 0 : (warp_rows <= 16 ? 1 : kParts) * groups;  // none of rows that do not exist
        bool released = false;
        int step = 0;
#pragma unroll 1
        do {
          uint32_t r[32];
          const int part = step >= groups ? 1 : 0, group = step - part * groups;
          if (step < steps) {
            tmem_load_16x64(tmem_rows + (static_cast<uint32_t>(part * 16) << 16) + static_cast<uint32_t>(acc) * kDpColumns + 64 * group, r);
            tmem_load_wait(r);
          }
          if (step + 1 >= steps) {
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
              if (is_leader) mbar_arrive(&smem->acc_empty[acc]);
              else pair_arrive_remote(&smem->acc_empty[acc], 0);
            }
            released = true;
          }
          if (step >= steps) break;
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const int row = row_in_tile + 16 * part + 8 * half;
            if (row >= tile.rows) continue;
            uint32_t v[8];
#pragma unroll
            for (int g = 0; g < 8; ++g)
              v[g] = pack_bf16x2(__fmul_rn(alpha, __uint_as_float(r[4 * g + 2 * half])),
                                 __fmul_rn(alpha, __uint_as_float(r[4 * g + 2 * half + 1])));
            const int column = n * kDpColumns + 64 * group + (lane & 3) * 16;
            // read back by the weighted reduce right after this launch: L2 is asked to keep it
            asm volatile("st.global.L2::cache_hint.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8}, %9;" ::"l"(
                             p.out + static_cast<size_t>(tile.row0 + row) * kHidden + column),
                         "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "l"(keep_in_l2)
                         : "memory");
          }
          ++step;
        } while (!released);
        if (++acc == kDpAccStages) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
    }
  }

  tc_fence_before_sync();
  // Both CTAs stay until neither can still receive a remote arrive, a copy or a commit.
  cluster_sync_all();
  if (warp == kDpMmaWarp) {
    tc_fence_after_sync();
    __syncwarp();
    pair_tmem_dealloc(tmem_base, kDpTmemColumns);
  }
}

}  // namespace

int prepare_grouped_down_pairs() {
  return static_cast<int>(cudaFuncSetAttribute(grouped_down_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(kDpSmemBytes)));
}

void launch_grouped_down_pairs(const GemmOperands& op, const RoutePlan& plan, int sm_count, cudaStream_t stream) {
  DownPairParams p{};
  p.alpha = op.alpha;
  p.out = static_cast<__nv_bfloat16*>(op.out);
  p.expert_offsets = plan.expert_offsets;
  p.scale_row_offsets = plan.scale_row_offsets;
  p.status = plan.status;
  p.early_weights = op.early_weights;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(sm_count & ~1));
  config.blockDim = dim3(kDpThreads);
  config.dynamicSmemBytes = kDpSmemBytes;
  config.stream = stream;
  cudaLaunchAttribute attributes[2];
  attributes[0].id = cudaLaunchAttributeClusterDimension;
  attributes[0].val.clusterDim.x = 2;
  attributes[0].val.clusterDim.y = 1;
  attributes[0].val.clusterDim.z = 1;
  attributes[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attributes[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attributes;
  config.numAttrs = 2;
  cudaLaunchKernelEx(&config, grouped_down_pair_kernel, op.map_a, op.map_down_a_sf, op.map_down_pieces, op.map_down_b_sf, p);
}

}  // namespace gv
