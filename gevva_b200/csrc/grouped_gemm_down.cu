// The grouped w2 GEMM of prefill-sized batches: rows of an expert's 128-row tiles against its 2816 output
// columns, K = 704.
//
// What bounds it.  At 4096 tokens the launch reads 143 MB of weights and writes 184 MB of rows: about
// 50 us of HBM time (measured copy rate), against 20 us of tensor-pipe time.  As a general 128 x 256
// tile GEMM (an accumulator per item of three K blocks, activations fetched again for every item,
// results through a staging tile) it took 75 us, and 37.8, 49 and 230 us at 1024, 2048 and 16384 tokens:
// the accumulator's hand-over was not overlapped, and shared memory, which has to carry the MMAs' operand
// reads, the arriving operands and the staged results, had no bandwidth left.  Here 35.7, 46, 70 and 227:
//   * an item is 192 output columns (15 to a row tile, the last of 128): two accumulators fit beside the
//     scales in tensor memory, so that draining one overlaps the next item's MMAs.  128-column items with
//     three accumulators took 76 us at 4096 tokens (an MMA and its share of the scale copies take 105 cycles to issue at
//     any N up to 128 and 111 at 192), 256-column items with one 80;
//   * a unit of work is a row tile against three of its items, and the tile's activations and their scales are
//     fetched and copied once a unit;
//   * scale copies and MMAs are issued by one thread (see there);
//   * results go from tensor memory to global memory without shared memory.  tcgen05.ld.16x256b gives the
//     four lanes of a quad the columns 8g + 2t, 8g + 2t + 1 of a row (t the lane in the quad, g = 0..7 the
//     register pair).  The weight rows are therefore taken in the order in which those are columns
//     16t + 2g, 16t + 2g + 1 of memory: a lane holds 16 consecutive columns and a quad stores a whole
//     128-byte line of a row.  The order costs nothing: it is a five-dimensional view of the same weights
//     ([64-column group][g][t][pair] with strides of 64, 2, 16 and 1 rows), and the scales have a
//     re-tiled copy made at runner creation.
// Units that do not fill a round are dealt out item by item where that is shorter (us alone, all in units -> so): 700 tokens 33.6 -> 33.1, 1000 36.0 -> 35.5, Zipf(1.1)
// 36.9 -> 35.3, 2048 46.2 -> 44.8, 2304 56.3 -> 53.7; two layers of 700 tokens 219.3 -> 216.6, 1000 234.2 -> 231.9, 2048 314.1 -> 311.4.
// From 2560 tokens on grouped_gemm_down_pair.cu takes its place. What is left is the way between an SM and L2, which stores and TMA loads share: the stores of
// an item (48 KB) raise the wait for its operands from 500 to 1700 cycles.
//
// Roles (8 warps): 0 fetches weights, 1 copies scale factors and issues MMAs, 2 fetches activations, 4..7 the
// epilogue (a quarter of the rows each; four more warps made no difference).  Every wait is bounded.
#include "gv_common.cuh"
#include "gv_gemm_parts.cuh"
#include "gv_launchers.h"

namespace gv {

namespace {

constexpr int kDnStages = 5;                    // weight stages: one K block of 192 output columns each
constexpr int kDnSlots = 4;                     // K blocks of row tiles: the tile at work and the start of the next
constexpr int kDnKBlocks = 3;                   // 704 = 256 + 256 + 192
constexpr int kDnLastMmas = 3;
constexpr int kDnAtoms = kInter / 64;           // 11 scale atoms a tile
constexpr int kDnColumns = 192;                 // output columns of an item (MMA N)
constexpr int kDnTiles = (kHidden + kDnColumns - 1) / kDnColumns;       // 15
constexpr int kDnLastColumns = kHidden - (kDnTiles - 1) * kDnColumns;   // 128
constexpr int kDnUnitTiles = 3;                 // items of a unit
constexpr int kDnTileUnits = kDnTiles / kDnUnitTiles;
static_assert(kDnTiles % kDnUnitTiles == 0, "units of whole items");
static_assert(kDnLastColumns == 128, "the last item is an N = 128 MMA");
// Tensor memory: two accumulators, the scales of the row tile at work (four columns an MMA), two K blocks'
// weight scales (eight columns an MMA).
constexpr int kDnAccStages = 2;
constexpr int kDnSfbBuffers = 2;
constexpr uint32_t kDnSfaColumn = kDnAccStages * kDnColumns;
constexpr uint32_t kDnSfbColumn = kDnSfaColumn + kDnAtoms * 4;
constexpr uint32_t kDnTmemColumns = 512;
static_assert(kDnSfbColumn + kDnSfbBuffers * 32 <= kDnTmemColumns, "tensor memory budget");
constexpr int kDnTokenBytes = 128 * kTileKBytes;            // 16 KiB
constexpr int kDnWeightBytes = kDnColumns * kTileKBytes;    // 24 KiB
constexpr int kDnWeightSfBytes = 2 * kSfStageBytes;
constexpr int kDnWeightWarp = 0, kDnMmaWarp = 1, kDnTokenWarp = 2, kDnEpilogueWarp = 4;
constexpr int kDnEpilogueWarps = 4;
constexpr int kDnThreads = (kDnEpilogueWarp + kDnEpilogueWarps) * 32;

struct alignas(1024) DownSmem {
  uint8_t a[kDnSlots][kDnTokenBytes];
  uint8_t b[kDnStages][kDnWeightBytes];
  uint8_t sfa[kDnSlots][kSfStageBytes];
  uint8_t sfb[kDnStages][kDnWeightSfBytes];
  uint64_t a_full[kDnSlots], a_empty[kDnSlots];
  uint64_t b_full[kDnStages], b_empty[kDnStages];
  uint64_t acc_full[kDnAccStages], acc_empty[kDnAccStages];
  uint32_t tmem_base;
  volatile int abort;
};
constexpr size_t kDnSmemBytes = sizeof(DownSmem) + 1024;
static_assert(kDnSmemBytes <= 232448, "shared memory budget of one sm_100 CTA");

struct DownParams {
  const uint8_t* a_scales;             // w2 operand scale regions
  const uint8_t* b_scales;             // launch_retile_w2_scales
  const float* alpha;
  __nv_bfloat16* out;
  const unsigned long long* row_dest;  // optional: address of each output row (may be peer memory)
  const int* tile_expert;
  const int* expert_offsets;
  const int* scale_row_offsets;
  const int* num_m_tiles;
  const int* tile_first;               // optional
  int* status;
  bool early_weights;
};

// A row tile of an expert and kDnUnitTiles of its column tiles [begin, end).
struct DownUnit {
  int tile, begin, end;
  int expert;
};

// Units are numbered row tile by row tile and dealt to the CTAs in snake order, so that at any time the
// grid works on neighbouring row tiles and an expert's weights are fetched from HBM once.  (Equal
// contiguous stretches, which keep a row tile resident for all its columns, read the weights once per
// row tile: 80 us instead of 75 at 4096 tokens, 340 instead of 230 at 16384.)
struct DownSchedule {
  const DownParams& p;
  int round, first, units;
  __device__ DownSchedule(const DownParams& params) : p(params) {
    round = 0;
    first = p.tile_first ? p.tile_first[0] : 0;
    units = p.num_m_tiles[0] * kDnTileUnits;
  }
  __device__ bool next(DownUnit& unit) {
    const int grid = static_cast<int>(gridDim.x);
    const int index = round * grid + ((round & 1) ? grid - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x));
    ++round;
    // What does not fill a round is dealt out item by item where that makes the last CTAs' way shorter.
    const int whole = units / grid * grid, over = kDnUnitTiles * (units - whole) <= (kDnUnitTiles - 1) * grid ? index - whole : -1;
    const int number = over < 0 ? index : whole + over / kDnUnitTiles;
    if (number >= units) return false;  // only the last round is incomplete
    unit.tile = first + number / kDnTileUnits;
    unit.begin = number % kDnTileUnits * kDnUnitTiles;
    unit.end = unit.begin + kDnUnitTiles;
    if (over >= 0) {
      unit.begin += over % kDnUnitTiles;
      unit.end = unit.begin + 1;
    }
    unit.expert = p.tile_expert[unit.tile];
    return true;
  }
};

__device__ __forceinline__ void tma_load_5d(void* smem_dst, const void* tensor_map, uint64_t* bar, int x, int group) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %4, %4, %5}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(tensor_map), "r"(smem_u32(bar)), "r"(x), "r"(0), "r"(group)
      : "memory");
}

__device__ __forceinline__ void down_copy_sf(uint32_t tmem_address, uint32_t lo) {
  constexpr uint32_t hi = (128u >> 4) | (1u << 14);  // 8 rows x 16 B, no swizzle
  asm volatile("{\n\t.reg .b64 d;\n\tmov.b64 d, {%1, %2};\n\ttcgen05.cp.cta_group::1.32x128b.warpx4 [%0], d;\n\t}" ::"r"(tmem_address),
               "r"(lo), "r"(hi)
               : "memory");
}

__device__ __forceinline__ void down_mma(uint32_t tmem_acc, uint32_t a_lo, uint32_t b_lo, uint32_t tmem_sfa, uint32_t tmem_sfb,
                                         uint32_t descriptor, bool accumulate) {
  constexpr uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);  // 8 rows x 128 B, 128B swizzle
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 d0, d1;\n\t"
      "setp.ne.b32 p, %7, 0;\n\t"
      "mov.b64 d0, {%1, %3};\n\t"
      "mov.b64 d1, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], d0, d1, %4, [%5], [%6], p;\n\t}" ::"r"(tmem_acc),
      "r"(a_lo), "r"(b_lo), "r"(hi), "r"(descriptor), "r"(tmem_sfa), "r"(tmem_sfb), "r"(accumulate ? 1u : 0u)
      : "memory");
}

__global__ void __launch_bounds__(kDnThreads, 1)
grouped_down_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const DownParams p) {
  extern __shared__ uint8_t smem_raw[];
  DownSmem* smem = reinterpret_cast<DownSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kDnSlots; ++s) {
      mbar_init(&smem->a_full[s], 1);
      mbar_init(&smem->a_empty[s], 1);
    }
    for (int s = 0; s < kDnStages; ++s) {
      mbar_init(&smem->b_full[s], 1);
      mbar_init(&smem->b_empty[s], 1);
    }
    for (int s = 0; s < kDnAccStages; ++s) {
      mbar_init(&smem->acc_full[s], 1);
      mbar_init(&smem->acc_empty[s], kDnEpilogueWarps);
    }
    smem->abort = 0;
    fence_barrier_init();
    prefetch_tensor_map(&map_a);
    prefetch_tensor_map(&map_b);
  }
  if (warp == kDnMmaWarp) {
    tmem_alloc(&smem->tmem_base, kDnTmemColumns);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = smem->tmem_base;
  // The weights (and the plan) come from before the previous kernel, which let this one start after its own wait.
  if (!(p.early_weights && warp == kDnWeightWarp)) {
    grid_dependency_wait();
    grid_launch_dependents();  // after the wait: whoever starts now may read what came before this kernel
  }

  DownSchedule schedule(p);
  DownUnit unit;
  bool ok = true;

  if (warp == kDnWeightWarp) {
    // ---------------- weights: every column tile of every unit, three K blocks each ----------------
    int stage = 0, issued = 0;
    uint32_t phase = 0;
    while (ok && schedule.next(unit)) {
      for (int n = unit.begin; ok && n < unit.end; ++n) {
        const uint8_t* sf = p.b_scales + static_cast<size_t>(unit.expert * kDnTiles + n) * (kDnKBlocks * kDnWeightSfBytes);
        for (int kb = 0; kb < kDnKBlocks; ++kb) {
          ok = __all_sync(0xffffffffu, wait_or_abort(&smem->b_empty[stage], phase ^ 1u, smem, p.status));
          if (!ok) break;
          if (elect_one()) {
            mbar_arrive_expect_tx(&smem->b_full[stage], kDnWeightBytes + kDnWeightSfBytes);
            tma_load_5d(smem->b[stage], &map_b, &smem->b_full[stage], kb * kTileKBytes,
                        unit.expert * (kHidden / 64) + (kDnColumns / 64) * n);
            bulk_load_1d(smem->sfb[stage], sf + kb * kDnWeightSfBytes, kDnWeightSfBytes, &smem->b_full[stage]);
          }
          __syncwarp();
          ++issued;
          if (++stage == kDnStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
    }
    if (!ok && lane == 0) {
      // unwinding: the copies already issued land before shared memory is given up
      const int pending = issued < kDnStages ? issued : kDnStages;
      for (int i = 0; i < pending; ++i) {
        if (--stage < 0) {
          stage = kDnStages - 1;
          phase ^= 1u;
        }
        mbar_wait_bounded(&smem->b_full[stage], phase, 40000000ll);
      }
    }
  } else if (warp == kDnTokenWarp) {
    // ---------------- activations: every unit's row tile once ----------------
    int slot = 0, issued = 0;
    uint32_t phase = 0;
    while (ok && schedule.next(unit)) {
      const int row = p.expert_offsets[unit.expert] + unit.tile * kTileM - p.scale_row_offsets[unit.expert];
      const uint8_t* sf = p.a_scales + static_cast<size_t>(unit.tile) * (kDnAtoms * kSfAtomBytes);
      for (int kb = 0; kb < kDnKBlocks; ++kb) {
        ok = __all_sync(0xffffffffu, wait_or_abort(&smem->a_empty[slot], phase ^ 1u, smem, p.status));
        if (!ok) break;
        if (elect_one()) {
          const uint32_t sf_bytes = static_cast<uint32_t>(kb + 1 == kDnKBlocks ? kDnLastMmas : 4) * kSfAtomBytes;
          mbar_arrive_expect_tx(&smem->a_full[slot], kDnTokenBytes + sf_bytes);
          tma_load_2d(smem->a[slot], &map_a, &smem->a_full[slot], kb * kTileKBytes, row);
          bulk_load_1d(smem->sfa[slot], sf + kb * kSfStageBytes, sf_bytes, &smem->a_full[slot]);
        }
        __syncwarp();
        ++issued;
        if (++slot == kDnSlots) {
          slot = 0;
          phase ^= 1u;
        }
      }
    }
    if (!ok && lane == 0) {
      const int pending = issued < kDnSlots ? issued : kDnSlots;
      for (int i = 0; i < pending; ++i) {
        if (--slot < 0) {
          slot = kDnSlots - 1;
          phase ^= 1u;
        }
        mbar_wait_bounded(&smem->a_full[slot], phase, 40000000ll);
      }
    }
  } else if (warp == kDnMmaWarp) {
    // ---------------- scale copies and MMAs, in one thread ----------------
    // They execute in order, so two buffers for the weight scales are enough.  A copier thread of its own, with
    // a barrier each way, costs more than it hides: a K block of N = 256 takes 846 cycles that way against
    // 688 here (no loads; 512 of MMAs).  The scales of a row tile are copied once a unit.
    const uint32_t a_lo0 = (smem_u32(smem->a[0]) & 0x3ffffu) >> 4, b_lo0 = (smem_u32(smem->b[0]) & 0x3ffffu) >> 4;
    const uint32_t sfa_lo0 = (smem_u32(smem->sfa[0]) & 0x3ffffu) >> 4, sfb_lo0 = (smem_u32(smem->sfb[0]) & 0x3ffffu) >> 4;
    const bool leader = elect_one();
    int stage = 0, buffer = 0, acc = 0, slot0 = 0;  // slot0: the unit's first K block
    uint32_t phase = 0, acc_phase = 0, slot0_phase = 0;
    while (ok && schedule.next(unit)) {
      for (int n = unit.begin; ok && n < unit.end; ++n) {
        ok = __all_sync(0xffffffffu, wait_or_abort(&smem->acc_empty[acc], acc_phase ^ 1u, smem, p.status));
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t descriptor = n + 1 == kDnTiles ? kInstrDesc<kDnLastColumns> : kInstrDesc<kDnColumns>;
        const uint32_t tmem_acc = tmem_base + static_cast<uint32_t>(acc) * kDnColumns;
#pragma unroll
        for (int kb = 0; kb < kDnKBlocks; ++kb) {
          constexpr int kMmas[kDnKBlocks] = {4, 4, kDnLastMmas};
          const int slot = slot0 + kb < kDnSlots ? slot0 + kb : slot0 + kb - kDnSlots;
          if (n == unit.begin)
            ok = wait_or_abort(&smem->a_full[slot], slot < slot0 ? slot0_phase ^ 1u : slot0_phase, smem, p.status);
          if (ok) ok = wait_or_abort(&smem->b_full[stage], phase, smem, p.status);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          if (leader) {
            const uint32_t tmem_sfa = tmem_base + kDnSfaColumn + static_cast<uint32_t>(16 * kb);
            const uint32_t tmem_sfb = tmem_base + kDnSfbColumn + static_cast<uint32_t>(buffer) * 32;
            if (n == unit.begin) {
              const uint32_t sfa = sfa_lo0 + static_cast<uint32_t>(slot) * (kSfStageBytes >> 4);
#pragma unroll
              for (int j = 0; j < kMmas[kb]; ++j) down_copy_sf(tmem_sfa + 4 * j, sfa + 32 * j);
            }
            const uint32_t sfb = sfb_lo0 + static_cast<uint32_t>(stage) * (kDnWeightSfBytes >> 4);
            const uint32_t a = a_lo0 + static_cast<uint32_t>(slot) * (kDnTokenBytes >> 4);
            const uint32_t b = b_lo0 + static_cast<uint32_t>(stage) * (kDnWeightBytes >> 4);
#pragma unroll
            for (int j = 0; j < kMmas[kb]; ++j) {
              down_copy_sf(tmem_sfb + 8 * j, sfb + 32 * j);
              down_copy_sf(tmem_sfb + 8 * j + 4, sfb + 128 + 32 * j);
            }
#pragma unroll
            for (int j = 0; j < kMmas[kb]; ++j)
              down_mma(tmem_acc, a + 2 * j, b + 2 * j, tmem_sfa + 4 * j, tmem_sfb + 8 * j, descriptor, (kb | j) != 0);
            tc_commit(&smem->b_empty[stage]);
            if (n + 1 == unit.end) tc_commit(&smem->a_empty[slot]);
            if (kb + 1 == kDnKBlocks) tc_commit(&smem->acc_full[acc]);
          }
          buffer ^= 1;
          if (++stage == kDnStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (++acc == kDnAccStages) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
      slot0 += kDnKBlocks;
      if (slot0 >= kDnSlots) {
        slot0 -= kDnSlots;
        slot0_phase ^= 1u;
      }
    }
  } else if (warp >= kDnEpilogueWarp) {
    // ---------------- epilogue ----------------
    // 64 columns of 16 rows at a time.
    static_assert(kDnEpilogueWarps == 4, "a quarter of the rows each");
    const int quarter = warp & 3;                        // the tensor-memory lanes this warp may read
    constexpr int kParts = 2;                            // 16-row parts of the quarter
    const int row_in_tile = quarter * 32 + (lane >> 2);  // and 8, 16 and 24 further down
    const uint32_t tmem_rows = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    unsigned long long keep_in_l2;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(keep_in_l2));
    int acc = 0;
    uint32_t acc_phase = 0;
    while (ok && schedule.next(unit)) {
      const int row0 = p.expert_offsets[unit.expert] + unit.tile * kTileM - p.scale_row_offsets[unit.expert] + row_in_tile;
      const int row_end = p.expert_offsets[unit.expert + 1];
      const float alpha = p.alpha[unit.expert];
      for (int n = unit.begin; n < unit.end; ++n) {
        ok = __all_sync(0xffffffffu, wait_or_abort(&smem->acc_full[acc], acc_phase, smem, p.status));
        if (!ok) break;
        tc_fence_after_sync();
        const int groups = n + 1 == kDnTiles ? kDnLastColumns / 64 : kDnColumns / 64;
#pragma unroll 1
        for (int part = 0; part < kParts; ++part) {
#pragma unroll 1
          for (int group = 0; group < groups; ++group) {
            uint32_t r[32];
            tmem_load_16x64(tmem_rows + (static_cast<uint32_t>(part * 16) << 16) + static_cast<uint32_t>(acc) * kDnColumns + 64 * group, r);
            tmem_load_wait(r);
            if (part + 1 == kParts && group + 1 == groups) {
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(&smem->acc_empty[acc]);
            }
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              const int row = row0 + 16 * part + 8 * half;
              if (row >= row_end) continue;
              uint32_t v[8];
#pragma unroll
              for (int g = 0; g < 8; ++g)
                v[g] = pack_bf16x2(__fmul_rn(alpha, __uint_as_float(r[4 * g + 2 * half])),
                                   __fmul_rn(alpha, __uint_as_float(r[4 * g + 2 * half + 1])));
              const int column = n * kDnColumns + 64 * group + (lane & 3) * 16;
              if (p.row_dest) {
                // expert-parallel combine: the row goes straight to its source rank's buffer
                uint4* remote = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.row_dest[row]) + column);
                remote[0] = make_uint4(v[0], v[1], v[2], v[3]);
                remote[1] = make_uint4(v[4], v[5], v[6], v[7]);
              } else {
                // read back by the weighted reduce right after this launch: L2 is asked to keep it
                asm volatile("st.global.L2::cache_hint.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8}, %9;" ::"l"(
                                 p.out + static_cast<size_t>(row) * kHidden + column),
                             "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "l"(keep_in_l2)
                             : "memory");
              }
            }
          }
        }
        if (++acc == kDnAccStages) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == kDnMmaWarp) {
    tc_fence_after_sync();
    __syncwarp();
    tmem_dealloc(tmem_base, kDnTmemColumns);
  }
}

// w2 block scales re-tiled for the kernel's column order: [expert][tile of 192 columns][K block][rows 0..127,
// 128..191][4 atoms of 512 bytes], byte (n%32)*16 + (n/32)*4 + k of an atom being the scale of MMA column n of
// that part (zero past K = 704 and past the tile).  One thread per byte.
__global__ void retile_w2_scales_kernel(const uint8_t* __restrict__ sidecar, uint8_t* __restrict__ tiled, int experts) {
  constexpr int groups = kInter / 16;  // 44
  const size_t index = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (index >= static_cast<size_t>(experts) * kDnTiles * kDnKBlocks * kDnWeightSfBytes) return;
  const int byte = static_cast<int>(index % kSfAtomBytes);
  size_t rest = index / kSfAtomBytes;
  const int mma = static_cast<int>(rest % 4);
  rest /= 4;
  const int half = static_cast<int>(rest % 2);
  rest /= 2;
  const int kb = static_cast<int>(rest % kDnKBlocks);
  rest /= kDnKBlocks;
  const int tile = static_cast<int>(rest % kDnTiles);
  const int expert = static_cast<int>(rest / kDnTiles);
  const int n = ((byte & 15) >> 2) * 32 + (byte >> 4);
  const int column = (n & 64) + ((n >> 1) & 3) * 16 + ((n >> 3) & 7) * 2 + (n & 1);
  const int atom = kb * 4 + mma;
  const int local = half * 128 + column, global = tile * kDnColumns + local;
  tiled[index] = atom < kDnAtoms && local < kDnColumns && global < kHidden ? sidecar[static_cast<size_t>(expert) * kHidden * groups +
                                           sf_offset(global, atom * 4 + (byte & 3), groups)]
                                 : 0;
}

}  // namespace

size_t retiled_w2_scale_bytes(int experts) {
  return static_cast<size_t>(experts) * kDnTiles * kDnKBlocks * kDnWeightSfBytes;
}

void launch_retile_w2_scales(const uint8_t* sidecar_scales, uint8_t* tiled, int experts, cudaStream_t stream) {
  const size_t total = retiled_w2_scale_bytes(experts);
  retile_w2_scales_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, stream>>>(sidecar_scales, tiled, experts);
}

int prepare_grouped_down() {
  return static_cast<int>(cudaFuncSetAttribute(grouped_down_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(kDnSmemBytes)));
}

void launch_grouped_down(const GemmOperands& op, const RoutePlan& plan, int sm_count, cudaStream_t stream) {
  DownParams p{};
  p.a_scales = op.a_scales;
  p.b_scales = op.down_scales;
  p.alpha = op.alpha;
  p.out = static_cast<__nv_bfloat16*>(op.out);
  p.row_dest = op.row_dest;
  p.tile_expert = plan.tile_expert;
  p.expert_offsets = plan.expert_offsets;
  p.scale_row_offsets = plan.scale_row_offsets;
  p.num_m_tiles = plan.num_m_tiles;
  p.tile_first = plan.tile_first;
  p.status = plan.status;
  p.early_weights = op.early_weights;
  if (op.serial_launch) {
    grouped_down_kernel<<<sm_count, kDnThreads, kDnSmemBytes, stream>>>(op.map_a, op.map_b_down, p);
    return;
  }
  launch_chained(grouped_down_kernel, dim3(sm_count), dim3(kDnThreads), kDnSmemBytes, stream, op.map_a, op.map_b_down, p);
}

}  // namespace gv
