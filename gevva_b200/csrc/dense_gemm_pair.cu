// The dense MLP's two FP8 projections of prefill-sized batches by CTA pairs: bf16 out[tokens, n] = E4M3 rows x E4M3 weights.
//
// What bounds it.  A 128 x 256 tile of one CTA (grouped_gemm.cu) takes in 48 KB a K block of 128 for 512 tensor-pipe cycles, and an SM
// takes in 73 bytes a cycle: 660 cycles.  A pair (tcgen05 cta_group::2, M = 256) computes 256 tokens x 256 columns with half of either
// operand in each CTA, 32 KB: 450 cycles, under the MMAs' 512.  The whole MLP, one CTA a tile -> pairs as they were first
// (us): 1 token 25.5 -> 22.8, 128 tokens 29.0 -> 24.8, 301 tokens 31.3 -> 25.1, 640 tokens 34.9 -> 30.1, 1024 tokens 38.0 -> 33.6, 2048 tokens 62.8 ->
// 54.2, 4096 tokens 106 -> 94 (of the last two 23 and 38 were its quantisers; 48 and 81 with those of today).
// 192 columns an item where that leaves the clusters less to do (the second projection at 2048 tokens: 88 items of 256 are two
// rounds of 74 clusters as 120 items of 192 are).  The weight rows are taken in the column order of grouped_gemm_down.cu, in copies of 32
// rows, so that a quad of lanes stores whole 128-byte lines of a row from registers.  Two accumulators of up to 256 columns fill
// tensor memory.  Every output is the sum of the same MMAs as in the one-CTA kernel.  The weight side waits for no earlier kernel (the MLP, us, all
// waiting -> so: 700 tokens 25.6 -> 24.7, 1024 29.4 -> 27.9, 2048 44.7 -> 41.9, 4096 77.3 -> 74.8).
//
// Roles of each CTA (8 warps): 0 fetches weights, 1 issues MMAs (in the first CTA, for both), 2 fetches activations, 4..7 the epilogue
// (a quarter of the rows each); one thread each but for the last.  Every wait is bounded.
#include "gv_common.cuh"
#include "gv_cta_pair.cuh"
#include "gv_gemm_parts.cuh"
#include "gv_launchers.h"

namespace gv {

namespace {

constexpr int kFpPieceRows = 32;
constexpr int kFpPieceBytes = kFpPieceRows * kTileKBytes;   // 4 KiB
constexpr int kFpTokenBytes = 128 * kTileKBytes;            // 16 KiB
constexpr int kFpAccStages = 2;
constexpr uint32_t kFpTmemColumns = 512;
constexpr int kFpUnroll = 2;                                // K blocks: a trip of a rolled loop takes 320 cycles whatever it loads
constexpr int kFpWeightWarp = 0, kFpMmaWarp = 1, kFpTokenWarp = 2, kFpEpilogueWarp = 4;
constexpr int kFpEpilogueWarps = 4;
constexpr int kFpThreads = (kFpEpilogueWarp + kFpEpilogueWarps) * 32;

template <int kN>
struct alignas(1024) DensePairSmem {
  static constexpr int kStages = kN == 256 ? 6 : 7;
  static constexpr int kWeightBytes = kN / 2 * kTileKBytes;  // this CTA's half
  uint8_t a[kStages][kFpTokenBytes];
  uint8_t b[kStages][kWeightBytes];
  uint64_t full[kStages];             // first CTA: the bytes have landed in both
  uint64_t empty[kStages];            // both CTAs: the MMAs that read them have completed
  uint64_t acc_full[kFpAccStages];    // both CTAs
  uint64_t acc_empty[kFpAccStages];   // first CTA: both CTAs' epilogues have copied the accumulator out
  uint32_t tmem_base;
  volatile int abort;
};

struct DensePairParams {
  __nv_bfloat16* out;
  int* status;
  int tokens, n_out;
  int k_blocks;    // of 128 bytes
  int last_mmas;   // MMAs (K = 32 each) of the last one
};

// Items are numbered row tile by row tile: the clusters that work at a time share their activations.
struct DensePairItem {
  int token0, column0;
  int pieces;  // 32-column pieces of each half: all of them but in the last item of a row
};
template <int kN>
__device__ __forceinline__ bool dense_pair_item(const DensePairParams& p, int round, uint32_t rank, DensePairItem& item) {
  const int columns = (p.n_out + kN - 1) / kN;
  const int index = round * (static_cast<int>(gridDim.x) >> 1) + (static_cast<int>(blockIdx.x) >> 1);
  const int tile = index / columns;
  item.token0 = tile * 256 + static_cast<int>(rank) * 128;
  item.column0 = (index - tile * columns) * kN;
  const int left = p.n_out - item.column0;
  item.pieces = (left < kN ? left : kN) / 2 / kFpPieceRows;
  return tile * 256 < p.tokens;
}

__device__ __forceinline__ void dense_pair_mma(uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t descriptor, uint32_t accumulate) {
  constexpr uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);  // 8 rows x 128 B, 128B swizzle
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"((static_cast<uint64_t>(hi) << 32) | a_lo), "l"((static_cast<uint64_t>(hi) << 32) | b_lo), "r"(descriptor), "r"(accumulate)
      : "memory");
}

template <int kN>
__global__ void __launch_bounds__(kFpThreads, 1)
dense_fp8_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const DensePairParams p) {
  using Smem = DensePairSmem<kN>;
  constexpr int kStages = Smem::kStages;
  constexpr int kPieces = kN / 2 / kFpPieceRows;
  extern __shared__ uint8_t smem_raw[];
  Smem* smem = reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_cta_rank();
  const bool is_leader = rank == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&smem->full[s], 2);   // the first CTA's two producers each announce both CTAs' byte count
      mbar_init(&smem->empty[s], 1);
    }
    for (int s = 0; s < kFpAccStages; ++s) {
      mbar_init(&smem->acc_full[s], 1);
      mbar_init(&smem->acc_empty[s], 2 * kFpEpilogueWarps);
    }
    smem->abort = 0;
    fence_barrier_init();
    prefetch_tensor_map(&map_a);
    prefetch_tensor_map(&map_b);
  }
  // Both CTAs run and their barriers exist before either touches the other's tensor memory or arrives there.
  __syncwarp();
  cluster_sync_all();
  if (warp == kFpMmaWarp) pair_tmem_alloc(&smem->tmem_base, kFpTmemColumns);  // the whole tensor memory
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = smem->tmem_base;
  // The weights come from before the previous kernel, which let this one start after its own wait.
  if (warp != kFpWeightWarp) {
    grid_dependency_wait();
    grid_launch_dependents();
  }

  DensePairItem item;
  bool ok = true;
  if (warp == kFpWeightWarp || warp == kFpTokenWarp) {
    // ---------------- producers ----------------
    if (elect_one()) {
      const bool weight_side = warp == kFpWeightWarp;
      const uint32_t full0 = is_leader ? smem_u32(&smem->full[0]) : cluster_map_shared(smem_u32(&smem->full[0]), 0);
      int stage = 0, issued = 0;
      uint32_t phase = 0;
      for (int round = 0; ok && dense_pair_item<kN>(p, round, rank, item); ++round) {
        const uint32_t both_bytes = 2u * (weight_side ? static_cast<uint32_t>(item.pieces) * kFpPieceBytes : kFpTokenBytes);
        const int piece0 = static_cast<int>(rank) * item.pieces, group0 = item.column0 / 64;
#pragma unroll kFpUnroll
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          ok = wait_or_abort(&smem->empty[stage], phase ^ 1u, smem, p.status);
          if (!ok) break;
          const uint32_t bar = full0 + 8 * stage;
          if (is_leader) mbar_arrive_expect_tx(&smem->full[stage], both_bytes);
          if (weight_side) {
#pragma unroll
            for (int j = 0; j < kPieces; ++j)
              if (j < item.pieces)
                pair_load_piece(smem->b[stage] + j * kFpPieceBytes, &map_b, bar, kb * kTileKBytes, (piece0 + j) & 1,
                                        group0 + ((piece0 + j) >> 1));
          } else {
            pair_load(smem->a[stage], &map_a, bar, kb * kTileKBytes, item.token0);  // (rows past the end are not stored)
          }
          ++issued;
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (!ok && is_leader) {
        // Unwinding: the copies already issued (by either CTA) land before shared memory is given up; the second CTA stays
        // resident until the cluster barrier at the end.
        const int pending = issued < kStages ? issued : kStages;
        for (int i = 0; i < pending; ++i) {
          if (--stage < 0) {
            stage = kStages - 1;
            phase ^= 1u;
          }
          mbar_wait_bounded(&smem->full[stage], phase, 40000000ll);
        }
      }
    }
    __syncwarp();
  } else if (warp == kFpMmaWarp) {
    // ---------------- first CTA: MMAs for both, in one thread ----------------
    if (is_leader && elect_one()) {
      const uint32_t a_lo0 = (smem_u32(smem->a[0]) & 0x3ffffu) >> 4, b_lo0 = (smem_u32(smem->b[0]) & 0x3ffffu) >> 4;
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool landed = false;  // the next stage's bytes have been seen
      for (int round = 0; ok && dense_pair_item<kN>(p, round, rank, item); ++round) {
        ok = wait_or_abort(&smem->acc_empty[acc], acc_phase ^ 1u, smem, p.status);
        if (!ok) break;
        tc_fence_after_sync();
        // fp32 accumulation (bit 4), E4M3 x E4M3, both K-major; N at [17,23) in units of 8, M = 256 at [24,29) in units of 16
        const uint32_t descriptor = (1u << 4) | (static_cast<uint32_t>(item.pieces * 2 * kFpPieceRows >> 3) << 17) | (static_cast<uint32_t>(256 >> 4) << 24);
        const uint32_t tmem_acc = tmem_base + static_cast<uint32_t>(acc) * kN;
#pragma unroll kFpUnroll
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!landed) ok = wait_or_abort(&smem->full[stage], phase, smem, p.status);
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t a = a_lo0 + static_cast<uint32_t>(stage) * (kFpTokenBytes >> 4);
          const uint32_t b = b_lo0 + static_cast<uint32_t>(stage) * (Smem::kWeightBytes >> 4);
          uint64_t* const empty = &smem->empty[stage];
          if (++stage == kStages) {
            stage = 0;
            phase ^= 1u;
          }
          const int mmas = kb + 1 == p.k_blocks ? p.last_mmas : 4;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j < mmas) dense_pair_mma(tmem_acc, a + 2 * j, b + 2 * j, descriptor, (kb | j) != 0 ? 1u : 0u);
          landed = mbar_try_wait(&smem->full[stage], phase);
          pair_commit_both(empty);
          if (kb + 1 == p.k_blocks) pair_commit_both(&smem->acc_full[acc]);
        }
        if (++acc == kFpAccStages) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
    }
    __syncwarp();
  } else if (warp >= kFpEpilogueWarp) {
    // ---------------- epilogue: 64 columns of 16 rows at a time ----------------
    const int quarter = warp & 3;                        // the tensor-memory lanes this warp may read
    const int row_in_tile = quarter * 32 + (lane >> 2);  // and 8, 16 and 24 further down
    const uint32_t tmem_rows = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int round = 0; ok && dense_pair_item<kN>(p, round, rank, item); ++round) {
      ok = __all_sync(0xffffffffu, wait_or_abort(&smem->acc_full[acc], acc_phase, smem, p.status));
      if (!ok) break;
      tc_fence_after_sync();
      const int groups = item.pieces;                                        // of 64 columns
      const int warp_rows = p.tokens - item.token0 - quarter * 32;           // of this warp's quarter that exist
      const int steps = warp_rows <= 0 ? 0 : (warp_rows <= 16 ? 1 : 2) * groups;
      bool released = false;
      int step = 0;
#pragma unroll 1
      do {
        uint32_t r[32];
        const int part = step >= groups ? 1 : 0, group = step - part * groups;
        if (step < steps) {
          tmem_load_16x64(tmem_rows + (static_cast<uint32_t>(part * 16) << 16) + static_cast<uint32_t>(acc) * kN + 64 * group, r);
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
          const int token = item.token0 + row_in_tile + 16 * part + 8 * half;
          if (token >= p.tokens) continue;
          uint32_t v[8];
#pragma unroll
          for (int g = 0; g < 8; ++g)
            v[g] = pack_bf16x2(__uint_as_float(r[4 * g + 2 * half]), __uint_as_float(r[4 * g + 2 * half + 1]));
          asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(
                           p.out + static_cast<size_t>(token) * p.n_out + item.column0 + 64 * group + (lane & 3) * 16),
                       "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                       : "memory");
        }
        ++step;
      } while (!released);
      if (++acc == kFpAccStages) {
        acc = 0;
        acc_phase ^= 1u;
      }
    }
  }

  tc_fence_before_sync();
  // Both CTAs stay until neither can still receive a remote arrive, a copy or a commit.
  cluster_sync_all();
  if (warp == kFpMmaWarp) {
    tc_fence_after_sync();
    __syncwarp();
    pair_tmem_dealloc(tmem_base, kFpTmemColumns);
  }
}

template <int kN>
constexpr size_t dense_pair_smem_bytes() {
  return sizeof(DensePairSmem<kN>) + 1024;
}
static_assert(dense_pair_smem_bytes<256>() <= 232448 && dense_pair_smem_bytes<192>() <= 232448, "shared memory budget");

// A cluster's rounds of items times what a K block of an item takes: its MMAs, or its 16 KB of activations and its weights at 73 bytes a
// cycle, whichever is longer.
int dense_pair_cost(int tokens, int n_out, int columns, int clusters) {
  const int items = (tokens + 255) / 256 * ((n_out + columns - 1) / columns);
  return (items + clusters - 1) / clusters * (columns == 256 ? 512 : 393);
}

template <int kN>
void launch_variant(const GemmOperands& op, const DensePairParams& p, int sm_count, cudaStream_t stream) {
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(sm_count & ~1));
  config.blockDim = dim3(kFpThreads);
  config.dynamicSmemBytes = dense_pair_smem_bytes<kN>();
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
  cudaLaunchKernelEx(&config, dense_fp8_pair_kernel<kN>, op.map_a, op.map_down_pieces, p);
}

}  // namespace

int prepare_dense_pairs() {
  cudaError_t e = cudaFuncSetAttribute(dense_fp8_pair_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(dense_pair_smem_bytes<256>()));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(dense_fp8_pair_kernel<192>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(dense_pair_smem_bytes<192>()));
  return static_cast<int>(e);
}

void launch_dense_pairs(const GemmOperands& op, int tokens, int* status, int sm_count, cudaStream_t stream) {
  DensePairParams p{};
  p.out = static_cast<__nv_bfloat16*>(op.out);
  p.status = status;
  p.tokens = tokens;
  p.n_out = op.n_out;
  p.k_blocks = (op.k_in + kTileKBytes - 1) / kTileKBytes;
  p.last_mmas = (op.k_in - (p.k_blocks - 1) * kTileKBytes) / 32;
  const int clusters = sm_count / 2;
  if (dense_pair_cost(tokens, op.n_out, 192, clusters) < dense_pair_cost(tokens, op.n_out, 256, clusters))
    launch_variant<192>(op, p, sm_count, stream);
  else
    launch_variant<256>(op, p, sm_count, stream);
}

}  // namespace gv
