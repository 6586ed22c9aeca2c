// Router projection fused with top-8 routing, for sm_100a.
//
// The reference computes the router logits with a library GEMM and then routes
// (src/cuda/runtime/prefill.cuh:414-422, :1203-1210: cublasGemmEx / cuBLASLt FP8
// [tokens,2816] x [128,2816]^T -> bf16 [tokens,128], followed by
// route_128_top8_kernel<<<tokens,128>>>).  Here both are one kernel and the logits never
// reach HBM: tokens sit on MMA-M (16 to 128 per tile), the 128 experts on MMA-N, K = 2816.
//
// A tile (of 16, 32 or 64 tokens in batches of up to 2048) has its K range cut into four slices (two, or one, in batches of many tiles;
// eight for batches of at most 512 tokens), of which each CTA of the tile's cluster has one, or two where clusters of one CTA a slice
// would not all run at once: a
// 4096-token batch runs on 128 SMs and a decode-sized batch streams the router matrix through
// eight SMs instead of one.  Each
// CTA accumulates its slices in tensor memory, each by itself (tcgen05.mma kind::f16 for bf16 operands,
// kind::f8f6f4 for E4M3).  Tile row r belongs to CTA r % split of the cluster: every CTA stores
// its fp32 partial sums (128 a row and slice) row by row straight into the owners' shared memory (posted
// st.shared::cluster stores, behind a cluster barrier that says that the owners run), and after a second cluster barrier each owner sums the partials of its
// rows (a tile's / split) in the order of the slices (a fixed order: results do not depend on timing), adds the optional
// per-expert bias, rounds to bf16 as the GEMM would have stored it, and routes its rows (gv_route.cuh): a warp per
// token where it has at most two a warp, else four lanes per token.
//
// Roles per CTA: warp 0 TMA producer, warp 1 MMA issuer and owner of tensor memory, warps
// from 2 on epilogue (thread = accumulator row, the columns shared by warps of equal lanes).  Every mbarrier wait is bounded (status word
// kWaitTimeout); the cluster barrier is reached by every thread whatever happened before.
#include "gv_common.cuh"
#include "gv_launchers.h"
#include "gv_route.cuh"

namespace gv {

namespace {

// K slices per token tile = CTAs per cluster x slices of a CTA: 8 for small batches, else 4, 2 or 1, with one slice a CTA where that
// keeps the launch within one wave of SMs (a tile's pass is a chain of latencies, so waves cost more
// than depth), else two.
// Epilogue warps.  CTAs of 128-row tiles that keep 64 or 128 rows for themselves route them four lanes a row in one pass of sixteen warps
// (four -> sixteen, us alone: 6000 tokens 15.8 -> 14.6, 8192 16.9 -> 15.7, 12000 25.3 -> 22.0, 16384 28.5 -> 25.2; a layer of 16384 tokens 793 -> 777; with 32 rows,
// up to 4608 tokens, 12.2 -> 12.5 at 4096).  64 rows keep eight busy (four -> eight, us alone: 37 tokens 5.9 -> 5.5, 64 6.7 -> 6.4, 613 9.0 -> 8.2, 1024 9.2 -> 8.4,
// 2048 10.0 -> 9.1); with fewer rows eight are 0.1 slower than four.
template <int kRows, int kSplit> constexpr int kRpEpilogueWarps = kRows == 64 ? 8 : kRows == 128 && kSplit <= 2 ? 16 : 4;
template <int kRows, int kSplit> constexpr int kRpThreads = (2 + kRpEpilogueWarps<kRows, kSplit>) * 32;
// Rows of a tile.  In batches of up to 2048 tokens the launch is a chain of latencies, and the fewer rows a cluster has, the fewer partial sums
// each CTA has to send, reduce and route.  128 -> 64 rows, us alone: 9.7 -> 6.8 at 128 and 200 tokens, 10.2 -> 7.6 at 512, 10.2 -> 9.3 at 1024, 10.5 -> 9.7
// at 2048; above, the clusters no longer run all at once (2368 tokens: 11.0 against 17.3).  64 -> 32 rows: 37 tokens 5.5 -> 5.2, 64 6.2 -> 5.4,
// 200 6.4 -> 5.6, 400 6.7 -> 5.8, but 512, whose 16 clusters of eight do not run all at once, 6.7 -> 10.3.  32 -> 16 rows: 37 tokens 5.2 -> 4.9,
// 64 5.4 -> 4.9, 128 5.4 -> 5.0; whole layers 37 tokens 69.6 -> 69.2 us, 64 75.3 -> 75.1, 128 76.4 -> 76.6, each
// hardly beyond its spread: with more tokens the experts' CTAs start late on the SMs of a router's CTAs, so 16 rows are taken up to 64 tokens only.
// The K split, which decides the order of the sums, depends on the number of 128-row tiles either way.
constexpr int kSmallTile = 64, kSmallTileTokens = 2048;
constexpr int tile_rows(int tokens) { return tokens <= 64 ? 16 : tokens <= 400 ? 32 : tokens <= kSmallTileTokens ? kSmallTile : kTileM; }
template <int kRows, int kSplit> constexpr int kWarpRows = 2 * kRpEpilogueWarps<kRows, kSplit>;  // rows of a CTA up to which a warp routes a row (two each); above, a quad of lanes does
// 128-row tiles whose clusters of four, or of two, all run at once on 148 SMs (a CTA fills an SM, and a cluster lies within a GPC).  With more, half as many
// CTAs a tile sum two slices of K each, so that the sums stay the same up to the number of tiles from which K has fewer slices (a second wave of the clusters
// before, us alone: 4352 tokens 21.3 -> 15.8, 5120 21.8 -> 16.0, 9600 29.9 -> 24.6; a layer of 4700 tokens 283.9 -> 280.3, of 10000 492.5 -> 485.3).
constexpr int kTilesOfFour = 33, kFourSlicesTiles = 40, kTilesOfTwo = 74, kTwoSlicesTiles = 80;
constexpr int kRpTileBytes = kTileM * kTileKBytes;  // 16 KiB: 128 rows of one 128-byte K block

// kRows: token rows of a tile.  Below 128, with eight CTAs a tile, the five or six K blocks of each all fit the ring; the MMA, whose
// M is 128, reads what lies behind the tile (always inside this structure) as its further rows, whose results nobody looks at.
// kSlices: K slices of a CTA, summed up for themselves.
template <int kRows, int kSlices>
struct alignas(1024) RouterSmem {
  static constexpr int kStages = kRows <= 64 ? 6 : kSlices == 1 ? 5 : 3;
  static constexpr int kTokenBytes = kRows * kTileKBytes;
  uint8_t a[kStages][kTokenBytes];
  uint8_t b[kStages][kRpTileBytes];
  // Partial sums of this CTA's rows as received from the CTAs of the cluster (its own included):
  // [source][local row][128 floats]; the 16-byte chunks of a row are permuted
  // (received_chunk_position) so that neither the row-wise stores nor the reduce's reads, where
  // four lanes share a row, meet in a bank.
  float received[kSlices * kRows * kExperts];   // [kSplit * kSlices][kRows / kSplit rows][128 floats]
  uint64_t full[kStages];
  uint64_t empty[kStages];
  uint64_t acc_full[kSlices];
  uint32_t tmem_base;
  volatile int abort;
  __nv_bfloat16 expert_scale[kExperts];
};

// Position of 16-byte chunk `chunk` (0..31) inside local row `row`: the chunk's low three bits are
// XORed with (row + 2 * (chunk / 8)) % 8.  For a fixed chunk, eight consecutive rows fall into eight
// different bank groups (the stores); for a fixed chunk % 8, two consecutive rows times the four
// column quarters do too (the loads of a quarter-warp).
__device__ __forceinline__ int received_chunk_position(int chunk, int row) {
  return chunk ^ ((row + 2 * (chunk >> 3)) & 7);
}

template <int kRows, int kSlices> constexpr size_t router_smem_bytes() { return sizeof(RouterSmem<kRows, kSlices>) + 1024; }
static_assert(router_smem_bytes<64, 1>() <= 232448 && router_smem_bytes<128, 1>() <= 232448 && router_smem_bytes<128, 2>() <= 232448,
              "shared memory budget of one sm_100 CTA");

struct RouterParams {
  const float* bias;                   // optional f32 [128], added before the bf16 rounding
  const __nv_bfloat16* expert_scale;   // bf16 [128]
  float* weights;                      // f32 [tokens, 8]
  int* ids;                            // i32 [tokens, 8]
  __nv_bfloat16* logits_out;           // optional bf16 [tokens, 128]
  const float* activation_scales;      // E4M3 form: f32 [tokens]
  const float* weight_scale;           // E4M3 form: f32 [1]
  int* status;                         // optional device status word
  int tokens;
  int k_blocks;                        // 128-byte K blocks per row
};

// Instruction descriptors: fp32 accumulate (bit 4), both operands K-major, N at [17,23) in units
// of 8, M at [24,29) in units of 16; operand formats at [7,10) and [10,13): BF16 = 1 in
// kind::f16, E4M3 = 0 in kind::f8f6f4.
constexpr uint32_t kIdescBase = (1u << 4) | (static_cast<uint32_t>(kExperts >> 3) << 17) |
                                (static_cast<uint32_t>(kTileM >> 4) << 24);
constexpr uint32_t kIdescBf16 = kIdescBase | (1u << 7) | (1u << 10);
constexpr uint32_t kIdescE4m3 = kIdescBase;

// The four MMAs of one 128-byte K block (K = 16 bf16 or 32 E4M3 values each, 32 bytes apart).
template <bool kFp8>
__device__ __forceinline__ void issue_router_k_block(uint32_t tmem_acc, uint32_t a_lo, uint32_t b_lo,
                                                     uint32_t accumulate) {
  constexpr uint32_t hi = (1024u >> 4) | (1u << 14) | (2u << 29);  // 8 rows x 128 B groups, 128B swizzle
#define GV_RP_MMA(kind, j, pred)                                     \
  "add.u32 lo, %1, " #j "*2;\n\t"                                    \
  "mov.b64 d0, {lo, %3};\n\t"                                        \
  "add.u32 lo, %2, " #j "*2;\n\t"                                    \
  "mov.b64 d1, {lo, %3};\n\t"                                        \
  "tcgen05.mma.cta_group::1.kind::" kind " [%0], d0, d1, %4, " pred ";\n\t"
#define GV_RP_BLOCK(kind)                                                                            \
  asm volatile("{\n\t.reg .pred p, pt;\n\t.reg .b32 lo;\n\t.reg .b64 d0, d1;\n\t"                     \
               "setp.ne.b32 p, %5, 0;\n\tsetp.eq.b32 pt, 0, 0;\n\t"                                   \
               GV_RP_MMA(kind, 0, "p") GV_RP_MMA(kind, 1, "pt") GV_RP_MMA(kind, 2, "pt")              \
               GV_RP_MMA(kind, 3, "pt") "}"                                                           \
               ::"r"(tmem_acc), "r"(a_lo), "r"(b_lo), "r"(hi), "r"(kFp8 ? kIdescE4m3 : kIdescBf16),    \
                 "r"(accumulate)                                                                      \
               : "memory")
  if constexpr (kFp8) {
    GV_RP_BLOCK("f8f6f4");
  } else {
    GV_RP_BLOCK("f16");
  }
#undef GV_RP_BLOCK
#undef GV_RP_MMA
}

template <bool kFp8, int kSplit, int kRows, int kSlices>
__global__ void __launch_bounds__(kRpThreads<kRows, kSplit>, 1)
route_project_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                     const RouterParams p) {
  using Smem = RouterSmem<kRows, kSlices>;
  constexpr int kRpStages = Smem::kStages;
  extern __shared__ uint8_t smem_raw[];
  Smem* smem = reinterpret_cast<Smem*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_cta_rank();
  constexpr int kOwnRows = kRows / kSplit;   // tile rows this CTA reduces and routes
  const int m_tile = static_cast<int>(blockIdx.x) / kSplit;
  constexpr int kSources = kSplit * kSlices;
  const int slice0 = static_cast<int>(rank) * kSlices;
  const int kb_begin = slice0 * p.k_blocks / kSources;
  const int kb_end = (slice0 + kSlices) * p.k_blocks / kSources;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kRpStages; ++s) {
      mbar_init(&smem->full[s], 1);
      mbar_init(&smem->empty[s], 1);
    }
    for (int s = 0; s < kSlices; ++s) mbar_init(&smem->acc_full[s], 1);
    smem->abort = 0;
    fence_barrier_init();
    prefetch_tensor_map(&map_x);
    prefetch_tensor_map(&map_w);
  }
  if (warp == 1) {
    tmem_alloc(&smem->tmem_base, kSlices * kExperts);
    tmem_relinquish();
  }
  // The next kernel of the stream (launched with programmatic serialization) may take its place on
  // the SMs now; it waits at its own top for this grid to complete.
  grid_launch_dependents();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  // A CTA's shared memory may be written by its peers once it runs: every thread says so here, and waits for all others where its
  // warp would store to them (the wait is over by then: it lies behind the K blocks).
  if (kSplit > 1) cluster_arrive_relaxed();
  const uint32_t tmem_base = smem->tmem_base;
  // While the previous kernel drains, this CTA's slice of the router matrix is asked into L2 (a hint: the
  // loads themselves come after the wait); a model's other weights have pushed it out since last time.
  if (m_tile == 0 && warp == 0 && elect_one())
    for (int kb = kb_begin; kb < kb_end; ++kb)
      asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(&map_w), "r"(kb * kTileKBytes), "r"(0)
                   : "memory");
  grid_dependency_wait();  // the previous kernel of the stream has completed and its writes are visible

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    int stage = 0;
    uint32_t phase = 0;
    int issued = 0;
    bool ok = true;
    for (int kb = kb_begin; kb < kb_end; ++kb) {
      ok = __all_sync(0xffffffffu, wait_or_abort(&smem->empty[stage], phase ^ 1u, smem, p.status));
      if (!ok) break;
      if (elect_one()) {
        mbar_arrive_expect_tx(&smem->full[stage], static_cast<uint32_t>(Smem::kTokenBytes + kRpTileBytes));
        tma_load_2d(smem->a[stage], &map_x, &smem->full[stage], kb * kTileKBytes, m_tile * kRows);
        tma_load_2d(smem->b[stage], &map_w, &smem->full[stage], kb * kTileKBytes, 0);
      }
      __syncwarp();
      ++issued;
      if (++stage == kRpStages) {
        stage = 0;
        phase ^= 1u;
      }
    }
    if (!ok && lane == 0) {
      // let the copies already issued land before shared memory is given up
      const int pending = issued < kRpStages ? issued : kRpStages;
      int s = stage;
      uint32_t ph = phase;
      for (int i = 0; i < pending; ++i) {
        if (--s < 0) {
          s = kRpStages - 1;
          ph ^= 1u;
        }
        mbar_wait_bounded(&smem->full[s], ph, 40000000ll);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    int stage = 0;
    uint32_t phase = 0;
    const uint32_t a_lo0 = (smem_u32(smem->a[0]) & 0x3ffffu) >> 4;
    const uint32_t b_lo0 = (smem_u32(smem->b[0]) & 0x3ffffu) >> 4;
    const bool leader = elect_one();
    int slice = 0;
    bool fresh = true;  // the slice's first K block
    for (int kb = kb_begin; kb < kb_end; ++kb) {
      if (!wait_or_abort(&smem->full[stage], phase, smem, p.status)) break;
      if (leader) {
        issue_router_k_block<kFp8>(tmem_base + static_cast<uint32_t>(slice) * kExperts, a_lo0 + static_cast<uint32_t>(stage) * (Smem::kTokenBytes >> 4),
                                   b_lo0 + static_cast<uint32_t>(stage) * (kRpTileBytes >> 4),
                                   fresh ? 0u : 1u);
        tc_commit(&smem->empty[stage]);
      }
      fresh = false;
      if (kb + 1 == (slice0 + slice + 1) * p.k_blocks / kSources) {
        if (leader) tc_commit(&smem->acc_full[slice]);
        ++slice;
        fresh = true;
      }
      if (++stage == kRpStages) {
        stage = 0;
        phase ^= 1u;
      }
    }
  } else {
    // ---------------- epilogue, part 1: partial sums to the rows' owners ----------------
    // (the per-expert scale, which part 2 would otherwise look up behind its last comparison)
    if (threadIdx.x - 64 < kExperts) smem->expert_scale[threadIdx.x - 64] = p.expert_scale[threadIdx.x - 64];
    const int quarter = warp & 3;  // the tensor-memory lanes this warp may read
    constexpr int kParts = 4 / (kRpEpilogueWarps<kRows, kSplit> / 4);  // the columns of a row are shared by the quarter's warps
    const int first_part = (warp - 2) / 4 * kParts;
    const int row = quarter * 32 + lane;
    const int owner = row % kSplit;
    const int owner_row = row / kSplit;
    // rows past the end of the batch (most rows of a decode-sized batch) are not sent; the
    // tensor-memory loads are warp-wide, so a warp takes part if any of its 32 rows exists
    const bool row_exists = row < kRows && m_tile * kRows + row < p.tokens;
    const bool warp_has_rows = quarter * 32 < kRows && m_tile * kRows + quarter * 32 < p.tokens;
    if (kSplit > 1) {
      __syncwarp();
      cluster_wait();
    }
#pragma unroll 1
    for (int slice = 0; slice < kSlices; ++slice) {
      if (!warp_has_rows || !__all_sync(0xffffffffu, wait_or_abort(&smem->acc_full[slice], 0, smem, p.status))) break;
      tc_fence_after_sync();
      const uint32_t remote_row =
          cluster_map_shared(smem_u32(smem->received + ((slice0 + slice) * kOwnRows + owner_row) * kExperts),
                             static_cast<uint32_t>(owner));
#pragma unroll 1
      for (int part = first_part; part < first_part + kParts; ++part) {
        uint32_t r[32];
        tmem_load_32x32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + slice * kExperts + part * 32, r);
        tmem_load_wait(r);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int chunk = part * 8 + i;
          if (row_exists)
            cluster_store_uint4(remote_row + (static_cast<uint32_t>(received_chunk_position(chunk, owner_row)) << 4),
                              make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]));
        }
      }
      tc_fence_before_sync();
    }
  }

  if (kSplit > 1 && warp < 2) {  // (the epilogue's warps have waited for the cluster's start above)
    __syncwarp();
    cluster_wait();
  }
  // Every thread of every CTA of the cluster arrives here, also after a failed wait.  The barrier
  // orders the posted stores above before the owners' reads below; after it no CTA touches another
  // CTA's shared memory, so a CTA may finish while its peers still work.
  cluster_sync_all();

  if (warp >= 2 && !smem->abort) {
    // ---------------- epilogue, part 2: reduce this CTA's rows and route them ----------------
    const int tile_rows = p.tokens - m_tile * kRows;   // may exceed the tile
    // rows kSplit * i + rank < tile_rows
    const int own_rows = tile_rows >= kRows ? kOwnRows : (tile_rows - static_cast<int>(rank) + kSplit - 1) / kSplit;
    constexpr int kWarps = kRpEpilogueWarps<kRows, kSplit>;
    const bool few = kOwnRows <= kWarpRows<kRows, kSplit> || own_rows <= kWarpRows<kRows, kSplit>;
    if (few) {
      // a few rows: one warp per row, four logits a lane (a third of the quads' chain)
      for (int row_local = warp - 2; row_local < own_rows; row_local += kWarps) {
        const int token = m_tile * kRows + row_local * kSplit + static_cast<int>(rank);
        float4 acc = make_float4(0, 0, 0, 0);
#pragma unroll
        for (int source = 0; source < kSources; ++source) {
          const float4 v = reinterpret_cast<const float4*>(
              smem->received + (source * kOwnRows + row_local) * kExperts)[received_chunk_position(lane, row_local)];
          acc = source == 0 ? v
                            : make_float4(__fadd_rn(acc.x, v.x), __fadd_rn(acc.y, v.y), __fadd_rn(acc.z, v.z), __fadd_rn(acc.w, v.w));
        }
        if (p.bias) {
          const float4 b = __ldg(reinterpret_cast<const float4*>(p.bias) + lane);
          acc = make_float4(__fadd_rn(acc.x, b.x), __fadd_rn(acc.y, b.y), __fadd_rn(acc.z, b.z), __fadd_rn(acc.w, b.w));
        }
        const __nv_bfloat162 lo = __floats2bfloat162_rn(acc.x, acc.y);
        const __nv_bfloat162 hi = __floats2bfloat162_rn(acc.z, acc.w);
        const uint2 packed = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        if (p.logits_out) reinterpret_cast<uint2*>(p.logits_out + static_cast<size_t>(token) * kExperts)[lane] = packed;
        const float rescale = kFp8 ? __fmul_rn(p.activation_scales[token], p.weight_scale[0]) : 1.0f;
        route_top8_warp(packed, lane, kFp8, rescale, smem->expert_scale, p.weights + static_cast<size_t>(token) * kTopK,
                        p.ids + static_cast<size_t>(token) * kTopK);
      }
    }
    if constexpr (kOwnRows > kWarpRows<kRows, kSplit>) if (!few) {
    static_assert(kOwnRows % 8 == 0 && kOwnRows <= 8 * kWarps, "128-row tiles: a row for every four lanes, in one pass");
    const int t = threadIdx.x - 64;
    const int part = t & 3;         // columns [32 * part, 32 * part + 32)
    if (8 * (warp - 2) < kOwnRows && 8 * (warp - 2) < own_rows) {
      const int row_local = t >> 2;   // tile row kSplit * row_local + rank
      const int token = m_tile * kRows + row_local * kSplit + static_cast<int>(rank);
      const bool valid = token < p.tokens;
      float4 acc[8];
#pragma unroll
      for (int source = 0; source < kSources; ++source) {
        const float4* source_row =
            reinterpret_cast<const float4*>(smem->received + (source * kOwnRows + row_local) * kExperts);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 v = source_row[received_chunk_position(part * 8 + i, row_local)];
          if (source == 0) {
            acc[i] = v;
          } else {
            acc[i].x = __fadd_rn(acc[i].x, v.x);
            acc[i].y = __fadd_rn(acc[i].y, v.y);
            acc[i].z = __fadd_rn(acc[i].z, v.z);
            acc[i].w = __fadd_rn(acc[i].w, v.w);
          }
        }
      }
      uint32_t packed[16];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float4 v = acc[i];
        if (p.bias) {
          const float4 b = __ldg(reinterpret_cast<const float4*>(p.bias) + part * 8 + i);
          v.x = __fadd_rn(v.x, b.x);
          v.y = __fadd_rn(v.y, b.y);
          v.z = __fadd_rn(v.z, b.z);
          v.w = __fadd_rn(v.w, b.w);
        }
        const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y);
        const __nv_bfloat162 hi = __floats2bfloat162_rn(v.z, v.w);
        packed[2 * i] = *reinterpret_cast<const uint32_t*>(&lo);
        packed[2 * i + 1] = *reinterpret_cast<const uint32_t*>(&hi);
      }
      const size_t safe_token = valid ? static_cast<size_t>(token) : 0;
      if (p.logits_out && valid) {
        uint4* out = reinterpret_cast<uint4*>(p.logits_out + safe_token * kExperts + 32 * part);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          out[i] = make_uint4(packed[4 * i], packed[4 * i + 1], packed[4 * i + 2], packed[4 * i + 3]);
      }
      // the reference's rescale of an unscaled FP8 GEMM output (routing_sampling.cuh:405-411)
      const float rescale = kFp8 ? __fmul_rn(p.activation_scales[safe_token], p.weight_scale[0]) : 1.0f;
      route_top8_quad(packed, part, kFp8, rescale, valid, smem->expert_scale, p.weights + safe_token * kTopK,
                      p.ids + safe_token * kTopK);
    }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    __syncwarp();
    tmem_dealloc(tmem_base, kSlices * kExperts);
  }
}

template <bool kFp8, int kSplit, int kRows, int kSlices = 1>
cudaError_t launch_variant(const CUtensorMap& map_x, const CUtensorMap& map_w, const RouterParams& p,
                           cudaStream_t stream) {
  static bool prepared[64] = {};
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  if (device >= 0 && device < 64 && !prepared[device]) {
    e = cudaFuncSetAttribute(route_project_kernel<kFp8, kSplit, kRows, kSlices>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(router_smem_bytes<kRows, kSlices>()));
    if (e != cudaSuccess) return e;
    prepared[device] = true;
  }
  const int m_tiles = (p.tokens + kRows - 1) / kRows;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(m_tiles * kSplit));
  config.blockDim = dim3(kRpThreads<kRows, kSplit>);
  config.dynamicSmemBytes = router_smem_bytes<kRows, kSlices>();
  config.stream = stream;
  // Clusters of kSplit CTAs; and the launch may begin while the previous kernel of the stream is
  // still running (the kernel waits at grid_dependency_wait before it reads or writes global memory),
  // so that its set-up hides behind a predecessor that lets its dependents go early.
  cudaLaunchAttribute attribute[2];
  attribute[0].id = cudaLaunchAttributeClusterDimension;
  attribute[0].val.clusterDim.x = kSplit;
  attribute[0].val.clusterDim.y = 1;
  attribute[0].val.clusterDim.z = 1;
  attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[1].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attribute;
  config.numAttrs = 2;
  return cudaLaunchKernelEx(&config, route_project_kernel<kFp8, kSplit, kRows, kSlices>, map_x, map_w, p);
}

template <bool kFp8>
cudaError_t launch_split(const CUtensorMap& map_x, const CUtensorMap& map_w, const RouterParams& p,
                         cudaStream_t stream) {
  const int m_tiles = (p.tokens + kTileM - 1) / kTileM;
  const int tile = tile_rows(p.tokens);
  if (tile == 16) return launch_variant<kFp8, 8, 16>(map_x, map_w, p, stream);
  if (tile == 32) return launch_variant<kFp8, 8, 32>(map_x, map_w, p, stream);
  if (m_tiles <= 4) return launch_variant<kFp8, 8, kSmallTile>(map_x, map_w, p, stream);
  if (tile == kSmallTile) return launch_variant<kFp8, 4, kSmallTile>(map_x, map_w, p, stream);
  if (m_tiles <= kTilesOfFour) return launch_variant<kFp8, 4, kTileM>(map_x, map_w, p, stream);
  if (m_tiles <= kFourSlicesTiles) return launch_variant<kFp8, 2, kTileM, 2>(map_x, map_w, p, stream);
  if (m_tiles <= kTilesOfTwo) return launch_variant<kFp8, 2, kTileM>(map_x, map_w, p, stream);
  if (m_tiles <= kTwoSlicesTiles) return launch_variant<kFp8, 1, kTileM, 2>(map_x, map_w, p, stream);
  return launch_variant<kFp8, 1, kTileM>(map_x, map_w, p, stream);
}

}  // namespace

int launch_route_project(const void* x, const void* router_w, bool fp8, const float* bias,
                         const void* expert_scale_bf16, float* weights, int* ids, void* logits_out,
                         const float* activation_scales, const float* weight_scale, int tokens, int* status,
                         cudaStream_t stream) {
  const uint64_t row_bytes = fp8 ? kHidden : 2 * kHidden;
  CUtensorMap map_x, map_w;
  if (!make_operand_tensor_map(&map_x, x, static_cast<uint64_t>(tokens), row_bytes, tile_rows(tokens)) ||
      !make_operand_tensor_map(&map_w, router_w, kExperts, row_bytes, kTileM))
    return static_cast<int>(cudaErrorInvalidValue);
  RouterParams p{};
  p.bias = bias;
  p.expert_scale = static_cast<const __nv_bfloat16*>(expert_scale_bf16);
  p.weights = weights;
  p.ids = ids;
  p.logits_out = static_cast<__nv_bfloat16*>(logits_out);
  p.activation_scales = activation_scales;
  p.weight_scale = weight_scale;
  p.status = status;
  p.tokens = tokens;
  p.k_blocks = static_cast<int>(row_bytes / kTileKBytes);
  const cudaError_t e = fp8 ? launch_split<true>(map_x, map_w, p, stream) : launch_split<false>(map_x, map_w, p, stream);
  return static_cast<int>(e);
}

}  // namespace gv
