// Grouped GEMM on CTA pairs (tcgen05 cta_group::2) for the NT, NN and TN layouts.
//
// Two CTAs of a cluster share one 256 x 256 accumulator tile; the even CTA issues
// `tcgen05.mma.cta_group::2` with M = 256, every CTA loads 128 of the 256 M rows and half of the N
// columns with its own TMA loads (nothing is multicast), and its tensor memory receives the
// accumulator lanes of its own M rows.  Per 64-deep K step a CTA pulls 32 KB through L2 where the
// single-CTA kernel pulls 48.
//
// TN (weight gradients): M and N are the matrix's own rows and columns.
//
// NT / NN: the operands are exchanged - the WEIGHTS' output columns lie on the MMA's M side and the
// group's rows (tokens) on its N side, because N may be any multiple of 16: a group's rows are split
// into the fewest tiles of at most 256 rows, all of (nearly) the same length, so a group of 300 rows
// costs two tiles of 150 instead of 256 + 256.  With rows on the M side a tile is 128 (single CTA)
// or 256 rows whatever the group holds; for 64 ragged groups of 512 rows that is 12 % and 25 % of
// the multiplications.  The accumulator then holds the transposed tile: lanes are output columns.  It
// is read in the fragment layout that stmatrix transposes on the way into the row-major staging
// buffer, so the fused epilogues and the coalesced / TMA stores are those of the single-CTA kernel.
//
// What bounds the mainloop (dense 8192 x 14336 x 4096 bf16, share of the tensor pipe's cycles): one
// commit per CTA and a warp-synchronous issue loop 0.81; one multicast commit 0.89; that and a loop
// run by ONE thread 0.95 (1674 TFLOP/s against 1447 of cuBLAS, burst).  NN 0.84 -> 0.98, TN 0.79 -> 0.92.
// The single-CTA kernel's loop reaches 0.88 / 0.90 / 0.78 at more power per multiplication, which the
// board's cap turns into time on long launches.
//
// The GLU forward with its two weight operands stays on the single-CTA kernel: as a pair its two
// accumulators leave room for 128 tokens a tile, and every weight byte then serves half as many of them
// (8192 x 4096 x 14336, 8 groups, sustained: 898 TFLOP/s against 1038).
//
// Synchronisation between the two CTAs:
//   NT / NN  full[stage] lives in the even CTA and expects the bytes of both CTAs'
//            loads (the odd CTA's TMA completes on the even CTA's barrier).
//   TN       (ragged K) full[stage] of the even CTA counts two arrivals.
//            For a whole K block the even CTA's producer makes both and expects the bytes of
//            both CTAs, exactly as above.  The last K block of a group may end inside the
//            block: the rows past the group must be cleared in BOTH CTAs before the MMA reads
//            them.  For that block the odd CTA's loads complete on its own tail[stage]
//            barrier; its MMA warp (otherwise idle) waits there, clears the rows and makes the
//            second arrival on the even CTA's full[stage]; the even CTA clears its own rows
//            after the wait and issues the MMAs.
//   empty[stage], tmem_full[s]   one per CTA; the MMA thread's commit arrives on both;
//   tmem_empty[s]  lives in the even CTA; the epilogue warps of both CTAs arrive on it.
// Every wait is bounded as in the single-CTA kernel; a pair always works inside one group.  Launches
// that wait for peers' rows or store into peers' buffers stay on the single-CTA kernel.
#pragma once

#include "grouped_gemm_kernel.cuh"

namespace mb {
namespace gemm {

constexpr int kPairBlockN = 256;
// Kernel variants: epilogues without and with auxiliary operands (which need buffers for them).
constexpr int kPairPlain = 0, kPairAux = 1;
// Twelve epilogue warps, three per lane quarter: with eight, each scheduler had two warps of long
// dependent chains and issued in a third of its cycles while the tensor pipe waited for accumulators
// (contractions of 512 to 1024, where a tile's multiplications take less time than its epilogue).
// 14 warps are allocated as 16: 128 registers a thread.
constexpr int kPairEpilogueWarps = 12;
constexpr int kPairSubs = kPairEpilogueWarps / 4;
constexpr int kPairProducerWarp = kPairEpilogueWarps;
constexpr int kPairMmaWarp = kPairEpilogueWarps + 1;
constexpr int kPairThreads = (kPairEpilogueWarps + 2) * 32;
template <int MODE>
struct PairConfig {
  static constexpr int kStages = MODE == kPairPlain ? 5 : 4;
  static constexpr int kMBytes = kABytes;                                  // this CTA's 128 rows of the M side
  static constexpr int kNBytes = (kPairBlockN / 2) * kBlockK * 2;          // this CTA's half of the N side
  static constexpr int kTileRows = 256;                                    // NT / NN: most tokens of a tile
  static constexpr int kTileBytes = kStages * (kMBytes + kNBytes);
  static constexpr int kStagingBytes = kPairEpilogueWarps * 2048;          // one 32 x 32 chunk per warp
  static constexpr int kChunkBuffers = MODE == kPairAux ? 4 : 2;           // two outgoing, two auxiliary
  static constexpr int kBarBytes = 256;
  static constexpr int kSmemBytes = kTileBytes + kChunkBuffers * kStagingBytes + kBarBytes + 2 * kSmallGroups * 4 + 1024;
  static_assert(kSmemBytes <= 232448, "shared memory of one CTA");
};
constexpr int kTokenBox = 64;      // rows of a token box (NT / NN)

struct PairTile {
  int group;
  int row0;        // NT / NN: first token; TN: first output row of this CTA's half inside the group
  int rows;        // NT / NN: tokens of the tile; TN: valid output rows of this CTA's half
  int n0;          // NT / NN: first output column of this CTA's half; TN: first column of the tile
  int k_begin;
  int k_len;
};

// Three outputs of the GLU backward in one pass over the chunk, from one evaluation of the activation:
// dz1 goes to the staging buffer as it is produced, dz2 and h wait packed in registers.
template <typename T, int ACT, bool FRAG>
__device__ __forceinline__ void epilogue_emit_dglu(const uint32_t (&raw)[32], const PackedRow& a1, const PackedRow& a2,
                                                   Staging& stage, int64_t off, int64_t row_stride, int rows_ok, int cols,
                                                   int lane, int col, const GemmParams& p, TmaOut tma) {
  uint4 w2[4], w3[4];
  if (p.store_tma) stage_acquire(stage, lane);
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    float dz1[8], dz2[8], h[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float acc = __uint_as_float(raw[v * 8 + j]);
      const float z1 = packed_at<T>(a1, v * 8 + j), z2 = packed_at<T>(a2, v * 8 + j);
      float d, a;
      dact_values<T, ACT>(acc, z1, d, a);
      dz1[j] = d * z2;
      dz2[j] = acc * a;
      h[j] = a * z2;
    }
    uint4 w;
    w.x = pack2<T>(dz1[0], dz1[1]); w.y = pack2<T>(dz1[2], dz1[3]); w.z = pack2<T>(dz1[4], dz1[5]); w.w = pack2<T>(dz1[6], dz1[7]);
    w2[v].x = pack2<T>(dz2[0], dz2[1]); w2[v].y = pack2<T>(dz2[2], dz2[3]);
    w2[v].z = pack2<T>(dz2[4], dz2[5]); w2[v].w = pack2<T>(dz2[6], dz2[7]);
    w3[v].x = pack2<T>(h[0], h[1]); w3[v].y = pack2<T>(h[2], h[3]);
    w3[v].z = pack2<T>(h[4], h[5]); w3[v].w = pack2<T>(h[6], h[7]);
    stage_put<FRAG>(stage.buf, lane, v, w);
  }
#pragma unroll
  for (int which = 0; which < 3; ++which) {
    T* out = static_cast<T*>(which == 0 ? p.c : (which == 1 ? p.out2 : p.out3));
    if (out == nullptr) continue;
    if (which > 0) {
      if (p.store_tma) stage_acquire(stage, lane);
#pragma unroll
      for (int v = 0; v < 4; ++v) stage_put<FRAG>(stage.buf, lane, v, which == 1 ? w2[v] : w3[v]);
    }
    if (tma.on) {
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(p.out_map + which, smem_u32(stage.buf), col, tma.row);
        bulk_commit_group();
      }
      stage_flip(stage);
    } else {
      __syncwarp();
      stage_store<T>(stage.buf, out + off, row_stride, rows_ok, cols, lane);
      __syncwarp();
    }
  }
}

template <typename T, bool FRAG>
__device__ __forceinline__ void epilogue_dglu(const uint32_t (&raw)[32], const PackedRow& a1, const PackedRow& a2,
                                              Staging& stage, int64_t off, int rows_ok, int cols, int lane, int col,
                                              const GemmParams& p, TmaOut tma) {
  switch (p.act) {
    case kActGeluTanh: epilogue_emit_dglu<T, kActGeluTanh, FRAG>(raw, a1, a2, stage, off, p.N, rows_ok, cols, lane, col, p, tma); break;
    case kActSilu: epilogue_emit_dglu<T, kActSilu, FRAG>(raw, a1, a2, stage, off, p.N, rows_ok, cols, lane, col, p, tma); break;
    case kActRelu: epilogue_emit_dglu<T, kActRelu, FRAG>(raw, a1, a2, stage, off, p.N, rows_ok, cols, lane, col, p, tma); break;
    case kActGeluErf: epilogue_emit_dglu<T, kActGeluErf, FRAG>(raw, a1, a2, stage, off, p.N, rows_ok, cols, lane, col, p, tma); break;
    default: epilogue_emit_dglu<T, kActIdentity, FRAG>(raw, a1, a2, stage, off, p.N, rows_ok, cols, lane, col, p, tma); break;
  }
}

// FULL: the exact activations, in kernels of their own.  In one kernel with the others they made both spill, and
// training passes that never use them took 1 to 2 % longer (32768 x 768 x 3072, 64 experts: 1484 us against 1465).
template <typename T, int LAYOUT, int MODE, bool FULL>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
grouped_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                         const __grid_constant__ GemmParams p) {
  using Cfg = PairConfig<MODE>;
  constexpr bool AUX = MODE == kPairAux;
  constexpr bool kTn = LAYOUT == kTN;
  constexpr bool kMMn = LAYOUT != kNT;       // M side MN-major: weights [K, N] (NN), activations (TN)
  constexpr bool kNMn = kTn;                 // N side MN-major
  constexpr int kStages = Cfg::kStages;
  constexpr int kTileRows = Cfg::kTileRows;
  constexpr bool kIsBf16 = std::is_same<T, __nv_bfloat16>::value;
  constexpr int kTnBytes = Cfg::kMBytes + Cfg::kNBytes;
  static_assert(!AUX || LAYOUT != kTN, "weight gradients have no auxiliary operands");

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* smem_m = smem;
  uint8_t* smem_n = smem + kStages * Cfg::kMBytes;
  // Staging buffers directly after the operand ring (1024-byte aligned for the swizzled TMA stores).
  uint8_t* staging = smem + Cfg::kTileBytes;
  uint8_t* aux_buf = staging + 2 * Cfg::kStagingBytes;                            // AUX: two chunks per warp
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + Cfg::kChunkBuffers * Cfg::kStagingBytes);
  uint64_t* full_bar = bars;
  uint64_t* empty_bar = bars + kStages;
  uint64_t* tmem_full_bar = bars + 2 * kStages;
  uint64_t* tmem_empty_bar = bars + 2 * kStages + 2;
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_base_slot + 1);
  uint64_t* tail_bar = bars + 2 * kStages + 5;   // [kStages] TN, odd CTA: loads of a ragged last K block
  uint64_t* aux_bar = bars + 3 * kStages + 5;    // [warps] AUX: this warp's auxiliary chunk has landed
  static_assert((3 * kStages + 5 + kPairEpilogueWarps) * 8 <= Cfg::kBarBytes, "barriers");
  int* s_row_end = reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(bars) + Cfg::kBarBytes);
  int* s_tile_end = s_row_end + kSmallGroups;    // inclusive prefix sum of token tiles per group (NT / NN)

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int G = p.num_groups;
  const uint32_t cta = cluster_ctarank();        // 0: issues the MMAs, 1: its partner
  const int pair_id = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;

  // ---- one-time setup ---------------------------------------------------------
  if (warp == 0) group_tables(p.bins, G, p.rows_total, kTileRows, s_row_end, kTn ? nullptr : s_tile_end, lane);
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_u32(&full_bar[s]), kTn ? 2 : 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
      mbar_init(smem_u32(&tail_bar[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&tmem_full_bar[s]), 1);
      mbar_init(smem_u32(&tmem_empty_bar[s]), 2 * kPairEpilogueWarps);
    }
    for (int s = 0; s < kPairEpilogueWarps; ++s) mbar_init(smem_u32(&aux_bar[s]), 1);
    fence_barrier_init();
    prefetch_tensormap(&tmap_a);
    prefetch_tensormap(&tmap_b);
  }
  if (warp == kPairMmaWarp) tmem_alloc_pair(smem_u32(tmem_base_slot), 2 * kPairBlockN);
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();          // both CTAs' barriers and tensor memory exist before either is used
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_base_slot;
  const bool concat = LAYOUT == kNN && p.k_concat != 0;

  // ---- tile schedule (every role of both CTAs decodes the same sequence) ------------
  const int num_nb = (p.N + kPairBlockN - 1) / kPairBlockN;
  const int num_mb_tn = (p.M + 2 * kBlockM - 1) / (2 * kBlockM);
  const int total_tiles = kTn ? G * num_mb_tn * num_nb : (G > 0 ? s_tile_end[G - 1] : 0) * num_nb;
  auto decode = [&](int t) {
    PairTile tile;
    if constexpr (kTn) {
      const int per_group = num_mb_tn * num_nb;
      tile.group = t / per_group;
      const int r = t - tile.group * per_group;
      const int mb_i = r / num_nb;
      tile.n0 = (r - mb_i * num_nb) * kPairBlockN;
      tile.row0 = mb_i * 2 * kBlockM + int(cta) * kBlockM;
      tile.rows = max(0, min(kBlockM, p.M - tile.row0));
      tile.k_begin = tile.group ? s_row_end[tile.group - 1] : 0;
      tile.k_len = s_row_end[tile.group] - tile.k_begin;
    } else {
      // Bands of column tiles with the token tiles outside, as in the single-CTA kernel.
      int lo = 0, hi = G - 1;
      const int key = t / num_nb;              // group boundaries are multiples of num_nb tiles
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (s_tile_end[mid] <= key) lo = mid + 1; else hi = mid;
      }
      tile.group = lo;
      const int tile_begin = lo ? s_tile_end[lo - 1] : 0;
      const int tiles = s_tile_end[lo] - tile_begin;
      const int u = t - tile_begin * num_nb;
      const int band_n = p.band_n > 0 ? p.band_n : kBandN;
      const int band = u / (tiles * band_n);
      const int r = u - band * tiles * band_n;
      const int width = min(band_n, num_nb - band * band_n);
      const int local = r / width;
      tile.n0 = (band * band_n + (r - local * width)) * kPairBlockN + int(cta) * kBlockM;
      const int row_start = lo ? s_row_end[lo - 1] : 0;
      const int rows = s_row_end[lo] - row_start;
      // Equal shares, rounded up to the 16 columns an MMA steps by.  A share is at most kTileRows, so the
      // last one is never empty.
      const int share = ((rows + tiles - 1) / tiles + 15) & ~15;
      tile.row0 = row_start + local * share;
      tile.rows = min(share, rows - local * share);
      tile.k_begin = 0;
      tile.k_len = p.K;
    }
    return tile;
  };
  // A decode is a search and four divisions, some 1500 cycles of one warp's time: every role's warp
  // decodes 32 of its tiles at once, one per lane, and fetches them by shuffles.
  PairTile cached;
  int cached_window = -1;
  auto fetch = [&](int i) {                    // i-th tile of this pair; the whole warp, i not decreasing
    if ((i >> 5) != cached_window) {
      cached_window = i >> 5;
      const int t = pair_id + ((i & ~31) + lane) * num_pairs;
      if (t < total_tiles) cached = decode(t);
    }
    PairTile tile;
    const int src = i & 31;
    tile.group = __shfl_sync(0xffffffffu, cached.group, src);
    tile.row0 = __shfl_sync(0xffffffffu, cached.row0, src);
    tile.rows = __shfl_sync(0xffffffffu, cached.rows, src);
    tile.n0 = __shfl_sync(0xffffffffu, cached.n0, src);
    tile.k_begin = kTn ? __shfl_sync(0xffffffffu, cached.k_begin, src) : 0;
    tile.k_len = kTn ? __shfl_sync(0xffffffffu, cached.k_len, src) : p.K;
    return tile;
  };
  const int my_tiles = pair_id < total_tiles ? (total_tiles - pair_id + num_pairs - 1) / num_pairs : 0;
  auto mma_cols = [](const PairTile& tile) { return (tile.rows + 15) & ~15; };   // NT / NN

  // Clears the rows of the last K block of a TN tile that lie past the group (one warp).
  auto clear_tail = [&](const PairTile& tile, int kb, int stage) {
    const int valid = tile.k_len - kb * kBlockK;
    if (valid < kBlockK) {
      uint8_t* m_tile = smem_m + stage * Cfg::kMBytes;
      uint8_t* n_tile = smem_n + stage * Cfg::kNBytes;
      const int tail_chunks = (kBlockK - valid) * 8;   // 16-byte chunks per box
      constexpr int kABoxes = kBlockM / 64, kBBoxes = kPairBlockN / 2 / 64;
      // After the last group that has rows the memory may never have been written: both operands are cleared.
      const bool at_end = tile.k_begin + tile.k_len >= s_row_end[G - 1];   // no later group has rows
      const int boxes = at_end ? kABoxes + kBBoxes : kABoxes;
      for (int box = 0; box < boxes; ++box) {
        uint8_t* base = (box < kABoxes) ? m_tile + box * kBoxBytes : n_tile + (box - kABoxes) * kBoxBytes;
        uint4* rows = reinterpret_cast<uint4*>(base + valid * 128);
        for (int i = lane; i < tail_chunks; i += 32) rows[i] = make_uint4(0, 0, 0, 0);
      }
      fence_proxy_async_smem();
    }
    __syncwarp();
  };

  if (warp == kPairProducerWarp) {
    // ======================= TMA producer (both CTAs) ============================
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int i = 0; i < my_tiles; ++i) {
      const PairTile tile = fetch(i);
      if (lane == 0 && ok) {
        const int num_kb1 = (tile.k_len + kBlockK - 1) / kBlockK;
        const int num_kb = concat ? 2 * num_kb1 : num_kb1;
        const int half = kTn ? 0 : mma_cols(tile) / 2;                  // tokens this CTA loads (NT / NN)
        const int boxes = (half + kTokenBox - 1) / kTokenBox;
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1u, abort_flag, p.status, kErrProducer, kWaitLimitNs);
          if (!ok) break;
          const uint32_t m_dst = smem_u32(smem_m + stage * Cfg::kMBytes);
          const uint32_t n_dst = smem_u32(smem_n + stage * Cfg::kNBytes);
          if constexpr (kTn) {
            const bool ragged = kb == num_kb - 1 && (tile.k_len & (kBlockK - 1)) != 0;
            uint32_t bar;
            if (cta == 0) {
              bar = smem_u32(&full_bar[stage]);
              if (ragged) {
                mbar_arrive_expect_tx(bar, kTnBytes);       // the partner arrives after clearing its tail
              } else {
                mbar_arrive_expect_tx(bar, 2 * kTnBytes);
                mbar_arrive(bar);
              }
            } else if (ragged) {
              bar = smem_u32(&tail_bar[stage]);
              mbar_arrive_expect_tx(bar, kTnBytes);
            } else {
              bar = map_to_cta(smem_u32(&full_bar[stage]), 0);
            }
            const int krow = tile.k_begin + kb * kBlockK;
            const int n_half = tile.n0 + int(cta) * (kPairBlockN / 2);        // this CTA's columns of b
#pragma unroll
            for (int j = 0; j < kBlockM / 64; ++j)
              tma_load_2d_pair(m_dst + j * kBoxBytes, &tmap_a, bar, tile.row0 + 64 * j, krow);
#pragma unroll
            for (int j = 0; j < kPairBlockN / 2 / 64; ++j)
              tma_load_2d_pair(n_dst + j * kBoxBytes, &tmap_b, bar, n_half + 64 * j, krow);
          } else {
            // The stage's "full" barrier is the even CTA's; it counts the bytes of both CTAs.
            const uint32_t bar = map_to_cta(smem_u32(&full_bar[stage]), 0);
            if (cta == 0)
              mbar_arrive_expect_tx(smem_u32(&full_bar[stage]),
                                    2 * (Cfg::kMBytes + boxes * (kTokenBox * kBlockK * 2)));
            // Second operand pair of a concatenated contraction: same coordinates, other tensors.
            const bool second = concat && kb >= num_kb1;
            const int kk = second ? kb - num_kb1 : kb;
            const CUtensorMap* tokens = second ? &p.a2_map : &tmap_a;
            const CUtensorMap* weights = second ? &p.b2_map : &tmap_b;
            if constexpr (LAYOUT == kNT) {
              tma_load_2d_pair(m_dst, weights, bar, kk * kBlockK, tile.group * p.N + tile.n0);
            } else {
#pragma unroll
              for (int j = 0; j < kBlockM / 64; ++j)
                tma_load_2d_pair(m_dst + j * kBoxBytes, weights, bar, tile.n0 + 64 * j,
                                 tile.group * p.K + kk * kBlockK);
            }
            for (int j = 0; j < boxes; ++j)
              tma_load_2d_pair(n_dst + j * (kTokenBox * kBlockK * 2), tokens, bar, kk * kBlockK,
                               tile.row0 + int(cta) * half + kTokenBox * j);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
      }
      __syncwarp();
    }
  } else if (warp == kPairMmaWarp) {
    if (cta == 0) {
      // ======================= MMA issuer (even CTA) ===============================
      int stage = 0;
      uint32_t phase = 0;
      int acc_stage = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      // The MMAs of one K step, by one thread.
      auto issue = [&](uint32_t d_tmem, uint32_t idesc, int s, bool first) {
        const uint32_t m_base = smem_u32(smem_m + s * Cfg::kMBytes);
        const uint32_t n_base = smem_u32(smem_n + s * Cfg::kNBytes);
#pragma unroll
        for (int k = 0; k < kBlockK / kUmmaK; ++k) {
          const uint64_t n_desc = kNMn ? smem_desc_sw128(n_base + k * (kUmmaK * 128), kBoxBytes, 1024)
                                       : smem_desc_sw128(n_base + k * (kUmmaK * 2), 16, 1024);
          const uint64_t m_desc = kMMn ? smem_desc_sw128(m_base + k * (kUmmaK * 128), kBoxBytes, 1024)
                                       : smem_desc_sw128(m_base + k * (kUmmaK * 2), 16, 1024);
          const uint32_t accumulate = (first && k == 0) ? 0u : 1u;
          umma_f16_pair(d_tmem, m_desc, n_desc, idesc, accumulate);
        }
        umma_commit_pair(smem_u32(&empty_bar[s]));    // the stage is reusable in both CTAs once these retire
      };
      for (int i = 0; i < my_tiles && ok; ++i) {
        const PairTile tile = fetch(i);
        const int num_kb = ((tile.k_len + kBlockK - 1) / kBlockK) * (concat ? 2 : 1);
        const uint32_t idesc =
            instr_desc_f16(kIsBf16, kMMn, kNMn, 2 * kBlockM, kTn ? kPairBlockN : mma_cols(tile));
        const uint32_t d_tmem = tmem_base + acc_stage * kPairBlockN;
        const bool ragged = kTn && (tile.k_len & (kBlockK - 1)) != 0;
        const int whole = ragged ? num_kb - 1 : num_kb;
        if (lane == 0) {
          ok = mbar_wait(smem_u32(&tmem_empty_bar[acc_stage]), acc_phase ^ 1u, abort_flag, p.status, kErrMmaTmem,
                         kWaitLimitNs);
          tcgen05_fence_after();
          int s = stage;
          uint32_t ph = phase;
          for (int kb = 0; kb < whole && ok; ++kb) {
            ok = mbar_wait(smem_u32(&full_bar[s]), ph, abort_flag, p.status, kErrMmaFull, kWaitLimitNs);
            if (!ok) break;
            tcgen05_fence_after();
            issue(d_tmem, idesc, s, kb == 0);
            if (++s == kStages) { s = 0; ph ^= 1u; }
          }
        }
        __syncwarp();
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        if (!ok) break;
        phase ^= uint32_t((stage + whole) / kStages) & 1u;
        stage = (stage + whole) % kStages;
        if constexpr (kTn) {
          if (ragged) {
            ok = mbar_wait(smem_u32(&full_bar[stage]), phase, abort_flag, p.status, kErrMmaFull, kWaitLimitNs);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            clear_tail(tile, num_kb - 1, stage);
            tcgen05_fence_after();
            if (lane == 0) issue(d_tmem, idesc, stage, whole == 0);
            __syncwarp();
            if (++stage == kStages) { stage = 0; phase ^= 1u; }
          }
        }
        if (lane == 0) {
          if (num_kb > 0) {
            umma_commit_pair(smem_u32(&tmem_full_bar[acc_stage]));
          } else {   // empty group: nothing to wait for, the epilogue writes zeros
            mbar_arrive(smem_u32(&tmem_full_bar[acc_stage]));
            mbar_arrive_remote(map_to_cta(smem_u32(&tmem_full_bar[acc_stage]), 1));
          }
        }
        __syncwarp();
        if (++acc_stage == 2) { acc_stage = 0; acc_phase ^= 1u; }
      }
    } else if constexpr (kTn) {
      // ======================= tail clearing and hand-over (odd CTA, TN) ===========
      int stage = 0;
      uint32_t tail_phases = 0;      // bit s: parity of the next use of tail[s]
      bool ok = true;
      for (int i = 0; i < my_tiles && ok; ++i) {
        const PairTile tile = fetch(i);
        const int num_kb = (tile.k_len + kBlockK - 1) / kBlockK;
        if (num_kb == 0) continue;
        const int last = (stage + num_kb - 1) % kStages;      // ring stage of the tile's last K block
        stage = (stage + num_kb) % kStages;
        if ((tile.k_len & (kBlockK - 1)) == 0) continue;      // whole blocks only: nothing to clear
        ok = mbar_wait(smem_u32(&tail_bar[last]), (tail_phases >> last) & 1u, abort_flag, p.status, kErrMmaFull,
                       kWaitLimitNs);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tail_phases ^= 1u << last;
        clear_tail(tile, num_kb - 1, last);
        if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&full_bar[last]), 0));
        __syncwarp();
      }
    }
  } else if (warp < kPairEpilogueWarps) {
    // ======================= epilogue warps (both CTAs, own 128 accumulator lanes) ====
    const int quarter = warp & 3;
    const int sub = warp >> 2;                  // which of the three warps of that quarter
    Staging stage{staging + warp * 2048, p.store_tma != 0 ? Cfg::kStagingBytes : 0};
    uint8_t* const aux1 = aux_buf + warp * 2048;
    uint8_t* const aux2 = aux1 + Cfg::kStagingBytes;
    const uint32_t my_aux_bar = smem_u32(&aux_bar[warp]);
    uint32_t aux_phase = 0;
    const bool need2 = AUX && p.epilogue == kEpiDGlu;
    int acc_stage = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    float2 sq_sum = make_float2(0.f, 0.f);      // sum of squares of what this thread stored (p.sqnorm)
    // Chunk `ci` of a tile: 32 rows x 32 columns of the output.
    //   TN       rows are this warp's lanes, chunks walk the columns;
    //   NT / NN  columns are this warp's lanes, chunks walk the rows (tokens).
    // A tile's chunks are dealt to the quarter's warps where the previous tile's left off.
    auto chunk_count = [&](const PairTile& tile) {
      if constexpr (kTn) return tile.rows > quarter * 32 ? (min(kPairBlockN, p.N - tile.n0) + 31) / 32 : 0;
      else return tile.n0 + quarter * 32 < p.N ? (tile.rows + 31) / 32 : 0;
    };
    auto first_chunk = [&](int dealt) { return (sub + kPairSubs - dealt) % kPairSubs; };
    auto chunk_row = [&](const PairTile& tile, int ci) {
      return kTn ? tile.group * p.M + tile.row0 + quarter * 32 : tile.row0 + ci * 32;
    };
    auto chunk_col = [&](const PairTile& tile, int ci) { return kTn ? tile.n0 + ci * 32 : tile.n0 + quarter * 32; };
    // Auxiliary operands of a chunk come by TMA (rows past the tile are loaded too and never used) into
    // this warp's buffers; the next chunk's, of the next tile where need be, are requested as soon as this
    // chunk's are in registers.
    auto request_aux = [&](const PairTile& tile, int ci) {
      if (lane == 0) {
        const int col = chunk_col(tile, ci), row = chunk_row(tile, ci);
        mbar_arrive_expect_tx(my_aux_bar, need2 ? 4096 : 2048);
        tma_load_2d(smem_u32(aux1), &p.aux_map[0], my_aux_bar, col, row);
        if (need2) tma_load_2d(smem_u32(aux2), &p.aux_map[1], my_aux_bar, col, row);
      }
    };
    PairTile next{};
    if (my_tiles > 0) next = fetch(0);
    int dealt = 0;                              // chunks dealt so far, modulo kPairSubs
    bool requested = false;                     // AUX: this warp's next chunk is on its way
    for (int i = 0; i < my_tiles && ok; ++i) {
      const PairTile tile = next;
      const bool has_k = tile.k_len > 0;
      const int chunks = chunk_count(tile), first = first_chunk(dealt);
      const int next_dealt = (dealt + chunks) % kPairSubs;
      if (i + 1 < my_tiles) next = fetch(i + 1);
      if constexpr (AUX) {
        if (!requested && first < chunks) {
          request_aux(tile, first);
          requested = true;
        }
      }
      ok = mbar_wait(smem_u32(&tmem_full_bar[acc_stage]), acc_phase, abort_flag, p.status, kErrEpilogue,
                     kWaitLimitNs);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tcgen05_fence_after();
      const uint32_t taddr = tmem_base + (uint32_t(quarter * 32) << 16) + acc_stage * kPairBlockN;
      auto load_acc = [&](int column, uint32_t (&raw)[32]) {
        if constexpr (kTn) {
          tmem_ld_32x32(taddr + column, raw);
        } else {
          tmem_ld_16x256_x4(taddr + column, raw);
          tmem_ld_16x256_x4(taddr + (16u << 16) + column, raw + 16);
        }
        tmem_ld_wait();
        if (p.alpha != 1.f) {
#pragma unroll
          for (int k = 0; k < 32; ++k) raw[k] = __float_as_uint(__uint_as_float(raw[k]) * p.alpha);
        }
      };
#pragma unroll 1
      for (int ci = first; ci < chunks; ci += kPairSubs) {
        const int col = chunk_col(tile, ci), out_row = chunk_row(tile, ci), cols = min(32, p.N - col);
        const int rows_ok = kTn ? min(32, tile.rows - quarter * 32) : min(32, tile.rows - ci * 32);
        const int64_t off = int64_t(out_row) * p.N + col;
        const TmaOut tma{p.store_tma != 0 && rows_ok == 32, out_row};
        uint32_t raw[32];
        if constexpr (AUX) {
          PackedRow a1, a2;
          ok = mbar_wait(my_aux_bar, aux_phase, abort_flag, p.status, kErrEpilogue, kWaitLimitNs);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          aux_phase ^= 1u;
          stage_read_row<true>(aux1, lane, a1);
          if (need2) stage_read_row<true>(aux2, lane, a2);
          __syncwarp();
          if (ci + kPairSubs < chunks) {
            request_aux(tile, ci + kPairSubs);
          } else {
            const int nf = first_chunk(next_dealt);
            requested = i + 1 < my_tiles && nf < chunk_count(next);
            if (requested) request_aux(next, nf);
          }
          load_acc(ci * 32, raw);
          if constexpr (FULL)
            epilogue_by_act<T, kEpiDAct, true, 1>(raw, a1, a2, stage, off, p.N, rows_ok, cols, lane, p, nullptr, col, tma);
          else switch (p.epilogue) {
            case kEpiAdd: epilogue_chunk<T, kEpiAdd, kActIdentity, true>(raw, a1, a2, stage, off, p.N, rows_ok, cols, lane, p, nullptr, col, tma); break;
            case kEpiDAct: epilogue_by_act<T, kEpiDAct, true, 0>(raw, a1, a2, stage, off, p.N, rows_ok, cols, lane, p, nullptr, col, tma); break;
            case kEpiGlu: epilogue_by_act<T, kEpiGlu, true>(raw, a1, a2, stage, off, p.N, rows_ok, cols, lane, p, nullptr, col, tma); break;
            default: epilogue_dglu<T, true>(raw, a1, a2, stage, off, rows_ok, cols, lane, col, p, tma); break;
          }
        } else {
          PackedRow unused;
          if (has_k) {
            load_acc(ci * 32, raw);
            if constexpr (kTn) {
              if (p.sqnorm != nullptr && lane < rows_ok) {
#pragma unroll
                for (int k = 0; k < 32; k += 2) {
                  const float2 v = make_float2(__uint_as_float(raw[k]), __uint_as_float(raw[k + 1]));
                  if (k < cols) sq_sum = __ffma2_rn(v, v, sq_sum);
                }
              }
            }
          } else {
#pragma unroll
            for (int k = 0; k < 32; ++k) raw[k] = 0u;
          }
          if (!FULL && (kTn || p.epilogue == kEpiNone))
            epilogue_chunk<T, kEpiNone, kActIdentity, !kTn>(raw, unused, unused, stage, off, p.N, rows_ok, cols, lane, p,
                                                            nullptr, col, tma);
          else
            epilogue_by_act<T, kEpiAct, !kTn, FULL ? 1 : 0>(raw, unused, unused, stage, off, p.N, rows_ok, cols, lane, p, nullptr, col,
                                              tma);
        }
      }
      if (!ok) break;
      dealt = next_dealt;
      tcgen05_fence_before();
      __syncwarp();
      // The accumulator stage is free for the next MMA once every epilogue warp of BOTH CTAs has read it.
      if (lane == 0) mbar_arrive_remote(map_to_cta(smem_u32(&tmem_empty_bar[acc_stage]), 0));
      if (++acc_stage == 2) { acc_stage = 0; acc_phase ^= 1u; }
    }
    if (p.store_tma && lane == 0) bulk_wait_all();   // bulk stores complete before the CTA retires
    if constexpr (kTn) {
      if (p.sqnorm != nullptr) {                     // one atomic per warp and launch
        float total = sq_sum.x + sq_sum.y;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) total += __shfl_xor_sync(0xffffffffu, total, off);
        if (lane == 0 && ok) atomicAdd(p.sqnorm, total);
      }
    }
    // Rows past the last group are defined as zero.
    if (!kTn && p.zero_tail) {
      const int last = G > 0 ? s_row_end[G - 1] : 0;
      const int64_t begin = int64_t(last) * p.N, end = int64_t(p.rows_total) * p.N;
      const int64_t tid = int64_t(blockIdx.x) * (kPairEpilogueWarps * 32) + threadIdx.x;
      const int64_t stride = int64_t(gridDim.x) * (kPairEpilogueWarps * 32);
      for (int64_t i = begin + tid * 8; i < end; i += stride * 8) {
        const uint4 z = make_uint4(0, 0, 0, 0);
        if (p.c) *reinterpret_cast<uint4*>(static_cast<T*>(p.c) + i) = z;
        if (p.out2) *reinterpret_cast<uint4*>(static_cast<T*>(p.out2) + i) = z;
        if (p.out3) *reinterpret_cast<uint4*>(static_cast<T*>(p.out3) + i) = z;
      }
    }
  }

  // ---- teardown: neither CTA may release shared or tensor memory the other still uses ----
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == kPairMmaWarp) {
    if (*abort_flag != 0) {
      const uint64_t t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 2000000ull) __nanosleep(1000);
    }
    tcgen05_fence_after();
    tmem_dealloc_pair(tmem_base, 2 * kPairBlockN);
  }
}

// Launches on at most as many CTA pairs as the device can keep resident at once: tiles are
// assigned round-robin to the pairs of the grid, so a pair that only starts after another has
// finished would double the run time.
template <typename T, int LAYOUT, int MODE, bool FULL>
cudaError_t launch_pair_kernel(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int grid,
                               cudaStream_t stream) {
  constexpr int kPairSmemBytes = PairConfig<MODE>::kSmemBytes;
  auto kernel = grouped_gemm_pair_kernel<T, LAYOUT, MODE, FULL>;
  static int max_pairs[64] = {0};
  int dev = 0;
  cudaError_t rc = cudaGetDevice(&dev);
  if (rc != cudaSuccess) return rc;
  if (max_pairs[dev & 63] == 0) {
    rc = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmemBytes);
    if (rc != cudaSuccess) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(kPairThreads, 1, 1);
    cfg.dynamicSmemBytes = kPairSmemBytes;
    int clusters = 0;
    rc = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
    if (rc != cudaSuccess || clusters < 1) {
      (void)cudaGetLastError();
      clusters = 1 << 20;   // unknown: keep the caller's grid
    }
    max_pairs[dev & 63] = clusters;
  }
  grid = 2 * min(grid / 2, max_pairs[dev & 63]);
  if (grid < 2) return cudaErrorInvalidValue;
  kernel<<<grid, kPairThreads, kPairSmemBytes, stream>>>(ta, tb, p);
  return cudaGetLastError();
}

template <typename T, int LAYOUT>
cudaError_t launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int grid,
                        cudaStream_t stream) {
  if constexpr (LAYOUT != kTN) {
    const bool full = p.act >= kActGeluTanhFull && (p.epilogue == kEpiAct || p.epilogue == kEpiDAct);
    if (p.epilogue != kEpiNone && p.epilogue != kEpiAct)
      return full ? launch_pair_kernel<T, LAYOUT, kPairAux, true>(ta, tb, p, grid, stream)
                  : launch_pair_kernel<T, LAYOUT, kPairAux, false>(ta, tb, p, grid, stream);
    if (full) return launch_pair_kernel<T, LAYOUT, kPairPlain, true>(ta, tb, p, grid, stream);
  }
  return launch_pair_kernel<T, LAYOUT, kPairPlain, false>(ta, tb, p, grid, stream);
}

}  // namespace gemm
}  // namespace mb
