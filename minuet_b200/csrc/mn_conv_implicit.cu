// Fused (implicit-GEMM) forward pass of a sparse convolution, fp16/bf16.
//
// The reference gathers every (source, target) pair row into a padded buffer,
// multiplies bucket by bucket with cuBLAS and scatters the products back
// (csrc/minuet/cuda/functions/sparse_convolution.cu:505-661); every pair row
// crosses HBM four times.  Here one persistent kernel owns 128 consecutive TARGET
// rows at a time and accumulates ALL kernel offsets of that tile in one TMEM
// accumulator:
//   producers   (4 or 8 warps): warp w fetches, for every active offset and k-block, the
//               128-byte slices of the source rows that feed its share of the target rows
//               (cp.async straight into the 128-byte-swizzled A tile, zeros where the
//               kernel map has no entry)
//   MMA warp    allocates TMEM and issues tcgen05.mma over (offset, k-block)
//   weight warp starts the TMA load of every stage's weight tile
//   index warp  copies every step's index block, eight steps ahead
//   epilogue    (8 or 4 warps): TMEM -> registers -> optional per-channel scale/shift
//               (folded BatchNorm or bias), residual add, ReLU -> the output rows
// so that features are read once per pair (mostly from L2), outputs are written
// once, and no pair-row buffer exists.  Offsets with no pair inside a tile are
// skipped through a per-tile bit mask.  The neighbour table [O, T] (source row
// of target t under mask row p, or -1) is derived once per kernel map from the
// masks by mn_build_neighbor_table.  Every barrier wait is bounded (status bit 2).
//
// What bounds it.  Up to 128 columns and with three or more pairs a row the memory does not: indices that are all -1,
// sequential or random take the same time.  Up to 64 columns a CTA's step of some 1000 cycles (2 CTAs per SM) is the chain of
// one producer warp (wait, eight indices a lane, eight copies), before that it was the one warp that
// sent index blocks and weights both.  From 128 columns on shared memory: per 64-channel step of 128 rows the gathered rows and
// weights are written (16 KB and 128 bytes a column) and read again by the MMAs, at 128 bytes a cycle 512 cycles
// for 256 of MMA at 128 columns (measured 595 to 650), 768 for 512 at 256 (726 to 804).  There the
// gather shows too, behind a ring of four stages: 524k rows 256->256, nine offsets, 408 us with indices of -1, 473
// sequential, 506 random.  Sparser maps: the epilogue (see there).  A warp needs five cycles per dependent
// instruction, so every role's loop is kept short: the issuing warps stay converged and elect
// one lane only around the instruction itself (issued from a divergent lane-0 branch every MMA
// took about 150 cycles of register moves), the index blocks arrive eight steps ahead and a lane
// reads the indices of all its rows with one load, and the next stage's barrier is probed before
// the current stage is worked on (a wait that finds its phase complete costs 200 cycles, a probe 60).
#include "mn_sort.cuh"
#include "mn_tc.cuh"

#include <algorithm>

namespace mn {

namespace {

using namespace tc;

constexpr int kGatherWarps = 12;       // producer and epilogue warps together: 8 + 4 or 4 + 8
constexpr int kImCtas = 2;             // CTAs per SM the register file allows
constexpr int kBM = 128;
constexpr int kBK = 64;
constexpr int kUmmaK = 16;
constexpr int kMaxStages = 8;
constexpr int kMaxN = 256;
constexpr int kIdxSlots = 8;           // steps the index blocks run ahead
constexpr int kTileSlots = 3;          // tiles that a CTA holds at most beside the one it works on (see the index warp)
constexpr int kMaxSub = 2;             // 128-row sub-tiles per CTA tile
constexpr int kResSlot = 32 * 64;      // bytes of 32 columns of 32 rows of the residual
constexpr int kNBlock = kBK * 128;     // kMapNMajor: bytes of one block of 64 columns of a weight tile

// What feeds the kernel: a kernel map; the same with weights as they are, [O, K, N], as N-major
// tiles; the product rows of a pair list; the rows of one dense product (the 1x1x1 convolution),
// whose tiles TMA fetches whole.
enum ImMode { kMap = 0, kMapNMajor = 1, kPairRows = 2, kDense = 3 };
// (one dense product: no rows to gather and no index blocks, so that a producer's place does for the tiles' warp)
constexpr int threads_of(int mode) { return (kGatherWarps + (mode == kDense ? 2 : 3)) * 32; }

struct ImArgs {
  const uint8_t *in;          // [S, K] 16-bit
  const int32_t *nbr;         // [O, pitch]
  const uint32_t *tile_bits;  // [tiles]
  const int32_t *order;       // [O] or NULL
  const float *scale;         // [N] or NULL
  const float *shift;         // [N] or NULL
  const uint8_t *residual;    // [T, N] 16-bit or NULL
  int32_t *status;
  int64_t T;
  int64_t pitch;              // of the neighbour table: T rounded up to 128
  int32_t K, N, n_pad, k_blocks, stages, a_bytes, stage_bytes, elem_is_bf16, num_tiles, relu;
  int32_t claims;             // tiles are handed out; 0: every gridDim-th is a CTA's
  int32_t wide;        // rows of the output and the residual start on 32-byte boundaries
  int32_t acc_bufs;    // accumulator sets in TMEM (2 when 2 * sub * n_pad <= 512, else 1)
  int32_t n_tiles128;  // entries of tile_bits
  int32_t num_offsets; // O
  int32_t tmem_cols;   // TMEM columns this CTA allocates
  int32_t zero;        // 0
  // pair mode (step 1 of the pair-list forward): the rows are PRODUCT rows, row r reads
  // source row nbr[r], every tile has exactly one "offset" whose weight matrix follows from
  // the mask row that owns the tile, and the fp32 accumulators are stored as they are
  int32_t pair_rows;                            // mask rows in pair_tile_prefix
  int32_t pair_tile_prefix[MN_MAX_PAIR_ROWS + 1];
  float *out_f32;                               // [T, N]
  const int32_t *perm;   // [T] or NULL: tile row r is target row perm[r] (nbr is in tile-row order)
  uint8_t *out16;        // [T, N] 16-bit output
};

// mask row that owns 128-row tile `tile` of the product buffer
__device__ __forceinline__ int pair_row_of_tile(const ImArgs &a, int tile) {
  int lo = 0, hi = a.pair_rows;   // last p with prefix[p] <= tile
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (a.pair_tile_prefix[mid] <= tile) lo = mid; else hi = mid;
  }
  return lo;
}

// 16-byte asynchronous copy; src_bytes = 0 writes 16 zero bytes instead.  It writes through the
// generic proxy, like a store: the MMA issuer fences after the stage barrier.
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void *src, uint32_t src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes)
               : "memory");
}

// One 32-byte sector of global memory per lane.
__device__ __forceinline__ void ld_global_32(const void *src, uint32_t *r) {
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                 "=r"(r[7])
               : "l"(src));
}

__device__ __forceinline__ void ld_global_16(const void *src, uint32_t *r) {
  const uint4 v = *reinterpret_cast<const uint4 *>(src);
  r[0] = v.x; r[1] = v.y; r[2] = v.z; r[3] = v.w;
}

__device__ __forceinline__ void ld_shared_16(uint32_t src, uint32_t *r) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(src) : "memory");
}

__device__ __forceinline__ void st_global_32(void *dst, const uint32_t *r) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

template <bool kBf16>
__device__ __forceinline__ float elem_to_f32(uint16_t v) {
  if (kBf16) return __uint_as_float((uint32_t)v << 16);
  return __half2float(__ushort_as_half(v));
}

// Loads that are issued where they stand: an ordinary read-only load may be moved down to its
// first use, a step or a tile later, where its whole latency would be waited for.
__device__ __forceinline__ int32_t load_ahead_1(const void *src) {
  int32_t v;
  asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(v) : "l"(src));
  return v;
}

// Asks for the next block of this grid that has not started, which will then not start: its number comes to
// `answer` (16 bytes) and completes `bar`.  Not to be called again once the answer was "none".
__device__ __forceinline__ void claim_block(void *answer, uint64_t *bar) {
  mbar_expect_tx(bar, 16u);
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
                   smem_u32(answer)), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ int claimed_block(const void *answer) {      // -1: none
  uint32_t got, x = 0u;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 v;\n\t"
      "ld.shared.b128 v, [%2];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, v;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "mov.u32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, _, _, _}, v;\n\t}"
      : "=r"(got), "=r"(x) : "r"(smem_u32(answer)) : "memory");
  return got != 0u ? (int)x : -1;
}

// Offset bits of the sub-tiles of a CTA tile (pair and dense mode: one offset each): the request and, later, the
// value.  A request under a condition would be waited for where the branch joins.
template <int kSub, int kMode>
__device__ __forceinline__ void request_bits(const ImArgs &args, int tile, uint32_t (&raw)[kSub]) {
#pragma unroll
  for (int h = 0; h < kSub; h++)
    raw[h] = kMode > kMapNMajor ? 1u : (uint32_t)load_ahead_1(args.tile_bits + min(max(tile, 0) * kSub + h, args.n_tiles128 - 1));
}

template <int kSub>
__device__ __forceinline__ void take_bits(const ImArgs &args, int tile, const uint32_t (&raw)[kSub],
                                          uint32_t (&hb)[kSub]) {
#pragma unroll
  for (int h = 0; h < kSub; h++)
    hb[h] = tile >= 0 && tile * kSub + h < args.n_tiles128 ? raw[h] : 0u;
}

template <int kSub>
__device__ __forceinline__ uint32_t union_of(const uint32_t (&hb)[kSub]) {
  uint32_t u = 0u;
#pragma unroll
  for (int h = 0; h < kSub; h++) u |= hb[h];
  return u;
}

// kSub: sub-tiles per CTA tile (they share every weight tile); kLpr: lanes that copy one
// 128-byte slice (4 where a source row has at most 64 bytes: half the copies, twice the rows
// per copy); kProdWarps: 4 producer and 8 epilogue warps or 8 and 4; kStaged: the epilogue's
// residual comes through shared memory.
template <int kSub, int kLpr, int kProdWarps, int kMode, bool kStaged>
__global__ void __launch_bounds__(threads_of(kMode), kImCtas)
conv_implicit_kernel(const __grid_constant__ ImArgs args,
                     const __grid_constant__ CUtensorMap map_a,     // kDense: features [S, K]
                     const __grid_constant__ CUtensorMap map_b) {   // weights^T [O, N, K]; kMapNMajor: weights [O, K, N]
  constexpr bool kPairs = kMode == kPairRows, kNMajor = kMode == kMapNMajor;
  constexpr int kProdRows = 128 / kProdWarps;               // rows of a sub-tile per producer warp
  constexpr int kMmaWarp = kProdWarps, kTmaWarp = kProdWarps + 1, kIdxWarp = kMode == kDense ? 0 : kProdWarps + 2;
  constexpr int kEpiWarp = threads_of(kMode) / 32 - (kGatherWarps - kProdWarps);
  constexpr int kEpiCols = (kGatherWarps - kProdWarps) / 4;   // epilogue warps per quarter of the rows
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t bar_full[kMaxStages], bar_empty[kMaxStages];
  __shared__ uint64_t bar_acc_full[2], bar_acc_empty[2];
  __shared__ uint64_t bar_idx_full[kIdxSlots], bar_idx_empty[kIdxSlots];
  __shared__ uint64_t bar_tile_full[kTileSlots], bar_tile_empty[kTileSlots], bar_claim;
  __shared__ __align__(16) uint4 s_claim;
  __shared__ int32_t s_tile[kTileSlots];
  __shared__ uint32_t s_tile_bits[kTileSlots][kSub];
  __shared__ uint32_t s_idx_has[kIdxSlots];
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;
  __shared__ __align__(16) float s_scale[kMaxN], s_shift[kMaxN];

  uint8_t *stage_base = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  int32_t *idx_ring = reinterpret_cast<int32_t *>(stage_base + (size_t)args.stages * args.stage_bytes);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int stages = args.stages;
  const uint32_t tmem_cols = (uint32_t)args.tmem_cols;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; s++) {
      // every producer lane + the weight tile's expect_tx
      mbar_init(&bar_full[s], kMode == kDense ? 1 : kProdWarps * 32 + 1);
      mbar_init(&bar_empty[s], 1);
    }
    for (int a = 0; a < 2; a++) { mbar_init(&bar_acc_full[a], 1); mbar_init(&bar_acc_empty[a], 4 * kEpiCols); }
    if (kMode != kDense)
      for (int i = 0; i < kIdxSlots; i++) { mbar_init(&bar_idx_full[i], 33); mbar_init(&bar_idx_empty[i], kProdWarps * 32); }
    if (args.claims != 0) {
      // read by the weight warp, the MMA warp and the epilogue warps
      for (int i = 0; i < kTileSlots; i++) { mbar_init(&bar_tile_full[i], 1); mbar_init(&bar_tile_empty[i], 2 + 4 * kEpiCols); }
      mbar_init(&bar_claim, 1);
    }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  wait_for_predecessor();
  // the first tile's offset bits, on their way while the rest is set up
  const int own_tile = args.num_tiles - 1 - (int)blockIdx.x;      // (the grid has no more blocks than tiles)
  uint32_t raw[kSub];
  if (warp == kIdxWarp) request_bits<kSub, kMode>(args, own_tile, raw);
  if (!kPairs && (args.scale != nullptr || args.shift != nullptr)) {
    for (int c = threadIdx.x; c < args.n_pad; c += threads_of(kMode)) {
      s_scale[c] = args.scale != nullptr && c < args.N ? __ldg(args.scale + c) : 1.f;
      s_shift[c] = args.shift != nullptr && c < args.N ? __ldg(args.shift + c) : 0.f;
    }
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&s_tmem_base)), "r"(tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  release_successor();   // every block has its tensor memory before another kernel's block can ask for some
  const uint32_t tmem_base = s_tmem_base;
  volatile int *abort_flag = &s_abort;
  // This CTA's tile after `tile` and its offset bits, for the warps of the roles that follow them (-1: no more).
  // The first is the block's own, which every role knows by itself; `turn` counts the others.
  uint32_t turn = 0;
  auto next_tile = [&](int &tile, uint32_t (&hb)[kSub]) {
    const uint32_t slot = turn % kTileSlots, phase = turn / kTileSlots & 1u;
    turn++;
    if (args.claims == 0) {
      tile = kMode > kMapNMajor ? max(tile - (int)gridDim.x, -1) : -1;   // (a map's grid has all its tiles then)
#pragma unroll
      for (int h = 0; h < kSub; h++) hb[h] = kMode > kMapNMajor ? 1u : 0u;
      return true;
    }
    if (!mbar_wait_warp(false, &bar_tile_full[slot], phase, abort_flag, args.status)) return false;
    tile = s_tile[slot];
    uint32_t seen = (uint32_t)tile;
#pragma unroll
    for (int h = 0; h < kSub; h++) { hb[h] = s_tile_bits[slot][h]; seen |= hb[h]; }
    __syncwarp();
    // (the loads have returned: the arrival's address depends on them, see the producers)
    if (lane == 0) mbar_arrive(&bar_tile_empty[slot] + (seen & (uint32_t)args.zero));
    return true;
  };

  if (kMode != kDense && warp < kProdWarps) {
    // ------------------------------ producers ---------------------------------
    // Lane l of warp w copies 16-byte piece l % kLpr of rows r0 .. r0 + kRpl - 1 of every
    // sub-tile, r0 = 16 w + kRpl (l / kLpr): the lane's indices are consecutive in the index
    // block (one 8- or 16-byte shared-memory load per offset and sub-tile), and a warp-wide
    // copy reads whole 128-byte lines.  Each lane's arrival on the stage barrier fires when its
    // copies have landed.
    constexpr int kRpl = kProdRows * kLpr / 32;   // rows per lane and sub-tile
    const int chunk = lane % kLpr;
    const int r0 = warp * kProdRows + (lane / kLpr) * kRpl;
    const uint32_t ring = smem_u32(stage_base);
    const uint32_t row_bytes = (uint32_t)args.K * 2u;
    uint32_t dst0[kRpl];                           // place of the lane's pieces inside a sub-tile
#pragma unroll
    for (int i = 0; i < kRpl; i++)
      dst0[i] = (uint32_t)(r0 + i) * 128u + (uint32_t)((chunk ^ ((r0 + i) & 7)) << 4);
    int stage = 0, slot = 0;
    uint32_t phase = 0, slot_phase = 0;
    bool alive = true;
    bool ready = mbar_test(&bar_empty[0], 1u), indices = false;
    while (alive) {
      if (!indices && !mbar_wait(&bar_idx_full[slot], slot_phase, abort_flag, args.status)) break;
      const uint32_t has = s_idx_has[slot];        // sub-tiles that have this offset; 0: no more steps
      int32_t q[kSub][kRpl];
#pragma unroll
      for (int h = 0; h < kSub; h++) {
        const int32_t *at = idx_ring + (slot * kSub + h) * kBM + r0;
        if (kRpl == 2) {
          const int2 v = *reinterpret_cast<const int2 *>(at);
          q[h][0] = v.x; q[h][1] = v.y;
        } else {
#pragma unroll
          for (int i = 0; i + 3 < kRpl; i += 4) {
            const int4 v = *reinterpret_cast<const int4 *>(at + i);
            q[h][i] = v.x; q[h][i + 1] = v.y; q[h][i + 2] = v.z; q[h][i + 3] = v.w;
          }
        }
      }
      if (has == 0u) break;
      // The slot may be refilled only once the loads above have RETURNED, not when they have been
      // issued: behind a queue of copies they were overtaken by the arrival and read the block of
      // eight steps later (one launch in a hundred on freshly built tables).  So every lane arrives for
      // its own loads, at an address that depends on their values through a mask that is zero at run
      // time and unknown to the compiler: whatever the slot holds (a sub-tile without this offset
      // leaves its block as it was, at first uninitialised), the arrival goes to this slot's
      // barrier.  No step of this loop waits for the warp: a lane that gave up leaves alone.
      // (One arrival per warp after a reduction over its lanes: 256->256 0.2 % slower, the rest the same.)
      uint32_t seen = 0u;
#pragma unroll
      for (int h = 0; h < kSub; h++)
#pragma unroll
        for (int i = 0; i < kRpl; i++) seen |= (uint32_t)q[h][i];
      mbar_arrive(&bar_idx_empty[slot] + (seen & (uint32_t)args.zero));
      if (++slot == kIdxSlots) { slot = 0; slot_phase ^= 1u; }
      indices = mbar_test(&bar_idx_full[slot], slot_phase);   // of the next step
      for (int kb = 0; kb < args.k_blocks; kb++) {
        if (!ready && !mbar_wait(&bar_empty[stage], phase ^ 1u, abort_flag, args.status)) {
          alive = false;
          break;
        }
        const uint32_t sa = ring + (uint32_t)(stage * args.stage_bytes);
        const int kcol = kb * kBK + chunk * 8;
        const uint8_t *src = args.in + kcol * 2;
        const bool inside = kcol < args.K;
        uint64_t *full = &bar_full[stage];
        if (++stage == stages) { stage = 0; phase ^= 1u; }
        ready = mbar_test(&bar_empty[stage], phase ^ 1u);   // of the next stage
#pragma unroll
        for (int h = 0; h < kSub; h++) {
          // a sub-tile without this offset has no index block, and no MMA reads its rows
          if (kSub > 1 && ((has >> h) & 1u) == 0u) continue;
#pragma unroll
          for (int i = 0; i < kRpl; i++) {
            const bool valid = q[h][i] >= 0 && inside;
            cp_async_16(sa + (uint32_t)(h * kBM * 128) + dst0[i],
                        valid ? src + (uint64_t)(uint32_t)q[h][i] * row_bytes : args.in, valid ? 16u : 0u);
          }
        }
        // this lane's arrival fires when its copies above have landed: no stall here
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(full))
                     : "memory");
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");   // nothing of this lane is in flight at exit
  } else if (warp == kMmaWarp) {
    // ------------------------------ MMA issuer --------------------------------
    const uint32_t fmt = args.elem_is_bf16 ? 1u : 0u;
    const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) |
                           ((uint32_t)(args.n_pad >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24) |
                           (kNMajor ? 1u << 16 : 0u);
    const uint64_t desc0 = umma_desc(smem_u32(stage_base));
    const uint64_t desc_b = kNMajor ? mn_major_desc(smem_u32(stage_base), kNBlock) : desc0;
    const uint32_t b_hi = (uint32_t)(desc_b >> 32), b_lo = (uint32_t)desc_b + ((uint32_t)args.a_bytes >> 4);
    constexpr uint32_t b_next = kNMajor ? kUmmaK * 128 / 16 : kUmmaK * 2 / 16;   // 16 steps along K
    const uint32_t desc_hi = (uint32_t)(desc0 >> 32), desc_lo = (uint32_t)desc0;
    const uint32_t stage_step = (uint32_t)args.stage_bytes >> 4;
    const int last_nk = (args.K - (args.k_blocks - 1) * kBK + kUmmaK - 1) / kUmmaK;
    int stage = 0, acc = 0;
    uint32_t phase = 0, acc_phase = 0;
    bool alive = true;
    bool ready = mbar_test(&bar_full[0], 0u);
    int tile = own_tile;
    uint32_t hb[kSub];
    request_bits<kSub, kMode>(args, tile, hb);
    take_bits<kSub>(args, tile, hb, hb);
    while (alive && tile >= 0) {
      uint32_t rest = union_of<kSub>(hb);
      if (!mbar_wait_warp(false, &bar_acc_empty[acc], acc_phase ^ 1u, abort_flag, args.status)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tmem_d = tmem_base + (uint32_t)(acc * kSub * args.n_pad);
      uint32_t begun = 0u;                                   // sub-tiles that have products already
      for (; alive && rest != 0u; rest &= rest - 1u) {
        const int p = __ffs(rest) - 1;
        for (int kb = 0; kb < args.k_blocks; kb++) {
          if (!mbar_wait_warp(ready, &bar_full[stage], phase, abort_flag, args.status)) { alive = false; break; }
          if (kMode != kDense) fence_generic_to_async();
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t lo = desc_lo + (uint32_t)stage * stage_step, lo_b = b_lo + (uint32_t)stage * stage_step;
          const int nk = kb + 1 < args.k_blocks ? kBK / kUmmaK : last_nk;
          uint64_t *empty = &bar_empty[stage];
          if (++stage == stages) { stage = 0; phase ^= 1u; }
          ready = mbar_test(&bar_full[stage], phase);      // of the next stage
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < kBK / kUmmaK; k++) {
              if (k < nk) {
                const uint64_t db = umma_desc_at(b_hi, lo_b + k * b_next);
#pragma unroll
                for (int h = 0; h < kSub; h++)                 // one weight tile, the sub-tiles that need it
                  if (kSub == 1 || ((hb[h] >> p) & 1u) != 0u)
                    umma_f16(tmem_d + (uint32_t)(h * args.n_pad),
                             umma_desc_at(desc_hi, lo + h * (kBM * 128 / 16) + k * (kUmmaK * 2 / 16)), db,
                             idesc, k == 0 && kb == 0 ? (begun >> h) & 1u : 1u);
              }
            }
            umma_commit(empty);
          }
        }
#pragma unroll
        for (int h = 0; h < kSub; h++) begun |= ((hb[h] >> p) & 1u) << h;
      }
      if (!alive) break;
      if (elect_one()) umma_commit(&bar_acc_full[acc]);
      if (++acc == args.acc_bufs) { acc = 0; acc_phase ^= 1u; }
      alive = next_tile(tile, hb);
    }
  } else if (warp == kTmaWarp) {
    // ------------------------------ weight tiles -------------------------------
    const uint32_t b_bytes = (uint32_t)(args.stage_bytes - args.a_bytes);
    const int my_order = lane < args.num_offsets && args.order != nullptr ? __ldg(args.order + lane) : lane;
    bool alive = true;
    int stage = 0;
    uint32_t phase = 0;
    bool ready = mbar_test(&bar_empty[0], 1u);
    int tile = own_tile;
    uint32_t hb[kSub];
    request_bits<kSub, kMode>(args, tile, hb);
    take_bits<kSub>(args, tile, hb, hb);
    while (alive && tile >= 0) {
      uint32_t rest = union_of<kSub>(hb);
      const int pair_row = kPairs ? pair_row_of_tile(args, tile) : 0;
      while (alive && rest != 0u) {
        const int p = kPairs ? pair_row : __ffs(rest) - 1;
        rest &= rest - 1u;
        const int widx = __shfl_sync(0xffffffffu, my_order, p);
        for (int kb = 0; kb < args.k_blocks; kb++) {
          if (!mbar_wait_warp(ready, &bar_empty[stage], phase ^ 1u, abort_flag, args.status)) { alive = false; break; }
          uint8_t *sb = stage_base + (size_t)stage * args.stage_bytes + args.a_bytes;
          uint64_t *full = &bar_full[stage];
          if (++stage == stages) { stage = 0; phase ^= 1u; }
          ready = mbar_test(&bar_empty[stage], phase ^ 1u);
          if (elect_one()) {
            mbar_expect_tx(full, b_bytes + (kMode == kDense ? (uint32_t)args.a_bytes : 0u));
            if (kMode == kDense) tma_load_2d(sb - args.a_bytes, &map_a, kb * kBK, tile * kBM, full);
            if (kNMajor) {
              for (int n = 0; n < args.n_pad; n += 64)
                tma_load_3d(sb + n / 64 * kNBlock, &map_b, n, kb * kBK, widx, full);
            } else {
              tma_load_3d(sb, &map_b, kb * kBK, 0, widx, full);
            }
          }
          __syncwarp();
        }
      }
      if (alive) alive = next_tile(tile, hb);
    }
  } else if (warp == kIdxWarp) {
    // ------------------------------ tiles and index blocks ---------------------
    // Tiles are handed out while the kernel runs: a CTA starts with the tile of its own number, counted from the last,
    // and takes over the tiles of blocks that have not started (cluster launch control) as it needs them, at most
    // kTileSlots before its epilogue.  With four the last CTAs had tiles left when others had none, with two the answer to a
    // request shows between tiles of few steps.  us, two / three / four: 464k rows 32->32 of 1.15 pairs with a residual 28.5 /
    // 28.7 / 29.5, 105k rows 128->128 of 3 with one 45.7 / 47.9 / 48.2, 420k 120.5 / 120.9 / 123.8; 290k rows 128->256 of 1.1
    // 53.1 / 52.0 / 52.0, 464k 192->48 of 1.15 45.8 / 44.9 / 44.4, 879k rows to strided ones 64->16 35.1 / 34.4 / 34.4.  Rows with many and rare offsets sort to the end, so the dear tiles go first.
    // With every gridDim-th tile for a CTA the busiest had 1.2 to 1.7 times the average of steps (one to
    // four clouds).  us, before / now: 406k rows of 3.4 pairs 64->64 70 / 59, 128->128 137 / 110, 256->256 328 /
    // 271; 1.8M of 9.3 256->256 3090 / 2810; 31k of 16.7 84 / 79.  The block's own tile is nobody's news, and where no
    // block waits for a place nothing is asked for: small layers had lost 0.2 us to that (20k rows 64->64, one offset, 5.30
    // dealt out, 5.50 asked for, 5.00 now; 128->128 6.32 / 6.63 / 6.12).
    //
    // 128 entries of the neighbour table per step and sub-tile, up to kIdxSlots steps ahead of the
    // producers, so that they never wait for an index from memory (loaded by the producers
    // themselves, even two steps ahead, they cost a quarter of the time).  A lane copies 16 bytes of
    // a block: no lane has to be elected, no byte count announced.  In one warp with the weight tiles a
    // step took that warp 1000 cycles and bound the layers of up to 64 channels (us, before / now: 464k rows
    // 32->32, 1.15 pairs a row, 37.7 / 32.8; 64->64 45 / 42; 406k 64->64, 3.4 pairs, 74.6 / 68; 123k 64->64,
    // 16.7 pairs, 70 / 62; 406k 64->128 90 / 86).
    const uint32_t ring = smem_u32(idx_ring) + (uint32_t)lane * 16u;
    int tile = own_tile;
    uint32_t phase = 0, claim_phase = 0, publish_phase = 0;
    int publish_slot = 0;
    bool claim_open = false;                       // an answer is on its way
    auto publish = [&](const uint32_t (&hb)[kSub]) {
      if (!mbar_wait_warp(false, &bar_tile_empty[publish_slot], publish_phase ^ 1u, abort_flag, args.status)) return false;
      if (lane == 0) {
        s_tile[publish_slot] = tile;
#pragma unroll
        for (int h = 0; h < kSub; h++) s_tile_bits[publish_slot][h] = hb[h];
        mbar_arrive(&bar_tile_full[publish_slot]);
      }
      __syncwarp();
      if (++publish_slot == kTileSlots) { publish_slot = 0; publish_phase ^= 1u; }
      return true;
    };
    int slot = 0;
    bool ready = true;
    // one step of the tile at `src`: offsets p of the sub-tiles in `has`; 0 marks the end
    auto send = [&](const int32_t *src, uint32_t has) {
      if (!mbar_wait_warp(ready, &bar_idx_empty[slot], phase ^ 1u, abort_flag, args.status)) return false;
      const uint32_t dst = ring + (uint32_t)(slot * kSub) * (kBM * 4);
#pragma unroll
      for (int h = 0; h < kSub; h++)
        if ((has >> h) & 1u) cp_async_16(dst + h * (kBM * 4), src + h * kBM, 16u);
      uint64_t *full = &bar_idx_full[slot];
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(full)) : "memory");
      if (lane == 0) {
        s_idx_has[slot] = has;
        mbar_arrive(full);
      }
      if (++slot == kIdxSlots) { slot = 0; phase ^= 1u; }
      ready = mbar_test(&bar_idx_empty[slot], phase ^ 1u);
      return true;
    };
    bool alive = true;
    while (alive) {
      uint32_t hb[kSub];
      take_bits<kSub>(args, tile, raw, hb);
      if (args.claims != 0 && tile != own_tile) alive = publish(hb);
      if (!alive || tile < 0) break;
      const int32_t *blocks = args.nbr + (int64_t)tile * (kSub * kBM) + lane * 4;
      for (uint32_t rest = kMode == kDense ? 0u : union_of<kSub>(hb); alive && rest != 0u; rest &= rest - 1u) {
        const int p = __ffs(rest) - 1;
        uint32_t has = 0u;
#pragma unroll
        for (int h = 0; h < kSub; h++) has |= ((hb[h] >> p) & 1u) << h;
        alive = send(blocks + (int64_t)p * args.pitch, has);
      }
      if (!alive) break;
      if (args.claims == 0) {
        tile = kPairs ? max(tile - (int)gridDim.x, -1) : -1;
        if (tile < 0) break;
        continue;
      }
      // the next tile, no earlier: a CTA that holds tiles it has not begun keeps them from one that is done
      if (lane == 0) {
        fence_generic_to_async();                  // the answer before has been read
        claim_block(&s_claim, &bar_claim);
      }
      claim_open = true;
      __syncwarp();
      if (!mbar_wait_warp(false, &bar_claim, claim_phase, abort_flag, args.status)) break;
      claim_open = false;
      claim_phase ^= 1u;
      const int block = claimed_block(&s_claim);
      __syncwarp();
      tile = block >= 0 ? args.num_tiles - 1 - block : -1;
      request_bits<kSub, kMode>(args, tile, raw);
    }
    if (alive && tile < 0 && kMode != kDense) send(args.nbr, 0u);
    // an answer that is still on its way lands before this block's shared memory goes
    if (claim_open) {
      for (uint32_t spin = 0; spin < 4096u && !mbar_try_wait(&bar_claim, claim_phase); spin++) {}
    }
    asm volatile("cp.async.wait_all;" ::: "memory");   // nothing of this lane is in flight at exit
  } else if (warp >= kEpiWarp) {
    // ------------------------------ epilogue ----------------------------------
    // A lane owns one accumulator row and takes it 16 columns at a time: one 32-byte store
    // (a whole sector of the output row, wherever perm puts it) and, with a residual, one
    // 32-byte load requested while the piece before is rounded and stored.  Two warps share a
    // quarter of the rows where there are eight: they take alternate pieces.  Stores stay 32 bytes a lane: rows
    // written by four lanes together (an exchange between lanes or through shared memory before) took the
    // same time or longer.
    // This role bounds the levels with few pairs a row (64->64, 1.15 pairs a row: the first tile of a CTA is in
    // flight after 8 us, then 2.3 a tile).  Not by the latency of its instructions, although every piece is a chain
    // of some 100: two groups of epilogue warps with a tile each took the same time.  What it spends is
    // the issue of scattered accesses: 32 lanes that each touch a line of their own.  It must not spill:
    // next to 200 KB of shared memory L1 keeps no local memory, and each reload of a spilled
    // register was a trip to L2 (with 32 bytes of spills 918k rows 32->32 took 66 us, without
    // 52; the pieces' registers are therefore single, not double, buffered).
    // tcgen05.ld reads the quarter of the tensor memory that the warp's number names
    const int quarter = warp & 3, group = (warp - kEpiWarp) >> 2;
    // two warps of a quarter take alternate pieces, or neighbouring ones where they copy residuals
    constexpr int kStep = kStaged ? 1 : kEpiCols;
    // (residuals are copied at three or four pieces)
    const int n = args.N, pieces = args.n_pad / 16, share = kStaged && kEpiCols == 2 ? 2 : (pieces + kEpiCols - 1) / kEpiCols;
    const int first_piece = kStaged ? group * share : group;
    const int last_piece = kStaged ? min(pieces, first_piece + share) : pieces;
    const bool affine = args.scale != nullptr || args.shift != nullptr;
    int acc = 0;
    uint32_t acc_phase = 0;
    // Row of the output (and of the residual) that this lane's accumulator row belongs to, per sub-tile (-1: none):
    // requested a tile ahead, so that the residual rows of the next tile can be on their way while this one is
    // worked on.
    const bool permuted = kMode <= kMapNMajor && args.perm != nullptr;
    auto table_row = [&](int tile, int h) { return ((int64_t)tile * kSub + h) * kBM + quarter * 32 + lane; };
    auto request_rows = [&](int tile, int32_t (&rows)[kSub]) {
#pragma unroll
      for (int h = 0; h < kSub; h++)
        if (permuted) rows[h] = load_ahead_1(args.perm + min(table_row(max(tile, 0), h), args.T - 1));
    };
    auto take_row = [&](int tile, int h, int32_t raw_row) {
      const int64_t row = table_row(tile, h);
      return tile >= 0 && row < args.T ? (permuted ? raw_row : (int32_t)row) : -1;
    };
    int32_t grow[kSub], next_rows[kSub] = {};
    int tile = own_tile, next = own_tile;
    uint32_t hb[kSub], next_hb[kSub];
    request_rows(tile, next_rows);
    request_bits<kSub, kMode>(args, tile, hb);
    take_bits<kSub>(args, tile, hb, hb);
    // Residuals of 33 to 64 columns come through a ring of this warp's own, one use of it (two pieces) ahead:
    // four lanes copy 64 bytes of a row, where a lane that reads its own row's pieces makes every load
    // 32 lines of 128 bytes.  64->64, us: 464k rows of 1.15 pairs 55.3 -> 48.5, 406k of 3.4 81 -> 76, 298k of 9.3
    // 94 -> 92, 2.7M of 1.15 229 -> 186.
    const uint32_t res_ring = smem_u32(idx_ring + kIdxSlots * kSub * kBM) + (uint32_t)((warp - kEpiWarp) * 2 * kResSlot);
    uint32_t res_turn = 0;                                    // the slot that is read next
    // copies the residual's pieces q and q + 1 of the quarter's rows (`row`: this lane's, -1: none)
    auto stage_residual = [&](uint32_t turn, int32_t row, int q) {
      const int k = lane & 3, c = q * 16 + k * 8;
      const bool inside = c < min(n, last_piece * 16);
      const uint32_t slot = res_ring + turn * kResSlot + (uint32_t)(lane >> 2) * 64u;
#pragma unroll
      for (int i = 0; i < 4; i++) {                           // rows 8 i + lane / 4
        const int32_t from = __shfl_sync(0xffffffffu, row, (lane >> 2) + 8 * i);
        if (from >= 0 && inside)
          cp_async_16(slot + (uint32_t)(i * 512) + ((uint32_t)(k ^ ((lane >> 3) & 3)) << 4),
                      args.residual + ((int64_t)from * n + c) * 2, 16u);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (kStaged && first_piece < last_piece) stage_residual(0u, take_row(tile, 0, next_rows[0]), first_piece);
    while (tile >= 0) {
#pragma unroll
      for (int h = 0; h < kSub; h++) grow[h] = take_row(tile, h, next_rows[h]);
      if (!next_tile(next, next_hb)) break;
      request_rows(next, next_rows);
      uint32_t res[8];
      // rows that are no whole number of 16-byte pieces (kDense): 8-byte pieces
      auto load_narrow = [&](const uint8_t *src, int c) {
        if (kMode == kDense && (n & 7) != 0) {
#pragma unroll
          for (int i = 0; i < 4; i++)
            if (c + 4 * i < n) {
              const uint2 v = *reinterpret_cast<const uint2 *>(src + 8 * i);
              res[2 * i] = v.x; res[2 * i + 1] = v.y;
            }
          return;
        }
        if (c < n) ld_global_16(src, res);
        if (c + 8 < n) ld_global_16(src + 16, res + 4);
      };
      auto load_residual = [&](int h, int c) {
#pragma unroll
        for (int i = 0; i < 8; i++) res[i] = 0u;
        if (args.residual == nullptr || grow[h] < 0) return;
        const uint8_t *src = args.residual + ((int64_t)grow[h] * n + c) * 2;
        if (args.wide && c + 16 <= n) {
          ld_global_32(src, res);
        } else {
          load_narrow(src, c);
        }
      };
      if (!kPairs && !kStaged) load_residual(0, first_piece * 16);
      if (!mbar_wait_warp(false, &bar_acc_full[acc], acc_phase, abort_flag, args.status)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (!kPairs && !kStaged && args.residual != nullptr) {
#pragma unroll
        for (int h = 0; h < kSub; h++) {
          const int32_t ahead = take_row(next, h, next_rows[h]);
          if (ahead < 0) continue;
          const uint8_t *row = args.residual + (int64_t)ahead * n * 2;
          for (int off = 0; off < n * 2; off += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + off));
        }
      }
#pragma unroll (kStaged ? 1 : kSub)
      for (int h = 0; h < kSub; h++) {
        // (kStaged: one body for both sub-tiles, two of them spill; no index into registers then)
        auto row_now = [&]() {
          if constexpr (kStaged) return h == 0 ? grow[0] : grow[kSub - 1];
          else return grow[h];
        };
        auto bits_now = [&]() {
          if constexpr (kStaged) return h == 0 ? hb[0] : hb[kSub - 1];
          else return hb[h];
        };
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) +
                               (uint32_t)((acc * kSub + h) * args.n_pad);
        auto piece = [&](int q) {
          uint32_t cur[16];
          __syncwarp();
          tmem_ld_32x16(taddr + (uint32_t)q * 16, cur);
          const bool more = q + kStep < last_piece;
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (!more && h + 1 == kSub) {
            // the last read of this accumulator set: the next tile's MMAs may have it
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            if (lane == 0) mbar_arrive(&bar_acc_empty[acc]);
          }
          const int c = q * 16;
          if (kPairs) {
            if (row_now() < 0) return;
            // pair mode: the fp32 accumulators of this row go out as they are
            float *dst = args.out_f32 + (int64_t)row_now() * n + c;
#pragma unroll
            for (int i = 0; i < 4; i++)
              if (c + 4 * i < n)
                *reinterpret_cast<float4 *>(dst + 4 * i) =
                    make_float4(__uint_as_float(cur[4 * i]), __uint_as_float(cur[4 * i + 1]),
                                __uint_as_float(cur[4 * i + 2]), __uint_as_float(cur[4 * i + 3]));
            return;
          }
          // one uniform branch per step of the epilogue and 16 independent values inside each: with
          // the branches inside the loop over the values a piece took 1300 cycles of latencies
          float f[16];
#pragma unroll
          for (int i = 0; i < 16; i++) f[i] = bits_now() == 0u ? 0.f : __uint_as_float(cur[i]);
          if (affine) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
              const float4 sc = *reinterpret_cast<const float4 *>(s_scale + c + 4 * i);
              const float4 sh = *reinterpret_cast<const float4 *>(s_shift + c + 4 * i);
              f[4 * i] = f[4 * i] * sc.x + sh.x;
              f[4 * i + 1] = f[4 * i + 1] * sc.y + sh.y;
              f[4 * i + 2] = f[4 * i + 2] * sc.z + sh.z;
              f[4 * i + 3] = f[4 * i + 3] * sc.w + sh.w;
            }
          }
          if (kStaged || args.residual != nullptr) {
            if (kStaged) {
              const uint32_t row = res_ring + res_turn * kResSlot + (uint32_t)lane * 64u;
              const uint32_t k = (uint32_t)((q - first_piece) & 1) * 2u ^ ((uint32_t)lane >> 1 & 3u);
              ld_shared_16(row + (k << 4), res);
              ld_shared_16(row + ((k ^ 1u) << 4), res + 4);
            }
            if (args.elem_is_bf16) {
#pragma unroll
              for (int i = 0; i < 8; i++) {
                f[2 * i] += elem_to_f32<true>((uint16_t)(res[i] & 0xffffu));
                f[2 * i + 1] += elem_to_f32<true>((uint16_t)(res[i] >> 16));
              }
            } else {
#pragma unroll
              for (int i = 0; i < 8; i++) {
                f[2 * i] += elem_to_f32<false>((uint16_t)(res[i] & 0xffffu));
                f[2 * i + 1] += elem_to_f32<false>((uint16_t)(res[i] >> 16));
              }
            }
          }
          if (kStaged) {
          } else if (more) load_residual(h, (q + kStep) * 16);
          else if (h + 1 < kSub) load_residual(h + 1, first_piece * 16);
          if (args.relu) {
#pragma unroll
            for (int i = 0; i < 16; i++) f[i] = fmaxf(f[i], 0.f);
          }
          if (row_now() < 0) return;
          uint32_t out[8];
          if (args.elem_is_bf16) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
              __nv_bfloat162 pk = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
              out[i] = *reinterpret_cast<uint32_t *>(&pk);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 8; i++) {
              __half2 pk = __floats2half2_rn(f[2 * i], f[2 * i + 1]);
              out[i] = *reinterpret_cast<uint32_t *>(&pk);
            }
          }
          uint8_t *dst = args.out16 + ((int64_t)row_now() * n + c) * 2;
          if (args.wide && c + 16 <= n) {
            st_global_32(dst, out);
          } else if (kMode == kDense && (n & 7) != 0) {
#pragma unroll
            for (int i = 0; i < 4; i++)
              if (c + 4 * i < n) *reinterpret_cast<uint2 *>(dst + 8 * i) = make_uint2(out[2 * i], out[2 * i + 1]);
          } else {
            if (c < n) *reinterpret_cast<uint4 *>(dst) = make_uint4(out[0], out[1], out[2], out[3]);
            if (c + 8 < n) *reinterpret_cast<uint4 *>(dst + 16) = make_uint4(out[4], out[5], out[6], out[7]);
          }
        };
        if (kEpiCols > 1 && first_piece >= last_piece && h + 1 == kSub) {   // no columns for this warp
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          if (lane == 0) mbar_arrive(&bar_acc_empty[acc]);
        }
        if constexpr (kStaged) {
          for (int q0 = first_piece; q0 < last_piece; q0 += 2) {
            __syncwarp();                                     // every lane has read the slot that is filled now
            const bool same = kEpiCols == 1 && q0 + 2 < last_piece;
            const int32_t row = same ? row_now() : h + 1 < kSub ? grow[kSub - 1] : take_row(next, 0, next_rows[0]);
            stage_residual(res_turn ^ 1u, row, same ? q0 + 2 : first_piece);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            for (int q = q0; q < min(q0 + 2, last_piece); q++) piece(q);
            res_turn ^= 1u;
            if (kEpiCols == 2) break;
          }
        } else {
          for (int q = first_piece; q < last_piece; q += kStep) piece(q);
        }
      }
      if (++acc == args.acc_bufs) { acc = 0; acc_phase ^= 1u; }
      tile = next;
#pragma unroll
      for (int h = 0; h < kSub; h++) hb[h] = next_hb[h];
    }
    asm volatile("cp.async.wait_all;" ::: "memory");   // nothing of this lane is in flight at exit
  }

  // ------------------------------ teardown ------------------------------------
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (s_abort) {
    for (int i = 0; i < 2000; i++) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(tmem_cols)
                 : "memory");
  }
}

// ---- neighbour table from masks --------------------------------------------------
struct CumSizes {
  int64_t cum[MN_MAX_OFFSETS + 1];
};

// Rows of a block of rank_to_source_kernel, four loads a thread in flight: with one, the launch was the
// rate at which 11 000 blocks start (105k rows, 27 offsets: 14.6 us).
constexpr int kRankRows = 1024;

// src_of_rank[cum[p] + source_masks[p, s]] = s.  Masks without hit words are a caller's own: a rank
// that their sizes have no place for, or that only one side has, makes no pair (the ranks start
// as -1).
__global__ void __launch_bounds__(256)
rank_to_source_kernel(const int32_t *__restrict__ source_masks, int64_t S, int O,
                      const __grid_constant__ CumSizes cs, int32_t *__restrict__ src_of_rank) {
  begin_early();
  const int p = blockIdx.y;
  const int32_t *mask = source_masks + (int64_t)p * S;
  const int64_t size = cs.cum[p + 1] - cs.cum[p];
  int32_t *out = src_of_rank + cs.cum[p];
  for (int64_t s0 = (int64_t)blockIdx.x * kRankRows + threadIdx.x; s0 < S; s0 += (int64_t)gridDim.x * kRankRows) {
    int m[kRankRows / 256];
#pragma unroll
    for (int i = 0; i < kRankRows / 256; i++) m[i] = s0 + i * 256 < S ? __ldg(mask + s0 + i * 256) : -1;
#pragma unroll
    for (int i = 0; i < kRankRows / 256; i++)
      if (m[i] >= 0 && m[i] < size) out[m[i]] = (int32_t)(s0 + i * 256);
  }
}

// the same from the sources' hit words: a source row reads only the mask entries of the
// offsets it takes part in (E entries instead of O * S)
__global__ void __launch_bounds__(256)
rank_to_source_bits_kernel(const int32_t *__restrict__ source_masks,
                           const uint32_t *__restrict__ source_bits, int64_t S,
                           const __grid_constant__ CumSizes cs, int32_t *__restrict__ src_of_rank) {
  begin_early();
  const int64_t gsz = (int64_t)gridDim.x * blockDim.x;
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < S; s += gsz) {
    for (uint32_t rest = __ldg(source_bits + s); rest != 0u; rest &= rest - 1u) {
      const int p = __ffs(rest) - 1;
      const int m = __ldg(source_masks + (int64_t)p * S + s);
      if (m >= 0) src_of_rank[cs.cum[p] + m] = (int32_t)s;
    }
  }
}

// nbr[p, r] = source row feeding target perm[r] (perm == NULL: target r) under mask row p
// (or -1); bit p of tile_bits[r / 128] is set when any row of that 128-row tile has such a
// source.  With the targets' hit words (`bits`) only the (tile, p) blocks whose bit is set
// are written, and a row looks its source up only for the offsets of its own word: the rest
// of the table is never read by the forward pass, which checks tile_bits first.  The rows of
// the table are `pitch` (T rounded up to 128) entries apart and -1 past T, so that the forward
// pass reads whole tiles with vector loads.
// What bounds it: a chain of dependent loads per thread.  With the offsets one after the other it was two trips
// to L2 for each of them (105k rows, 27 offsets: 19.5 us); the loads of kTableBatch offsets are in flight together.
constexpr int kTableBatch = 9;

__global__ void __launch_bounds__(128)
neighbor_table_kernel(const int32_t *__restrict__ target_masks, int64_t T, int64_t pitch, int O,
                      const __grid_constant__ CumSizes cs,
                      const int32_t *__restrict__ src_of_rank, const int32_t *__restrict__ perm,
                      const uint32_t *__restrict__ bits, int32_t *__restrict__ nbr,
                      uint32_t *__restrict__ tile_bits) {
  begin_early();
  __shared__ uint32_t s_bits;
  if (threadIdx.x == 0) s_bits = 0u;
  __syncthreads();
  const int64_t r = (int64_t)blockIdx.x * 128 + threadIdx.x;
  const int64_t t = (r < T && perm != nullptr) ? (int64_t)__ldg(perm + r) : r;
  if (bits != nullptr) {
    const uint32_t mine = r < T ? __ldg(bits + t) : 0u;
    const uint32_t warp_or = __reduce_or_sync(0xffffffffu, mine);
    if ((threadIdx.x & 31) == 0 && warp_or != 0u) atomicOr(&s_bits, warp_or);
    __syncthreads();
    const uint32_t tile = s_bits;
    if (threadIdx.x == 0) tile_bits[blockIdx.x] = tile;
    for (uint32_t rest = tile; rest != 0u;) {
      int p[kTableBatch], v[kTableBatch];
#pragma unroll
      for (int i = 0; i < kTableBatch; i++) {
        p[i] = rest != 0u ? __ffs(rest) - 1 : -1;
        rest &= rest - 1u;
        v[i] = p[i] >= 0 && ((mine >> p[i]) & 1u) ? __ldg(target_masks + (int64_t)p[i] * T + t) : -1;
      }
#pragma unroll
      for (int i = 0; i < kTableBatch; i++)
        if (v[i] >= 0) v[i] = __ldg(src_of_rank + cs.cum[p[i]] + v[i]);
#pragma unroll
      for (int i = 0; i < kTableBatch; i++)
        if (p[i] >= 0) nbr[(int64_t)p[i] * pitch + r] = v[i];
    }
    return;
  }
  uint32_t mine = 0u;
  for (int p0 = 0; p0 < O; p0 += kTableBatch) {
    int v[kTableBatch];
#pragma unroll
    for (int i = 0; i < kTableBatch; i++)
      v[i] = r < T && p0 + i < O ? __ldg(target_masks + (int64_t)(p0 + i) * T + t) : -1;
#pragma unroll
    for (int i = 0; i < kTableBatch; i++) {
      const int p = p0 + i;
      if (p >= O) break;
      const bool pair = v[i] >= 0 && v[i] < cs.cum[p + 1] - cs.cum[p];
      v[i] = pair ? __ldg(src_of_rank + cs.cum[p] + v[i]) : -1;
    }
#pragma unroll
    for (int i = 0; i < kTableBatch; i++) {
      if (p0 + i >= O) break;
      nbr[(int64_t)(p0 + i) * pitch + r] = v[i];
      mine |= (v[i] >= 0 ? 1u : 0u) << (p0 + i);
    }
  }
  mine = __reduce_or_sync(0xffffffffu, mine);
  if ((threadIdx.x & 31) == 0 && mine != 0u) atomicOr(&s_bits, mine);
  __syncthreads();
  if (threadIdx.x == 0) tile_bits[blockIdx.x] = s_bits;
}

// Rows of a neighbour table are sorted by hit word inside chunks of 2^shift rows (rows come in
// coordinate order, so a chunk is a region of space).  Over the whole table the order is best for
// skipping offsets, but a tile then gathers from everywhere, and once the feature rows outgrow the
// 126 MB L2 each of a row's pairs is a DRAM access of its own: 4.7M rows of 128 channels with 9.3
// pairs each took 4.5 ms (1.35 slots computed per pair); in chunks of 2^17 or 2^18 rows they take
// 2.8 ms (1.7 slots per pair), 1.9M rows of 256 channels 4.7 -> 4.15 ms.  Chunks from 2^16 to 2^19
// rows differ by less than 5 %.  With fewer than three pairs a row there is little to find again
// in L2 and the skipped offsets are worth more (7.1M rows of 32 channels, 1.6 pairs: 0.57 ms
// without chunks, 0.65 with), and half a million rows fit L2.  At most 32 chunks, and 32 key bits
// in all: another pass of the sort would cost more than smaller chunks give.
inline int row_chunk_shift(int64_t T, int64_t pairs, int64_t O) {
  const int chunk_bits = (int)std::min<int64_t>(5, 32 - O);
  if (T < (1 << 19) || pairs < 3 * T || chunk_bits <= 0) return 31;
  return std::max(17, rsort::bits_for(T) - chunk_bits);
}

}  // namespace

namespace {

template <int kSub, int kLpr, int kProdWarps, int kMode, bool kStaged = false>
mn_status launch_implicit(const ImArgs &a, const TcSizing &sizing, const CUtensorMap &map_a,
                          const CUtensorMap &map_b, cudaStream_t st) {
  auto kernel = conv_implicit_kernel<kSub, kLpr, kProdWarps, kMode, kStaged>;
  MN_RETURN_IF(allow_max_shared_memory(reinterpret_cast<const void *>(kernel)));
  ImArgs args = a;
  const int at_once = kNumSMs * sizing.ctas_per_sm;
  // Tiles of one offset cost the same and are dealt out up to some ten a CTA, with one CTA an SM always; narrow rows are
  // handed out.  1x1x1 layers, us, dealt out / handed out: 64->64 120k rows 7.3 / 8.2, 320k 13.6 / 15.7, 460k 21.3 / 21.0,
  // 1.5 M 70 / 58, with a residual 240k 19.0 / 19.5, 320k 28.0 / 26.6; 64->20 460k 13.5 / 14.8, with one 17.1 / 18.4, 700k
  // 25.0 / 21.4; 256->256 700k 141 / 147; 32->32 120k 7.2 / 7.1, 460k 19.3 / 17.8.  Pair products 32->32 103 / 105 (2184
  // tiles), 729 / 720 (30 754).
  int64_t dealt = 1;
  if (kMode > kMapNMajor && (kMode == kPairRows || a.K > 32))
    dealt = sizing.ctas_per_sm == 1 ? a.num_tiles : a.residual == nullptr || a.n_pad <= 32 ? 13 : 8;
  args.claims = a.num_tiles > dealt * at_once ? 1 : 0;
  const int grid = args.claims != 0 ? a.num_tiles : std::min(a.num_tiles, at_once);
  MN_LAUNCH(kMode == kPairRows ? "conv_implicit_kernel<pairs>" : kMode == kDense ? "conv_implicit_kernel<dense>"
                                                                                 : "conv_implicit_kernel", st,
            launch_early(kernel, (unsigned)grid, threads_of(kMode), sizing.smem_bytes, st, args, map_a, map_b));
  return MN_OK;
}

template <int kMode, bool kStaged>
mn_status launch_map(const ImArgs &a, int sub, const TcSizing &sizing, const CUtensorMap &map_b, cudaStream_t st) {
  if (sub == 1)
    return a.K <= 32 ? launch_implicit<1, 4, 4, kMode, kStaged>(a, sizing, map_b, map_b, st)
                     : launch_implicit<1, 8, 4, kMode, kStaged>(a, sizing, map_b, map_b, st);
  return a.K <= 32 ? launch_implicit<2, 4, 8, kMode, kStaged>(a, sizing, map_b, map_b, st)
                   : launch_implicit<2, 8, 8, kMode, kStaged>(a, sizing, map_b, map_b, st);
}

}  // namespace

mn_status launch_pair_products(const PairPlan &plan, int64_t S, int64_t c_in, int64_t c_out, bool bf16,
                               const void *sources, const void *weights_t, int O,
                               const int32_t *pair_src, const int32_t *order, float *products,
                               int32_t *status_dev, cudaStream_t st) {
  (void)S;
  MN_CHECK_ARG(plan.total_rows > 0 && plan.total_rows % kBM == 0 && plan.total_rows < (1ll << 31),
               "pair products: bad product row count");
  MN_CHECK_ARG(((reinterpret_cast<uintptr_t>(sources) | reinterpret_cast<uintptr_t>(products) |
                 reinterpret_cast<uintptr_t>(weights_t) | reinterpret_cast<uintptr_t>(pair_src)) & 15) == 0,
               "pair products: arrays must be 16-byte aligned");
  ImArgs a{};
  a.in = static_cast<const uint8_t *>(sources);
  a.nbr = pair_src;
  a.tile_bits = nullptr;
  a.order = order;
  a.status = status_dev;
  a.T = plan.total_rows;
  a.K = (int)c_in;
  a.N = (int)c_out;
  a.n_pad = (int)align_up((size_t)c_out, 16);
  a.k_blocks = (int)div_up(c_in, kBK);
  a.n_tiles128 = (int)(plan.total_rows / kBM);
  a.pitch = plan.total_rows;
  a.acc_bufs = 2;
  a.a_bytes = kBM * kBK * 2;
  a.stage_bytes = a.a_bytes + a.n_pad * kBK * 2;
  const TcSizing sizing = size_tc_kernel(a.stage_bytes, a.acc_bufs * a.n_pad, kMaxStages, kImCtas, kIdxSlots * kMaxSub * kBM * 4, kMaxStages);
  a.stages = sizing.stages;
  a.tmem_cols = sizing.tmem_cols;
  a.num_offsets = O;
  a.elem_is_bf16 = bf16 ? 1 : 0;
  a.num_tiles = a.n_tiles128;
  a.pair_rows = plan.num_rows;
  for (int p = 0; p <= MN_MAX_PAIR_ROWS; p++) a.pair_tile_prefix[p] = plan.tile_prefix[p];
  a.out_f32 = products;
  CUtensorMap map_b;
  MN_RETURN_IF(make_kmajor_map(&map_b, weights_t, bf16, c_in, c_out, O, a.n_pad));
  return c_in <= 32 ? launch_implicit<1, 4, 8, kPairRows>(a, sizing, map_b, map_b, st)
                    : launch_implicit<1, 8, 8, kPairRows>(a, sizing, map_b, map_b, st);
}

// out = relu?((features @ weights) * scale + shift + residual), c_out a multiple of 4
mn_status launch_dense_rows(int64_t rows, int64_t c_in, int64_t c_out, bool bf16, const void *features,
                            const void *weights_t, const float *scale, const float *shift, const void *residual,
                            bool relu, void *out, int32_t *status_dev, cudaStream_t st) {
  ImArgs a{};
  a.scale = scale;
  a.shift = shift;
  a.residual = static_cast<const uint8_t *>(residual);
  a.out16 = static_cast<uint8_t *>(out);
  a.status = status_dev;
  a.T = rows;
  a.K = (int)c_in;
  a.N = (int)c_out;
  a.n_pad = (int)align_up((size_t)c_out, 16);
  a.k_blocks = (int)div_up(c_in, kBK);
  a.n_tiles128 = a.num_tiles = (int)div_up(rows, kBM);
  a.acc_bufs = 2;
  a.a_bytes = kBM * kBK * 2;
  a.stage_bytes = a.a_bytes + a.n_pad * kBK * 2;
  const TcSizing sizing = size_tc_kernel(a.stage_bytes, a.acc_bufs * a.n_pad, kMaxStages, kImCtas, kIdxSlots * kMaxSub * kBM * 4, kMaxStages);
  a.stages = sizing.stages;
  a.tmem_cols = sizing.tmem_cols;
  a.num_offsets = 1;
  a.elem_is_bf16 = bf16 ? 1 : 0;
  a.relu = relu ? 1 : 0;
  a.wide = c_out % 16 == 0 && ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(residual)) & 31) == 0;
  CUtensorMap map_a, map_b;
  MN_RETURN_IF(make_kmajor_map(&map_a, features, bf16, c_in, rows, 0, kBM));
  MN_RETURN_IF(make_kmajor_map(&map_b, weights_t, bf16, c_in, c_out, 1, a.n_pad));
  return launch_implicit<1, 8, 4, kDense>(a, sizing, map_a, map_b, st);
}

}  // namespace mn

using namespace mn;

extern "C" int mn_implicit_supported(int64_t O, int64_t c_in, int64_t c_out, mn_dtype dtype) {
  return (dtype == MN_F16 || dtype == MN_BF16) && O >= 1 && O <= 32 && c_in >= 8 && c_in % 8 == 0 &&
         c_out >= 8 && c_out % 8 == 0 && c_out <= 256;
}

extern "C" size_t mn_neighbor_table_workspace_bytes(const int32_t *sizes_host, int64_t O, int64_t T) {
  int64_t e = 0;
  for (int64_t p = 0; p < O; p++) e += sizes_host[p];
  const size_t n = (size_t)std::max<int64_t>(T, 1);
  const size_t sort = 2 * align_up(n * 8, 256) + rsort::workspace_bytes(T);
  return align_up((size_t)std::max<int64_t>(e, 1) * sizeof(int32_t), 256) + sort + 1024;
}

extern "C" mn_status mn_build_neighbor_table(const int32_t *source_masks,
                                             const int32_t *target_masks,
                                             const int32_t *sizes_host, int64_t O, int64_t S,
                                             int64_t T, const uint32_t *source_bits,
                                             const uint32_t *target_bits,
                                             int32_t *nbr_out, uint32_t *tile_bits_out,
                                             int32_t *perm_out, int32_t *ctrl, void *ws_ptr,
                                             size_t ws_bytes, void *stream) {
  MN_CHECK_ARG(O >= 1 && O <= 32, "neighbor table: %lld offsets (supported: 1..32)", (long long)O);
  MN_CHECK_ARG(S >= 0 && T >= 0 && T < (1ll << 31) && sizes_host != nullptr,
               "neighbor table: bad arguments");
  if (T == 0) return MN_OK;
  MN_CHECK_ARG(source_masks != nullptr && target_masks != nullptr && nbr_out != nullptr &&
                   tile_bits_out != nullptr, "neighbor table: null pointer");
  MN_CHECK_ARG(perm_out == nullptr || (target_bits != nullptr && ctrl != nullptr),
               "neighbor table: a row permutation needs the targets' hit words and a control block");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  CumSizes cs{};
  for (int64_t p = 0; p < O; p++) {
    MN_CHECK_ARG(sizes_host[p] >= 0 && sizes_host[p] <= std::min(S, T), "neighbor table: bad size");
    cs.cum[p + 1] = cs.cum[p] + sizes_host[p];
  }
  Workspace ws(ws_ptr, ws_bytes);
  int32_t *src_of_rank = ws.take<int32_t>((size_t)std::max<int64_t>(cs.cum[O], 1));
  MN_CHECK_WS(ws);
  if (perm_out != nullptr) {
    // stable sort of the rows by hit word: perm[r] = target row at position r
    uint64_t *keys = ws.take<uint64_t>(T), *keys_tmp = ws.take<uint64_t>(T);
    MN_CHECK_WS(ws);
    rsort::Args a{};
    a.keys[0] = keys; a.keys[1] = keys_tmp;
    a.n = T;
    a.first_bit = rsort::bits_for(T);
    const int chunk_shift = row_chunk_shift(T, cs.cum[O], O);
    a.bits = (int)O + (T > (1ll << chunk_shift) ? rsort::bits_for(((T - 1) >> chunk_shift) + 1) : 0);
    a.status = ctrl + MN_CTRL_STATUS;
    a.index32 = perm_out;
    MN_RETURN_IF(rsort::run(a, HitWordKeys{target_bits, (int32_t)O, a.first_bit, chunk_shift}, ws, st));
  }
  if (target_bits == nullptr)
    MN_CHECK_CUDA(cudaMemsetAsync(src_of_rank, 0xff, sizeof(int32_t) * (size_t)std::max<int64_t>(cs.cum[O], 1), st));
  // a scattered 4-byte read costs a 32-byte sector: worth it while the pairs are fewer than
  // an eighth of the mask entries
  if (S > 0 && source_bits != nullptr && cs.cum[O] * 8 < O * S) {
    const int blocks = (int)std::min<int64_t>(kNumSMs * 16, div_up(S, 256));
    MN_LAUNCH("rank_to_source_bits_kernel", st,
              launch_early(rank_to_source_bits_kernel, blocks, 256, 0, st, source_masks, source_bits, S, cs,
                                                                  src_of_rank));
  } else if (S > 0) {
    const dim3 grid((unsigned)std::min<int64_t>(kNumSMs * 4, div_up(S, kRankRows)), (unsigned)O);
    MN_LAUNCH("rank_to_source_kernel", st,
              launch_early(rank_to_source_kernel, grid, 256, 0, st, source_masks, S, (int)O, cs, src_of_rank));
  }
  MN_LAUNCH("neighbor_table_kernel", st,
            launch_early(neighbor_table_kernel, (unsigned)div_up(T, 128), 128, 0, st, 
                target_masks, T, (int64_t)align_up((size_t)T, kBM), (int)O, cs, src_of_rank, perm_out,
                target_bits, nbr_out, tile_bits_out));
  return MN_OK;
}

extern "C" size_t mn_implicit_workspace_bytes(int64_t O, int64_t c_in, int64_t c_out) {
  return align_up((size_t)O * c_in * c_out * 2, 1024) + 1024;
}

extern "C" mn_status mn_sparse_convolution_forward_implicit(
    int64_t S, int64_t T, int64_t O, int64_t c_in, int64_t c_out, mn_dtype dtype,
    const void *sources, const void *weights, const void *weights_t_in, const int32_t *nbr,
    const uint32_t *tile_bits, const int32_t *perm,
    const int32_t *order, const float *scale, const float *shift, const void *residual, int relu,
    double pairs_per_row, int sub_hint, void *targets_out, int32_t *status_dev, void *ws_ptr,
    size_t ws_bytes, void *stream) {
  if (!mn_implicit_supported(O, c_in, c_out, dtype)) {
    set_error("implicit forward: needs fp16/bf16, at most 32 offsets, channels multiple of 8, "
              "c_out <= 256 (got O=%lld c_in=%lld c_out=%lld dtype=%d)", (long long)O,
              (long long)c_in, (long long)c_out, (int)dtype);
    return MN_ERR_UNSUPPORTED;
  }
  MN_CHECK_ARG(S >= 0 && T >= 0 && T < (1ll << 31) && S < (1ll << 31), "implicit forward: bad sizes");
  if (T == 0) return MN_OK;
  MN_CHECK_ARG((weights != nullptr || weights_t_in != nullptr) && nbr != nullptr && tile_bits != nullptr &&
                   targets_out != nullptr && status_dev != nullptr && (S == 0 || sources != nullptr),
               "implicit forward: null pointer");
  MN_CHECK_ARG(((reinterpret_cast<uintptr_t>(sources) | reinterpret_cast<uintptr_t>(targets_out) |
                 reinterpret_cast<uintptr_t>(residual) | reinterpret_cast<uintptr_t>(nbr)) & 15) == 0,
               "implicit forward: feature arrays and the neighbour table must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool bf16 = dtype == MN_BF16;
  // Weights that were not transposed once are read as they are, as N-major tiles, where a call has
  // few steps: the transposition is a launch of 3 to 10 us, an N-major step a little slower than a
  // K-major one.  With fewer than two pairs a row the MMAs wait for the rest anyway (464k rows
  // 64->64, 1.15 pairs: 56.3 -> 53.8 us; 168k rows 64->128, 1.4 pairs: 23.4 -> 20.5 us); up to four
  // tiles per SM (two per CTA where two CTAs share one) the launch is what counts (53k rows
  // 256->256: 95.5 -> 92.1 us, 30k rows 32->96: 13.9 -> 12.0 us).  The line is drawn through these few
  // layers: 200k rows 64->64 with 3 pairs a row would lose 1 of 115 us beyond it.  TMA needs the
  // weights on a 16-byte boundary.
  Workspace ws(ws_ptr, ws_bytes);
  const void *weights_t = weights_t_in;
  const bool n_major = weights_t == nullptr && (reinterpret_cast<uintptr_t>(weights) & 15) == 0 &&
                       (pairs_per_row < 2.0 || div_up(T, kBM) <= 4 * kNumSMs);
  if (n_major) {
    weights_t = weights;
  } else if (weights_t == nullptr) {
    char *mine = ws.take<char>(align_up((size_t)O * c_in * c_out * 2, 1024));
    MN_CHECK_WS(ws);
    MN_RETURN_IF(launch_transpose_weights(weights, mine, (int)O, (int)c_in, (int)c_out, bf16, st));
    weights_t = mine;
  }

  ImArgs a{};
  a.in = static_cast<const uint8_t *>(sources);
  a.nbr = nbr;
  a.tile_bits = tile_bits;
  a.order = order;
  a.scale = scale;
  a.shift = shift;
  a.residual = static_cast<const uint8_t *>(residual);
  a.perm = perm;
  a.out16 = static_cast<uint8_t *>(targets_out);
  a.status = status_dev;
  a.T = T;
  a.K = (int)c_in;
  a.N = (int)c_out;
  a.n_pad = (int)align_up((size_t)c_out, 16);
  a.k_blocks = (int)div_up(c_in, kBK);
  a.n_tiles128 = (int)div_up(T, kBM);
  // One sub-tile: four producer and eight epilogue warps (918k rows 32->32 52 -> 50 us against
  // eight and four, 243k rows 128->256 with stride 2 90 -> 78 us, 464k rows 64->64 45 -> 42 us); two
  // sub-tiles: twice the rows to fetch per step, eight producers (128->128 with 9.4 pairs a row 387
  // against 395 us).
  // Sub-tiles per CTA tile.  The two sub-tiles of a CTA tile share the steps' bookkeeping and the weight
  // tile of a stage, at the price of a shallower ring, fewer epilogue warps and tiles twice as large; a sub-tile
  // is skipped in the steps of offsets that only the other one has.  It pays where the bookkeeping
  // bounds a step and every CTA has several tiles.  us, 1 / 2 sub-tiles, of one layer at a time (14k tiles and more: at the
  // power limit, near 1.5 GHz).  32->32: 938 tiles of 1.15 pairs a row 10.6 / 15.2, 2026 of 1.1 15.2 / 16.7, 1849 of 5.4
  // 40.3 / 37.7, 3629 of 1.15 22.4 / 20.8, 57k of 1.15 279 / 226.  64->64: 3176 of 3.5 49.0 / 49.4, with a residual 54.6 /
  // 57.7, 5456 of 5.4 153 / 145, 57k of 1.15 365 / 332, with one 447 / 462, 37k of 9.3 1077 / 982.  Beyond 64 columns few
  // pairs leave the epilogue as the bound, which has half the warps with two.  64->128: 57k of 1.15 537 / 758, 50k of 3.4
  // 1033 / 1111, 5456 of 5.4 189 / 182, 9257 of 9.3 345 / 327, 878 of 12.6 39.8 / 40.3, with a residual 49.5 / 53.8.  128->128:
  // 12.6k of 3.5 416 / 415, with one 592 / 612, 10.1k of 7.5 541 / 527 and 683 / 638, 2331 of 9.3 153 / 148, 1083 of 7.2
  // 58.7 / 59.3.  More input channels are more steps a tile, and without a residual the epilogue has less to do.  Without / with
  // one: 192->128, 3.0k tiles of 3.0 117 / 115, 145 / 154; 4.8k of 2.6 158 / 154, 199 / 215; 4.8k of 2.0 125 / 126, 168 / 193;
  // 2.6k of 4.6 144 / 138, 167 / 171; 5.1k of 4.6 298 / 285, 341 / 339.  256->128, 4.8k of 2.6 203 / 195, 243 / 252; 10.4k of 3.0 484 /
  // 460, 585 / 610; 5.1k of 4.6 387 / 375, 439 / 436.  128->128, 3.0k of 3.0 88.2 / 88.6, 117 / 130; 4.8k of 2.6 118 / 118,
  // 161 / 184; 10.4k of 3.0 273 / 262, 364 / 408; 5.1k of 4.6 214 / 204, 256 / 262.  128->96 5.2k of 3.0 141 / 144, 10.4k 236 / 231.
  // 128->64 0.96 to 1.04, 256->256 336 / 404.  Callers that have timed the layer pass their own choice.
  int sub = sub_hint;
  if (sub <= 0) {
    const double tiles = a.n_tiles128;
    sub = 1;
    if (c_in <= 32 && a.n_pad <= 32) {
      if (tiles >= 24 * kNumSMs) sub = 2;
    } else if (c_in <= 64 && a.n_pad <= 64) {
      if (pairs_per_row >= 3.0 && tiles >= 16 * kNumSMs && tiles * pairs_per_row >= 16384) sub = 2;
    } else if (a.n_pad > 64 && a.n_pad <= 128) {
      const bool many = tiles >= 32 * kNumSMs;
      const double line = a.residual != nullptr ? (c_in > 128 && many ? 3.6 : 5.0) : c_in > 128 ? 2.5 : c_in > 64 && many ? 3.0 : 5.0;
      if (pairs_per_row >= line && tiles >= 16 * kNumSMs) sub = 2;
    }
  }
  MN_CHECK_ARG(sub_hint <= 4 && (sub_hint <= 0 || sub_hint * a.n_pad <= 512),
               "implicit forward: %d sub-tiles of %d columns do not fit TMEM", sub_hint, a.n_pad);
  sub = std::min(sub, kMaxSub);
  a.pitch = (int64_t)align_up((size_t)T, kBM);
  a.acc_bufs = 2 * sub * a.n_pad <= 512 ? 2 : 1;
  a.a_bytes = sub * kBM * kBK * 2;
  a.stage_bytes = a.a_bytes + (n_major ? (int)div_up(a.n_pad, 64) * kNBlock : a.n_pad * kBK * 2);
  // The residual's ring: two slots of 32 rows per epilogue warp.  At 32 columns rows of 64 bytes are two sectors for
  // two lanes either way (464k rows, 1.15 pairs: 37.9 / 39.8 us, 336k, 7 pairs 61.4 / 63.5), and beyond 64 the
  // 32 KB are a stage or two of the ring.
  const bool staged = residual != nullptr && a.n_pad > 32 && a.n_pad <= 64;
  const int rings = kIdxSlots * sub * kBM * 4 + (staged ? (sub == 1 ? 8 : 4) * 2 * kResSlot : 0);
  const TcSizing sizing = size_tc_kernel(a.stage_bytes, a.acc_bufs * sub * a.n_pad, kMaxStages, kImCtas, rings, kMaxStages);
  a.stages = sizing.stages;
  a.tmem_cols = sizing.tmem_cols;
  a.num_offsets = (int)O;
  a.elem_is_bf16 = bf16 ? 1 : 0;
  a.num_tiles = (int)div_up(a.n_tiles128, sub);
  a.relu = relu ? 1 : 0;
  a.wide = c_out % 16 == 0 && ((reinterpret_cast<uintptr_t>(targets_out) |
                                reinterpret_cast<uintptr_t>(residual)) & 31) == 0;

  CUtensorMap map_b;
  MN_RETURN_IF(n_major ? make_kmajor_map(&map_b, weights_t, bf16, c_out, c_in, O, kBK)
                       : make_kmajor_map(&map_b, weights_t, bf16, c_in, c_out, O, a.n_pad));
  if (n_major)
    return staged ? launch_map<kMapNMajor, true>(a, sub, sizing, map_b, st)
                           : launch_map<kMapNMajor, false>(a, sub, sizing, map_b, st);
  return staged ? launch_map<kMap, true>(a, sub, sizing, map_b, st) : launch_map<kMap, false>(a, sub, sizing, map_b, st);
}
