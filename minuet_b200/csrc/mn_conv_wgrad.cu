// Weight gradients of a sparse convolution: for every kernel offset k
//   dW[k] = sum over the pairs (s, t) of k of x[s]^T dout[t]      ([c_in, c_out], fp32 sums)
// The reference has no backward pass.  One launch covers all offsets: the pairs of an offset
// are cut into items, a block owns one item, fetches both rows of every pair straight into
// shared memory and leaves one partial matrix; a second launch adds the partial matrices of
// an offset in item order (no atomics: the same bits every time) and converts.
//
// wgrad_tc_kernel (fp16/bf16): the contraction runs over PAIRS, so the gathered rows are
// used as they lie in memory, channels contiguous: both operands are M/N-major tiles of
// 64 channels x 64 pairs with 128-byte swizzle, and no transpose exists anywhere.
// wgrad_simt_kernel (fp32, and the 16-bit shapes the tensor-core kernel does not take):
// FFMA outer products over the same tiles.
//
// Bound: both rows of every pair come from L2 (E (c_in + c_out) e bytes; the arrays
// themselves fit it), the products are 2 E c_in c_out flop.  200 000 indoor voxels, 64 -> 64,
// fp16 (600 000 pairs): 39 us for the two launches, against 4.2 ms for the index selections and
// one library GEMM per offset that stood here (27 host reads and 700 launches on top).
#include "mn_tc.cuh"

#include <algorithm>

namespace mn {

namespace {

using namespace tc;

constexpr int kPairRows = 128;    // the pairs of an offset start on multiples of this in the lists

// Where the pairs of every mask row lie in the pair lists, and how they are cut into items.
struct WgradPlan {
  int64_t row_begin[MN_MAX_OFFSETS + 1];   // first list entry of mask row p
  int32_t item_prefix[MN_MAX_OFFSETS + 1]; // first item of mask row p
  int32_t num_rows;                        // O
  int32_t item_rows;                       // list entries per item, a multiple of 64
};

struct WgradArgs {
  const void *x;             // [S, c_in]
  const void *g;             // [T, c_out]
  const int32_t *pair_src;   // source row of every pair, -1 in the padding; null: row i of both arrays is pair i (FFMA only)
  const int32_t *pair_dst;   // target row of every pair, -1 in the padding
  float *partial;            // [items, c_in, c_out]
  int32_t *status;
  int64_t rows;              // of both arrays, where there are no lists
  int32_t c_in, c_out, n_pad;
  int32_t a_blocks, b_blocks;   // 64-channel blocks of one stage
  int32_t m_tiles;              // 128-channel accumulator tiles of this block
  int32_t stages, stage_bytes, tmem_cols, elem_is_bf16;
};

__device__ __forceinline__ int row_of_item(const WgradPlan &plan, int item) {
  int lo = 0, hi = plan.num_rows;   // last p with item_prefix[p] <= item
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (plan.item_prefix[mid] <= item) lo = mid; else hi = mid;
  }
  return lo;
}

// ---------------------------------------------------------------------------
// pair lists
// ---------------------------------------------------------------------------

// list[row_begin[p] + masks[p, r]] = r for every entry of the masks; with `bits` (hit words)
// only the entries that exist are looked at.
// What bounds it: a row's loads, when they follow one another (the stores between them keep the order).  With
// kPairBatch of them in flight: 27 offsets of 58 800 rows 7.7 us -> 5.5, of 15 700 rows 12.5 -> 7 (more pairs a row).
constexpr int kPairBatch = 9;

__global__ void __launch_bounds__(256)
pair_side_kernel(const int32_t *__restrict__ masks, const uint32_t *__restrict__ bits, int64_t rows,
                 const __grid_constant__ WgradPlan plan, int32_t *__restrict__ list) {
  begin_early();
  const int64_t gsz = (int64_t)gridDim.x * blockDim.x;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gsz) {
    if (bits != nullptr) {
      for (uint32_t w = __ldg(bits + r); w != 0u;) {
        int p[kPairBatch], m[kPairBatch];
#pragma unroll
        for (int i = 0; i < kPairBatch; i++) {
          p[i] = w != 0u ? __ffs(w) - 1 : 0;
          m[i] = w != 0u ? __ldg(masks + (int64_t)p[i] * rows + r) : -1;
          w &= w - 1u;
        }
#pragma unroll
        for (int i = 0; i < kPairBatch; i++)
          if (m[i] >= 0) list[plan.row_begin[p[i]] + m[i]] = (int32_t)r;
      }
    } else {
      const int p = blockIdx.y;
      const int m = __ldg(masks + (int64_t)p * rows + r);
      // a caller's own masks: a rank beyond the row's list makes no pair
      if (m >= 0 && m < plan.row_begin[p + 1] - plan.row_begin[p]) list[plan.row_begin[p] + m] = (int32_t)r;
    }
  }
}

// ---------------------------------------------------------------------------
// fp16 / bf16
// ---------------------------------------------------------------------------
constexpr int kWgWarps = 8;             // producers; all of them write the result
constexpr int kWgMmaWarp = kWgWarps;
constexpr int kWgThreads = (kWgWarps + 1) * 32;
constexpr int kWgRows = 64;             // pairs per stage
constexpr int kWgBlock = kWgRows * 128; // bytes of 64 pairs x 64 channels
constexpr int kWgMaxStages = 8;

__device__ __forceinline__ void wg_copy_16(uint32_t dst, const void *src, uint32_t src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes)
               : "memory");
}

// issued where it stands (an ordinary read-only load may be moved down to its first use)
__device__ __forceinline__ int2 load_pair_rows(const int32_t *src) {
  int2 v;
  asm volatile("ld.global.nc.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(src));
  return v;
}

__global__ void __launch_bounds__(kWgThreads, 2)
wgrad_tc_kernel(const __grid_constant__ WgradArgs a, const __grid_constant__ WgradPlan plan) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ uint64_t bar_full[kWgMaxStages], bar_empty[kWgMaxStages], bar_done;
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;
  uint8_t *stage_base = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int stages = a.stages;
  const int item = blockIdx.x;
  const int p = row_of_item(plan, item);
  const int64_t first = plan.row_begin[p] + (int64_t)(item - plan.item_prefix[p]) * plan.item_rows;
  const int64_t last = min(plan.row_begin[p + 1], first + plan.item_rows);
  const int n_stage = (int)((last - first) / kWgRows);
  const int c0 = blockIdx.y * (a.a_blocks * 64);   // first input channel of this block

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; s++) {
      mbar_init(&bar_full[s], kWgWarps * 32);
      mbar_init(&bar_empty[s], 1);
    }
    mbar_init(&bar_done, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  wait_for_predecessor();
  if (warp == kWgMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&s_tmem_base)), "r"((uint32_t)a.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  release_successor();   // every block has its tensor memory before another kernel's block can ask for some
  const uint32_t tmem_base = s_tmem_base;
  volatile int *abort_flag = &s_abort;

  if (warp < kWgWarps) {
    // Warp w fetches pairs 8w .. 8w + 7 of every stage: eight lanes copy one 128-byte slice
    // (64 channels) of a row, two rows per lane; the list entries of the next stage are on
    // their way while this one is copied.
    const int chunk = lane & 7;
    const int r0 = warp * 8 + (lane >> 3) * 2;
    const uint32_t ring = smem_u32(stage_base);
    uint32_t dst0[2];
#pragma unroll
    for (int i = 0; i < 2; i++)
      dst0[i] = (uint32_t)(r0 + i) * 128u + (uint32_t)((chunk ^ ((r0 + i) & 7)) << 4);
    const int32_t *ps = a.pair_src + first + r0, *pd = a.pair_dst + first + r0;
    int stage = 0;
    uint32_t phase = 0;
    bool alive = true;
    auto copy = [&](int2 s, int2 t) {
      if (!mbar_wait(&bar_empty[stage], phase ^ 1u, abort_flag, a.status)) { alive = false; return; }
      const uint32_t sa = ring + (uint32_t)(stage * a.stage_bytes);
      const uint8_t *x = static_cast<const uint8_t *>(a.x), *g = static_cast<const uint8_t *>(a.g);
      for (int b = 0; b < a.a_blocks; b++) {
        const int c = c0 + b * 64 + chunk * 8;
        const bool in = c < a.c_in;
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const int row = i == 0 ? s.x : s.y;
          const bool valid = in && row >= 0;
          wg_copy_16(sa + (uint32_t)(b * kWgBlock) + dst0[i],
                     valid ? x + ((int64_t)row * a.c_in + c) * 2 : x, valid ? 16u : 0u);
        }
      }
      const uint32_t sb = sa + (uint32_t)(a.a_blocks * kWgBlock);
      for (int b = 0; b < a.b_blocks; b++) {
        const int c = b * 64 + chunk * 8;
        const bool in = c < a.c_out;
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const int row = i == 0 ? t.x : t.y;
          const bool valid = in && row >= 0;
          wg_copy_16(sb + (uint32_t)(b * kWgBlock) + dst0[i],
                     valid ? g + ((int64_t)row * a.c_out + c) * 2 : g, valid ? 16u : 0u);
        }
      }
      asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&bar_full[stage]))
                   : "memory");
      if (++stage == stages) { stage = 0; phase ^= 1u; }
    };
    int2 s0 = load_pair_rows(ps), t0 = load_pair_rows(pd), s1 = s0, t1 = t0;
    for (int st = 0; alive && st < n_stage; st += 2) {
      if (st + 1 < n_stage) {
        s1 = load_pair_rows(ps + (int64_t)(st + 1) * kWgRows);
        t1 = load_pair_rows(pd + (int64_t)(st + 1) * kWgRows);
      }
      copy(s0, t0);
      if (!alive || st + 1 >= n_stage) break;
      if (st + 2 < n_stage) {
        s0 = load_pair_rows(ps + (int64_t)(st + 2) * kWgRows);
        t0 = load_pair_rows(pd + (int64_t)(st + 2) * kWgRows);
      }
      copy(s1, t1);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    // ---- the partial matrix: lanes are input channels, columns output channels -----------
    __syncwarp();
    if (mbar_wait_warp(false, &bar_done, 0u, abort_flag, a.status)) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int quarter = warp & 3, half = warp >> 2;     // two warps share a lane quarter
      float *out = a.partial + (int64_t)item * a.c_in * a.c_out;
      for (int mt = 0; mt < a.m_tiles; mt++) {
        const int c = c0 + mt * 128 + quarter * 32 + lane;
        for (int col = half * 16; col < a.n_pad; col += 32) {
          uint32_t v[16];
          __syncwarp();
          tmem_ld_32x16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(mt * a.n_pad + col), v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (c < a.c_in && c - c0 < a.a_blocks * 64) {
            float *dst = out + (int64_t)c * a.c_out + col;
#pragma unroll
            for (int i = 0; i < 4; i++)
              if (col + 4 * i < a.c_out)
                *reinterpret_cast<float4 *>(dst + 4 * i) =
                    make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]),
                                __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]));
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
  } else {
    // ------------------------------ MMA issuer --------------------------------
    const uint32_t fmt = a.elem_is_bf16 ? 1u : 0u;
    const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (1u << 15) | (1u << 16) |
                           ((uint32_t)(a.n_pad >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    const uint64_t base = mn_major_desc(smem_u32(stage_base), kWgBlock);
    const uint32_t desc_hi = (uint32_t)(base >> 32), desc_lo = (uint32_t)base;
    const uint32_t stage_step = (uint32_t)a.stage_bytes >> 4;
    const uint32_t b_off = (uint32_t)(a.a_blocks * kWgBlock) >> 4;
    // an accumulator tile with one block of channels reads that block twice; rows 64..127 of
    // its result are not stored
    const uint32_t one_block = (uint32_t)(kWgBlock >> 4) << 16;
    int stage = 0;
    uint32_t phase = 0;
    bool alive = true;
    for (int st = 0; st < n_stage; st++) {
      if (!mbar_wait_warp(false, &bar_full[stage], phase, abort_flag, a.status)) { alive = false; break; }
      fence_generic_to_async();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t lo = desc_lo + (uint32_t)stage * stage_step;
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < kWgRows / 16; k++) {
          const uint64_t db = umma_desc_at(desc_hi, lo + b_off + k * (2048 >> 4));
          for (int mt = 0; mt < a.m_tiles; mt++) {
            const bool single = mt * 2 + 1 >= a.a_blocks;
            const uint32_t alo = lo + (uint32_t)(mt * 2 * kWgBlock >> 4) + k * (2048 >> 4);
            umma_f16(tmem_base + (uint32_t)(mt * a.n_pad), umma_desc_at(desc_hi, single ? alo - one_block : alo),
                     db, idesc, (st | k) != 0 ? 1u : 0u);
          }
        }
        umma_commit(&bar_empty[stage]);
      }
      if (++stage == stages) { stage = 0; phase ^= 1u; }
    }
    if (alive && elect_one()) umma_commit(&bar_done);
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (s_abort) {
    for (int i = 0; i < 2000; i++) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == kWgMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"((uint32_t)a.tmem_cols)
                 : "memory");
  }
}

// ---------------------------------------------------------------------------
// FFMA
// ---------------------------------------------------------------------------
template <typename T> __device__ __forceinline__ float wg_to_f32(T v);
template <> __device__ __forceinline__ float wg_to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float wg_to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float wg_to_f32<__nv_bfloat16>(__nv_bfloat16 v) {
  return __bfloat162float(v);
}
template <typename T> __device__ __forceinline__ T wg_from_f32(float v);
template <> __device__ __forceinline__ float wg_from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __half wg_from_f32<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 wg_from_f32<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}

constexpr int kWsThreads = 128;
constexpr int kWsRows = 32;      // pairs per stage
constexpr int kWsStages = 3;

constexpr int kWsIdxSlots = 8;   // stages whose list entries are kept; the copies of a stage ask for those of kWsIdxAhead later
constexpr int kWsIdxAhead = kWsStages;

// A block owns a BM x BN tile of one item's matrix; a thread 8 x TN of it, 4 rows in each half (and 4
// columns in each half, TN == 8).  The threads form kGroups groups that take every kGroups-th
// pair of a stage and are added up at the end, two by two.  kVec: rows of both arrays can be
// copied 16 bytes at a time (fp32, channels a multiple of 4, aligned).  kLists: pairs are named by the lists, otherwise
// pair i is row i of both arrays (an instance of its own: as a branch it cost the layers with lists 3 to 5 %, 200k rows
// 32 x 32 with 13.5 pairs 180.5 -> 190.4 us).
//
// What bounds it: FFMA issue and the copies' latency.  With 8 x 4 sums a thread, and the list entries read
// from memory before every copy, 586k pairs 64 x 64 took 230 us (products at the FFMA rate: 65 us), now
// 124; 196k pairs 128 x 64 122 -> 96; 52k pairs 256 x 128 141 -> 115 (both with the host's part).  Small tiles
// keep 8 x 4: their copies need the warps that 128 registers a thread would cost.  The ring of a 64 x 64 tile
// (48 KB) lets four blocks share an SM, so its registers are limited for four (for six they spilled).
template <typename T, int BM, int BN, int TN, bool kVec, bool kLists>
__global__ void __launch_bounds__(kWsThreads, TN == 8 || BM + BN == 128 ? 4 : 6)
wgrad_simt_kernel(const __grid_constant__ WgradArgs a, const __grid_constant__ WgradPlan plan, int n_tiles) {
  begin_early();
  constexpr int kHalves = TN / 4, kTileThreads = BM * BN / (8 * TN);
  constexpr int kGroups = kWsThreads / kTileThreads;
  constexpr int kStageFloats = kWsRows * (BM + BN);
  extern __shared__ __align__(16) float s_wg[];      // [kWsStages][kWsRows][BM | BN]
  __shared__ int32_t s_pair[kWsIdxSlots][2][kWsRows];   // source and target rows of a stage's pairs
  const int item = blockIdx.x;
  const int p = row_of_item(plan, item);
  const int64_t first = plan.row_begin[p] + (int64_t)(item - plan.item_prefix[p]) * plan.item_rows;
  const int64_t last = min(plan.row_begin[p + 1], first + plan.item_rows);
  const int n_stage = (int)((last - first) / kWsRows);
  const int m0 = (int)(blockIdx.y / n_tiles) * BM, n0 = (int)(blockIdx.y % n_tiles) * BN;
  const int tid = threadIdx.x;
  const int group = tid / kTileThreads, tt = tid % kTileThreads;
  const int tx = tt % (BN / TN), ty = tt / (BN / TN);
  const T *x = static_cast<const T *>(a.x), *g = static_cast<const T *>(a.g);

  auto load_pairs = [&](int st) {
    if (tid < 2 * kWsRows && st < n_stage) {
      const int side = tid / kWsRows, r = tid % kWsRows;
      if constexpr (!kLists) {
        const int64_t row = first + (int64_t)st * kWsRows + r;
        s_pair[st % kWsIdxSlots][side][r] = row < a.rows ? (int)row : -1;
      } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&s_pair[st % kWsIdxSlots][side][r])),
                     "l"((side ? a.pair_dst : a.pair_src) + first + (int64_t)st * kWsRows + r)
                     : "memory");
      }
    }
  };
  auto load_stage = [&](int st) {
    float *buf = s_wg + (st % kWsStages) * kStageFloats;
    const int32_t *src = s_pair[st % kWsIdxSlots][0], *dst = s_pair[st % kWsIdxSlots][1];
    if constexpr (kVec) {
      constexpr int kCa = BM / 4, kCb = BN / 4;
#pragma unroll
      for (int i = tid; i < kWsRows * kCa; i += kWsThreads) {
        const int r = i / kCa, c = m0 + (i % kCa) * 4;
        const int row = src[r];
        const bool valid = row >= 0 && c < a.c_in;
        wg_copy_16(smem_u32(buf + r * (BM + BN) + (i % kCa) * 4), valid ? x + (int64_t)row * a.c_in + c : x,
                   valid ? 16u : 0u);
      }
#pragma unroll
      for (int i = tid; i < kWsRows * kCb; i += kWsThreads) {
        const int r = i / kCb, c = n0 + (i % kCb) * 4;
        const int row = dst[r];
        const bool valid = row >= 0 && c < a.c_out;
        wg_copy_16(smem_u32(buf + r * (BM + BN) + BM + (i % kCb) * 4),
                   valid ? g + (int64_t)row * a.c_out + c : g, valid ? 16u : 0u);
      }
    } else {
      // element by element: fp32 as copies in flight, 16-bit values through registers, eight at a time
      auto side = [&](const T *in, const int32_t *rows, int channels, int first_c, int width, int at) {
        constexpr int kBatch = 8;
        for (int i0 = tid; i0 < kWsRows * width; i0 += kBatch * kWsThreads) {
          float v[kBatch];
#pragma unroll
          for (int q = 0; q < kBatch; q++) {
            const int i = i0 + q * kWsThreads, r = i / width, c = first_c + i % width;
            v[q] = 0.f;
            if (i >= kWsRows * width) continue;
            const int row = rows[r];
            const bool valid = row >= 0 && c < channels;
            const T *from = valid ? in + (int64_t)row * channels + c : in;
            if constexpr (sizeof(T) == 4) {
              asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                               smem_u32(buf + r * (BM + BN) + at + i % width)), "l"(from), "r"(valid ? 4u : 0u)
                           : "memory");
            } else if (valid) {
              v[q] = wg_to_f32<T>(*from);
            }
          }
          if constexpr (sizeof(T) != 4) {
#pragma unroll
            for (int q = 0; q < kBatch; q++) {
              const int i = i0 + q * kWsThreads;
              if (i < kWsRows * width) buf[i / width * (BM + BN) + at + i % width] = v[q];
            }
          }
        }
      };
      side(x, src, a.c_in, m0, BM, 0);
      side(g, dst, a.c_out, n0, BN, BM);
    }
    load_pairs(st + kWsIdxAhead);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float acc[8][TN];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < TN; j++) acc[i][j] = 0.f;
  for (int st = 0; st < kWsIdxAhead; st++) load_pairs(st);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  for (int st = 0; st < kWsStages - 1; st++) {
    if (st < n_stage) load_stage(st);
    else asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int st = 0; st < n_stage; st++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kWsStages - 2) : "memory");
    __syncthreads();
    // (the list entries of the stage asked for here came with the copies of stage st - 1 at the latest)
    if (st + kWsStages - 1 < n_stage) load_stage(st + kWsStages - 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    const float *buf = s_wg + (st % kWsStages) * kStageFloats;
#pragma unroll 4
    for (int r = group; r < kWsRows; r += kGroups) {
      const float *row = buf + r * (BM + BN);
      float av[8], bv[TN];
      *reinterpret_cast<float4 *>(av) = *reinterpret_cast<const float4 *>(row + ty * 4);
      *reinterpret_cast<float4 *>(av + 4) = *reinterpret_cast<const float4 *>(row + BM / 2 + ty * 4);
#pragma unroll
      for (int h = 0; h < kHalves; h++)
        *reinterpret_cast<float4 *>(bv + 4 * h) = *reinterpret_cast<const float4 *>(row + BM + h * (BN / kHalves) + tx * 4);
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  // the groups add up in the ring, which is free now: the upper half to the lower one, until one is left
  static_assert(kGroups / 2 * BM * BN <= kWsStages * kStageFloats, "the groups' sums must fit the ring");
#pragma unroll
  for (int half = kGroups / 2; half > 0; half /= 2) {
    __syncthreads();
    float *mine = s_wg + (group % half) * (BM * BN) + tt * 4;
    if (group >= half && group < 2 * half) {
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int h = 0; h < kHalves; h++)
          *reinterpret_cast<float4 *>(mine + (i * kHalves + h) * kTileThreads * 4) =
              make_float4(acc[i][4 * h], acc[i][4 * h + 1], acc[i][4 * h + 2], acc[i][4 * h + 3]);
    }
    __syncthreads();
    if (group < half) {
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int h = 0; h < kHalves; h++) {
          const float4 v = *reinterpret_cast<const float4 *>(mine + (i * kHalves + h) * kTileThreads * 4);
          acc[i][4 * h] += v.x; acc[i][4 * h + 1] += v.y; acc[i][4 * h + 2] += v.z; acc[i][4 * h + 3] += v.w;
        }
    }
  }
  if (group == 0) {
    float *out = a.partial + (int64_t)item * a.c_in * a.c_out;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int c = m0 + i / 4 * (BM / 2) + ty * 4 + i % 4;
      if (c >= a.c_in) continue;
#pragma unroll
      for (int h = 0; h < kHalves; h++) {
        const int n = n0 + h * (BN / kHalves) + tx * 4;
        float *dst = out + (int64_t)c * a.c_out + n;
        if (a.c_out % 4 == 0) {
          if (n < a.c_out) *reinterpret_cast<float4 *>(dst) = make_float4(acc[i][4 * h], acc[i][4 * h + 1], acc[i][4 * h + 2], acc[i][4 * h + 3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++)
            if (n + j < a.c_out) dst[j] = acc[i][4 * h + j];
        }
      }
    }
  }
}

// grad_w[order[p]] = sum of the partial matrices of mask row p: kRuns runs of them, each in item order, then
// the sums of the runs.  (One run of up to a hundred items per element is a chain of trips to L2.)
constexpr int kWrThreads = 256;
template <typename T, int kRuns>
__global__ void __launch_bounds__(kWrThreads)
wgrad_reduce_kernel(const float *__restrict__ partial, const __grid_constant__ WgradPlan plan,
                    const int32_t *__restrict__ order, int64_t matrix, T *__restrict__ grad_w) {
  begin_early();
  constexpr int kElems = kWrThreads / kRuns;
  __shared__ float s_sum[kRuns][kElems];
  const int p = blockIdx.y;
  const int k = order != nullptr ? __ldg(order + p) : p;
  const int run = threadIdx.x / kElems, e = threadIdx.x % kElems;
  const int n = plan.item_prefix[p + 1] - plan.item_prefix[p];
  const int begin = plan.item_prefix[p] + (int)((int64_t)n * run / kRuns);
  const int end = plan.item_prefix[p] + (int)((int64_t)n * (run + 1) / kRuns);
  for (int64_t i0 = (int64_t)blockIdx.x * kElems; i0 < matrix; i0 += (int64_t)gridDim.x * kElems) {
    const int64_t i = i0 + e;
    float sum = 0.f;
    if (i < matrix) {
#pragma unroll 8
      for (int it = begin; it < end; it++) sum += __ldg(partial + (int64_t)it * matrix + i);
    }
    if (kRuns > 1) {
      s_sum[run][e] = sum;
      __syncthreads();
      if (run == 0) {
#pragma unroll
        for (int q = 1; q < kRuns; q++) sum += s_sum[q][e];
      }
      __syncthreads();
    }
    if (run == 0 && i < matrix) grad_w[(int64_t)k * matrix + i] = wg_from_f32<T>(sum);
  }
}

bool wgrad_tc_takes(int64_t c_in, int64_t c_out, mn_dtype dtype) {
  return (dtype == MN_F16 || dtype == MN_BF16) && c_in % 8 == 0 && c_out % 8 == 0 && c_out <= 256;
}

int64_t list_rows(const int32_t *sizes, int64_t O) {
  int64_t rows = 0;
  for (int64_t p = 0; p < O; p++) rows += (int64_t)align_up((size_t)sizes[p], kPairRows);
  return rows;
}

struct SimtTile { int bm, bn; };
SimtTile simt_tile(int64_t c_in, int64_t c_out) {
  return SimtTile{c_in > 32 ? 64 : 32, c_out > 32 ? 64 : 32};
}

// Items of every mask row.  One wave of blocks at the kernel's occupancy is aimed at; an item of the tensor-core
// kernel is at least 512 pairs (its partial matrix is written and read once more), one of the FFMA kernel 128: a block
// takes 40 ns a pair.  One offset of 2000 pairs 128 x 64: 25.2 us with 512, 14.2 with 256, 9.2 with 128; 60 000 pairs
// 32 x 20 have 16.1, 14.0, 16.8; all the layers of a UNet's training step (58 800 rows) 2.05, 1.98, 1.98 ms.
WgradPlan make_wgrad_plan(const int32_t *sizes, int64_t O, int64_t c_in, int64_t c_out, mn_dtype dtype) {
  WgradPlan plan{};
  plan.num_rows = (int32_t)O;
  const int64_t total = list_rows(sizes, O);
  int64_t blocks = kNumSMs * 2, least = 512;
  if (wgrad_tc_takes(c_in, c_out, dtype)) {
    blocks /= div_up(c_in, 256);
  } else {
    const SimtTile t = simt_tile(c_in, c_out);
    least = kPairRows;
    blocks = std::max<int64_t>(1, kNumSMs * 4 / (div_up(c_in, t.bm) * div_up(c_out, t.bn)));
  }
  const int64_t want = std::max<int64_t>(least, div_up(total, std::max<int64_t>(1, blocks - O / 2)));
  plan.item_rows = (int32_t)align_up((size_t)want, kPairRows);
  int64_t row = 0;
  int32_t items = 0;
  for (int64_t p = 0; p < MN_MAX_OFFSETS; p++) {
    plan.row_begin[p] = row;
    plan.item_prefix[p] = items;
    if (p < O) {
      const int64_t rows = (int64_t)align_up((size_t)sizes[p], kPairRows);
      row += rows;
      items += (int32_t)div_up(rows, plan.item_rows);
    }
  }
  plan.row_begin[MN_MAX_OFFSETS] = row;
  plan.item_prefix[MN_MAX_OFFSETS] = items;
  return plan;
}

template <typename T, int BM, int BN, int TN, bool kVec>
mn_status launch_wgrad_simt(const WgradArgs &a, const WgradPlan &plan, int items, cudaStream_t st) {
  auto kernel = wgrad_simt_kernel<T, BM, BN, TN, kVec, true>;
  if constexpr (sizeof(T) == 4) {
    if (a.pair_src == nullptr) kernel = wgrad_simt_kernel<T, BM, BN, TN, kVec, false>;
  }
  const int n_tiles = (int)div_up(a.c_out, BN);
  const dim3 grid((unsigned)items, (unsigned)(div_up(a.c_in, BM) * n_tiles));
  const size_t smem = (size_t)kWsStages * kWsRows * (BM + BN) * sizeof(float);
  MN_RETURN_IF(allow_max_shared_memory(reinterpret_cast<const void *>(kernel)));
  MN_LAUNCH("wgrad_simt_kernel", st, launch_early(kernel, grid, kWsThreads, smem, st, a, plan, n_tiles));
  return MN_OK;
}

template <typename T, int BM, int BN>
mn_status run_wgrad_simt(const WgradArgs &a, const WgradPlan &plan, int items, cudaStream_t st) {
  if constexpr (sizeof(T) == 4) {
    if (a.c_in % 4 == 0 && a.c_out % 4 == 0 &&
        ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.g)) & 15) == 0)
      return launch_wgrad_simt<T, BM, BN, (BM + BN > 64 ? 8 : 4), true>(a, plan, items, st);
  }
  return launch_wgrad_simt<T, BM, BN, 4, false>(a, plan, items, st);
}

template <typename T>
mn_status run_wgrad_simt_t(const WgradArgs &a, const WgradPlan &plan, int items, cudaStream_t st) {
  const SimtTile t = simt_tile(a.c_in, a.c_out);
  if (t.bm == 64) return t.bn == 64 ? run_wgrad_simt<T, 64, 64>(a, plan, items, st)
                                    : run_wgrad_simt<T, 64, 32>(a, plan, items, st);
  return t.bn == 64 ? run_wgrad_simt<T, 32, 64>(a, plan, items, st)
                    : run_wgrad_simt<T, 32, 32>(a, plan, items, st);
}

template <typename T>
mn_status run_wgrad_reduce(const float *partial, const WgradPlan &plan, const int32_t *order, int64_t O,
                           int64_t matrix, void *grad_w, cudaStream_t st) {
  // Four runs where one offset has many items: 32 x 32 with 115 of them 7.3 -> 3.8 us, 64 x 64 with 90 18 -> 7;
  // with 31 or fewer the larger number of small blocks costs as much (128 x 128 with 8: 4.8 -> 8.9).
  int32_t most = 0;
  for (int64_t p = 0; p < O; p++) most = std::max(most, plan.item_prefix[p + 1] - plan.item_prefix[p]);
  const bool runs = most >= 40;
  const dim3 grid((unsigned)std::min<int64_t>(div_up(matrix, runs ? kWrThreads / 4 : kWrThreads), 256), (unsigned)O);
  if (runs) {
    MN_LAUNCH("wgrad_reduce_kernel", st, launch_early(wgrad_reduce_kernel<T, 4>, grid, kWrThreads, 0, st, partial, plan,
                                                      order, matrix, static_cast<T *>(grad_w)));
  } else {
    MN_LAUNCH("wgrad_reduce_kernel", st, launch_early(wgrad_reduce_kernel<T, 1>, grid, kWrThreads, 0, st, partial, plan,
                                                      order, matrix, static_cast<T *>(grad_w)));
  }
  return MN_OK;
}

mn_status check_sizes(const int32_t *sizes, int64_t O, int64_t S, int64_t T) {
  MN_CHECK_ARG(O >= 1 && O <= MN_MAX_OFFSETS && S >= 0 && T >= 0 && S < (1ll << 31) && T < (1ll << 31) &&
                   sizes != nullptr, "weight gradient: bad shape");
  for (int64_t p = 0; p < O; p++)
    MN_CHECK_ARG(sizes[p] >= 0 && sizes[p] <= std::min(S, T), "weight gradient: bad size");
  return MN_OK;
}

}  // namespace
}  // namespace mn

using namespace mn;

extern "C" int64_t mn_pair_list_rows(const int32_t *sizes_host, int64_t O) {
  if (sizes_host == nullptr || O < 1 || O > MN_MAX_OFFSETS) return 0;
  return list_rows(sizes_host, O);
}

extern "C" mn_status mn_build_pair_lists(const int32_t *source_masks, const int32_t *target_masks,
                                         const uint32_t *source_bits, const uint32_t *target_bits,
                                         const int32_t *sizes_host, int64_t O, int64_t S, int64_t T,
                                         int32_t *pair_src_out, int32_t *pair_dst_out, void *stream) {
  MN_RETURN_IF(check_sizes(sizes_host, O, S, T));
  const WgradPlan plan = make_wgrad_plan(sizes_host, O, 1, 1, MN_F32);   // row_begin only
  const int64_t rows = plan.row_begin[MN_MAX_OFFSETS];
  if (rows == 0) return MN_OK;
  MN_CHECK_ARG(source_masks != nullptr && target_masks != nullptr && pair_src_out != nullptr &&
                   pair_dst_out != nullptr, "pair lists: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  for (int side = 0; side < 2; side++) {
    int32_t *list = side ? pair_dst_out : pair_src_out;
    const int64_t n = side ? T : S;
    const uint32_t *bits = O <= 32 ? (side ? target_bits : source_bits) : nullptr;
    MN_CHECK_CUDA(cudaMemsetAsync(list, 0xff, sizeof(int32_t) * rows, st));   // padding: no row
    const dim3 grid((unsigned)std::min<int64_t>(kNumSMs * 8, div_up(n, 256)), bits != nullptr ? 1u : (unsigned)O);
    MN_LAUNCH("pair_side_kernel", st,
              launch_early(pair_side_kernel, grid, 256, 0, st, side ? target_masks : source_masks, bits, n, plan, list));
  }
  return MN_OK;
}

extern "C" size_t mn_weight_gradient_workspace_bytes(const int32_t *sizes_host, int64_t O, int64_t c_in,
                                                     int64_t c_out, mn_dtype dtype) {
  if (sizes_host == nullptr || O < 1 || O > MN_MAX_OFFSETS) return 0;
  const WgradPlan plan = make_wgrad_plan(sizes_host, O, c_in, c_out, dtype);
  return (size_t)std::max(plan.item_prefix[MN_MAX_OFFSETS], 1) * c_in * c_out * sizeof(float) + 1024;
}

extern "C" mn_status mn_sparse_convolution_weight_gradient(
    int64_t S, int64_t T, int64_t O, int64_t c_in, int64_t c_out, mn_dtype dtype, const void *sources,
    const void *grad_targets, const int32_t *pair_src, const int32_t *pair_dst, const int32_t *order,
    const int32_t *sizes_host, void *grad_weights_out, int32_t *status_dev, void *ws_ptr,
    size_t ws_bytes, void *stream) {
  MN_RETURN_IF(check_sizes(sizes_host, O, S, T));
  MN_CHECK_ARG(c_in >= 1 && c_out >= 1 && c_in * c_out < (1ll << 31), "weight gradient: bad channels");
  MN_CHECK_ARG(dtype == MN_F32 || dtype == MN_F16 || dtype == MN_BF16, "weight gradient: unknown dtype %d", (int)dtype);
  MN_CHECK_ARG(grad_weights_out != nullptr && status_dev != nullptr, "weight gradient: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const WgradPlan plan = make_wgrad_plan(sizes_host, O, c_in, c_out, dtype);
  const int items = plan.item_prefix[MN_MAX_OFFSETS];
  Workspace ws(ws_ptr, ws_bytes);
  float *partial = ws.take<float>((size_t)std::max(items, 1) * c_in * c_out);
  MN_CHECK_WS(ws);
  if (items > 0) {
    MN_CHECK_ARG(sources != nullptr && grad_targets != nullptr && pair_src != nullptr && pair_dst != nullptr,
                 "weight gradient: null pointer");
    WgradArgs a{};
    a.x = sources; a.g = grad_targets;
    a.pair_src = pair_src; a.pair_dst = pair_dst;
    a.partial = partial; a.status = status_dev;
    a.c_in = (int)c_in; a.c_out = (int)c_out;
    a.n_pad = (int)align_up((size_t)c_out, 16);
    a.elem_is_bf16 = dtype == MN_BF16;
    const bool aligned = ((reinterpret_cast<uintptr_t>(sources) | reinterpret_cast<uintptr_t>(grad_targets)) & 15) == 0 &&
                         ((reinterpret_cast<uintptr_t>(pair_src) | reinterpret_cast<uintptr_t>(pair_dst)) & 7) == 0;
    if (wgrad_tc_takes(c_in, c_out, dtype) && aligned) {
      a.a_blocks = (int)div_up(std::min<int64_t>(c_in, 256), 64);
      a.b_blocks = (int)div_up(c_out, 64);
      a.m_tiles = (int)div_up(a.a_blocks, 2);
      a.stage_bytes = (a.a_blocks + a.b_blocks) * kWgBlock;
      const TcSizing z = size_tc_kernel(a.stage_bytes, a.m_tiles * a.n_pad, kWgMaxStages, 2, 0, kWgMaxStages);
      a.stages = z.stages;
      a.tmem_cols = z.tmem_cols;
      MN_RETURN_IF(allow_max_shared_memory(reinterpret_cast<const void *>(wgrad_tc_kernel)));
      const dim3 grid((unsigned)items, (unsigned)div_up(c_in, 256));
      MN_LAUNCH("wgrad_tc_kernel", st, launch_early(wgrad_tc_kernel, grid, kWgThreads, z.smem_bytes, st, a, plan));
    } else if (dtype == MN_F32) {
      MN_RETURN_IF(run_wgrad_simt_t<float>(a, plan, items, st));
    } else if (dtype == MN_F16) {
      MN_RETURN_IF(run_wgrad_simt_t<__half>(a, plan, items, st));
    } else {
      MN_RETURN_IF(run_wgrad_simt_t<__nv_bfloat16>(a, plan, items, st));
    }
  }
  const int64_t matrix = c_in * c_out;
  switch (dtype) {
    case MN_F32: return run_wgrad_reduce<float>(partial, plan, order, O, matrix, grad_weights_out, st);
    case MN_F16: return run_wgrad_reduce<__half>(partial, plan, order, O, matrix, grad_weights_out, st);
    default: return run_wgrad_reduce<__nv_bfloat16>(partial, plan, order, O, matrix, grad_weights_out, st);
  }
}

// ---------------------------------------------------------------------------
// x^T g: the weight gradient of a 1x1x1 convolution, fp32
// ---------------------------------------------------------------------------
// One offset whose pair i is row i of both arrays, so no lists.  A library GEMM sees a small matrix and a long
// contraction and gives it few blocks (58 800 rows x 96 x 20: 26); here the rows are cut into items for a wave of
// them.  60 000 rows 32 x 20: 148 us -> 17, 96 x 20 157 -> 24, 192 x 128 151 -> 81, and a smaller error against
// fp64 (96 x 20: 2.1e-8 -> 7e-9 of the terms' sum).  What bounds it: the chain of an item and of the sums over
// the items up to some 20 000 rows, FFMA issue beyond.
extern "C" size_t mn_dense_weight_gradient_workspace_bytes(int64_t rows, int64_t c_in, int64_t c_out) {
  if (rows < 0 || rows > INT32_MAX - kPairRows) return 0;
  const int32_t size = (int32_t)rows;
  return mn_weight_gradient_workspace_bytes(&size, 1, c_in, c_out, MN_F32);
}

extern "C" mn_status mn_dense_weight_gradient(int64_t rows, int64_t c_in, int64_t c_out, const float *x, const float *g,
                                              float *grad_weight_out, void *ws_ptr, size_t ws_bytes, void *stream) {
  MN_CHECK_ARG(rows >= 0 && rows <= INT32_MAX - kPairRows, "dense weight gradient: bad number of rows");
  MN_CHECK_ARG(c_in >= 1 && c_out >= 1 && c_in < (1 << 20) && c_out < (1 << 20) && c_in * c_out < (1ll << 31),
               "dense weight gradient: bad channels");
  MN_CHECK_ARG(grad_weight_out != nullptr && (rows == 0 || (x != nullptr && g != nullptr)),
               "dense weight gradient: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int32_t size = (int32_t)rows;
  const WgradPlan plan = make_wgrad_plan(&size, 1, c_in, c_out, MN_F32);
  const int items = plan.item_prefix[MN_MAX_OFFSETS];
  Workspace ws(ws_ptr, ws_bytes);
  float *partial = ws.take<float>((size_t)std::max(items, 1) * c_in * c_out);
  MN_CHECK_WS(ws);
  if (items > 0) {
    WgradArgs a{};
    a.x = x; a.g = g; a.partial = partial; a.rows = rows;
    a.c_in = (int)c_in; a.c_out = (int)c_out;
    MN_RETURN_IF(run_wgrad_simt_t<float>(a, plan, items, st));
  }
  return run_wgrad_reduce<float>(partial, plan, nullptr, 1, c_in * c_out, grad_weight_out, st);
}
