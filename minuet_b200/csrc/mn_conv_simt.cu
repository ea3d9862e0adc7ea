// Fused (implicit-GEMM) forward pass of a sparse convolution in fp32.
//
// fp32 features must not go through the tensor cores (TF32 keeps 10 mantissa bits), so this
// is the output-stationary kernel of mn_conv_implicit.cu on FFMA units: a block owns BM
// consecutive rows of the neighbour table (targets sorted by hit word) and 32 output
// channels, keeps their sums in shared memory and walks the offsets that its rows have; source
// rows are fetched through the table straight into shared memory.
//
// Order of the sums: every offset's product is a chain of its own over the input channels,
// and the products are added in mask-row order (the centre, the largest, last).  That is the
// order of the reference's GEMM and scatter and of the explicit path, bit for bit; a network
// with ReLUs turns a last-bit difference in its forward pass into visible differences of its
// gradients.
//
// The unit of work is a warp's: the product of one offset's weights with up to 32 of the block's rows
// that have the offset, picked from anywhere in the block, so that next to no zeros are multiplied.  A
// block lists these items offset by offset and deals them out to its warps in turn; each warp
// runs its own ring of copies and waits for no other, except that products enter the sums in the
// order of the list, handed from warp to warp.  So the offsets of a tile are worked on side by side, and a
// tile with 27 of them is no chain of 27 steps that the whole chip waits for.
//
// Few rows (the coarse levels of a network) leave SMs without a block, and a block of eight warps with 27
// items runs four products one after the other: there a cluster of eight blocks shares a tile's
// list.  Every product stays in the shared memory of the block that made it, and after a barrier of the
// cluster each block adds the products of some of the rows, in the same order.
#include "mn_common.cuh"

#include <algorithm>

namespace mn {

namespace {

constexpr int kCsK = 16;          // input channels per step
constexpr int kCsRows = 32;       // rows and columns of a warp's product
constexpr int kCsStageFloats = 2 * kCsK * kCsRows;   // rows [32][16] (pieces swizzled), weights [16][32]
constexpr int kCsMaxOffsets = 32;

struct CsArgs {
  const float *in;            // [S, K]
  const float *weights;       // [O, K, N]
  const int32_t *nbr;         // [O, pitch]
  const uint32_t *tile_bits;  // [ceil(T / 128)]
  const int32_t *order;       // [O] or NULL
  const int32_t *perm;        // [T] or NULL
  const float *scale, *shift, *residual;
  float *out;                 // [T, N]
  int64_t T, pitch;
  int32_t K, N, k_steps, relu;
};

__device__ __forceinline__ void cs_copy_16(void *dst, const void *src, uint32_t src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cs_copy_4(void *dst, const void *src, uint32_t src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(src_bytes)
               : "memory");
}

__device__ __forceinline__ float cs_epilogue(float f, const CsArgs &a, int64_t row, int c) {
  if (a.scale != nullptr) f *= __ldg(a.scale + c);
  if (a.shift != nullptr) f += __ldg(a.shift + c);
  if (a.residual != nullptr) f += __ldg(a.residual + row * a.N + c);
  return a.relu ? fmaxf(f, 0.f) : f;
}
__device__ __forceinline__ float4 cs_epilogue(float4 v, const CsArgs &a, int64_t row, int c) {
  float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; j++)
    if (c + j < a.N) f[j] = cs_epilogue(f[j], a, row, c + j);
  return make_float4(f[0], f[1], f[2], f[3]);
}

// Barrier between a warp and the one that its neighbour's products follow (64 threads).
__device__ __forceinline__ void cs_turn_wait(int id) {
  __syncwarp();
  asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
}
__device__ __forceinline__ void cs_turn_pass(int id) {
  __threadfence_block();
  __syncwarp();
  asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory");
}

// Blocks of a cluster: what every block wrote before its arrival can be read by the others after their wait.
__device__ __forceinline__ void cs_cluster_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cs_cluster_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the value at `at` in the shared memory of another block of the cluster
__device__ __forceinline__ float cs_load_from(const float *at, int block) {
  uint32_t addr;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(addr) : "r"((uint32_t)__cvta_generic_to_shared(at)), "r"(block));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

// BM x (32 kCols) sums per block of W warps or per cluster of kCluster of them, a product of 32 x 32 per warp,
// 8 x 4 of it per thread.  Blocks take the tiles from the last to the first: the rows with rare
// offsets sort to the end, and their tiles take longest.  At most cs_cap offsets are looked at at a
// time (index blocks in shared memory).  kVec: rows of the features and of the weights can be copied 16
// bytes at a time.  kFew: an item of up to 16 rows costs half as much (maps of 3.5 pairs a row: 32-row tiles
// take 15 % less time, at 20 pairs 3 % more); not for the tall blocks of large maps, whose items are full.
//
// What bounds it: issue and latency at 12 to 16 warps per SM (registers and shared memory allow no more).
// With one product per instruction, of 56 M warp instructions of a layer of 3.6k rows 128->128 with 14.5
// pairs 38 M ran on the FMA pipe, and a scheduler issued in 61 % of the cycles; with two (the same rate of
// products, half the issue slots) layers of 15k rows 64->64 with 12.3 pairs take 75 instead of 85 us, 41k 32->32
// with 7.7 45 instead of 48.5, 3.4k 128->128 79 instead of 89, 700 rows 256->256 103 instead of 113.  The weight
// gradients, whose tiles are 8 x 8, gain nothing by it.  Sparse maps: the
// chain tile bits -> index blocks -> rows before a block's first product.
//
// Against a block of 64 x 64 (or 32 x 32) sums in registers that walked its tile's offsets one after
// the other, and a second launch for maps of few rows (us): 59k rows 32->32, 3 pairs 67 -> 34; 42k
// 64->32, 7.5 pairs 146 -> 78; 16k 64->64, 12.5 pairs 137 -> 85; 16k 128->64 262 -> 150; 3.6k 128->128,
// 14.5 pairs 108 -> 95; 196k 64->64, 3 pairs 228 -> 213; 50k 32->32, 1.1 pairs 29 -> 15; 59k 3->32 98 -> 21.
// Where every row of a 64 x 64 or 128 x 32 block has every offset, a warp's items are all those of its own rows and
// columns and nothing is handed over.  Maps of 20 and more pairs a row in blocks like that are what the block with
// sums in registers was better at, whose warps shared the copies of the weights: 250k rows 64->64, 23.9 pairs 1370
// -> 1579 us, 16->16 308 -> 329, 60k 256->256 5030 -> 5300; with 11 pairs 0.53 to 0.8 of its time.
// Clusters against that second launch, 8 to 21 pairs: 13 rows 256->256 25 -> 15, 64->64 16 -> 8; 130 rows 128->128 23
// -> 15; 325 rows 256->64 37 -> 26; 700 rows 256->256 137 -> 120 (3.5 pairs 79 -> 60).
constexpr int cs_cap(int bm, int cluster) { return bm == 32 || cluster > 1 ? kCsMaxOffsets : 16; }
// items of one block of a cluster at most
constexpr int cs_share(int bm, int cluster) { return kCsMaxOffsets * (bm / kCsRows) / cluster; }
constexpr size_t cs_smem(int bm, int cols, int warps, int stages, int cluster) {
  return (size_t)warps * stages * kCsStageFloats * 4 + (size_t)cs_cap(bm, cluster) * bm * 5 +
         (size_t)(cluster > 1 ? cs_share(bm, cluster) * kCsRows : bm * cols) * kCsRows * 4;
}

template <int BM, int kCols, int W, int kStages, int kCluster, bool kVec>
__global__ void __launch_bounds__(W * 32, W == 4 ? (cs_smem(BM, kCols, W, kStages, kCluster) <= 55 * 1024 ? 4 : 3) : 2)
conv_simt_kernel(const __grid_constant__ CsArgs a) {
  begin_early();
  constexpr int kThreads = W * 32, kSubs = BM / 32, kCap = cs_cap(BM, kCluster), kSumCols = kCols * kCsRows;
  constexpr int kTeam = W * kCluster;                // warps of a tile
  constexpr bool kDirect = BM > 32 && kCluster == 1;
  constexpr bool kOwn = kDirect && kSubs * kCols == W;
  constexpr bool kFew = BM == 32 || kCluster > 1;
  static_assert(kCluster == 1 || (kCols == 1 && kCap == kCsMaxOffsets), "clusters: one list of items per tile");
  extern __shared__ __align__(16) float s_mem[];
  __shared__ int32_t s_active[kCsMaxOffsets], s_weight[kCsMaxOffsets];
  __shared__ uint8_t s_have[kCap];                // rows that have the offset
  __shared__ uint16_t s_items[kCap * kSubs * kCols];   // offset of the chunk | 32 of its rows << 5 | 32 columns << 8
  __shared__ uint8_t s_first[kCap];               // an offset's first item
  __shared__ uint32_t s_present;                  // offsets that have items
  __shared__ bool s_own;
  __shared__ int32_t s_count, s_perm[BM];
  // the sums [BM][kSumCols]; in a cluster the products of this block's items [item][32][32]
  float *s_sum = s_mem + W * kStages * kCsStageFloats;
  constexpr int kSums = kCluster > 1 ? cs_share(BM, kCluster) * kCsRows * kCsRows : BM * kSumCols;
  int32_t *s_idx = reinterpret_cast<int32_t *>(s_sum + kSums);          // [kCap][BM]: source rows, then those that exist
  // [kCap][BM]: the block's rows they feed; in a cluster the other way round, a row's place among them (none: 0xff)
  uint8_t *s_row = reinterpret_cast<uint8_t *>(s_idx + kCap * BM);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = lane % 8, ty = lane / 8;
  const int rank = (int)(blockIdx.x % kCluster);                         // of this block in its cluster
  const int64_t r0 = (int64_t)((gridDim.x - 1 - blockIdx.x) / kCluster) * BM;
  const int n0 = blockIdx.y * kSumCols;
  float *ring = s_mem + warp * kStages * kCsStageFloats;

  const uint32_t bits = __ldg(a.tile_bits + r0 / 128);
  const int n_bits = __popc(bits);
  if (warp == 0 && ((bits >> lane) & 1u)) {
    const int j = __popc(bits & ((1u << lane) - 1u));
    s_active[j] = lane;
    s_weight[j] = a.order != nullptr ? __ldg(a.order + lane) : lane;
  }
  // where the rows go: needed last, asked for first
  for (int e = tid; e < BM; e += kThreads)
    if (a.perm != nullptr && r0 + e < a.T) cs_copy_4(s_perm + e, a.perm + r0 + e, 4u);
  const int tiles = kCols == 1 || n0 + kCsRows >= a.N ? 1 : kCols;      // of 32 columns
  auto clear_sums = [&]() {
    for (int e = tid; e < BM * kSumCols / 4; e += kThreads)
      reinterpret_cast<float4 *>(s_sum)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  };
  const bool vec_out = a.N % 4 == 0;
  auto store_row = [&](float4 v, int64_t r, int c) {
    const int64_t t = a.perm != nullptr ? (int64_t)s_perm[r - r0] : r;
    v = cs_epilogue(v, a, t, c);
    float *dst = a.out + t * a.N + c;
    if (vec_out) {
      *reinterpret_cast<float4 *>(dst) = v;
    } else {
      const float f[4] = {v.x, v.y, v.z, v.w};
      for (int j = 0; j < 4 && c + j < a.N; j++) dst[j] = f[j];
    }
  };
  // One offset, and every row has it (most blocks of a sparse map): the products are the sums.
  bool direct = false;
  int n_items = 0;
  if (kCluster == 1 && n_bits == 0) clear_sums();

  for (int chunk = 0; chunk < n_bits; chunk += kCap) {
    __syncthreads();
    // index blocks of these offsets (their loads are in flight together), the rows that have them
    const int n_chunk = min(kCap, n_bits - chunk);
    for (int e = tid; e < n_chunk * (BM / 4); e += kThreads) {
      const int j = e / (BM / 4), i = (e % (BM / 4)) * 4;
      cs_copy_16(s_idx + j * BM + i, a.nbr + (int64_t)s_active[chunk + j] * a.pitch + r0 + i, 16u);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    for (int j = warp; j < n_chunk; j += W) {
      int32_t source[kSubs];
#pragma unroll
      for (int sub = 0; sub < kSubs; sub++) source[sub] = s_idx[j * BM + sub * 32 + lane];
      __syncwarp();
      int n = 0;
#pragma unroll
      for (int sub = 0; sub < kSubs; sub++) {
        const uint32_t hit = __ballot_sync(0xffffffffu, source[sub] >= 0);
        if (source[sub] >= 0) {
          const int at = n + __popc(hit & ((1u << lane) - 1u));
          s_idx[j * BM + at] = source[sub];
          if (kCluster == 1) s_row[j * BM + at] = (uint8_t)(sub * 32 + lane);
          else s_row[j * BM + sub * 32 + lane] = (uint8_t)at;
        } else if (kCluster > 1) {
          s_row[j * BM + sub * 32 + lane] = (uint8_t)0xff;
        }
        n += __popc(hit);
      }
      if (n + lane < BM) s_idx[j * BM + n + lane] = -1;       // up to a whole item
      if (lane == 0) s_have[j] = (uint8_t)n;
    }
    __syncthreads();
    const int n_rows = (int)min((int64_t)BM, a.T - r0);
    direct = kDirect && n_bits == 1 && s_have[0] == n_rows;
    if (kCluster == 1 && chunk == 0 && !direct) clear_sums();
    if (warp == 0) {
      const int mine = lane < n_chunk ? (s_have[lane % kCap] + 31) / 32 * tiles : 0;
      int end = mine;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, end, d);
        if (lane >= d) end += t;
      }
      if (kCluster > 1 && lane < n_chunk) s_first[lane % kCap] = (uint8_t)(end - mine);
      for (int g = 0; g < mine; g++) s_items[end - mine + g] = (uint16_t)(lane | ((g / tiles) << 5) | ((g % tiles) << 8));
      if (lane == 31) s_count = end;
      if constexpr (kCluster > 1) {
        const uint32_t present = __ballot_sync(0xffffffffu, mine > 0);
        if (lane == 0) s_present = present;
      }
      // every row has every offset: item i is that of the 32 rows and columns of warp i % W, and of no other
      if constexpr (kOwn) {
        const bool whole = __all_sync(0xffffffffu, lane >= n_chunk || s_have[lane % kCap] == n_rows);
        if (lane == 0) s_own = whole && tiles == kCols && n_rows > BM - 32;
      }
    }
    __syncthreads();
    n_items = s_count;
    const bool own = kOwn && s_own;
    // item i is worked on by block i % kCluster, so that a tile with few items has them on as many SMs
    const int first_item = warp * kCluster + rank;
    const int n_step = (n_items > first_item ? (n_items - first_item + kTeam - 1) / kTeam : 0) * a.k_steps;

    // kFew: rows 16 to 31 of an item of up to 16 are neither copied nor multiplied (rare offsets: a few rows each)
    auto few_rows = [&](int entry) { return kFew && (int)s_have[entry & 31] - ((entry >> 5) & 7) * kCsRows <= kCsRows / 2; };
    // the cursor of the copies: item, first channel, ring stage; the item's rows and weights
    int l_item = first_item, l_k = 0, l_stage = 0;
    const float *l_src[kCsRows / 8], *l_w = nullptr;
    uint32_t l_valid = 0u;
    bool l_few = false;
    auto load_step = [&]() {
      float *sa = ring + l_stage * kCsStageFloats, *sb = sa + kCsK * kCsRows;
      const int item = s_items[l_item], j = item & 31;
      const int32_t *idx = s_idx + j * BM + ((item >> 5) & 7) * 32;
      const int c0 = n0 + (item >> 8) * kCsRows;
      if constexpr (kVec) {
        const int c = (lane & 3) * 4;
        if (l_k == 0) {
          if (kFew) l_few = few_rows(item);
          l_w = a.weights + ((int64_t)s_weight[chunk + j] * a.K + ty) * a.N + c0 + tx * 4;
          l_valid = 0u;
#pragma unroll
          for (int i = 0; i < kCsRows / 8; i++) {
            const int row = idx[i * 8 + (lane >> 2)];
            l_src[i] = a.in + (int64_t)max(row, 0) * a.K + c;
            l_valid |= (row >= 0 ? 1u : 0u) << i;
          }
        }
        const uint32_t valid = l_k + c < a.K ? l_valid : 0u;
        const int place = (((lane & 3) ^ ((lane >> 3) & 3)) << 2);   // pieces of row r: position ^ (r >> 1) & 3
#pragma unroll
        for (int i = 0; i < kCsRows / 8; i++)
          if (i < kCsRows / 16 || !kFew || !l_few) cs_copy_16(sa + (i * 8 + (lane >> 2)) * kCsK + place, (valid >> i) & 1u ? l_src[i] + l_k : a.in,
                     (valid >> i) & 1u ? 16u : 0u);
        const bool col = c0 + tx * 4 < a.N;
#pragma unroll
        for (int i = 0; i < kCsK / 4; i++) {
          const bool in = col && l_k + i * 4 + ty < a.K;
          cs_copy_16(sb + (i * 4 + ty) * kCsRows + tx * 4, in ? l_w + i * 4 * (int64_t)a.N : a.weights, in ? 16u : 0u);
        }
        l_w += kCsK * (int64_t)a.N;
      } else {
        const float *w = a.weights + ((int64_t)s_weight[chunk + j] * a.K + l_k) * a.N + c0 + lane;
        const bool col = c0 + lane < a.N, item_few = few_rows(item);
        for (int k = 0; k < kCsK && l_k + k < a.K; k += 4) {      // the channels that are multiplied
          const int c = k + (lane & 3);
          const int place = (((k >> 2) ^ ((lane >> 3) & 3)) << 2) | (lane & 3);
#pragma unroll
          for (int i = 0; i < kCsRows / 8; i++) {
            if (kFew && i >= kCsRows / 16 && item_few) break;
            const int r = i * 8 + (lane >> 2), row = idx[r];
            const bool valid = row >= 0 && l_k + c < a.K;
            cs_copy_4(sa + r * kCsK + place, valid ? a.in + (int64_t)row * a.K + l_k + c : a.in, valid ? 4u : 0u);
          }
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const bool valid = col && l_k + k + i < a.K;
            cs_copy_4(sb + (k + i) * kCsRows + lane, valid ? w + (int64_t)(k + i) * a.N : a.weights, valid ? 4u : 0u);
          }
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      l_k += kCsK;
      if (l_k >= a.K) { l_k = 0; l_item += kTeam; }
      if (++l_stage == kStages) l_stage = 0;
    };
    for (int s = 0; s < kStages - 1; s++) {
      if (s < n_step) load_step();
      else asm volatile("cp.async.commit_group;" ::: "memory");
    }

    f32_pair acc[8][2];                            // 8 rows x 4 columns
#pragma unroll
    for (int i = 0; i < 8; i++) acc[i][0] = acc[i][1] = 0u;
    int place[4];                                  // of the four-channel pieces of this lane's rows
#pragma unroll
    for (int k = 0; k < 4; k++) place[k] = ty * kCsK + ((k ^ (ty >> 1)) << 2);
    int item = first_item, k0 = 0, stage = 0;
    bool few = n_step > 0 && few_rows(s_items[item]);
    auto next_item = [&]() {
      item += kTeam;
      k0 = 0;
      if (kFew && item < n_items) few = few_rows(s_items[item]);
    };
    for (int step = 0; step < n_step; step++) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
      __syncwarp();
      if (step + kStages - 1 < n_step) load_step();
      else asm volatile("cp.async.commit_group;" ::: "memory");
      const float *sa = ring + stage * kCsStageFloats, *sb = sa + kCsK * kCsRows + tx * 4;
      const int kmax = min(kCsK, a.K - k0);        // zeros up to a multiple of 4
      if (++stage == kStages) stage = 0;
      k0 += kCsK;
#pragma unroll
      for (int k = 0; k < kCsK; k += 4) {
        if (k < kmax) {
          float4 av[8], bv[4];
#pragma unroll
          for (int i = 0; i < 8; i++)
            if (i < 4 || !kFew || !few)
              av[i] = *reinterpret_cast<const float4 *>(sa + i * 4 * kCsK + place[(k / 4) ^ (2 * (i & 1))]);
#pragma unroll
          for (int j = 0; j < 4; j++) bv[j] = *reinterpret_cast<const float4 *>(sb + (k + j) * kCsRows);
#pragma unroll
          for (int i = 0; i < 8; i++) {
            if (kFew && i >= 4 && few) continue;
            const float ak[4] = {av[i].x, av[i].y, av[i].z, av[i].w};
#pragma unroll
            for (int j = 0; j < 4; j++) {
              const f32_pair a2 = make_pair_f32(ak[j], ak[j]);
              fma_pair_f32(a2, make_pair_f32(bv[j].x, bv[j].y), acc[i][0]);
              fma_pair_f32(a2, make_pair_f32(bv[j].z, bv[j].w), acc[i][1]);
            }
          }
        }
      }
      if (k0 < a.K) continue;
      // the product is complete: it is added when the items before it have been
      const int entry = s_items[item], j0 = entry & 31, first = ((entry >> 5) & 7) * 32 + ty;
      const int left = s_have[j0] - first;
      const uint8_t *rows = s_row + j0 * BM + first;
      if constexpr (kCluster > 1) {
        float4 *product = reinterpret_cast<float4 *>(s_sum + (item / kCluster * kCsRows + ty) * kCsRows) + tx;
#pragma unroll
        for (int i = 0; i < 8; i++) {
          if (4 * i < left) product[i * 4 * (kCsRows / 4)] = split_pairs_f32(acc[i][0], acc[i][1]);
          acc[i][0] = acc[i][1] = 0u;
        }
        next_item();
        continue;
      }
      if (kDirect && direct) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const int c = n0 + (entry >> 8) * kCsRows + tx * 4;
          if (4 * i < left && c < a.N)
            store_row(split_pairs_f32(acc[i][0], acc[i][1]), r0 + first + 4 * i, c);
          acc[i][0] = acc[i][1] = 0u;
        }
        next_item();
        continue;
      }
      if (W > 1 && !own && item > 0) cs_turn_wait(1 + warp);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        if (4 * i < left) {
          float4 *sum = reinterpret_cast<float4 *>(s_sum + rows[4 * i] * kSumCols + (entry >> 8) * kCsRows) + tx;
          const float4 mine = split_pairs_f32(acc[i][0], acc[i][1]);
          float4 v = *sum;
          v.x += mine.x; v.y += mine.y; v.z += mine.z; v.w += mine.w;
          *sum = v;
        }
        acc[i][0] = acc[i][1] = 0u;
      }
      if (W > 1 && !own && item + 1 < n_items) {
        cs_turn_pass(1 + (warp + 1) % W);
      }
      next_item();
    }
  }
  if constexpr (kCluster > 1) {
    // every block adds the products of some rows, read from where they are, in the order of the list
    constexpr int kRows = BM / kCluster, kBatch = 8;
    asm volatile("cp.async.wait_all;" ::: "memory");      // (s_perm of a tile without offsets)
    cs_cluster_arrive();
    cs_cluster_wait();
    const uint32_t present = n_bits > 0 ? s_present : 0u;
    const int c = n0 + lane;
    for (int r = rank * kRows + warp; r < (rank + 1) * kRows; r += W) {
      float sum = 0.f;
      for (uint32_t left = present; left != 0u;) {
        float v[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; q++) {
          const int j = left != 0u ? __ffs(left) - 1 : 0;
          const int at = left != 0u ? s_row[j * BM + r] : 0xff;
          left &= left - 1u;
          v[q] = 0.f;
          if (at == 0xff) continue;
          const int item = s_first[j] + at / kCsRows;
          v[q] = cs_load_from(s_sum + (item / kCluster * kCsRows + at % kCsRows) * kCsRows + lane, item % kCluster);
        }
#pragma unroll
        for (int q = 0; q < kBatch; q++) sum += v[q];     // (a zero for a row without the offset changes no bit)
      }
      if (r0 + r < a.T && c < a.N) {
        const int64_t t = a.perm != nullptr ? (int64_t)s_perm[r] : r0 + r;
        a.out[t * a.N + c] = cs_epilogue(sum, a, t, c);
      }
    }
    cs_cluster_arrive();
    cs_cluster_wait();                                    // the others have read this block's products
    return;
  }
  if (kDirect && direct) return;
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  for (int e = tid; e < BM * kSumCols / 4; e += kThreads) {
    const int64_t r = r0 + e / (kSumCols / 4);
    const int c = n0 + (e % (kSumCols / 4)) * 4;
    if (r < a.T && c < a.N) store_row(reinterpret_cast<const float4 *>(s_sum)[e], r, c);
  }
}

template <int BM, int kCols, int W, int kStages, int kCluster = 1>
mn_status launch_cs(const CsArgs &a, cudaStream_t st) {
  const bool vec = a.K % 4 == 0 && a.N % 4 == 0 &&
                   ((reinterpret_cast<uintptr_t>(a.in) | reinterpret_cast<uintptr_t>(a.weights)) & 15) == 0;
  constexpr size_t smem = cs_smem(BM, kCols, W, kStages, kCluster);
  const dim3 grid((unsigned)(div_up(a.T, BM) * kCluster), (unsigned)div_up(a.N, kCols * kCsRows));
  static thread_local bool sized[kMaxDevices] = {false};
  int device = 0;
  MN_CHECK_CUDA(cudaGetDevice(&device));
  MN_CHECK_ARG(device >= 0 && device < kMaxDevices, "fp32 forward: device index %d out of range", device);
  const auto with_vec = conv_simt_kernel<BM, kCols, W, kStages, kCluster, true>;
  const auto by_element = conv_simt_kernel<BM, kCols, W, kStages, kCluster, false>;
  if (!sized[device]) {
    MN_CHECK_CUDA(cudaFuncSetAttribute(with_vec, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    MN_CHECK_CUDA(cudaFuncSetAttribute(by_element, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    sized[device] = true;
  }
  MN_LAUNCH("conv_simt_kernel", st, launch_early_clusters(vec ? with_vec : by_element, kCluster, grid, W * 32, smem, st, a));
  return MN_OK;
}

}  // namespace
}  // namespace mn

using namespace mn;

extern "C" size_t mn_implicit_fp32_workspace_bytes(int64_t, int64_t, int64_t) { return 0; }

extern "C" mn_status mn_sparse_convolution_forward_implicit_fp32(
    int64_t S, int64_t T, int64_t O, int64_t c_in, int64_t c_out, const float *sources,
    const float *weights, const int32_t *nbr, const uint32_t *tile_bits, const int32_t *perm,
    const int32_t *order, const float *scale, const float *shift, const float *residual, int relu,
    float *targets_out, void *ws_ptr, size_t ws_bytes, void *stream) {
  MN_CHECK_ARG(O >= 1 && O <= kCsMaxOffsets, "fp32 forward: %lld offsets (supported: 1..%d)", (long long)O,
               kCsMaxOffsets);
  MN_CHECK_ARG(S >= 0 && T >= 0 && T < (1ll << 31) && S < (1ll << 31) && c_in >= 1 && c_out >= 1 &&
                   c_out <= 65535 * 32ll, "fp32 forward: bad sizes");
  if (T == 0) return MN_OK;
  MN_CHECK_ARG(weights != nullptr && nbr != nullptr && tile_bits != nullptr && targets_out != nullptr &&
                   (S == 0 || sources != nullptr), "fp32 forward: null pointer");
  CsArgs a{};
  a.in = sources; a.weights = weights; a.nbr = nbr; a.tile_bits = tile_bits;
  a.order = order; a.perm = perm;
  a.scale = scale; a.shift = shift; a.residual = residual; a.relu = relu ? 1 : 0;
  a.out = targets_out;
  a.T = T; a.pitch = (int64_t)align_up((size_t)T, 128);
  a.K = (int)c_in; a.N = (int)c_out;
  a.k_steps = (int)div_up(c_in, kCsK);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  (void)ws_ptr;             // products and sums stay on the chip
  (void)ws_bytes;
  MN_CHECK_ARG((reinterpret_cast<uintptr_t>(nbr) & 15) == 0 &&
                   (c_out % 4 != 0 || (reinterpret_cast<uintptr_t>(targets_out) & 15) == 0),
               "fp32 forward: the output and the neighbour table must be 16-byte aligned");
  // Tall blocks waste fewest products (an item holds up to 32 rows with the offset) and pay the lookup of
  // their index blocks over more rows, short ones fill the chip.  Measured, us for blocks of 128 x 32 /
  // 64 x 64 / 64 x 32 / 32 x 32 sums: 232k rows 16->16 31 / 41 / 40 / 80; 200k 48->48 77 / 69 / 95 / 181;
  // 59k 32->32 42 / 40 / 34 / 43; 16k 64->64 156 / 130 / 95 / 84; 3.6k 128->128 185 / 190 / 140 / 95.  Eight
  // warps instead of four where blocks of 32 rows leave half the chip idle: 700 rows 256->256 136 -> 121,
  // 5k rows 256->64 60 -> 50.
  // Clusters as long as their blocks run in one wave (three per SM): of 32 rows up to 48 tiles, of 64 rows (half
  // the items where offsets are rare) up to 55.  us for clusters of 32 rows / of 64 rows / eight warps (with a
  // loop body of its own for items of up to 16 rows, some 5 % slower in the clusters than now): 325
  // rows 256->64, 19 pairs, 22 tiles 28 / 36 / 79; 325 rows 256->256, 88 tiles 69 / 67 / 80, with 3.2 pairs 49 / 34
  // / 56; 1.5k 128->128, 188 tiles 83 / 78 / 65.  A second wave of them pays for deep products where the
  // blocks of eight warps are a few more than the SMs: 700 rows 256->256, 88 tiles of 64 rows, 21 pairs 133 /
  // 128 / 122, 3.5 pairs 93 / 63 / 85.
  const int64_t columns = div_up(c_out, kCsRows);
  const int64_t tall = div_up(T, 128) * columns, mid = div_up(T, 64) * columns, low = div_up(T, 32) * columns;
  if (low <= 48) return launch_cs<32, 1, 4, 3, 8>(a, st);
  if (mid <= 55 || (c_in >= 256 && 2 * mid >= kNumSMs && 3 * mid <= 2 * kNumSMs)) return launch_cs<64, 1, 4, 2, 8>(a, st);
  if (tall >= 8 * kNumSMs) return columns > 1 ? launch_cs<64, 2, 4, 2>(a, st) : launch_cs<128, 1, 4, 2>(a, st);
  if (mid >= 4 * kNumSMs) return launch_cs<64, 1, 4, 3>(a, st);
  if (2 * low >= 5 * kNumSMs) return launch_cs<32, 1, 4, 3>(a, st);
  return launch_cs<32, 1, 8, 2>(a, st);
}
