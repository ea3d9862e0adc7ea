// Stable radix sort of 64-bit keys, shared by the map step, voxelisation and the neighbour
// tables: one launch that makes the keys and counts their digits, then one launch per 9-bit
// digit.  The scheme is published: one sweep per digit (Adinets and Merrill, "Onesweep", 2022) with
// decoupled look-back (Merrill and Garland, 2016).
//
// A digit pass moves every key once: a block takes the next tile of keys, ranks them in
// registers (equal digits of a warp find each other with match.any), learns how many keys of
// each digit the tiles before it hold by looking back over their published counts (every thread
// follows one or two digits; a tile publishes its own count at once and the running total as soon as it
// knows it), reorders the tile in shared memory and writes it out in runs.  Tiles are numbered
// in the order in which blocks start, so a block only ever waits for blocks that already run;
// the waits are bounded all the same (status bit 4).  An index that travels with the keys sits
// in their low bits where both fit 64 bits (8 bytes per key and pass instead of 12), in an array
// of its own otherwise.
//
// A pass is bound by latency at small sizes (two dependent rounds of loads and the look-back)
// and by instruction issue at large ones.  The kernel it replaces, one cooperative launch with
// two grid-wide barriers per pass and every block reading every block's counts, took 12 us per
// pass at 120 000 keys and 147 us at 7.3 million.
#pragma once

#include "mn_grid.cuh"
#include "mn_pack.cuh"

#include <algorithm>
#include <type_traits>

namespace mn {
namespace rsort {

constexpr int kThreads = 256;                 // of the key kernel
constexpr int kBits = 9;
constexpr int kDigits = 1 << kBits;
constexpr int kMaxPasses = 8;                 // more than 64 / kBits
constexpr uint32_t kSpinLimit = 1u << 22;

struct Args {
  uint64_t *keys[2];          // ping-pong buffers; the keys start in [0]
  int32_t *vals[2];           // index array of its own, or NULL
  int64_t n;
  int32_t first_bit;          // lowest key bit that is sorted on
  int32_t bits;               // sorted bits; < 0: the key layout's total_bits
  SpecRef spec;
  uint32_t *hist;             // [kMaxPasses][kDigits], zeroed
  uint32_t *next_tile;        // [kMaxPasses], zeroed
  uint32_t *state;            // [passes][tiles][kDigits], zeroed
  int32_t *result_in_second;  // out (may be NULL): 1 when the result is in keys[1]
  int32_t *status;            // device status word
  int32_t tiles;
  uint32_t wait_limit;        // polls of the look-back before it gives up; 0: kSpinLimit
  // the last pass may write the index (low `first_bit` bits of the key, or vals) instead of keys
  int32_t *index32;
  int64_t *index64;
};

__device__ __forceinline__ int passes_of(const Args &a) {
  const int bits = a.bits >= 0 ? a.bits : spec_of(a.spec).total_bits;
  const int p = (bits + kBits - 1) / kBits;
  return p < 1 ? 1 : (p > kMaxPasses ? kMaxPasses : p);
}

// The row that the low bits of a sorted key name (31 at most).
__device__ __forceinline__ int32_t index_of(uint64_t key, uint64_t mask, int64_t n) {
  return (int32_t)min((uint32_t)key & (uint32_t)mask, (uint32_t)n - 1u);
}

__device__ __forceinline__ unsigned lanes_below() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Makes the keys and counts the digits of all passes.  The layout is read once per thread and a
// row's cloud looked for next to the last one's: with a search and a dozen loads of the layout per
// row 7.3 million rows in 64 clouds took 136 us.  A digit that a whole warp shares (the high
// digits of sorted input, most digits of hit words) is added once.
template <typename Source>
__global__ void __launch_bounds__(kThreads)
sort_keys_kernel(const __grid_constant__ Args a, const __grid_constant__ Source source) {
  begin_early();
  __shared__ uint32_t s_hist[kMaxPasses][kDigits];
  const int passes = passes_of(a);
  for (int i = threadIdx.x; i < passes * kDigits; i += kThreads) (&s_hist[0][0])[i] = 0u;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  // A block's keys are consecutive (rows of one cloud mostly), a thread takes two at a time.
  const auto layout = source.layout();
  int hint = 0;
  const int64_t per_block = ((a.n + gridDim.x - 1) / gridDim.x + kThreads - 1) / kThreads * kThreads;
  const int64_t begin = blockIdx.x * per_block, end = min(a.n, begin + per_block);
  for (int64_t i0 = begin; i0 < end; i0 += 2 * kThreads) {
    const int64_t i[2] = {i0 + threadIdx.x, i0 + kThreads + threadIdx.x};
    uint64_t key[2];
    unsigned live[2];
#pragma unroll
    for (int j = 0; j < 2; j++) key[j] = i[j] < end ? source(i[j], layout, hint) : 0ull;
#pragma unroll
    for (int j = 0; j < 2; j++) {
      live[j] = __ballot_sync(0xffffffffu, i[j] < end);
      if (i[j] < end) {
        a.keys[0][i[j]] = key[j];
        if (a.vals[0] != nullptr) a.vals[0][i[j]] = (int32_t)i[j];
        // slots that a timed-out pass leaves out must hold an index all the same
        if (a.index32 != nullptr) a.index32[i[j]] = (int32_t)i[j];
        if (a.index64 != nullptr) a.index64[i[j]] = i[j];
      }
    }
    for (int p = 0; p < passes; p++) {
#pragma unroll
      for (int j = 0; j < 2; j++) {
        if (live[j] == 0u) continue;
        const int leader = __ffs(live[j]) - 1;
        const bool valid = i[j] < end;
        const unsigned d = (unsigned)(key[j] >> (a.first_bit + p * kBits)) & (kDigits - 1);
        const unsigned d0 = __shfl_sync(0xffffffffu, d, leader);
        if (__all_sync(0xffffffffu, d == d0 || !valid)) {
          if (lane == leader) atomicAdd(&s_hist[p][d0], (uint32_t)__popc(live[j]));
        } else if (valid) {
          atomicAdd(&s_hist[p][d], 1u);
        }
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * kDigits; i += kThreads) {
    const uint32_t v = (&s_hist[0][0])[i];
    if (v != 0u) atomicAdd(a.hist + i, v);
  }
}

// exclusive prefix of one value per thread over the block; s_part: [warps]
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t *s_part, int lane, int warp) {
  uint32_t inc = v;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, s);
    if (lane >= s) inc += t;
  }
  if (lane == 31) s_part[warp] = inc;
  __syncthreads();
  uint32_t before = 0;
  for (int w = 0; w < warp; w++) before += s_part[w];
  __syncthreads();
  return before + inc - v;
}

// A thread looks after kPer consecutive digits: two of them with 256 threads, one with 512.
template <int kThr, int kItems, int kBlocks, bool kVals>
__global__ void __launch_bounds__(kThr, kBlocks)
sort_pass_kernel(const __grid_constant__ Args a, int pass) {
  begin_early();
  constexpr int kTile = kThr * kItems, kWarps = kThr / 32, kPer = kDigits / kThr;
  // the tile's keys; before that, the warps' counts per digit, then their first positions inside the
  // tile's digit (at most kTile)
  constexpr int kShared = kTile * 8 > kWarps * kDigits * 2 ? kTile * 8 : kWarps * kDigits * 2;
  __shared__ __align__(16) unsigned char s_raw[kShared];
  uint64_t *s_key = reinterpret_cast<uint64_t *>(s_raw);
  uint16_t (*s_cnt)[kDigits] = reinterpret_cast<uint16_t (*)[kDigits]>(s_raw);
  __shared__ uint32_t s_local[kDigits];              // first position of a digit inside the tile
  __shared__ uint32_t s_dest[kDigits];               // its first position in the output, minus s_local
  __shared__ uint32_t s_part[kWarps];
  __shared__ int s_tile;
  const int passes = passes_of(a);
  if (pass >= passes) return;
  const bool last_pass = pass + 1 == passes;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = lanes_below();
  if (tid == 0) s_tile = (int)atomicAdd(a.next_tile + pass, 1u);
  for (int i = tid; i < kWarps * kDigits / 2; i += kThr) reinterpret_cast<uint32_t *>(&s_cnt[0][0])[i] = 0u;
  uint32_t totals[kPer], all = 0u;
#pragma unroll
  for (int i = 0; i < kPer; i++) totals[i] = __ldcg(a.hist + pass * kDigits + kPer * tid + i);
  __syncthreads();
  const int tile = s_tile;
  if (tile >= a.tiles) return;
  if (tile == 0 && tid == 0 && last_pass && a.result_in_second != nullptr) *a.result_in_second = passes & 1;

  const uint64_t *kin = a.keys[pass & 1];
  const int shift = a.first_bit + pass * kBits;
  const int64_t base = (int64_t)tile * kTile + warp * (kItems * 32) + lane;
  uint64_t key[kItems];
#pragma unroll
  for (int j = 0; j < kItems; j++) key[j] = base + j * 32 < a.n ? __ldcg(kin + base + j * 32) : ~0ull;
  // where this thread's digits start in the output (every block adds up the totals itself), while the keys come
#pragma unroll
  for (int i = 0; i < kPer; i++) all += totals[i];
  const uint32_t digit_start = block_exclusive(all, s_part, lane, warp);
  // ---- rank inside the warp: position among the equal digits of the warp's slice ------------
  uint16_t rank[kItems];
  uint16_t *mine = s_cnt[warp];
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const bool valid = base + j * 32 < a.n;
    const unsigned d = valid ? (unsigned)(key[j] >> shift) & (kDigits - 1) : (unsigned)kDigits;
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    uint32_t before = 0;
    if (valid) before = mine[d];
    __syncwarp();
    if (valid && (peers & lt) == 0u) mine[d] = (uint16_t)(before + __popc(peers));
    rank[j] = (uint16_t)(before + __popc(peers & lt));
    __syncwarp();
  }
  __syncthreads();
  // ---- per digit: the warps' first positions, the tile's count ---------------------------------
  uint32_t count[kPer] = {};
#pragma unroll
  for (int w = 0; w < kWarps; w++) {
    if constexpr (kPer == 2) {
      uint32_t *at = reinterpret_cast<uint32_t *>(s_cnt[w]) + tid;    // two digits
      const uint32_t c = *at;
      *at = count[0] | (count[1] << 16);
      count[0] += c & 0xffffu;
      count[1] += c >> 16;
    } else {
      const uint32_t c = s_cnt[w][tid];
      s_cnt[w][tid] = (uint16_t)count[0];
      count[0] += c;
    }
  }
  // A published word: 2 * value + (running total ? 1 : 0) + 1; 0: nothing yet.  A thread's words are
  // one access, so two of them say the same about what they hold.
  using Word = std::conditional_t<kPer == 2, uint64_t, uint32_t>;
  constexpr int kWords = kDigits / kPer;
  volatile Word *state = reinterpret_cast<Word *>(a.state + ((size_t)pass * a.tiles) * kDigits) + tid;
  auto publish = [&](const uint32_t (&v)[kPer], uint32_t mark) {
    Word w = (Word)(2u * v[0] + mark);
    if constexpr (kPer == 2) w |= (Word)(2u * v[1] + mark) << 32;
    state[(size_t)tile * kWords] = w;
  };
  publish(count, tile == 0 ? 2u : 1u);
  uint32_t sum = 0u;
#pragma unroll
  for (int i = 0; i < kPer; i++) sum += count[i];
  uint32_t local = block_exclusive(sum, s_part, lane, warp);
  // ---- look back: keys of these digits in the tiles before --------------------------------------
  uint32_t before[kPer] = {};
  if (tile > 0) {
    // kLook tiles at a time, their words in flight together.  Where all tiles run at once the running totals
    // spread over them in sqrt(2 tiles / kLook) trips to L2, and eight at a time save a microsecond of a pass
    // (all passes of 27 bits, us, one / 4 / 8 / 16 at a time: 12k keys 21.1 / 18.4 / 19.7 / 20.1; 60k 28.3 /
    // 23.5 / 24.6 / 25.0; 120k 35.2 / 33.8 / 30.9 / 30.7).  Where tiles follow one another the total is found
    // close by, and words read beyond it cost more than they save (1.9 M 119 / 125 / 131 / 136).
    constexpr int kLook = kThr == 256 && kItems == 4 ? 8 : 1;
    uint32_t spins = 0;
    for (int prev = tile - 1; prev >= 0;) {
      Word v[kLook];
#pragma unroll
      for (int q = 0; q < kLook; q++) v[q] = prev >= q ? state[(size_t)(prev - q) * kWords] : (Word)0;
      bool done = false;
      int taken = 0;                                  // up to the first that has not been published
#pragma unroll
      for (int q = 0; q < kLook; q++) {
        const uint32_t x = (uint32_t)v[q];
        if (done || taken < q || x == 0u) continue;
        taken++;
        before[0] += (x - 1u) >> 1;
        if constexpr (kPer == 2) before[1] += ((uint32_t)(v[q] >> 32) - 1u) >> 1;
        done = ((x - 1u) & 1u) != 0u;
      }
      if (done) break;
      prev -= taken;
      if (taken == 0 && ++spins > a.wait_limit) { atomicOr(a.status, MN_STATUS_GRID_TIMEOUT); break; }
    }
    uint32_t upto[kPer];
#pragma unroll
    for (int i = 0; i < kPer; i++) upto[i] = before[i] + count[i];
    publish(upto, 2u);
  }
  uint32_t start = digit_start;
#pragma unroll
  for (int i = 0; i < kPer; i++) {
    s_local[kPer * tid + i] = local;
    s_dest[kPer * tid + i] = start + before[i] - local;
    local += count[i];
    start += totals[i];
  }
  __syncthreads();
  // ---- reorder in shared memory, write in runs -------------------------------------------------
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const unsigned d = (unsigned)(key[j] >> shift) & (kDigits - 1);
    if (base + j * 32 < a.n) rank[j] = (uint16_t)(s_local[d] + s_cnt[warp][d] + rank[j]);
  }
  __syncthreads();                                    // the counts have been read: keys take their place
#pragma unroll
  for (int j = 0; j < kItems; j++)
    if (base + j * 32 < a.n) s_key[rank[j]] = key[j];
  __syncthreads();
  const int in_tile = (int)min((int64_t)kTile, a.n - (int64_t)tile * kTile);
  const bool write_index = last_pass && (a.index32 != nullptr || a.index64 != nullptr);
  uint64_t *kout = a.keys[(pass & 1) ^ 1];
  const uint64_t index_mask = (1ull << a.first_bit) - 1ull;
  uint32_t dest[kItems];
#pragma unroll
  for (int j = 0; j < kItems; j++) {
    const int i = j * kThr + tid;
    if (i < in_tile) {
      const uint64_t k = s_key[i];
      // After a look-back that timed out (status bit 4) keys may land on one another and leave
      // slots of the output with what the buffer held before: positions stay inside the arrays here,
      // and so does every index that is read out of a key, here and in the kernels that follow.
      dest[j] = min(s_dest[(unsigned)(k >> shift) & (kDigits - 1)] + (uint32_t)i, (uint32_t)a.n - 1u);
      if (!write_index) kout[dest[j]] = k;
      else if (!kVals && a.index32 != nullptr) a.index32[dest[j]] = index_of(k, index_mask, a.n);
      else if (!kVals) a.index64[dest[j]] = index_of(k, index_mask, a.n);
    }
  }
  if (kVals) {
    // the index array follows the same way
    int32_t *s_val = reinterpret_cast<int32_t *>(s_key);
    const int32_t *vin = a.vals[pass & 1];
    int32_t val[kItems];
#pragma unroll
    for (int j = 0; j < kItems; j++) val[j] = base + j * 32 < a.n ? __ldcg(vin + base + j * 32) : 0;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kItems; j++)
      if (base + j * 32 < a.n) s_val[rank[j]] = val[j];
    __syncthreads();
    int32_t *vout = a.vals[(pass & 1) ^ 1];
#pragma unroll
    for (int j = 0; j < kItems; j++) {
      const int i = j * kThr + tid;
      if (i < in_tile) {
        const int32_t v = (int32_t)min((uint32_t)s_val[i], (uint32_t)a.n - 1u);
        if (!write_index) vout[dest[j]] = v;
        else if (a.index32 != nullptr) a.index32[dest[j]] = v;
        else a.index64[dest[j]] = v;
      }
    }
  }
}

// Threads and keys per thread of a tile, and its blocks per SM.  Every tile that runs at the same time lengthens
// the look-back, so tiles are large: 4096 keys, with 512 threads up to two tiles per SM and with 256 beyond,
// three to an SM (80 registers; at 128 registers and two, 7.3 M keys took 7 % longer) while that is one wave and a hundredth
// (the few tiles over start as soon as others end).  Four to an SM (64 registers, 8 bytes spilled, 28 with an index array)
// pay beyond, and tiles of 3072 keys where the second wave would be small.  Up to one tile of 1024 keys per SM a pass is shorter with
// those; beyond, up to 606k keys, the large ones leave SMs without a tile and are faster all the same.  Measured,
// all passes, us for 256 x 4 / 512 x 8 / 256 x 16: 30k keys 29 / 37 / 39; 120k 45 / 51 / 53; 250k 64 / 59 / 62;
// 464k 80 / 74 / 78; 900k 115 / 94 / 100; 1.9 M 184 / 141 / 127; 7.3 M 755 / 491 / 445.  36 bits, 256 x 16 with three
// / with four blocks / 256 x 12 with four: 1.5 M 129 / 150 / 132; 1.9 M 147 / 157 / 140; 2.1 M 165 / 159 / 156;
// 2.4 M 188 / 164 / 182; 7.3 M 417 / 390 / 406.  At the line, 256 x 16 with three / 256 x 12 with four, 42 bits: 1.83 M 167 / 173,
// 1.85 M 170 / 175, 1.87 M 175 / 173; 63 bits and an index array: 1.82 M 254 / 261, 1.85 M 266 / 259, 1.91 M 292 / 266; past the
// small second wave 256 x 16 with three / with four, an index array: 2.4 M 373 / 317, 3.5 M 442 / 442, 7.3 M 826 / 782.
struct TileShape { int threads, items, blocks; };
constexpr int64_t kFewKeys = 1024ll * kNumSMs;
constexpr int64_t kOneWave = 3 * 4096ll * kNumSMs, kHardlyTwo = kOneWave + kOneWave / 100, kSmallSecondWave = kOneWave + kOneWave / 5;
inline TileShape tile_shape(int64_t n) {
  if (n < kFewKeys) return TileShape{256, 4, 4};
  if (n < 2 * 4096ll * kNumSMs) return TileShape{512, 8, 2};
  if (n <= kHardlyTwo) return TileShape{256, 16, 3};
  return n <= kSmallSecondWave ? TileShape{256, 12, 4} : TileShape{256, 16, 4};
}
inline int64_t tiles_of(int64_t n) {
  const TileShape s = tile_shape(n);
  return div_up(std::max<int64_t>(n, 1), (int64_t)s.threads * s.items);
}
inline size_t control_words(int64_t n, int passes) {
  return (size_t)kMaxPasses * kDigits + 64 + (size_t)passes * tiles_of(n) * kDigits;
}
// Enough for any number of keys up to n: small tiles are more than the large ones of a larger number of keys.
inline size_t workspace_bytes(int64_t n) {
  size_t words = 0;
  for (int64_t keys : {n, kFewKeys - 1, kSmallSecondWave})
    words = std::max(words, control_words(std::min(n, keys), kMaxPasses));
  return align_up(words * sizeof(uint32_t), 256) + 256;
}

inline int bits_for(int64_t values) {    // bits that tell `values` different values apart, at least 1
  int b = 1;
  while ((1ll << b) < values) b++;
  return b;
}

template <int kThr, int kItems, int kBlocks>
mn_status launch_passes(const Args &a, int launches, cudaStream_t st) {
  for (int p = 0; p < launches; p++) {
    if (a.vals[0] != nullptr) {
      MN_LAUNCH("sort_pass_kernel", st, launch_early(sort_pass_kernel<kThr, kItems, kBlocks, true>, a.tiles, kThr, 0, st, a, p));
    } else {
      MN_LAUNCH("sort_pass_kernel", st, launch_early(sort_pass_kernel<kThr, kItems, kBlocks, false>, a.tiles, kThr, 0, st, a, p));
    }
  }
  return MN_OK;
}

// Stable sort on key bits [first_bit, first_bit + bits) (bits < 0: the key layout's, known on
// the device).  `a` comes with keys, n, bits, spec and what the last pass writes.
template <typename Source>
mn_status run(Args a, const Source &source, Workspace &ws, cudaStream_t st) {
  MN_CHECK_ARG(a.n > 0 && a.n < (1ll << 31) - 1, "radix sort: n = %lld exceeds 2^31-2", (long long)a.n);
  a.tiles = (int32_t)tiles_of(a.n);
  if (a.wait_limit == 0) a.wait_limit = kSpinLimit;
  // bits that only the device knows: no more than fit above the index
  const int bits = a.bits >= 0 ? a.bits : 64 - a.first_bit;
  const int launches = std::min(kMaxPasses, std::max(1, (bits + kBits - 1) / kBits));
  uint32_t *control = ws.take<uint32_t>(control_words(a.n, kMaxPasses));
  MN_CHECK_WS(ws);
  a.hist = control;
  a.next_tile = control + kMaxPasses * kDigits;
  a.state = a.next_tile + 64;
  MN_CHECK_CUDA(cudaMemsetAsync(control, 0, control_words(a.n, launches) * sizeof(uint32_t), st));
  // Every block adds its counts to the digits' totals: no more blocks than run at once, two keys a thread at least
  // (1184 blocks of one key a thread: 120k points 12.5 -> 10.9 us, 464k rows 20.5 -> 16.9, 1.9 M points 32.8 -> 29)
  const int blocks = (int)std::min<int64_t>(kNumSMs * 4, div_up(a.n, 2 * kThreads));
  MN_LAUNCH("sort_keys_kernel", st, launch_early(sort_keys_kernel<Source>, blocks, kThreads, 0, st, a, source));
  const TileShape shape = tile_shape(a.n);
  if (shape.threads == 512) return launch_passes<512, 8, 2>(a, launches, st);
  if (shape.items == 4) return launch_passes<256, 4, 4>(a, launches, st);
  if (shape.items == 12) return launch_passes<256, 12, 4>(a, launches, st);
  return shape.blocks == 3 ? launch_passes<256, 16, 3>(a, launches, st) : launch_passes<256, 16, 4>(a, launches, st);
}

}  // namespace rsort

// Where keys come from.  (Outside any unnamed namespace: kernels are instantiated on these.)
struct CoordKeys {            // coordinate rows, floored to a target stride and packed
  const int32_t *coords;
  const int64_t *batch_dims;
  int32_t ndim, num_clouds, index_bits;   // index_bits > 0: the row index goes below the key
  PackParams pack;
  int32_t *status;
  __device__ __forceinline__ mn_keyspec layout() const { return spec_of(pack.spec); }
  __device__ __forceinline__ uint64_t operator()(int64_t r, const mn_keyspec &spec, int &hint) const {
    int c[4] = {0, 0, 0, 0};
    for (int k = 0; k < ndim; k++) c[k] = __ldg(coords + r * ndim + k);
    const uint64_t g = batch_dims != nullptr ? cloud_near(batch_dims, num_clouds, r, hint) : 0;
    bool bad = false;
    const uint64_t key = pack_one(c, ndim, g, spec, pack, bad);
    if (bad) atomicOr(status, MN_STATUS_KEY_BOX);
    return index_bits > 0 ? (key << index_bits) | (uint64_t)r : key;
  }
};

// Keys of one pass of the dimension-by-dimension sort: the coordinate of dimension `dim`
// (dim >= 0; sign bit flipped, so that unsigned order is signed order) or the cloud (dim < 0) of
// the row that currently sits at position i, the row itself below.
struct DimensionKeys {
  const int32_t *coords;
  const int32_t *perm;
  const int64_t *batch_dims;
  int32_t ndim, dim, num_clouds, index_bits;
  __device__ __forceinline__ int layout() const { return 0; }
  __device__ __forceinline__ uint64_t operator()(int64_t i, int, int &) const {
    const int64_t row = perm != nullptr ? perm[i] : i;
    const uint64_t k = dim >= 0 ? (uint64_t)((uint32_t)__ldg(coords + row * ndim + dim) ^ 0x80000000u)
                                : (uint64_t)cloud_of(batch_dims, num_clouds, row);
    return (k << index_bits) | (uint64_t)row;
  }
};

// Sort keys of a neighbour table's row permutation: the row's hit word with its bits reversed, so
// that rows with the same set of offsets become neighbours and whole tiles can skip the offsets
// none of their rows has.  Mask rows are in ascending size order, so the reversal makes the RARE
// offsets the most significant key bits: the few rows that have a rare offset end up together
// instead of sprinkling it over many tiles.  The key is the reversed word's position in the
// reflected Gray sequence: neighbouring keys differ in one offset instead of many (2-5 % fewer
// offsets per tile than binary order).  Rows stay within their chunk of 2^chunk_shift rows, whose
// number sits on top.  The row itself sits below.
struct HitWordKeys {
  const uint32_t *bits;
  int32_t num_offsets, index_bits, chunk_shift;
  __device__ __forceinline__ int layout() const { return 0; }
  __device__ __forceinline__ uint64_t operator()(int64_t i, int, int &) const {
    uint32_t r = __brev(__ldg(bits + i)) >> (32 - num_offsets);
    r ^= r >> 1; r ^= r >> 2; r ^= r >> 4; r ^= r >> 8; r ^= r >> 16;
    return ((((uint64_t)(i >> chunk_shift) << num_offsets) | (uint64_t)r) << index_bits) | (uint64_t)i;
  }
};

// Voxels of floating-point points: floor(point / size) in the points' own type.
template <typename F>
struct VoxelPoints {
  const F *points;
  F size[4];
  int32_t ndim;
  __device__ __forceinline__ void operator()(int64_t r, int (&c)[4]) const {
#pragma unroll
    for (int k = 0; k < 4; k++) c[k] = k < ndim ? (int)floor(__ldg(points + r * ndim + k) / size[k]) : 0;
  }
};

template <typename F>
struct VoxelKeys {
  VoxelPoints<F> voxel;
  const int64_t *batch_dims;
  int32_t num_clouds, index_bits;
  PackParams pack;
  __device__ __forceinline__ mn_keyspec layout() const { return spec_of(pack.spec); }
  __device__ __forceinline__ uint64_t operator()(int64_t r, const mn_keyspec &spec, int &hint) const {
    int c[4];
    voxel(r, c);
    const uint64_t g = batch_dims != nullptr ? cloud_near(batch_dims, num_clouds, r, hint) : 0;
    bool bad = false;
    return (pack_one(c, voxel.ndim, g, spec, pack, bad) << index_bits) | (uint64_t)r;
  }
};

}  // namespace mn
