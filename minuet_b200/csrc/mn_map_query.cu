// Map step, part 2: kernel-map search, sizes, size order and masks.
//
// The reference builds the kernel map in two traversals
// (csrc/minuet/cuda/functions/query_sorted_index.cu:14-119): a global binary
// search per (256-source block, offset) for target borders, then a per-target
// binary search inside one source block staged in shared memory
// (kernels/query_sorted_index_with_offsets.cuh:60-76); sizes, order and masks
// follow as a reduce-by-key, a torch.sort, a DeviceSelect, two memsets and a
// scatter kernel (functions/scan.cu:221-365, minuet/nn/convolutions.py:156-170).
//
// Here the map build is two launches over packed 64-bit keys.
//
// search_kernel: a block owns 512 consecutive rows (targets).  Two
// warp-cooperative 32-ary ballot searches find the window of the sorted table
// (sources) that can match the tile over all offsets; the window is staged in
// shared memory as a hash set of CELLS (32 consecutive values of the last
// dimension -> {cell id, 32-bit occupancy}, 8-byte slots, linear probing): the
// offsets that differ only in the last dimension (a "group", split so that its
// span is at most 14) are answered by ONE lookup per row, of 16 bytes, i.e. two slots at once.
// What bounds it: instructions and their latency, at five blocks per SM.  A tile of 7.3 million rows and
// 27 offsets took 35 000 cycles, 12 000 of them before its window was known and 19 400 in lookups;
// now 7 500 (layout, keys and tile ends in one trip, the hash cleared before the wait for the kernel
// before, bounds looked for near the tile where the rows are the table) and 13 000 (strips that lie in one cell,
// keys of 32 bits, the few longer probes of a warp in one loop at the end).  464k rows, four
// maps: 138 -> 99 us of searches; 7.3 million, two maps: 634 -> 534 us.  Keys in two cells cost what they save where few and
// long groups ask (build of 1 x 1 x 5 dilated by 7, 464k rows: 31.0 -> 31.9 us; 3 x 3 x 3 dilated by 4 77 -> 72, 50k uniform
// rows 6 % more).  Lanes that add up their bits of a cell before one inserts it: 0.9 of the time on full grids,
// 1.04 on scans, not kept.  Tiles whose window does not fit the hash are
// processed group range by group range, and ranges that still do not fit fall
// back to binary search in global memory.  The kernel writes kernel-map rows
// or, for the fused build, one 32-bit word of per-offset hit bits per row.
//
// emit_masks_kernel (cooperative launch, all blocks resident): every block
// and every warp of it owns a contiguous range of 32-row segments.  Phase 1
// counts the hits per offset of the range (32x32 bit-matrix transposes turn 32
// hit words into 32 per-offset row masks); one grid barrier later every block
// knows its rank offset per offset and the total sizes, hence the stable size
// order; phase 2 turns each segment's row masks into ranks and writes every
// mask row of it with one 128-byte store per warp.  No memset, no select, no
// scatter, no separate scan kernel.  For submanifold maps (sources == targets,
// symmetric offsets) the source mask of offset o is read off the hit bits of
// the mirrored offset.
#include "mn_sort.cuh"

#include <algorithm>
#include <vector>

namespace mn {

namespace {

constexpr int kQThreads = 256;
constexpr int kQWarps = kQThreads / 32;
constexpr int kQRows = 2;                    // rows per thread
constexpr int kQTile = kQThreads * kQRows;   // 512 rows per block
constexpr int kQSlots = 4096;                // hash slots of 8 bytes: {cell, occupancy}
// Table keys per hashed stage.  A key near a cell's start is in two cells: the load factor is at most
// (1 + span / step) * 1280 / 4096, 0.33 for 3 x 3 x 3 and 0.56 for the longest groups (span 14, step 18).
constexpr int kQMaxWindow = 1280;
constexpr int kQMaxSpan = 14;                // last-dimension span of one group
constexpr uint32_t kQPad = 64;               // relative keys start at kQPad
constexpr uint32_t kHashEmpty = 0xffffffffu;
constexpr uint64_t kRelLimit = 0xffffffffull - 4ull * kQPad;
constexpr uint64_t kNarrow = 1ull << 29;
constexpr uint32_t kQNowhere = 0xffffffe0u;  // relative key in a cell past every window's (below kRelLimit + kQPad)

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Warp-cooperative 32-ary search in global memory: lower bound (first index
// with t[i] >= q) or upper bound (first index with t[i] > q) inside [lo, hi).
// Every lane probes one pivot per round, a ballot narrows the range 32-fold;
// ~4 rounds for half a million keys.  All 32 lanes must call with identical
// arguments.
__device__ __forceinline__ int64_t warp_bound(const uint64_t *__restrict__ t, int64_t lo,
                                              int64_t hi, uint64_t q, bool upper, int lane) {
  for (int round = 0; round < 16; round++) {
    const int64_t len = hi - lo;
    if (len <= 0) break;
    const int64_t stride = (len + 31) >> 5;
    const int64_t idx = lo + (int64_t)(lane + 1) * stride - 1;
    bool pred = false;
    if (idx < hi) {
      const uint64_t v = __ldg(t + idx);
      pred = upper ? (v <= q) : (v < q);
    }
    const int c = __popc(__ballot_sync(0xffffffffu, pred));
    if (stride == 1) return lo + c;
    const int64_t nlo = min(lo + (int64_t)c * stride, hi);
    hi = min(hi, nlo + stride - 1);
    lo = nlo;
  }
  return lo;
}

// The same for a bound that is probably near a known place (the tile's own rows, where the rows are
// the table): one round of probes at doubling distances, then the search between two of them.
// Lower bound of q <= t[at] (upper false), upper bound of q >= t[at] (upper true), at inside [0, n).
__device__ __forceinline__ int64_t warp_bound_near(const uint64_t *__restrict__ t, int64_t n, int64_t at, uint64_t q,
                                                   bool upper, int lane) {
  constexpr int64_t kFirst = 16;
  const int64_t idx = upper ? at + (kFirst << lane) : at - (kFirst << lane);
  bool inside = false;                       // the bound lies beyond this probe
  if (idx >= 0 && idx < n) {
    const uint64_t v = __ldg(t + idx);
    inside = upper ? v <= q : v >= q;
  }
  const int c = __popc(__ballot_sync(0xffffffffu, inside));
  const int64_t near = c > 0 ? kFirst << (c - 1) : 0, far = kFirst << min(c, 31);
  if (upper) return warp_bound(t, at + near + 1, min(at + far, n), q, true, lane);
  return warp_bound(t, max(at - far + 1, (int64_t)0), at - near, q, false, lane);
}

struct SearchArgs {
  const uint64_t *rows;
  const uint64_t *table;
  int64_t n_rows;
  int64_t n_table;
  int32_t *kernel_map;     // kMap:  [O, n_rows]
  uint32_t *hit_words;     // kBits / kBitsRev: [n_rows]
  uint32_t *table_words;   // kBitsRev: [n_table], zeroed; bit o of entry s is set when row t hits s
  int32_t n_tiles;
};

// Cells overlap: cell c holds the keys from c * step to c * step + 31, step = 32 - (largest span of a group),
// rounded down to even, so that the strip that a group asks for lies in one cell, and a key near the start of a
// cell is in the one before too.  (In cells side by side one strip in sixteen crossed into the next, i.e. one in
// almost every warp.)  The quotient is exact: k / 2 < 2^31, magic = ceil(2^35 / (step / 2)), step / 2 in 9..16.
struct CellStep {
  uint32_t step, magic;
  __device__ __forceinline__ uint32_t cell(uint32_t k) const { return (uint32_t)(((uint64_t)(k >> 1) * magic) >> 35); }
};
inline CellStep cell_step(const OffsetTable &t) {
  int span = 0;
  for (int g = 0; g < t.num_groups; g++)
    span = std::max(span, t.off[t.member[t.group_begin[g + 1] - 1]][t.ndim - 1] -
                              t.off[t.member[t.group_begin[g]]][t.ndim - 1]);
  const uint32_t half = (uint32_t)(32 - span) / 2;
  return CellStep{2 * half, (uint32_t)(((1ull << 35) + half - 1) / half)};
}

// One launch can serve two searches (e.g. targets->sources and sources->targets).
struct SearchPair {
  SearchArgs a[2];
  OffsetTable tab[2];
  SpecRef spec;
  CellStep cells[2];
  int32_t tiles0;   // blocks of the first search
};

// kMap: kernel-map rows; kBits: per-row hit words; kBitsRev: hit words of the rows
// and, through atomicOr at the matched table position, of the table entries
// (one search then serves both masks of a map whose two sides differ).
enum SearchMode { kMap = 0, kBits = 1, kBitsRev = 2 };

MN_MARKS_DECL(g_marks_search);
MN_MARKS_DECL(g_marks_emit);

// First of the two slots that a lookup reads at once.
__device__ __forceinline__ uint32_t hash_slot(uint32_t c) {
  return (c * 0x9E3779B1u) >> 20 & ~1u;  // top 12 bits: 4096 slots
}

__device__ __forceinline__ uint32_t insert_cell(uint2 *slots, uint32_t c, uint32_t bit) {
  uint32_t h = hash_slot(c);
  for (int probe = 0; probe < kQSlots; probe++) {
    const uint32_t old = atomicCAS(&slots[h].x, kHashEmpty, c);
    if (old == kHashEmpty || old == c) break;
    h = (h + 1) & (kQSlots - 1);
  }
  atomicOr(&slots[h].y, 1u << bit);
  return h;
}

template <int kMode>
__global__ void __launch_bounds__(kQThreads, kMode == kBits ? 5 : 4)
search_kernel(const __grid_constant__ SearchPair sp) {
  constexpr bool kPos = kMode != kBits;   // table positions are needed
  // blocks [0, tiles0) serve direction 0, the rest direction 1 (rows and table swapped)
  const int dir = (int)blockIdx.x >= sp.tiles0 ? 1 : 0;
  const int bid = (int)blockIdx.x - dir * sp.tiles0;
  const SearchArgs &a = sp.a[dir];
  const OffsetTable &tab = sp.tab[dir];
  const CellStep cells = sp.cells[dir];
  __shared__ __align__(16) uint2 s_slots[kQSlots];
  __shared__ uint16_t s_hpos[kPos ? kQSlots : 2];   // first position of a cell
  __shared__ int64_t s_delta[MN_MAX_OFFSETS];
  __shared__ int64_t s_gdelta[MN_MAX_OFFSETS];       // per group: delta of its first member
  __shared__ uint32_t s_gmeta[MN_MAX_OFFSETS];       // first offset | members << 8 | stride << 16
  __shared__ int64_t s_glo[MN_MAX_OFFSETS], s_ghi[MN_MAX_OFFSETS];
  __shared__ int64_t s_slo[MN_MAX_OFFSETS], s_shi[MN_MAX_OFFSETS];
  __shared__ uint8_t s_stage_gbeg[MN_MAX_OFFSETS + 1];
  __shared__ int32_t s_num_stages;
  __shared__ int64_t s_union[2];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int O = tab.num_offsets, G = tab.num_groups;
  const int last = tab.ndim - 1;
  const int64_t tile0 = (int64_t)bid * kQTile;
  const int tile_rows = (int)min((int64_t)kQTile, a.n_rows - tile0);
  const int64_t row0 = tile0 + tid * kQRows;
  auto clear_slots = [&]() {
    uint4 *clear = reinterpret_cast<uint4 *>(s_slots);
    for (int i = tid; i < kQSlots / 2; i += kQThreads)
      clear[i] = make_uint4(kHashEmpty, 0u, kHashEmpty, 0u);   // two {cell, mask} slots
  };
  // what needs no memory of the GPU, while the kernel before this one drains
  clear_slots();
  for (int g = tid; g < G; g += kQThreads) {
    const int mb = tab.group_begin[g], me = tab.group_begin[g + 1];
    const int o_first = tab.member[mb];
    // stride: member i is offset o_first + i and sits i * stride values further along the last dimension; 0: no such
    // order (a dilated kernel's members were looked up one by one in the parameters, two dependent reads each)
    const int stride = me - mb > 1 ? tab.off[tab.member[mb + 1]][last] - tab.off[o_first][last] : 1;
    bool regular = true;
    for (int m = mb; m < me; m++)
      regular &= tab.member[m] == o_first + (m - mb) &&
                 tab.off[tab.member[m]][last] - tab.off[o_first][last] == (m - mb) * stride;
    s_gmeta[g] = (uint32_t)o_first | ((uint32_t)(me - mb) << 8) | ((regular ? (uint32_t)stride : 0u) << 16);
  }
  begin_early();
  MN_MARK(g_marks_search, 0);

  // one trip to memory: the rows' keys, the tile's ends and the key layout together
  uint64_t key[kQRows];
  bool live[kQRows];
  if (tid * kQRows + kQRows <= tile_rows && (reinterpret_cast<uintptr_t>(a.rows) & 15) == 0) {
    const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2 *>(a.rows + row0));
    key[0] = v.x; key[1] = v.y;
    live[0] = live[1] = true;
  } else {
#pragma unroll
    for (int j = 0; j < kQRows; j++) {
      live[j] = tid * kQRows + j < tile_rows;
      key[j] = live[j] ? __ldg(a.rows + row0 + j) : 0ull;
    }
  }
  const uint64_t kfirst = __ldg(a.rows + tile0);
  const uint64_t klast = __ldg(a.rows + tile0 + tile_rows - 1);
  {
    const mn_keyspec &spec = spec_of(sp.spec);
    int shift[MN_MAX_NDIM];
#pragma unroll
    for (int k = 0; k < MN_MAX_NDIM; k++) shift[k] = k < tab.ndim ? spec.shift[k] : 0;
    for (int o = tid; o < O; o += kQThreads) {
      int64_t d = 0;
#pragma unroll
      for (int k = 0; k < MN_MAX_NDIM; k++)
        if (k < tab.ndim) d += (int64_t)tab.off[o][k] * ((int64_t)1 << shift[k]);
      s_delta[o] = d;
    }
  }
  __syncthreads();
  for (int g = tid; g < G; g += kQThreads) s_gdelta[g] = s_delta[tab.member[tab.group_begin[g]]];
  MN_MARK(g_marks_search, 1);

  // window of the table over all offsets: members are ordered by delta
  if (warp < 2) {
    const uint64_t q = warp == 0 ? kfirst + (uint64_t)s_delta[tab.member[0]]
                                 : klast + (uint64_t)s_delta[tab.member[O - 1]];
    // rows that are the table: the window surrounds the tile
    const bool own = a.rows == a.table && a.n_rows == a.n_table && (warp == 0 ? q <= kfirst : q >= klast);
    const int64_t r = own ? warp_bound_near(a.table, a.n_table, warp == 0 ? tile0 : tile0 + tile_rows - 1, q, warp == 1, lane)
                          : warp_bound(a.table, 0, a.n_table, q, warp == 1, lane);
    if (lane == 0) s_union[warp] = r;
  }
  __syncthreads();
  {
    const int64_t ulo = s_union[0], uhi = max(s_union[0], s_union[1]);
    bool one_stage = uhi - ulo <= kQMaxWindow;
    if (one_stage && uhi > ulo)
      one_stage = __ldg(a.table + uhi - 1) - __ldg(a.table + ulo) < kRelLimit;
    if (one_stage) {
      if (tid == 0) {
        s_num_stages = 1;
        s_stage_gbeg[0] = 0;
        s_stage_gbeg[1] = (uint8_t)G;
        s_slo[0] = ulo;
        s_shi[0] = uhi;
      }
    } else {
      // per-group windows inside the union window, then consecutive groups are
      // merged into stages for as long as their joint window fits the hash
      for (int g = warp; g < G; g += kQWarps) {
        const int mb = tab.group_begin[g], me = tab.group_begin[g + 1];
        const uint64_t qlo = kfirst + (uint64_t)s_delta[tab.member[mb]];
        const uint64_t qhi = klast + (uint64_t)s_delta[tab.member[me - 1]];
        const int64_t lo = warp_bound(a.table, ulo, uhi, qlo, false, lane);
        const int64_t hi = warp_bound(a.table, ulo, uhi, qhi, true, lane);
        if (lane == 0) { s_glo[g] = lo; s_ghi[g] = max(lo, hi); }
      }
      __syncthreads();
      if (tid == 0) {
        int ns = 0, g = 0;
        while (g < G) {
          s_stage_gbeg[ns] = (uint8_t)g;
          int64_t lo = s_glo[g], hi = s_ghi[g];
          g++;
          if (hi - lo <= kQMaxWindow) {
            while (g < G) {
              const int64_t nlo = min(lo, s_glo[g]), nhi = max(hi, s_ghi[g]);
              if (nhi - nlo > kQMaxWindow) break;
              lo = nlo; hi = nhi; g++;
            }
          }
          s_slo[ns] = lo;
          s_shi[ns] = hi;
          ns++;
        }
        s_stage_gbeg[ns] = (uint8_t)G;
        s_num_stages = ns;
      }
    }
  }
  __syncthreads();
  MN_MARK(g_marks_search, 2);

  uint32_t bits[kQRows] = {0u, 0u};
  const bool in_pairs = kMode == kMap && (a.n_rows & 1) == 0 &&
                        (reinterpret_cast<uintptr_t>(a.kernel_map) & 7) == 0 && live[kQRows - 1];
  const int num_stages = s_num_stages;
  bool clean = true;                          // no keys in the hash yet
  for (int st = 0; st < num_stages; st++) {
    const int gb = s_stage_gbeg[st], ge = s_stage_gbeg[st + 1];
    const int64_t lo = s_slo[st], hi = s_shi[st];
    const int wn = (int)min(hi - lo, (int64_t)kQMaxWindow + 1);
    bool hashed = hi - lo <= kQMaxWindow;
    uint64_t base = 0;
    if (hashed && wn > 0) {
      base = __ldg(a.table + lo);
      hashed = __ldg(a.table + hi - 1) - base < kRelLimit;
    }
    if (hashed) {
      if (!clean) {
        clear_slots();
        __syncthreads();
      }
      clean = false;
      MN_MARK(g_marks_search, 3);
      // relative keys start at kQPad, so that a query below the window stays non-negative
      for (int w = tid; w < wn; w += kQThreads) {
        const uint32_t k = (uint32_t)(__ldg(a.table + lo + w) - base) + kQPad;
        // the table is sorted: a cell's keys follow one another, and all but the first have a predecessor in it
        uint32_t pk = 0;
        if (kPos && w > 0) pk = (uint32_t)(__ldg(a.table + lo + w - 1) - base) + kQPad;
        const uint32_t c = cells.cell(k), at = k - c * cells.step;
        const uint32_t h = insert_cell(s_slots, c, at);
        if (kPos && (w == 0 || pk < k - at)) s_hpos[h] = (uint16_t)w;
        if (at + cells.step < 32u) {
          const uint32_t h1 = insert_cell(s_slots, c - 1u, at + cells.step);
          if (kPos && (w == 0 || pk < k - at - cells.step)) s_hpos[h1] = (uint16_t)w;
        }
      }
      __syncthreads();
      MN_MARK(g_marks_search, 4);
      int64_t rel[kQRows];
#pragma unroll
      for (int j = 0; j < kQRows; j++)   // a dead row gets a value that no window can reach
        rel[j] = live[j] ? (int64_t)(key[j] - base) + kQPad : (int64_t)1 << 62;
      // Where window, rows and offsets span less than 2^29 the relative keys are sums of 32 bits: what
      // falls outside the window is in no cell of it (a dead row's sums are off by 2^31).  A window without
      // keys has no last one.
      const int64_t first_delta = s_delta[tab.member[0]], last_delta = s_delta[tab.member[O - 1]];
      const bool narrow = wn > 0 && __ldg(a.table + hi - 1) - base < kNarrow && (int64_t)(kfirst - base) > -(int64_t)kNarrow &&
                          (int64_t)(klast - base) < (int64_t)kNarrow && first_delta > -(int64_t)kNarrow &&
                          last_delta < (int64_t)kNarrow;
      auto relative = [&](int j, int g) {
        if (narrow) return (uint32_t)rel[j] + (uint32_t)s_gdelta[g] + (live[j] ? 0u : 0x80000000u);
        const uint64_t t0 = (uint64_t)(rel[j] + s_gdelta[g]);
        return t0 < kRelLimit + kQPad ? (uint32_t)t0 : kQNowhere;   // the window's last key may be kQPad past the limit
      };
      // what the offsets of group g find for row j: the strip of its cell from `sh` on
      auto found_strip = [&](int j, uint32_t meta, uint32_t mask, uint32_t sh, uint32_t slot) {
        const uint32_t o_first = meta & 0xffu, members = (meta >> 8) & 0xffu;
        const uint32_t strip = (mask >> sh) & ((1u << members) - 1u);
        bits[j] |= strip << o_first;
        if (kMode == kBitsRev && strip != 0u) {
          // entries of a cell follow one another
          uint32_t *at = a.table_words + lo + s_hpos[slot] + __popc(mask & ((1u << sh) - 1u));
          for (uint32_t rest = strip; rest != 0u; rest &= rest - 1u, at++)
            atomicOr(at, (rest & (0u - rest)) << o_first);
        }
      };
      auto member_of = [&](int g, uint32_t meta, int m, int &o, uint32_t &de) {
        const int o_first = (int)(meta & 0xffu);
        const uint32_t stride = meta >> 16;
        o = stride != 0u ? o_first + m : tab.member[tab.group_begin[g] + m];
        de = stride != 0u ? (uint32_t)m * stride : (uint32_t)(tab.off[o][last] - tab.off[o_first][last]);   // sh + de < 32
      };
      // The same for the thread's rows together, where a member at a time is looked at: a map's entries of two rows
      // are one store.  (Not unrolled: beside it the strips, which most maps are made of, lost 3 %: 7.3 M rows 3 x 3 x 3, build,
      // 636 -> 618 us; dilated by 4 841 -> 786.)
      auto found_by_member = [&](int g, uint32_t meta, const uint32_t (&mask)[kQRows], const uint32_t (&sh)[kQRows],
                                 const uint32_t (&slot)[kQRows]) {
        const int members = (int)((meta >> 8) & 0xffu);
        int32_t first[kQRows];
#pragma unroll
        for (int j = 0; j < kQRows; j++) first[j] = kPos ? (int32_t)(lo + s_hpos[slot[j]]) : 0;
#pragma unroll 1
        for (int m = 0; m < members; m++) {
          int o;
          uint32_t de;
          member_of(g, meta, m, o, de);
          int32_t idx[kQRows];
#pragma unroll
          for (int j = 0; j < kQRows; j++) {
            const uint32_t below = mask[j] & ((1u << (sh[j] + de)) - 1u), hit = mask[j] >> (sh[j] + de) & 1u;
            idx[j] = hit != 0u ? first[j] + __popc(below) : -1;
            if (kMode != kMap) {
              bits[j] |= hit << o;
              if (kMode == kBitsRev && hit != 0u) atomicOr(a.table_words + idx[j], 1u << o);
            }
          }
          if (kMode == kMap) {
            int32_t *dst = a.kernel_map + (int64_t)o * a.n_rows + row0;
            if (in_pairs) {
              *reinterpret_cast<int2 *>(dst) = make_int2(idx[0], idx[1]);
            } else {
#pragma unroll
              for (int j = 0; j < kQRows; j++) if (live[j]) dst[j] = idx[j];
            }
          }
        }
      };
      // and for one row whose lookup was put off: its offsets have found nothing so far
      auto found_late = [&](int j, int g, uint32_t mask, uint32_t sh, uint32_t slot) {
        const uint32_t meta = s_gmeta[g];
        if (kMode != kMap && (meta >> 16) == 1u) {
          found_strip(j, meta, mask, sh, slot);
          return;
        }
        const int members = (int)((meta >> 8) & 0xffu);
#pragma unroll 1
        for (int m = 0; m < members; m++) {
          int o;
          uint32_t de;
          member_of(g, meta, m, o, de);
          if ((mask >> (sh + de) & 1u) == 0u) continue;
          const int32_t idx = kPos ? (int32_t)(lo + s_hpos[slot] + __popc(mask & ((1u << (sh + de)) - 1u))) : 0;
          if (kMode == kMap) {
            if (live[j]) a.kernel_map[(int64_t)o * a.n_rows + row0 + j] = idx;
          } else {
            bits[j] |= 1u << o;
            if (kMode == kBitsRev) atomicOr(a.table_words + idx, 1u << o);
          }
        }
      };
      // Linear probing over {cell, mask} slots.  The first two slots are one load and hold nearly all answers;
      // a lookup that has to go on is put off (its offsets have found nothing so far) until the others are
      // through, so that a warp goes round the probing loop for its few of them together.
      for (int g0 = gb; g0 < ge; g0 += 32) {
        const int g1 = min(ge, g0 + 32);
        uint32_t open[kQRows] = {0u, 0u};
#pragma unroll 3
        for (int g = g0; g < g1; g++) {
          uint32_t mask[kQRows], sh[kQRows], slot[kQRows];
#pragma unroll
          for (int j = 0; j < kQRows; j++) {
            const uint32_t q = relative(j, g), c = cells.cell(q);
            sh[j] = q - c * cells.step;
            slot[j] = hash_slot(c);
            const uint4 v = *reinterpret_cast<const uint4 *>(s_slots + slot[j]);
            const bool second = v.z == c;
            mask[j] = v.x == c ? v.y : second ? v.w : 0u;
            if (v.x != c && !second && v.z != kHashEmpty) open[j] |= 1u << (g - g0);
            slot[j] += second ? 1u : 0u;
          }
          const uint32_t meta = s_gmeta[g];
          if (kMode == kMap || (meta >> 16) != 1u) {
            found_by_member(g, meta, mask, sh, slot);
          } else {
#pragma unroll
            for (int j = 0; j < kQRows; j++) found_strip(j, meta, mask[j], sh[j], slot[j]);
          }
        }
#pragma unroll
        for (int j = 0; j < kQRows; j++) {
          for (; open[j] != 0u; open[j] &= open[j] - 1u) {
            const int g = g0 + __ffs(open[j]) - 1;
            const uint32_t q = relative(j, g), c = cells.cell(q);
            uint32_t slot = hash_slot(c) + 1u;
            uint2 v;
            int probe = 0;
            do {
              slot = (slot + 1u) & (kQSlots - 1);
              v = s_slots[slot];
            } while (v.x != c && v.x != kHashEmpty && ++probe < kQSlots);
            if (v.x == c) found_late(j, g, v.y, q - c * cells.step, slot);
          }
        }
      }
      __syncthreads();
    } else {
      // ---- window too large or too wide for the hash: binary search in global memory
      for (int g = gb; g < ge; g++) {
        const int mb = tab.group_begin[g], me = tab.group_begin[g + 1];
        const int64_t glo = s_glo[g], ghi = s_ghi[g];
        int64_t pos[kQRows];
#pragma unroll
        for (int j = 0; j < kQRows; j++) {
          const uint64_t q0 = key[j] + (uint64_t)s_delta[tab.member[mb]];
          int64_t l = glo, h = ghi;
          while (l < h) {
            const int64_t mid = (l + h) >> 1;
            if (__ldg(a.table + mid) < q0) l = mid + 1; else h = mid;
          }
          pos[j] = l;
        }
        for (int m = mb; m < me; m++) {
          const int o = tab.member[m];
          int32_t idx[kQRows];
#pragma unroll
          for (int j = 0; j < kQRows; j++) {
            const uint64_t q = key[j] + (uint64_t)s_delta[o];
            int64_t p = pos[j];
            uint64_t v = ~0ull;
            while (p < ghi) {   // at most kQMaxSpan steps: the table holds distinct keys
              v = __ldg(a.table + p);
              if (v >= q) break;
              p++;
              v = ~0ull;
            }
            pos[j] = p;
            idx[j] = (live[j] && v == q) ? (int32_t)p : -1;
          }
          if (kMode == kMap) {
            int32_t *dst = a.kernel_map + (int64_t)o * a.n_rows + row0;
#pragma unroll
            for (int j = 0; j < kQRows; j++) if (live[j]) dst[j] = idx[j];
          } else {
#pragma unroll
            for (int j = 0; j < kQRows; j++) {
              if (idx[j] >= 0) {
                bits[j] |= 1u << o;
                if (kMode == kBitsRev) atomicOr(a.table_words + idx[j], 1u << o);
              }
            }
          }
        }
      }
    }
  }

  MN_MARK(g_marks_search, 5);
  if (kMode != kMap) {
    if (live[kQRows - 1] && (reinterpret_cast<uintptr_t>(a.hit_words) & 7) == 0) {
      *reinterpret_cast<uint2 *>(a.hit_words + row0) = make_uint2(bits[0], bits[1]);
    } else {
#pragma unroll
      for (int j = 0; j < kQRows; j++) if (live[j]) a.hit_words[row0 + j] = bits[j];
    }
  }
}

// ---------------------------------------------------------------------------
// masks from hit words (fused build)
// ---------------------------------------------------------------------------
constexpr int kEThreads = 512;
constexpr int kEWarps = kEThreads / 32;
constexpr int kESegs = 4;             // 32-row segments a warp takes at a time
constexpr int kEUnit = kESegs * 32;

struct EmitArgs {
  const uint32_t *words_t;   // [T] hit bits of target rows
  const uint32_t *words_s;   // [S] hit bits of source rows (== words_t when mirrored)
  int32_t *target_masks;     // [O, T]
  int32_t *source_masks;     // [O, S]
  int32_t *order_out;        // [O] offset at mask row p
  int32_t *sizes_out;        // [O + 1] size of mask row p, then a copy of the status word
  int32_t *sizes_host;       // the same in host memory, or NULL
  uint32_t *bits_t;          // optional [T]: bit p set when mask row p has an entry for the target
  uint32_t *bits_s;          // optional [S]: the same for the sources
  int32_t *agg;              // workspace [64 pairs][grid]: hit counts of every block's rows;
                             // pair = direction * 32 + offset
  int32_t *ctrl;
  int64_t T, S;
  int32_t units_t, units_s;  // kEUnit-row units of the targets / the sources
  int32_t num_offsets;
  int32_t reorder;
  uint8_t mirror[32];        // source direction: which offset's bit to read
};

// Transpose of the 32x32 bit matrix held one row per lane: on return lane j
// holds column j (bit i = bit j of lane i's input).
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane) {
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) {
    const uint32_t low = s == 16 ? 0x0000ffffu : s == 8 ? 0x00ff00ffu : s == 4 ? 0x0f0f0f0fu
                       : s == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, s);
    x = (lane & s) ? ((x & ~low) | ((y & ~low) >> s)) : ((x & low) | ((y & low) << s));
  }
  return x;
}

// A warp owns consecutive 128-row units of the target rows followed by the source rows, lane p
// the running rank of mask row p; a mask row of a unit is four 128-byte stores of the whole warp.
// After the grid-wide barrier no warp waits for another one: with 512-row tiles staged in shared
// memory and three block barriers a tile the kernel spent half its time in those barriers where
// the masks are narrow (7.3M + 7.1M rows, 8 offsets: 301 us, now 160; 464k + 464k rows 28, now
// 18 us).  With 27 offsets it is bound by the bytes it writes (1.58 GB in 355 us either way).
// More than two blocks of 16 warps per SM make it slower: too many rows are open at a time.
__global__ void __launch_bounds__(kEThreads, 2)
emit_masks_kernel(const __grid_constant__ EmitArgs e) {
  release_successor();
  __shared__ int32_t s_wcnt[2][32][kEWarps + 1];        // per direction / offset: warp counts, then warp bases
  __shared__ int32_t s_first[2][32], s_size[32], s_ord[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int O = e.num_offsets;
  const int G = (int)gridDim.x, b = (int)blockIdx.x;
  const int64_t total_units = (int64_t)e.units_t + e.units_s, workers = (int64_t)G * kEWarps;
  const int64_t me = (int64_t)b * kEWarps + warp;
  const int begin = (int)(total_units * me / workers), end = (int)(total_units * (me + 1) / workers);
  const unsigned lt = lanemask_lt();
  const int my_mirror = lane < O ? e.mirror[lane] : 0;

  MN_MARK(g_marks_emit, 0);
  auto fetch_words = [&](int unit, uint32_t (&w)[kESegs]) {
    const int dir = unit >= e.units_t ? 1 : 0;
    const int64_t n = unit < end ? (dir ? e.S : e.T) : 0;
    const int64_t r = (int64_t)(unit - (dir ? e.units_t : 0)) * kEUnit + lane;
    const uint32_t *words = dir ? e.words_s : e.words_t;
#pragma unroll
    for (int k = 0; k < kESegs; k++) w[k] = r + 32 * k < n ? __ldg(words + r + 32 * k) : 0u;
  };

  // ---- phase 1: hits per offset of this warp's rows -------------------------------
  {
    int cnt0 = 0, cnt1 = 0;   // lane o: hits of offset o, per direction
    uint32_t w[kESegs], next[kESegs];
    fetch_words(begin, w);
    for (int unit = begin; unit < end; unit++) {
      fetch_words(unit + 1, next);
#pragma unroll
      for (int k = 0; k < kESegs; k++) {
        const int c = __popc(transpose32(w[k], lane));
        if (unit >= e.units_t) cnt1 += c; else cnt0 += c;
        w[k] = next[k];
      }
    }
    cnt1 = __shfl_sync(0xffffffffu, cnt1, my_mirror);
    if (lane < O) { s_wcnt[0][lane][warp] = cnt0; s_wcnt[1][lane][warp] = cnt1; }
  }
  __syncthreads();
  if (tid < 64) {
    int sum = 0;
    if ((tid & 31) < O)
      for (int w = 0; w < kEWarps; w++) {
        const int c = s_wcnt[tid >> 5][tid & 31][w];
        s_wcnt[tid >> 5][tid & 31][w] = sum;
        sum += c;
      }
    e.agg[(int64_t)tid * G + b] = sum;
  }
  __syncthreads();
  MN_MARK(g_marks_emit, 1);
  grid_barrier(e.ctrl, (unsigned)G);
  MN_MARK(g_marks_emit, 2);

  // ---- totals and this block's first ranks: every block adds up the other blocks' counts
  // itself (a few hundred 4-byte reads per pair), which is cheaper than a second barrier ------
  // (a warp's four pairs together: one after the other they were eight dependent trips to L2, 3.5 us of every map)
  {
    constexpr int kPairs = 64 / kEWarps, kBatch = 5;
    int all[kPairs] = {}, before[kPairs] = {};
    for (int b0 = lane; b0 < G; b0 += 32 * kBatch) {
      int v[kPairs][kBatch];
#pragma unroll
      for (int q = 0; q < kPairs; q++) {
        const int pair = warp + q * kEWarps;
        const int32_t *row = e.agg + (int64_t)pair * G;
#pragma unroll
        for (int i = 0; i < kBatch; i++)
          v[q][i] = (pair & 31) < O && b0 + 32 * i < G ? __ldcg(row + b0 + 32 * i) : 0;
      }
#pragma unroll
      for (int q = 0; q < kPairs; q++)
#pragma unroll
        for (int i = 0; i < kBatch; i++) {
          all[q] += v[q][i];
          before[q] += b0 + 32 * i < b ? v[q][i] : 0;
        }
    }
#pragma unroll
    for (int q = 0; q < kPairs; q++) {
      const int pair = warp + q * kEWarps;
      const int sum = __reduce_add_sync(0xffffffffu, all[q]), mine = __reduce_add_sync(0xffffffffu, before[q]);
      if (lane == 0 && (pair & 31) < O) {
        s_first[pair >> 5][pair & 31] = mine;
        if (pair < 32) s_size[pair] = sum;
      }
    }
  }
  if (tid < 32) s_ord[tid] = 0;
  __syncthreads();
  if (tid < O) {
    int pos = tid;
    if (e.reorder) {
      // stable ascending sizes: ties keep the offset order
      const int mine = s_size[tid];
      pos = 0;
      for (int j = 0; j < O; j++) {
        const int other = s_size[j];
        pos += (other < mine) || (other == mine && j < tid);
      }
    }
    s_ord[pos] = tid;
    if (b == 0) {
      e.order_out[pos] = tid;
      e.sizes_out[pos] = s_size[tid];
      if (e.sizes_host != nullptr) e.sizes_host[pos] = s_size[tid];
    }
  }
  if (b == 0 && tid == 0) {
    const int32_t status = e.ctrl[MN_CTRL_STATUS];
    e.sizes_out[O] = status;
    if (e.sizes_host != nullptr) e.sizes_host[O] = status;
  }
  __syncthreads();
  // from here on lane p stands for mask row p
  const int ord = s_ord[lane];
  const int plane_of[2] = {ord, __shfl_sync(0xffffffffu, my_mirror, ord)};
  int run[2];
#pragma unroll
  for (int d = 0; d < 2; d++)
    run[d] = lane < O ? s_first[d][ord] + s_wcnt[d][ord][warp] : 0;

  MN_MARK(g_marks_emit, 5);
  // ---- phase 2: ranks ------------------------------------------------------------------
  uint32_t w[kESegs], next[kESegs];
  fetch_words(begin, w);
  for (int unit = begin; unit < end; unit++) {
    fetch_words(unit + 1, next);
    const int dir = unit >= e.units_t ? 1 : 0;
    const int64_t n = dir ? e.S : e.T, r = (int64_t)(unit - (dir ? e.units_t : 0)) * kEUnit + lane;
    const int left = (int)min(n - r, (int64_t)kEUnit);   // rows from this lane's first one on
    uint32_t *bits_out = dir ? e.bits_s : e.bits_t;
    uint32_t plane[kESegs], seen = 0u;
    int count = 0;
#pragma unroll
    for (int k = 0; k < kESegs; k++) {
      plane[k] = __shfl_sync(0xffffffffu, transpose32(w[k], lane), dir ? plane_of[1] : plane_of[0]);
      if (lane >= O) plane[k] = 0u;
      seen |= plane[k];
      count += __popc(plane[k]);
      // hit word of every row in mask-row order (bit p <-> mask row p), for the
      // convolution kernels that walk a row's pairs without scanning the masks
      if (bits_out != nullptr) {
        const uint32_t by_row = transpose32(plane[k], lane);
        if (32 * k < left) bits_out[r + 32 * k] = by_row;
      }
      w[k] = next[k];
    }
    const unsigned any = __ballot_sync(0xffffffffu, seen != 0u);
    const int first_rank = dir ? run[1] : run[0];
    int32_t *dst = (dir ? e.source_masks : e.target_masks) + r;
    for (int p = 0; p < O; p++, dst += n) {
      int v[kESegs];
#pragma unroll
      for (int k = 0; k < kESegs; k++) v[k] = -1;
      if ((any >> p) & 1u) {
        int rank = __shfl_sync(0xffffffffu, first_rank, p);
#pragma unroll
        for (int k = 0; k < kESegs; k++) {
          const uint32_t pl = __shfl_sync(0xffffffffu, plane[k], p);
          if ((pl >> lane) & 1u) v[k] = rank + __popc(pl & lt);
          rank += __popc(pl);
        }
      }
#pragma unroll
      for (int k = 0; k < kESegs; k++)
        if (32 * k < left) dst[32 * k] = v[k];
    }
    if (dir) run[1] += count; else run[0] += count;
  }
  MN_MARK(g_marks_emit, 6);
}

__global__ void identity_order_kernel(int O, int32_t *order_out, int32_t *sizes_out, int32_t *sizes_host,
                                      const int32_t *ctrl) {
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o < O) order_out[o] = o;
  if (o <= O) {
    const int32_t v = o < O ? 0 : ctrl[MN_CTRL_STATUS];
    sizes_out[o] = v;
    if (sizes_host != nullptr) sizes_host[o] = v;
  }
}

// ---------------------------------------------------------------------------
// reference-API pieces that start from a materialised kernel map
// ---------------------------------------------------------------------------
constexpr int kMTile = 1024;     // rows per tile of the kernels below
constexpr int kMThreads = 256;

// counts[o, tile] = valid entries of kernel_map[o, tile * kMTile ...)
__global__ void __launch_bounds__(kMThreads)
map_count_kernel(const int32_t *__restrict__ kernel_map, int64_t T, int n_tiles,
                 int32_t *__restrict__ counts, int32_t *__restrict__ sizes_atomic) {
  const int o = blockIdx.y, tile = blockIdx.x;
  const int64_t t0 = (int64_t)tile * kMTile;
  int c = 0;
#pragma unroll
  for (int j = 0; j < kMTile / kMThreads; j++) {
    const int64_t t = t0 + j * kMThreads + threadIdx.x;
    if (t < T) c += __ldg(kernel_map + (int64_t)o * T + t) != -1;
  }
  c = __reduce_add_sync(0xffffffffu, c);
  __shared__ int s[kMThreads / 32];
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int tot = 0;
    for (int w = 0; w < kMThreads / 32; w++) tot += s[w];
    if (counts != nullptr) counts[(int64_t)o * n_tiles + tile] = tot;
    if (sizes_atomic != nullptr && tot != 0) atomicAdd(sizes_atomic + o, tot);
  }
}

// Block o turns row o of counts ([O, tiles]) into its exclusive prefix, in place.
__global__ void __launch_bounds__(1024)
scan_tiles_kernel(int32_t *__restrict__ counts, int n) {
  __shared__ int32_t s_warp[32];
  __shared__ int32_t s_carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int32_t *row = counts + (int64_t)blockIdx.x * n;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (int b0 = 0; b0 < n; b0 += 1024) {
    const int b = b0 + threadIdx.x;
    const int32_t v = b < n ? row[b] : 0;
    int32_t inc = v;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const int32_t t = __shfl_up_sync(0xffffffffu, inc, s);
      if (lane >= s) inc += t;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    int32_t before = s_carry;
    for (int w = 0; w < warp; w++) before += s_warp[w];
    if (b < n) row[b] = before + inc - v;
    __syncthreads();
    if (threadIdx.x == 1023) s_carry = before + inc;
    __syncthreads();
  }
}

// rank valid entries of row o by t; write the target mask densely and the
// source mask (pre-filled with -1) by scatter
__global__ void __launch_bounds__(kMThreads)
map_masks_kernel(const int32_t *__restrict__ kernel_map, int64_t S, int64_t T, int n_tiles,
                 const int32_t *__restrict__ prefix, int32_t *__restrict__ source_masks,
                 int32_t *__restrict__ target_masks) {
  const int o = blockIdx.y, tile = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t t0 = (int64_t)tile * kMTile + threadIdx.x * 4;
  int32_t s_idx[4];
  int mine = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    s_idx[i] = (t0 + i < T) ? __ldg(kernel_map + (int64_t)o * T + t0 + i) : -1;
    mine += s_idx[i] != -1;
  }
  int inc = mine;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, s);
    if (lane >= s) inc += t;
  }
  __shared__ int s_w[kMThreads / 32];
  if (lane == 31) s_w[warp] = inc;
  __syncthreads();
  int r = prefix[(int64_t)o * n_tiles + tile] + inc - mine;
  for (int w = 0; w < warp; w++) r += s_w[w];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    if (t0 + i < T) {
      const bool v = s_idx[i] != -1;
      target_masks[(int64_t)o * T + t0 + i] = v ? r : -1;
      if (v) source_masks[(int64_t)o * S + s_idx[i]] = r;
      r += v;
    }
  }
}

void fill_search_args(SearchArgs *a, const uint64_t *rows, int64_t n_rows, const uint64_t *table,
                      int64_t n_table, int32_t *kernel_map, uint32_t *hit_words) {
  *a = SearchArgs{};
  a->rows = rows; a->table = table; a->n_rows = n_rows; a->n_table = n_table;
  a->kernel_map = kernel_map; a->hit_words = hit_words;
  a->n_tiles = (int)div_up(n_rows, kQTile);
}

// Launches one search, or two in the same grid when `second` is given.
mn_status run_search(int mode, const mn_keyspec &spec, const SearchArgs &first,
                     const OffsetTable &tab_first, const SearchArgs *second,
                     const OffsetTable *tab_second, cudaStream_t st) {
  thread_local static SearchPair sp;   // ~5 KB: kept off the stack; passed by value per launch
  sp.a[0] = first;
  sp.tab[0] = tab_first;
  sp.cells[0] = cell_step(tab_first);
  sp.spec = make_spec_ref(spec);
  sp.tiles0 = first.n_tiles;
  int blocks = first.n_tiles;
  if (second != nullptr) {
    sp.a[1] = *second;
    sp.tab[1] = *tab_second;
    sp.cells[1] = cell_step(*tab_second);
    blocks += second->n_tiles;
  }
  if (blocks == 0) return MN_OK;
  {
    LaunchScope scope(mode == kMap ? "search_kernel<map>" : mode == kBits ? "search_kernel<bits>"
                                                                         : "search_kernel<bits,rev>", st);
    if (mode == kMap) launch_early(search_kernel<kMap>, blocks, kQThreads, 0, st, sp);
    else if (mode == kBits) launch_early(search_kernel<kBits>, blocks, kQThreads, 0, st, sp);
    else launch_early(search_kernel<kBitsRev>, blocks, kQThreads, 0, st, sp);
  }
  MN_CHECK_LAUNCH();
  return MN_OK;
}

}  // namespace

mn_status make_offset_table(const int32_t *offsets, int64_t O, int ndim, int sign,
                            const mn_keyspec *spec, OffsetTable *out) {
  MN_CHECK_ARG(offsets != nullptr && spec != nullptr, "offset table: null pointer");
  MN_CHECK_ARG(O >= 1 && O <= MN_MAX_OFFSETS, "offset table: %lld offsets (supported: 1..%d)",
               (long long)O, MN_MAX_OFFSETS);
  MN_CHECK_ARG(ndim == spec->ndim, "offset table: ndim %d differs from the key spec's %d", ndim,
               spec->ndim);
  *out = OffsetTable{};
  out->num_offsets = (int32_t)O;
  out->ndim = ndim;
  for (int64_t o = 0; o < O; o++)
    for (int k = 0; k < ndim; k++) {
      const int64_t v = (int64_t)sign * offsets[o * ndim + k];
      MN_CHECK_ARG(v >= -(int64_t)spec->margin && v <= (int64_t)spec->margin,
                   "offset %lld exceeds the key margin %d", (long long)v, spec->margin);
      out->off[o][k] = (int32_t)v;
    }
  std::vector<int> idx(O);
  for (int64_t o = 0; o < O; o++) idx[o] = (int)o;
  std::stable_sort(idx.begin(), idx.end(), [&](int x, int y) {
    for (int k = 0; k < ndim; k++)
      if (out->off[x][k] != out->off[y][k]) return out->off[x][k] < out->off[y][k];
    return false;
  });
  // a group: same offset in every dimension but the last, last-dimension span <= kQMaxSpan
  int g = 0, first = 0;
  for (int64_t i = 0; i < O; i++) {
    out->member[i] = (uint8_t)idx[i];
    bool new_group = i == 0;
    if (i > 0) {
      for (int k = 0; k + 1 < ndim; k++)
        new_group |= out->off[idx[i]][k] != out->off[idx[i - 1]][k];
      new_group |= out->off[idx[i]][ndim - 1] - out->off[first][ndim - 1] > kQMaxSpan;
    }
    if (new_group) {
      out->group_begin[g++] = (uint8_t)i;
      first = idx[i];
    }
  }
  out->group_begin[g] = (uint8_t)O;
  out->num_groups = g;
  return MN_OK;
}

}  // namespace mn

using namespace mn;

extern "C" size_t mn_map_workspace_bytes(int64_t S, int64_t T, int64_t O) {
  const int64_t n = std::max<int64_t>(std::max(S, T), 1);
  size_t sort = 2 * align_up((size_t)n * 8, 256) + 2 * align_up((size_t)n * 4, 256) +
                rsort::workspace_bytes(n) + align_up((size_t)div_up(n, 2048) * 4, 256) + 512;
  const int64_t tiles = div_up(S, kMTile) + div_up(T, kMTile) + 2;
  size_t map = align_up((size_t)S * 4, 256) + align_up((size_t)T * 4, 256) +
               2 * align_up((size_t)std::max<int64_t>(O, 1) * tiles * 4, 256) +
               align_up((size_t)kMaxCoopBlocks * 64 * 4, 256) + 4 * 1024;
  size_t bbox = (size_t)kNumSMs * 4 * 8 * 4 + 256;
  return std::max(std::max(sort, map), bbox) + 4096;
}

extern "C" mn_status mn_query_sorted_index_with_offsets(
    const uint64_t *source_keys, int64_t S, const uint64_t *target_keys, int64_t T,
    const int32_t *offsets, int64_t O, const mn_keyspec *spec, int32_t *kernel_map_out,
    void *stream) {
  MN_CHECK_ARG(S >= 0 && T >= 0, "query: negative size");
  MN_CHECK_ARG(spec != nullptr, "query: null key spec");
  MN_CHECK_ARG(S < (1ll << 31) && T < (1ll << 31), "query: more than 2^31-1 rows");
  OffsetTable tab;
  MN_RETURN_IF(make_offset_table(offsets, O, spec->ndim, +1, spec, &tab));
  if (T == 0) return MN_OK;
  MN_CHECK_ARG(target_keys != nullptr && kernel_map_out != nullptr && (S == 0 || source_keys != nullptr),
               "query: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (S == 0) {
    MN_CHECK_CUDA(cudaMemsetAsync(kernel_map_out, 0xff, sizeof(int32_t) * O * T, st));
    return MN_OK;
  }
  SearchArgs a;
  fill_search_args(&a, target_keys, T, source_keys, S, kernel_map_out, nullptr);
  return run_search(kMap, *spec, a, tab, nullptr, nullptr, st);
}

extern "C" mn_status mn_compute_kernel_map_sizes(const int32_t *kernel_map, int64_t O, int64_t T,
                                                 int32_t *sizes_out, void *stream) {
  MN_CHECK_ARG(O >= 0 && T >= 0 && O <= 65535, "sizes: bad shape");
  if (O == 0) return MN_OK;
  MN_CHECK_ARG(sizes_out != nullptr, "sizes: null output");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  MN_CHECK_CUDA(cudaMemsetAsync(sizes_out, 0, sizeof(int32_t) * O, st));
  if (T == 0) return MN_OK;
  MN_CHECK_ARG(kernel_map != nullptr, "sizes: null kernel map");
  const int n_tiles = (int)div_up(T, kMTile);
  MN_LAUNCH("map_count_kernel", st,
            map_count_kernel<<<dim3(n_tiles, (unsigned)O), kMThreads, 0, st>>>(
                kernel_map, T, n_tiles, nullptr, sizes_out));
  return MN_OK;
}

extern "C" mn_status mn_compute_kernel_map_masks(const int32_t *kernel_map, int64_t O, int64_t S,
                                                 int64_t T, int32_t *source_masks_out,
                                                 int32_t *target_masks_out, void *ws_ptr,
                                                 size_t ws_bytes, void *stream) {
  MN_CHECK_ARG(O >= 0 && S >= 0 && T >= 0, "masks: bad shape");
  MN_CHECK_ARG(O <= MN_MAX_OFFSETS, "masks: %lld offsets (supported: up to %d)", (long long)O,
               MN_MAX_OFFSETS);
  if (O == 0) return MN_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (S > 0) {
    MN_CHECK_ARG(source_masks_out != nullptr, "masks: null source mask");
    MN_CHECK_CUDA(cudaMemsetAsync(source_masks_out, 0xff, sizeof(int32_t) * O * S, st));
  }
  if (T == 0) return MN_OK;
  MN_CHECK_ARG(kernel_map != nullptr && target_masks_out != nullptr, "masks: null pointer");
  Workspace ws(ws_ptr, ws_bytes);
  const int n_tiles = (int)div_up(T, kMTile);
  int32_t *counts = ws.take<int32_t>((size_t)O * n_tiles);
  MN_CHECK_WS(ws);
  MN_LAUNCH("map_count_kernel", st,
            map_count_kernel<<<dim3(n_tiles, (unsigned)O), kMThreads, 0, st>>>(
                kernel_map, T, n_tiles, counts, nullptr));
  MN_LAUNCH("scan_tiles_kernel", st, scan_tiles_kernel<<<(unsigned)O, 1024, 0, st>>>(counts, n_tiles));
  MN_LAUNCH("map_masks_kernel", st,
            map_masks_kernel<<<dim3(n_tiles, (unsigned)O), kMThreads, 0, st>>>(
                kernel_map, S, T, n_tiles, counts, source_masks_out, target_masks_out));
  return MN_OK;
}

extern "C" mn_status mn_build_kernel_map(const uint64_t *source_keys, int64_t S,
                                         const uint64_t *target_keys, int64_t T,
                                         const int32_t *offsets, int64_t O,
                                         const mn_keyspec *spec, int reorder,
                                         int32_t *source_masks_out, int32_t *target_masks_out,
                                         int32_t *order_out, int32_t *sizes_out,
                                         uint32_t *source_bits_out, uint32_t *target_bits_out,
                                         int32_t *sizes_host, int32_t *ctrl, void *ws_ptr,
                                         size_t ws_bytes, void *stream) {
  MN_CHECK_ARG(S >= 0 && T >= 0, "build_kernel_map: negative size");
  MN_CHECK_ARG(spec != nullptr, "build_kernel_map: null key spec");
  MN_CHECK_ARG(S < (1ll << 31) && T < (1ll << 31), "build_kernel_map: more than 2^31-1 rows");
  if (O > 32) {
    set_error("build_kernel_map: the fused build handles up to 32 offsets (got %lld); use "
              "mn_query_sorted_index_with_offsets + mn_compute_kernel_map_masks", (long long)O);
    return MN_ERR_UNSUPPORTED;
  }
  MN_CHECK_ARG(order_out != nullptr && sizes_out != nullptr && ctrl != nullptr,
               "build_kernel_map: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int ndim = spec->ndim;
  OffsetTable fwd;
  MN_RETURN_IF(make_offset_table(offsets, O, ndim, +1, spec, &fwd));

  if (T == 0 || S == 0) {
    // nothing can match: every mask entry is -1, every size 0
    if (S > 0) MN_CHECK_CUDA(cudaMemsetAsync(source_masks_out, 0xff, sizeof(int32_t) * O * S, st));
    if (T > 0) MN_CHECK_CUDA(cudaMemsetAsync(target_masks_out, 0xff, sizeof(int32_t) * O * T, st));
    if (S > 0 && source_bits_out != nullptr) MN_CHECK_CUDA(cudaMemsetAsync(source_bits_out, 0, sizeof(uint32_t) * S, st));
    if (T > 0 && target_bits_out != nullptr) MN_CHECK_CUDA(cudaMemsetAsync(target_bits_out, 0, sizeof(uint32_t) * T, st));
    MN_LAUNCH("identity_order_kernel", st,
              identity_order_kernel<<<1, MN_MAX_OFFSETS + 32, 0, st>>>((int)O, order_out, sizes_out, sizes_host, ctrl));
    return MN_OK;
  }
  MN_CHECK_ARG(source_keys != nullptr && target_keys != nullptr && source_masks_out != nullptr &&
                   target_masks_out != nullptr, "build_kernel_map: null pointer");

  // mirrored offset of every offset, if the table is symmetric
  bool symmetric = true;
  uint8_t neg[MN_MAX_OFFSETS] = {0};
  for (int64_t o = 0; o < O && symmetric; o++) {
    int found = -1;
    for (int64_t j = 0; j < O && found < 0; j++) {
      bool same = true;
      for (int k = 0; k < ndim; k++) same &= offsets[j * ndim + k] == -offsets[o * ndim + k];
      if (same) found = (int)j;
    }
    if (found < 0) symmetric = false; else neg[o] = (uint8_t)found;
  }
  const bool mirrored = symmetric && source_keys == target_keys && S == T;

  // grid of the cooperative emission kernel: every block resident at once
  static thread_local int coresident_for[kMaxDevices] = {0};
  int device = 0;
  MN_CHECK_CUDA(cudaGetDevice(&device));
  MN_CHECK_ARG(device >= 0 && device < kMaxDevices, "build_kernel_map: device index %d out of range", device);
  int &coresident = coresident_for[device];
  if (coresident == 0) {
    coresident = std::min(kMaxCoopBlocks, max_coresident_blocks(emit_masks_kernel, kEThreads, 0));
    if (coresident <= 0) {
      coresident = 0;
      set_error("build_kernel_map: cannot size the cooperative grid");
      return MN_ERR_CUDA;
    }
  }
  const int units_t = (int)div_up(T, kEUnit), units_s = (int)div_up(S, kEUnit);
  const int grid = (int)std::min<int64_t>(div_up((int64_t)units_t + units_s, 2), coresident);

  Workspace ws(ws_ptr, ws_bytes);
  uint32_t *words_t = ws.take<uint32_t>(T);
  uint32_t *words_s = mirrored ? words_t : ws.take<uint32_t>(S);
  int32_t *agg = ws.take<int32_t>((size_t)grid * 64);
  MN_CHECK_WS(ws);

  SearchArgs fwd_args;
  fill_search_args(&fwd_args, target_keys, T, source_keys, S, nullptr, words_t);
  if (mirrored) {
    MN_RETURN_IF(run_search(kBits, *spec, fwd_args, fwd, nullptr, nullptr, st));
  } else {
    // one search with the targets as rows; every hit also sets its bit in the word of the
    // source it found, so the source side needs no search of its own
    MN_CHECK_CUDA(cudaMemsetAsync(words_s, 0, sizeof(uint32_t) * S, st));
    fwd_args.table_words = words_s;
    MN_RETURN_IF(run_search(kBitsRev, *spec, fwd_args, fwd, nullptr, nullptr, st));
  }

  EmitArgs e{};
  e.words_t = words_t; e.words_s = words_s;
  e.target_masks = target_masks_out; e.source_masks = source_masks_out;
  e.order_out = order_out; e.sizes_out = sizes_out; e.sizes_host = sizes_host; e.agg = agg; e.ctrl = ctrl;
  e.bits_t = target_bits_out; e.bits_s = source_bits_out;
  e.T = T; e.S = S; e.units_t = units_t; e.units_s = units_s;
  e.num_offsets = (int)O; e.reorder = reorder ? 1 : 0;
  for (int64_t o = 0; o < O; o++) e.mirror[o] = mirrored ? neg[o] : (uint8_t)o;
  void *params[] = {&e};
  {
    LaunchScope scope("emit_masks_kernel", st);
    MN_CHECK_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void *>(emit_masks_kernel), dim3(grid),
                                              dim3(kEThreads), params, 0, st));
  }
  MN_CHECK_LAUNCH();
  return MN_OK;
}

#ifdef MN_PHASE_TIMING
// Debug build only: copies the phase marks of the last search (which = 0) or mask
// emission (which = 1) launch to the host (blocking).
extern "C" int mn_debug_marks_query(int which, long long *out, int count) {
  const size_t bytes = sizeof(long long) * (size_t)std::min(count, 2048 * 16);
  cudaError_t e = which == 0 ? cudaMemcpyFromSymbol(out, g_marks_search, bytes)
                             : cudaMemcpyFromSymbol(out, g_marks_emit, bytes);
  return e == cudaSuccess ? 0 : 1;
}
#endif
