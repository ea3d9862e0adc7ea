// Map step, part 1: radix sort of packed keys, unique, the fused target
// coordinate build of strided convolutions, and voxelisation.
//
// The reference sorts with cub::DeviceRadixSort::SortPairs over all 8*sizeof(key)
// bits (csrc/minuet/cuda/functions/arg_sort_coodrinates.cu:346-357) and removes
// duplicates with cub::DeviceScan + a compaction kernel
// (csrc/minuet/cuda/functions/unique_coordinates.cu:16-101).  Here the sort is a
// hand-written stable LSD radix sort that only visits the key bits the bounding
// box uses, and unique/compaction is one count + scan + compact pipeline that can
// also unpack keys back to coordinates.
#include "mn_sort.cuh"

#include <algorithm>
#include <climits>
#include <mutex>

namespace mn {

namespace {

// ---------------------------------------------------------------------------
// unique: count -> scan -> compact
// ---------------------------------------------------------------------------
constexpr int kUqThreads = 256;
constexpr int kUqItems = 8;
constexpr int kUqTile = kUqThreads * kUqItems;  // 2048 rows per block

struct RowsView {  // sorted coordinate rows
  const int32_t *coords;
  const int64_t *batch_dims;
  int num_clouds;
  int ndim;
  int64_t n;
  // true when row i closes a run: it differs from row i+1, is the last row, or
  // row i+1 opens a new cloud (unique_coordinates.cu:16-26, 57-70)
  __device__ __forceinline__ bool closes(int64_t i) const {
    if (i + 1 >= n) return true;
    bool same = true;
    for (int k = 0; k < ndim; k++) same &= coords[i * ndim + k] == coords[(i + 1) * ndim + k];
    if (!same) return true;
    if (batch_dims != nullptr) {
      int lo = 0, hi = num_clouds;  // is i+1 a cloud start?
      while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (batch_dims[mid] < i + 1) lo = mid + 1; else hi = mid;
      }
      if (batch_dims[lo] == i + 1) return true;
    }
    return false;
  }
};

template <typename View>
__global__ void __launch_bounds__(kUqThreads)
unique_count_kernel(const View v, uint32_t *__restrict__ block_counts) {
  const int64_t base = (int64_t)blockIdx.x * kUqTile + (int64_t)threadIdx.x * kUqItems;
  uint32_t c = 0;
#pragma unroll
  for (int j = 0; j < kUqItems; j++) {
    int64_t i = base + j;
    if (i < v.n && v.closes(i)) c++;
  }
  c = __reduce_add_sync(0xffffffffu, c);
  __shared__ uint32_t s[kUqThreads / 32];
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < kUqThreads / 32; w++) t += s[w];
    block_counts[blockIdx.x] = t;
  }
}

// Single block: exclusive scan of the block counts in place, total -> *total
// (and, when given, *total64).
__global__ void __launch_bounds__(1024)
scan_blocks_kernel(uint32_t *__restrict__ counts, int nblocks, uint32_t *__restrict__ total,
                   int64_t *__restrict__ total64) {
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_carry;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (int b0 = 0; b0 < nblocks; b0 += 1024) {
    const int b = b0 + threadIdx.x;
    const uint32_t v = b < nblocks ? counts[b] : 0u;
    uint32_t inc = v;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      uint32_t t = __shfl_up_sync(0xffffffffu, inc, s);
      if (lane >= s) inc += t;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = s_warp[lane], winc = w;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        uint32_t t = __shfl_up_sync(0xffffffffu, winc, s);
        if (lane >= s) winc += t;
      }
      s_warp[lane] = winc - w;
    }
    __syncthreads();
    const uint32_t carry = s_carry;
    if (b < nblocks) counts[b] = carry + s_warp[warp] + inc - v;
    __syncthreads();
    if (threadIdx.x == 1023) s_carry = carry + s_warp[warp] + inc;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *total = s_carry;
    if (total64 != nullptr) *total64 = s_carry;
  }
}

struct CoordSink {  // reference-API unique: rows + inclusive index array
  const int32_t *coords;
  int ndim;
  int32_t *out_rows;
  int64_t *indices;  // [n+1]
  __device__ __forceinline__ void index(int64_t i, uint32_t inclusive) const {
    indices[i + 1] = inclusive;
  }
  __device__ __forceinline__ void emit(int64_t i, uint32_t pos) const {
    for (int k = 0; k < ndim; k++) out_rows[(int64_t)pos * ndim + k] = coords[i * ndim + k];
  }
};

template <typename View, typename Sink>
__global__ void __launch_bounds__(kUqThreads)
unique_compact_kernel(const View v, const Sink sink, const uint32_t *__restrict__ block_offsets) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = (int64_t)blockIdx.x * kUqTile + (int64_t)threadIdx.x * kUqItems;
  bool flag[kUqItems];
  uint32_t c = 0;
#pragma unroll
  for (int j = 0; j < kUqItems; j++) {
    int64_t i = base + j;
    flag[j] = i < v.n && v.closes(i);
    c += flag[j];
  }
  uint32_t inc = c;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    uint32_t t = __shfl_up_sync(0xffffffffu, inc, s);
    if (lane >= s) inc += t;
  }
  __shared__ uint32_t s_warp[kUqThreads / 32];
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  uint32_t run = block_offsets[blockIdx.x] + inc - c;
  for (int w = 0; w < warp; w++) run += s_warp[w];
#pragma unroll
  for (int j = 0; j < kUqItems; j++) {
    int64_t i = base + j;
    if (i < v.n) {
      if (flag[j]) sink.emit(i, run);
      run += flag[j];
      sink.index(i, run);
    }
  }
}

// ---------------------------------------------------------------------------
// unique over sorted keys (strided target coordinates): one cooperative kernel
// ---------------------------------------------------------------------------
// Every block owns a contiguous chunk of the sorted keys.  It counts the keys
// that open a run (differ from their predecessor), a grid barrier later sums
// the counts of the blocks before it, and walks the chunk again: every opening
// key goes to its rank in keys_out, is unpacked into a coordinate row, and, when
// it is the first key of its cloud, fills the cloud-start table.  The count,
// the cloud starts and a copy of the status word land in one int64 block
// (meta), so that the host needs a single small read.
constexpr int kUkThreads = 1024;
constexpr int kUkMaxBlocks = 256;                 // workspace sizing
constexpr int kUkWarps = kUkThreads / 32;

struct UniqueKeysArgs {
  const uint64_t *keys[2];           // sorted keys are in keys[*which] (which may be NULL: keys[0])
  const int32_t *which;
  int64_t n;
  SpecRef spec;
  uint64_t *keys_out;                // [n]
  int32_t *rows_out;                 // [n, ndim]
  int64_t *meta;                     // [num_clouds + 4]: count, cloud starts [num_clouds + 1], status, key bits
  int64_t *meta_host;                // the same in host memory, or NULL
  int32_t num_clouds;
  uint32_t *block_counts;            // workspace [grid]
  int32_t *ctrl;
  int32_t index_bits;                // low key bits that hold the row of the unsorted input
  int32_t *run_start;                // optional [n]: sorted position of every run's first key
  int64_t *inverse;                  // optional [n]: run of every row of the unsorted input
};

constexpr int kUkRounds = 8;                          // keys per thread and step
constexpr int kUkStep = kUkThreads * kUkRounds;       // 8192 keys per block and step

__global__ void __launch_bounds__(kUkThreads, 1)
unique_keys_kernel(const __grid_constant__ UniqueKeysArgs a) {
  release_successor();
  __shared__ uint32_t s_cnt[kUkRounds][kUkWarps];     // openers per (round, warp), then their prefix
  __shared__ uint32_t s_before, s_total, s_step_total;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = (int)gridDim.x, b = (int)blockIdx.x;
  const unsigned lt = (1u << lane) - 1u;
  const mn_keyspec &spec = spec_of(a.spec);
  const int ib = a.index_bits;
  const uint64_t index_mask = (1ull << ib) - 1ull;
  const uint64_t *keys = a.keys[a.which != nullptr ? (*a.which & 1) : 0];
  const int64_t per_block = ((a.n + G - 1) / G + kUkThreads - 1) / kUkThreads * kUkThreads;
  const int64_t c0 = min(a.n, (int64_t)b * per_block), c1 = min(a.n, c0 + per_block);

  // ---- count the run openers of this chunk (a key opens a run when it differs from
  // its predecessor); all loads of a step are issued before any is used -------------
  uint32_t mine = 0;
  for (int64_t s0 = c0; s0 < c1; s0 += kUkStep) {
    uint64_t k[kUkRounds], pk[kUkRounds];
#pragma unroll
    for (int j = 0; j < kUkRounds; j++) {
      const int64_t i = s0 + j * kUkThreads + tid;
      k[j] = i < c1 ? __ldcg(keys + i) : 0ull;
      pk[j] = (i < c1 && i > 0) ? __ldcg(keys + i - 1) : 0ull;
    }
#pragma unroll
    for (int j = 0; j < kUkRounds; j++) {
      const int64_t i = s0 + j * kUkThreads + tid;
      mine += (i < c1 && (i == 0 || (k[j] >> ib) != (pk[j] >> ib))) ? 1u : 0u;
    }
  }
  mine = __reduce_add_sync(0xffffffffu, mine);
  if (lane == 0) s_cnt[0][warp] = mine;
  __syncthreads();
  if (tid == 0) {
    uint32_t t = 0;
    for (int w = 0; w < kUkWarps; w++) t += s_cnt[0][w];
    a.block_counts[b] = t;
  }
  grid_barrier(a.ctrl, (unsigned)G);
  if (warp == 0) {
    uint32_t before = 0, all = 0;
    for (int bb = lane; bb < G; bb += 32) {
      const uint32_t v = __ldcg(a.block_counts + bb);
      all += v;
      if (bb < b) before += v;
    }
    before = __reduce_add_sync(0xffffffffu, before);
    all = __reduce_add_sync(0xffffffffu, all);
    if (lane == 0) { s_before = before; s_total = all; }
  }
  __syncthreads();
  uint32_t run = s_before;
  const uint32_t total = s_total;
  auto put_meta = [&](int64_t i, int64_t v) {
    a.meta[i] = v;
    if (a.meta_host != nullptr) a.meta_host[i] = v;   // a posted write; it lands before the launch has ended
  };

  // ---- compact, unpack, cloud starts ----------------------------------------------
  for (int64_t s0 = c0; s0 < c1; s0 += kUkStep) {
    uint64_t k[kUkRounds], pk[kUkRounds];
    unsigned votes[kUkRounds];
#pragma unroll
    for (int j = 0; j < kUkRounds; j++) {
      const int64_t i = s0 + j * kUkThreads + tid;
      k[j] = i < c1 ? __ldcg(keys + i) : 0ull;
      pk[j] = (i < c1 && i > 0) ? __ldcg(keys + i - 1) : 0ull;
    }
    __syncthreads();   // the prefix table of the previous step has been read
#pragma unroll
    for (int j = 0; j < kUkRounds; j++) {
      const int64_t i = s0 + j * kUkThreads + tid;
      const bool opens = i < c1 && (i == 0 || (k[j] >> ib) != (pk[j] >> ib));
      votes[j] = __ballot_sync(0xffffffffu, opens);
      if (lane == 0) s_cnt[j][warp] = __popc(votes[j]);
    }
    __syncthreads();
    if (warp == 0) {
      // exclusive prefix over the kUkRounds * kUkWarps counts, in (round, warp) order
      uint32_t v[kUkRounds], sum = 0;
#pragma unroll
      for (int j = 0; j < kUkRounds; j++) { v[j] = (&s_cnt[0][0])[lane * kUkRounds + j]; sum += v[j]; }
      uint32_t inc = sum;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, inc, s);
        if (lane >= s) inc += t;
      }
      uint32_t r = inc - sum;
#pragma unroll
      for (int j = 0; j < kUkRounds; j++) { (&s_cnt[0][0])[lane * kUkRounds + j] = r; r += v[j]; }
      if (lane == 31) s_step_total = inc;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kUkRounds; j++) {
      const int64_t i = s0 + j * kUkThreads + tid;
      const uint32_t pos = run + s_cnt[j][warp] + __popc(votes[j] & lt);   // openers before key i
      const bool opens = ((votes[j] >> lane) & 1u) != 0u;
      if (a.inverse != nullptr && i < c1)
        a.inverse[rsort::index_of(k[j], index_mask, a.n)] = (int64_t)(opens ? pos : pos - 1u);
      if (opens) {
        const uint64_t key = k[j] >> ib;
        if (a.keys_out != nullptr) a.keys_out[pos] = key;
        if (a.run_start != nullptr) a.run_start[pos] = (int32_t)i;
        for (int d = 0; d < spec.ndim; d++) {
          const uint64_t f = (key >> spec.shift[d]) & ((1ull << spec.bits[d]) - 1ull);
          a.rows_out[(int64_t)pos * spec.ndim + d] = (int32_t)((int64_t)f + spec.base[d]);
        }
        // first key of cloud c: every cloud after the previous key's cloud starts here
        const int64_t c_here = (int64_t)(key >> spec.cloud_shift);
        const int64_t c_prev = i == 0 ? -1 : (int64_t)(pk[j] >> ib >> spec.cloud_shift);
        for (int64_t g = c_prev + 1; g <= c_here && g <= a.num_clouds; g++) put_meta(1 + g, pos);
      }
    }
    run += s_step_total;
  }
  if (b == 0 && tid == 0) {
    put_meta(0, total);
    const int64_t c_last = a.n > 0 ? (int64_t)(__ldcg(keys + a.n - 1) >> ib >> spec.cloud_shift) : -1;
    for (int64_t g = c_last + 1; g <= a.num_clouds; g++) put_meta(1 + g, total);
    put_meta(a.num_clouds + 2, a.ctrl[MN_CTRL_STATUS]);
    put_meta(a.num_clouds + 3, spec.total_bits);
  }
}

__global__ void zero_index0_kernel(int64_t *indices) { indices[0] = 0; }

}  // namespace

namespace {

// Grid of a cooperative kernel with one 1024-thread block per SM, cached per device.
template <typename Kernel>
mn_status coop_grid_1024(Kernel kernel, size_t smem, int *cache, int *out) {
  int device = 0;
  MN_CHECK_CUDA(cudaGetDevice(&device));
  MN_CHECK_ARG(device >= 0 && device < kMaxDevices, "device index %d out of range", device);
  if (cache[device] == 0) {
    if (smem > 48 * 1024)
      MN_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    cache[device] = std::min(kUkMaxBlocks, max_coresident_blocks(kernel, 1024, smem));
    if (cache[device] <= 0) {
      cache[device] = 0;
      set_error("cannot size a cooperative grid on device %d", device);
      return MN_ERR_CUDA;
    }
  }
  *out = cache[device];
  return MN_OK;
}

CoordKeys make_coord_keys(const SortSource &source, const mn_keyspec &spec, int32_t *status) {
  CoordKeys k{};
  k.coords = source.coords;
  k.batch_dims = source.batch_dims;
  k.ndim = source.ndim;
  k.num_clouds = source.batch_dims != nullptr ? (int)source.num_clouds : 1;
  k.status = status;
  k.pack.spec = make_spec_ref(spec);
  for (int d = 0; d < 4; d++) k.pack.tstride[d] = 1;
  for (int d = 0; d < source.ndim; d++) {
    k.pack.tstride[d] = source.tstride != nullptr ? source.tstride[d] : 1;
    if (k.pack.tstride[d] != 1) k.pack.has_stride = 1;
  }
  return k;
}

mn_status launch_unique_keys(const UniqueKeysArgs &args, cudaStream_t st) {
  static thread_local int grid_cache[kMaxDevices] = {0};
  int coresident = 0;
  MN_RETURN_IF(coop_grid_1024(unique_keys_kernel, 0, grid_cache, &coresident));
  const int grid = (int)std::min<int64_t>(coresident, std::max<int64_t>(1, div_up(args.n, kUkStep / 4)));
  UniqueKeysArgs a = args;
  void *params[] = {&a};
  {
    LaunchScope scope("unique_keys_kernel", st);
    MN_CHECK_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<void *>(unique_keys_kernel), dim3(grid),
                                              dim3(kUkThreads), params, 0, st));
  }
  MN_CHECK_LAUNCH();
  return MN_OK;
}

}  // namespace

}  // namespace mn

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
using namespace mn;

extern "C" mn_status mn_arg_sort_coordinates(const int32_t *coords, int64_t n, int ndim,
                                             const int64_t *batch_dims, int64_t num_clouds,
                                             const mn_keyspec *spec, int64_t *index_out,
                                             int32_t *status_dev, void *ws_ptr,
                                             size_t ws_bytes, void *stream) {
  MN_CHECK_ARG(n >= 0 && ndim >= 1 && ndim <= MN_MAX_NDIM, "arg_sort: bad n/ndim");
  MN_CHECK_ARG(spec != nullptr && spec->ndim == ndim, "arg_sort: key spec missing or of another ndim");
  if (n == 0) return MN_OK;
  MN_CHECK_ARG(coords != nullptr && index_out != nullptr && status_dev != nullptr,
               "arg_sort: null pointer");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  Workspace ws(ws_ptr, ws_bytes);
  uint64_t *keys = ws.take<uint64_t>(n), *keys_tmp = ws.take<uint64_t>(n);
  int32_t *vals = ws.take<int32_t>(n), *vals_tmp = ws.take<int32_t>(n);
  MN_CHECK_WS(ws);
  MN_CHECK_ARG(spec->device_copy == nullptr, "arg_sort: needs a key spec whose layout is known on the host");
  rsort::Args a{};
  a.keys[0] = keys; a.keys[1] = keys_tmp;
  a.n = n;
  a.bits = spec->total_bits;
  a.spec = make_spec_ref(*spec);
  a.status = status_dev;
  a.index64 = index_out;
  CoordKeys k = make_coord_keys(SortSource{coords, batch_dims, num_clouds, ndim, nullptr}, *spec, status_dev);
  if (spec->total_bits + rsort::bits_for(n) <= 64) {
    a.first_bit = k.index_bits = rsort::bits_for(n);
  } else {
    a.vals[0] = vals; a.vals[1] = vals_tmp;    // the index does not fit below the key
  }
  return rsort::run(a, k, ws, st);
}

namespace mn {
struct GivenKeys {
  const uint64_t *keys;
  int32_t index_bits;
  __device__ __forceinline__ int layout() const { return 0; }
  __device__ __forceinline__ uint64_t operator()(int64_t i, int, int &) const {
    return (__ldg(keys + i) << index_bits) | (uint64_t)i;
  }
};
}  // namespace mn

extern "C" mn_status mn_arg_sort_keys(const uint64_t *keys_in, int64_t n, int bits, uint32_t wait_limit,
                                      int64_t *index_out, int32_t *status_dev, void *ws_ptr, size_t ws_bytes,
                                      void *stream) {
  MN_CHECK_ARG(n >= 0 && n < (1ll << 31) - 1, "arg_sort_keys: bad n");
  if (n == 0) return MN_OK;
  MN_CHECK_ARG(bits >= 1 && bits + rsort::bits_for(n) <= 64, "arg_sort_keys: the index does not fit below the key");
  MN_CHECK_ARG(keys_in != nullptr && index_out != nullptr && status_dev != nullptr, "arg_sort_keys: null pointer");
  Workspace ws(ws_ptr, ws_bytes);
  rsort::Args a{};
  a.keys[0] = ws.take<uint64_t>(n);
  a.keys[1] = ws.take<uint64_t>(n);
  MN_CHECK_WS(ws);
  a.n = n;
  a.first_bit = rsort::bits_for(n);
  a.bits = bits;
  a.wait_limit = wait_limit;
  a.status = status_dev;
  a.index64 = index_out;
  return rsort::run(a, GivenKeys{keys_in, a.first_bit}, ws, static_cast<cudaStream_t>(stream));
}

extern "C" mn_status mn_arg_sort_coordinates_by_dimension(
    const int32_t *coords, int64_t n, int ndim, const int64_t *batch_dims, int64_t num_clouds,
    int64_t *index_out, int32_t *ctrl, void *ws_ptr, size_t ws_bytes, void *stream) {
  MN_CHECK_ARG(n >= 0 && n < (1ll << 31) && ndim >= 1 && ndim <= MN_MAX_NDIM,
               "arg_sort_by_dimension: bad n/ndim");
  if (n == 0) return MN_OK;
  MN_CHECK_ARG(coords != nullptr && index_out != nullptr && ctrl != nullptr,
               "arg_sort_by_dimension: null pointer");
  if (batch_dims == nullptr) num_clouds = 1;
  MN_CHECK_ARG(num_clouds >= 1 && num_clouds < (1ll << 31), "arg_sort_by_dimension: bad num_clouds");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  Workspace ws(ws_ptr, ws_bytes);
  uint64_t *keys[2] = {ws.take<uint64_t>(n), ws.take<uint64_t>(n)};
  int32_t *perm[2] = {ws.take<int32_t>(n), ws.take<int32_t>(n)};
  MN_CHECK_WS(ws);
  const size_t fixed = ws.used;
  int cur = -1;           // perm[cur] holds the current permutation (after the first pass)
  // least significant key first: last dimension ... dimension 0, then the cloud
  const int last_dim = num_clouds > 1 ? -1 : 0;
  for (int dim = ndim - 1; dim >= last_dim; dim--) {
    rsort::Args a{};
    a.keys[0] = keys[0]; a.keys[1] = keys[1];
    a.n = n;
    a.first_bit = rsort::bits_for(n);
    a.bits = dim < 0 ? rsort::bits_for(num_clouds) : 32;
    a.status = ctrl;
    const int next = cur == 0 ? 1 : 0;
    if (dim == last_dim) a.index64 = index_out; else a.index32 = perm[next];
    Workspace sub(static_cast<char *>(ws_ptr) + fixed, ws_bytes - fixed);
    MN_RETURN_IF(rsort::run(a, DimensionKeys{coords, cur < 0 ? nullptr : perm[cur], batch_dims, ndim, dim,
                                             (int)num_clouds, a.first_bit}, sub, st));
    cur = next;
  }
  return MN_OK;
}

extern "C" mn_status mn_unique_coordinates(const int32_t *coords, int64_t n, int ndim,
                                           const int64_t *batch_dims, int64_t num_clouds,
                                           int32_t *unique_out, int64_t *indices_out,
                                           void *ws_ptr, size_t ws_bytes, void *stream) {
  MN_CHECK_ARG(n >= 0 && ndim >= 1 && ndim <= MN_MAX_NDIM, "unique: bad n/ndim");
  MN_CHECK_ARG(indices_out != nullptr, "unique: null indices");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  MN_LAUNCH("zero_index0_kernel", st, zero_index0_kernel<<<1, 1, 0, st>>>(indices_out));
  if (n == 0) return MN_OK;
  MN_CHECK_ARG(coords != nullptr && unique_out != nullptr, "unique: null pointer");
  MN_CHECK_ARG(n < (1ll << 31), "unique: n exceeds 2^31-1");
  Workspace ws(ws_ptr, ws_bytes);
  const int nblocks = (int)div_up(n, kUqTile);
  uint32_t *counts = ws.take<uint32_t>(nblocks);
  uint32_t *total = ws.take<uint32_t>(1);
  MN_CHECK_WS(ws);
  RowsView view{coords, batch_dims, batch_dims ? (int)num_clouds : 1, ndim, n};
  CoordSink sink{coords, ndim, unique_out, indices_out};
  MN_LAUNCH("unique_count_kernel", st, unique_count_kernel<RowsView><<<nblocks, kUqThreads, 0, st>>>(view, counts));
  MN_LAUNCH("scan_blocks_kernel", st, scan_blocks_kernel<<<1, 1024, 0, st>>>(counts, nblocks, total, nullptr));
  MN_LAUNCH("unique_compact_kernel", st, unique_compact_kernel<RowsView, CoordSink><<<nblocks, kUqThreads, 0, st>>>(view, sink, counts));
  return MN_OK;
}

extern "C" mn_status mn_downsample_coordinates(
    const int32_t *coords, int64_t n, int ndim, const int64_t *batch_dims, int64_t num_clouds,
    const int32_t *tstride, const mn_keyspec *spec, int32_t *unique_out, uint64_t *keys_out,
    int64_t *meta_out, int64_t *meta_host, int32_t *ctrl, void *ws_ptr, size_t ws_bytes, void *stream) {
  MN_CHECK_ARG(n >= 0 && ndim >= 1 && ndim <= MN_MAX_NDIM, "downsample: bad n/ndim");
  MN_CHECK_ARG(spec != nullptr && spec->ndim == ndim, "downsample: key spec missing or of another ndim");
  MN_CHECK_ARG(tstride != nullptr && meta_out != nullptr && ctrl != nullptr, "downsample: null pointer");
  MN_CHECK_ARG(n < (1ll << 31), "downsample: n exceeds 2^31-1");
  if (batch_dims == nullptr) num_clouds = 1;
  MN_CHECK_ARG(num_clouds >= 1, "downsample: num_clouds must be >= 1");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  MN_CHECK_ARG(n == 0 || (coords != nullptr && unique_out != nullptr && keys_out != nullptr),
               "downsample: null pointer");
  for (int k = 0; k < ndim; k++)
    MN_CHECK_ARG(tstride[k] >= 1 && tstride[k] - 1 <= spec->margin,
                 "downsample: stride %d needs a key margin >= %d (have %d)", tstride[k],
                 tstride[k] - 1, spec->margin);
  Workspace ws(ws_ptr, ws_bytes);
  uint64_t *keys = ws.take<uint64_t>(std::max<int64_t>(n, 1)), *keys_tmp = ws.take<uint64_t>(std::max<int64_t>(n, 1));
  int32_t *which = ws.take<int32_t>(1);
  uint32_t *block_counts = ws.take<uint32_t>(kUkMaxBlocks);
  MN_CHECK_WS(ws);
  if (n > 0) {
    rsort::Args sort{};
    sort.keys[0] = keys; sort.keys[1] = keys_tmp;
    sort.n = n;
    sort.bits = spec->total_bits > 0 ? spec->total_bits : -1;   // -1: a layout that only the device knows
    sort.spec = make_spec_ref(*spec);
    sort.result_in_second = which;
    sort.status = ctrl + MN_CTRL_STATUS;
    MN_RETURN_IF(rsort::run(sort, make_coord_keys(SortSource{coords, batch_dims, num_clouds, ndim, tstride}, *spec,
                                                  ctrl + MN_CTRL_STATUS), ws, st));
  }
  UniqueKeysArgs a{};
  a.keys[0] = keys; a.keys[1] = keys_tmp;
  a.which = n > 0 ? which : nullptr;
  a.n = n;
  a.spec = make_spec_ref(*spec);
  a.keys_out = keys_out;
  a.rows_out = unique_out;
  a.meta = meta_out;
  a.meta_host = meta_host;
  a.num_clouds = (int)num_clouds;
  a.block_counts = block_counts;
  a.ctrl = ctrl;
  return launch_unique_keys(a, st);
}

// ---------------------------------------------------------------------------
// voxelisation
// ---------------------------------------------------------------------------
// Box of the points' voxels -> keys with the point's index in their low bits -> sort -> unique ->
// means of the runs: one read of the number of voxels by the host at the end.  The steps one by
// one (library floor and division, arg sort, row gather, unique, mean; two host reads) took 235 us
// for a scan of 120 000 points and 865 us for two million indoor points, of which 360 us were a
// mean kernel with a warp per point.
namespace mn {

constexpr int kVbThreads = 256;

// Bounding box of the points' voxels and the key layout: every block leaves its box, the last one
// to arrive reduces them and writes the layout.  The ticket wraps back to zero by itself.
template <typename F>
__global__ void __launch_bounds__(kVbThreads)
voxel_box_kernel(const __grid_constant__ VoxelPoints<F> voxel, int64_t n, int64_t num_clouds,
                 int32_t *__restrict__ partial, uint32_t *ticket, mn_keyspec *spec_out) {
  int lo[4] = {INT_MAX, INT_MAX, INT_MAX, INT_MAX}, hi[4] = {INT_MIN, INT_MIN, INT_MIN, INT_MIN};
  const int64_t gsz = (int64_t)gridDim.x * kVbThreads;
#pragma unroll 4
  for (int64_t r = (int64_t)blockIdx.x * kVbThreads + threadIdx.x; r < n; r += gsz) {
    int c[4];
    voxel(r, c);
#pragma unroll
    for (int k = 0; k < 4; k++) { lo[k] = min(lo[k], c[k]); hi[k] = max(hi[k], c[k]); }
  }
  __shared__ int s_box[kVbThreads / 32][8];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto reduce = [&]() {         // the block's box in s_box[0]
#pragma unroll
    for (int k = 0; k < 4; k++) {
      lo[k] = __reduce_min_sync(0xffffffffu, lo[k]);
      hi[k] = __reduce_max_sync(0xffffffffu, hi[k]);
    }
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < 4; k++) { s_box[warp][k] = lo[k]; s_box[warp][4 + k] = hi[k]; }
    }
    __syncthreads();
    if (threadIdx.x < 8) {
      int v = s_box[0][threadIdx.x];
      for (int w = 1; w < kVbThreads / 32; w++)
        v = threadIdx.x < 4 ? min(v, s_box[w][threadIdx.x]) : max(v, s_box[w][threadIdx.x]);
      s_box[0][threadIdx.x] = v;
    }
    __syncthreads();
  };
  reduce();
  if (threadIdx.x < 8) partial[blockIdx.x * 8 + threadIdx.x] = s_box[0][threadIdx.x];
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
#pragma unroll
  for (int k = 0; k < 4; k++) { lo[k] = INT_MAX; hi[k] = INT_MIN; }
  for (int b = threadIdx.x; b < (int)gridDim.x; b += kVbThreads) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      lo[k] = min(lo[k], __ldcg(partial + b * 8 + k));
      hi[k] = max(hi[k], __ldcg(partial + b * 8 + 4 + k));
    }
  }
  reduce();
  if (threadIdx.x == 0) {
    mn_keyspec spec;
    compute_keyspec(s_box[0], voxel.ndim, num_clouds, 0, &spec);
    *spec_out = spec;
  }
}

template <typename T> __device__ __forceinline__ float vm_to_f32(T v);
template <> __device__ __forceinline__ float vm_to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float vm_to_f32<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float vm_to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T vm_from_f32(float v);
template <> __device__ __forceinline__ float vm_from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __half vm_from_f32<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 vm_from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// out[u] = mean of the feature rows of the points of run u, added in sorted order in fp32.
// `lanes` lanes share a voxel and take four consecutive channels each: a voxel holds one or two
// points of a few channels, so a warp per voxel would leave most lanes idle.
template <typename T>
__global__ void __launch_bounds__(256)
voxel_run_mean_kernel(const T *__restrict__ features, int channels, int lanes, const uint64_t *keys0,
                      const uint64_t *keys1, const int32_t *which, int index_bits,
                      const int32_t *__restrict__ run_start, const int64_t *__restrict__ meta, int64_t n,
                      T *__restrict__ out) {
  begin_early();
  const int64_t count = __ldg(meta);
  const uint64_t *keys = (*which & 1) ? keys1 : keys0;
  const uint64_t mask = (1ull << index_bits) - 1ull;
  const int64_t groups = (int64_t)gridDim.x * (256 / lanes);
  const int part = threadIdx.x % lanes;
  for (int64_t u = (int64_t)blockIdx.x * (256 / lanes) + threadIdx.x / lanes; u < count; u += groups) {
    const int64_t begin = __ldg(run_start + u);
    const int64_t end = u + 1 < count ? (int64_t)__ldg(run_start + u + 1) : n;
    const float inv = 1.0f / (float)(end - begin);
    for (int c0 = part * 4; c0 < channels; c0 += lanes * 4) {
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      for (int64_t j = begin; j < end; j++) {
        const T *row = features + (int64_t)rsort::index_of(__ldg(keys + j), mask, n) * channels + c0;
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (c0 + k < channels) acc[k] += vm_to_f32<T>(row[k]);
      }
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (c0 + k < channels) out[u * channels + c0 + k] = vm_from_f32<T>(acc[k] * inv);
    }
  }
}

namespace {

struct Runs {                 // sorted keys and the runs found in them
  uint64_t *keys, *keys_tmp;
  int32_t *which, *run_start;
  const int64_t *meta;
  int64_t n;
  int index_bits;
};

template <typename T>
mn_status run_mean(const void *features, int64_t channels, const Runs &r, void *out, cudaStream_t st) {
  int lanes = 1;
  while (lanes < 32 && lanes * 4 < channels) lanes *= 2;
  const int blocks = (int)std::min<int64_t>(kNumSMs * 32, div_up(r.n, 256 / lanes));
  MN_LAUNCH("voxel_run_mean_kernel", st,
            launch_early(voxel_run_mean_kernel<T>, blocks, 256, 0, st, static_cast<const T *>(features), (int)channels, lanes,
                                                             r.keys, r.keys_tmp, r.which, r.index_bits, r.run_start,
                                                             r.meta, r.n, static_cast<T *>(out)));
  return MN_OK;
}

template <typename F>
mn_status run_voxelize(const F *points, int64_t n, int ndim, const double *voxel_size, const int64_t *batch_dims,
                       int64_t num_clouds, const void *features, int64_t channels, mn_dtype dtype,
                       int32_t *voxels_out, int64_t *inverse_out, void *means_out, int64_t *meta_out,
                       int64_t *meta_host, cudaEvent_t meta_event, int32_t *ctrl, Workspace &ws, cudaStream_t st) {
  Runs r{};
  r.keys = ws.take<uint64_t>(n);
  r.keys_tmp = ws.take<uint64_t>(n);
  r.run_start = ws.take<int32_t>(n);
  r.which = ws.take<int32_t>(1);
  r.meta = meta_out;
  r.n = n;
  r.index_bits = rsort::bits_for(n);
  const int blocks = (int)std::min<int64_t>(kNumSMs * 4, div_up(n, kVbThreads));
  int32_t *partial = ws.take<int32_t>((size_t)blocks * 8);
  mn_keyspec *spec_dev = ws.take<mn_keyspec>(1);
  uint32_t *block_counts = ws.take<uint32_t>(kUkMaxBlocks);
  MN_CHECK_WS(ws);
  VoxelPoints<F> voxel{};
  voxel.points = points;
  voxel.ndim = ndim;
  for (int k = 0; k < 4; k++) voxel.size[k] = (F)(k < ndim ? voxel_size[k] : 1.0);
  MN_LAUNCH("voxel_box_kernel", st,
            voxel_box_kernel<F><<<blocks, kVbThreads, 0, st>>>(
                voxel, n, num_clouds, partial, reinterpret_cast<uint32_t *>(ctrl) + MN_CTRL_TICKET, spec_dev));
  mn_keyspec spec{};
  spec.ndim = ndim;
  spec.device_copy = spec_dev;
  rsort::Args sort{};
  sort.keys[0] = r.keys; sort.keys[1] = r.keys_tmp;
  sort.n = n;
  sort.first_bit = r.index_bits;
  sort.bits = -1;
  sort.spec = make_spec_ref(spec);
  sort.result_in_second = r.which;
  sort.status = ctrl + MN_CTRL_STATUS;
  VoxelKeys<F> source{};
  source.voxel = voxel;
  source.batch_dims = batch_dims;
  source.num_clouds = batch_dims != nullptr ? (int)num_clouds : 1;
  source.index_bits = r.index_bits;
  source.pack.spec = sort.spec;
  for (int k = 0; k < 4; k++) source.pack.tstride[k] = 1;
  MN_RETURN_IF(rsort::run(sort, source, ws, st));
  UniqueKeysArgs u{};
  u.keys[0] = r.keys; u.keys[1] = r.keys_tmp;
  u.which = r.which;
  u.n = n;
  u.spec = sort.spec;
  u.rows_out = voxels_out;
  u.meta = meta_out;
  u.meta_host = meta_host;
  u.num_clouds = (int)num_clouds;
  u.block_counts = block_counts;
  u.ctrl = ctrl;
  u.index_bits = r.index_bits;
  u.run_start = r.run_start;
  u.inverse = inverse_out;
  MN_RETURN_IF(launch_unique_keys(u, st));
  // the host goes on with the number of voxels while their means are still made
  if (meta_event != nullptr) MN_CHECK_CUDA(cudaEventRecord(meta_event, st));
  if (features == nullptr) return MN_OK;
  switch (dtype) {
    case MN_F32: return run_mean<float>(features, channels, r, means_out, st);
    case MN_F16: return run_mean<__half>(features, channels, r, means_out, st);
    default: return run_mean<__nv_bfloat16>(features, channels, r, means_out, st);
  }
}

}  // namespace
}  // namespace mn

extern "C" size_t mn_voxelize_workspace_bytes(int64_t n) {
  const size_t m = (size_t)std::max<int64_t>(n, 1);
  return 2 * align_up(m * 8, 256) + align_up(m * 4, 256) + rsort::workspace_bytes(n) +
         align_up((size_t)kNumSMs * 4 * 32, 256) + 8192;
}

extern "C" mn_status mn_voxelize(const void *points, int points_are_double, int64_t n, int ndim,
                                 const double *voxel_size, const int64_t *batch_dims, int64_t num_clouds,
                                 const void *features, int64_t channels, mn_dtype dtype, int32_t *voxels_out,
                                 int64_t *inverse_out, void *means_out, int64_t *meta_out, int64_t *meta_host,
                                 void *meta_event, int32_t *ctrl, void *ws_ptr, size_t ws_bytes, void *stream) {
  MN_CHECK_ARG(n >= 1 && n < (1ll << 31) - 1 && ndim >= 1 && ndim <= MN_MAX_NDIM, "voxelize: bad n/ndim");
  if (batch_dims == nullptr) num_clouds = 1;
  MN_CHECK_ARG(num_clouds >= 1 && num_clouds < (1ll << 31), "voxelize: bad num_clouds");
  MN_CHECK_ARG(points != nullptr && voxel_size != nullptr && voxels_out != nullptr && meta_out != nullptr && ctrl != nullptr,
               "voxelize: null pointer");
  MN_CHECK_ARG(features == nullptr || (means_out != nullptr && channels >= 1 && channels < (1 << 20) &&
                                       (dtype == MN_F32 || dtype == MN_F16 || dtype == MN_BF16)),
               "voxelize: bad features");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  Workspace ws(ws_ptr, ws_bytes);
  if (points_are_double)
    return run_voxelize(static_cast<const double *>(points), n, ndim, voxel_size, batch_dims, num_clouds, features,
                        channels, dtype, voxels_out, inverse_out, means_out, meta_out, meta_host,
                        static_cast<cudaEvent_t>(meta_event), ctrl, ws, st);
  return run_voxelize(static_cast<const float *>(points), n, ndim, voxel_size, batch_dims, num_clouds, features,
                      channels, dtype, voxels_out, inverse_out, means_out, meta_out, meta_host,
                      static_cast<cudaEvent_t>(meta_event), ctrl, ws, st);
}

// ---------------------------------------------------------------------------
// Allocation-free variant of mn_unique_coordinates
// ---------------------------------------------------------------------------
// Some hosts may not allocate device memory at the point where they need this
// op: code running inside a CUDA stream capture or under a framework that
// forbids allocator calls on its hot path, plugins handed a fixed memory
// budget at load time, or real-time loops that must not touch the driver's
// allocator.  For them the block counts and the total live in a fixed array
// inside the library image.  Every GPU that loads the library carries these
// 33 KB until the process exits.
namespace {
constexpr int64_t kStaticUniqueMaxRows = 16ll << 20;  // 16 Mi rows per call
constexpr int kStaticUniqueBlocks = (int)(kStaticUniqueMaxRows / kUqTile);  // 8192 block counts
constexpr int kStaticUniqueWords = kStaticUniqueBlocks + 64;                // + the total
}  // namespace

static __device__ __align__(256) uint32_t g_unique_scratch[kStaticUniqueWords];

// In host code `g_unique_scratch` is only a handle for the symbol, not a device
// address, so the address is looked up once per device (with that device
// current) and cached here.
static uint32_t *g_unique_scratch_addr[kMaxDevices] = {nullptr};
static std::mutex g_unique_scratch_mutex;

static mn_status unique_scratch_address(uint32_t **out) {
  int device = -1;
  MN_CHECK_CUDA(cudaGetDevice(&device));
  MN_CHECK_ARG(device >= 0 && device < kMaxDevices, "unique_static: device index %d out of range",
               device);
  std::lock_guard<std::mutex> lock(g_unique_scratch_mutex);
  if (g_unique_scratch_addr[device] == nullptr) {
    uint32_t *p = nullptr;
    MN_CHECK_CUDA(cudaGetSymbolAddress((void **)&p, g_unique_scratch));
    g_unique_scratch_addr[device] = p;
  }
  *out = g_unique_scratch_addr[device];
  return MN_OK;
}

extern "C" mn_status mn_unique_coordinates_static(const int32_t *coords, int64_t n, int ndim,
                                                  const int64_t *batch_dims, int64_t num_clouds,
                                                  int32_t *unique_out, int64_t *indices_out,
                                                  void *stream) {
  MN_CHECK_ARG(n >= 0 && ndim >= 1 && ndim <= MN_MAX_NDIM, "unique_static: bad n/ndim");
  MN_CHECK_ARG(indices_out != nullptr, "unique_static: null indices");
  if (n > kStaticUniqueMaxRows) {
    set_error("unique_static: %lld rows exceed the built-in scratch limit of %lld rows; call "
              "mn_unique_coordinates with a caller-provided workspace instead",
              (long long)n, (long long)kStaticUniqueMaxRows);
    return MN_ERR_BAD_ARG;
  }
  uint32_t *scratch = nullptr;
  MN_RETURN_IF(unique_scratch_address(&scratch));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  MN_LAUNCH("zero_index0_kernel", st, zero_index0_kernel<<<1, 1, 0, st>>>(indices_out));
  if (n == 0) return MN_OK;
  MN_CHECK_ARG(coords != nullptr && unique_out != nullptr, "unique_static: null pointer");
  const int nblocks = (int)div_up(n, kUqTile);
  uint32_t *counts = scratch;                       // [nblocks], every word written before read
  uint32_t *total = scratch + kStaticUniqueBlocks;  // [1]
  RowsView view{coords, batch_dims, batch_dims ? (int)num_clouds : 1, ndim, n};
  CoordSink sink{coords, ndim, unique_out, indices_out};
  MN_LAUNCH("unique_count_kernel", st,
            unique_count_kernel<RowsView><<<nblocks, kUqThreads, 0, st>>>(view, counts));
  MN_LAUNCH("scan_blocks_kernel", st,
            scan_blocks_kernel<<<1, 1024, 0, st>>>(counts, nblocks, total, nullptr));
  MN_LAUNCH("unique_compact_kernel", st,
            unique_compact_kernel<RowsView, CoordSink><<<nblocks, kUqThreads, 0, st>>>(view, sink, counts));
  return MN_OK;
}
