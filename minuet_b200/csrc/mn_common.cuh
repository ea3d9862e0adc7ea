// Shared declarations of the CUDA side: error plumbing, launch helpers, the key
// layout and the internal (C++-linkage) launchers that mn_api.cu wraps.
#pragma once

#include <cuda_runtime.h>
#include <utility>
#include <cuda_fp16.h>
#include <cuda_bf16.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>

#include "../../include/minuet_b200.h"

namespace mn {

constexpr int kNumSMs = 148;  // B200: 2 dies x 74 SMs
constexpr int kMaxDevices = 64;
constexpr int kMaxCoopBlocks = 1024;  // upper bound of a cooperative grid (workspace sizing)

// Key layout as a kernel parameter: the host copy, or (when the layout was
// derived on the device and never read back) a pointer to the device copy.
struct SpecRef {
  mn_keyspec host;
  const mn_keyspec *dev;
};
inline SpecRef make_spec_ref(const mn_keyspec &s) {
  SpecRef r;
  r.host = s;
  r.dev = static_cast<const mn_keyspec *>(s.device_copy);
  return r;
}
#ifdef __CUDACC__
__device__ __forceinline__ const mn_keyspec &spec_of(const SpecRef &r) {
  return r.dev != nullptr ? *r.dev : r.host;
}
#endif

void set_error(const char *fmt, ...);

#define MN_CHECK_ARG(cond, ...)                      \
  do {                                               \
    if (!(cond)) {                                   \
      ::mn::set_error(__VA_ARGS__);                  \
      return MN_ERR_BAD_ARG;                         \
    }                                                \
  } while (0)

#define MN_CHECK_CUDA(expr)                                                   \
  do {                                                                        \
    cudaError_t e__ = (expr);                                                 \
    if (e__ != cudaSuccess) {                                                 \
      ::mn::set_error("%s:%d CUDA error: %s", __FILE__, __LINE__,             \
                      cudaGetErrorString(e__));                               \
      return MN_ERR_CUDA;                                                     \
    }                                                                         \
  } while (0)

#define MN_CHECK_LAUNCH() MN_CHECK_CUDA(cudaGetLastError())

// Counts the launch and, while profiling is on (mn_profile_enable), brackets it
// with a pair of CUDA events on the launching stream.
struct LaunchScope {
  LaunchScope(const char *name, cudaStream_t st);
  ~LaunchScope();
  cudaStream_t st_;
  const char *name_;
  cudaEvent_t begin_, end_;   // both null unless this launch is being timed
};

#define MN_LAUNCH(name, st, ...)                  \
  do {                                            \
    {                                             \
      ::mn::LaunchScope scope__(name, st);        \
      __VA_ARGS__;                                \
    }                                             \
    MN_CHECK_LAUNCH();                            \
  } while (0)

// Dependent launches.  A kernel launched with launch_early may be given to the SMs while the kernel
// before it in the stream still drains; it starts with begin_early(), which returns when that
// kernel is complete and its writes are visible, and then lets the next one do the same.  Every
// block calls it before anything else that touches global memory or allocates tensor memory,
// and before any return, so that "complete" covers all the kernels before it.  It takes launch
// latency, block scheduling and the first instruction fetches out of the chains of short kernels
// that a map or a network is made of.
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void release_successor() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void begin_early() {
  wait_for_predecessor();
  release_successor();
}

// The same in clusters of `cluster` blocks along x (grid.x a multiple of it).
template <typename... Params, typename... Args>
inline void launch_early_clusters(void (*kernel)(Params...), unsigned cluster, dim3 grid, dim3 block, size_t smem,
                                  cudaStream_t st, Args &&...args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2]{};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  (void)cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);   // errors: MN_CHECK_LAUNCH
}

template <typename... Params, typename... Args>
inline void launch_early(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                         Args &&...args) {
  launch_early_clusters(kernel, 1u, grid, block, smem, st, std::forward<Args>(args)...);
}

// Optional phase timing of a kernel (builds with -DMN_PHASE_TIMING only): thread 0
// of the first blocks stores its SM cycle counter at numbered points into a
// file-local array that a debug entry point copies out.
#ifdef MN_PHASE_TIMING
#define MN_MARKS_DECL(name) static __device__ long long name[2048 * 16]
#define MN_MARK(name, slot)                                                          \
  do {                                                                               \
    if (threadIdx.x == 0 && blockIdx.x < 2048) name[blockIdx.x * 16 + (slot)] = clock64(); \
  } while (0)
#else
#define MN_MARKS_DECL(name)
#define MN_MARK(name, slot) do {} while (0)
#endif

#define MN_RETURN_IF(expr)              \
  do {                                  \
    mn_status s__ = (expr);             \
    if (s__ != MN_OK) return s__;       \
  } while (0)

inline int64_t div_up(int64_t a, int64_t b) { return (a + b - 1) / b; }
inline size_t align_up(size_t a, size_t b) { return (a + b - 1) / b * b; }

// Bump allocator over the caller's workspace; never touches the driver.
struct Workspace {
  char *base;
  size_t size;
  size_t used = 0;
  bool overflow = false;
  Workspace(void *p, size_t n) : base(static_cast<char *>(p)), size(n) {}
  template <typename T>
  T *take(size_t count) {
    size_t bytes = align_up(count * sizeof(T), 256);
    if (base == nullptr || used + bytes > size) {
      overflow = true;
      used += bytes;
      return nullptr;
    }
    T *p = reinterpret_cast<T *>(base + used);
    used += bytes;
    return p;
  }
};

#define MN_CHECK_WS(ws)                                                        \
  do {                                                                         \
    if ((ws).overflow) {                                                       \
      ::mn::set_error("workspace too small: need %zu bytes, have %zu",         \
                      (ws).used, (ws).size);                                   \
      return MN_ERR_WORKSPACE;                                                 \
    }                                                                          \
  } while (0)

// Offsets regrouped for the search kernel: offsets that share every dimension
// but the last form a group, and inside a group the queries of one row grow
// with the member index, so one binary search serves the whole group.
struct OffsetTable {
  int32_t num_offsets;
  int32_t num_groups;
  int32_t ndim;
  int32_t pad_;
  int32_t off[MN_MAX_OFFSETS][MN_MAX_NDIM];  // effective (sign folded) offsets
  uint8_t member[MN_MAX_OFFSETS];            // offset indices, group by group
  uint8_t group_begin[MN_MAX_OFFSETS + 1];   // prefix into member[]
};

mn_status make_offset_table(const int32_t *offsets, int64_t O, int ndim, int sign,
                            const mn_keyspec *spec, OffsetTable *out);

// Problem table of the grouped GEMM over offsets, passed to the kernels by value.
struct GemmTable {
  int32_t num_problems;
  int32_t tile_rows;                          // rows per tile the prefix was built for
  int32_t tile_prefix[MN_MAX_OFFSETS + 2];    // prefix of row tiles over problems
  int32_t rows[MN_MAX_OFFSETS + 1];
  int32_t weight_row[MN_MAX_OFFSETS + 1];     // mask row whose weight matrix to use
  const void *a[MN_MAX_OFFSETS + 1];          // first A row of the problem
  void *c[MN_MAX_OFFSETS + 1];                // first C row of the problem
  int64_t a_row[MN_MAX_OFFSETS + 1];          // that row's index inside its operand array
  uint8_t direct[MN_MAX_OFFSETS + 1];         // 1: A is the input feature matrix, 0: gather buffer
};

// Operand arrays of the tensor-core GEMM (TMA addresses whole arrays, not rows).
struct TcOperands {
  const void *gathered = nullptr;   // [gathered_rows, c_in]
  int64_t gathered_rows = 0;
  const void *sources = nullptr;    // [source_rows, c_in]
  int64_t source_rows = 0;
  void *products = nullptr;         // [gathered_rows, c_out]: outputs of the buffered problems
  void *out = nullptr;              // [out_rows, c_out]: output of the direct problem
  int64_t out_rows = 0;
  void *weights_t = nullptr;        // scratch for the transposed weights [O, c_out, c_in]
  int num_weights = 0;              // O
  int32_t *status = nullptr;        // device status word
};

// Tensor-core grouped GEMM (mn_gemm_tc.cu); *handled = false when the shape or
// dtype is outside what it covers and the caller must use the SIMT kernel.
mn_status launch_gemm_tc(const GemmTable &tab, const TcOperands &ops, int c_in, int c_out,
                         mn_dtype dtype, const void *weights, const int32_t *order,
                         cudaStream_t st, bool *handled);
bool gemm_tc_supported(int c_in, int c_out, mn_dtype dtype);
size_t gemm_tc_workspace_bytes(int64_t O, int64_t c_in, int64_t c_out);

// ---- launchers (defined in the .cu files) ---------------------------------
mn_status launch_bbox(const int32_t *a, int64_t na, const int32_t *b, int64_t nb,
                      int ndim, int32_t *minmax_dev, Workspace &ws, cudaStream_t st);
mn_status launch_pack(const int32_t *coords, int64_t n, int ndim,
                      const int64_t *batch_dims, int64_t num_clouds,
                      const int32_t *tstride, const mn_keyspec &spec,
                      uint64_t *keys_out, int32_t *status_dev, cudaStream_t st);
// Coordinate rows a sort builds its keys from (floored to tstride when given).
struct SortSource {
  const int32_t *coords;
  const int64_t *batch_dims;
  int64_t num_clouds;
  int ndim;
  const int32_t *tstride;   // host, may be NULL
};

// Two fp32 sums in a register pair: one instruction multiplies a factor into both, each with the
// rounding of fmaf.  It runs at half the rate of fmaf, so that the sums take as long, but leaves half of
// the issue slots to loads and addresses.
typedef unsigned long long f32_pair;
__device__ __forceinline__ f32_pair make_pair_f32(float x, float y) {
  f32_pair v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
  return v;
}
__device__ __forceinline__ float4 split_pairs_f32(f32_pair xy, f32_pair zw) {
  float4 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(xy));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.z), "=f"(v.w) : "l"(zw));
  return v;
}
__device__ __forceinline__ void fma_pair_f32(f32_pair a, f32_pair b, f32_pair &sum) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(sum) : "l"(a), "l"(b));
}

}  // namespace mn
