// Native host path: the bookkeeping around the library's launches that a program pays for
// on every call (outputs, workspaces, plans of kernel maps, choice of the algorithm,
// autograd), as a CPython module over ATen tensors.  The kernels stay behind the C ABI of
// include/minuet_b200.h, which this module binds at run time, so that whatever library the
// Python side loaded is the one that runs.
//
// A layer on a small cloud is bound by host time: one launch of a few microseconds took 55 us
// of interpreter and ctypes work, a kernel map 98; from here 14 and 38.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/custom_class.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <memory>
#include <mutex>
#include <optional>
#include <string>
#include <vector>

#include "../../include/minuet_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

// ---------------------------------------------------------------------------
// the library
// ---------------------------------------------------------------------------
#define MN_HOST_FUNCTIONS(X)                                                                      \
  X(mn_last_error) X(mn_keyspec_device) X(mn_pack_keys) X(mn_downsample_coordinates)              \
  X(mn_map_workspace_bytes) X(mn_build_kernel_map) X(mn_implicit_supported)                       \
  X(mn_neighbor_table_workspace_bytes) X(mn_build_neighbor_table) X(mn_implicit_workspace_bytes)  \
  X(mn_sparse_convolution_forward_implicit)                                                       \
  X(mn_sparse_convolution_forward_implicit_fp32) X(mn_pairs_supported) X(mn_pair_rows)            \
  X(mn_build_pair_list) X(mn_pairs_workspace_bytes) X(mn_sparse_convolution_forward_pairs)        \
  X(mn_conv_workspace_bytes) X(mn_sparse_convolution_forward) X(mn_apply_epilogue)                \
  X(mn_dense_supported) X(mn_dense_workspace_bytes) X(mn_dense_forward) X(mn_dense_forward_simt)  \
  X(mn_pair_list_rows) X(mn_build_pair_lists) X(mn_weight_gradient_workspace_bytes)               \
  X(mn_sparse_convolution_weight_gradient) X(mn_voxelize_workspace_bytes) X(mn_voxelize)           \
  X(mn_dense_weight_gradient_workspace_bytes) X(mn_dense_weight_gradient)

struct Api {
#define MN_DECLARE(name) decltype(&::name) name = nullptr;
  MN_HOST_FUNCTIONS(MN_DECLARE)
#undef MN_DECLARE
  void *handle = nullptr;
} api;

void bind(const std::string &path) {
  void *handle = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (handle == nullptr) throw std::runtime_error(std::string("cannot load ") + path + ": " + dlerror());
#define MN_BIND(name)                                                         \
  api.name = reinterpret_cast<decltype(api.name)>(dlsym(handle, #name));      \
  if (api.name == nullptr) throw std::runtime_error(path + " has no " #name);
  MN_HOST_FUNCTIONS(MN_BIND)
#undef MN_BIND
  api.handle = handle;
}

void raise_status(mn_status status, const char *what) {
  const std::string msg = std::string(what) + ": " + api.mn_last_error();
  if (status == MN_ERR_UNSUPPORTED) {
    py::gil_scoped_acquire gil;
    PyErr_SetString(PyExc_NotImplementedError, msg.c_str());
    throw py::error_already_set();
  }
  throw std::runtime_error(msg);
}
inline void check(mn_status status, const char *what) {
  if (status != MN_OK) raise_status(status, what);
}
inline void check_cuda(cudaError_t e, const char *what) {
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

[[noreturn]] void not_on_gpu() {
  py::gil_scoped_acquire gil;
  PyErr_SetString(PyExc_NotImplementedError, "minuet_b200 runs on CUDA tensors only (no CPU path)");
  throw py::error_already_set();
}

// A trace would record nothing of a call into this module but its result, as a constant.
void refuse_tracing() {
  if (torch::jit::tracer::isTracing())
    throw std::runtime_error("sparse convolutions cannot be traced by torch.jit.trace");
}

// A kernel follows the operand's pointer: one on the host, or on another GPU than `like`, would be
// an illegal access there.
void require_device(const Tensor &t, const Tensor &like, const char *what) {
  if (!t.is_cuda()) not_on_gpu();
  if (t.get_device() != like.get_device())
    throw std::runtime_error(std::string(what) + " must be on the device of its input (cuda:" +
                             std::to_string(like.get_device()) + ") but is on cuda:" + std::to_string(t.get_device()));
}
void require_device(const OptTensor &t, const Tensor &like, const char *what) {
  if (t.has_value() && t->defined()) require_device(*t, like, what);
}

// ---------------------------------------------------------------------------
// memory, streams
// ---------------------------------------------------------------------------
inline cudaStream_t stream_of(const Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

inline Tensor empty_on(const Tensor &t, at::IntArrayRef sizes, at::ScalarType dtype) {
  return at::empty(sizes, t.options().dtype(dtype).requires_grad(false));
}

// Scratch of one library call, from the stream-ordered caching allocator.
inline Tensor workspace(const Tensor &like, size_t bytes) {
  return at::empty({(int64_t)std::max<size_t>(bytes, 256)}, like.options().dtype(at::kByte).requires_grad(false));
}

template <typename T>
inline T *raw(const OptTensor &t) {
  return t.has_value() && t->defined() ? static_cast<T *>(t->data_ptr()) : nullptr;
}
template <typename T>
inline T *raw(const Tensor &t) {
  return t.defined() ? static_cast<T *>(t.data_ptr()) : nullptr;
}

// The MN_CTRL_WORDS control block of (device, current stream): word 0 is the status word.
// One per stream, because kernels of different streams may overlap; never freed, as a stream
// of torch's pool is not either.  A stream that is first used inside a capture gets one per capture: it
// comes from the graph's memory and is zeroed by the graph, so nothing outside may count on it.
struct ControlBlock {
  Tensor words;
  unsigned long long capture = 0;      // of the capture that made it, 0: none
};
std::mutex ctrl_mutex;
std::map<std::pair<int, cudaStream_t>, ControlBlock> &ctrl_blocks() {
  static auto *blocks = new std::map<std::pair<int, cudaStream_t>, ControlBlock>;   // outlives the CUDA context
  return *blocks;
}

Tensor control_block(int device) {
  const cudaStream_t st = c10::cuda::getCurrentCUDAStream(device).stream();
  std::lock_guard<std::mutex> lock(ctrl_mutex);
  ControlBlock &b = ctrl_blocks()[{device, st}];
  if (b.words.defined() && b.capture == 0) return b.words;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  check_cuda(cudaStreamGetCaptureInfo(st, &status, &id), "control block");
  if (status != cudaStreamCaptureStatusActive) id = 0;
  if (!b.words.defined() || b.capture != id) {
    b.words = at::zeros({MN_CTRL_WORDS}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, device));
    b.capture = id;
  }
  return b.words;
}
inline int32_t *ctrl_of(const Tensor &t) { return static_cast<int32_t *>(control_block(t.get_device()).data_ptr()); }

// Whether the work before an event has ended.  The "not ready" of such a query is no error of this
// thread; errors that other calls have left are theirs to report.
bool ended(cudaEvent_t event) {
  const cudaError_t e = cudaEventQuery(event);
  if (e == cudaErrorNotReady && cudaPeekAtLastError() == cudaErrorNotReady) (void)cudaGetLastError();
  return e == cudaSuccess;
}

// Small pinned buffers with an event each, for device-to-host copies that the host waits for
// later (or never).  A buffer given back while its copy is still in flight is not handed out
// before the copy has ended; at most kKeep are kept.
class PinnedPool {
 public:
  static constexpr size_t kBytes = 8192;
  static constexpr size_t kKeep = 64;
  struct Buffer {
    void *host = nullptr;
    cudaEvent_t event = nullptr;
    int device = -1;
  };
  Buffer take(int device) {
    {
      std::lock_guard<std::mutex> lock(mutex_);
      for (size_t i = 0; i < free_.size(); i++) {
        if (free_[i].device == device && ended(free_[i].event)) {
          Buffer b = free_[i];
          free_.erase(free_.begin() + (long)i);
          return b;
        }
      }
    }
    Buffer b;
    b.device = device;
    check_cuda(cudaHostAlloc(&b.host, kBytes, cudaHostAllocDefault), "pinned buffer");
    check_cuda(cudaEventCreateWithFlags(&b.event, cudaEventDisableTiming), "pinned buffer");
    return b;
  }
  void give(Buffer b) {
    if (b.host == nullptr) return;
    std::lock_guard<std::mutex> lock(mutex_);
    if (free_.size() < kKeep) {
      free_.push_back(b);
      return;
    }
    (void)cudaEventSynchronize(b.event);
    (void)cudaEventDestroy(b.event);
    (void)cudaFreeHost(b.host);
  }

 private:
  std::mutex mutex_;
  std::vector<Buffer> free_;
};
PinnedPool &pinned_pool() {
  static PinnedPool *pool = new PinnedPool;   // outlives every plan, whatever the order of exits
  return *pool;
}

// Host memory that the kernels of one library call write a few values to, and the event after it: the
// read needs no copy (a copy of a few bytes is 3 us on the stream, and 2 to 9 us pass before it starts).
// Not used (host() is NULL) for more than a buffer holds and inside a stream capture, where a
// replay would write to memory that has been given back.
class Reply {
 public:
  Reply(const Tensor &like, size_t bytes) : stream_(stream_of(like)) {
    if (bytes <= PinnedPool::kBytes && c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None)
      buffer_ = pinned_pool().take(like.get_device());
  }
  Reply(const Reply &) = delete;
  ~Reply() {
    if (used()) pinned_pool().give(written());   // a call that has failed may have launched some of its kernels
  }
  bool used() const { return buffer_.host != nullptr; }
  template <typename T>
  T *host() const { return static_cast<T *>(buffer_.host); }
  // for a call that records the event itself, once the values are complete
  cudaEvent_t event() {
    recorded_ = used();
    return buffer_.event;
  }
  // The buffer, its event recorded behind the call; empty if it is not used.
  PinnedPool::Buffer written() {
    if (used() && !recorded_) (void)cudaEventRecord(buffer_.event, stream_);
    PinnedPool::Buffer b = buffer_;
    buffer_ = {};
    return b;
  }

 private:
  cudaStream_t stream_;
  PinnedPool::Buffer buffer_;
  bool recorded_ = false;
};

[[noreturn]] void raise_device_status(int value, int device) {
  py::gil_scoped_acquire gil;
  py::module_::import("minuet_b200.engine").attr("raise_on_status")(value, device);
  throw std::runtime_error("device status " + std::to_string(value));
}

// Non-blocking look at the status word: queues a copy of it and returns the first non-zero value
// of the copies that have landed (0: none).
int poll_status(int device) {
  static std::mutex mutex;
  static auto *queues = new std::map<int, std::vector<PinnedPool::Buffer>>;
  std::lock_guard<std::mutex> lock(mutex);
  auto &queue = (*queues)[device];
  while (!queue.empty() && ended(queue.front().event)) {
    const int value = *static_cast<int32_t *>(queue.front().host);
    pinned_pool().give(queue.front());
    queue.erase(queue.begin());
    if (value != 0) return value;
  }
  if (queue.size() < 8) {
    c10::cuda::CUDAGuard guard(device);
    const cudaStream_t st = c10::cuda::getCurrentCUDAStream(device).stream();
    PinnedPool::Buffer b = pinned_pool().take(device);
    check_cuda(cudaMemcpyAsync(b.host, control_block(device).data_ptr(), sizeof(int32_t), cudaMemcpyDeviceToHost, st),
               "status word");
    check_cuda(cudaEventRecord(b.event, st), "status word");
    queue.push_back(b);
  }
  return 0;
}

// ---------------------------------------------------------------------------
// key layouts and coordinates
// ---------------------------------------------------------------------------
struct KeyLayout {
  mn_keyspec spec{};
  Tensor dev;      // device copy of the layout, alive as long as this object

  ~KeyLayout() { pinned_pool().give(bits_); }
  // The kernel also writes the width of the keys here: where it has landed by the time a sort is
  // launched, no digit too many is (a digit pass that finds nothing to do is 2-4 us).
  void expect_bits(PinnedPool::Buffer written) { bits_ = written; }
  void look_for_bits() {
    if (spec.total_bits > 0 || bits_.host == nullptr) return;
    if (ended(bits_.event)) spec.total_bits = *static_cast<int32_t *>(bits_.host);
  }

 private:
  PinnedPool::Buffer bits_;
};

struct Offsets {
  std::vector<int32_t> table;   // [O, ndim]
  int64_t count = 0;
  int ndim = 0;
  int reach = 0;                // largest absolute value
};

std::shared_ptr<Offsets> make_offsets(const std::vector<std::vector<int32_t>> &rows, int ndim) {
  auto o = std::make_shared<Offsets>();
  o->count = (int64_t)rows.size();
  o->ndim = ndim;
  for (const auto &r : rows)
    for (int32_t v : r) {
      o->table.push_back(v);
      o->reach = std::max(o->reach, std::abs(v));
    }
  return o;
}

// Bounding box, key layout and the keys of `coords` in one launch, all left on the device.
std::pair<std::shared_ptr<KeyLayout>, Tensor> root_keys(const Tensor &coords, const OptTensor &batch_dims,
                                                        int64_t num_clouds, int margin) {
  if (!coords.is_cuda()) not_on_gpu();
  require_device(batch_dims, coords, "batch_dims");
  c10::cuda::CUDAGuard guard(coords.get_device());
  auto layout = std::make_shared<KeyLayout>();
  layout->dev = empty_on(coords, {256}, at::kByte);
  Tensor keys = empty_on(coords, {coords.size(0)}, at::kLong);
  Tensor ws = workspace(coords, api.mn_map_workspace_bytes(0, 0, 0));
  Reply bits(coords, sizeof(int32_t));
  check(api.mn_keyspec_device(raw<int32_t>(coords), coords.size(0), (int)coords.size(1), raw<int64_t>(batch_dims),
                              std::max<int64_t>(num_clouds, 1), margin, layout->dev.data_ptr(), &layout->spec,
                              raw<uint64_t>(keys), bits.host<int32_t>(), ctrl_of(coords), ws.data_ptr(),
                              (size_t)ws.numel(), stream_of(coords)),
        "keyspec_device");
  layout->expect_bits(bits.written());
  return {layout, keys};
}

Tensor pack_keys(const Tensor &coords, const OptTensor &batch_dims, KeyLayout &layout) {
  if (!coords.is_cuda()) not_on_gpu();
  require_device(batch_dims, coords, "batch_dims");
  c10::cuda::CUDAGuard guard(coords.get_device());
  Tensor keys = empty_on(coords, {coords.size(0)}, at::kLong);
  const int64_t nb = batch_dims.has_value() ? batch_dims->numel() - 1 : 1;
  check(api.mn_pack_keys(raw<int32_t>(coords), coords.size(0), (int)coords.size(1), raw<int64_t>(batch_dims), nb,
                         nullptr, &layout.spec, raw<uint64_t>(keys), ctrl_of(coords), stream_of(coords)),
        "pack_keys");
  return keys;
}

mn_dtype dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return MN_F32;
    case at::kHalf: return MN_F16;
    case at::kBFloat16: return MN_BF16;
    default:
      throw std::runtime_error(std::string("Cannot find implementation of sparse convolution for ") + c10::toString(t));
  }
}

// Blocking read of a small int64 tensor.
std::vector<int64_t> read_back(const Tensor &t) {
  std::vector<int64_t> host((size_t)t.numel());
  Tensor h = t.cpu();
  std::copy_n(static_cast<int64_t *>(h.data_ptr()), host.size(), host.begin());
  return host;
}

// What `reply` holds, or where the values did not fit it what `t` holds on the device.
std::vector<int64_t> read_reply(Reply &reply, const Tensor &t) {
  if (!reply.used()) return read_back(t);
  const PinnedPool::Buffer b = reply.written();
  const cudaError_t e = cudaEventSynchronize(b.event);
  std::vector<int64_t> host((size_t)t.numel());
  if (e == cudaSuccess) std::copy_n(static_cast<int64_t *>(b.host), host.size(), host.begin());
  pinned_pool().give(b);
  check_cuda(e, "device-to-host read");
  return host;
}

// Output coordinates of a strided level: (rows, keys, cloud starts on the device, cloud starts on
// the host).  One blocking read, of the number of rows (it sets the shapes of what follows).
std::tuple<Tensor, Tensor, Tensor, std::vector<int64_t>> downsample(const Tensor &coords, const OptTensor &batch_dims,
                                                                    const std::vector<int32_t> &tstride,
                                                                    KeyLayout &layout) {
  if (!coords.is_cuda()) not_on_gpu();
  require_device(batch_dims, coords, "batch_dims");
  c10::cuda::CUDAGuard guard(coords.get_device());
  const int64_t n = coords.size(0), ndim = coords.size(1);
  const int64_t nb = batch_dims.has_value() ? batch_dims->numel() - 1 : 1;
  Tensor unique = empty_on(coords, {n, ndim}, at::kInt);
  Tensor keys = empty_on(coords, {n}, at::kLong);
  Tensor meta = empty_on(coords, {nb + 4}, at::kLong);   // count, cloud starts, status, key bits
  Tensor ws = workspace(coords, api.mn_map_workspace_bytes(n, n, 1));
  layout.look_for_bits();
  Reply reply(coords, sizeof(int64_t) * (size_t)(nb + 4));
  check(api.mn_downsample_coordinates(raw<int32_t>(coords), n, (int)ndim, raw<int64_t>(batch_dims), nb,
                                      tstride.data(), &layout.spec, raw<int32_t>(unique), raw<uint64_t>(keys),
                                      raw<int64_t>(meta), reply.host<int64_t>(), ctrl_of(coords), ws.data_ptr(),
                                      (size_t)ws.numel(), stream_of(coords)),
        "downsample_coordinates");
  const std::vector<int64_t> host = read_reply(reply, meta);
  if (host[(size_t)nb + 2] != 0) raise_device_status((int)host[(size_t)nb + 2], coords.get_device());
  layout.spec.total_bits = (int32_t)host[(size_t)nb + 3];   // later levels launch no digit too many
  const int64_t count = host[0];
  return {unique.narrow(0, 0, count), keys.narrow(0, 0, count), meta.narrow(0, 1, nb + 1),
          std::vector<int64_t>(host.begin() + 1, host.begin() + nb + 2)};
}

// Distinct voxels of floating-point points: (voxels, cloud starts, inverse or None, means or None), or
// None when the voxels' box is too wide for keys that carry the point's index.
std::optional<std::tuple<Tensor, Tensor, OptTensor, OptTensor>> voxelize(const Tensor &points_in,
                                                                         const std::vector<double> &voxel_size,
                                                                         const OptTensor &batch_dims, bool inverse,
                                                                         const OptTensor &features_in) {
  at::NoGradGuard no_grad;
  if (!points_in.is_cuda()) not_on_gpu();
  require_device(batch_dims, points_in, "batch_dims");
  require_device(features_in, points_in, "features");
  c10::cuda::CUDAGuard guard(points_in.get_device());
  const Tensor points = points_in.contiguous();
  const int64_t n = points.size(0), ndim = points.size(1);
  const int64_t nb = batch_dims.has_value() ? batch_dims->numel() - 1 : 1;
  OptTensor features, means, inv;
  if (features_in.has_value()) {
    features = features_in->contiguous();
    means = empty_on(*features, {n, features->size(1)}, features->scalar_type());
  }
  if (inverse) inv = empty_on(points, {n}, at::kLong);
  Tensor voxels = empty_on(points, {n, ndim}, at::kInt);
  Tensor meta = empty_on(points, {nb + 4}, at::kLong);
  Tensor ws = workspace(points, api.mn_voxelize_workspace_bytes(n));
  Reply reply(points, sizeof(int64_t) * (size_t)(nb + 4));
  check(api.mn_voxelize(points.data_ptr(), points.scalar_type() == at::kDouble, n, (int)ndim, voxel_size.data(),
                        raw<int64_t>(batch_dims), nb, raw<void>(features), features.has_value() ? features->size(1) : 0,
                        features.has_value() ? dtype_code(features->scalar_type()) : MN_F32, raw<int32_t>(voxels),
                        raw<int64_t>(inv), raw<void>(means), raw<int64_t>(meta), reply.host<int64_t>(),
                        reply.event(), ctrl_of(points), ws.data_ptr(), (size_t)ws.numel(), stream_of(points)),
        "voxelize");
  const std::vector<int64_t> host = read_reply(reply, meta);
  int index_bits = 1;
  while ((1ll << index_bits) < n) index_bits++;
  if (host[(size_t)nb + 3] + index_bits > 64) return std::nullopt;
  if (host[(size_t)nb + 2] != 0) raise_device_status((int)host[(size_t)nb + 2], points.get_device());
  const int64_t count = host[0];
  if (means.has_value()) means = means->narrow(0, 0, count);
  return std::make_tuple(voxels.narrow(0, 0, count), meta.narrow(0, 1, nb + 1), inv, means);
}

// ---------------------------------------------------------------------------
// plans of kernel maps
// ---------------------------------------------------------------------------
// Device memory that a plan makes on first use belongs to the stream of the call that made it: calls on
// other streams wait until it is there, and the allocator does not hand it out again before
// they are through.  (A capture begins on an idle device and may not wait for work outside itself.)
bool capturing() {
  return c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
}

class Made {
 public:
  Made() = default;
  Made(const Made &) = delete;
  ~Made() {
    if (event_ != nullptr) (void)cudaEventDestroy(event_);
  }
  void here(c10::DeviceIndex device) {
    device_ = device;
    stream_ = c10::cuda::getCurrentCUDAStream(device).stream();
    check_cuda(cudaEventCreateWithFlags(&event_, cudaEventDisableTiming), "plan");
    check_cuda(cudaEventRecord(event_, stream_), "plan");
  }
  bool elsewhere() const { return c10::cuda::getCurrentCUDAStream(device_).stream() != stream_ && !capturing(); }
  void join(std::initializer_list<Tensor> memory) const {
    const c10::cuda::CUDAStream now = c10::cuda::getCurrentCUDAStream(device_);
    check_cuda(cudaStreamWaitEvent(now.stream(), event_, 0), "plan");
    for (const Tensor &t : memory)
      if (t.defined()) c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), now);
  }

 private:
  c10::DeviceIndex device_ = 0;
  cudaStream_t stream_ = nullptr;
  cudaEvent_t event_ = nullptr;
};

struct Neighbours {
  Tensor nbr, tile_bits, perm;
};

// What the convolutions derive from a kernel map, once: the pair counts on the host, hit words,
// neighbour tables and pair lists.  `swapped` asks for the map with its two sides exchanged (a
// transposed convolution, an input gradient).  Holds no masks: they belong to the caller.
struct Plan {
  int64_t O = 0, S = 0, T = 0;
  Tensor bits_s, bits_t;                 // hit words of the two sides (undefined: none)
  // what calls have made so far (a call inside a stream capture keeps nothing: its work is not done
  // before the graph is replayed)
  Neighbours nb[2][2];                   // [swapped][rows sorted by hit word]
  Tensor pair_src[2][2];                 // [swapped][shortcut], of the pair-list forward
  Tensor lists;                          // [2, rows]: source and target row of every pair
  Made nb_made[2][2], pair_src_made[2][2], lists_made;
  int last_algorithm = 0;                // of the last forward: 1 explicit, 2 implicit
  // held while a call looks things up or makes them: a backward pass runs on a thread of its own.
  // Never waited for with the GIL held (its holder may need the GIL to raise).
  std::recursive_mutex mutex;
  using Lock = std::lock_guard<std::recursive_mutex>;

  Plan(int64_t o, int64_t s, int64_t t) : O(o), S(s), T(t) {}
  ~Plan() {
    if (pending_) pinned_pool().give(buffer_);
  }
  Plan(const Plan &) = delete;

  void set_sizes(const std::vector<int32_t> &v) {
    sizes_ = v;
    total_ = 0;
    for (int32_t n : sizes_) total_ += n;
    known_ = true;
  }
  // The sizes and the status word behind them come with a copy that is already in flight.  Inside a stream
  // capture they do not: every replay makes the map anew, with the sizes of the coordinates that it finds, and
  // would write them to a buffer that may have been given back.
  void expect_sizes(const Tensor &sizes_and_status) {
    captured_ = capturing();
    if (captured_) return;
    const cudaStream_t st = stream_of(sizes_and_status);
    buffer_ = pinned_pool().take(sizes_and_status.get_device());
    pending_ = true;
    check_cuda(cudaMemcpyAsync(buffer_.host, sizes_and_status.data_ptr(), sizeof(int32_t) * (size_t)(O + 1),
                               cudaMemcpyDeviceToHost, st), "kernel map sizes");
    check_cuda(cudaEventRecord(buffer_.event, st), "kernel map sizes");
  }
  const std::vector<int32_t> &sizes() {
    Lock lock(mutex);
    if (!known_) {
      if (captured_)
        throw std::runtime_error("the pair counts of a kernel map that was built inside a stream capture are not known "
                                 "to the host: build the map outside, or pass copies of its masks and sizes");
      if (!pending_) throw std::runtime_error("the sizes of this kernel map are not known");
      const cudaError_t e = cudaEventSynchronize(buffer_.event);
      const int32_t *host = static_cast<const int32_t *>(buffer_.host);
      std::vector<int32_t> v(host, host + O);
      const int32_t status = host[O];
      const int device = buffer_.device;
      check_cuda(e, "kernel map sizes");
      if (status != 0) raise_device_status(status, device);   // now and whenever asked again
      pinned_pool().give(buffer_);
      buffer_ = {};
      pending_ = false;
      set_sizes(v);
    }
    return sizes_;
  }
  // the same, written by the kernel itself
  void expect_sizes(PinnedPool::Buffer written) {
    buffer_ = written;
    pending_ = true;
  }
  int64_t pairs() {
    sizes();
    return total_;
  }

 private:
  std::vector<int32_t> sizes_;
  int64_t total_ = 0;
  bool known_ = false, pending_ = false, captured_ = false;
  PinnedPool::Buffer buffer_;
};
using PlanPtr = std::shared_ptr<Plan>;

// Masks, order and sizes from packed keys (up to 32 offsets) and the plan of the map.
std::tuple<Tensor, Tensor, Tensor, Tensor, PlanPtr> build_map(const Tensor &source_keys, const Tensor &target_keys,
                                                              const Offsets &offsets, KeyLayout &layout,
                                                              bool reorder) {
  c10::cuda::CUDAGuard guard(source_keys.get_device());
  const int64_t S = source_keys.numel(), T = target_keys.numel(), O = offsets.count;
  Tensor sm = empty_on(source_keys, {O, S}, at::kInt);
  Tensor tm = empty_on(source_keys, {O, T}, at::kInt);
  // one allocation for the small outputs: order [O], sizes + status word [O + 1] and the per-row
  // hit words [S], [T] (each part starts on a 256-byte boundary)
  auto pad = [](int64_t n) { return (n + 63) / 64 * 64; };
  const int64_t base = 2 * pad(O + 1);
  Tensor small = empty_on(source_keys, {base + pad(S) + pad(T)}, at::kInt);
  int32_t *p = raw<int32_t>(small);
  auto plan = std::make_shared<Plan>(O, S, T);
  plan->bits_s = small.narrow(0, base, S);
  plan->bits_t = small.narrow(0, base + pad(S), T);
  const bool same = source_keys.data_ptr() == target_keys.data_ptr() && S == T;
  Tensor ws = workspace(source_keys, api.mn_map_workspace_bytes(S, T, O));
  const uint64_t *sk = raw<uint64_t>(source_keys);
  const uint64_t *tk = same ? sk : raw<uint64_t>(target_keys);
  Reply reply(source_keys, sizeof(int32_t) * (size_t)(O + 1));
  check(api.mn_build_kernel_map(sk, S, tk, T, offsets.table.data(), O, &layout.spec, reorder ? 1 : 0,
                                raw<int32_t>(sm), raw<int32_t>(tm), p, p + pad(O + 1),
                                reinterpret_cast<uint32_t *>(p + base),
                                reinterpret_cast<uint32_t *>(p + base + pad(S)), reply.host<int32_t>(),
                                ctrl_of(source_keys), ws.data_ptr(), (size_t)ws.numel(), stream_of(source_keys)),
        "build_kernel_map");
  if (reply.used()) plan->expect_sizes(reply.written());
  else plan->expect_sizes(small.narrow(0, pad(O + 1), O + 1));
  return {sm, tm, small.narrow(0, 0, O), small.narrow(0, pad(O + 1), O), plan};
}

Neighbours neighbours(Plan &plan, bool swapped, bool reorder, const Tensor &sm, const Tensor &tm) {
  const Tensor &sb = swapped ? plan.bits_t : plan.bits_s, &tb = swapped ? plan.bits_s : plan.bits_t;
  const bool sorted = reorder && tb.defined();
  Plan::Lock lock(plan.mutex);
  Neighbours &n = plan.nb[swapped][sorted];
  if (n.nbr.defined()) {
    const Made &made = plan.nb_made[swapped][sorted];
    if (made.elsewhere()) made.join({n.nbr, n.tile_bits, n.perm});
    return n;
  }
  c10::cuda::CUDAGuard guard(tm.get_device());
  const int64_t O = plan.O, S = swapped ? plan.T : plan.S, T = swapped ? plan.S : plan.T;
  const auto &sizes = plan.sizes();
  // rows of the table start on 128-row tiles (the kernels read whole tiles)
  const int64_t pitch = (T + 127) / 128 * 128;
  Tensor nbr = empty_on(tm, {O, pitch}, at::kInt).narrow(1, 0, T);
  Tensor tile_bits = empty_on(tm, {(T + 127) / 128}, at::kInt), perm;
  if (sorted) perm = empty_on(tm, {T}, at::kInt);
  Tensor ws = workspace(tm, api.mn_neighbor_table_workspace_bytes(sizes.data(), O, T));
  check(api.mn_build_neighbor_table(raw<int32_t>(sm), raw<int32_t>(tm), sizes.data(), O, S, T,
                                    sorted ? raw<uint32_t>(sb) : nullptr, sorted ? raw<uint32_t>(tb) : nullptr,
                                    raw<int32_t>(nbr), raw<uint32_t>(tile_bits), raw<int32_t>(perm), ctrl_of(tm),
                                    ws.data_ptr(), (size_t)ws.numel(), stream_of(tm)),
        "build_neighbor_table");
  if (!capturing()) {
    plan.nb_made[swapped][sorted].here((c10::DeviceIndex)tm.get_device());
    n = {nbr, tile_bits, perm};
  }
  return {nbr, tile_bits, perm};
}

// Source row of every product row of the pair-list forward; undefined when the map has no hit words.
Tensor pair_sources(Plan &plan, bool swapped, bool shortcut, const Tensor &sm) {
  const Tensor &sb = swapped ? plan.bits_t : plan.bits_s;
  if (!sb.defined()) return {};
  Tensor &t = plan.pair_src[swapped][shortcut];
  if (t.defined()) {
    const Made &made = plan.pair_src_made[swapped][shortcut];
    if (made.elsewhere()) made.join({t});
    return t;
  }
  const int64_t O = plan.O, S = swapped ? plan.T : plan.S, T = swapped ? plan.S : plan.T;
  const auto &sizes = plan.sizes();
  Tensor list = empty_on(sm, {std::max<int64_t>(api.mn_pair_rows(sizes.data(), O, S, T, shortcut), 1)}, at::kInt);
  check(api.mn_build_pair_list(raw<int32_t>(sm), raw<uint32_t>(sb), sizes.data(), O, S, T, shortcut,
                               raw<int32_t>(list), stream_of(sm)),
        "build_pair_list");
  if (!capturing()) {
    plan.pair_src_made[swapped][shortcut].here((c10::DeviceIndex)sm.get_device());
    t = list;
  }
  return list;
}

// ---------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------
enum Algorithm { kAuto = 0, kExplicit = 1, kImplicit = 2 };

// Rough cost of one 16-bit forward pass in milliseconds, fitted to 144 layers of 2 500 to 918 000
// rows, 8 to 256 channels and 1 to 20 pairs per row (the fused kernel within 25 % of most, pair
// lists within a factor of two; of the 144 choices four are wrong, all at 12 000 rows and by less
// than 3 us).  Pair lists move every non-centre pair row three times (16-bit read, fp32 product
// written and read back) and every row twice in the centre product.  The fused kernel pays per
// 128-row tile and per offset of a tile, of which the row permutation leaves a tile a little over
// the pairs per row.  It is the faster one nearly everywhere, up to 9 times where pairs are many;
// the neighbour table it needs is built once per map.  Of maps with a pair or more per row (8 and 27
// offsets, 500 to 8 million rows, 8 to 256 channels) the estimate gives none to the pair lists: they
// run on request, and where most targets have no pair at all.
double estimate_ms(bool implicit, double S, double T, double O, double c_in, double c_out, double pairs,
                   bool shortcut, bool reorder) {
  if (implicit) {
    const double tiles = std::ceil(T / 128);
    const double present = reorder ? std::min(O, 1.0 + 1.4 * std::max(pairs / std::max(T, 1.0) - 1.0, 0.0)) : O;
    return 0.0177 + tiles * (4.0e-6 + 1.7e-8 * (c_in + c_out)) +
           1.6e-6 * tiles * present * std::ceil(c_in / 64) * (1.05 + c_out / 128);
  }
  const double rest = pairs - (shortcut ? std::min(S, T) : 0.0);
  return 0.022 + (rest * (8.0 * c_out + 2.0 * c_in) + 2.0 * (S * std::max(c_in, 32.0) + T * std::max(c_out, 32.0))) / 1.8e9;
}

struct ConvOptions {
  bool shortcut = false;
  int algorithm = kAuto;      // the call's or the module's choice
  int sub_tiles = 0;
  int gather_tile = 1, scatter_tile = 1;
  bool has_threshold = true;
  double threshold = -1;
  bool reorder = true;
  bool relu = false;
};

int pick_algorithm(Plan &plan, bool swapped, int64_t c_in, int64_t c_out, mn_dtype code, const ConvOptions &o) {
  const int64_t T = swapped ? plan.S : plan.T, S = swapped ? plan.T : plan.S;
  if (T == 0) return kExplicit;
  // fp32: one kernel for any channel counts, whose sums are the explicit path's bit for bit, so
  // that a call (or a tuned configuration) that asks for that path gets its result too; the path
  // itself is for more than 32 offsets
  if (code == MN_F32) return plan.O > 32 ? kExplicit : kImplicit;
  if (o.algorithm == kExplicit) return kExplicit;
  if (!api.mn_implicit_supported(plan.O, c_in, c_out, code)) return kExplicit;
  if (o.algorithm == kImplicit) return kImplicit;
  // without hit words the explicit path would gather and scatter through HBM
  if (!api.mn_pairs_supported(plan.O, c_in, c_out, code) || !plan.bits_t.defined()) return kImplicit;
  const bool shortcut = o.shortcut && plan.O > 0 && plan.sizes().back() == S && S == T;
  const double pairs = (double)plan.pairs();
  const bool implicit = estimate_ms(true, S, T, plan.O, c_in, c_out, pairs, shortcut, o.reorder) <
                        estimate_ms(false, S, T, plan.O, c_in, c_out, pairs, shortcut, o.reorder);
  return implicit ? kImplicit : kExplicit;
}

Tensor zero_channels(const Tensor &t, int64_t dim, int64_t pad) {
  auto sizes = t.sizes().vec();
  sizes[(size_t)dim] += pad;
  Tensor out = at::zeros(sizes, t.options().requires_grad(false));
  out.narrow(dim, 0, t.size(dim)).copy_(t);
  return out;
}

// TMA reads transposed weights, from a 16-byte boundary; off one the call transposes its own (a
// weight that is a view into a flat parameter buffer, its own transpose in the backward pass).
void drop_misaligned(OptTensor &w_t) {
  if (w_t.has_value() && (reinterpret_cast<uintptr_t>(w_t->data_ptr()) & 15) != 0) w_t = std::nullopt;
}

Tensor run_forward(Plan &plan, bool swapped, Tensor x, Tensor w, const Tensor &sm, const Tensor &tm,
                   const OptTensor &order, OptTensor w_t, const OptTensor &scale, const OptTensor &shift,
                   const OptTensor &residual, const ConvOptions &o) {
  const int64_t O = plan.O, S = swapped ? plan.T : plan.S, T = swapped ? plan.S : plan.T;
  const mn_dtype code = dtype_code(w.scalar_type());
  const int64_t c_out = w.size(2);
  Plan::Lock lock(plan.mutex);
  if (code != MN_F32 && w.size(1) % 8 != 0 && c_out % 8 == 0) {
    // few input channels (a network's first layer): zero channels up to a multiple of 8 put the
    // layer on the tensor-core paths instead of gather - FFMA GEMM - scatter
    const int64_t pad = 8 - w.size(1) % 8;
    x = zero_channels(x, 1, pad);
    w = zero_channels(w, 1, pad);
    w_t = std::nullopt;
  }
  drop_misaligned(w_t);
  const int64_t c_in = w.size(1);
  const auto &sizes = plan.sizes();
  const int choice = pick_algorithm(plan, swapped, c_in, c_out, code, o);
  plan.last_algorithm = choice;
  // weights that only their transpose is read of may stay a view (an input gradient's)
  if (choice != kImplicit || code == MN_F32 || !w_t.has_value()) w = w.contiguous();
  Tensor out = empty_on(x, {T, c_out}, w.scalar_type());
  if (T == 0) return out;
  const cudaStream_t st = stream_of(x);
  const int32_t *ord = raw<int32_t>(order);
  const float *sc = raw<float>(scale), *sh = raw<float>(shift);
  const void *res = raw<void>(residual);
  if (choice == kImplicit) {
    const Neighbours n = neighbours(plan, swapped, o.reorder, sm, tm);
    const int32_t *perm = raw<int32_t>(n.perm), *nbr = raw<int32_t>(n.nbr);
    const uint32_t *tiles = raw<uint32_t>(n.tile_bits);
    if (code == MN_F32) {
      check(api.mn_sparse_convolution_forward_implicit_fp32(
                S, T, O, c_in, c_out, raw<float>(x), raw<float>(w), nbr, tiles, perm, ord, sc, sh,
                static_cast<const float *>(res), o.relu, raw<float>(out), nullptr, 0, st),
            "sparse_convolution_forward_implicit_fp32");
      return out;
    }
    Tensor ws;                             // for the transposed weights, where the call makes them itself
    if (!w_t.has_value()) ws = workspace(x, api.mn_implicit_workspace_bytes(O, c_in, c_out));
    check(api.mn_sparse_convolution_forward_implicit(
              S, T, O, c_in, c_out, code, x.data_ptr(), w.data_ptr(), raw<void>(w_t), nbr, tiles, perm, ord, sc,
              sh, res, o.relu, (double)plan.pairs() / (double)std::max<int64_t>(T, 1), o.sub_tiles, out.data_ptr(),
              ctrl_of(x), raw<void>(ws), ws.defined() ? (size_t)ws.numel() : 0, st),
          "sparse_convolution_forward_implicit");
    return out;
  }
  // sparse maps with hit words: pair lists, fp32 products, one rounding
  if (code != MN_F32 && api.mn_pairs_supported(O, c_in, c_out, code)) {
    const Tensor src = pair_sources(plan, swapped, o.shortcut, sm);
    if (src.defined()) {
      const Tensor &tb = swapped ? plan.bits_s : plan.bits_t;
      Tensor ws = workspace(x, api.mn_pairs_workspace_bytes(sizes.data(), O, S, T, c_in, c_out, o.shortcut));
      check(api.mn_sparse_convolution_forward_pairs(
                S, T, O, c_in, c_out, code, x.data_ptr(), w.data_ptr(), raw<void>(w_t), raw<int32_t>(tm),
                raw<uint32_t>(tb), raw<int32_t>(src), ord, sizes.data(), o.shortcut, sc, sh, res, o.relu,
                out.data_ptr(), ctrl_of(x), ws.data_ptr(), (size_t)ws.numel(), st),
            "sparse_convolution_forward_pairs");
      return out;
    }
  }
  Tensor ws = workspace(x, api.mn_conv_workspace_bytes(sizes.data(), O, S, T, c_in, c_out, code, o.shortcut,
                                                       o.has_threshold, o.threshold));
  check(api.mn_sparse_convolution_forward(
            S, T, O, c_in, c_out, code, x.data_ptr(), w.data_ptr(), raw<int32_t>(sm), raw<int32_t>(tm), ord,
            sizes.data(), o.gather_tile, o.scatter_tile, o.shortcut, o.has_threshold, o.threshold, out.data_ptr(),
            ctrl_of(x), ws.data_ptr(), (size_t)ws.numel(), st),
        "sparse_convolution_forward");
  if (sc != nullptr || sh != nullptr || res != nullptr || o.relu)
    check(api.mn_apply_epilogue(out.data_ptr(), T, c_out, code, sc, sh, res, o.relu, st), "apply_epilogue");
  return out;
}

// Per-channel factors and sums of an epilogue.
void check_channels(const OptTensor &v, const Tensor &like, int64_t c_out, const char *what) {
  if (!v.has_value()) return;
  require_device(v, like, what);
  if (v->numel() < c_out)
    throw std::runtime_error(std::string(what) + " must have one value per output channel (" + std::to_string(c_out) +
                             ") but has " + std::to_string(v->numel()));
}

void check_transposed(const OptTensor &w_t, const Tensor &w) {
  if (!w_t.has_value()) return;
  require_device(w_t, w, "weights_t");
  if (w_t->numel() != w.numel() || w_t->scalar_type() != w.scalar_type() || !w_t->is_contiguous())
    throw std::runtime_error("weights_t must be transpose_weights(weights)");
}

// Devices, shapes, types and layouts that every forward needs; the messages are the reference's.
void check_operands(const Plan &plan, bool swapped, const Tensor &x, const Tensor &w, const Tensor &sm,
                    const Tensor &tm, const OptTensor &order) {
  if (!x.is_cuda()) not_on_gpu();
  require_device(w, x, "weights");
  require_device(sm, x, "source_masks");
  require_device(tm, x, "target_masks");
  require_device(order, x, "kernel_map_order");
  if (order.has_value() && order->numel() < plan.O)
    throw std::runtime_error("kernel_map_order must have one entry per offset (" + std::to_string(plan.O) + ")");
  if (w.dim() != 3) throw std::runtime_error("weights must be a 3-D tensor but found " + std::to_string(w.dim()) + "-D");
  if (w.size(0) != plan.O)
    throw std::runtime_error("source_masks, weights and kernel_map_sizes must have one row per offset (" +
                             std::to_string(plan.O) + ")");
  if (x.dim() != 2 || x.size(1) != w.size(1))
    throw std::runtime_error("sources must be [N, " + std::to_string(w.size(1)) + "] but found another shape");
  if (x.scalar_type() != w.scalar_type())
    throw std::runtime_error(std::string("sources (") + c10::toString(x.scalar_type()) + ") and weights (" +
                             c10::toString(w.scalar_type()) + ") must share one dtype");
  const int64_t S = swapped ? plan.T : plan.S;
  if (x.size(0) != S)
    throw std::runtime_error("sources has " + std::to_string(x.size(0)) + " rows but the masks describe " +
                             std::to_string(S));
}

OptTensor as_f32(const OptTensor &v) {
  if (!v.has_value()) return v;
  return v->detach().to(at::kFloat).contiguous();
}

Tensor conv_forward(const PlanPtr &plan, bool swapped, const Tensor &x, const Tensor &w, const Tensor &sm,
                    const Tensor &tm, const OptTensor &order, const OptTensor &w_t, const OptTensor &scale,
                    const OptTensor &shift, const OptTensor &residual, const ConvOptions &o) {
  at::NoGradGuard no_grad;
  refuse_tracing();
  check_operands(*plan, swapped, x, w, sm, tm, order);
  check_transposed(w_t, w);
  check_channels(scale, x, w.size(2), "scale");
  check_channels(shift, x, w.size(2), "shift");
  c10::cuda::CUDAGuard guard(x.get_device());
  OptTensor res;
  if (residual.has_value()) {
    require_device(residual, x, "residual");
    res = residual->contiguous();
    const int64_t T = swapped ? plan->S : plan->T;
    if (res->dim() != 2 || res->size(0) != T || res->size(1) != w.size(2) || res->scalar_type() != w.scalar_type())
      throw std::runtime_error("residual must be [N_out, C_out] in the feature dtype");
  }
  return run_forward(*plan, swapped, x.contiguous(), w.contiguous(), sm, tm, order, w_t, as_f32(scale),
                     as_f32(shift), res, o);
}

// ---------------------------------------------------------------------------
// autograd
// ---------------------------------------------------------------------------
// With pairs (s, t) under offset k: out[t] += x[s] W[k], hence dx[s] += dout[t] W[k]^T -- the
// same convolution with the two sides exchanged and every weight matrix transposed, run by the
// same kernels -- and dW[k] = sum over the pairs of x[s]^T dout[t].  Both are differentiable in turn:
// a backward pass that keeps a graph (create_graph) is made of the same two functions, the gradients
// of dW under u being dx[s] += dout[t] u[k]^T and ddout[t] += x[s] u[k].
struct PlanHolder : torch::CustomClassHolder {
  PlanPtr plan;
  ConvOptions options;
};
using Holder = c10::intrusive_ptr<PlanHolder>;

Holder flipped(const Holder &holder) {
  auto other = c10::make_intrusive<PlanHolder>();
  other->plan = holder->plan;
  other->options = holder->options;
  std::swap(other->options.gather_tile, other->options.scatter_tile);
  return other;
}

Tensor weight_gradient(Plan &plan, bool swapped, const Tensor &x, const Tensor &g, const Tensor &sm,
                       const Tensor &tm, const OptTensor &order) {
  const int64_t O = plan.O, S = swapped ? plan.T : plan.S, T = swapped ? plan.S : plan.T;
  const int64_t c_in = x.size(1), c_out = g.size(1);
  const mn_dtype code = dtype_code(x.scalar_type());
  const auto &sizes = plan.sizes();
  const cudaStream_t st = stream_of(x);
  Plan::Lock lock(plan.mutex);
  Tensor lists = plan.lists;
  if (lists.defined()) {
    if (plan.lists_made.elsewhere()) plan.lists_made.join({lists});
  } else {
    // the two lists in the map's own direction
    lists = empty_on(sm, {2, std::max<int64_t>(api.mn_pair_list_rows(sizes.data(), O), 1)}, at::kInt);
    const Tensor &s = swapped ? tm : sm, &t = swapped ? sm : tm;
    int32_t *p = raw<int32_t>(lists);
    check(api.mn_build_pair_lists(raw<int32_t>(s), raw<int32_t>(t), raw<uint32_t>(plan.bits_s),
                                  raw<uint32_t>(plan.bits_t), sizes.data(), O, plan.S, plan.T, p,
                                  p + lists.size(1), st),
          "build_pair_lists");
    if (!capturing()) {
      plan.lists_made.here((c10::DeviceIndex)sm.get_device());
      plan.lists = lists;
    }
  }
  const int32_t *src = raw<int32_t>(lists), *dst = src + lists.size(1);
  if (swapped) std::swap(src, dst);
  Tensor grad = empty_on(x, {O, c_in, c_out}, x.scalar_type());
  Tensor ws = workspace(x, api.mn_weight_gradient_workspace_bytes(sizes.data(), O, c_in, c_out, code));
  check(api.mn_sparse_convolution_weight_gradient(S, T, O, c_in, c_out, code, x.data_ptr(), g.data_ptr(),
                                                  src, dst, raw<int32_t>(order), sizes.data(), grad.data_ptr(),
                                                  ctrl_of(x), ws.data_ptr(), (size_t)ws.numel(), st),
        "sparse_convolution_weight_gradient");
  return grad;
}

// What a function keeps of a kernel map for its backward pass.  The masks are no saved variables
// (those made in inference mode cannot be), so writes into them are counted here.
struct MapRef {
  Tensor sm, tm;
  OptTensor order;
  bool swapped;
  Holder holder;

  std::vector<int64_t> versions() const {
    std::vector<int64_t> v;
    for (const Tensor &t : {sm, tm, order.value_or(Tensor())})
      v.push_back(!t.defined() || t.is_inference() ? 0 : (int64_t)t._version());
    return v;
  }
  void save(torch::autograd::AutogradContext *ctx) const {
    ctx->saved_data["masks"] = std::vector<Tensor>{sm, tm};
    if (order.has_value()) ctx->saved_data["order"] = *order;
    ctx->saved_data["versions"] = versions();
    ctx->saved_data["swapped"] = swapped;
    ctx->saved_data["plan"] = c10::IValue::make_capsule(holder);
  }
  static MapRef load(torch::autograd::AutogradContext *ctx) {
    const auto masks = ctx->saved_data["masks"].toTensorVector();
    MapRef m{masks[0], masks[1], std::nullopt, ctx->saved_data["swapped"].toBool(),
             c10::static_intrusive_pointer_cast<PlanHolder>(ctx->saved_data["plan"].toCapsule())};
    const auto it = ctx->saved_data.find("order");
    if (it != ctx->saved_data.end()) m.order = it->second.toTensor();
    if (ctx->saved_data["versions"].toIntVector() != m.versions())
      throw std::runtime_error("one of the variables needed for gradient computation has been modified by an inplace "
                               "operation: the kernel map of a sparse convolution");
    return m;
  }
};

// A gradient that torch knows to be zero (sgn's) comes without memory.
Tensor with_memory(const Tensor &grad) { return grad._is_zerotensor() ? grad.clone() : grad; }

struct WeightGradient : torch::autograd::Function<WeightGradient> {
  static Tensor forward(torch::autograd::AutogradContext *ctx, const Tensor &x, const Tensor &g, const Tensor &sm,
                        const Tensor &tm, const OptTensor &order, bool swapped, Holder holder);
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext *ctx,
                                                 torch::autograd::variable_list grads);
};

struct Convolution : torch::autograd::Function<Convolution> {
  static Tensor forward(torch::autograd::AutogradContext *ctx, const Tensor &x, const Tensor &w,
                        const Tensor &sm, const Tensor &tm, const OptTensor &order, bool swapped, Holder holder) {
    at::AutoDispatchBelowADInplaceOrView below;
    c10::cuda::CUDAGuard guard(x.get_device());
    ctx->save_for_backward({x, w});
    MapRef{sm, tm, order, swapped, holder}.save(ctx);
    return run_forward(*holder->plan, swapped, x, w, sm, tm, order, std::nullopt, std::nullopt, std::nullopt,
                       std::nullopt, holder->options);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext *ctx,
                                                 torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1];
    c10::cuda::CUDAGuard guard(x.get_device());
    const MapRef m = MapRef::load(ctx);
    Tensor grad_x, grad_w;
    if (at::GradMode::is_enabled()) {
      const Tensor g = with_memory(grads[0]).to(w.scalar_type()).contiguous();
      if (ctx->needs_input_grad(0))
        grad_x = Convolution::apply(g, w.transpose(1, 2).contiguous(), m.tm, m.sm, m.order, !m.swapped,
                                    flipped(m.holder));
      if (ctx->needs_input_grad(1))
        grad_w = WeightGradient::apply(x, g, m.sm, m.tm, m.order, m.swapped, m.holder);
      return {grad_x, grad_w, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    }
    at::AutoDispatchBelowADInplaceOrView below;
    Plan &plan = *m.holder->plan;
    const Tensor g = with_memory(grads[0]).to(w.scalar_type()).contiguous();
    if (ctx->needs_input_grad(0)) {
      // [O, c_out, c_in] weights; their transpose, which the tensor-core kernels read, is w
      grad_x = run_forward(plan, !m.swapped, g, w.transpose(1, 2), m.tm, m.sm, m.order,
                           w.scalar_type() == at::kFloat ? OptTensor() : OptTensor(w), std::nullopt, std::nullopt,
                           std::nullopt, flipped(m.holder)->options);
    }
    if (ctx->needs_input_grad(1)) grad_w = weight_gradient(plan, m.swapped, x, g, m.sm, m.tm, m.order);
    return {grad_x, grad_w, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Tensor WeightGradient::forward(torch::autograd::AutogradContext *ctx, const Tensor &x, const Tensor &g,
                               const Tensor &sm, const Tensor &tm, const OptTensor &order, bool swapped,
                               Holder holder) {
  at::AutoDispatchBelowADInplaceOrView below;
  c10::cuda::CUDAGuard guard(x.get_device());
  ctx->save_for_backward({x, g});
  MapRef{sm, tm, order, swapped, holder}.save(ctx);
  return weight_gradient(*holder->plan, swapped, x, g, sm, tm, order);
}

torch::autograd::variable_list WeightGradient::backward(torch::autograd::AutogradContext *ctx,
                                                        torch::autograd::variable_list grads) {
  const auto saved = ctx->get_saved_variables();
  const Tensor &x = saved[0], &g = saved[1];
  c10::cuda::CUDAGuard guard(x.get_device());
  const MapRef m = MapRef::load(ctx);
  const Tensor u = with_memory(grads[0]).to(x.scalar_type()).contiguous();
  Tensor grad_x, grad_g;
  if (ctx->needs_input_grad(0))
    grad_x = Convolution::apply(g, u.transpose(1, 2).contiguous(), m.tm, m.sm, m.order, !m.swapped, flipped(m.holder));
  if (ctx->needs_input_grad(1)) grad_g = Convolution::apply(x, u, m.sm, m.tm, m.order, m.swapped, m.holder);
  return {grad_x, grad_g, Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
}

Tensor conv_autograd(const PlanPtr &plan, bool swapped, const Tensor &x, const Tensor &w, const Tensor &sm,
                     const Tensor &tm, const OptTensor &order, const ConvOptions &o) {
  refuse_tracing();
  check_operands(*plan, swapped, x, w, sm, tm, order);
  auto holder = c10::make_intrusive<PlanHolder>();
  holder->plan = plan;
  holder->options = o;
  return Convolution::apply(x.contiguous(), w.contiguous(), sm, tm, order, swapped, holder);
}

// ---------------------------------------------------------------------------
// 1x1x1 convolutions
// ---------------------------------------------------------------------------
std::pair<Tensor, bool> dense_forward(const Tensor &features_in, const Tensor &weight_in, const OptTensor &scale,
                                      const OptTensor &shift, const OptTensor &residual, bool relu,
                                      OptTensor w_t) {
  at::NoGradGuard no_grad;
  refuse_tracing();
  if (!features_in.is_cuda()) not_on_gpu();
  require_device(weight_in, features_in, "weight");
  if (features_in.dim() != 2 || weight_in.dim() != 2 || features_in.size(1) != weight_in.size(0))
    throw std::runtime_error("features must be [N, C_in] and weight [C_in, C_out]");
  check_transposed(w_t, weight_in);
  drop_misaligned(w_t);
  check_channels(scale, features_in, weight_in.size(1), "scale");
  check_channels(shift, features_in, weight_in.size(1), "shift");
  if (residual.has_value()) {
    require_device(residual, features_in, "residual");
    if (residual->numel() != features_in.size(0) * weight_in.size(1) ||
        residual->scalar_type() != features_in.scalar_type())
      throw std::runtime_error("residual must be [N, C_out] in the feature dtype");
  }
  c10::cuda::CUDAGuard guard(features_in.get_device());
  const Tensor features = features_in.contiguous(), weight = weight_in.contiguous();
  const int64_t rows = features.size(0), c_in = features.size(1), c_out = weight.size(1);
  const mn_dtype code = dtype_code(features.scalar_type());
  Tensor out = empty_on(features, {rows, c_out}, features.scalar_type());
  const OptTensor sc = as_f32(scale), sh = as_f32(shift);
  const OptTensor res = residual.has_value() ? OptTensor(residual->contiguous()) : OptTensor();
  const cudaStream_t st = stream_of(features);
  const bool tensor_core = code != MN_F32 && api.mn_dense_supported(c_in, c_out, code);
  if (tensor_core) {
    Tensor ws = workspace(features, w_t.has_value() ? 0 : api.mn_dense_workspace_bytes(c_in, c_out));
    check(api.mn_dense_forward(rows, c_in, c_out, code, features.data_ptr(), weight.data_ptr(), raw<void>(w_t),
                               raw<float>(sc), raw<float>(sh), raw<void>(res), relu, out.data_ptr(),
                               ctrl_of(features), ws.data_ptr(), (size_t)ws.numel(), st),
          "dense_forward");
  } else {
    // fp32 and the shapes the tensor-core kernel does not take: the FFMA grouped-GEMM kernel
    check(api.mn_dense_forward_simt(rows, c_in, c_out, code, features.data_ptr(), weight.data_ptr(),
                                    raw<float>(sc), raw<float>(sh), raw<void>(res), relu, out.data_ptr(), st),
          "dense_forward_simt");
  }
  return {out, tensor_core};
}

// x w in training, differentiated as torch does, except that x^T g may be a kernel of its own (own_gradient_pays; with
// fewer rows, or more weights, it never is: 512 rows 192 x 128 7.6 us in torch, 9.4 here).
bool dense_product_takes(const Tensor &x, const Tensor &w) {
  if (x.dim() != 2 || w.dim() != 2 || x.size(0) < 1024 || w.numel() > (1 << 16) ||
      (w.numel() > (1 << 15) && x.size(0) > (1 << 17)))
    return false;
  return w.requires_grad() && x.is_cuda() && w.is_cuda() && x.get_device() == w.get_device() &&
         x.scalar_type() == at::kFloat && w.scalar_type() == at::kFloat && x.layout() == at::kStrided &&
         w.layout() == at::kStrided && x.size(1) == w.size(0) && w.numel() > 0 && x.is_contiguous() && !x.is_neg() &&
         !w.is_neg() && !x.is_inference() && !w.is_inference() && x.size(0) < INT32_MAX - 4096;
}

// A tensor whose values lie at its data pointer, and nothing that watches torch's own operations: gradients may
// come batched, dual or wrapped where the forward pass was none of these.
bool plain_values(const Tensor &t) {
  for (const auto key : {c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                         c10::DispatchKey::FuncTorchVmapMode, c10::DispatchKey::Batched, c10::DispatchKey::Functionalize,
                         c10::DispatchKey::Python, c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor})
    if (t.key_set().has(key)) return false;
  return t.is_cuda() && t.layout() == at::kStrided && t.scalar_type() == at::kFloat && !t._fw_grad(0).defined() &&
         !c10::impl::TorchDispatchModeTLS::any_modes_set();
}

// Where x^T g is faster in the library's kernel than in torch's GEMM, us, torch / here.  One channel is a matrix times a
// vector there: 400k rows 96 x 1 46 / 163.  Channels in fours: 1000 rows 128 x 64 10.3 / 8.8; 60k rows 32 x 20 148 / 18, 96 x
// 20 156 / 25, 192 x 128 152 / 83.  Channels that are not are copied one by one here, and torch is good at few of them into
// many: 1024 rows 32 x 13 18.8 / 8.6, 65 x 65 11.1 / 14.7, 8000 rows 7 x 64 10.1 / 13.2, 30k rows 42 / 17, 400k 88 / 99.  Matrices
// of many tiles keep torch's GEMM busy too: 256 x 256 131k rows 444 / 391, 240k 708 / 738; 160 x 200 400k rows 899 / 878, 1 M
// 2144 / 2178; 65 x 65 131k rows 224 / 165, 400k 414 / 490; 4 x 4096 100k rows 708 / 677, 131k 785 / 887.
// A caller who allows TF32 has a faster GEMM there: 60k rows 32 x 20 64 / 18, 64 x 64 66 / 26, 128 x 64 68 / 37, 192 x 128 77 /
// 83; 131k rows 256 x 256 137 / 391; 4000 rows 64 x 64 9.1 / 11.1, 16k 17.8 / 12.6; 400k rows 128 x 64 171 / 169, 1 M 269 / 387.
bool own_gradient_pays(int64_t rows, int64_t c_in, int64_t c_out) {
  if (c_in == 1 || c_out == 1) return false;
  const bool fours = c_in % 4 == 0 && c_out % 4 == 0;
  if (!fours && c_out > 32 && rows < (c_in < 32 ? 1 << 14 : 1 << 11)) return false;
  auto tiled = [](int64_t c) { return c <= 32 ? 32 : (c + 63) / 64 * 64; };
  const int64_t tiles = tiled(c_in) * tiled(c_out), cost = fours ? tiles : 3 * tiles;
  if ((cost > (1 << 15) || (!fours && c_out > 32)) &&
      (double)rows * (double)std::max<int64_t>(cost, 1 << 15) > 1.3e10)
    return false;
  const auto precision = at::globalContext().float32Precision(at::Float32Backend::CUDA, at::Float32Op::MATMUL);
  if (precision == at::Float32Precision::IEEE || precision == at::Float32Precision::NONE) return true;
  return tiles <= 32 * 32 || (tiles <= 128 * 64 && rows >= 8192 && (double)rows * (double)tiles <= 3.3e9);
}

struct DenseProduct : torch::autograd::Function<DenseProduct> {
  static Tensor forward(torch::autograd::AutogradContext *ctx, const Tensor &x, const Tensor &w) {
    at::AutoDispatchBelowADInplaceOrView below;
    ctx->save_for_backward({x, w});
    return at::mm(x, w);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext *ctx,
                                                 torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &w = saved[1];
    c10::cuda::CUDAGuard guard(x.get_device());
    Tensor grad_x, grad_w;
    if (ctx->needs_input_grad(0)) grad_x = at::mm(grads[0], w.t());
    if (ctx->needs_input_grad(1)) {
      if (at::GradMode::is_enabled() || !plain_values(grads[0]) || !plain_values(x) || !x.is_contiguous() ||
          !own_gradient_pays(x.size(0), w.size(0), w.size(1))) {
        grad_w = at::mm(x.t(), grads[0]);
      } else {
        at::AutoDispatchBelowADInplaceOrView below;
        const Tensor g = grads[0].contiguous();
        grad_w = empty_on(x, {w.size(0), w.size(1)}, at::kFloat);
        Tensor ws = workspace(x, api.mn_dense_weight_gradient_workspace_bytes(x.size(0), w.size(0), w.size(1)));
        check(api.mn_dense_weight_gradient(x.size(0), w.size(0), w.size(1), raw<float>(x), raw<float>(g),
                                           raw<float>(grad_w), ws.data_ptr(), (size_t)ws.numel(), stream_of(x)),
              "dense_weight_gradient");
      }
    }
    return {grad_x, grad_w};
  }
};

Tensor dense_product(const Tensor &x, const Tensor &w) {
  refuse_tracing();
  if (!dense_product_takes(x, w))
    throw std::runtime_error("dense_product: operands that dense_product_takes() does not take");
  return DenseProduct::apply(x, w);
}

OptTensor optional(const Tensor &t) { return t.defined() ? OptTensor(t) : OptTensor(); }

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  using NoGil = py::call_guard<py::gil_scoped_release>;
  m.def("bind", &bind);
  m.def("control_block", &control_block);
  m.def("poll_status", &poll_status);
  py::class_<KeyLayout, std::shared_ptr<KeyLayout>>(m, "KeyLayout")
      .def_property_readonly("margin", [](KeyLayout &k) { return k.spec.margin; })
      .def_property_readonly("address", [](KeyLayout &k) { return reinterpret_cast<uintptr_t>(&k.spec); });
  py::class_<Offsets, std::shared_ptr<Offsets>>(m, "Offsets")
      .def(py::init(&make_offsets))
      .def_readonly("count", &Offsets::count)
      .def_readonly("reach", &Offsets::reach);
  m.def("root_keys", &root_keys);
  m.def("pack_keys", &pack_keys);
  m.def("downsample", &downsample, NoGil());
  m.def("voxelize", &voxelize, NoGil());
  py::class_<Plan, PlanPtr>(m, "Plan")
      .def(py::init<int64_t, int64_t, int64_t>())
      .def("set_sizes", &Plan::set_sizes)
      .def("expect_sizes", py::overload_cast<const Tensor &>(&Plan::expect_sizes))
      .def("sizes", [](Plan &p) { return p.sizes(); }, NoGil())
      .def("pairs", &Plan::pairs, NoGil())
      .def_property_readonly("source_bits", [](Plan &p) { return optional(p.bits_s); })
      .def_property_readonly("target_bits", [](Plan &p) { return optional(p.bits_t); })
      .def_readonly("last_algorithm", &Plan::last_algorithm)
      .def("neighbours", [](Plan &p, bool swapped, bool reorder, const Tensor &sm, const Tensor &tm) {
        const Neighbours n = neighbours(p, swapped, reorder, sm, tm);
        return std::make_tuple(n.nbr, n.tile_bits, optional(n.perm));
      }, NoGil());
  m.def("build_map", &build_map, NoGil());
  py::class_<ConvOptions>(m, "ConvOptions")
      .def(py::init([](bool shortcut, int algorithm, int sub_tiles, int gather_tile, int scatter_tile,
                       std::optional<double> threshold, bool reorder, bool relu) {
        ConvOptions o;
        o.shortcut = shortcut;
        o.algorithm = algorithm;
        o.sub_tiles = sub_tiles;
        o.gather_tile = gather_tile;
        o.scatter_tile = scatter_tile;
        o.has_threshold = threshold.has_value();
        o.threshold = threshold.value_or(0.0);
        o.reorder = reorder;
        o.relu = relu;
        return o;
      }));
  m.def("estimate_ms", &estimate_ms);
  m.def("conv_forward", &conv_forward, NoGil());
  m.def("conv_autograd", &conv_autograd, NoGil());
  m.def("dense_forward", &dense_forward, NoGil());
  m.def("dense_product_takes", &dense_product_takes);
  m.def("dense_product", &dense_product, NoGil());
}
