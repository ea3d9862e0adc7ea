// Fused (implicit-GEMM) forward pass of a sparse convolution in fp32.
//
// fp32 features must not go through the tensor cores (TF32 keeps 10 mantissa bits), so this
// is the output-stationary kernel of mn_conv_implicit.cu on FFMA units: a block owns BM
// consecutive rows of the neighbour table (targets sorted by hit word) and BN output
// channels, keeps the BM x BN sums in registers and walks the offsets that any of its rows
// has; source rows are fetched through the table straight into shared memory.  Gather buffer,
// product buffer and scatter pass of the explicit path do not exist: they were 15 of the 20 ms
// that the forward and input-gradient products of a UNet training step took on 60 000 voxels.
//
// Order of the sums: every offset's product is a chain of its own over the input channels,
// and the products are added in mask-row order (the centre, the largest, last).  That is the
// order of the reference's GEMM and scatter and of the explicit path, bit for bit; a network
// with ReLUs turns a last-bit difference in its forward pass into visible differences of its
// gradients.
//
// Few rows (the coarse levels of a network) leave most of the chip without a block, and then
// an offset takes the same time as on a full chip: below one block per SM the offsets of a
// tile are spread over blocks (grid.z), each product goes to a buffer, and a second launch
// adds them in the same order and applies the epilogue.
#include "mn_common.cuh"

#include <algorithm>
#include <type_traits>

namespace mn {

namespace {

constexpr int kCsK = 32;          // input channels per step
constexpr int kCsPitch = kCsK + 4;
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
  float *products;            // [O, T, N] in table order (offsets spread over blocks), or NULL
  int64_t T, pitch;
  int32_t K, N, k_steps, splits, relu;
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

__device__ __forceinline__ float4 cs_epilogue(float4 v, const CsArgs &a, int64_t row, int c) {
  float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; j++) {
    if (c + j < a.N) {
      if (a.scale != nullptr) f[j] *= __ldg(a.scale + c + j);
      if (a.shift != nullptr) f[j] += __ldg(a.shift + c + j);
      if (a.residual != nullptr) f[j] += __ldg(a.residual + row * a.N + c + j);
      if (a.relu) f[j] = fmaxf(f[j], 0.f);
    }
  }
  return make_float4(f[0], f[1], f[2], f[3]);
}

// BM x BN sums per block, 8 x 4 per thread.  A warp owns kRows consecutive rows: it fetches them
// itself and leaves out the offsets that none of them has.  Blocks take the tiles from the last
// to the first: the rows with rare offsets sort to the end, a handful of rows per offset, and
// such a tile takes several times as long as one that has the centre only.  kVec: rows of the
// features and of the weights can be copied 16 bytes at a time.
template <int BM, int BN, int kStages, bool kVec>
__global__ void __launch_bounds__(BM * BN / 32, BN == 32 ? 12 : 3)
conv_simt_kernel(const __grid_constant__ CsArgs a) {
  begin_early();
  constexpr int kThreads = BM * BN / 32, kWarps = kThreads / 32;
  constexpr int kRows = BM / kWarps;                   // rows of a warp: 32 or 16
  constexpr int kStageFloats = BM * kCsPitch + kCsK * BN;
  extern __shared__ __align__(16) float s_mem[];      // [stages][A | B], then the index blocks
  __shared__ int32_t s_active[kCsMaxOffsets], s_weight[kCsMaxOffsets];
  __shared__ uint8_t s_warps[kCsMaxOffsets];
  __shared__ uint32_t s_rows[kCsMaxOffsets][BM / 32];   // bit r: row r has this offset
  __shared__ int32_t s_count;
  int32_t *s_idx = reinterpret_cast<int32_t *>(s_mem + kStages * kStageFloats);   // [active][BM]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = lane % (BN / 4), ty = lane / (BN / 4);
  const int64_t r0 = (int64_t)(gridDim.x - 1 - blockIdx.x) * BM;
  const int n0 = blockIdx.y * BN;

  // index blocks of all the offsets this tile has (their loads are in flight together); an
  // offset of the 128-row tile that none of these BM rows has is dropped
  const uint32_t bits = __ldg(a.tile_bits + r0 / 128);
  const int n_bits = __popc(bits);
  if (warp == 0 && ((bits >> lane) & 1u)) {
    const int j = __popc(bits & ((1u << lane) - 1u));
    s_active[j] = lane;
    s_weight[j] = a.order != nullptr ? __ldg(a.order + lane) : lane;
  }
  __syncthreads();
  for (int e = tid; e < n_bits * (BM / 4); e += kThreads) {
    const int j = e / (BM / 4), i = (e % (BM / 4)) * 4;
    cs_copy_16(s_idx + j * BM + i, a.nbr + (int64_t)s_active[j] * a.pitch + r0 + i, 16u);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  for (int j = warp; j < n_bits; j += kWarps) {
    uint32_t warps = 0u;               // bit w: warp w has a row with this offset
#pragma unroll
    for (int i = 0; i < BM / 32; i++) {
      const uint32_t hit = __ballot_sync(0xffffffffu, s_idx[j * BM + i * 32 + lane] >= 0);
      if (lane == 0) s_rows[j][i] = hit;
      if (kRows == 32) warps |= (hit != 0u ? 1u : 0u) << i;
      else warps |= ((hit & 0xffffu) != 0u ? 1u : 0u) << (2 * i) | ((hit >> 16) != 0u ? 2u : 0u) << (2 * i);
    }
    if (lane == 0) s_warps[j] = (uint8_t)warps;
  }
  __syncthreads();
  if (tid == 0) {
    // compact in place: entry i becomes offset | index block << 8 | warps << 16
    int n = 0;
    for (int j = 0; j < n_bits; j++) {
      if (s_warps[j] == 0) continue;
      s_weight[n] = s_weight[j];
      s_active[n++] = s_active[j] | (j << 8) | ((int)s_warps[j] << 16);
    }
    s_count = n;
  }
  __syncthreads();
  const int n_all = s_count;
  const int o_begin = (int)((int64_t)n_all * blockIdx.z / a.splits);
  const int o_end = (int)((int64_t)n_all * (blockIdx.z + 1) / a.splits);
  const int n_step = (o_end - o_begin) * a.k_steps;

  // rows of this warp that an entry's offset has, and whether it lacks some of them anywhere
  constexpr uint32_t kAll = kRows == 32 ? 0xffffffffu : 0xffffu;
  auto rows_of = [&](int entry) {
    return (s_rows[(entry >> 8) & 0xff][warp * kRows / 32] >> (warp * kRows % 32)) & kAll;
  };
  const uint32_t lane_rows = lane < n_all ? rows_of(s_active[lane]) : 0u;
  const bool lacking = __any_sync(0xffffffffu, lane_rows != 0u && lane_rows != kAll);

  // the cursor of the copies: offset, first channel, ring stage
  int l_off = o_begin, l_k = 0, l_stage = 0;
  auto load_step = [&]() {
    float *sa = s_mem + l_stage * kStageFloats + warp * kRows * kCsPitch;
    float *sb = s_mem + l_stage * kStageFloats + BM * kCsPitch;
    const int entry = s_active[l_off];
    const int k0 = l_k;
    const int32_t *idx = s_idx + ((entry >> 8) & 0xff) * BM + warp * kRows;
    const bool mine = ((entry >> (16 + warp)) & 1) != 0;
    const float *w = a.weights + ((int64_t)s_weight[l_off] * a.K + k0) * a.N + n0;
    if constexpr (kVec) {
      if (mine) {
        const int c = (lane % (kCsK / 4)) * 4;
        const bool inside = k0 + c < a.K;
        const float *src = a.in + k0 + c;
#pragma unroll
        for (int i = 0; i < kRows / 4; i++) {
          const int r = i * 4 + lane / (kCsK / 4);
          const int row = idx[r];
          const bool valid = row >= 0 && inside;
          cs_copy_16(sa + r * kCsPitch + c, valid ? src + (int64_t)row * a.K : a.in, valid ? 16u : 0u);
        }
      }
      const int c = (tid % (BN / 4)) * 4;
      const bool inside = n0 + c < a.N;
#pragma unroll
      for (int i = 0; i < kCsK * (BN / 4) / kThreads; i++) {
        const int r = i * (kThreads / (BN / 4)) + tid / (BN / 4);
        const bool valid = inside && k0 + r < a.K;
        cs_copy_16(sb + r * BN + c, valid ? w + r * a.N + c : a.weights, valid ? 16u : 0u);
      }
    } else {
      for (int e = mine ? lane : kRows * kCsK; e < kRows * kCsK; e += 32) {
        const int r = e / kCsK, c = e % kCsK;
        const int row = idx[r];
        const bool valid = row >= 0 && k0 + c < a.K;
        cs_copy_4(sa + r * kCsPitch + c, valid ? a.in + (int64_t)row * a.K + k0 + c : a.in, valid ? 4u : 0u);
      }
      for (int e = tid; e < kCsK * BN; e += kThreads) {
        const int r = e / BN, c = e % BN;
        const bool valid = k0 + r < a.K && n0 + c < a.N;
        cs_copy_4(sb + r * BN + c, valid ? w + r * a.N + c : a.weights, valid ? 4u : 0u);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    l_k += kCsK;
    if (l_k >= a.K) { l_k = 0; l_off++; }
    if (++l_stage == kStages) l_stage = 0;
  };

  const int c = n0 + tx * 4;
  const bool vec_out = a.N % 4 == 0;
  auto store4 = [&](float *dst, float4 v) {
    if (vec_out) {
      *reinterpret_cast<float4 *>(dst) = v;
    } else {
      const float f[4] = {v.x, v.y, v.z, v.w};
      for (int j = 0; j < 4 && c + j < a.N; j++) dst[j] = f[j];
    }
  };
  float acc[8][4], sum[8][4];
  auto run = [&](auto select) {
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) acc[i][j] = sum[i][j] = 0.f;
    for (int s = 0; s < kStages - 1; s++) {
      if (s < n_step) load_step();
      else asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int off = o_begin, k0 = 0, stage = 0;
    for (int step = 0; step < n_step; step++) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
      __syncthreads();
      if (step + kStages - 1 < n_step) load_step();
      else asm volatile("cp.async.commit_group;" ::: "memory");
      const float *sb = s_mem + stage * kStageFloats + BM * kCsPitch;
      const float *sa = s_mem + stage * kStageFloats + (warp * kRows + ty) * kCsPitch;
      const int entry = s_active[off];
      const int kmax = min(kCsK, a.K - k0);                  // zeros up to a multiple of 4
      const bool complete = k0 + kCsK >= a.K;                // the last step of this offset
      if (++stage == kStages) stage = 0;
      k0 += kCsK;
      if (complete) { k0 = 0; off++; }
      if (((entry >> (16 + warp)) & 1) == 0) continue;      // none of this warp's rows
#pragma unroll 2
      for (int k = 0; k < kmax; k += 4) {
        float4 av[8], bv[4];
#pragma unroll
        for (int i = 0; i < 8; i++)
          av[i] = *reinterpret_cast<const float4 *>(sa + i * (kRows / 8) * kCsPitch + k);
#pragma unroll
        for (int j = 0; j < 4; j++) bv[j] = *reinterpret_cast<const float4 *>(sb + (k + j) * BN + tx * 4);
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const float ak[4] = {av[i].x, av[i].y, av[i].z, av[i].w};
#pragma unroll
          for (int j = 0; j < 4; j++) {
            acc[i][0] = fmaf(ak[j], bv[j].x, acc[i][0]);
            acc[i][1] = fmaf(ak[j], bv[j].y, acc[i][1]);
            acc[i][2] = fmaf(ak[j], bv[j].z, acc[i][2]);
            acc[i][3] = fmaf(ak[j], bv[j].w, acc[i][3]);
          }
        }
      }
      if (complete) {
        if (a.products != nullptr) {
          float *out = a.products + (int64_t)(entry & 0xff) * a.T * a.N;
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const int64_t r = r0 + warp * kRows + ty + i * (kRows / 8);
            if (c < a.N && r < a.T)
              store4(out + r * a.N + c, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
          }
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const bool add = !decltype(select)::value || ((rows_of(entry) >> (ty + i * (kRows / 8))) & 1u) != 0u;
#pragma unroll
          for (int j = 0; j < 4; j++) {
            if (add) sum[i][j] += acc[i][j];
            acc[i][j] = 0.f;
          }
        }
      }
    }
  };
  // A row of a warp that lacks an offset multiplies zeros, which adds NaN to it where a weight is not
  // finite.  Such a NaN must not reach it, and a select per row and offset costs 4 % of a dense
  // layer: a block whose sums end with a NaN, and where some rows lack an offset, runs once more
  // with the select.  (Products that go to the buffer are picked by row when they are added.)
  run(std::false_type());
  if (a.products == nullptr) {
    bool bad = false;
    if (lacking) {
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) bad |= sum[i][j] != sum[i][j];
    }
    if (__syncthreads_or(bad)) {
      l_off = o_begin; l_k = 0; l_stage = 0;
      run(std::true_type());
    }
  }

  if (c >= a.N || a.products != nullptr) return;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int64_t r = r0 + warp * kRows + ty + i * (kRows / 8);
    if (r >= a.T) break;
    const int64_t t = a.perm != nullptr ? (int64_t)__ldg(a.perm + r) : r;
    store4(a.out + t * a.N + c, cs_epilogue(make_float4(sum[i][0], sum[i][1], sum[i][2], sum[i][3]), a, t, c));
  }
}

// out[perm[r]] = epilogue(sum of the products of row r's pairs, in mask-row order)
__global__ void __launch_bounds__(256)
conv_simt_add_kernel(const __grid_constant__ CsArgs a) {
  begin_early();
  const int per_row = (a.N + 3) / 4;
  const int64_t total = a.T * per_row, gsz = (int64_t)gridDim.x * blockDim.x;
  const bool vec = a.N % 4 == 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gsz) {
    const int64_t r = i / per_row;
    const int c = (int)(i - r * per_row) * 4;
    float f[4] = {0.f, 0.f, 0.f, 0.f};
    for (uint32_t w = __ldg(a.tile_bits + r / 128); w != 0u; w &= w - 1u) {
      const int p = __ffs(w) - 1;
      if (__ldg(a.nbr + (int64_t)p * a.pitch + r) < 0) continue;
      const float *src = a.products + ((int64_t)p * a.T + r) * a.N + c;
      if (vec) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(src));
        f[0] += v.x; f[1] += v.y; f[2] += v.z; f[3] += v.w;
      } else {
        for (int j = 0; j < 4 && c + j < a.N; j++) f[j] += __ldg(src + j);
      }
    }
    const int64_t t = a.perm != nullptr ? (int64_t)__ldg(a.perm + r) : r;
    const float4 v = cs_epilogue(make_float4(f[0], f[1], f[2], f[3]), a, t, c);
    float *dst = a.out + t * a.N + c;
    if (vec) {
      *reinterpret_cast<float4 *>(dst) = v;
    } else {
      const float g[4] = {v.x, v.y, v.z, v.w};
      for (int j = 0; j < 4 && c + j < a.N; j++) dst[j] = g[j];
    }
  }
}

struct CsShape { int bm, bn, splits; };

// 64 x 64 sums per block; 32 x 32, one warp, where there are at most 32 output channels (such
// layers sit on the fine levels, whose maps are sparse: small tiles keep the rows with rare
// offsets from holding up others).  Offsets are spread over blocks where the tiles alone leave
// an SM without a block of 128 threads: the products then cross memory twice, which a full chip
// does not win back.
CsShape cs_shape(int64_t T, int64_t O, int64_t N) {
  CsShape s{};
  s.bn = N <= 32 ? 32 : 64;
  s.bm = N <= 32 ? 32 : 64;
  const int64_t blocks = div_up(T, s.bm) * div_up(N, s.bn);
  const int64_t fill = N <= 32 ? 4 * kNumSMs : kNumSMs;
  s.splits = blocks >= fill ? 1 : (int)std::min<int64_t>(O, div_up(3 * fill, std::max<int64_t>(blocks, 1)));
  return s;
}

template <int BM, int BN, int kStages>
mn_status launch_cs(const CsArgs &a, int64_t O, cudaStream_t st) {
  const bool vec = a.K % 4 == 0 && a.N % 4 == 0 &&
                   ((reinterpret_cast<uintptr_t>(a.in) | reinterpret_cast<uintptr_t>(a.weights)) & 15) == 0;
  constexpr size_t ring = (size_t)kStages * (BM * kCsPitch + kCsK * BN) * sizeof(float);
  const size_t smem = ring + (size_t)O * BM * sizeof(int32_t);
  const dim3 grid((unsigned)div_up(a.T, BM), (unsigned)div_up(a.N, BN), (unsigned)a.splits);
  static thread_local bool sized[kMaxDevices] = {false};
  int device = 0;
  MN_CHECK_CUDA(cudaGetDevice(&device));
  MN_CHECK_ARG(device >= 0 && device < kMaxDevices, "fp32 forward: device index %d out of range", device);
  if (!sized[device]) {
    const int most = (int)(ring + (size_t)kCsMaxOffsets * BM * sizeof(int32_t));
    MN_CHECK_CUDA(cudaFuncSetAttribute(conv_simt_kernel<BM, BN, kStages, true>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    MN_CHECK_CUDA(cudaFuncSetAttribute(conv_simt_kernel<BM, BN, kStages, false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    sized[device] = true;
  }
  if (vec) {
    MN_LAUNCH("conv_simt_kernel", st, launch_early(conv_simt_kernel<BM, BN, kStages, true>, grid, BM * BN / 32, smem, st, a));
  } else {
    MN_LAUNCH("conv_simt_kernel", st, launch_early(conv_simt_kernel<BM, BN, kStages, false>, grid, BM * BN / 32, smem, st, a));
  }
  return MN_OK;
}

}  // namespace
}  // namespace mn

using namespace mn;

extern "C" size_t mn_implicit_fp32_workspace_bytes(int64_t T, int64_t O, int64_t c_out) {
  const CsShape s = cs_shape(T, O, c_out);
  return s.splits == 1 ? 256 : (size_t)O * std::max<int64_t>(T, 1) * c_out * sizeof(float) + 256;
}

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
  const CsShape s = cs_shape(T, O, c_out);
  CsArgs a{};
  a.in = sources; a.weights = weights; a.nbr = nbr; a.tile_bits = tile_bits;
  a.order = order; a.perm = perm;
  a.scale = scale; a.shift = shift; a.residual = residual; a.relu = relu ? 1 : 0;
  a.out = targets_out;
  a.T = T; a.pitch = (int64_t)align_up((size_t)T, 128);
  a.K = (int)c_in; a.N = (int)c_out;
  a.k_steps = (int)div_up(c_in, kCsK);
  a.splits = s.splits;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (s.splits > 1) {
    Workspace ws(ws_ptr, ws_bytes);
    a.products = ws.take<float>((size_t)O * T * c_out);
    MN_CHECK_WS(ws);
  }
  MN_CHECK_ARG((reinterpret_cast<uintptr_t>(nbr) & 15) == 0 &&
                   (c_out % 4 != 0 || ((reinterpret_cast<uintptr_t>(targets_out) |
                                        reinterpret_cast<uintptr_t>(a.products)) & 15) == 0),
               "fp32 forward: the output and the neighbour table must be 16-byte aligned");
  MN_RETURN_IF(s.bn == 32 ? (launch_cs<32, 32, 2>(a, O, st)) : (launch_cs<64, 64, 3>(a, O, st)));
  if (s.splits > 1) {
    const int64_t total = T * div_up(c_out, 4);
    const int blocks = (int)std::min<int64_t>(kNumSMs * 8, div_up(total, 256));
    MN_LAUNCH("conv_simt_add_kernel", st, launch_early(conv_simt_add_kernel, blocks, 256, 0, st, a));
  }
  return MN_OK;
}
