// Stand-alone launches of the element-wise / row-wise operators.
#include "elementwise.cuh"
#include "row_tasks.cuh"
#include "host_common.h"

using namespace maco;

namespace {

// What the two kernels below do not take: RoPE, row-wise operators on rows that are not whole aligned vectors or are
// longer than the register form holds, strided operands. One CTA per chunk of rows.
__global__ void __launch_bounds__(128, 4) elt_kernel(uint32_t type, MacoEltArgs a, int rows_per_cta) {
  MacoEltArgs mine = a;
  mine.row0 = a.row0 + blockIdx.x * rows_per_cta;
  int left = a.rows - blockIdx.x * rows_per_cta;
  mine.rows = left < rows_per_cta ? left : rows_per_cta;
  if (mine.rows <= 0) return;
  elt_run(type, mine, threadIdx.x, blockDim.x);
}

// RMSNorm, LayerNorm and softmax, bound by memory: the row is fetched once, with all loads of a thread in flight, and stays
// in registers between the reduction and the result. TEAM threads own a row: a warp up to 64 vectors, 128 threads
// up to 1024, 256 up to 2048; V vectors a thread. One B200, 8192 x 5120 bf16, against one warp per row reading it twice: RMSNorm 42 -> 30 us
// (5.5 TB/s), LayerNorm 51 -> 36 us, softmax 58 -> 38 us; 16384 x 64: 48 -> 12 us (the call's host time).
constexpr int kRowMaxV = 8;
template <int TEAM>
__device__ __forceinline__ float team_reduce(float v, bool max, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float w = __shfl_xor_sync(0xffffffffu, v, o);
    v = max ? fmaxf(v, w) : v + w;
  }
  if constexpr (TEAM > 32) {
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = red[0];
#pragma unroll
    for (int i = 1; i < TEAM / 32; ++i) v = max ? fmaxf(v, red[i]) : v + red[i];
  }
  return v;
}

template <int DT, int OP, int TEAM, int V>
__global__ void __launch_bounds__(TEAM > 128 ? TEAM : 128) row_kernel(MacoEltArgs a) {
  using Vec = VecOf<DT>;
  __shared__ float red[2][8];                       // one per reduction of a row (one row per team)
  const int t = threadIdx.x % TEAM;
  const long long r = TEAM < 128 ? (long long)blockIdx.x * (128 / TEAM) + threadIdx.x / TEAM : blockIdx.x;
  if (r >= a.rows) return;                          // (whole warps; from TEAM = 128 on the grid is exact)
  const int n = a.cols / Vec::kN;
  const uint4* x = reinterpret_cast<const uint4*>(a.in0) + r * n;
  uint4* out = reinterpret_cast<uint4*>(a.out) + r * n;
  uint4 raw[V];
#pragma unroll
  for (int i = 0; i < V; ++i) if (t + i * TEAM < n) raw[i] = x[t + i * TEAM];
  float s = 0.f, mx = -INFINITY, mean = 0.f, scale;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    if (t + i * TEAM < n) {
      const Vec v = vec_unpack<DT>(raw[i]);
#pragma unroll
      for (int j = 0; j < Vec::kN; ++j) {
        if constexpr (OP == MACO_TASK_RMSNORM) s += v.v[j] * v.v[j];
        else if constexpr (OP == MACO_TASK_LAYERNORM) s += v.v[j];
        else mx = fmaxf(mx, v.v[j]);
      }
    }
  }
  if constexpr (OP == MACO_TASK_RMSNORM) {
    scale = rsqrtf(team_reduce<TEAM>(s, false, red[0]) / a.cols + a.f0);
  } else {
    if constexpr (OP == MACO_TASK_LAYERNORM) mean = team_reduce<TEAM>(s, false, red[0]) / a.cols;
    else mx = team_reduce<TEAM>(mx, true, red[0]);
    s = 0.f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      if (t + i * TEAM < n) {
        const Vec v = vec_unpack<DT>(raw[i]);
#pragma unroll
        for (int j = 0; j < Vec::kN; ++j) {
          if constexpr (OP == MACO_TASK_LAYERNORM) s += (v.v[j] - mean) * (v.v[j] - mean);
          else s += __expf(v.v[j] - mx);
        }
      }
    }
    s = team_reduce<TEAM>(s, false, red[1]);
    scale = OP == MACO_TASK_LAYERNORM ? rsqrtf(s / a.cols + a.f0) : 1.f / s;
  }
  const uint4* w = reinterpret_cast<const uint4*>(a.in1);
  const uint4* b = reinterpret_cast<const uint4*>(a.in2);
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int c = t + i * TEAM;
    if (c < n) {
      Vec v = vec_unpack<DT>(raw[i]);
      if constexpr (OP == MACO_TASK_SOFTMAX) {
#pragma unroll
        for (int j = 0; j < Vec::kN; ++j) v.v[j] = __expf(v.v[j] - mx) * scale;
      } else {
        const Vec wv = vec_unpack<DT>(w[c]);
        if constexpr (OP == MACO_TASK_RMSNORM) {
#pragma unroll
          for (int j = 0; j < Vec::kN; ++j) v.v[j] = v.v[j] * scale * wv.v[j];
        } else {
          const Vec bv = vec_unpack<DT>(b[c]);
#pragma unroll
          for (int j = 0; j < Vec::kN; ++j) v.v[j] = (v.v[j] - mean) * scale * wv.v[j] + bv.v[j];
        }
      }
      out[c] = vec_pack<DT>(v);
    }
  }
}

template <int DT, int OP>
bool launch_rows(const MacoEltArgs& a, cudaStream_t stream) {
  const int n = a.cols / VecOf<DT>::kN;
  const unsigned warp_rows = ((unsigned)a.rows + 3) / 4;
  if (n <= 32) row_kernel<DT, OP, 32, 1><<<warp_rows, 128, 0, stream>>>(a);
  else if (n <= 64) row_kernel<DT, OP, 32, 2><<<warp_rows, 128, 0, stream>>>(a);
  else if (n <= 128) row_kernel<DT, OP, 128, 1><<<a.rows, 128, 0, stream>>>(a);
  else if (n <= 256) row_kernel<DT, OP, 128, 2><<<a.rows, 128, 0, stream>>>(a);
  else if (n <= 512) row_kernel<DT, OP, 128, 4><<<a.rows, 128, 0, stream>>>(a);
  else if (n <= 768) row_kernel<DT, OP, 128, 6><<<a.rows, 128, 0, stream>>>(a);
  else if (n <= 128 * kRowMaxV) row_kernel<DT, OP, 128, kRowMaxV><<<a.rows, 128, 0, stream>>>(a);
  else if (n <= 256 * kRowMaxV) row_kernel<DT, OP, 256, kRowMaxV><<<a.rows, 256, 0, stream>>>(a);
  else return false;
  return true;
}

template <int DT>
bool launch_rows_op(uint32_t type, const MacoEltArgs& a, cudaStream_t stream) {
  switch (type) {
    case MACO_TASK_RMSNORM: return launch_rows<DT, MACO_TASK_RMSNORM>(a, stream);
    case MACO_TASK_LAYERNORM: return launch_rows<DT, MACO_TASK_LAYERNORM>(a, stream);
    case MACO_TASK_SOFTMAX: return launch_rows<DT, MACO_TASK_SOFTMAX>(a, stream);
    default: return false;
  }
}

// Point-wise operators over contiguous tensors, bound by memory: the tensor is one run of 16-byte vectors whatever its row
// length (rows of odd length went element by element before), and its last few elements go one by one. One B200:
// GELU of 8192 x 5120 bf16 50 -> 29 us, of 16384 x 4001 669 -> 44 us; ADD of 16384 x 4001 1041 -> 60 us.
constexpr int kFlatU = 4;                            // vectors a thread has in flight per operand
template <int DT, int OP>
__global__ void __launch_bounds__(256) flat_kernel(const void* in0, const void* in1, void* out, long long total, float f0, float f1) {
  using Vec = VecOf<DT>;
  constexpr bool bin = elt_is_binary(OP);
  const long long nvec = total / Vec::kN, first = (long long)blockIdx.x * (256 * kFlatU) + threadIdx.x;
  const uint4* x = reinterpret_cast<const uint4*>(in0);
  const uint4* y = reinterpret_cast<const uint4*>(in1);
  uint4 xr[kFlatU], yr[kFlatU];
#pragma unroll
  for (int u = 0; u < kFlatU; ++u) if (first + u * 256 < nvec) xr[u] = x[first + u * 256];
  if constexpr (bin) {
#pragma unroll
    for (int u = 0; u < kFlatU; ++u) if (first + u * 256 < nvec) yr[u] = y[first + u * 256];
  }
#pragma unroll
  for (int u = 0; u < kFlatU; ++u) {
    if (first + u * 256 < nvec) {
      Vec v = vec_unpack<DT>(xr[u]);
      Vec w;
      if constexpr (bin) w = vec_unpack<DT>(yr[u]);
#pragma unroll
      for (int j = 0; j < Vec::kN; ++j) v.v[j] = elt_op<DT, OP>(v.v[j], bin ? w.v[j] : 0.f, f0, f1);
      reinterpret_cast<uint4*>(out)[first + u * 256] = vec_pack<DT>(v);
    }
  }
  const long long rest = nvec * Vec::kN + threadIdx.x;
  if (blockIdx.x == gridDim.x - 1 && rest < total)
    store1(out, rest, DT, elt_op<DT, OP>(load1(in0, rest, DT), bin ? load1(in1, rest, DT) : 0.f, f0, f1));
}

// Start of an MLP's backward pass, dz = f * (a - target) * gelu'(z), bound by memory (four tensors once each).
// It was two passes of tasks in the persistent kernel with a rounded tensor in between, whose 28 KB of staging per SM held each at
// about 2 TB/s: 320 us of the backward pass for 8192 x 4096.
template <int DT>
__global__ void __launch_bounds__(256) mse_gelu_bwd_kernel(const uint4* a, const uint4* target, const uint4* z, uint4* dz, long long nvec, float f) {
  using Vec = VecOf<DT>;
  const long long first = (long long)blockIdx.x * (256 * 2) + threadIdx.x;
  uint4 ar[2], tr[2], zr[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) if (first + u * 256 < nvec) { ar[u] = a[first + u * 256]; tr[u] = target[first + u * 256]; zr[u] = z[first + u * 256]; }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    if (first + u * 256 < nvec) {
      const Vec av = vec_unpack<DT>(ar[u]), tv = vec_unpack<DT>(tr[u]);
      Vec v = vec_unpack<DT>(zr[u]);
#pragma unroll
      for (int j = 0; j < Vec::kN; ++j) v.v[j] = f * (av.v[j] - tv.v[j]) * gelu_tanh_grad(v.v[j]);
      dz[first + u * 256] = vec_pack<DT>(v);
    }
  }
}

template <int DT>
bool launch_flat(uint32_t type, const MacoEltArgs& a, cudaStream_t stream) {
  const long long total = (long long)a.rows * a.cols, per = 256ll * kFlatU * VecOf<DT>::kN;
  const long long grid = (total + per - 1) / per;
  if (grid > 0x7fffffffll) return false;
#define MACO_FLAT_CASE(T) \
  case T: flat_kernel<DT, T><<<(unsigned)grid, 256, 0, stream>>>(a.in0, a.in1, a.out, total, a.f0, a.f1); return true;
  switch (type) {
    MACO_FLAT_CASE(MACO_TASK_GELU)
    MACO_FLAT_CASE(MACO_TASK_SILU)
    MACO_FLAT_CASE(MACO_TASK_SCALE)
    MACO_FLAT_CASE(MACO_TASK_ADD)
    MACO_FLAT_CASE(MACO_TASK_SILU_GATE)
    MACO_FLAT_CASE(MACO_TASK_GELU_BWD)
    MACO_FLAT_CASE(MACO_TASK_AXPBY)
    MACO_FLAT_CASE(MACO_TASK_COPY)
    default: return false;
  }
#undef MACO_FLAT_CASE
}

// Contiguous rows and 16-byte aligned bases take the kernels above; a row-wise operator also needs rows of whole vectors
// (so that every row, and the parameters beside it, starts on a vector).
bool launch_contiguous(uint32_t type, const MacoEltArgs& a, cudaStream_t stream) {
  auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  if (a.ld_in != a.cols || a.ld_out != a.cols || !aligned(a.in0) || !aligned(a.in1) || !aligned(a.in2) || !aligned(a.out)) return false;
  const bool rowwise = type == MACO_TASK_RMSNORM || type == MACO_TASK_LAYERNORM || type == MACO_TASK_SOFTMAX;
  if (rowwise) {
    if (a.cols % (a.dtype == MACO_DT_F32 ? 4 : 8) != 0) return false;
    if (a.dtype == MACO_DT_BF16) return launch_rows_op<MACO_DT_BF16>(type, a, stream);
    if (a.dtype == MACO_DT_F16) return launch_rows_op<MACO_DT_F16>(type, a, stream);
    return launch_rows_op<MACO_DT_F32>(type, a, stream);
  }
  if (a.dtype == MACO_DT_BF16) return launch_flat<MACO_DT_BF16>(type, a, stream);
  if (a.dtype == MACO_DT_F16) return launch_flat<MACO_DT_F16>(type, a, stream);
  return launch_flat<MACO_DT_F32>(type, a, stream);
}

}  // namespace

extern "C" int maco_elementwise(int type, const void* in0, const void* in1, const void* in2, void* out, int rows,
                                int cols, int dtype, int ld_in, int ld_out, float f0, float f1, int i0, int i1,
                                void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (rows <= 0 || cols <= 0) return 0;
  MacoEltArgs a;
  a.in0 = in0; a.in1 = in1; a.in2 = in2; a.out = out; a.row0 = 0; a.rows = rows; a.cols = cols; a.dtype = dtype;
  a.ld_in = ld_in; a.ld_out = ld_out; a.f0 = f0; a.f1 = f1; a.i0 = i0; a.i1 = i1;
  if (launch_contiguous((uint32_t)type, a, stream)) {
    MACO_CHECK_CUDA(cudaGetLastError());
    return 0;
  }
  const int sms = maco_host::sm_count();
  // 128-thread CTAs, four resident per SM; several waves so that the tail is short.
  long long work = (long long)rows * cols;
  int target_ctas = (int)((work + 16383) / 16384);
  if (target_ctas > sms * 16) target_ctas = sms * 16;
  if (target_ctas < 1) target_ctas = 1;
  int rows_per_cta = (rows + target_ctas - 1) / target_ctas;
  if (rows_per_cta < 1) rows_per_cta = 1;
  int grid = (rows + rows_per_cta - 1) / rows_per_cta;
  elt_kernel<<<grid, 128, 0, stream>>>((uint32_t)type, a, rows_per_cta);
  MACO_CHECK_CUDA(cudaGetLastError());
  return 0;
}

// `total` elements of 16-bit tensors, a multiple of 8; all four bases 16-byte aligned.
extern "C" int maco_mse_gelu_bwd(const void* a, const void* target, const void* z, void* dz, long long total, int dtype, float f, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (total <= 0) return 0;
  const uintptr_t bases = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(target) | reinterpret_cast<uintptr_t>(z) | reinterpret_cast<uintptr_t>(dz);
  const long long nvec = total / 8, grid = (nvec + 511) / 512;
  if (total % 8 != 0 || (bases & 15) != 0 || grid > 0x7fffffffll || (dtype != MACO_DT_BF16 && dtype != MACO_DT_F16)) {
    maco_host::set_error("maco_mse_gelu_bwd: 16-bit tensors of whole, aligned 16-byte vectors only");
    return -1;
  }
  auto v = [](const void* p) { return reinterpret_cast<const uint4*>(p); };
  if (dtype == MACO_DT_BF16) mse_gelu_bwd_kernel<MACO_DT_BF16><<<(unsigned)grid, 256, 0, stream>>>(v(a), v(target), v(z), reinterpret_cast<uint4*>(dz), nvec, f);
  else mse_gelu_bwd_kernel<MACO_DT_F16><<<(unsigned)grid, 256, 0, stream>>>(v(a), v(target), v(z), reinterpret_cast<uint4*>(dz), nvec, f);
  MACO_CHECK_CUDA(cudaGetLastError());
  return 0;
}
