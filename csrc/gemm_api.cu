// Host launchers for the GEMM operators.
//
//   maco_gemm        tcgen05 / TMEM / TMA pipeline (bf16 or fp16 inputs, 16-byte aligned rows)
//   maco_gemm_simt   CUDA cores: fp32 inputs (gemm_f32.cuh), and 16-bit inputs that TMA cannot address
//
// Both compute D = epilogue(alpha * op(A) · op(B)^T) with A logically [M,K] and B logically
// [N,K]; `a_mn` / `b_mn` say that the operand is stored transposed ([K,M] / [K,N] row-major).
#include "gemm_f32.cuh"
#include "host_common.h"

using namespace maco;

namespace {

// Optional per-CTA cycle counters of the stand-alone GEMM kernels (8 x int64 per CTA), off unless set.
long long* g_gemm_dbg = nullptr;

template <int BN, int STAGES, bool A_MN, bool B_MN, bool BESIDE>
int launch_gemm(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmEpilogue& epi, int K, uint32_t idesc,
                int max_ctas, uint64_t budget_ns, cudaStream_t stream) {
  using L = GemmSmemLayout<BN, STAGES>;
  auto kern = gemm_tcgen05_kernel<BN, STAGES, A_MN, B_MN, false, BESIDE>;
  static bool attr_set[64] = {};
  int dev = 0;
  MACO_CHECK_CUDA(cudaGetDevice(&dev));
  if (!attr_set[dev]) {
    MACO_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotalBytes + kEpiBlockBytes));
    attr_set[dev] = true;
  }
  const int m_tiles = (epi.M + kBM - 1) / kBM, n_tiles = (epi.N + BN - 1) / BN;
  int grid = m_tiles * n_tiles;
  int sms = maco_host::sm_count();
  if (max_ctas > 0 && max_ctas < sms) sms = max_ctas;
  if (grid > sms) grid = sms;
  if (grid <= 0) return 0;
  uint32_t* status = maco_host::status_device_ptr();
  kern<<<grid, kGemmThreads, L::kTotalBytes + kEpiBlockBytes, stream>>>(tmA, tmB, epi, K, idesc, budget_ns, status, g_gemm_dbg);
  MACO_CHECK_CUDA(cudaGetLastError());
  return 0;
}

// Products whose epilogue has a second tensor take the kernel instances that hold that epilogue.
bool has_second(const GemmEpilogue& e) {
  return e.mode == MACO_EPI_GELU_DUAL || (e.mode == MACO_EPI_GELU_BWD && e.out_type != MACO_DT_F32 && e.bias == nullptr);
}

template <int BN, int STAGES, bool BESIDE>
int dispatch_major(bool a_mn, bool b_mn, const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmEpilogue& epi,
                   int K, uint32_t idesc, int max_ctas, uint64_t budget_ns, cudaStream_t stream) {
  if (!a_mn && !b_mn) return launch_gemm<BN, STAGES, false, false, BESIDE>(tmA, tmB, epi, K, idesc, max_ctas, budget_ns, stream);
  if (!a_mn && b_mn) return launch_gemm<BN, STAGES, false, true, BESIDE>(tmA, tmB, epi, K, idesc, max_ctas, budget_ns, stream);
  if (a_mn && !b_mn) return launch_gemm<BN, STAGES, true, false, BESIDE>(tmA, tmB, epi, K, idesc, max_ctas, budget_ns, stream);
  return launch_gemm<BN, STAGES, true, true, BESIDE>(tmA, tmB, epi, K, idesc, max_ctas, budget_ns, stream);
}

// fp32 operands on the tensor cores (kind::tf32): K-major operands only, 128 x 256 tiles.
int launch_gemm_tf32(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmEpilogue& epi, int K, uint32_t idesc,
                     int max_ctas, uint64_t budget_ns, cudaStream_t stream) {
  using L = GemmSmemLayout<256, 4>;
  auto kern = gemm_tcgen05_kernel<256, 4, false, false, true, false>;
  static bool attr_set[64] = {};
  int dev = 0;
  MACO_CHECK_CUDA(cudaGetDevice(&dev));
  if (!attr_set[dev]) {
    MACO_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotalBytes + kEpiBlockBytes));
    attr_set[dev] = true;
  }
  int grid = ((epi.M + kBM - 1) / kBM) * ((epi.N + 255) / 256);
  int sms = maco_host::sm_count();
  if (max_ctas > 0 && max_ctas < sms) sms = max_ctas;
  if (grid > sms) grid = sms;
  if (grid <= 0) return 0;
  kern<<<grid, kGemmThreads, L::kTotalBytes + kEpiBlockBytes, stream>>>(tmA, tmB, epi, K, idesc, budget_ns, maco_host::status_device_ptr(), g_gemm_dbg);
  MACO_CHECK_CUDA(cudaGetLastError());
  return 0;
}

// Two-CTA tiles: clusters of two CTAs, 256 x BN per pair.
template <int BN, bool A_MN, bool B_MN, bool BESIDE>
int launch_gemm_pair(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmEpilogue& epi, int K, uint32_t idesc,
                     int max_ctas, uint64_t budget_ns, cudaStream_t stream) {
  using L = PairSmemLayout<kPairStages>;
  auto kern = gemm_tcgen05_pair_kernel<BN, A_MN, B_MN, BESIDE>;
  static bool attr_set[64] = {};
  int dev = 0;
  MACO_CHECK_CUDA(cudaGetDevice(&dev));
  if (!attr_set[dev]) {
    MACO_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kTotalBytes + kEpiBlockBytes));
    attr_set[dev] = true;
  }
  const int m_pairs = (epi.M + 2 * kBM - 1) / (2 * kBM), n_tiles = (epi.N + BN - 1) / BN;
  int pairs = m_pairs * n_tiles;
  int sms = maco_host::sm_count();
  if (max_ctas > 0 && max_ctas < sms) sms = max_ctas;
  if (pairs > sms / 2) pairs = sms / 2;
  if (pairs <= 0) return 0;
  uint32_t* status = maco_host::status_device_ptr();
  kern<<<2 * pairs, kGemmThreads, L::kTotalBytes + kEpiBlockBytes, stream>>>(tmA, tmB, epi, K, idesc, budget_ns, status, g_gemm_dbg);
  MACO_CHECK_CUDA(cudaGetLastError());
  return 0;
}

template <int BN, bool BESIDE>
int dispatch_major_pair(bool a_mn, bool b_mn, const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmEpilogue& epi,
                        int K, uint32_t idesc, int max_ctas, uint64_t budget_ns, cudaStream_t stream) {
  if (!a_mn && !b_mn) return launch_gemm_pair<BN, false, false, BESIDE>(tmA, tmB, epi, K, idesc, max_ctas, budget_ns, stream);
  if (!a_mn && b_mn) return launch_gemm_pair<BN, false, true, BESIDE>(tmA, tmB, epi, K, idesc, max_ctas, budget_ns, stream);
  if (a_mn && !b_mn) return launch_gemm_pair<BN, true, false, BESIDE>(tmA, tmB, epi, K, idesc, max_ctas, budget_ns, stream);
  return launch_gemm_pair<BN, true, true, BESIDE>(tmA, tmB, epi, K, idesc, max_ctas, budget_ns, stream);
}

// ---- CUDA-core GEMM for 16-bit operands without TMA alignment: 64x64 tile, 256 threads, 4x4 outputs per thread --------
template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }

template <typename T>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const T* __restrict__ A, const T* __restrict__ B, long long sam, long long sak, long long sbn,
                 long long sbk, GemmEpilogue e, int K) {
  __shared__ float sA[16][64 + 1];
  __shared__ float sB[16][64 + 1];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int m0 = blockIdx.y * 64, n0 = blockIdx.x * 64;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += 16) {
    for (int i = threadIdx.x; i < 64 * 16; i += 256) {
      int r = i >> 4, kk = i & 15;
      int m = m0 + r, n = n0 + r, k = k0 + kk;
      sA[kk][r] = (m < e.M && k < K) ? to_f32<T>(A[m * sam + k * sak]) : 0.f;
      sB[kk][r] = (n < e.N && k < K) ? to_f32<T>(B[n * sbn + k * sbk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { a[i] = sA[kk][ty * 4 + i]; b[i] = sB[kk][tx * 4 + i]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= e.M) continue;
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= e.N) continue;
      simt_store(e, m, n, acc[i][j]);
    }
  }
}

template <int BM, int BN, int TM, int TN>
int launch_gemm_f32(const F32Operand& A, const F32Operand& B, const GemmEpilogue& e, int K, int split, bool chained, cudaStream_t stream) {
  using T = F32Tile<BM, BN, TM, TN>;
  auto kern = gemm_f32_kernel<BM, BN, TM, TN>;
  static bool attr_set[64] = {};
  int dev = 0;
  MACO_CHECK_CUDA(cudaGetDevice(&dev));
  if (!attr_set[dev]) {
    MACO_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmemBytes));
    attr_set[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((e.N + BN - 1) / BN * split, (e.M + BM - 1) / BM);
  cfg.blockDim = dim3(T::kThreads);
  cfg.dynamicSmemBytes = T::kSmemBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {(unsigned)split, 1, 1};
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // begins when the blocks in front of it have ended
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = chained ? 2 : 1;
  MACO_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, A, B, e, K, split));
  return 0;
}

// Tile and K split of an fp32 GEMM. 64 x 64 tiles (half an LDS per FMA of the 32 x 32 ones) as soon as they give every SM
// one; below that 32 x 32, and 8 x 64 for at most eight rows, where a 32-row tile would spend three quarters of its
// FMAs on padding. While the tiles leave SMs idle the split doubles, as long as each block keeps two k-steps.
int dispatch_gemm_f32(const F32Operand& A, const F32Operand& B, const GemmEpilogue& e, int K, cudaStream_t stream, bool chained = false) {
  const long long sms = maco_host::sm_count();
  auto tiles = [&](int bm, int bn) { return (long long)((e.M + bm - 1) / bm) * ((e.N + bn - 1) / bn); };
  auto split_for = [&](long long t) {
    int s = 1;
    const int steps = (K + kF32BK - 1) / kF32BK;
    while (s < kF32MaxSplit && t * s < sms && steps >= 4 * s) s *= 2;
    return s;
  };
  if (e.M <= 8) return launch_gemm_f32<8, 64, 1, 4>(A, B, e, K, split_for(tiles(8, 64)), chained, stream);
  if (tiles(64, 64) >= sms) return launch_gemm_f32<64, 64, 4, 4>(A, B, e, K, 1, chained, stream);
  return launch_gemm_f32<32, 32, 2, 4>(A, B, e, K, split_for(tiles(32, 32)), chained, stream);
}

F32Operand f32_operand(const void* p, long long s_row, long long s_k, int rows) {
  const bool vec = s_k == 1 && s_row % 4 == 0 && (reinterpret_cast<uintptr_t>(p) & 15) == 0;
  return F32Operand{(const float*)p, s_row, s_k, rows, vec ? 1 : 0};
}

}  // namespace

extern "C" {

// One fp32 GEMM of a chain (arguments as in maco_gemm_simt).
struct MacoF32Gemm {
  const void *A, *B;
  void* D;
  const void* bias;
  long long sam, sak, sbn, sbk, ldd;
  int M, N, K, mode, bias_type, out_type;
};

// The fp32 GEMMs of a graph in order on one stream, each behind the one in front of it: one call for the host, and launches that follow
// each other as soon as the previous one's blocks have ended (no kernel here starts its successor earlier). Two layers of 32 rows: 41 us
// through one Python call each, of which 17 us a launch on the host; 14 us now.
int maco_gemm_f32_chain(const MacoF32Gemm* g, int n, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  for (int i = 0; i < n; ++i) {
    GemmEpilogue e = {};
    e.out = g[i].D; e.bias = g[i].bias; e.ld_out = g[i].ldd; e.mode = g[i].mode; e.out_type = g[i].out_type;
    e.bias_type = g[i].bias_type; e.M = g[i].M; e.N = g[i].N; e.alpha = 1.f;
    const int rc = dispatch_gemm_f32(f32_operand(g[i].A, g[i].sam, g[i].sak, g[i].M), f32_operand(g[i].B, g[i].sbn, g[i].sbk, g[i].N), e, g[i].K,
                                     stream, i > 0);
    if (rc != 0) return rc;
  }
  return 0;
}

// Cycle counters of the stand-alone GEMM kernels: `buf` (device memory, 8 x int64 per CTA, or null to switch
// them off) receives per CTA [0] producer cycles waiting for a free stage, [1] MMA warp waiting for a free
// accumulator, [2] MMA warp waiting for operands, [3] MMA warp total, [4] producer total. Word [7] of the buffer
// is read as experiment switches (results are then meaningless): 1 = epilogue does the barrier handshake only,
// 8 = the first CTA pair also logs a %globaltimer time line of its producer and MMA loops behind word 4096.
void maco_gemm_set_debug(long long* buf) { g_gemm_dbg = buf; }

// Returns 0 on success; -2 means "operands are not TMA-addressable, use maco_gemm_simt".
int maco_gemm(const void* A, const void* B, void* D, int M, int N, int K, long long lda, long long ldb,
              long long ldd, int a_mn, int b_mn, int ab_type, int out_type, int mode, const void* bias,
              int bias_type, const void* aux, long long ld_aux, int aux_type, float alpha, int bn, int max_ctas,
              double wait_budget_ms, void* stream_, int cta_pair) {
  // cta_pair: 0 = choose (two-CTA tiles when the 256 x bn tiles cover every SM pair), 1 = one-CTA tiles, 2 = two-CTA tiles
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (M <= 0 || N <= 0) return 0;
  if (ab_type != MACO_DT_BF16 && ab_type != MACO_DT_F16) { maco_host::set_error("maco_gemm: inputs must be bf16 or fp16"); return -2; }
  if (K <= 0) { maco_host::set_error("maco_gemm: K must be positive"); return -2; }
  if (bn == 0) {
    const int m_tiles = (M + kBM - 1) / kBM;
    const int sms = maco_host::sm_count();
    bn = (N <= 128 || m_tiles * ((N + 255) / 256) < sms) ? 128 : 256;
    if (mode == MACO_EPI_SWIGLU) bn = 256;
  }
  if (bn != 128 && bn != 256) { maco_host::set_error("maco_gemm: bn must be 0, 128 or 256"); return -1; }
  // Output rows are written with 16-byte vectors.
  const int out_vec = out_type == MACO_DT_F32 ? 4 : 8;
  if ((reinterpret_cast<uintptr_t>(D) & 15) != 0 || (ldd % out_vec) != 0) {
    maco_host::set_error("maco_gemm: output base and row stride must be 16-byte aligned");
    return -2;
  }
  bool pair = cta_pair == 2;
  if (cta_pair == 0) {
    // One- / two-CTA tiles, one B200, us: 2048 x 2048 x 2048 23.2 / 21.4, 1000 x 4096 x 4096 37.6 / 33.5, 2048 x 4096 x 1024 21.0 / 21.2. Short of that
    // line the two-CTA form is the faster one too where K is long (1024 x 2048 x 8192 39.1 / 33.5, 512 x 4096 x 4096 23.3 / 21.2; 1024 x 2048 x
    // 2048 15.5 / 15.4): callers with such products ask for it.
    const int sms = maco_host::sm_count();
    pair = ((M + 255) / 256) * ((N + bn - 1) / bn) >= sms / 2;
  }
  CUtensorMap tmA, tmB;
  int r;
  if (!a_mn) r = maco_host::encode_tmap_2d(&tmA, A, 2, M, K, lda * 2, kBK, kBM);
  else       r = maco_host::encode_tmap_2d(&tmA, A, 2, K, M, lda * 2, 64, kBK);
  if (r != 0) return r == -2 ? -2 : -1;
  if (!b_mn) r = maco_host::encode_tmap_2d(&tmB, B, 2, N, K, ldb * 2, kBK, pair ? bn / 2 : bn);
  else       r = maco_host::encode_tmap_2d(&tmB, B, 2, K, N, ldb * 2, 64, kBK);
  if (r != 0) return r == -2 ? -2 : -1;
  GemmEpilogue e;
  e.out = D; e.bias = bias; e.aux = aux; e.ld_out = ldd; e.ld_aux = ld_aux; e.mode = mode; e.out_type = out_type;
  e.bias_type = bias_type; e.aux_type = aux_type; e.M = M; e.N = N; e.alpha = alpha; e.aux_pack = 0;
  const uint64_t budget_ns = (uint64_t)((wait_budget_ms > 0 ? wait_budget_ms : 2000.0) * 1e6);
  const bool second = has_second(e);
  if (pair) {
    const uint32_t idesc2 = make_idesc(ab_type == MACO_DT_BF16 ? 1u : 0u, 2 * kBM, bn, a_mn ? 1u : 0u, b_mn ? 1u : 0u);
    auto run = bn == 256 ? (second ? dispatch_major_pair<256, true> : dispatch_major_pair<256, false>)
                         : (second ? dispatch_major_pair<128, true> : dispatch_major_pair<128, false>);
    return run(a_mn, b_mn, tmA, tmB, e, K, idesc2, max_ctas, budget_ns, stream);
  }
  const uint32_t idesc = make_idesc(ab_type == MACO_DT_BF16 ? 1u : 0u, kBM, bn, a_mn ? 1u : 0u, b_mn ? 1u : 0u);
  auto run = bn == 256 ? (second ? dispatch_major<256, 4, true> : dispatch_major<256, 4, false>)
                       : (second ? dispatch_major<128, 6, true> : dispatch_major<128, 6, false>);
  return run(a_mn, b_mn, tmA, tmB, e, K, idesc, max_ctas, budget_ns, stream);
}

// fp32 inputs on the tensor cores as TF32 (10-bit mantissa: an opt-in, the default fp32 path is maco_gemm_simt).
// A [M, K] and B [N, K] row-major fp32 with 16-byte aligned rows; same epilogues as maco_gemm.
// Returns -2 when the operands are not TMA-addressable.
int maco_gemm_tf32(const void* A, const void* B, void* D, int M, int N, int K, long long lda, long long ldb, long long ldd,
                   int out_type, int mode, const void* bias, int bias_type, const void* aux, long long ld_aux,
                   int aux_type, float alpha, int max_ctas, double wait_budget_ms, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || mode == MACO_EPI_SWIGLU) { maco_host::set_error("maco_gemm_tf32: K must be positive; no SwiGLU epilogue"); return -2; }
  const int out_vec = out_type == MACO_DT_F32 ? 4 : 8;
  if ((reinterpret_cast<uintptr_t>(D) & 15) != 0 || (ldd % out_vec) != 0) {
    maco_host::set_error("maco_gemm_tf32: output base and row stride must be 16-byte aligned");
    return -2;
  }
  CUtensorMap tmA, tmB;
  int r = maco_host::encode_tmap_2d(&tmA, A, 4, M, K, lda * 4, kBK / 2, kBM);
  if (r != 0) return r == -2 ? -2 : -1;
  r = maco_host::encode_tmap_2d(&tmB, B, 4, N, K, ldb * 4, kBK / 2, 256);
  if (r != 0) return r == -2 ? -2 : -1;
  GemmEpilogue e;
  e.out = D; e.bias = bias; e.aux = aux; e.ld_out = ldd; e.ld_aux = ld_aux; e.mode = mode; e.out_type = out_type;
  e.bias_type = bias_type; e.aux_type = aux_type; e.M = M; e.N = N; e.alpha = alpha; e.aux_pack = 0;
  const uint64_t budget_ns = (uint64_t)((wait_budget_ms > 0 ? wait_budget_ms : 2000.0) * 1e6);
  return launch_gemm_tf32(tmA, tmB, e, K, make_idesc(2u, kBM, 256, 0u, 0u), max_ctas, budget_ns, stream);
}

// Element strides: A(m,k) = A[m*sam + k*sak], B(n,k) = B[n*sbn + k*sbk].
int maco_gemm_simt(const void* A, const void* B, void* D, int M, int N, int K, long long sam, long long sak,
                   long long sbn, long long sbk, long long ldd, int ab_type, int out_type, int mode, const void* bias,
                   int bias_type, const void* aux, long long ld_aux, int aux_type, float alpha, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (M <= 0 || N <= 0) return 0;
  GemmEpilogue e;
  e.out = D; e.bias = bias; e.aux = aux; e.ld_out = ldd; e.ld_aux = ld_aux; e.mode = mode; e.out_type = out_type;
  e.bias_type = bias_type; e.aux_type = aux_type; e.M = M; e.N = N; e.alpha = alpha; e.aux_pack = 0;
  if (ab_type == MACO_DT_F32) {
    return dispatch_gemm_f32(f32_operand(A, sam, sak, M), f32_operand(B, sbn, sbk, N), e, K, stream);
  }
  dim3 grid((N + 63) / 64, (M + 63) / 64);
  if (ab_type == MACO_DT_F16)
    gemm_simt_kernel<__half><<<grid, 256, 0, stream>>>((const __half*)A, (const __half*)B, sam, sak, sbn, sbk, e, K);
  else
    gemm_simt_kernel<__nv_bfloat16><<<grid, 256, 0, stream>>>((const __nv_bfloat16*)A, (const __nv_bfloat16*)B, sam, sak, sbn, sbk, e, K);
  MACO_CHECK_CUDA(cudaGetLastError());
  return 0;
}

}  // extern "C"
