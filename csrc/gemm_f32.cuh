// fp32 GEMM on the CUDA cores, for inputs that keep all their bits:  D = epilogue(A · B^T), any strides.
//
// Bound by latency at the sizes it is called for (tens of rows): a 64 x 64 tile per block with one synchronous 16-deep
// load per step left 32 x 1024 x 512 to 16 of 148 SMs and took about 100 us, against a few us of weight traffic. Here
//  * the tile shrinks with the problem, and the blocks of one cluster (up to 8) split K and add their partial
//    tiles through distributed shared memory, in rank order: no workspace, no second launch, same sum every time;
//  * k-steps of 32 stream through a cp.async pipeline of three to six stages: 16 bytes a copy where K is contiguous and
//    rows are 16-byte aligned, else 4 bytes a copy along whichever dimension is contiguous;
//  * a thread owns rows ty + i * TY and columns tx + j * TX and reads four k at once: eight consecutive rows of pitch
//    36 floats fall into different banks, so a warp's LDS.128 is one wavefront (4 x 4 outputs: 8 reads for 64 FMAs).
// One B200, launch included (16 us of it is the host): 32 x 1024 x 512 75 -> 17 us, 32 x 512 x 1024 144 -> 17 us,
// 1 x 2048 x 2048 261 -> 17 us (35 us with three stages instead of six), 512 x 2048 x 2048 379 -> 148 us.
#pragma once
#include "gemm_tcgen05.cuh"

namespace maco {

constexpr int kF32BK = 32, kF32Pitch = kF32BK + 4, kF32MaxSplit = 8;

struct F32Operand {
  const float* p;
  long long s_row, s_k;     // element strides
  int rows, vec;            // vec: 16-byte copies are aligned and k-contiguous
};

template <int ROWS, int NT>
MACO_DEVICE void f32_load_stage(float* dst, const F32Operand& o, int row0, int k0, int k_end, int tid) {
  if (o.vec) {
#pragma unroll
    for (int i = tid; i < ROWS * (kF32BK / 4); i += NT) {
      const int r = i / (kF32BK / 4), k = k0 + (i % (kF32BK / 4)) * 4;
      const int left = (row0 + r < o.rows) ? min(4, k_end - k) : 0;
      const float* src = left > 0 ? o.p + (row0 + r) * o.s_row + k : o.p;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                   :: "r"(smem_u32(dst + r * kF32Pitch + (k - k0))), "l"(src), "r"(left > 0 ? left * 4 : 0) : "memory");
    }
  } else {
#pragma unroll 4
    for (int i = tid; i < ROWS * kF32BK; i += NT) {
      const int r = o.s_k == 1 ? i / kF32BK : i % ROWS, kk = o.s_k == 1 ? i % kF32BK : i / ROWS;
      const bool in = row0 + r < o.rows && k0 + kk < k_end;
      const float* src = in ? o.p + (row0 + r) * o.s_row + (k0 + kk) * o.s_k : o.p;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                   :: "r"(smem_u32(dst + r * kF32Pitch + kk)), "l"(src), "r"(in ? 4 : 0) : "memory");
    }
  }
}

MACO_DEVICE void simt_store(const GemmEpilogue& e, int m, int n, float acc) {
  float v = acc * e.alpha;
  if (e.bias != nullptr) v += epi_bias(e, n);
  if (e.mode == MACO_EPI_GELU) v = gelu_tanh_f32(v);
  else if (e.mode == MACO_EPI_SILU) v = silu(v);
  else if (e.mode == MACO_EPI_GELU_BWD) v *= gelu_tanh_grad_f32(epi_load_aux(e, m, n));
  else if (e.mode == MACO_EPI_RESIDUAL) v += epi_load_aux(e, m, n);
  const long long o = (long long)m * e.ld_out + n;
  if (e.out_type == MACO_DT_F32) {
    float* p = reinterpret_cast<float*>(e.out) + o;
    *p = (e.mode == MACO_EPI_F32_ACC) ? *p + v : v;
  } else if (e.out_type == MACO_DT_F16) {
    reinterpret_cast<__half*>(e.out)[o] = __float2half_rn(v);
  } else {
    reinterpret_cast<__nv_bfloat16*>(e.out)[o] = __float2bfloat16_rn(v);
  }
}

template <int BM, int BN, int TM, int TN>
struct F32Tile {
  static constexpr int kStages = BM * BN > 2048 ? 3 : 6;      // small tiles: more loads in flight; 55 to 62 KB either way
  static constexpr int kTX = BN / TN, kTY = BM / TM, kThreads = kTX * kTY;
  static constexpr int kStageFloats = (BM + BN) * kF32Pitch;
  static constexpr int kSmemBytes = kStages * kStageFloats * 4;
  static_assert(kTX % 8 == 0 && kTY % 4 == 0 && BM * BN <= kStages * kStageFloats, "tile shape");
};

// grid: x = column tiles * split (the cluster is the `split` blocks of one tile), y = row tiles
template <int BM, int BN, int TM, int TN>
__global__ void __launch_bounds__(F32Tile<BM, BN, TM, TN>::kThreads)
gemm_f32_kernel(F32Operand A, F32Operand B, GemmEpilogue e, int K, int split) {
  using T = F32Tile<BM, BN, TM, TN>;
  constexpr int NT = T::kThreads;
  extern __shared__ __align__(16) float f32_smem[];
  asm volatile("griddepcontrol.wait;" ::: "memory");   // (launched behind another one of a chain: its results are complete)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = (lane & 7) + 8 * (warp % (T::kTX / 8)), ty = (lane >> 3) + 4 * (warp / (T::kTX / 8));
  const int rank = blockIdx.x % split;
  const int m0 = blockIdx.y * BM, n0 = (int)(blockIdx.x / split) * BN;
  const int steps_all = (K + kF32BK - 1) / kF32BK, per = (steps_all + split - 1) / split;
  const int k_begin = rank * per * kF32BK, k_end = min(K, k_begin + per * kF32BK);
  const int steps = k_end > k_begin ? (k_end - k_begin + kF32BK - 1) / kF32BK : 0;
  auto load = [&](int i) {
    if (i < steps) {
      float* st = f32_smem + (i % T::kStages) * T::kStageFloats;
      f32_load_stage<BM, NT>(st, A, m0, k_begin + i * kF32BK, k_end, tid);
      f32_load_stage<BN, NT>(st + BM * kF32Pitch, B, n0, k_begin + i * kF32BK, k_end, tid);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[TM][TN] = {};
  for (int i = 0; i < T::kStages - 1; ++i) load(i);
  for (int i = 0; i < steps; ++i) {
    asm volatile("cp.async.wait_group %0;" :: "n"(T::kStages - 2) : "memory");
    __syncthreads();                                  // step i has landed; step i - 1's stage is free
    load(i + T::kStages - 1);
    const float* sa = f32_smem + (i % T::kStages) * T::kStageFloats;
    const float* sb = sa + BM * kF32Pitch;
#pragma unroll
    for (int k = 0; k < kF32BK; k += 4) {
      float4 a[TM], b[TN];
#pragma unroll
      for (int r = 0; r < TM; ++r) a[r] = *reinterpret_cast<const float4*>(sa + (ty + r * T::kTY) * kF32Pitch + k);
#pragma unroll
      for (int c = 0; c < TN; ++c) b[c] = *reinterpret_cast<const float4*>(sb + (tx + c * T::kTX) * kF32Pitch + k);
#pragma unroll
      for (int r = 0; r < TM; ++r)
#pragma unroll
        for (int c = 0; c < TN; ++c) {
          acc[r][c] = fmaf(a[r].x, b[c].x, acc[r][c]);
          acc[r][c] = fmaf(a[r].y, b[c].y, acc[r][c]);
          acc[r][c] = fmaf(a[r].z, b[c].z, acc[r][c]);
          acc[r][c] = fmaf(a[r].w, b[c].w, acc[r][c]);
        }
    }
  }
  if (split == 1) {
#pragma unroll
    for (int r = 0; r < TM; ++r)
#pragma unroll
      for (int c = 0; c < TN; ++c) {
        const int m = m0 + ty + r * T::kTY, n = n0 + tx + c * T::kTX;
        if (m < e.M && n < e.N) simt_store(e, m, n, acc[r][c]);
      }
    return;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                                    // the stages are read and no copy is in flight: they hold the partial tile now
#pragma unroll
  for (int r = 0; r < TM; ++r)
#pragma unroll
    for (int c = 0; c < TN; ++c) f32_smem[(ty + r * T::kTY) * BN + tx + c * T::kTX] = acc[r][c];
  cluster_arrive();
  cluster_wait();
  const uint32_t part = smem_u32(f32_smem);
  for (int i = rank * NT + tid; i < BM * BN; i += split * NT) {
    float v[kF32MaxSplit];
#pragma unroll
    for (int s = 0; s < kF32MaxSplit; ++s) {
      v[s] = 0.f;
      if (s < split) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v[s]) : "r"(mapa_u32(part + i * 4, s)) : "memory");
    }
    float sum = v[0];
#pragma unroll
    for (int s = 1; s < kF32MaxSplit; ++s) if (s < split) sum += v[s];
    const int m = m0 + i / BN, n = n0 + i % BN;
    if (m < e.M && n < e.N) simt_store(e, m, n, sum);
  }
  cluster_arrive();                                   // no block leaves while another may still read its partial tile
  cluster_wait();
}

}  // namespace maco
