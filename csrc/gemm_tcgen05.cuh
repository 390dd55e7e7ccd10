// Warp-specialised tcgen05 GEMM pipeline for sm_100a.
//
//   D[M,N] = epilogue( A[M,K] · B[N,K]^T )      A, B: bf16 or fp16;  accumulate fp32 in TMEM
//
// This replaces the reference's scalar one-thread-per-output GEMM task
// (maco/csrc/maco_worker.cuh:36-57) and the torch.mm call its live runtime makes
// (maco/task_graph/runtime.py:188-209).
//
// One CTA = 6 warps:
//   warp 0      TMA producer   cp.async.bulk.tensor tiles -> 128B-swizzled smem ring
//   warp 1      MMA issuer     one elected lane issues tcgen05.mma (128 x BN x 16) into a TMEM accumulator
//   warps 2..5  epilogue       tcgen05.ld the accumulator (one TMEM lane quarter per warp),
//                              apply the fused epilogue, store to global (local or peer memory)
// The accumulator is double buffered in TMEM (2 x BN columns) so the epilogue of tile i runs
// under the main loop of tile i+1. All hand-offs are mbarriers; every wait is bounded and a
// wait that runs out sets a CTA-wide abort word, after which all roles drain and the CTA frees
// its TMEM and returns.
//
// Warps 0 and 1 run converged and elect the lane that issues (elect.sync) in each k-block. tcgen05.mma, cp.async.bulk.tensor and their
// operands live on the warp-uniform datapath: in code that one lane runs under `lane == 0` the compiler cannot know that, and serialises
// every such instruction over the lanes that may be active, about 100 cycles apiece. A k-block then took 0.32 us to issue whatever its size,
// more than its products (0.13 us for 128 x 128) and more than the loads. One B200, lane 0 / elected lane, us: 1024 x 2048 x 8192 in
// 256 x 128 tiles 58 / 34, 8192 x 4096 x 4096 in 256 x 256 tiles 205 / 185 (one-CTA tiles 205 / 195).
//
// Operands may be K-major (row-major [rows, K]) or MN-major (row-major [K, rows]); the latter is
// what the backward GEMMs need (wgrad = dY^T · X contracts over the token dimension).
#pragma once
#include <cuda.h>
#include "maco_atoms.cuh"
#include "maco_types.h"

namespace maco {

constexpr int kBM = 128;       // tile rows  (UMMA M)
constexpr int kBK = 64;        // k-block: 64 x 2 B = one 128-byte swizzle row
constexpr int kUmmaK = 16;     // K per tcgen05.mma for 16-bit inputs
constexpr int kGemmThreads = 192;

// BN is the tile width a task uses; SBN (>= BN) sizes the ring's stages, so tasks of different
// BN can share one ring with identical stage addresses and barrier phases.
template <int BN, int STAGES, int SBN = BN>
struct GemmSmemLayout {
  static constexpr int kABytes = kBM * kBK * 2;
  static constexpr int kBBytes = BN * kBK * 2;
  static constexpr int kLoadBytes = kABytes + kBBytes;          // bytes one k-step brings in
  static constexpr int kStageBytes = kABytes + SBN * kBK * 2;   // distance between stages
  static constexpr int kRingBytes = STAGES * kStageBytes;
  // after the ring: full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2], tmem slot, abort word
  static constexpr int kCtrlBytes = 256;
  static constexpr int kTotalBytes = kRingBytes + kCtrlBytes + 1024;   // +1024: manual alignment slack
  static_assert(2 * STAGES * 8 + 4 * 8 + 16 <= kCtrlBytes, "control block too small");
};

struct GemmCtrl {
  uint64_t* full;        // [STAGES]  TMA -> MMA
  uint64_t* empty;       // [STAGES]  MMA -> TMA
  uint64_t* tmem_full;   // [2]       MMA -> epilogue
  uint64_t* tmem_empty;  // [2]       epilogue -> MMA
  uint32_t* tmem_slot;
  volatile uint32_t* abort_word;
};

template <int BN, int STAGES, int SBN = BN>
MACO_DEVICE GemmCtrl gemm_ctrl(uint8_t* smem_base) {
  using L = GemmSmemLayout<BN, STAGES, SBN>;
  GemmCtrl c;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_base + L::kRingBytes);
  c.full = bars;
  c.empty = bars + STAGES;
  c.tmem_full = bars + 2 * STAGES;
  c.tmem_empty = bars + 2 * STAGES + 2;
  c.tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  c.abort_word = reinterpret_cast<volatile uint32_t*>(c.tmem_slot + 1);
  return c;
}

// Raster order: groups of 8 tile-rows sweep all tile-columns, so CTAs that run together
// share A row-blocks and B column-blocks in L2.
MACO_DEVICE void gemm_tile_coords(int tile, int m_tiles, int n_tiles, int& m_blk, int& n_blk) {
  const int G = 8;
  int per_group = G * n_tiles;
  int g = tile / per_group;
  int first_m = g * G;
  int gsize = min(G, m_tiles - first_m);
  int r = tile - g * per_group;
  m_blk = first_m + r % gsize;
  n_blk = r / gsize;
}

// ---- producer: a whole, converged warp -------------------------------------------------------
// Loads one (128 x 64) A block and one (BN x 64) B block per k-step. K-major operands take one
// box; MN-major operands take one 64-wide box per 64 rows (each box is a 64x64 swizzle panel).
template <int BN, int STAGES, bool A_MN, bool B_MN, int SBN = BN>
MACO_DEVICE bool gemm_produce_tile(uint8_t* smem, const GemmCtrl& c, const CUtensorMap* tmA,
                                   const CUtensorMap* tmB, int m0, int n0, int k0, int k_blocks,
                                   uint32_t& it, uint64_t budget_ns, long long* prof = nullptr, int k_step = kBK,
                                   int b_blocked_row0 = -1, uint32_t b_ahead = 0) {
  // b_ahead: the first b_ahead k-blocks have their stage armed and B on its way already (gemm_produce_b_ahead)
  // b_blocked_row0 >= 0: B is stored tile by tile ([N / BN][K / 64][BN][64], see ops.block_weight) and its tensor map
  // is the 2-D view [rows, 64]; k-block kb of this tile is the contiguous BN x 64 block at row b_blocked_row0 + kb * BN.
  // (A K-major [N, K] weight read once from HBM comes in as BN separate 128-byte pieces per box, one per DRAM
  // page; the blocked form streams at the rate of a plain copy.)
  // k_step: elements per 128-byte k-block (64 for 16-bit operands, 32 for fp32 operands run as TF32)
  using L = GemmSmemLayout<BN, STAGES, SBN>;
  m0 = warp_uniform(m0); n0 = warp_uniform(n0); k0 = warp_uniform(k0); k_blocks = warp_uniform(k_blocks);
  b_blocked_row0 = warp_uniform(b_blocked_row0); b_ahead = warp_uniform(b_ahead);
  // stage index and phase advance incrementally: the loop is one instruction stream, and a division
  // per k-block is a measurable part of it
  uint32_t s = it % STAGES, ph = (it / STAGES) & 1;
  uint8_t* sa = smem + s * L::kStageBytes;
  int k = k0;
  for (int kb = 0; kb < k_blocks; ++kb, k += k_step) {
    const long long t0 = prof ? clock64() : 0;
    const bool b_done = (uint32_t)kb < b_ahead;
    if (!b_done && !mbar_wait_warp(&c.empty[s], ph ^ 1, budget_ns, c.abort_word)) { it += kb; return false; }
    if (prof) prof[0] += clock64() - t0;
    if (elect_one()) {
      if (!b_done) mbar_arrive_expect_tx(&c.full[s], L::kLoadBytes);
      uint8_t* sb = sa + L::kABytes;
      if constexpr (!A_MN) {
        tma_load_2d(sa, tmA, &c.full[s], k, m0);
      } else {
#pragma unroll
        for (int j = 0; j < kBM / 64; ++j) tma_load_2d(sa + j * 8192, tmA, &c.full[s], m0 + j * 64, k);
      }
      if constexpr (!B_MN) {
        if (b_done) {}
        else if (b_blocked_row0 >= 0) tma_load_2d(sb, tmB, &c.full[s], 0, b_blocked_row0 + kb * BN);
        else tma_load_2d(sb, tmB, &c.full[s], k, n0);
      } else {
#pragma unroll
        for (int j = 0; j < BN / 64; ++j) tma_load_2d(sb + j * 8192, tmB, &c.full[s], n0 + j * 64, k);
      }
    }
    if (++s == STAGES) { s = 0; ph ^= 1; sa = smem; } else { sa += L::kStageBytes; }
  }
  it += k_blocks;
  return true;
}

// The B half of a tile's first k-blocks (K-major B), ahead of everything the tile waits for: arms each stage for both
// operands and loads B; gemm_produce_tile then brings in A. At most STAGES k-blocks; `ahead` counts them.
template <int BN, int STAGES, int SBN = BN>
MACO_DEVICE bool gemm_produce_b_ahead(uint8_t* smem, const GemmCtrl& c, const CUtensorMap* tmB, int n0, int k0, int k_blocks,
                                      uint32_t it, uint64_t budget_ns, int b_blocked_row0, uint32_t& ahead) {
  using L = GemmSmemLayout<BN, STAGES, SBN>;
  n0 = warp_uniform(n0); k0 = warp_uniform(k0); k_blocks = warp_uniform(k_blocks); b_blocked_row0 = warp_uniform(b_blocked_row0);
  const uint32_t most = k_blocks < STAGES ? (uint32_t)k_blocks : (uint32_t)STAGES;
  for (ahead = 0; ahead < most; ++ahead) {
    const uint32_t u = it + ahead, s = u % STAGES, ph = (u / STAGES) & 1;
    if (!mbar_wait_warp(&c.empty[s], ph ^ 1, budget_ns, c.abort_word)) return false;
    if (elect_one()) {
      mbar_arrive_expect_tx(&c.full[s], L::kLoadBytes);
      uint8_t* sb = smem + s * L::kStageBytes + L::kABytes;
      if (b_blocked_row0 >= 0) tma_load_2d(sb, tmB, &c.full[s], 0, b_blocked_row0 + (int)ahead * BN);
      else tma_load_2d(sb, tmB, &c.full[s], k0 + (int)ahead * kBK, n0);
    }
  }
  return true;
}

// After an abort: give loads that are still in flight a bounded time to land before the CTA
// leaves (their destination is this CTA's shared memory).
template <int STAGES>
MACO_DEVICE void gemm_drain_loads(const GemmCtrl& c, uint32_t issued) {
  uint32_t first = issued > STAGES ? issued - STAGES : 0;
  for (uint32_t i = first; i < issued; ++i) {
    uint64_t t0 = globaltimer_ns();
    while (!mbar_try_wait(&c.full[i % STAGES], (i / STAGES) & 1)) {
      if (globaltimer_ns() - t0 > 2000000ull) break;
    }
  }
}

// ---- MMA issuer: a whole, converged warp (the elected lane is the same one each time, so its commits cover its products) -----
template <int BN, int STAGES, bool A_MN, bool B_MN, int SBN = BN, bool TF32 = false>
MACO_DEVICE bool gemm_mma_tile(uint8_t* smem, const GemmCtrl& c, uint32_t tmem_base, uint32_t idesc,
                               int k_blocks, uint32_t& it, uint32_t tile_seq, uint64_t budget_ns,
                               long long* prof = nullptr) {
  using L = GemmSmemLayout<BN, STAGES, SBN>;
  const uint32_t acc = tile_seq & 1, acc_ph = (tile_seq >> 1) & 1;
  k_blocks = warp_uniform(k_blocks); idesc = warp_uniform(idesc);
  long long t0 = prof ? clock64() : 0;
  if (!mbar_wait_warp(&c.tmem_empty[acc], acc_ph ^ 1, budget_ns, c.abort_word)) return false;
  if (prof) prof[1] += clock64() - t0;
  tc_fence_after();
  const uint32_t d_tmem = warp_uniform(tmem_base) + acc * SBN;
  // K-major: 8-row groups are 1024 B apart (SBO); a K step of 16 elements is 32 B inside the swizzled row.
  // MN-major: 64-row panels are 8192 B apart (LBO), 8-k groups 1024 B apart (SBO); a K step of 16 is two groups
  // = 2048 B. The descriptors' high words are constant; the low word is the start address in 16-byte units.
  const uint64_t da0 = A_MN ? make_smem_desc(0, 8192, 1024, 2) : make_smem_desc(0, 16, 1024, 2);
  const uint64_t db0 = B_MN ? make_smem_desc(0, 8192, 1024, 2) : make_smem_desc(0, 16, 1024, 2);
  const uint32_t a_hi = (uint32_t)(da0 >> 32), b_hi = (uint32_t)(db0 >> 32);
  const uint32_t a_lbo = (uint32_t)da0, b_lbo = (uint32_t)db0;          // leading-dimension offset field (bits 16-29)
  constexpr uint32_t kStepA = (A_MN ? 2048 : 32) >> 4, kStepB = (B_MN ? 2048 : 32) >> 4;
  constexpr uint32_t kStage16 = L::kStageBytes >> 4, kAB16 = L::kABytes >> 4;
  const uint32_t base_lo = (smem_u32(smem) & 0x3FFFFu) >> 4;
  uint32_t s = it % STAGES, ph = (it / STAGES) & 1;
  uint32_t a_lo = base_lo + s * kStage16;
  for (int kb = 0; kb < k_blocks; ++kb) {
    if (prof) t0 = clock64();
    if (!mbar_wait_warp(&c.full[s], ph, budget_ns, c.abort_word)) { it += kb; return false; }
    if (prof) prof[2] += clock64() - t0;
    if (elect_one()) {
      const uint32_t b_lo = a_lo + kAB16;
#pragma unroll
      for (int k = 0; k < kBK / kUmmaK; ++k) {
        // low descriptor words: start address (bits 0-13, never carries: shared memory is below 256 KB) | leading offset
        // fp32 operands (TF32): 8 elements of 4 bytes per MMA, the same 32-byte step inside the swizzled row
        const uint32_t add = k == 0 ? (kb != 0 ? 1u : 0u) : 1u;
        if constexpr (TF32) tc_mma_tf32_lo(d_tmem, (a_lo + k * kStepA) | a_lbo, a_hi, (b_lo + k * kStepB) | b_lbo, b_hi, idesc, add);
        else tc_mma_f16_lo(d_tmem, (a_lo + k * kStepA) | a_lbo, a_hi, (b_lo + k * kStepB) | b_lbo, b_hi, idesc, add);
      }
      tc_commit(&c.empty[s]);        // frees the smem stage once these MMAs have read it
    }
    if (++s == STAGES) { s = 0; ph ^= 1; a_lo = base_lo; } else { a_lo += kStage16; }
  }
  it += k_blocks;
  if (elect_one()) tc_commit(&c.tmem_full[acc]);      // accumulator complete -> epilogue
  return true;
}

// ---- epilogue ------------------------------------------------------------------------------
MACO_DEVICE float epi_bias(const GemmEpilogue& e, int col) {
  if (e.bias == nullptr) return 0.f;
  if (e.bias_type == MACO_DT_F32) return reinterpret_cast<const float*>(e.bias)[col];
  if (e.bias_type == MACO_DT_F16) return __half2float(reinterpret_cast<const __half*>(e.bias)[col]);
  return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(e.bias)[col]);
}

MACO_DEVICE uint32_t epi_pack(int out_type, float a, float b) {
  if (out_type == MACO_DT_F16) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  return pack_bf16x2(a, b);
}

// Stores 32 consecutive columns of one row. `v` holds fp32 values already transformed.
MACO_DEVICE void epi_store_row32(const GemmEpilogue& e, void* out_base, long long row, int col0,
                                 int ncols_valid, const float (&v)[32]) {
  if (e.out_type == MACO_DT_F32) {
    float* p = reinterpret_cast<float*>(out_base) + row * e.ld_out + col0;
    if (e.mode == MACO_EPI_F32_ATOMIC || e.mode == MACO_EPI_SPLITK_FUSED) {
      // split-K: several tiles add into the same fp32 block; vector reductions at the L2
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        if (j + 4 <= ncols_valid) {
          asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};"
                       :: "l"(p + j), "f"(v[j]), "f"(v[j + 1]), "f"(v[j + 2]), "f"(v[j + 3]) : "memory");
        } else {
          for (int t = j; t < ncols_valid && t < j + 4; ++t) atomicAdd(p + t, v[t]);
        }
      }
    } else if (e.mode == MACO_EPI_F32_ACC) {
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        if (j + 4 <= ncols_valid) {
          float4 o = *reinterpret_cast<float4*>(p + j);
          o.x += v[j]; o.y += v[j + 1]; o.z += v[j + 2]; o.w += v[j + 3];
          *reinterpret_cast<float4*>(p + j) = o;
        } else {
          for (int t = j; t < ncols_valid && t < j + 4; ++t) p[t] += v[t];
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        if (j + 4 <= ncols_valid) {
          *reinterpret_cast<float4*>(p + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        } else {
          for (int t = j; t < ncols_valid && t < j + 4; ++t) p[t] = v[t];
        }
      }
    }
  } else {
    uint16_t* p = reinterpret_cast<uint16_t*>(out_base) + row * e.ld_out + col0;
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
      if (j + 8 <= ncols_valid) {
        uint4 o;
        o.x = epi_pack(e.out_type, v[j], v[j + 1]);
        o.y = epi_pack(e.out_type, v[j + 2], v[j + 3]);
        o.z = epi_pack(e.out_type, v[j + 4], v[j + 5]);
        o.w = epi_pack(e.out_type, v[j + 6], v[j + 7]);
        *reinterpret_cast<uint4*>(p + j) = o;
      } else {
        for (int t = j; t < ncols_valid && t < j + 8; ++t) {
          uint32_t w = epi_pack(e.out_type, v[t], 0.f);
          p[t] = (uint16_t)(w & 0xffffu);
        }
      }
    }
  }
}

MACO_DEVICE float epi_load_aux(const GemmEpilogue& e, long long row, int col) {
  const uint16_t* p = reinterpret_cast<const uint16_t*>(e.aux) + row * e.ld_aux + col;
  if (e.aux_type == MACO_DT_F16) return __half2float(*reinterpret_cast<const __half*>(p));
  return __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(p));
}

// The 32 aux values beside one row's 32-column chunk: four 16-byte loads issued together when the chunk is
// whole and aligned (one 2-byte load per element otherwise). Values past `valid` are 0.
MACO_DEVICE void epi_load_aux32(const GemmEpilogue& e, long long row, int col0, int valid, float (&a)[32]) {
  const uint16_t* p = reinterpret_cast<const uint16_t*>(e.aux) + row * e.ld_aux + col0;
  if (valid == 32 && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    uint4 q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = reinterpret_cast<const uint4*>(p)[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t w[4] = {q[i].x, q[i].y, q[i].z, q[i].w};
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float2 f = e.aux_type == MACO_DT_F16 ? __half22float2(*reinterpret_cast<const __half2*>(&w[t])) : unpack_bf16x2(w[t]);
        a[i * 8 + 2 * t] = f.x; a[i * 8 + 2 * t + 1] = f.y;
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) a[j] = j < valid ? epi_load_aux(e, row, col0 + j) : 0.f;
  }
}

// Consumes one finished accumulator. Called by all 32 lanes of each of the 4 epilogue warps.
// `out_base` lets a caller redirect the tile (for example into a peer GPU's buffer);
// `row_off` is added to the tile's row index when storing (for scatter into per-rank slabs).
// Staged stores: tiles that leave the GPU (a peer's heap) are first written to shared memory and
// then sent as one 128-byte bulk copy per row and 64-column group. Per-thread 16-byte stores to
// peer memory reach only a small fraction of NVLink bandwidth; the bulk engine writes full lines.
constexpr int kEpiStageRowBytes = 144;                       // 128 bytes of data + 16 of padding (bank spread)
constexpr int kEpiStageWarpBytes = 32 * kEpiStageRowBytes;   // one epilogue warp: 32 rows
constexpr int kEpiStageBytes = 4 * kEpiStageWarpBytes;

MACO_DEVICE void epi_stage_chunk(uint8_t* srow, int half, int out_type, const float (&v)[32]) {
  uint4* dst = reinterpret_cast<uint4*>(srow + half * 64);
#pragma unroll
  for (int j = 0; j < 32; j += 8) {
    uint4 o;
    o.x = epi_pack(out_type, v[j], v[j + 1]); o.y = epi_pack(out_type, v[j + 2], v[j + 3]);
    o.z = epi_pack(out_type, v[j + 4], v[j + 5]); o.w = epi_pack(out_type, v[j + 6], v[j + 7]);
    dst[j >> 3] = o;
  }
}

MACO_DEVICE void epi_stage_chunk_f32(uint8_t* srow, const float (&v)[32]) {
  uint4* dst = reinterpret_cast<uint4*>(srow);
#pragma unroll
  for (int j = 0; j < 32; j += 4)
    dst[j >> 2] = make_uint4(__float_as_uint(v[j]), __float_as_uint(v[j + 1]), __float_as_uint(v[j + 2]), __float_as_uint(v[j + 3]));
}

// Extra destinations of a tile: the same values are also stored at bases[k] + off for k < n
// (used to broadcast a partial result into every rank's staging slot).
struct EpiBroadcast {
  int n;
  uint8_t* const* bases;
  unsigned long long off;
};

// The common tiles of the persistent kernel: whole columns into this GPU's memory and no bias (plain 16-bit store, SwiGLU,
// rows scattered by record). Same arithmetic as gemm_epilogue_tile below without its other modes around it, which cost a few
// hundred bytes of spills per thread and tile with a 28 KB L1 to hold them: the entry function goes from 636 / 1284 bytes
// stored / loaded to 308 / 404 with this form inlined and the general one behind a call.
MACO_DEVICE bool epi_is_lean(const GemmEpilogue& e, int n0, int bn) {
  const bool plain = e.mode == MACO_EPI_STORE || e.mode == MACO_EPI_F32_STORE;
  return e.out_type != MACO_DT_F32 && e.bias == nullptr && n0 + bn <= e.N && (plain || e.mode == MACO_EPI_SWIGLU || e.mode == MACO_EPI_SCATTER_ROWS);
}
template <int SBN>
MACO_DEVICE bool gemm_epilogue_lean(int bn, const GemmCtrl& c, uint32_t tmem_base, const GemmEpilogue& e, void* out_base, long long row_off,
                                    int m0, int n0, uint32_t tile_seq, uint64_t budget_ns, uint32_t pair_empty_bar, int row_limit) {
  const uint32_t q = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
  const uint32_t acc = tile_seq & 1;
  uint32_t ok = 1;
  if (lane == 0) ok = mbar_wait(&c.tmem_full[acc], (tile_seq >> 1) & 1, budget_ns, c.abort_word) ? 1u : 0u;
  ok = __shfl_sync(0xffffffffu, ok, 0);
  if (!ok) return false;
  tc_fence_after();
  const int row = m0 + (int)(q * 32 + lane), dt = e.out_type;
  const bool scatter = e.mode == MACO_EPI_SCATTER_ROWS, swiglu = e.mode == MACO_EPI_SWIGLU;
  const bool row_ok = row < e.M && (!scatter || row < row_limit);
  long long out_row = row + row_off;
  float row_weight = 1.f;
  if (scatter && row_ok) {
    const int4 rec = reinterpret_cast<const int4*>(e.aux)[row];
    out_row = (long long)rec.x * e.bias_type + rec.y;
    row_weight = __int_as_float(rec.z);
  }
  const float alpha = e.alpha;
  uint8_t* dst = reinterpret_cast<uint8_t*>(out_base) + (out_row * e.ld_out + (swiglu ? n0 / 2 : n0)) * 2;
  const uint32_t t_row = tmem_base + ((q * 32u) << 16) + acc * SBN;
  const int cols = swiglu ? bn / 2 : bn;
#pragma unroll 1
  for (int col = 0; col < cols; col += 32) {
    uint32_t r[32];
    tmem_ld_32x32(t_row + col, r);
    if (swiglu) {
      uint32_t u[32];
      tmem_ld_32x32(t_row + cols + col, u);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(silu_16(__uint_as_float(r[j])) * __uint_as_float(u[j]));
    } else {
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * alpha);
    }
    uint32_t w[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) w[j] = epi_pack(dt, __uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
    if (scatter) {
      // the expert's output row is rounded to the output type first (what a separate return pass would read)
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float2 f = dt == MACO_DT_F16 ? __half22float2(*reinterpret_cast<const __half2*>(&w[j])) : unpack_bf16x2(w[j]);
        w[j] = epi_pack(dt, f.x * row_weight, f.y * row_weight);
      }
    }
    if (row_ok) {
#pragma unroll
      for (int j = 0; j < 16; j += 4) reinterpret_cast<uint4*>(dst)[j >> 2] = make_uint4(w[j], w[j + 1], w[j + 2], w[j + 3]);
    }
    dst += 64;
    __syncwarp();
  }
  tc_fence_before();
  if (pair_empty_bar == 0) {
    mbar_arrive(&c.tmem_empty[acc]);
  } else {
    __syncwarp();
    if (lane == 0) mbar_arrive_cluster(pair_empty_bar + acc * 8);
  }
  return true;
}

// Rows of a warp's 32 accumulator rows on their way to global memory. A thread holds one row (its TMEM lane), so a vector store straight
// from its registers touches 32 lines with half a sector each (L2 counted 3.3 sectors written per sector of output); through a block of
// shared memory every instruction moves whole sectors of a few rows. PIECES 16-byte pieces a row (8 or 4), swizzled by the row: free of
// bank conflicts in both directions. The block is the calling warp's own. `row_ptr(r)`: where row r of the 32 starts in this column
// group, null for a row that does not exist.
constexpr int kEpiWarpBytes = 6144;                    // a warp's: 32 rows of 128 bytes, or three blocks of 32 rows of 64 bytes (gemm_epilogue_beside)
constexpr int kEpiBlockBytes = 4 * kEpiWarpBytes;
template <int PIECES>
MACO_DEVICE uint32_t epi_piece(uint32_t block, uint32_t row, uint32_t piece) {
  return PIECES == 8 ? block + row * 128u + ((piece ^ (row & 7u)) << 4) : block + row * 64u + ((piece ^ ((row >> 1) & 3u)) << 4);
}
MACO_DEVICE void epi_sts(uint32_t saddr, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" :: "r"(saddr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
MACO_DEVICE uint4 epi_lds(uint32_t saddr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(saddr) : "memory");
  return v;
}
// Block to global memory; a barrier of the warp in front and behind.
template <int PIECES, typename RowFn>
MACO_DEVICE void epi_flush_rows(uint32_t block, uint32_t lane, RowFn row_ptr) {
  __syncwarp();
#pragma unroll 4
  for (uint32_t i = 0; i < PIECES; ++i) {
    const uint32_t r = i * (32 / PIECES) + lane / PIECES;
    const uint4 v = epi_lds(epi_piece<PIECES>(block, r, lane % PIECES));
    uint8_t* dst = row_ptr(r);
    if (dst != nullptr) reinterpret_cast<uint4*>(dst)[lane % PIECES] = v;
  }
  __syncwarp();
}
MACO_DEVICE float2 epi_unpack(int type, uint32_t w) { return type == MACO_DT_F16 ? __half22float2(*reinterpret_cast<const __half2*>(&w)) : unpack_bf16x2(w); }

// Whole columns into this GPU's memory: fp32 rows, and 16-bit ones with a bias, GELU or SiLU; and plain 16-bit tiles, with or without a bias,
// that end early at a whole step. Same results as gemm_epilogue_tile below (SiLU by silu_16: other steps, the same 16-bit values),
// in steps of 16 columns so that nothing lives in local memory: the persistent kernel leaves its L1 28 KB, a spilled value of the
// column loop is a miss to L2 two times in three, and one warp per scheduler has nothing to cover it with (32 columns at a time,
// with GELU: 20 local loads per 32 columns). fp32 rows go through `block`; 16-bit rows do not (a short chain per step counts for more there: through
// the block, products of K = 256 without a term took 79 us instead of 65). One B200, graph linears
// with GELU, us, before / now: 2048 x 4096 x 4096 76 / 58, 4096 x 8192 x 1024 170 / 99, 8192 x 4096 x 256 159 / 90.
MACO_DEVICE bool epi_is_stepped(const GemmEpilogue& e, int n0, int bn) {
  const bool f32 = e.out_type == MACO_DT_F32, plain = e.mode == MACO_EPI_STORE || e.mode == MACO_EPI_F32_STORE;
  // A plain 16-bit tile may end early, at a whole step: the few columns of a router (expert layer of 256 tokens 100.3 us with the general epilogue,
  // 94.0 this way). Not in gemm_epilogue_lean: its loop with a length of its own took 196 us instead of 186 for SwiGLU tiles of 8 k-blocks.
  if (n0 + bn > e.N) return !f32 && plain && (e.N - n0) % 16 == 0;
  return f32 ? plain : (e.mode == MACO_EPI_GELU || e.mode == MACO_EPI_SILU || (plain && e.bias != nullptr));
}
template <int SBN>
MACO_DEVICE bool gemm_epilogue_stepped(int bn, const GemmCtrl& c, uint32_t tmem_base, const GemmEpilogue& e, void* out_base, long long row_off,
                                       int m0, int n0, uint32_t tile_seq, uint64_t budget_ns, uint32_t pair_empty_bar, uint8_t* block) {
  const uint32_t q = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
  const uint32_t acc = tile_seq & 1;
  uint32_t ok = 1;
  if (lane == 0) ok = mbar_wait(&c.tmem_full[acc], (tile_seq >> 1) & 1, budget_ns, c.abort_word) ? 1u : 0u;
  ok = __shfl_sync(0xffffffffu, ok, 0);
  if (!ok) return false;
  tc_fence_after();
  const int row0 = m0 + (int)(q * 32), dt = e.out_type, mode = e.mode;
  const bool f32 = dt == MACO_DT_F32, bias = e.bias != nullptr;
  const int rows = min(32, e.M - row0);                                // of this warp (may be <= 0)
  const int cols = min(bn, e.N - n0);
  const float alpha = e.alpha;
  const long long pitch = e.ld_out * (f32 ? 4 : 2);
  uint8_t* dst = reinterpret_cast<uint8_t*>(out_base) + (row0 + row_off + (f32 ? 0 : (int)lane)) * pitch + (long long)n0 * (f32 ? 4 : 2);
  const uint32_t t_row = tmem_base + ((q * 32u) << 16) + acc * SBN;
  const uint32_t mine = smem_u32(block) + q * kEpiWarpBytes;
#pragma unroll 1
  for (int col = rows > 0 ? 0 : cols; col < cols; col += 16) {
    uint32_t r[16];
    tmem_ld_32x16(t_row + col, r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * alpha);
    if (bias) {
      const float b = epi_bias(e, n0 + col + (int)(lane & 15));
#pragma unroll
      for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __shfl_sync(0xffffffffu, b, j));
    }
    if (f32) {
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j)
        epi_sts(epi_piece<8>(mine, lane, (col & 16) / 4 + j), make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]));
      if (col & 16) {
        epi_flush_rows<8>(mine, lane, [&](uint32_t k) -> uint8_t* { return (int)k < rows ? dst + k * pitch : nullptr; });
        dst += 128;
      }
      continue;
    }
    if (mode == MACO_EPI_GELU) {
#pragma unroll
      for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(gelu_tanh(__uint_as_float(r[j])));
    } else if (mode == MACO_EPI_SILU) {
#pragma unroll
      for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(silu_16(__uint_as_float(r[j])));
    }
    uint32_t w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = epi_pack(dt, __uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
    if ((int)lane < rows) {
      reinterpret_cast<uint4*>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
      reinterpret_cast<uint4*>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
    dst += 32;
    __syncwarp();
  }
  tc_fence_before();
  if (pair_empty_bar == 0) {
    mbar_arrive(&c.tmem_empty[acc]);
  } else {
    __syncwarp();
    if (lane == 0) mbar_arrive_cluster(pair_empty_bar + acc * 8);
  }
  return true;
}

// Tiles with a second tensor beside the result, 16-bit, whole columns, no bias, 16-byte rows: the result times gelu'(aux)
// (MACO_EPI_GELU_BWD), the result and its GELU (MACO_EPI_GELU_DUAL: stand-alone products), the result and its sum with aux
// (MACO_EPI_RESIDUAL_DUAL: graphs). DUAL: which of the last two a kernel has code for. In steps of 16 columns as above; aux comes in by cp.async, whole sectors of eight rows an instruction, up to three groups of 32 columns ahead
// without a register held for it. One B200, us, before (32 columns at a time, aux in registers, the operators in one function with 12 local loads per step)
// / now: linear + add of 8192 x 4096 x 256 180 / 110, 2048 x 4096 x 4096 84 / 66; training stack of four 4096 x 4096 layers 2788 / 2595.
template <int DUAL>
MACO_DEVICE bool epi_is_beside(const GemmEpilogue& e, int n0, int bn) {
  const bool res = DUAL == MACO_EPI_RESIDUAL_DUAL && e.mode == DUAL;
  const uintptr_t p = reinterpret_cast<uintptr_t>(e.aux) | (uintptr_t)(e.ld_aux * 2) | (res ? reinterpret_cast<uintptr_t>(e.bias) : 0);
  return (e.mode == MACO_EPI_GELU_BWD || e.mode == DUAL) && (res || e.bias == nullptr) && n0 + bn <= e.N &&
         e.out_type != MACO_DT_F32 && (p & 15) == 0;
}
template <int SBN, int MODE>
__device__ __noinline__ bool gemm_epilogue_beside_as(int bn, const GemmCtrl& c, uint32_t tmem_base, const GemmEpilogue& e_in, void* out_base,
                                                long long row_off, int m0, int n0, uint32_t tile_seq, uint64_t budget_ns,
                                                uint32_t pair_empty_bar, uint8_t* block) {
  const uint32_t q = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31, acc = tile_seq & 1;
  const int row0 = m0 + (int)(q * 32), dt = e_in.out_type, at = e_in.aux_type;
  const int rows = min(32, e_in.M - row0);                             // of this warp (may be <= 0)
  constexpr bool dual = MODE == MACO_EPI_GELU_DUAL, res = MODE == MACO_EPI_RESIDUAL_DUAL;
  const float alpha = e_in.alpha;
  const long long pitch = e_in.ld_out * 2, aux_pitch = e_in.ld_aux * 2;
  uint8_t* dst = reinterpret_cast<uint8_t*>(out_base) + (row0 + row_off + (int)lane) * pitch + n0 * 2;
  uint8_t* aux = reinterpret_cast<uint8_t*>(const_cast<void*>(e_in.aux)) + (long long)row0 * aux_pitch + n0 * 2;
  uint8_t* second = dual ? aux + lane * aux_pitch : reinterpret_cast<uint8_t*>(const_cast<void*>(e_in.bias)) + (row0 + row_off + (int)lane) * pitch + n0 * 2;
  const uint32_t mine = smem_u32(block) + q * kEpiWarpBytes;
  uint32_t in = 0;                                     // which of the three 2 KB blocks is filled next
  int fetched = dual ? bn : 0;
  auto fetch = [&] {                                   // 32 columns of aux, and always a group for the waits to count
    if (fetched < bn) {
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i) {
        const uint32_t r = i * 8 + (lane >> 2);
        if ((int)r < rows) cp_async16(epi_piece<4>(mine + in, r, lane & 3), aux + r * aux_pitch + fetched * 2 + (lane & 3) * 16);
      }
      fetched += 32;
      in = in + 2048u == kEpiWarpBytes ? 0u : in + 2048u;
    }
    cp_async_commit();
  };
  uint32_t ok = 1;
  if (lane == 0) ok = mbar_wait(&c.tmem_full[acc], (tile_seq >> 1) & 1, budget_ns, c.abort_word) ? 1u : 0u;
  ok = __shfl_sync(0xffffffffu, ok, 0);
  if (!ok) return false;
  tc_fence_after();
  fetch();                                             // (behind the accumulator's barrier: what the tile depends on has happened)
  fetch();
  fetch();
  const uint32_t t_row = tmem_base + ((q * 32u) << 16) + acc * SBN;
  uint32_t cur = mine;
#pragma unroll 1
  for (int col = rows > 0 ? 0 : bn; col < bn;) {
    cp_async_wait<2>();
    __syncwarp();
#pragma unroll 1
    for (uint32_t piece = 0; piece < 4; piece += 2, col += 16) {
      uint32_t r[16], w[8], g[8];
      tmem_ld_32x16(t_row + col, r);
      if (!dual) {
        const uint4 a = epi_lds(epi_piece<4>(cur, lane, piece)), b = epi_lds(epi_piece<4>(cur, lane, piece + 1));
        g[0] = a.x; g[1] = a.y; g[2] = a.z; g[3] = a.w; g[4] = b.x; g[5] = b.y; g[6] = b.z; g[7] = b.w;
      }
      tmem_ld_wait();
      if (dual || res) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          w[j] = epi_pack(dt, __uint_as_float(r[2 * j]) * alpha, __uint_as_float(r[2 * j + 1]) * alpha);
          const float2 z = epi_unpack(dt, w[j]);
          if (dual) {
            g[j] = epi_pack(at, gelu_tanh(z.x), gelu_tanh(z.y));
          } else {
            const float2 x = epi_unpack(at, g[j]);
            g[j] = epi_pack(dt, z.x + x.x, z.y + x.y);
          }
        }
        if ((int)lane < rows) {
          reinterpret_cast<uint4*>(second)[0] = make_uint4(g[0], g[1], g[2], g[3]);
          reinterpret_cast<uint4*>(second)[1] = make_uint4(g[4], g[5], g[6], g[7]);
        }
        second += 32;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 z = epi_unpack(at, g[j]);
          w[j] = epi_pack(dt, __uint_as_float(r[2 * j]) * alpha * gelu_tanh_grad(z.x), __uint_as_float(r[2 * j + 1]) * alpha * gelu_tanh_grad(z.y));
        }
      }
      if ((int)lane < rows) {
        reinterpret_cast<uint4*>(dst)[0] = make_uint4(w[0], w[1], w[2], w[3]);
        reinterpret_cast<uint4*>(dst)[1] = make_uint4(w[4], w[5], w[6], w[7]);
      }
      dst += 32;
      __syncwarp();                                    // tcgen05.ld takes a converged warp; and every lane has read its row of the block that is filled next
    }
    cur = cur + 2048u == mine + kEpiWarpBytes ? mine : cur + 2048u;
    fetch();
  }
  cp_async_wait<0>();
  tc_fence_before();
  if (pair_empty_bar == 0) {
    mbar_arrive(&c.tmem_empty[acc]);
  } else {
    __syncwarp();
    if (lane == 0) mbar_arrive_cluster(pair_empty_bar + acc * 8);
  }
  return true;
}

// (a function per operator: together they keep more values than a callee of the persistent kernel has registers for)
template <int SBN, int DUAL>
MACO_DEVICE bool gemm_epilogue_beside(int bn, const GemmCtrl& c, uint32_t tmem_base, const GemmEpilogue& e, void* out_base, long long row_off,
                                      int m0, int n0, uint32_t tile_seq, uint64_t budget_ns, uint32_t pair_empty_bar, uint8_t* block) {
  if (e.mode == MACO_EPI_GELU_BWD)
    return gemm_epilogue_beside_as<SBN, MACO_EPI_GELU_BWD>(bn, c, tmem_base, e, out_base, row_off, m0, n0, tile_seq, budget_ns, pair_empty_bar, block);
  return gemm_epilogue_beside_as<SBN, DUAL>(bn, c, tmem_base, e, out_base, row_off, m0, n0, tile_seq, budget_ns, pair_empty_bar, block);
}

// (DUAL: with this mode that writes a second tensor, or 0, for tiles of such a product that are ragged or not aligned)
template <int BN, int SBN, int DUAL>
MACO_DEVICE bool gemm_epilogue_tile(const GemmCtrl& c, uint32_t tmem_base, const GemmEpilogue& e_in,
                                    void* out_base, long long row_off, int m0, int n0,
                                    uint32_t tile_seq, uint64_t budget_ns, const EpiBroadcast* bc = nullptr,
                                    uint8_t* stage = nullptr, uint32_t pair_empty_bar = 0, int row_limit = 0x7fffffff) {
  // private copy: the record lives in global memory; read in place, its fields would be loaded again after
  // every store of the tile (the stores could alias it)
  const GemmEpilogue e = e_in;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t q = warp & 3;     // TMEM lane quarter this warp may read
  const uint32_t acc = tile_seq & 1, acc_ph = (tile_seq >> 1) & 1;
  uint32_t ok = 1;
  if (lane == 0) ok = mbar_wait(&c.tmem_full[acc], acc_ph, budget_ns, c.abort_word) ? 1u : 0u;
  ok = __shfl_sync(0xffffffffu, ok, 0);
  if (!ok) return false;
  tc_fence_after();
  const int row = m0 + q * 32 + lane;
  const bool scatter = e.mode == MACO_EPI_SCATTER_ROWS;
  const bool row_ok = row < e.M && (!scatter || row < row_limit);
  // scatter: this thread's row has its own destination row and weight (one 16-byte record per row)
  long long out_row = row + row_off;
  float row_weight = 1.f;
  if (scatter && row_ok) {
    const int4 rec = reinterpret_cast<const int4*>(e.aux)[row];
    out_row = (long long)rec.x * e.bias_type + rec.y;
    row_weight = __int_as_float(rec.z);
  }
  // staged path: 16-bit output, tile completely inside the output columns (uniform over the CTA)
  const int out_cols = e.mode == MACO_EPI_SWIGLU ? e.N / 2 : e.N;
  const int tile_col0 = e.mode == MACO_EPI_SWIGLU ? n0 / 2 : n0;
  const int tile_cols = e.mode == MACO_EPI_SWIGLU ? BN / 2 : BN;
  // (fp32 tiles that are plain stores take the same path: 32 columns are one 128-byte row chunk)
  const bool f32_out = e.out_type == MACO_DT_F32;
  const bool staged = stage != nullptr && (!f32_out || e.mode == MACO_EPI_F32_STORE) && tile_col0 + tile_cols <= out_cols &&
                      e.mode != MACO_EPI_F32_ACC;
  uint8_t* srow = stage != nullptr ? stage + q * kEpiStageWarpBytes + lane * kEpiStageRowBytes : nullptr;
  auto flush_group = [&](int gcol) {
    fence_proxy_async_smem();
    __syncwarp();
    if (row_ok) {
      const long long eoff = (out_row * e.ld_out + gcol) * (f32_out ? 4 : 2);
      if (bc == nullptr) {
        bulk_store(reinterpret_cast<uint8_t*>(out_base) + eoff, srow, 128);
      } else {
        for (int k = 0; k < bc->n; ++k) bulk_store(bc->bases[k] + bc->off + eoff, srow, 128);
      }
      tma_store_commit();
    }
    tma_store_wait_read<0>();
    __syncwarp();
  };
  const uint32_t t_row = tmem_base + ((q * 32u) << 16) + acc * SBN;
  if (e.mode == MACO_EPI_SWIGLU) {
    // Columns [0, BN/2) of the tile hold the gate projection, [BN/2, BN) the up projection of
    // the same BN/2 output features (weights are interleaved that way when the graph is built).
#pragma unroll 1
    for (int ch = 0; ch < BN / 64; ++ch) {
      uint32_t g[32], u[32];
      tmem_ld_32x32(t_row + ch * 32, g);
      tmem_ld_32x32(t_row + BN / 2 + ch * 32, u);
      tmem_ld_wait();
      float v[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = silu(__uint_as_float(g[j])) * __uint_as_float(u[j]);
      const int col0 = n0 / 2 + ch * 32;
      const int valid = min(32, e.N / 2 - col0);
      if (staged) {
        if (row_ok) epi_stage_chunk(srow, ch & 1, e.out_type, v);
        if (ch & 1) flush_group(col0 - 32);
      } else if (row_ok && valid > 0) {
        if (bc == nullptr) epi_store_row32(e, out_base, out_row, col0, valid, v);
        else for (int k = 0; k < bc->n; ++k) epi_store_row32(e, bc->bases[k] + bc->off, out_row, col0, valid, v);
      }
      __syncwarp();
    }
  } else {
#pragma unroll 1
    for (int ch = 0; ch < BN / 32; ++ch) {
      uint32_t r[32];
      tmem_ld_32x32(t_row + ch * 32, r);
      tmem_ld_wait();
      const int col0 = n0 + ch * 32;
      const int valid = min(32, e.N - col0);
      if (row_ok && valid > 0) {
      float v[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]) * e.alpha;
      if (scatter) {
        // the expert's output row is rounded to the output type first (what a separate return pass would read)
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const uint32_t pk = epi_pack(e.out_type, v[j], v[j + 1]);
          const float2 f = e.out_type == MACO_DT_F16 ? __half22float2(*reinterpret_cast<const __half2*>(&pk)) : unpack_bf16x2(pk);
          v[j] = f.x * row_weight; v[j + 1] = f.y * row_weight;
        }
      }
      if (e.bias != nullptr && e.mode != MACO_EPI_SPLITK_FUSED && !(DUAL == MACO_EPI_RESIDUAL_DUAL && e.mode == DUAL)) {     // (those keep counters / an output there)
#pragma unroll
        for (int j = 0; j < 32; ++j) if (j < valid) v[j] += epi_bias(e, col0 + j);
      }
      if (e.mode == MACO_EPI_GELU) {
        if (f32_out) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = gelu_tanh_f32_call(v[j]);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = gelu_tanh(v[j]);
        }
      } else if (e.mode == MACO_EPI_GELU_BWD) {
        float ax[32];
        epi_load_aux32(e, row, col0, valid, ax);
        if (f32_out) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] *= gelu_tanh_grad_f32_call(ax[j]);
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] *= gelu_tanh_grad(ax[j]);
        }
      } else if (DUAL == MACO_EPI_RESIDUAL_DUAL && e.mode == DUAL) {
        uint16_t* sum = reinterpret_cast<uint16_t*>(const_cast<void*>(e.bias)) + out_row * e.ld_out + col0;
        float ax[32];
        epi_load_aux32(e, row, col0, valid, ax);
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const uint32_t z = epi_pack(e.out_type, v[j], 0.f);
          const float f = e.out_type == MACO_DT_F16 ? __half22float2(*reinterpret_cast<const __half2*>(&z)).x : unpack_bf16x2(z).x;
          if (j < valid) sum[j] = (uint16_t)(epi_pack(e.out_type, f + ax[j], 0.f) & 0xffffu);
        }
      } else if (DUAL == MACO_EPI_GELU_DUAL && e.mode == DUAL) {
        uint16_t* act = reinterpret_cast<uint16_t*>(const_cast<void*>(e.aux)) + row * e.ld_aux + col0;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const uint32_t z = epi_pack(e.out_type, v[j], 0.f);
          const float f = e.out_type == MACO_DT_F16 ? __half22float2(*reinterpret_cast<const __half2*>(&z)).x : unpack_bf16x2(z).x;
          if (j < valid) act[j] = (uint16_t)(epi_pack(e.aux_type, gelu_tanh(f), 0.f) & 0xffffu);
        }
      } else if (e.mode == MACO_EPI_SILU) {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = silu(v[j]);
      } else if (e.mode == MACO_EPI_RESIDUAL) {
        const int n_aux = e.aux_pack & 15;
        if (n_aux <= 1) {
          float ax[32];
          epi_load_aux32(e, row, col0, valid, ax);
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] += ax[j];
        } else {
          // several blocks (a reduce-scatter's staging slots): the tile sums them all into its accumulator
          const int skip = (e.aux_pack >> 4) & 15;
          const long long slot_rows = e.aux_pack >> 8;
          for (int sl = 0; sl < n_aux; ++sl) {
            if (sl == skip) continue;
            float ax[32];
            epi_load_aux32(e, row + sl * slot_rows, col0, valid, ax);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] += ax[j];
          }
        }
      }
      if (staged) {
        if (row_ok) {
          if (f32_out) epi_stage_chunk_f32(srow, v);
          else epi_stage_chunk(srow, ch & 1, e.out_type, v);
        }
      } else if (bc == nullptr) epi_store_row32(e, out_base, out_row, col0, valid, v);
      else for (int k = 0; k < bc->n; ++k) epi_store_row32(e, bc->bases[k] + bc->off, out_row, col0, valid, v);
      }
      if (staged && f32_out) flush_group(col0);
      else if (staged && (ch & 1)) flush_group(col0 - 32);
      __syncwarp();
    }
  }
  if (staged) tma_store_wait<0>();     // bulk stores complete before the tile is signalled
  tc_fence_before();
  if (pair_empty_bar == 0) {
    mbar_arrive(&c.tmem_empty[acc]);
  } else {
    // two-CTA tile: the pair leader's barrier collects one arrival per epilogue warp of both CTAs
    __syncwarp();
    if (lane == 0) mbar_arrive_cluster(pair_empty_bar + acc * 8);
  }
  return true;
}

// ---- CTA set-up / tear-down shared by every kernel built on this pipeline ------------------------
template <int BN, int STAGES>
MACO_DEVICE uint8_t* gemm_cta_setup(uint8_t* dyn_smem, GemmCtrl& c, uint32_t& tmem_base, bool alloc_tmem = true) {
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dyn_smem) + 1023) & ~uintptr_t(1023));
  c = gemm_ctrl<BN, STAGES>(smem);
  const uint32_t warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&c.full[s], 1); mbar_init(&c.empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&c.tmem_full[a], 1); mbar_init(&c.tmem_empty[a], 128); }
    *c.abort_word = 0;
    fence_mbar_init();
  }
  if (threadIdx.x == 32) *c.tmem_slot = 0;
  __syncwarp();
  if (warp == 1 && alloc_tmem) {
    tmem_alloc(c.tmem_slot, 2 * BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  tmem_base = *c.tmem_slot;
  return smem;
}

template <int BN>
MACO_DEVICE void gemm_cta_teardown(const GemmCtrl& c, uint32_t tmem_base, uint32_t* status, bool had_tmem = true) {
  tc_fence_before();
  __syncthreads();
  if ((threadIdx.x >> 5) == 1 && had_tmem) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BN);
  }
  if (threadIdx.x == 0 && *c.abort_word != 0 && status != nullptr) st_relaxed_sys_u32(status, MACO_STATUS_TIMEOUT);
}

// ---- two-CTA tiles (cta_group::2) -----------------------------------------------------------------
// A pair of CTAs (one cluster) computes a 256 x BN tile: each CTA loads its own 128 rows of A and its own
// half (BN/2 rows) of B, the leader issues tcgen05.mma.cta_group::2 (M = 256), which reads both CTAs' shared
// memory and writes each CTA's 128 accumulator rows into that CTA's TMEM. Per k-step a CTA brings in
// 16 KB + BN/2 * 128 B instead of 16 KB + BN * 128 B: a third less shared-memory and L2 traffic per FLOP at
// BN = 256, and six 32 KB stages where the one-CTA form has four of 48 KB. The two row blocks of a pair
// need not be adjacent. Loads carry no multicast: each CTA fetches what it needs itself.
template <int STAGES>
struct PairSmemLayout {
  static constexpr int kABytes = kBM * kBK * 2;
  static constexpr int kBBytesMax = 128 * kBK * 2;
  static constexpr int kStageBytes = kABytes + kBBytesMax;
  static constexpr int kRingBytes = STAGES * kStageBytes;
  static constexpr int kCtrlBytes = 256;
  static constexpr int kTotalBytes = kRingBytes + kCtrlBytes + 1024;
  static_assert(2 * STAGES * 8 + 4 * 8 + 16 <= kCtrlBytes, "control block too small");
};

template <int STAGES>
MACO_DEVICE GemmCtrl pair_ctrl(uint8_t* smem_base) {
  using L = PairSmemLayout<STAGES>;
  GemmCtrl c;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_base + L::kRingBytes);
  c.full = bars;
  c.empty = bars + STAGES;
  c.tmem_full = bars + 2 * STAGES;
  c.tmem_empty = bars + 2 * STAGES + 2;
  c.tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
  c.abort_word = reinterpret_cast<volatile uint32_t*>(c.tmem_slot + 1);
  return c;
}

// Producer of one CTA of the pair. `n0` is the tile's first column; this CTA loads B rows
// [n0 + rank * BN/2, n0 + (rank + 1) * BN/2). All bytes of both CTAs are credited to the LEADER's full barrier
// by the TMA units themselves. (Measured alternative: loads completing on each CTA's own barrier plus a thread
// of the second CTA that forwards an arrival to the leader took twice as long per k-block.)
template <int BN, int STAGES, bool A_MN, bool B_MN>
MACO_DEVICE bool pair_produce_tile(uint8_t* smem, const GemmCtrl& c, uint32_t rank, const CUtensorMap* tmA,
                                   const CUtensorMap* tmB, int m0, int n0, int k0, int k_blocks, uint32_t& it,
                                   uint64_t budget_ns, long long* prof = nullptr) {
  using L = PairSmemLayout<STAGES>;
  constexpr int kBHalf = BN / 2;
  constexpr uint32_t kPairBytes = 2u * (L::kABytes + kBHalf * kBK * 2);
  const uint32_t full0 = mapa_u32(smem_u32(&c.full[0]), 0);
  m0 = warp_uniform(m0); n0 = warp_uniform(n0); k0 = warp_uniform(k0); k_blocks = warp_uniform(k_blocks);
  const int nb0 = n0 + (int)rank * kBHalf;
  uint32_t s = it % STAGES, ph = (it / STAGES) & 1;
  uint8_t* sa = smem + s * L::kStageBytes;
  int k = k0;
  for (int kb = 0; kb < k_blocks; ++kb, k += kBK) {
    const long long t0 = prof ? clock64() : 0;
    if (!mbar_wait_warp(&c.empty[s], ph ^ 1, budget_ns, c.abort_word)) { it += kb; return false; }
    if (prof) prof[0] += clock64() - t0;
    if (prof && prof[4] && prof[5] < 512) reinterpret_cast<uint64_t*>(prof[4])[2 * prof[5]] = globaltimer_ns();
    if (elect_one()) {
      uint8_t* sb = sa + L::kABytes;
      if (rank == 0) mbar_arrive_expect_tx(&c.full[s], kPairBytes);
      const uint32_t bar = full0 + s * 8;
      if constexpr (!A_MN) {
        tma_load_2d_pair(sa, tmA, bar, k, m0);
      } else {
#pragma unroll
        for (int j = 0; j < kBM / 64; ++j) tma_load_2d_pair(sa + j * 8192, tmA, bar, m0 + j * 64, k);
      }
      if constexpr (!B_MN) {
        tma_load_2d_pair(sb, tmB, bar, k, nb0);
      } else {
#pragma unroll
        for (int j = 0; j < kBHalf / 64; ++j) tma_load_2d_pair(sb + j * 8192, tmB, bar, nb0 + j * 64, k);
      }
    }
    if (prof && prof[4] && prof[5] < 512) { reinterpret_cast<uint64_t*>(prof[4])[2 * prof[5] + 1] = globaltimer_ns(); ++prof[5]; }
    if (++s == STAGES) { s = 0; ph ^= 1; sa = smem; } else { sa += L::kStageBytes; }
  }
  it += k_blocks;
  return true;
}

// MMA issuer: the pair's leader only. `peer_*` are the shared::cluster addresses of the other CTA's barriers.
template <int BN, int STAGES, bool A_MN, bool B_MN>
MACO_DEVICE bool pair_mma_tile(uint8_t* smem, const GemmCtrl& c, uint32_t tmem_base, uint32_t idesc, int k_blocks,
                               uint32_t& it, uint32_t tile_seq, uint64_t budget_ns, long long* prof = nullptr) {
  using L = PairSmemLayout<STAGES>;
  const uint32_t acc = tile_seq & 1, acc_ph = (tile_seq >> 1) & 1;
  const uint32_t empty0 = smem_u32(&c.empty[0]), tfull0 = smem_u32(&c.tmem_full[0]);
  k_blocks = warp_uniform(k_blocks); idesc = warp_uniform(idesc);
  long long t0 = prof ? clock64() : 0;
  if (!mbar_wait_warp(&c.tmem_empty[acc], acc_ph ^ 1, budget_ns, c.abort_word)) return false;
  if (prof) prof[1] += clock64() - t0;
  tc_fence_after();
  const uint32_t d_tmem = warp_uniform(tmem_base) + acc * 256;
  const uint64_t da0 = A_MN ? make_smem_desc(0, 8192, 1024, 2) : make_smem_desc(0, 16, 1024, 2);
  const uint64_t db0 = B_MN ? make_smem_desc(0, 8192, 1024, 2) : make_smem_desc(0, 16, 1024, 2);
  const uint32_t a_hi = (uint32_t)(da0 >> 32), b_hi = (uint32_t)(db0 >> 32);
  const uint32_t a_lbo = (uint32_t)da0, b_lbo = (uint32_t)db0;          // leading-dimension offset field (bits 16-29)
  constexpr uint32_t kStepA = (A_MN ? 2048 : 32) >> 4, kStepB = (B_MN ? 2048 : 32) >> 4;
  constexpr uint32_t kStage16 = L::kStageBytes >> 4, kAB16 = L::kABytes >> 4;
  const uint32_t base_lo = (smem_u32(smem) & 0x3FFFFu) >> 4;
  uint32_t s = it % STAGES, ph = (it / STAGES) & 1;
  uint32_t a_lo = base_lo + s * kStage16;
  for (int kb = 0; kb < k_blocks; ++kb) {
    if (prof) t0 = clock64();
    if (!mbar_wait_warp(&c.full[s], ph, budget_ns, c.abort_word)) { it += kb; return false; }
    if (prof) prof[2] += clock64() - t0;
    if (prof && prof[4] && prof[5] < 512) reinterpret_cast<uint64_t*>(prof[4])[2 * prof[5]] = globaltimer_ns();
    if (elect_one()) {
      const uint32_t b_lo = a_lo + kAB16;
#pragma unroll
      for (int k = 0; k < kBK / kUmmaK; ++k)
        tc_mma2_f16_lo(d_tmem, (a_lo + k * kStepA) | a_lbo, a_hi, (b_lo + k * kStepB) | b_lbo, b_hi, idesc, k == 0 ? (kb != 0 ? 1u : 0u) : 1u);
      tc_commit2_both(empty0 + s * 8); // both CTAs may refill the stage once these MMAs have read it
    }
    if (prof && prof[4] && prof[5] < 512) { reinterpret_cast<uint64_t*>(prof[4])[2 * prof[5] + 1] = globaltimer_ns(); ++prof[5]; }
    if (++s == STAGES) { s = 0; ph ^= 1; a_lo = base_lo; } else { a_lo += kStage16; }
  }
  it += k_blocks;
  if (elect_one()) tc_commit2_both(tfull0 + acc * 8);   // accumulator complete -> both CTAs' epilogues
  return true;
}

template <int STAGES>
MACO_DEVICE uint8_t* pair_cta_setup(uint8_t* dyn_smem, GemmCtrl& c, uint32_t& tmem_base) {
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dyn_smem) + 1023) & ~uintptr_t(1023));
  c = pair_ctrl<STAGES>(smem);
  const uint32_t warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&c.full[s], 1); mbar_init(&c.empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&c.tmem_full[a], 1); mbar_init(&c.tmem_empty[a], 8); }   // 4 warps x 2 CTAs
    *c.abort_word = 0;
    fence_mbar_init();
  }
  if (threadIdx.x == 32) *c.tmem_slot = 0;
  __syncwarp();
  if (warp == 1) {
    tmem_alloc2(c.tmem_slot, 512);
    tmem_relinquish2();
  }
  tc_fence_before();
  __syncthreads();
  cluster_arrive();            // the other CTA's barriers are initialised before anything is sent to them
  cluster_wait();
  tc_fence_after();
  tmem_base = *c.tmem_slot;
  return smem;
}

MACO_DEVICE void pair_cta_teardown(const GemmCtrl& c, uint32_t tmem_base, uint32_t* status) {
  tc_fence_before();
  __syncthreads();
  cluster_arrive();            // neither CTA frees TMEM or leaves while the other may still touch its memory
  cluster_wait();
  if ((threadIdx.x >> 5) == 1) {
    tc_fence_after();
    tmem_dealloc2(tmem_base, 512);
  }
  if (threadIdx.x == 0 && *c.abort_word != 0 && status != nullptr) st_relaxed_sys_u32(status, MACO_STATUS_TIMEOUT);
}

constexpr int kPairStages = 6;

// Stand-alone GEMM on two-CTA tiles: grid = 2 x (number of CTA pairs), launched as clusters of two. BESIDE: with the out-of-line epilogue of
// tiles that have a second tensor. It takes the kernel's parameters by reference, which puts them on the stack (120 bytes) and costs some
// registers, so that products without such a tensor have instances of their own. With it / without, one B200, us: 512 x 2048 x 2048 plain
// 24.2 / 20.5, 4096^3 plain 119 / 112, with GELU 173 / 147, 8192 x 4096 x 4096 plain 201 / 190, with GELU 288 / 242.
template <int BN, bool A_MN, bool B_MN, bool BESIDE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
gemm_tcgen05_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                         GemmEpilogue epi, int K, uint32_t idesc, uint64_t budget_ns, uint32_t* status, long long* dbg) {
  extern __shared__ uint8_t dyn_smem[];
  GemmCtrl c;
  uint32_t tmem_base;
  uint8_t* smem = pair_cta_setup<kPairStages>(dyn_smem, c, tmem_base);
  // optional cycle counters per CTA: [0] producer waiting for a free stage, [1] MMA waiting for a free
  // accumulator, [2] MMA waiting for operands, [3] MMA warp total, [4] producer total
  // [3]: experiment switches, see maco_gemm_set_debug; [4], [5]: optional time-line log (switch 8, first pair only):
  // words 4096 + 2048 * cta + {0: producer, 1024: MMA warp} + 2 * i + {0: wait over, 1: issue done}, %globaltimer ns
  long long prof[6] = {0, 0, 0, dbg != nullptr ? dbg[7] : 0, 0, 0};
  long long* pp = dbg != nullptr ? prof : nullptr;
  const int variant = (int)prof[3];
  if (dbg != nullptr && (variant & 8) && blockIdx.x < 2)
    prof[4] = reinterpret_cast<long long>(dbg + 4096 + 2048 * blockIdx.x + ((threadIdx.x >> 5) == 1 ? 1024 : 0));
  const long long t_begin = clock64();
  const uint32_t rank = cluster_ctarank();
  const int m_pairs = (epi.M + 2 * kBM - 1) / (2 * kBM), n_tiles = (epi.N + BN - 1) / BN;
  const int num_tiles = m_pairs * n_tiles;
  const int k_blocks = (K + kBK - 1) / kBK;
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const uint32_t warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const uint32_t tempty_leader = mapa_u32(smem_u32(&c.tmem_empty[0]), 0);
  uint8_t* block = smem + PairSmemLayout<kPairStages>::kRingBytes + PairSmemLayout<kPairStages>::kCtrlBytes;

  if (warp == 0) {
    if (lane == 0) { tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB); }
    __syncwarp();
    {
      uint32_t it = 0;
      bool ok = true;
      for (int tile = pair; ok && tile < num_tiles; tile += num_pairs) {
        int mp, nb;
        gemm_tile_coords(tile, m_pairs, n_tiles, mp, nb);
        ok = pair_produce_tile<BN, kPairStages, A_MN, B_MN>(smem, c, rank, &tmA, &tmB, (mp * 2 + (int)rank) * kBM, nb * BN, 0,
                                                            k_blocks, it, budget_ns, pp);
      }
      // after an abort the leader's barriers count both CTAs' bytes; the other CTA stays until the leader
      // reaches the teardown (cluster barrier)
      if (!ok && rank == 0) gemm_drain_loads<kPairStages>(c, it);
      if (dbg != nullptr && lane == 0) { dbg[blockIdx.x * 8 + 0] = prof[0]; dbg[blockIdx.x * 8 + 4] = clock64() - t_begin; }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0) {
      uint32_t it = 0, seq = 0;
      bool ok = true;
      for (int tile = pair; ok && tile < num_tiles; tile += num_pairs, ++seq)
        ok = pair_mma_tile<BN, kPairStages, A_MN, B_MN>(smem, c, tmem_base, idesc, k_blocks, it, seq, budget_ns, pp);
      if (dbg != nullptr && lane == 0) { dbg[blockIdx.x * 8 + 1] = prof[1]; dbg[blockIdx.x * 8 + 2] = prof[2]; dbg[blockIdx.x * 8 + 3] = clock64() - t_begin; }
    }
    __syncwarp();
  } else {
    uint32_t seq = 0;
    bool ok = true;
    for (int tile = pair; ok && tile < num_tiles; tile += num_pairs, ++seq) {
      int mp, nb;
      gemm_tile_coords(tile, m_pairs, n_tiles, mp, nb);
      if (variant & 1) {           // experiment: barrier handshake only
        if (lane == 0) ok = mbar_wait(&c.tmem_full[seq & 1], (seq >> 1) & 1, budget_ns, c.abort_word);
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(tempty_leader + (seq & 1) * 8);
        continue;
      }
      if (BESIDE && epi_is_beside<MACO_EPI_GELU_DUAL>(epi, nb * BN, BN))
        ok = gemm_epilogue_beside<256, MACO_EPI_GELU_DUAL>(BN, c, tmem_base, epi, epi.out, 0, (mp * 2 + (int)rank) * kBM, nb * BN, seq, budget_ns, tempty_leader, block);
      else if (!BESIDE && epi_is_stepped(epi, nb * BN, BN))
        ok = gemm_epilogue_stepped<256>(BN, c, tmem_base, epi, epi.out, 0, (mp * 2 + (int)rank) * kBM, nb * BN, seq, budget_ns, tempty_leader, block);
      else
        ok = gemm_epilogue_tile<BN, 256, BESIDE ? MACO_EPI_GELU_DUAL : 0>(c, tmem_base, epi, epi.out, 0, (mp * 2 + (int)rank) * kBM, nb * BN, seq, budget_ns,
                                                 nullptr, nullptr, tempty_leader);
    }
  }
  pair_cta_teardown(c, tmem_base, status);
}

// ---- stand-alone persistent GEMM kernel ---------------------------------------------------------
template <int BN, int STAGES, bool A_MN, bool B_MN, bool TF32, bool BESIDE>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    GemmEpilogue epi, int K, uint32_t idesc, uint64_t budget_ns, uint32_t* status, long long* dbg) {
  extern __shared__ uint8_t dyn_smem[];
  GemmCtrl c;
  uint32_t tmem_base;
  uint8_t* smem = gemm_cta_setup<BN, STAGES>(dyn_smem, c, tmem_base);
  long long prof[4] = {0, 0, 0, dbg != nullptr ? dbg[7] : 0};   // see gemm_tcgen05_pair_kernel
  long long* pp = dbg != nullptr ? prof : nullptr;
  const int variant = (int)prof[3];
  const long long t_begin = clock64();

  const int m_tiles = (epi.M + kBM - 1) / kBM, n_tiles = (epi.N + BN - 1) / BN;
  const int num_tiles = m_tiles * n_tiles;
  constexpr int kStepElems = TF32 ? kBK / 2 : kBK;
  const int k_blocks = (K + kStepElems - 1) / kStepElems;
  const uint32_t warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  uint8_t* block = smem + GemmSmemLayout<BN, STAGES>::kRingBytes + GemmSmemLayout<BN, STAGES>::kCtrlBytes;

  if (warp == 0) {
    if (lane == 0) { tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB); }
    __syncwarp();
    {
      uint32_t it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x) {
        int mb, nb;
        gemm_tile_coords(tile, m_tiles, n_tiles, mb, nb);
        ok = gemm_produce_tile<BN, STAGES, A_MN, B_MN>(smem, c, &tmA, &tmB, mb * kBM, nb * BN, 0, k_blocks, it, budget_ns, pp, kStepElems);
      }
      if (!ok) gemm_drain_loads<STAGES>(c, it);
      if (dbg != nullptr && lane == 0) { dbg[blockIdx.x * 8 + 0] = prof[0]; dbg[blockIdx.x * 8 + 4] = clock64() - t_begin; }
    }
    __syncwarp();
  } else if (warp == 1) {
    {
      uint32_t it = 0, seq = 0;
      bool ok = true;
      for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x, ++seq)
        ok = gemm_mma_tile<BN, STAGES, A_MN, B_MN, BN, TF32>(smem, c, tmem_base, idesc, k_blocks, it, seq, budget_ns, pp);
      if (dbg != nullptr && lane == 0) { dbg[blockIdx.x * 8 + 1] = prof[1]; dbg[blockIdx.x * 8 + 2] = prof[2]; dbg[blockIdx.x * 8 + 3] = clock64() - t_begin; }
    }
    __syncwarp();
  } else {
    uint32_t seq = 0;
    bool ok = true;
    for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x, ++seq) {
      int mb, nb;
      gemm_tile_coords(tile, m_tiles, n_tiles, mb, nb);
      if (variant & 1) {           // experiment: barrier handshake only
        if (lane == 0) ok = mbar_wait(&c.tmem_full[seq & 1], (seq >> 1) & 1, budget_ns, c.abort_word);
        ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        mbar_arrive(&c.tmem_empty[seq & 1]);
        continue;
      }
      if (BESIDE && epi_is_beside<MACO_EPI_GELU_DUAL>(epi, nb * BN, BN))
        ok = gemm_epilogue_beside<BN, MACO_EPI_GELU_DUAL>(BN, c, tmem_base, epi, epi.out, 0, mb * kBM, nb * BN, seq, budget_ns, 0, block);
      else if (!BESIDE && epi_is_stepped(epi, nb * BN, BN))
        ok = gemm_epilogue_stepped<BN>(BN, c, tmem_base, epi, epi.out, 0, mb * kBM, nb * BN, seq, budget_ns, 0, block);
      else
        ok = gemm_epilogue_tile<BN, BN, BESIDE ? MACO_EPI_GELU_DUAL : 0>(c, tmem_base, epi, epi.out, 0, mb * kBM, nb * BN, seq, budget_ns);
    }
  }
  gemm_cta_teardown<BN>(c, tmem_base, status);
}

}  // namespace maco
