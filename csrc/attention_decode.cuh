// Split-KV decode attention for grouped-query attention (one KV head shared by G <= 8 query
// heads, head_dim 128), as tasks of the persistent kernel, plus the merge of the split partials.
//
// The reference only names ATTENTION / SOFTMAX in its task enum (maco/csrc/maco_types.h:48,53)
// and computes attention as softmax(QK^T)V with O(S^2) memory in an example
// (examples/test_overlap_attention.py:111-113). Decode attention is bound by streaming the KV
// cache from HBM, so the task reads every K and V row exactly once with 16-byte loads, keeps the
// G query rows in shared memory and carries the usual running (max, sum, output) triple, which
// also is what a ring / context-parallel merge needs.
//
// Task ATTENTION, arguments in MacoEltArgs:
//   in0 = q [G, 128]   in1 = K rows [rows, ld_in]   in2 = V rows [rows, ld_in]   (bf16 or fp16)
//   out = fp32 partial: o[G*128] (unnormalised), m[G], l[G]
//   rows = keys in this split, cols = 128, i0 = G, f0 = softmax scale
// Task ATTN_MERGE:
//   in0 = partials [i1 splits][G*128 + 2G] fp32, out = o [G, 128] (dtype), i0 = G, i1 = splits
#pragma once
#include <cuda.h>
#include "elementwise.cuh"

namespace maco {

constexpr int kAttnD = 128;
constexpr int kAttnMaxG = 8;

__device__ __forceinline__ void attn_bar() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// Shared memory needed by attn_decode_task.
constexpr int kAttnVStageKeys = 64;
constexpr int kAttnScratchBytes = (2 * kAttnMaxG * kAttnD + 8 * kAttnMaxG) * 4 + kAttnVStageKeys * kAttnD * 2;

template <int DTT>
__device__ __noinline__ void attn_decode_task_t(const MacoEltArgs& ar, int tid, uint8_t* scratch) {
  const MacoEltArgs a = ar;
  const int G = a.i0 < kAttnMaxG ? a.i0 : kAttnMaxG;
  float* q_s = reinterpret_cast<float*>(scratch);                 // [G][128]
  float* p_s = q_s + kAttnMaxG * kAttnD;                          // [G][128] probabilities of the chunk
  float* red = p_s + kAttnMaxG * kAttnD;                          // [4][G] cross-warp scratch
  uint16_t* v_s = reinterpret_cast<uint16_t*>(red + 8 * kAttnMaxG);   // [64][128] staged V rows (16-byte aligned)
  const int warp = tid >> 5, lane = tid & 31;
  for (int i = tid; i < G * kAttnD; i += 128) q_s[i] = load1(a.in0, i, DTT) * a.f0;
  float m_run[kAttnMaxG], l_run[kAttnMaxG], o[kAttnMaxG];
#pragma unroll
  for (int g = 0; g < kAttnMaxG; ++g) { m_run[g] = -INFINITY; l_run[g] = 0.f; o[g] = 0.f; }
  attn_bar();
  const uint16_t* K = reinterpret_cast<const uint16_t*>(a.in1);
  const uint16_t* V = reinterpret_cast<const uint16_t*>(a.in2);
  for (int base = 0; base < a.rows; base += 128) {
    const int j = base + tid;
    const bool valid = j < a.rows;
    float s[kAttnMaxG];
#pragma unroll
    for (int g = 0; g < kAttnMaxG; ++g) s[g] = 0.f;
    // one key row per thread: all 16 vector loads of the row are issued before the first use
    uint4 kr[kAttnD / 8];
    const uint4* krow = reinterpret_cast<const uint4*>(K + (long long)(valid ? j : 0) * a.ld_in);
#pragma unroll
    for (int v = 0; v < kAttnD / 8; ++v) kr[v] = valid ? ld_global_nc_v4(krow + v) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int v = 0; v < kAttnD / 8; ++v) {
      float kf[8];
      const uint32_t w[4] = {kr[v].x, kr[v].y, kr[v].z, kr[v].w};
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        float2 f = DTT == MACO_DT_BF16 ? unpack_bf16x2(w[t]) : __half22float2(*reinterpret_cast<const __half2*>(&w[t]));
        kf[2 * t] = f.x; kf[2 * t + 1] = f.y;
      }
#pragma unroll
      for (int g = 0; g < kAttnMaxG; ++g) {
        if (g < G) {
          const float4 q0 = *reinterpret_cast<const float4*>(q_s + g * kAttnD + v * 8);
          const float4 q1 = *reinterpret_cast<const float4*>(q_s + g * kAttnD + v * 8 + 4);
          s[g] += q0.x * kf[0] + q0.y * kf[1] + q0.z * kf[2] + q0.w * kf[3] + q1.x * kf[4] + q1.y * kf[5] +
                  q1.z * kf[6] + q1.w * kf[7];
        }
      }
    }
    // chunk maximum per head
#pragma unroll
    for (int g = 0; g < kAttnMaxG; ++g) {
      float mx = warp_max(valid ? s[g] : -INFINITY);
      if (lane == 0) red[warp * kAttnMaxG + g] = mx;
    }
    attn_bar();
    float corr[kAttnMaxG];
#pragma unroll
    for (int g = 0; g < kAttnMaxG; ++g) {
      const float cm = fmaxf(fmaxf(red[g], red[kAttnMaxG + g]), fmaxf(red[2 * kAttnMaxG + g], red[3 * kAttnMaxG + g]));
      const float m_new = fmaxf(m_run[g], cm);
      corr[g] = (m_run[g] == -INFINITY) ? 0.f : __expf(m_run[g] - m_new);
      const float pj = valid ? __expf(s[g] - m_new) : 0.f;
      p_s[g * kAttnD + tid] = pj;
      s[g] = pj;
      m_run[g] = m_new;
    }
    attn_bar();                                   // red consumed, p_s complete
#pragma unroll
    for (int g = 0; g < kAttnMaxG; ++g) {
      float sm = warp_sum(s[g]);
      if (lane == 0) red[warp * kAttnMaxG + g] = sm;
    }
#pragma unroll
    for (int g = 0; g < kAttnMaxG; ++g) o[g] *= corr[g];
    // P·V: V rows are staged 64 at a time with coalesced 16-byte loads (8 per thread in flight);
    // thread `tid` then owns output dimension `tid` of every head and reads the staged rows.
    const int nk = min(128, a.rows - base);
    for (int h0 = 0; h0 < nk; h0 += kAttnVStageKeys) {
      const int hk = min(kAttnVStageKeys, nk - h0);
      const uint4* vsrc = reinterpret_cast<const uint4*>(V + (long long)(base + h0) * a.ld_in);
      const int nvec = hk * (kAttnD / 8);
      if (a.ld_in == kAttnD) {
#pragma unroll
        for (int u = 0; u < kAttnVStageKeys * (kAttnD / 8) / 128; ++u) {
          const int i = tid + u * 128;
          if (i < nvec) reinterpret_cast<uint4*>(v_s)[i] = ld_global_nc_v4(vsrc + i);
        }
      } else {
        for (int i = tid; i < nvec; i += 128)
          reinterpret_cast<uint4*>(v_s)[i] = ld_global_nc_v4(reinterpret_cast<const uint4*>(V + (long long)(base + h0 + i / 16) * a.ld_in) + (i & 15));
      }
      attn_bar();
      int jj = 0;
      for (; jj + 4 <= hk; jj += 4) {
        float vv[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const uint16_t raw = v_s[(jj + t) * kAttnD + tid];
          vv[t] = DTT == MACO_DT_BF16 ? __uint_as_float((uint32_t)raw << 16) : __half2float(*reinterpret_cast<const __half*>(&raw));
        }
#pragma unroll
        for (int g = 0; g < kAttnMaxG; ++g) {
          if (g < G) {
            const float4 pp = *reinterpret_cast<const float4*>(p_s + g * kAttnD + h0 + jj);
            o[g] += pp.x * vv[0] + pp.y * vv[1] + pp.z * vv[2] + pp.w * vv[3];
          }
        }
      }
      for (; jj < hk; ++jj) {
        const uint16_t raw = v_s[jj * kAttnD + tid];
        const float v1 = DTT == MACO_DT_BF16 ? __uint_as_float((uint32_t)raw << 16) : __half2float(*reinterpret_cast<const __half*>(&raw));
#pragma unroll
        for (int g = 0; g < kAttnMaxG; ++g) if (g < G) o[g] += p_s[g * kAttnD + h0 + jj] * v1;
      }
      attn_bar();                                 // v_s free for the next half
    }
#pragma unroll
    for (int g = 0; g < kAttnMaxG; ++g)
      l_run[g] = l_run[g] * corr[g] + red[g] + red[kAttnMaxG + g] + red[2 * kAttnMaxG + g] + red[3 * kAttnMaxG + g];
    attn_bar();                                   // red and p_s free for the next chunk
  }
  float* out = reinterpret_cast<float*>(a.out);
#pragma unroll
  for (int g = 0; g < kAttnMaxG; ++g) if (g < G) out[g * kAttnD + tid] = o[g];
  if (tid < G) {
    float mg = -INFINITY, lg = 0.f;
#pragma unroll
    for (int g = 0; g < kAttnMaxG; ++g) if (g == tid) { mg = m_run[g]; lg = l_run[g]; }
    out[G * kAttnD + tid] = mg;
    out[G * kAttnD + G + tid] = lg;
  }
}

// ---- streaming form -----------------------------------------------------------------------------
// Decode attention of one key range of one (sequence, kv head), bound by streaming K and V out of HBM. A TMA warp
// brings 128-key chunks of K and V (two boxes of 64 dims x 128 keys each, 128-byte swizzle) through a ring of six 32 KB
// stages (192 KB in flight per SM); four warps consume it. Warp w owns keys [32 w, 32 w + 32) of every chunk and
// keeps its own softmax state, so there is no barrier among the warps before the range is done:
//
//   S^T[key, head] = K . Q^T       keys on the M = 16 side, the G <= 8 heads are the N = 8 columns
//   P = exp2(S - m)                m is lazy: it moves only when a score exceeds it by more than kAttnLazyMargin
//   O^T[dim, head] += V^T . P      V through ldmatrix.trans, P turned into the B operand by movmatrix
//
// Warp-level mma.sync on purpose. The op does 4 G flops per byte of K / V read (0.05 of the tensor rate at the HBM rate),
// so what counts is the latency from "chunk landed" to "stage free". The tcgen05 form of this task (128 x 16 x 128
// products from shared memory, scores read back from TMEM, P staged for all warps behind a block barrier, one thread
// issuing) needed about 1.9 us per 64 KB chunk and SM against 1.4 us at the HBM rate; a warp's chain here (16 ldmatrix,
// 16 + 16 mma, two exponentials per lane and key pair) takes about 0.4 us per chunk with the four warps side by side.
// 537 MB of K / V (batch 16, 8 kv heads, 8192 keys, one B200): 117 us through the tcgen05 form, 86-87 us through this one (6.2 TB/s).
constexpr int kAttnStages = 6;
constexpr int kAttnStageBytes = 32768;               // one 128-key chunk of K or of V
constexpr int kAttnHalfBytes = 16384;                // its 64-dim half
constexpr float kAttnLazyMargin = 11.5f;             // in log2 units: P <= 2^11.5 (e^8) between two moves of the reference
constexpr int kAttnTcScratchBytes = 1024 + 4 * kAttnMaxG * kAttnD * 4;

// K / V tensor maps: 4-D (dim, key, head, batch); a chunk that runs past the last key reads zeros.
MACO_DEVICE void attn_load_box(void* dst, const void* tmap, uint64_t* bar, int x, int key, int head, int batch, uint64_t pol) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cta.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5, %6}], [%2], %7;"
      :: "r"(smem_u32(dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(x), "r"(key), "r"(head), "r"(batch), "l"(pol) : "memory");
}
MACO_DEVICE uint64_t attn_evict_first() {            // every K / V row is read once
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
// Both stages of one chunk (K, then V); a whole, converged warp. `ait` counts stage uses.
MACO_DEVICE bool attn_load_chunk(uint8_t* ring, uint64_t* full, uint64_t* empty, const void* tmK, const void* tmV, int key, int head, int batch,
                                 uint32_t& ait, uint64_t pol, uint64_t budget_ns, volatile uint32_t* abort_word) {
#pragma unroll
  for (int kv = 0; kv < 2; ++kv, ++ait) {
    const uint32_t s = ait % kAttnStages;
    if (!mbar_wait_warp(&empty[s], ((ait / kAttnStages) & 1) ^ 1, budget_ns, abort_word)) return false;
    if (elect_one()) {
      mbar_arrive_expect_tx(&full[s], kAttnStageBytes);
      uint8_t* dst = ring + (size_t)s * kAttnStageBytes;
      const void* tm = kv == 0 ? tmK : tmV;
      attn_load_box(dst, tm, &full[s], 0, key, head, batch, pol);
      attn_load_box(dst + kAttnHalfBytes, tm, &full[s], 64, key, head, batch, pol);
    }
  }
  return true;
}

MACO_DEVICE float attn_ex2(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
MACO_DEVICE void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
MACO_DEVICE void ldsm_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
MACO_DEVICE uint32_t movmatrix_trans(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}
template <int DTT>
MACO_DEVICE void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (DTT == MACO_DT_BF16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Two values rounded to 16 bits in one register; `r`: what they became.
template <int DTT>
MACO_DEVICE uint32_t attn_pack2(float x, float y, float2& r) {
  if constexpr (DTT == MACO_DT_BF16) {
    const uint32_t w = pack_bf16x2(x, y);
    r = unpack_bf16x2(w);
    return w;
  } else {
    const __half2 h = __floats2half2_rn(x, y);
    r = __half22float2(h);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
}

// A bounded wait of a whole warp with one verdict. Every lane waits for itself (the data must be visible to it); the vote keeps
// a warp together whose lanes gave up and saw the phase complete at the same moment.
MACO_DEVICE bool attn_wait_warp(uint64_t* bar, uint32_t parity, uint64_t budget_ns, volatile uint32_t* abort_word) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, budget_ns, abort_word)) != 0;
}

// 128 threads: attention of `rows` keys for the G query rows at `q`. On return (all threads behind a barrier) thread
// `tid` holds output dimension `tid` of every head: o[g] unnormalised, under the reference M[g] (log2 units) with
// denominator L[g]. `ait`: ring uses before this range (advanced); `bar`: barrier of the 128 threads.
//
// SPLIT_P keeps the probabilities at (nearly) fp32: each is the sum of two 16-bit values, hi and lo, and O takes one more product per
// 16 keys for lo; the denominator sums the unrounded ones. fp16 has few exponent bits, so there the probabilities are scaled by 2^12
// and the reference may lag by 2^3.5 only: products stay below 65504 and what lo drops is 2^-37 of the largest probability.
// (The extra mma all but hide behind the K / V stream: 16 x 8 heads x 8192 keys 87.1 us with them, 85.7 us without.)
template <int DTT, bool SPLIT_P, typename BarFn>
MACO_DEVICE bool attn_consume_range(const void* q, int G, int rows, float scale_log2, uint8_t* ring, uint64_t* full, uint64_t* empty,
                                    uint32_t& ait, uint8_t* scratch, int tid, uint64_t budget_ns, volatile uint32_t* abort_word, BarFn bar,
                                    float (&o)[kAttnMaxG], float (&M)[kAttnMaxG], float (&L)[kAttnMaxG]) {
  const int warp = tid >> 5, lane = tid & 31, hc = 2 * (lane & 3);     // this lane's two heads (columns of S^T and O^T)
  constexpr bool kScaled = SPLIT_P && DTT == MACO_DT_F16;
  constexpr float kMargin = kScaled ? 3.5f : kAttnLazyMargin, kShift = kScaled ? 12.f : 0.f;
  uint32_t qf[8][2];                                 // Q as the B operand: head lane / 4, dims 16 k + 2 (lane % 4) + {0, 1, 8, 9}
  {
    const uint32_t* qrow = reinterpret_cast<const uint32_t*>(q) + (lane >> 2) * (kAttnD / 2) + (lane & 3);
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int h = 0; h < 2; ++h) qf[k][h] = (lane >> 2) < G ? qrow[k * 8 + h * 4] : 0u;
  }
  float acc[8][4];                                   // O^T: dims 16 t + lane / 4 (+ 8), heads hc, hc + 1
#pragma unroll
  for (int t = 0; t < 8; ++t)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[t][j] = 0.f;
  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
  // ldmatrix row addresses inside a 64-dim half: K rows in order, V rows with the two 8-key blocks on the upper lanes
  const uint32_t k_row = (uint32_t)(warp * 32 + (lane & 15)), k_chunk = (uint32_t)(lane >> 4);
  const uint32_t v_row = (uint32_t)(warp * 32 + (lane & 7) + ((lane >> 4) & 1) * 8), v_chunk = (uint32_t)((lane >> 3) & 1);
  const uint32_t ring_s = smem_u32(ring);
  const uint32_t ait_end = ait + 2u * (uint32_t)((rows + 127) / 128);
  bool ok;
#pragma unroll 1
  for (int base = 0; base < rows; base += 128, ait += 2) {
    const int n_w = rows - base - warp * 32;         // keys of this warp in the chunk (may be <= 0 or more than 32)
    const uint32_t sk = ait % kAttnStages, sv = (ait + 1) % kAttnStages;
    if (!attn_wait_warp(&full[sk], (ait / kAttnStages) & 1, budget_ns, abort_word)) break;
    uint32_t pb[2][2], pl[2][2];                     // P and, with SPLIT_P, what its rounding left
    if (n_w > 0) {
      float s[2][4];
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[t][j] = 0.f;
      const uint32_t kb = ring_s + sk * kAttnStageBytes + k_row * 128;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t off = (uint32_t)(k >> 2) * kAttnHalfBytes + (((((uint32_t)k & 3) * 2 + k_chunk) ^ (k_row & 7)) << 4);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          uint32_t a[4];
          ldsm_x4(kb + t * 2048 + off, a);
          mma_16816<DTT>(s[t], a, qf[k][0], qf[k][1]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[sk]);
      float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int key = t * 16 + (lane >> 2) + (j >> 1) * 8;
          s[t][j] = key < n_w ? s[t][j] * scale_log2 : -INFINITY;
          if (j & 1) mx1 = fmaxf(mx1, s[t][j]); else mx0 = fmaxf(mx0, s[t][j]);
        }
      if (__any_sync(0xffffffffu, mx0 > m0 + kMargin || mx1 > m1 + kMargin)) {
#pragma unroll
        for (int d = 4; d < 32; d <<= 1) {
          mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, d));
          mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, d));
        }
        const float n0 = fmaxf(m0, mx0), n1 = fmaxf(m1, mx1);
        const float c0 = m0 == -INFINITY ? 0.f : attn_ex2(m0 - n0), c1 = m1 == -INFINITY ? 0.f : attn_ex2(m1 - n1);
        l0 *= c0; l1 *= c1;
#pragma unroll
        for (int t = 0; t < 8; ++t) { acc[t][0] *= c0; acc[t][1] *= c1; acc[t][2] *= c0; acc[t][3] *= c1; }
        m0 = n0; m1 = n1;
      }
      // (a block whose scores are all -inf leaves the reference at -inf: its probabilities are 0, not exp2(-inf + inf))
      const float r0 = (m0 == -INFINITY ? 0.f : m0) - kShift, r1 = (m1 == -INFINITY ? 0.f : m1) - kShift;
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          // without SPLIT_P the product uses the rounded probabilities, and the denominator sums the same ones
          const float p0 = attn_ex2(s[t][2 * h] - r0), p1 = attn_ex2(s[t][2 * h + 1] - r1);
          float2 r;
          const uint32_t w = attn_pack2<DTT>(p0, p1, r);
          pb[t][h] = movmatrix_trans(w);             // (key, head pair) -> (head, key pair): the B operand
          if constexpr (SPLIT_P) {
            float2 rest;
            pl[t][h] = movmatrix_trans(attn_pack2<DTT>(p0 - r.x, p1 - r.y, rest));
            l0 += p0; l1 += p1;
          } else {
            l0 += r.x; l1 += r.y;
          }
        }
    } else if (lane == 0) {
      mbar_arrive(&empty[sk]);
    }
    if (!attn_wait_warp(&full[sv], ((ait + 1) / kAttnStages) & 1, budget_ns, abort_word)) break;
    if (n_w > 0) {
      const uint32_t vb = ring_s + sv * kAttnStageBytes + v_row * 128;
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const uint32_t off = (uint32_t)(t >> 2) * kAttnHalfBytes + (((((uint32_t)t & 3) * 2 + v_chunk) ^ (v_row & 7)) << 4);
#pragma unroll
        for (int kt = 0; kt < 2; ++kt) {
          uint32_t a[4];
          ldsm_x4_trans(vb + kt * 2048 + off, a);
          mma_16816<DTT>(acc[t], a, pb[kt][0], pb[kt][1]);
          if constexpr (SPLIT_P) mma_16816<DTT>(acc[t], a, pl[kt][0], pl[kt][1]);
        }
      }
      __syncwarp();
    }
    if (lane == 0) mbar_arrive(&empty[sv]);
  }
  ait = ait_end;
  // combine the four warps: {m, l} per head and O per (head, dim) through shared memory
#pragma unroll
  for (int d = 4; d < 32; d <<= 1) {
    l0 += __shfl_xor_sync(0xffffffffu, l0, d);
    l1 += __shfl_xor_sync(0xffffffffu, l1, d);
  }
  float* red = reinterpret_cast<float*>(scratch);    // [4 warps][8 heads] m, then l; O behind it
  float* ro = red + 256;
  if (lane < 4) {
    red[warp * 8 + hc] = m0; red[warp * 8 + hc + 1] = m1;
    red[32 + warp * 8 + hc] = l0; red[32 + warp * 8 + hc + 1] = l1;
  }
#pragma unroll
  for (int t = 0; t < 8; ++t)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      ro[(warp * kAttnMaxG + hc + (j & 1)) * kAttnD + t * 16 + (lane >> 2) + (j >> 1) * 8] = acc[t][j];
  bar();
  // one verdict for all threads (a wait that ran out has set the abort word): callers leave or go on together
  if (tid == 0) red[128] = *abort_word != 0 ? 1.f : 0.f;
#pragma unroll
  for (int g = 0; g < kAttnMaxG; ++g) {
    M[g] = fmaxf(fmaxf(red[g], red[8 + g]), fmaxf(red[16 + g], red[24 + g]));
    o[g] = 0.f; L[g] = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float c = red[w * 8 + g] == -INFINITY ? 0.f : attn_ex2(red[w * 8 + g] - M[g]);
      L[g] += red[32 + w * 8 + g] * c;
      o[g] += ro[(w * kAttnMaxG + g) * kAttnD + tid] * c;
    }
  }
  bar();
  ok = red[128] == 0.f;
  bar();                                             // scratch may be used again
  return ok;
}

// One record {o[G][128], m[G], l[G]} (m in log2 units) of a key range.
MACO_DEVICE void attn_store_record(float* rec, int G, int tid, const float (&o)[kAttnMaxG], const float (&M)[kAttnMaxG], const float (&L)[kAttnMaxG]) {
#pragma unroll
  for (int g = 0; g < kAttnMaxG; ++g) {
    if (g < G) {
      rec[g * kAttnD + tid] = o[g];
      if (tid == g) { rec[G * kAttnD + g] = M[g]; rec[G * kAttnD + G + g] = L[g]; }
    }
  }
}
// Output rows from n records; `rec_of(i)` is the address of record i. The loads of two records are in flight together (one record per
// turn is a round trip to L2 each: six records, a 700-key cache cut into 128-key pieces, took 5 us).
constexpr int kAttnMergeAhead = 2;
template <int DTT, typename RecFn>
MACO_DEVICE void attn_merge_records(void* out, int G, int n, int tid, RecFn rec_of) {
  float M[kAttnMaxG], L[kAttnMaxG], acc[kAttnMaxG];
#pragma unroll
  for (int g = 0; g < kAttnMaxG; ++g) { M[g] = -INFINITY; L[g] = 0.f; acc[g] = 0.f; }
#pragma unroll 1
  for (int i0 = 0; i0 < n; i0 += kAttnMergeAhead) {
    float ms[kAttnMergeAhead][kAttnMaxG], ls[kAttnMergeAhead][kAttnMaxG], os[kAttnMergeAhead][kAttnMaxG];
#pragma unroll
    for (int i = 0; i < kAttnMergeAhead; ++i) {
      const bool have = i0 + i < n;
      const float* r = have ? rec_of(i0 + i) : nullptr;
#pragma unroll
      for (int g = 0; g < kAttnMaxG; ++g) {
        ms[i][g] = have && g < G ? __ldcg(r + G * kAttnD + g) : -INFINITY;
        ls[i][g] = have && g < G ? __ldcg(r + G * kAttnD + G + g) : 0.f;
        os[i][g] = have && g < G ? __ldcg(r + g * kAttnD + tid) : 0.f;
      }
    }
#pragma unroll
    for (int i = 0; i < kAttnMergeAhead; ++i)
#pragma unroll
      for (int g = 0; g < kAttnMaxG; ++g) {
        const float m = fmaxf(M[g], ms[i][g]);
        const float a = M[g] == -INFINITY ? 0.f : attn_ex2(M[g] - m), b = ms[i][g] == -INFINITY ? 0.f : attn_ex2(ms[i][g] - m);
        L[g] = L[g] * a + ls[i][g] * b;
        acc[g] = acc[g] * a + os[i][g] * b;
        M[g] = m;
      }
  }
#pragma unroll
  for (int g = 0; g < kAttnMaxG; ++g)
    if (g < G) store1(out, g * kAttnD + tid, DTT, L[g] > 0.f ? acc[g] / L[g] : 0.f);
}

// ---- the task of the persistent kernel: one key range of one (sequence, kv head) ----------------------------------
//   in0 = q rows, in1 = arrival counter of the (sequence, kv head), in2 = output rows, out = this range's record
//   row0 = first key, rows = keys, cols = index of the (sequence, kv head), f0 = softmax scale, f1 = index of the range,
//   i0 = G | first key a task of this program writes << 8 (0: every key waits for the task's conditions), i1 = ranges
//   ld_in = 128 and ld_out = tensor-map indices of K and V (+1 each, 16 bits each) mark this form
struct AttnPipe {
  uint8_t* ring;
  uint64_t* full;         // [kAttnStages]
  uint64_t* empty;        // [kAttnStages], four arrivals (one per consumer warp)
  uint64_t budget_ns;
  volatile uint32_t* abort_word;
};
MACO_DEVICE bool attn_pipelined(const MacoEltArgs& a) { return a.ld_in == kAttnD && a.rows > 0 && a.ld_out != 0; }
MACO_DEVICE uint32_t attn_stage_uses(const MacoEltArgs& a) { return 2u * (uint32_t)((a.rows + 127) / 128); }

// Waits (bounded) until the last uses of the attention ring have been released by the consumer: the
// operand memory may then be handed to another pipeline. A whole, converged warp.
MACO_DEVICE bool attn_ring_drained(const AttnPipe& pp, uint32_t ait) {
  for (uint32_t u = ait > (uint32_t)kAttnStages ? ait - kAttnStages : 0; u < ait; ++u)
    if (!mbar_wait_warp(&pp.empty[u % kAttnStages], (u / kAttnStages) & 1, pp.budget_ns, pp.abort_word)) return false;
  return true;
}

// After an abort: loads still in flight get a bounded time to land (their destination is this CTA's memory).
MACO_DEVICE void attn_drain_loads(const AttnPipe& pp, uint32_t ait) {
  for (uint32_t u = ait > (uint32_t)kAttnStages ? ait - kAttnStages : 0; u < ait; ++u) {
    const uint64_t t0 = globaltimer_ns();
    while (!mbar_try_wait(&pp.full[u % kAttnStages], (u / kAttnStages) & 1)) {
      if (globaltimer_ns() - t0 > 2000000ull) break;
    }
  }
}

// 128 general threads. The range that arrives last at the group's counter combines all of them (no separate merge task,
// no extra dependency hop); the counter only grows: i1 arrivals per launch.
template <int DTT, typename BarFn>
__device__ __noinline__ bool attn_task_t(const MacoEltArgs& ar, int tid, uint8_t* scratch, const AttnPipe& pipe, uint32_t& ait, volatile uint32_t* word,
                                         BarFn bar) {
  const MacoEltArgs a = ar;
  const AttnPipe pp = pipe;
  const int G = a.i0 & 0xff, S = a.i1;
  float o[kAttnMaxG], M[kAttnMaxG], L[kAttnMaxG];
  if (!attn_consume_range<DTT, false>(a.in0, G, a.rows, a.f0 * 1.4426950408889634f, pp.ring, pp.full, pp.empty, ait, scratch, tid, pp.budget_ns,
                               pp.abort_word, bar, o, M, L)) return false;
  void* out = const_cast<void*>(a.in2);
  if (S <= 1) {
#pragma unroll
    for (int g = 0; g < kAttnMaxG; ++g)
      if (g < G) store1(out, g * kAttnD + tid, DTT, L[g] > 0.f ? o[g] / L[g] : 0.f);
    return true;
  }
  float* rec = reinterpret_cast<float*>(a.out);
  attn_store_record(rec, G, tid, o, M, L);
  bar();
  if (tid == 0) {
    uint32_t* counter = reinterpret_cast<uint32_t*>(const_cast<void*>(a.in1));
    *word = ((atom_add_acq_rel_gpu_u32(counter, 1u) + 1u) % (uint32_t)S) == 0u ? 1u : 0u;
  }
  bar();
  if (*word != 0u) {
    const int n = G * kAttnD + 2 * G;
    const float* first = rec - (size_t)(int)a.f1 * n;
    attn_merge_records<DTT>(out, G, S, tid, [=](int i) { return first + (size_t)i * n; });
  }
  return true;
}

MACO_DEVICE void attn_decode_task(const MacoEltArgs& a, int tid, uint8_t* scratch) {
  if (a.dtype == MACO_DT_BF16) attn_decode_task_t<MACO_DT_BF16>(a, tid, scratch);
  else attn_decode_task_t<MACO_DT_F16>(a, tid, scratch);
}

// Combines the S split records {o[G][128], m[G], l[G]} of one (sequence, kv head): thread `tid` owns output
// dimension `tid` of every head. The loads of one split are independent of each other (8 heads in flight).
MACO_DEVICE void attn_merge_task(const MacoEltArgs& ar, int tid) {
  const MacoEltArgs a = ar;                              // private copy: stores cannot alias it
  const int G = a.i0 < kAttnMaxG ? a.i0 : kAttnMaxG, S = a.i1;
  const int rec = G * kAttnD + 2 * G;
  const float* part = reinterpret_cast<const float*>(a.in0);
  float M[kAttnMaxG], L[kAttnMaxG], acc[kAttnMaxG];
#pragma unroll
  for (int g = 0; g < kAttnMaxG; ++g) { M[g] = -INFINITY; L[g] = 0.f; acc[g] = 0.f; }
  for (int s = 0; s < S; ++s) {
#pragma unroll
    for (int g = 0; g < kAttnMaxG; ++g) if (g < G) M[g] = fmaxf(M[g], part[s * rec + G * kAttnD + g]);
  }
  for (int s = 0; s < S; ++s) {
    float ms[kAttnMaxG], ls[kAttnMaxG], os[kAttnMaxG];
#pragma unroll
    for (int g = 0; g < kAttnMaxG; ++g) {
      ms[g] = g < G ? part[s * rec + G * kAttnD + g] : -INFINITY;
      ls[g] = g < G ? part[s * rec + G * kAttnD + G + g] : 0.f;
      os[g] = g < G ? part[s * rec + g * kAttnD + tid] : 0.f;
    }
#pragma unroll
    for (int g = 0; g < kAttnMaxG; ++g) {
      const float w = (ms[g] == -INFINITY) ? 0.f : __expf(ms[g] - M[g]);
      L[g] += ls[g] * w;
      acc[g] += os[g] * w;
    }
  }
#pragma unroll
  for (int g = 0; g < kAttnMaxG; ++g) if (g < G) store1(a.out, g * kAttnD + tid, a.dtype, L[g] > 0.f ? acc[g] / L[g] : 0.f);
}

MACO_DEVICE void attn_run(uint32_t type, const MacoEltArgs& a, int tid, int nthreads, uint8_t* scratch) {
  (void)nthreads;
  if (type == MACO_TASK_ATTENTION) attn_decode_task(a, tid, scratch); else attn_merge_task(a, tid);
}

}  // namespace maco
