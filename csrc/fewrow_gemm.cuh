// Few-row GEMMs (decode: up to 64 tokens) as a weight stream, with the operands swapped.
//
//   out[token, feature] = op( sum_k x[token, k] * w[feature, k] ),  w read exactly once
//
// The op is bound by streaming w out of HBM, so the weights take the M = 128 rows of the instruction (128 features
// per tile) and the tokens its N columns (16, 32, 48 or 64): no MMA row and no shared memory is spent on padding a
// handful of tokens to 128, and a tile is 128 features wide instead of 256, so half as many partial sums per output
// are exchanged to keep every SM busy. A ring stage holds two k-blocks: 2 x 16 KB of weights and 2 x (tokens x 128) bytes
// of x, so the four 48 KB stages keep 128 KB of weights in flight per SM.
//
// Work split (ProgramBuilder.gemm_stream): equal parts of whole feature tiles, one part per worker; where the tiles do not divide well
// over the workers, all (feature tile, 128-wide k-step) pairs in one line, cut into one equal piece per worker. A part is a
// task that adds its fp32 sums into a [tokens, features] workspace. The accumulator has one feature per TMEM lane, so a
// warp's reduction instruction covers 128 consecutive bytes of one token's row. Whoever arrives last at a tile's counter finds
// every part summed and finishes the tile (operator, 16-bit store, workspace zeroed for the next launch) through shared
// memory in short loops; only that task signals the tile's event. (Zeroing in a pass of its own behind the signal cost 1 to 2 % where
// a worker has a second part, and gained nothing in a decode layer: 158.5 / 157.9 us at batch 64, 71.3 / 70.6 at batch 3.) A tile that
// is one part skips all that (few_direct).
// One B200, decode layer of batch 64: 190 -> 162 us with one part per worker instead of the line alone, 159 with few_direct.
#pragma once
#include "gemm_tcgen05.cuh"
#include "row_tasks.cuh"

namespace maco {

constexpr int kFewK = 2 * kBK;                       // k elements per stage
constexpr uint32_t kFewWBytes = 2u * kBM * kBK * 2u; // weight bytes per stage
constexpr uint8_t kFewFlag = 4;                      // MacoGemmArgs.b_mn bit of such a task
constexpr uint8_t kFewDirect = 8;                    // ... of one whose tile is one part: no workspace, no arrival
constexpr uint8_t kFewSplit = 16;                    // ... whose 128 rows are 64 gate features and the 64 up features of the same outputs

// Weights are read once per launch: evict-first keeps activations, workspaces and the kernel's own code in L2.
MACO_DEVICE uint64_t l2_evict_first() {
  uint64_t pol;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  return pol;
}
MACO_DEVICE void tma_load_2d_hint(void* smem_dst, const void* tmap, uint64_t* bar, int x, int y, uint64_t pol) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4}], [%2], %5;"
      :: "r"(smem_u32(smem_dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(x), "r"(y), "l"(pol) : "memory");
}

// ---- TMA warp (converged) ----------------------------------------------------------------------
template <int STAGES, int STAGE_BYTES>
MACO_DEVICE bool few_load_weights(uint8_t* smem, const GemmCtrl& c, const CUtensorMap* tmW, const MacoGemmArgs& g, uint32_t u,
                                  uint32_t step, uint64_t pol, uint64_t budget_ns) {
  const uint32_t s = u % STAGES, ph = (u / STAGES) & 1;
  if (!mbar_wait_warp(&c.empty[s], ph ^ 1, budget_ns, c.abort_word)) return false;
  const int k = warp_uniform(g.k0) + (int)step * kFewK, m0 = warp_uniform(g.m0);
  const bool split = warp_uniform((int)g.b_mn & kFewSplit) != 0;
  if (elect_one()) {
    mbar_arrive_expect_tx(&c.full[s], kFewWBytes + g.bn * (kFewK * 2u));
    uint8_t* sw = smem + s * STAGE_BYTES;
    if (split) {                                     // boxes of 64 rows (gate and up alternate in blocks of 128)
#pragma unroll 1
      for (int i = 0; i < 4; ++i) tma_load_2d_hint(sw + i * (kFewWBytes / 4), tmW, &c.full[s], k + (i >> 1) * kBK, m0 + (i & 1) * 128, pol);
    } else {
      tma_load_2d_hint(sw, tmW, &c.full[s], k, m0, pol);
      tma_load_2d_hint(sw + kFewWBytes / 2, tmW, &c.full[s], k + kBK, m0, pol);
    }
  }
  return true;
}
template <int STAGES, int STAGE_BYTES>
MACO_DEVICE void few_load_tokens(uint8_t* smem, const GemmCtrl& c, const CUtensorMap* tmX, const MacoGemmArgs& g, uint32_t u, uint32_t step) {
  const uint32_t s = u % STAGES;
  uint8_t* sx = smem + s * STAGE_BYTES + kFewWBytes;
  const int k = warp_uniform(g.k0) + (int)step * kFewK;
  const uint32_t half = warp_uniform(g.bn) * (kBK * 2u);
  if (elect_one()) {
    tma_load_2d(sx, tmX, &c.full[s], k, 0);
    tma_load_2d(sx + half, tmX, &c.full[s], k + kBK, 0);
  }
}

// ---- MMA warp (converged) ----------------------------------------------------------------------
template <int STAGES, int STAGE_BYTES, int ACC_COLS>
MACO_DEVICE bool few_mma_tile(uint8_t* smem, const GemmCtrl& c, uint32_t tmem_base, const MacoGemmArgs& g, uint32_t& it, uint32_t tile_seq,
                              uint64_t budget_ns) {
  const uint32_t acc = tile_seq & 1, acc_ph = (tile_seq >> 1) & 1, idesc = warp_uniform(g.idesc);
  const int steps = warp_uniform(g.k_blocks);
  if (!mbar_wait_warp(&c.tmem_empty[acc], acc_ph ^ 1, budget_ns, c.abort_word)) return false;
  tc_fence_after();
  const uint32_t d_tmem = warp_uniform(tmem_base) + acc * ACC_COLS;
  const uint64_t d0 = make_smem_desc(0, 16, 1024, 2);
  const uint32_t hi = (uint32_t)(d0 >> 32), lbo = (uint32_t)d0;
  const uint32_t base_lo = (smem_u32(smem) & 0x3FFFFu) >> 4, x_half = warp_uniform(g.bn) * (kBK * 2u) >> 4;
  for (int st = 0; st < steps; ++st) {
    const uint32_t u = it + (uint32_t)st, s = u % STAGES;
    if (!mbar_wait_warp(&c.full[s], (u / STAGES) & 1, budget_ns, c.abort_word)) { it = u; return false; }
    if (elect_one()) {
      uint32_t w_lo = base_lo + s * (STAGE_BYTES >> 4), x_lo = w_lo + (kFewWBytes >> 4);
#pragma unroll
      for (int half = 0; half < 2; ++half) {
#pragma unroll
        for (int k = 0; k < kBK / kUmmaK; ++k)
          tc_mma_f16_lo(d_tmem, (w_lo + k * 2) | lbo, hi, (x_lo + k * 2) | lbo, hi, idesc, half + k == 0 ? (st != 0 ? 1u : 0u) : 1u);
        w_lo += kFewWBytes >> 5;
        x_lo += x_half;
      }
      tc_commit(&c.empty[s]);
    }
  }
  it += (uint32_t)steps;
  if (elect_one()) tc_commit(&c.tmem_full[acc]);
  return true;
}

// ---- finishing pass of one feature tile (or gate / up pair of tiles): 128 threads --------------
MACO_DEVICE uint32_t few_pack2(int dtype, float x, float y) {
  if (dtype == MACO_DT_BF16) return pack_bf16x2(x, y);
  const __half2 h = __floats2half2_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&h);
}
MACO_DEVICE float2 few_unpack2(int dtype, uint32_t w) {
  return dtype == MACO_DT_BF16 ? unpack_bf16x2(w) : __half22float2(*reinterpret_cast<const __half2*>(&w));
}
MACO_DEVICE float4 few_lds_f4(uint32_t saddr) {
  const uint4 u = lds_v4(saddr);
  return make_float4(__uint_as_float(u.x), __uint_as_float(u.y), __uint_as_float(u.z), __uint_as_float(u.w));
}

// Operators 0 (store), 1 (SwiGLU: 128 gate features, then the 128 up features of the same outputs), 2 (+ residual):
// a unit is 8 output values of one token; a thread stages its own units, as many as the scratch block holds.
MACO_DEVICE void few_finish_rows(const MacoEltArgs& fa, int m0, int tid, uint8_t* scratch) {
  const int mode = fa.i0, dt = fa.dtype;
  const uint32_t V = mode == 1 ? 4u : (mode == 2 ? 3u : 2u), U = 14u / V;
  const int n0 = mode == 1 ? (m0 & ~255) : m0, c0 = mode == 1 ? n0 >> 1 : n0;
  float* ws = const_cast<float*>(reinterpret_cast<const float*>(fa.in0)) + n0;
  const uint16_t* aux = reinterpret_cast<const uint16_t*>(fa.in1) + c0;
  uint16_t* out = reinterpret_cast<uint16_t*>(fa.out) + c0;
  const uint32_t units = (uint32_t)fa.rows * 16u;
  const uint32_t s0 = smem_u32(scratch) + (uint32_t)tid * 16u;
#pragma unroll 1
  for (uint32_t base = 0; base < units; base += U * 128u) {
#pragma unroll 1
    for (uint32_t k = 0; k < U; ++k) {
      const uint32_t u = base + k * 128u + (uint32_t)tid;
      if (u < units) {
        const uint32_t t = u >> 4, col = (u & 15u) * 8u, s = s0 + k * V * 2048u;
        const float* src = ws + (size_t)t * fa.ld_in + col;
        cp_async16(s, src);
        cp_async16(s + 2048u, src + 4);
        if (mode == 1) { cp_async16(s + 4096u, src + 128); cp_async16(s + 6144u, src + 132); }
        else if (mode == 2) cp_async16(s + 4096u, aux + (size_t)t * fa.ld_out + col);
      }
    }
    cp_async_commit();
    cp_async_wait<0>();
#pragma unroll 1
    for (uint32_t k = 0; k < U; ++k) {
      const uint32_t u = base + k * 128u + (uint32_t)tid;
      if (u >= units) break;
      const uint32_t t = u >> 4, col = (u & 15u) * 8u, s = s0 + k * V * 2048u;
      float4* src = reinterpret_cast<float4*>(ws + (size_t)t * fa.ld_in + col);
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      src[0] = zero; src[1] = zero;
      const float4 a = few_lds_f4(s), b = few_lds_f4(s + 2048u);
      float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      if (mode == 1) {
        src[32] = zero; src[33] = zero;
        const float4 c = few_lds_f4(s + 4096u), d = few_lds_f4(s + 6144u);
        const float up[8] = {c.x, c.y, c.z, c.w, d.x, d.y, d.z, d.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = silu_16(v[j]) * up[j];
      } else if (mode == 2) {
        const uint4 r = lds_v4(s + 4096u);
        const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) { const float2 f = few_unpack2(dt, rw[j]); v[2 * j] += f.x; v[2 * j + 1] += f.y; }
      }
      *reinterpret_cast<uint4*>(out + (size_t)t * fa.ld_out + col) =
          make_uint4(few_pack2(dt, v[0], v[1]), few_pack2(dt, v[2], v[3]), few_pack2(dt, v[4], v[5]), few_pack2(dt, v[6], v[7]));
    }
  }
}

// Operator 3: the tile is one head of a fused QKV projection. One warp per token: QK-norm and RoPE for query and key
// heads, then into q or into the new token's cache row (see MacoQkRopeParams); a lane owns elements {2l, 2l + 1} of both
// halves of the head (the pairs RoPE rotates).
MACO_DEVICE void few_finish_qkrope(const MacoEltArgs& fa, int m0, int tid, uint8_t* scratch) {
  const MacoQkRopeParams q = *reinterpret_cast<const MacoQkRopeParams*>(fa.in1);
  const int warp = tid >> 5, lane = tid & 31, head = m0 >> 7, dt = q.dtype, M = fa.rows;
  const bool is_q = head < q.hq, is_v = head >= q.hq + q.hkv;
  float* ws = const_cast<float*>(reinterpret_cast<const float*>(fa.in0)) + m0;
  const uint32_t* wn = reinterpret_cast<const uint32_t*>(is_q ? q.q_norm : q.k_norm);
  const float2 w1 = few_unpack2(dt, wn[lane]), w2 = few_unpack2(dt, wn[32 + lane]);
  const uint8_t* cs = reinterpret_cast<const uint8_t*>(q.cos_sin);
  uint16_t* dst;
  long long pitch;
  if (is_q) {
    dst = reinterpret_cast<uint16_t*>(q.q_out) + head * 128; pitch = (long long)q.hq * 128;
  } else {
    dst = is_v ? reinterpret_cast<uint16_t*>(q.v_cache) + (head - q.hq - q.hkv) * q.kv_head_stride
               : reinterpret_cast<uint16_t*>(q.k_cache) + (head - q.hq) * q.kv_head_stride;
    dst += (long long)q.pos * 128; pitch = q.kv_batch_stride;
  }
  constexpr int kTok = 8;                            // tokens a warp stages at a time: 512 bytes of sums, 256 of cos / sin each
  uint8_t* mine = scratch + warp * (kTok * 768);
  const uint32_t s0 = smem_u32(mine);
#pragma unroll 1
  for (int t0 = warp * kTok; t0 < M; t0 += 4 * kTok) {
    const int n = min(kTok, M - t0);
#pragma unroll 1
    for (int j = 0; j < n; ++j) {
      cp_async16(s0 + j * 768 + lane * 16, ws + (size_t)(t0 + j) * fa.ld_in + lane * 4);
      if (lane < 16) cp_async16(s0 + j * 768 + 512 + lane * 16, cs + (size_t)(t0 + j) * 256 + lane * 16);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();
#pragma unroll 1
    for (int j = 0; j < n; ++j) {
      reinterpret_cast<float4*>(ws + (size_t)(t0 + j) * fa.ld_in)[lane] = make_float4(0.f, 0.f, 0.f, 0.f);
      const float2* x = reinterpret_cast<const float2*>(mine + j * 768);
      const uint32_t* c = reinterpret_cast<const uint32_t*>(mine + j * 768 + 512);
      // the projection's result in the layer's 16-bit type first (what a separate pass would have read)
      const float2 x1 = x[lane], x2 = x[32 + lane];
      uint32_t p1 = few_pack2(dt, x1.x, x1.y), p2 = few_pack2(dt, x2.x, x2.y);
      if (!is_v) {
        float2 a1 = few_unpack2(dt, p1), a2 = few_unpack2(dt, p2);
        const float2 cc = few_unpack2(dt, c[lane]), sn = few_unpack2(dt, c[32 + lane]);
        const float rstd = rsqrtf(warp_sum(a1.x * a1.x + a1.y * a1.y + a2.x * a2.x + a2.y * a2.y) / 128.f + q.eps);
        a1.x *= rstd * w1.x; a1.y *= rstd * w1.y; a2.x *= rstd * w2.x; a2.y *= rstd * w2.y;
        p1 = few_pack2(dt, a1.x * cc.x - a2.x * sn.x, a1.y * cc.y - a2.y * sn.y);
        p2 = few_pack2(dt, a2.x * cc.x + a1.x * sn.x, a2.y * cc.y + a1.y * sn.y);
      }
      uint32_t* o = reinterpret_cast<uint32_t*>(dst + (t0 + j) * pitch);
      o[lane] = p1; o[32 + lane] = p2;
    }
    __syncwarp();
  }
}

// A tile that is one part goes from the accumulator to the result through shared memory, 32 tokens at a time. Gate and up features of
// an output lie in one tile then (kFewSplit), so that SwiGLU needs no other worker. Against reductions into the workspace, an arrival
// and a finishing pass: 4 us instead of 11 at the end of a gate / up projection of 64 tokens.
template <int ACC_COLS, typename BarFn>
__device__ __noinline__ bool few_direct(const GemmCtrl& c, uint32_t tmem_base, const MacoEltArgs& fa, const MacoGemmArgs& g, int tid, uint32_t acc,
                                        bool ok, uint8_t* scratch, volatile uint32_t* word, BarFn bar) {
  const int M = fa.rows, mode = fa.i0, dt = fa.dtype, m0 = g.m0;
  const uint32_t lane = threadIdx.x & 31, quarter = (threadIdx.x >> 5) & 3;
  const uint32_t t_row = tmem_base + ((quarter * 32u) << 16) + acc * ACC_COLS;
  float* sums = reinterpret_cast<float*>(scratch);                     // [32 tokens][128 features]
  const int c0 = mode == 1 ? (m0 >> 8) * 128 + (m0 & 255) : m0;
  const uint32_t shift = mode == 1 ? 3 : 4;                            // 8-feature units per token: 8 or 16
#pragma unroll 1
  for (int t0 = 0; t0 < M; t0 += 32) {
    if (ok) {
#pragma unroll 1
      for (int h = 0; h < 32 && t0 + h < M; h += 16) {
        uint32_t r[16];
        tmem_ld_32x16(t_row + (uint32_t)(t0 + h), r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) sums[(h + j) * 128 + quarter * 32 + lane] = __uint_as_float(r[j]);
      }
      if (t0 + 32 >= M) {
        tc_fence_before();
        mbar_arrive(&c.tmem_empty[acc]);
      }
    }
    bar();
    if (t0 == 0) {                                                     // one verdict for all threads, as in few_epilogue
      if (tid == 0) *word = *c.abort_word != 0 ? 2u : 1u;
      bar();
      if (*word == 2u) return false;
    }
    const uint32_t units = (uint32_t)min(32, M - t0) << shift;
#pragma unroll 1
    for (uint32_t u = tid; u < units; u += 128) {
      const uint32_t t = u >> shift, col = (u & ((1u << shift) - 1u)) * 8u;
      const size_t o = (size_t)(t0 + (int)t) * fa.ld_out + c0 + col;
      const float4* src = reinterpret_cast<const float4*>(sums + t * 128 + col);
      const float4 a = src[0], b = src[1];
      float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      if (mode == 1) {
        const float4 e = src[16], f = src[17];
        const float up[8] = {e.x, e.y, e.z, e.w, f.x, f.y, f.z, f.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = silu_16(v[j]) * up[j];
      } else if (mode == 2) {
        const uint4 r = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(fa.in1) + o);
        const uint32_t rw[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) { const float2 f = few_unpack2(dt, rw[j]); v[2 * j] += f.x; v[2 * j + 1] += f.y; }
      }
      *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(fa.out) + o) =
          make_uint4(few_pack2(dt, v[0], v[1]), few_pack2(dt, v[2], v[3]), few_pack2(dt, v[4], v[5]), few_pack2(dt, v[6], v[7]));
    }
    if (t0 + 32 < M) bar();                                            // the sums are read before the next tokens' take their place
  }
  return true;
}

// ---- general warps ----------------------------------------------------------------------------
// Returns 0 on failure, 1 when other parts of the tile are still to come, 2 when this task finished the tile.
// `word`: a shared control word; `bar`: the barrier of the 128 threads.
// (out of line: inlined into the task loop it takes registers from the GEMM epilogue beside it)
template <int ACC_COLS, typename BarFn>
__device__ __noinline__ int few_epilogue(const GemmCtrl& c, uint32_t tmem_base, const GemmEpilogue& e, const MacoGemmArgs& g, int tid,
                                         uint32_t tile_seq, uint64_t budget_ns, uint8_t* scratch, volatile uint32_t* word, BarFn bar) {
  float* ws = reinterpret_cast<float*>(e.out);
  const long long ld = e.ld_out;
  const int M = e.N;                                 // tokens
  uint32_t* counter = reinterpret_cast<uint32_t*>(const_cast<void*>(e.bias)) + g.row_off;
  const MacoEltArgs* fin = reinterpret_cast<const MacoEltArgs*>(e.aux);
  const uint32_t lane = threadIdx.x & 31, quarter = (threadIdx.x >> 5) & 3;
  const uint32_t acc = tile_seq & 1;
  uint32_t ok = 1;
  if (lane == 0) ok = mbar_wait(&c.tmem_full[acc], (tile_seq >> 1) & 1, budget_ns, c.abort_word) ? 1u : 0u;
  ok = __shfl_sync(0xffffffffu, ok, 0);
  if (g.b_mn & kFewDirect) {
    if (ok) tc_fence_after();
    return few_direct<ACC_COLS>(c, tmem_base, *fin, g, tid, acc, ok != 0, scratch, word, bar) ? 2 : 0;
  }
  if (ok) {                                            // (a warp whose wait ran out still meets the others at both barriers below)
    tc_fence_after();
    const uint32_t t_row = tmem_base + ((quarter * 32u) << 16) + acc * ACC_COLS;
    float* dst = ws + g.m0 + (int)(quarter * 32u + lane);
#pragma unroll 1
    for (int t0 = 0; t0 < M; t0 += 16) {
      uint32_t r[16];
      tmem_ld_32x16(t_row + (uint32_t)t0, r);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (t0 + j < M) asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" :: "l"(dst + (t0 + j) * ld), "f"(__uint_as_float(r[j])) : "memory");
      }
    }
    tc_fence_before();
    mbar_arrive(&c.tmem_empty[acc]);
  }
  bar();                                             // every thread's reductions are issued before the arrival
  // One verdict for all threads. A wait that ran out has set the abort word or seen it set, in front of the barrier; the
  // warps must not act on their own results, or some would leave while others wait at the next barrier.
  if (tid == 0) *word = *c.abort_word != 0 ? 2u : (((atom_add_acq_rel_gpu_u32(counter, 1u) + 1u) % g.count_base) == 0u ? 1u : 0u);
  bar();
  const uint32_t verdict = *word;
  if (verdict != 1u) return verdict == 2u ? 0 : 1;
  const MacoEltArgs fa = *fin;
  if (fa.i0 == 3) few_finish_qkrope(fa, g.m0, tid, scratch);
  else few_finish_rows(fa, g.m0, tid, scratch);
  return 2;
}

}  // namespace maco
