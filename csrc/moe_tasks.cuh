// Mixture-of-experts tasks of the persistent kernel: top-k routing fused with the dispatch
// all-to-all, publication of the per-expert counts, and the weighted return (combine) of expert
// outputs, all over NVLink peer memory from inside the kernel.
//
//   TOPK (dispatch)   per token: softmax top-k over the router logits, a slot in the destination
//                     expert's receive slab (atomic counter), the token row staged in shared memory
//                     once and sent with one bulk copy per chosen expert straight into the slab of the
//                     GPU that owns the expert (the permute IS the store address), plus a 16-byte
//                     {token, k, weight} record beside it.
//   MOE_COUNTS        after the last dispatch task: this rank's counts go to the expert owners (more than one rank, or a task per
//                     expert tile); and at the end of the launch, with i0 = 1, the counters are cleared for the next one.
//   MOE_RETURN        per (expert, source rank, 128-row block): rows below the received count are
//                     scaled by their routing weight and sent back into the source rank's combine
//                     buffer at [token, k]; the source then sums the k rows of every token.
//
// The reference has none of this: its expert-parallel example uses equal splits on one GPU and a
// dummy all_to_all node (examples/benchmark_all_to_all.py:31-127). Receive slabs have a fixed
// capacity per (source, expert); a token that does not fit is dropped for that expert (its combine
// row is zeroed at the source) and counted, never silently lost.
#pragma once
#include "elementwise.cuh"
#include "comm_tasks.cuh"

namespace maco {

struct MoeMeta { int32_t token; int32_t k; float weight; int32_t _pad; };

// Order of routing: larger logit first, lower expert on equal logits. A 16-bit logit and its index make one 32-bit key whose
// unsigned order is that order (0: no expert), so an arg-max over a warp is one redux instruction.
MACO_DEVICE uint32_t moe_key(uint32_t bits16, int expert, int dtype) {
  const uint32_t mag = bits16 & 0x7fffu, inf = dtype == MACO_DT_BF16 ? 0x7f80u : 0x7c00u;
  // NaN: behind everything else; -0 is 0
  const uint32_t ord = mag > inf ? 0u : ((bits16 & 0x8000u) && mag != 0u ? 0x7fffu - mag : 0x8000u + mag);
  return ((ord + 1u) << 15) - 1u - (uint32_t)expert;
}
MACO_DEVICE float moe_key_logit(uint32_t key, int dtype) {
  const uint32_t ord = key >> 15;
  const uint16_t bits = (uint16_t)(ord >= 0x8000u ? ord - 0x8000u : 0x8000u | (0x7fffu - ord));
  return dtype == MACO_DT_BF16 ? __uint_as_float((uint32_t)bits << 16) : __half2float(*reinterpret_cast<const __half*>(&bits));
}

// Top-k routing and dispatch of tokens [row0, row0 + rows), a warp per token. The rows come into shared memory by bulk copy, up
// to 32 at a time, while the warps route their tokens, and leave from there, one copy per choice, lane k for choice k. A token's slot
// atomics are in flight while the next token is routed.
// Routing a token used to take 40 shuffles and its row went through registers into one buffer per warp, free again only when the
// token's copies had read it: 76 us for 4096 tokens of 2048, top-8 of 64, most of it one warp's chain of 7 x 10 us.
// False after a wait that ran out, in the threads whose wait it was.
template <typename Program>
MACO_DEVICE bool moe_topk_dispatch(const Program& p, const MacoEltArgs& ar, int tid, const BulkCtx* bc) {
  // private copies: descriptor and parameter block live in global memory; read in place every use inside the
  // loops would be a fresh load, because the loops' stores could alias them
  const MacoEltArgs a = ar;
  const MacoMoeParams m = *reinterpret_cast<const MacoMoeParams*>(a.in2);
  const int warp = tid >> 5, lane = tid & 31;
  const int E = m.experts, K = m.top_k, dt = m.dtype;
  const uint32_t row_bytes = (uint32_t)m.hidden * 2;
  const int batch = min(32, (int)(bc->nbuf * bc->buf_bytes / row_bytes));
  uint8_t* const rows_s = bc->buf;
  constexpr int kChunks = 4;                           // 64 logits a chunk, two neighbours per lane: up to 256 experts
  auto fetch = [&](int t, uint32_t (&v)[kChunks]) {
#pragma unroll
    for (int i = 0; i < kChunks; ++i) {
      const int e = 64 * i + 2 * lane;
      if (e < E) v[i] = *reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint16_t*>(m.logits) + (size_t)t * m.ld_logits + e);
    }
  };
  bool ok = true;                                      // (after a wait that ran out a warp sends no more but meets the others at every barrier)
  for (int b0 = 0; b0 < a.rows; b0 += batch) {
    const int n = min(batch, a.rows - b0), tok0 = a.row0 + b0;
    if (b0 != 0) {
      if (lane < K) tma_store_wait_read<0>();          // the rows before these have left the buffer
      asm volatile("bar.sync 1, 128;" ::: "memory");   // (and the phase word is this batch's)
    }
    const uint32_t parity = *bc->phase & 1u;
    if (tid == 0 && ok) {
      fence_proxy_async_all();
      mbar_arrive_expect_tx(&bc->bars[0], (uint32_t)n * row_bytes);
      const uint8_t* src = reinterpret_cast<const uint8_t*>(m.x) + (size_t)tok0 * row_bytes;
      for (int j = 0; j < n; ++j) bulk_load(rows_s + (size_t)j * row_bytes, src + (size_t)j * row_bytes, row_bytes, &bc->bars[0]);
    }
    uint32_t cur[kChunks] = {0, 0, 0, 0}, nxt[kChunks] = {0, 0, 0, 0};
    if (warp < n) fetch(tok0 + warp, cur);
    if (warp + 4 < n) fetch(tok0 + warp + 4, nxt);
    int p_j = -1, p_e = 0;                             // the token routed last: its rows leave one turn later
    float p_w = 0.f;
    uint32_t p_slot = 0;
    auto send = [&] {
      if (lane >= K) return;
      const int t = tok0 + p_j;
      if (p_slot < (uint32_t)m.capacity) {
        const int dst = p_e / m.experts_per_rank, el = p_e - dst * m.experts_per_rank;
        const size_t cell = ((size_t)el * p.world + p.rank) * m.capacity + p_slot;
        bulk_store(p.peer_heap[dst] + m.recv_off + cell * row_bytes, rows_s + (size_t)p_j * row_bytes, row_bytes);
        MoeMeta mm{t, lane, p_w, 0};
        *reinterpret_cast<uint4*>(p.peer_heap[dst] + m.meta_off + cell * sizeof(MoeMeta)) = *reinterpret_cast<uint4*>(&mm);
      } else {
        // dropped for this expert: its combine row contributes nothing
        uint4* comb_row = reinterpret_cast<uint4*>(reinterpret_cast<uint8_t*>(m.comb) + ((size_t)t * K + lane) * row_bytes);
        for (uint32_t i = 0; i < row_bytes / 16; ++i) comb_row[i] = make_uint4(0, 0, 0, 0);
        atomicAdd(&m.counts[E + 1], 1u);               // dropped (token, expert) pairs of this launch
      }
      tma_store_commit();
    };
    for (int j = warp; j < n; j += 4) {
      uint32_t key[2 * kChunks];
#pragma unroll
      for (int i = 0; i < kChunks; ++i) {
        const int e = 64 * i + 2 * lane;
        key[2 * i] = e < E ? moe_key(cur[i] & 0xffffu, e, dt) : 0u;
        key[2 * i + 1] = e + 1 < E ? moe_key(cur[i] >> 16, e + 1, dt) : 0u;
        cur[i] = nxt[i];
      }
      if (j + 8 < n) fetch(tok0 + j + 8, nxt);
      uint32_t mine = 0, first = 0;
#pragma unroll 1
      for (int k = 0; k < K; ++k) {
        uint32_t best = key[0];
#pragma unroll
        for (int i = 1; i < 2 * kChunks; ++i) best = max(best, key[i]);
        best = __reduce_max_sync(0xffffffffu, best);
#pragma unroll
        for (int i = 0; i < 2 * kChunks; ++i) if (key[i] == best) key[i] = 0u;      // (keys differ: their low bits name the expert)
        if (k == 0) first = best;
        if (k == lane) mine = best;
      }
      const float ex = lane < K ? __expf(moe_key_logit(mine, dt) - moe_key_logit(first, dt)) : 0.f;
      const float w = ex / warp_sum(ex);
      const int e = 0x7fff - (int)(mine & 0x7fffu);
      uint32_t slot = 0;
      if (lane < K) slot = atomicAdd(&m.counts[e], 1u);
      if (p_j < 0) {
        const uint64_t t0 = globaltimer_ns();
        while (ok && !mbar_try_wait(&bc->bars[0], parity)) {
          if (globaltimer_ns() - t0 <= p.budget_ns) continue;
          ok = false;                                  // (warp 0 has sent for the rows and gives them as long again to land)
          if (warp == 0) while (!mbar_try_wait(&bc->bars[0], parity) && globaltimer_ns() - t0 <= 2 * p.budget_ns) {}
        }
      } else if (ok) {
        send();
      }
      p_j = j; p_e = e; p_w = w; p_slot = slot;
    }
    if (ok && p_j >= 0) send();
    __syncwarp();
    asm volatile("bar.sync 1, 128;" ::: "memory");     // every warp has seen this batch's phase
    if (tid == 0) *bc->phase = *bc->phase ^ 1u;
  }
  if (lane < K) tma_store_wait<0>();                   // all rows have landed before the task signals
  return ok;
}

// End of a launch, when every rank has returned its rows: counters for the next one. in0: what this one counted per expert, for the
// host; in1 (one rank, or null): the same as received counts.
MACO_DEVICE void moe_reset_counts(const MacoEltArgs& a, int tid) {
  const MacoMoeParams m = *reinterpret_cast<const MacoMoeParams*>(a.in2);
  uint32_t* ready = reinterpret_cast<uint32_t*>(a.out);
  uint32_t* routed = reinterpret_cast<uint32_t*>(const_cast<void*>(a.in0));
  uint32_t* received = reinterpret_cast<uint32_t*>(const_cast<void*>(a.in1));
  for (int e = tid; e < m.experts; e += 128) {
    const uint32_t n = __ldcg(m.counts + e);           // (other SMs' atomics)
    routed[e] = n;
    if (received != nullptr) received[e] = min(n, (uint32_t)m.capacity);
    m.counts[e] = 0;
  }
  for (int i = tid; i < a.cols; i += 128) ready[i] = 0;
  if (tid == 0) {
    m.counts[m.experts] = m.counts[m.experts + 1];     // what the host reads: pairs dropped by this launch
    m.counts[m.experts + 1] = 0;
  }
}

// counts[e] of this rank -> cnt[world][experts_per_rank] on the owner of e (slot = this rank).
template <typename Program>
MACO_DEVICE void moe_publish_counts(const Program& p, const MacoEltArgs& a, int tid) {
  if (a.i0 == 1) return moe_reset_counts(a, tid);
  const MacoMoeParams m = *reinterpret_cast<const MacoMoeParams*>(a.in2);
  for (int e = tid; e < m.experts; e += 128) {
    const int dst = e / m.experts_per_rank, el = e % m.experts_per_rank;
    uint32_t c = m.counts[e];
    if (c > (uint32_t)m.capacity) c = m.capacity;
    reinterpret_cast<uint32_t*>(p.peer_heap[dst] + m.cnt_off)[p.rank * m.experts_per_rank + el] = c;
  }
}

// rows [row0, row0+rows) of slab (el = i0, source rank = i1): y row * weight -> source's comb[token, k].
// One warp per row; the next row and its record are fetched into registers before the warp waits for
// the bulk engine to have read the current row out of shared memory.
template <typename Program>
MACO_DEVICE void moe_return(const Program& p, const MacoEltArgs& ar, int tid, uint8_t* stage) {
  const MacoEltArgs a = ar;
  const MacoMoeParams m = *reinterpret_cast<const MacoMoeParams*>(a.in2);
  const int warp = tid >> 5, lane = tid & 31;
  const int el = a.i0, src = a.i1, H = m.hidden, K = m.top_k;
  const int row_bytes = H * 2;
  const int nvec = row_bytes >> 4;
  constexpr int kVecPerLane = 10;                      // 16-byte vectors of a row per lane: hidden <= 2560
  const uint32_t count = reinterpret_cast<const uint32_t*>(p.peer_heap[p.rank] + m.cnt_off)[src * m.experts_per_rank + el];
  uint8_t* srow = stage + (size_t)warp * row_bytes;
  const size_t slab = ((size_t)el * p.world + src) * m.capacity;
  const MoeMeta* meta = reinterpret_cast<const MoeMeta*>(p.peer_heap[p.rank] + m.meta_off) + slab;
  const uint8_t* y = reinterpret_cast<const uint8_t*>(m.y) + slab * row_bytes;
  const int r_end = min(a.row0 + a.rows, (int)count);
  uint4 yr[kVecPerLane];
  MoeMeta mm{0, 0, 0.f, 0};
  auto fetch = [&](int r) {
    mm = meta[r];
    const uint4* q = reinterpret_cast<const uint4*>(y + (size_t)r * row_bytes);
#pragma unroll
    for (int i = 0; i < kVecPerLane; ++i) if (lane + 32 * i < nvec) yr[i] = q[lane + 32 * i];
  };
  int r = a.row0 + warp;
  if (r < r_end) fetch(r);
  bool pending = false;
  for (; r < r_end; r += 4) {
    if (pending && lane == 0) tma_store_wait_read<0>();
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kVecPerLane; ++i) {
      if (lane + 32 * i < nvec) {
        uint32_t w[4] = {yr[i].x, yr[i].y, yr[i].z, yr[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float2 f = m.dtype == MACO_DT_BF16 ? unpack_bf16x2(w[j]) : __half22float2(*reinterpret_cast<__half2*>(&w[j]));
          f.x *= mm.weight; f.y *= mm.weight;
          if (m.dtype == MACO_DT_BF16) w[j] = pack_bf16x2(f.x, f.y);
          else { __half2 h = __floats2half2_rn(f.x, f.y); w[j] = *reinterpret_cast<uint32_t*>(&h); }
        }
        reinterpret_cast<uint4*>(srow)[lane + 32 * i] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
    const MoeMeta cur = mm;
    if (r + 4 < r_end) fetch(r + 4);
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      bulk_store(p.peer_heap[src] + m.comb_off + ((size_t)cur.token * K + cur.k) * row_bytes, srow, row_bytes);
      tma_store_commit();
    }
    pending = true;
  }
  if (lane == 0) tma_store_wait<0>();
}

// Combine: out[t] = sum over k of comb[t][k] for tokens [row0, row0 + rows). A token's K rows are one
// contiguous block of the combine buffer, so with the operand ring idle (`bc` given) the leader
// streams whole token blocks into shared memory with the bulk-copy engine, half of the slots always
// in flight while the other half is summed; without the ring the rows are read with vector loads.
template <typename Program>
__device__ __noinline__ bool moe_combine(const Program& p, const MacoEltArgs& ar, int tid, BulkCtx* bc) {
  const MacoEltArgs a = ar;
  const MacoMoeParams m = *reinterpret_cast<const MacoMoeParams*>(a.in2);
  const int K = m.top_k, dt = m.dtype;
  const uint32_t row_bytes = (uint32_t)m.hidden * 2, tb = row_bytes * (uint32_t)K, nvec = row_bytes >> 4;
  const uint8_t* comb = p.peer_heap[p.rank] + m.comb_off;
  uint8_t* out = reinterpret_cast<uint8_t*>(a.out);
  const int t_end = a.row0 + a.rows;
  auto bar = [] { asm volatile("bar.sync 1, 128;" ::: "memory"); };
  uint32_t nslot = bc != nullptr ? min(bc->nbuf, (bc->nbuf * bc->buf_bytes) / tb) & ~1u : 0u;
  if (nslot < 2) {
    for (uint32_t i = tid; i < (uint32_t)a.rows * nvec; i += 128) {
      const uint32_t r = i / nvec, v = i - r * nvec;
      const uint8_t* src = comb + (size_t)(a.row0 + r) * tb + ((size_t)v << 4);
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      for (int k = 0; k < K; ++k) add8(acc, *reinterpret_cast<const uint4*>(src + (size_t)k * row_bytes), dt);
      *reinterpret_cast<uint4*>(out + (size_t)(a.row0 + r) * row_bytes + ((size_t)v << 4)) = pack8(acc, 1.f, dt);
    }
    return true;
  }
  const uint32_t half = nslot >> 1;
  bool ok = true;
  auto issue = [&](uint32_t h, int t0) {                 // leader only
    for (uint32_t s = 0; s < half; ++s) {
      const int t = t0 + (int)s;
      if (t >= t_end) break;
      const uint32_t b = h * half + s;
      mbar_arrive_expect_tx(&bc->bars[b], tb);
      bulk_load(bc->buf + (size_t)b * tb, comb + (size_t)t * tb, tb, &bc->bars[b]);
    }
  };
  auto consume = [&](uint32_t h, int t0) {
    const uint32_t phase = *bc->phase;
    uint32_t used = 0;
    for (uint32_t s = 0; s < half; ++s) {
      const int t = t0 + (int)s;
      if (t >= t_end) break;
      const uint32_t b = h * half + s;
      used |= 1u << b;
      const uint64_t w0 = globaltimer_ns();
      while (!mbar_try_wait(&bc->bars[b], (phase >> b) & 1u)) {
        if (globaltimer_ns() - w0 > p.budget_ns) { ok = false; break; }
      }
      const uint8_t* src = bc->buf + (size_t)b * tb;
      for (uint32_t v = tid; v < nvec; v += 128) {
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int k = 0; k < K; ++k) add8(acc, *reinterpret_cast<const uint4*>(src + (size_t)k * row_bytes + ((size_t)v << 4)), dt);
        *reinterpret_cast<uint4*>(out + (size_t)t * row_bytes + ((size_t)v << 4)) = pack8(acc, 1.f, dt);
      }
    }
    bar();                                               // the half's buffers are consumed by everybody
    if (tid == 0) *bc->phase = phase ^ used;             // read again only after the next barrier
  };
  if (tid == 0) {
    fence_proxy_async_all();
    issue(0, a.row0);
    issue(1, a.row0 + (int)half);
  }
  for (int t0 = a.row0; t0 < t_end; t0 += (int)nslot) {
    consume(0, t0);
    if (tid == 0) issue(0, t0 + (int)nslot);
    consume(1, t0 + (int)half);
    if (tid == 0) issue(1, t0 + (int)half + (int)nslot);
  }
  bar();                                                 // the last phase word is visible before the next task reads it
  return ok;
}

}  // namespace maco
