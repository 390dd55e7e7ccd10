// The expert GEMMs of a mixture-of-experts layer as one task per worker.
//
// How many 128-row tiles an expert has is known only when dispatch has ended. With a task per tile of every slab's capacity
// (MACO_TF_COUNTED, still the form of the dynamic scheduler and of separate return tasks) half of 7,168 tasks were empty at 2-5 us each on three
// roles, and a tile of the down projection, 12 k-blocks or 4.5 us of MMA, took 15-20 us of waits, count reads, fences and
// signals. Here every role of a worker walks over the tiles that exist: tile t of the line
//   [gate / up tiles of slab 0, slab 1, ...][down tiles of slab 0, slab 1, ...]
// belongs to worker t mod shares, which each role derives from the received counts by itself. Consecutive tiles of a slab are the
// row blocks of one 256-column weight tile, so a weight tile is read by its workers at the same time. A down tile waits
// for the gate / up tiles of its row block (a counter per block, bumped by each of the four epilogue warps); these lie in front of
// every down tile in each worker's share, so the workers cannot wait for one another in a circle. Rows leave, scaled by their routing
// weight, for their source rank's combine buffer; one signal per worker says that all of its rows have.
#pragma once
#include "gemm_tcgen05.cuh"
#include "moe_tasks.cuh"

namespace maco {

struct ExpertTiles {
  const uint32_t* counts;
  int experts, world, capacity, tiles[2];     // local experts; column tiles of the two projections
  int t, step;                                // this share's next tile
  int base, el, src;                          // first tile of the slab (expert el, source rank src)
  int phase, slab, mb, nb, rows;              // the current tile: projection, slab, row block, column tile, rows of the slab

  MACO_DEVICE ExpertTiles(const MacoExpertArgs& a, int share)
      : counts(a.counts), experts(a.experts), world(a.world), capacity(a.capacity), tiles{a.inter / 128, a.hidden / 256}, t(share),
        step(a.shares), base(0), el(0), src(0), phase(0), slab(0), mb(0), nb(0), rows(0) {}

  MACO_DEVICE bool next() {
    while (true) {
      if (el == experts) {
        if (phase == 1) return false;
        phase = 1; el = 0; src = 0;
      }
      rows = min((int)counts[src * experts + el], capacity);     // (final: dispatch has ended everywhere)
      const int blocks = (rows + kBM - 1) / kBM, n = blocks * tiles[phase];
      if (t < base + n) {
        const int r = t - base;
        nb = r / blocks;
        mb = r - nb * blocks;
        slab = el * world + src;
        t += step;
        return true;
      }
      base += n;
      if (++src == world) { src = 0; ++el; }
    }
  }
};

// ---- TMA thread -------------------------------------------------------------------------------
template <int STAGES, typename Program, typename WaitFn>
__device__ __noinline__ bool experts_produce(const Program& p, const MacoExpertArgs& args, int share, uint8_t* smem, const GemmCtrl& c,
                                             const CUtensorMap* tmaps, uint32_t& it, WaitFn wait) {
  const MacoExpertArgs a = args;
  ExpertTiles tiles(a, share);
  const uint32_t gate_done = 4u * (uint32_t)tiles.tiles[0];
  while (tiles.next()) {
    const int m0 = tiles.slab * a.capacity + tiles.mb * kBM;
    bool ok;
    if (tiles.phase == 0) {
      ok = gemm_produce_tile<256, STAGES, false, false>(smem, c, tmaps + a.tmap_x, tmaps + a.tmap_w1, m0, (tiles.el * tiles.tiles[0] + tiles.nb) * 256, 0,
                                                        a.hidden / kBK, it, p.budget_ns);
    } else {
      // the first weights are on their way before the row block of activations is complete
      uint32_t ahead = 0;
      const int n0 = tiles.el * a.hidden + tiles.nb * 256;
      ok = gemm_produce_b_ahead<256, STAGES>(smem, c, tmaps + a.tmap_w2, n0, 0, a.inter / kBK, it, p.budget_ns, -1, ahead);
      if (!ok || !wait(a.ready + tiles.slab * (a.capacity / kBM) + tiles.mb, gate_done)) { it += ahead; return false; }
      fence_proxy_async_all();
      ok = gemm_produce_tile<256, STAGES, false, false>(smem, c, tmaps + a.tmap_act, tmaps + a.tmap_w2, m0, n0, 0, a.inter / kBK, it, p.budget_ns,
                                                        nullptr, kBK, -1, ahead);
    }
    if (!ok) return false;
  }
  return true;
}

// ---- MMA thread -------------------------------------------------------------------------------
template <int STAGES, typename Program>
__device__ __noinline__ bool experts_mma(const Program& p, const MacoExpertArgs& args, int share, uint8_t* smem, const GemmCtrl& c,
                                         uint32_t tmem_base, uint32_t& it, uint32_t& seq) {
  const MacoExpertArgs a = args;
  ExpertTiles tiles(a, share);
  while (tiles.next()) {
    if (!gemm_mma_tile<256, STAGES, false, false>(smem, c, tmem_base, a.idesc, (tiles.phase == 0 ? a.hidden : a.inter) / kBK, it, seq, p.budget_ns))
      return false;
    ++seq;
  }
  return true;
}

// ---- epilogue warps: the four run on their own --------------------------------------------------
// Returns the number of tiles, or -1 after a wait that ran out.
template <typename Program>
__device__ __noinline__ int experts_epilogue(const Program& p, const MacoExpertArgs& args, int share, const GemmCtrl& c, uint32_t tmem_base,
                                             uint32_t seq0) {
  const MacoExpertArgs a = args;
  ExpertTiles tiles(a, share);
  const uint32_t q = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
  const int dt = a.dtype;
  uint32_t seq = seq0;
  while (tiles.next()) {
    const uint32_t acc = seq & 1;
    const int row = tiles.mb * kBM + (int)(q * 32 + lane);
    const bool row_ok = row < tiles.rows;
    const long long cell = (long long)tiles.slab * a.capacity + row;
    uint8_t* dst;
    float weight = 1.f;
    if (tiles.phase == 0) {
      dst = reinterpret_cast<uint8_t*>(a.act) + (cell * a.inter + tiles.nb * 128) * 2;
    } else {
      int4 rec = make_int4(0, 0, 0, 0);
      if (row_ok) rec = reinterpret_cast<const int4*>(a.meta)[cell];
      weight = __int_as_float(rec.z);
      dst = p.peer_heap[tiles.src] + a.comb_off + (((long long)rec.x * a.top_k + rec.y) * a.hidden + tiles.nb * 256) * 2;
    }
    uint32_t ok = 1;
    if (lane == 0) ok = mbar_wait(&c.tmem_full[acc], (seq >> 1) & 1, p.budget_ns, c.abort_word) ? 1u : 0u;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (!ok) return -1;
    tc_fence_after();
    const uint32_t t_row = tmem_base + ((q * 32u) << 16) + acc * 256;
    if (tiles.phase == 0) {
#pragma unroll 1
      for (int col = 0; col < 128; col += 32) {
        uint32_t r[32], u[32], w[16];
        tmem_ld_32x32(t_row + col, r);
        tmem_ld_32x32(t_row + 128 + col, u);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j)
          w[j] = epi_pack(dt, silu(__uint_as_float(r[2 * j])) * __uint_as_float(u[2 * j]), silu(__uint_as_float(r[2 * j + 1])) * __uint_as_float(u[2 * j + 1]));
        if (row_ok) {
#pragma unroll
          for (int j = 0; j < 16; j += 4) reinterpret_cast<uint4*>(dst + col * 2)[j >> 2] = make_uint4(w[j], w[j + 1], w[j + 2], w[j + 3]);
        }
        __syncwarp();
      }
    } else {
#pragma unroll 1
      for (int col = 0; col < 256; col += 32) {
        uint32_t r[32], w[16];
        tmem_ld_32x32(t_row + col, r);
        tmem_ld_wait();
        // the expert's output row is rounded to the output type first (what a separate return pass would read)
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const uint32_t y = epi_pack(dt, __uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
          const float2 f = dt == MACO_DT_F16 ? __half22float2(*reinterpret_cast<const __half2*>(&y)) : unpack_bf16x2(y);
          w[j] = epi_pack(dt, f.x * weight, f.y * weight);
        }
        if (row_ok) {
#pragma unroll
          for (int j = 0; j < 16; j += 4) reinterpret_cast<uint4*>(dst + col * 2)[j >> 2] = make_uint4(w[j], w[j + 1], w[j + 2], w[j + 3]);
        }
        __syncwarp();
      }
    }
    tc_fence_before();
    mbar_arrive(&c.tmem_empty[acc]);
    if (tiles.phase == 0) {
      __syncwarp();
      if (lane == 0) {
        fence_acq_rel_gpu();
        red_add_relaxed_gpu_u32(a.ready + tiles.slab * (a.capacity / kBM) + tiles.mb, 1);
      }
    }
    ++seq;
  }
  return (int)(seq - seq0);
}

}  // namespace maco
