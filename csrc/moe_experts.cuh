// The expert GEMMs of a mixture-of-experts layer on one rank as one task per worker.
//
// How many 128-row tiles an expert has is known only when dispatch has ended. With a task per tile of every slab's capacity
// (MACO_TF_COUNTED, still the form of several ranks, of the dynamic scheduler and of separate return tasks) half of 7,168 tasks were empty at 2-5 us each on three
// roles, and a tile of the down projection, 12 k-blocks or 4.5 us of MMA, took 15-20 us of waits, count reads, fences and
// signals. Here every role of a worker walks over the tiles that exist: tile t of the line
//   [gate / up tiles of slab 0, slab 1, ...][down tiles of slab 0, slab 1, ...]
// belongs to worker t mod shares, which each role derives from the received counts by itself. Consecutive tiles of a slab are the
// row blocks of one 256-column weight tile, so a weight tile is read by its workers at the same time. A down tile waits
// for the gate / up tiles of its row block (a counter per block, bumped by each of the four epilogue warps); these lie in front of
// every down tile in each worker's share, so the workers cannot wait for one another in a circle. Rows leave, scaled by their routing
// weight, for the combine buffer; one signal per worker says that all of its rows have.
#pragma once
#include "gemm_tcgen05.cuh"
#include "moe_tasks.cuh"

namespace maco {

constexpr int kMaxSlabs = 256;                // experts of the layer, a slab each

// Row blocks per slab, in shared memory: counts read from global memory again for every tile were an L2 round trip per slab passed
// (each acquire of the SM empties its L1), 2-5 us between two tiles. `first`, `step`: the threads that fill the table.
MACO_DEVICE void expert_blocks(uint16_t* table, const MacoExpertArgs& a, int first, int step) {
#pragma unroll 4
  for (int i = first; i < a.experts; i += step)
    table[i] = (uint16_t)((min((int)__ldcg(a.counts + i), a.capacity) + kBM - 1) / kBM);      // (final: dispatch has ended)
}

struct ExpertTiles {
  const uint16_t* blocks;
  int slabs, tiles[2];                        // column tiles of the two projections
  int t, step, base;                          // this share's next tile; first tile of the slab
  int phase, slab, mb, nb;                    // the current tile: projection, slab, row block, column tile

  MACO_DEVICE ExpertTiles(const MacoExpertArgs& a, const uint16_t* table, int share)
      : blocks(table), slabs(a.experts), tiles{a.inter / 128, a.hidden / 256}, t(share), step(a.shares), base(0), phase(0), slab(0),
        mb(0), nb(0) {}

  MACO_DEVICE bool next() {
    while (true) {
      if (slab == slabs) {
        if (phase == 1) return false;
        phase = 1; slab = 0;
      }
      const int b = blocks[slab], n = b * (phase == 0 ? tiles[0] : tiles[1]), r = t - base;
      if (r < n) {
        nb = r / b;
        mb = r - nb * b;
        t += step;
        return true;
      }
      base += n;
      ++slab;
    }
  }
};

// ---- TMA warp (converged) ----------------------------------------------------------------------
template <int STAGES, typename Program, typename WaitFn>
__device__ __noinline__ bool experts_produce(const Program& p, const MacoExpertArgs& args, int share, uint16_t* table, uint8_t* smem, const GemmCtrl& c,
                                             const CUtensorMap* tmaps, uint32_t& it, WaitFn wait) {
  const MacoExpertArgs a = args;
  expert_blocks(table, a, threadIdx.x & 31, 32);
  __syncwarp();
  ExpertTiles tiles(a, table, share);
  const uint32_t gate_done = 4u * (uint32_t)tiles.tiles[0];
  while (tiles.next()) {
    const int m0 = tiles.slab * a.capacity + tiles.mb * kBM, el = tiles.slab;
    bool ok;
    if (tiles.phase == 0) {
      ok = gemm_produce_tile<256, STAGES, false, false>(smem, c, tmaps + a.tmap_x, tmaps + a.tmap_w1, m0, (el * tiles.tiles[0] + tiles.nb) * 256, 0,
                                                        a.hidden / kBK, it, p.budget_ns);
    } else {
      // A row block that is complete (all but the first ones of a share) goes on without a pause: the look at its counter is over before
      // the stages of the tile in front are free. Else the first weights are on their way while it is waited for.
      uint32_t ahead = 0;
      const int n0 = el * a.hidden + tiles.nb * 256;
      const uint32_t* ready = a.ready + tiles.slab * (a.capacity / kBM) + tiles.mb;
      // (one lane looks, for all)
      if (warp_uniform((threadIdx.x & 31) == 0 ? ld_acquire_gpu_u32(ready) : 0u) < gate_done) {
        ok = gemm_produce_b_ahead<256, STAGES>(smem, c, tmaps + a.tmap_w2, n0, 0, a.inter / kBK, it, p.budget_ns, -1, ahead);
        if (!ok || !wait(ready, gate_done)) { it += ahead; return false; }
      }
      __syncwarp();
      fence_proxy_async_all();
      ok = gemm_produce_tile<256, STAGES, false, false>(smem, c, tmaps + a.tmap_act, tmaps + a.tmap_w2, m0, n0, 0, a.inter / kBK, it, p.budget_ns,
                                                        nullptr, kBK, -1, ahead);
    }
    if (!ok) return false;
  }
  return true;
}

// ---- MMA warp (converged) ----------------------------------------------------------------------
template <int STAGES, typename Program>
__device__ __noinline__ bool experts_mma(const Program& p, const MacoExpertArgs& args, int share, uint16_t* table, uint8_t* smem, const GemmCtrl& c,
                                         uint32_t tmem_base, uint32_t& it, uint32_t& seq) {
  const MacoExpertArgs a = args;
  expert_blocks(table, a, threadIdx.x & 31, 32);
  __syncwarp();
  ExpertTiles tiles(a, table, share);
  while (tiles.next()) {
    if (!gemm_mma_tile<256, STAGES, false, false>(smem, c, tmem_base, a.idesc, (tiles.phase == 0 ? a.hidden : a.inter) / kBK, it, seq, p.budget_ns))
      return false;
    ++seq;
  }
  return true;
}

// ---- epilogue warps: the four run on their own --------------------------------------------------
// Returns the number of tiles, or -1 after a wait that ran out.
template <typename Program, typename BarFn>
__device__ __noinline__ int experts_epilogue(const Program& p, const MacoExpertArgs& args, int share, uint16_t* table, int tid, const GemmCtrl& c,
                                             uint32_t tmem_base, uint32_t seq0, uint8_t* block, BarFn bar) {
  const MacoExpertArgs a = args;
  expert_blocks(table, a, tid, 128);
  bar();
  ExpertTiles tiles(a, table, share);
  const uint32_t q = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
  const uint32_t mine = smem_u32(block) + q * kEpiWarpBytes;
  const int dt = a.dtype;
  uint32_t seq = seq0;
  while (tiles.next()) {
    const uint32_t acc = seq & 1;
    const bool down = tiles.phase != 0;
    const int row = tiles.mb * kBM + (int)(q * 32 + lane);
    const long long cell = (long long)tiles.slab * a.capacity + row;
    // both loads are back before the accumulator is complete
    const int rows = min((int)__ldcg(a.counts + tiles.slab), a.capacity);
    int4 rec = make_int4(0, 0, 0, 0);
    if (down) rec = reinterpret_cast<const int4*>(a.meta)[cell];        // (rows beyond the count hold old records, and are not written)
    const int valid = rows - (tiles.mb * kBM + (int)(q * 32));          // rows of this warp's 32 that hold a token (may be <= 0 or more)
    uint8_t* dst = down ? reinterpret_cast<uint8_t*>(a.comb) + tiles.nb * 512
                        : reinterpret_cast<uint8_t*>(a.act) + ((cell - lane) * a.inter + tiles.nb * 128) * 2;
    const int out_row = down ? rec.x * a.top_k + rec.y : (int)lane, pitch = (down ? a.hidden : a.inter) * 2;
    const float weight = __int_as_float(rec.z);
    // Rows leave in whole lines through shared memory where there are many of them (4096 tokens, 64 experts: 547 -> 515 us); a slab of less than
    // one row block has few, and the way through the block is only longer (256 tokens, 32 experts: 102.5 instead of 100.8).
    const bool lines = rows >= kBM;
    uint32_t ok = 1;
    if (lane == 0) ok = mbar_wait(&c.tmem_full[acc], (seq >> 1) & 1, p.budget_ns, c.abort_word) ? 1u : 0u;
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (!ok) return -1;
    tc_fence_after();
    const uint32_t t_row = tmem_base + ((q * 32u) << 16) + acc * 256;
    const int cols = down ? 256 : 128;
#pragma unroll 1
    for (int col = valid > 0 ? 0 : cols; col < cols; dst += 128) {      // (a warp without tokens has nothing to compute)
#pragma unroll 1
      for (uint32_t piece = 0; piece < 8; piece += 2, col += 16) {
        uint32_t r[16], w[8];
        tmem_ld_32x16(t_row + col, r);
        if (!down) {
          uint32_t u[16];
          tmem_ld_32x16(t_row + 128 + col, u);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(silu_16(__uint_as_float(r[j])) * __uint_as_float(u[j]));
        } else {
          tmem_ld_wait();
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = epi_pack(dt, __uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
        if (down) {
          // the expert's output row is rounded to the output type first (what a separate return pass would read)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float2 f = epi_unpack(dt, w[j]);
            w[j] = epi_pack(dt, f.x * weight, f.y * weight);
          }
        }
        if (lines) {
          epi_sts(epi_piece<8>(mine, lane, piece), make_uint4(w[0], w[1], w[2], w[3]));
          epi_sts(epi_piece<8>(mine, lane, piece + 1), make_uint4(w[4], w[5], w[6], w[7]));
        } else if ((int)lane < valid) {
          uint4* to = reinterpret_cast<uint4*>(dst + (long long)out_row * pitch) + piece;
          to[0] = make_uint4(w[0], w[1], w[2], w[3]);
          to[1] = make_uint4(w[4], w[5], w[6], w[7]);
        }
        __syncwarp();                                                   // (the lanes that stored and the others: tcgen05.ld takes a converged warp)
      }
      if (lines)
        epi_flush_rows<8>(mine, lane, [&](uint32_t r) -> uint8_t* {
          const int o = __shfl_sync(0xffffffffu, out_row, r);
          return (int)r < valid ? dst + (long long)o * pitch : nullptr;
        });
    }
    tc_fence_before();
    mbar_arrive(&c.tmem_empty[acc]);
    if (!down) {
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
