// Row-wise and point-wise tasks of the persistent kernel, staged through shared memory.
//
// What bounds a small task there is neither bandwidth nor arithmetic but the memory round trips and the code it
// walks through: a worker leaves 28 KB of L1 next to its 220 KB of shared memory, so register spills and re-reads
// of an unrolled body turn into L2 round trips (the unrolled RMSNorm of one 5120-wide row took 18,000-23,000 cycles:
// 850 bytes of spills per thread, and 9 KB of straight-line code fetched cold on every SM). These forms keep the row
// in shared memory instead of registers: every thread copies exactly the vectors it will use with cp.async (all of
// them in flight at once, no barrier needed to read them back) and then walks over them in short loops.
#pragma once
#include "elementwise.cuh"

namespace maco {

MACO_DEVICE uint4 lds_v4(uint32_t saddr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(saddr));
  return v;
}

// A 16-byte vector as 8 (16-bit types) or 4 (fp32) floats.
template <int DT> struct VecOf { static constexpr int kN = DT == MACO_DT_F32 ? 4 : 8; float v[kN]; };
template <int DT> MACO_DEVICE VecOf<DT> vec_unpack(uint4 u) {
  VecOf<DT> r;
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (DT == MACO_DT_F32) {
      r.v[i] = __uint_as_float(w[i]);
    } else {
      const float2 f = DT == MACO_DT_BF16 ? unpack_bf16x2(w[i]) : __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      r.v[2 * i] = f.x; r.v[2 * i + 1] = f.y;
    }
  }
  return r;
}
template <int DT> MACO_DEVICE uint4 vec_pack(const VecOf<DT>& r) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (DT == MACO_DT_F32) {
      w[i] = __float_as_uint(r.v[i]);
    } else if constexpr (DT == MACO_DT_BF16) {
      w[i] = pack_bf16x2(r.v[2 * i], r.v[2 * i + 1]);
    } else {
      const __half2 h = __floats2half2_rn(r.v[2 * i], r.v[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

constexpr uint32_t kRowScratch = 28672;                // shared memory the staged tasks may use
constexpr uint32_t kRowRed = 256;                      // of which: cross-warp reductions (2 x 2 x 4 floats used)

// Row-wise task (RMSNORM, LAYERNORM, SOFTMAX) on 128 threads. A team (one warp, or all four for tasks of fewer than
// four rows and for rows that four warps cannot hold side by side) owns a row at a time. Returns false when one
// row does not fit the scratch block or is not made of 16-byte vectors (elt_run handles those).
template <int DT>
__device__ __noinline__ bool row_task_staged(uint32_t type, const MacoEltArgs& ar, int tid, uint8_t* scratch) {
  constexpr int kN = VecOf<DT>::kN;
  const MacoEltArgs a = ar;
  if (!elt_vec_ok(a)) return false;
  const uint32_t nvec = (uint32_t)a.cols / kN, rb = nvec * 16;
  const uint32_t n_par = type == MACO_TASK_SOFTMAX ? 0u : (type == MACO_TASK_LAYERNORM ? 2u : 1u);
  const uint32_t room = kRowScratch - kRowRed;
  // parameter rows are staged when a row buffer still fits beside them, else read from global memory
  const bool par_s = n_par * rb + rb <= room;
  const uint32_t left = room - (par_s ? n_par * rb : 0u);
  if (rb > left) return false;
  const bool team_warp = a.rows >= 4 && 4 * rb <= left;
  const uint32_t teams = team_warp ? 4u : 1u;
  const bool two = teams * 2 * rb <= left && (uint32_t)a.rows > teams;
  const uint32_t lane = tid & 31, warp = tid >> 5;
  const uint32_t start = team_warp ? lane : (uint32_t)tid, step = team_warp ? 32u : 128u;
  const uint32_t s_red = smem_u32(scratch), s_par = s_red + kRowRed;
  const uint32_t s_buf = s_par + (par_s ? n_par * rb : 0u) + (team_warp ? warp * (two ? 2u : 1u) * rb : 0u);
  float* red = reinterpret_cast<float*>(scratch);
  const uint8_t* in = reinterpret_cast<const uint8_t*>(a.in0);
  const size_t in_pitch = (size_t)a.ld_in * (16 / kN), out_pitch = (size_t)a.ld_out * (16 / kN);
  auto fetch = [&](int r, uint32_t buf) {
    const uint8_t* src = in + (size_t)(a.row0 + r) * in_pitch;
#pragma unroll 1
    for (uint32_t v = start; v < nvec; v += step) cp_async16(s_buf + buf * rb + v * 16, src + (size_t)v * 16);
  };
  int r = team_warp ? (int)warp : 0;
  const int r_step = team_warp ? 4 : 1;
  if (par_s) {
#pragma unroll 1
    for (uint32_t v = tid; v < nvec; v += 128) {
      if (n_par > 0) cp_async16(s_par + v * 16, reinterpret_cast<const uint8_t*>(a.in1) + (size_t)v * 16);
      if (n_par > 1) cp_async16(s_par + rb + v * 16, reinterpret_cast<const uint8_t*>(a.in2) + (size_t)v * 16);
    }
  }
  if (r < a.rows) fetch(r, 0);
  cp_async_commit();
  if (team_warp && par_s && n_par > 0) {
    cp_async_wait<0>();                                // every warp reads parameter vectors that other warps copied
    asm volatile("bar.sync 1, 128;" ::: "memory");
  }
  if (two && r + r_step < a.rows) fetch(r + r_step, 1);
  cp_async_commit();
  uint32_t it = 0;
#pragma unroll 1
  for (; r < a.rows; r += r_step, ++it) {
    if (two) cp_async_wait<1>(); else cp_async_wait<0>();
    const uint32_t buf = two ? (it & 1u) : 0u, sb = s_buf + buf * rb;
    auto reduce = [&](float v, bool is_max, int which) {
      v = is_max ? warp_max(v) : warp_sum(v);
      if (team_warp) return v;
      float* slot = red + ((it & 1u) * 2 + which) * 4;
      if (lane == 0) slot[warp] = v;
      asm volatile("bar.sync 1, 128;" ::: "memory");
      return is_max ? fmaxf(fmaxf(slot[0], slot[1]), fmaxf(slot[2], slot[3])) : slot[0] + slot[1] + slot[2] + slot[3];
    };
    float acc = type == MACO_TASK_SOFTMAX ? -INFINITY : 0.f;
#pragma unroll 1
    for (uint32_t v = start; v < nvec; v += step) {
      const VecOf<DT> x = vec_unpack<DT>(lds_v4(sb + v * 16));
      if (type == MACO_TASK_SOFTMAX) {
#pragma unroll
        for (int j = 0; j < kN; ++j) acc = fmaxf(acc, x.v[j]);
      } else if (type == MACO_TASK_LAYERNORM) {
#pragma unroll
        for (int j = 0; j < kN; ++j) acc += x.v[j];
      } else {
#pragma unroll
        for (int j = 0; j < kN; ++j) acc += x.v[j] * x.v[j];
      }
    }
    acc = reduce(acc, type == MACO_TASK_SOFTMAX, 0);
    float sub = 0.f, mul;                              // out = (x - sub) * mul [* w + b], or exp(x - sub) * mul
    if (type == MACO_TASK_RMSNORM) {
      mul = rsqrtf(acc / a.cols + a.f0);
    } else {
      const bool soft = type == MACO_TASK_SOFTMAX;
      sub = soft ? acc : acc / a.cols;
      float s2 = 0.f;
#pragma unroll 1
      for (uint32_t v = start; v < nvec; v += step) {
        const VecOf<DT> x = vec_unpack<DT>(lds_v4(sb + v * 16));
#pragma unroll
        for (int j = 0; j < kN; ++j) { const float d = x.v[j] - sub; s2 += soft ? __expf(d) : d * d; }
      }
      s2 = reduce(s2, false, 1);
      mul = soft ? 1.f / s2 : rsqrtf(s2 / a.cols + a.f0);
    }
    uint8_t* dst = reinterpret_cast<uint8_t*>(a.out) + (size_t)(a.row0 + r) * out_pitch;
#pragma unroll 1
    for (uint32_t v = start; v < nvec; v += step) {
      VecOf<DT> x = vec_unpack<DT>(lds_v4(sb + v * 16));
      if (type == MACO_TASK_SOFTMAX) {
#pragma unroll
        for (int j = 0; j < kN; ++j) x.v[j] = __expf(x.v[j] - sub) * mul;
      } else {
        const VecOf<DT> w = vec_unpack<DT>(par_s ? lds_v4(s_par + v * 16) : reinterpret_cast<const uint4*>(a.in1)[v]);
#pragma unroll
        for (int j = 0; j < kN; ++j) x.v[j] = (x.v[j] - sub) * mul * w.v[j];
        if (type == MACO_TASK_LAYERNORM) {
          const VecOf<DT> b = vec_unpack<DT>(par_s ? lds_v4(s_par + rb + v * 16) : reinterpret_cast<const uint4*>(a.in2)[v]);
#pragma unroll
          for (int j = 0; j < kN; ++j) x.v[j] += b.v[j];
        }
      }
      *reinterpret_cast<uint4*>(dst + (size_t)v * 16) = vec_pack<DT>(x);
    }
    const int rn = r + (two ? 2 : 1) * r_step;         // this buffer's next row (a thread overwrites only vectors it has read)
    if (rn < a.rows) fetch(rn, buf);
    cp_async_commit();
  }
  cp_async_wait<0>();
  return true;
}

// Point-wise task on 128 threads: two stages of vectors per thread in flight (7 of one operand or 3 of two), consumed
// in a loop of one vector per turn. Same return value as row_task_staged.
template <int DT>
__device__ __noinline__ bool point_task_staged(uint32_t type, const MacoEltArgs& ar, int tid, uint8_t* scratch) {
  constexpr int kN = VecOf<DT>::kN;
  const MacoEltArgs a = ar;
  if (!elt_vec_ok(a)) return false;
  const bool bin = elt_is_binary(type);
  const uint32_t vpr = (uint32_t)a.cols / kN, total = (uint32_t)a.rows * vpr;
  const uint32_t per = bin ? 3u : 7u;                  // vectors per thread and stage
  const uint32_t s_mine = smem_u32(scratch) + (uint32_t)tid * 16;          // slot k of this thread: + k * 2048
  const size_t es = 16 / kN;
  const bool packed = a.ld_in == a.cols && a.ld_out == a.cols;
  const uint8_t* in0 = reinterpret_cast<const uint8_t*>(a.in0) + (size_t)a.row0 * a.ld_in * es;
  const uint8_t* in1 = reinterpret_cast<const uint8_t*>(a.in1) + (size_t)a.row0 * a.ld_in * es;
  uint8_t* out = reinterpret_cast<uint8_t*>(a.out) + (size_t)a.row0 * a.ld_out * es;
  auto off = [&](uint32_t i, int ld) {                 // byte offset of vector i
    if (packed) return (size_t)i * 16;
    const uint32_t r = i / vpr;
    return (size_t)r * ld * es + (size_t)(i - r * vpr) * 16;
  };
  auto issue = [&](uint32_t base, uint32_t stage) {
#pragma unroll 1
    for (uint32_t k = 0; k < per; ++k) {
      const uint32_t i = base + k * 128 + (uint32_t)tid;
      if (i < total) {
        const size_t o = off(i, a.ld_in);
        const uint32_t s = s_mine + (stage * 7 + k) * 2048;
        cp_async16(s, in0 + o);
        if (bin) cp_async16(s + 3 * 2048, in1 + o);
      }
    }
    cp_async_commit();
  };
  const uint32_t span = per * 128;
  issue(0, 0);
  issue(span, 1);
  uint32_t stage = 0;
#pragma unroll 1
  for (uint32_t base = 0; base < total; base += span, stage ^= 1u) {
    cp_async_wait<1>();
#pragma unroll 1
    for (uint32_t k = 0; k < per; ++k) {
      const uint32_t i = base + k * 128 + (uint32_t)tid;
      if (i >= total) break;
      const uint32_t s = s_mine + (stage * 7 + k) * 2048;
      VecOf<DT> x = vec_unpack<DT>(lds_v4(s)), y;
      if (bin) y = vec_unpack<DT>(lds_v4(s + 3 * 2048));
      switch (type) {
#define MACO_POINT_CASE(T, EXPR)                                   \
  case T:                                                          \
    _Pragma("unroll") for (int j = 0; j < kN; ++j) x.v[j] = EXPR;  \
    break;
        MACO_POINT_CASE(MACO_TASK_GELU, (elt_op<DT, MACO_TASK_GELU>(x.v[j], 0.f, 0.f, 0.f)))
        MACO_POINT_CASE(MACO_TASK_SILU, silu(x.v[j]))
        MACO_POINT_CASE(MACO_TASK_SCALE, x.v[j] * a.f0)
        MACO_POINT_CASE(MACO_TASK_ADD, x.v[j] + y.v[j])
        MACO_POINT_CASE(MACO_TASK_SILU_GATE, silu(x.v[j]) * y.v[j])
        MACO_POINT_CASE(MACO_TASK_GELU_BWD, (elt_op<DT, MACO_TASK_GELU_BWD>(x.v[j], y.v[j], 0.f, 0.f)))
        MACO_POINT_CASE(MACO_TASK_AXPBY, a.f0 * x.v[j] + a.f1 * y.v[j])
        default: break;                                // COPY
#undef MACO_POINT_CASE
      }
      *reinterpret_cast<uint4*>(out + off(i, a.ld_out)) = vec_pack<DT>(x);
    }
    issue(base + 2 * span, stage);
  }
  cp_async_wait<0>();
  return true;
}

// Staged form of a row-wise or point-wise task where it applies; everything else goes through elt_run.
MACO_DEVICE bool elt_run_staged(uint32_t type, const MacoEltArgs& a, int tid, uint8_t* scratch) {
  switch (type) {
    case MACO_TASK_RMSNORM: case MACO_TASK_LAYERNORM: case MACO_TASK_SOFTMAX:
      if (a.dtype == MACO_DT_BF16) return row_task_staged<MACO_DT_BF16>(type, a, tid, scratch);
      if (a.dtype == MACO_DT_F16) return row_task_staged<MACO_DT_F16>(type, a, tid, scratch);
      return row_task_staged<MACO_DT_F32>(type, a, tid, scratch);
    case MACO_TASK_GELU: case MACO_TASK_SILU: case MACO_TASK_SCALE: case MACO_TASK_ADD:
    case MACO_TASK_SILU_GATE: case MACO_TASK_GELU_BWD: case MACO_TASK_COPY: case MACO_TASK_AXPBY:
      if (a.dtype == MACO_DT_BF16) return point_task_staged<MACO_DT_BF16>(type, a, tid, scratch);
      if (a.dtype == MACO_DT_F16) return point_task_staged<MACO_DT_F16>(type, a, tid, scratch);
      return point_task_staged<MACO_DT_F32>(type, a, tid, scratch);
    default: return false;
  }
}

}  // namespace maco
