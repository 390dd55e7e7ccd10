// Stand-alone decode attention. Default: one CTA per SM streams an equal share of all (batch, kv-head, 128-key chunk)
// triples (attn_stream_kernel), a second launch merges the ranges cut by a share's end. With a caller-chosen split count
// or scratch: one CTA per (batch, kv-head, split) on the CUDA cores and a merge launch.
//
// Layouts (row-major, 16-bit):
//   q   [B, Hq, 128]          Hq = Hkv * G query heads, the G heads of one KV head are adjacent
//   k,v [B, Hkv, S, 128]      S = keys per sequence (cache length)
//   out [B, Hq, 128]
//   scratch fp32 [B * Hkv * splits, G*128 + 2G]   unnormalised partial outputs, running max and sum
#include "attention_decode.cuh"
#include "host_common.h"

using namespace maco;

namespace {

struct AttnParams {
  const void* q; const void* k; const void* v; void* out; float* scratch;
  int B, Hkv, G, S, splits, dtype;
  long long kv_batch_stride, kv_head_stride;   // in elements
  float scale;
};

__global__ void __launch_bounds__(128) attn_decode_kernel(AttnParams p) {
  __shared__ __align__(16) uint8_t scratch_smem[kAttnScratchBytes];
  const int split = blockIdx.x % p.splits;
  const int bh = blockIdx.x / p.splits;            // b * Hkv + kvh
  const int b = bh / p.Hkv, kvh = bh % p.Hkv;
  const int per = (p.S + p.splits - 1) / p.splits;
  const int s0 = split * per;
  int rows = p.S - s0;
  if (rows > per) rows = per;
  if (rows < 0) rows = 0;
  const int rec = p.G * kAttnD + 2 * p.G;
  MacoEltArgs a;
  const size_t esz = 2;
  a.in0 = reinterpret_cast<const uint8_t*>(p.q) + ((size_t)(b * p.Hkv + kvh) * p.G * kAttnD) * esz;
  const size_t kv_off = ((size_t)b * p.kv_batch_stride + (size_t)kvh * p.kv_head_stride + (size_t)s0 * kAttnD) * esz;
  a.in1 = reinterpret_cast<const uint8_t*>(p.k) + kv_off;
  a.in2 = reinterpret_cast<const uint8_t*>(p.v) + kv_off;
  a.out = p.scratch + (size_t)blockIdx.x * rec;
  a.row0 = 0; a.rows = rows; a.cols = kAttnD; a.dtype = p.dtype; a.ld_in = kAttnD; a.ld_out = 0;
  a.f0 = p.scale; a.f1 = 0.f; a.i0 = p.G; a.i1 = 0;
  attn_decode_task(a, threadIdx.x, scratch_smem);
}

__global__ void __launch_bounds__(128) attn_merge_kernel(AttnParams p) {
  const int bh = blockIdx.x;
  const int rec = p.G * kAttnD + 2 * p.G;
  MacoEltArgs a;
  a.in0 = p.scratch + (size_t)bh * p.splits * rec;
  a.in1 = nullptr; a.in2 = nullptr;
  a.out = reinterpret_cast<uint8_t*>(p.out) + (size_t)bh * p.G * kAttnD * 2;
  a.row0 = 0; a.rows = 0; a.cols = kAttnD; a.dtype = p.dtype; a.ld_in = 0; a.ld_out = 0;
  a.f0 = 0.f; a.f1 = 0.f; a.i0 = p.G; a.i1 = p.splits;
  attn_merge_task(a, threadIdx.x);
}

// ---- streaming form --------------------------------------------------------------------------
// 160 threads: four consumer warps and a TMA warp around a 192 KB ring, one CTA per SM. What bounds it is the HBM stream
// of K and V; the shares are equal to one 128-key chunk, so no SM runs a second wave, and a share that ends inside a
// (batch, kv-head) leaves a record of at most 4.2 KB. Batch 16 x 8 kv heads x 8192 keys (537 MB), one B200: 86-87 us (6.2 TB/s),
// against 117 us through a tcgen05 task of the persistent kernel.
struct AttnStreamParams {
  const void* q; void* out; float* scratch; uint32_t* status;
  int Hkv, G, S, chunks_per_head, groups;
  long long total;                                 // groups * chunks_per_head
  float scale;
};
constexpr int kStreamThreads = 160;
constexpr int kStreamSmem = 1024 + kAttnStages * kAttnStageBytes + kAttnTcScratchBytes + 128;

// (32-bit division where the product fits: 2^24 chunks times 148 shares)
MACO_DEVICE long long share_begin(const AttnStreamParams& p, int cta, int n) {
  return p.total < (1ll << 24) ? (long long)((uint32_t)p.total * (uint32_t)cta / (uint32_t)n) : p.total * cta / n;
}

template <int DTT>
__global__ void __launch_bounds__(kStreamThreads, 1)
attn_stream_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const AttnStreamParams p) {
  extern __shared__ uint8_t dyn_smem[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dyn_smem) + 1023) & ~uintptr_t(1023));
  uint8_t* scratch = ring + kAttnStages * kAttnStageBytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(scratch + kAttnTcScratchBytes);
  uint64_t* empty = full + kAttnStages;
  volatile uint32_t* abort_word = reinterpret_cast<volatile uint32_t*>(empty + kAttnStages);
  asm volatile("griddepcontrol.launch_dependents;");   // the merge waits for this grid's end anyway; its CTAs may take their places now
  if (threadIdx.x == 0) {
    for (int s = 0; s < kAttnStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 4); }
    *abort_word = 0;
    fence_mbar_init();
  }
  __syncthreads();
  constexpr uint64_t kBudgetNs = 2000000000ull;
  const long long begin = share_begin(p, blockIdx.x, gridDim.x), end = share_begin(p, blockIdx.x + 1, gridDim.x);
  uint32_t ait = 0;
  const int tid = threadIdx.x, warp = warp_uniform(tid >> 5);
  bool ok = true;
  for (long long pos = begin; pos < end && ok;) {
    const int group = p.total < (1ll << 24) ? (int)((uint32_t)pos / (uint32_t)p.chunks_per_head) : (int)(pos / p.chunks_per_head);
    const int c0 = (int)(pos - (long long)group * p.chunks_per_head);
    const int n = (int)min((long long)(p.chunks_per_head - c0), end - pos);
    const int key0 = c0 * 128, rows = min(p.S - key0, n * 128);
    if (warp == 4) {
      const uint64_t pol = attn_evict_first();
      const int b = group / p.Hkv, h = group - b * p.Hkv;
      for (int i = 0; i < n && ok; ++i)
        ok = attn_load_chunk(ring, full, empty, &tmK, &tmV, key0 + i * 128, h, b, ait, pol, kBudgetNs, abort_word);
    } else {
      float o[kAttnMaxG], M[kAttnMaxG], L[kAttnMaxG];
      auto bar = [] { attn_bar(); };
      const size_t row0 = (size_t)group * p.G * kAttnD * 2;
      ok = attn_consume_range<DTT, true>(reinterpret_cast<const uint8_t*>(p.q) + row0, p.G, rows, p.scale * 1.4426950408889634f, ring, full, empty, ait,
                                   scratch, tid, kBudgetNs, abort_word, bar, o, M, L);
      if (ok && n == p.chunks_per_head) {
#pragma unroll
        for (int g = 0; g < kAttnMaxG; ++g)
          if (g < p.G) store1(reinterpret_cast<uint8_t*>(p.out) + row0, g * kAttnD + tid, DTT, L[g] > 0.f ? o[g] / L[g] : 0.f);
      } else if (ok) {
        // slot 0: the range starts with the share, slot 1: it ends with it (attn_stream_merge_kernel uses the same rule)
        attn_store_record(p.scratch + ((size_t)blockIdx.x * 2 + (pos == begin ? 0 : 1)) * (p.G * kAttnD + 2 * p.G), p.G, tid, o, M, L);
      }
    }
    pos += n;
  }
  if (!ok && warp == 4) {                            // loads in flight land in this CTA's memory
    const AttnPipe pp{ring, full, empty, kBudgetNs, abort_word};
    attn_drain_loads(pp, ait);
  }
  __syncthreads();
  if (tid == 0 && *abort_word != 0 && p.status != nullptr) st_relaxed_sys_u32(p.status, MACO_STATUS_TIMEOUT);
}

// ONE_HEAD: a CTA per head. With all G heads of a group in one CTA a thread has registers for two records, and the twelve records of a cache
// of 1357 keys in 128-key shares were six round trips to L2 in a row (16.2 us for the call, 13.7 with a CTA per head and the call in C). Where a group has two or three
// records there is nothing to gain, and G times the CTAs cost (16 x 8 kv heads x 8192 keys 88.2 us, 89.3 with a CTA per head): see launch_stream.
constexpr int kMergeAhead = 8;
template <int DTT, bool ONE_HEAD>
__global__ void __launch_bounds__(128) attn_stream_merge_kernel(const AttnStreamParams p, int n_ctas) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int group = blockIdx.x, g = blockIdx.y, tid = threadIdx.x;
  const long long first = (long long)group * p.chunks_per_head, last = first + p.chunks_per_head - 1;
  // the CTA whose share holds chunk x: floor estimate, then exact (shares differ by at most one chunk)
  auto owner = [&](long long x) {
    int c = p.total < (1ll << 24) ? (int)((uint32_t)x * (uint32_t)n_ctas / (uint32_t)p.total) : (int)(x * n_ctas / p.total);
    while (c > 0 && share_begin(p, c, n_ctas) > x) --c;
    while (c + 1 < n_ctas && share_begin(p, c + 1, n_ctas) <= x) ++c;
    return c;
  };
  const int lo = owner(first), hi = owner(last), n = hi - lo + 1;
  if (n == 1) return;                                // one share held the whole group and wrote its rows
  const int rec = p.G * kAttnD + 2 * p.G;
  // a share behind the first one begins inside the group (slot 0); the first one may have begun in front of it (slot 1)
  const float* r0 = p.scratch + ((size_t)lo * 2 + (share_begin(p, lo, n_ctas) >= first ? 0 : 1)) * rec;
  const float* rest = p.scratch + (size_t)lo * 2 * rec;
  if constexpr (!ONE_HEAD) {
    attn_merge_records<DTT>(reinterpret_cast<uint8_t*>(p.out) + (size_t)group * p.G * kAttnD * 2, p.G, n, tid,
                            [&](int i) { return i == 0 ? r0 : rest + (size_t)i * 2 * rec; });
    return;
  }
  float M = -INFINITY, L = 0.f, acc = 0.f;
#pragma unroll 1
  for (int i0 = 0; i0 < n; i0 += kMergeAhead) {
    float ms[kMergeAhead], ls[kMergeAhead], os[kMergeAhead];
#pragma unroll
    for (int i = 0; i < kMergeAhead; ++i) {
      const bool have = i0 + i < n;
      const float* r = i0 + i == 0 ? r0 : rest + (size_t)(i0 + i) * 2 * rec;
      ms[i] = have ? __ldcg(r + p.G * kAttnD + g) : -INFINITY;
      ls[i] = have ? __ldcg(r + p.G * kAttnD + p.G + g) : 0.f;
      os[i] = have ? __ldcg(r + g * kAttnD + tid) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < kMergeAhead; ++i) {
      const float m = fmaxf(M, ms[i]);
      const float a = M == -INFINITY ? 0.f : attn_ex2(M - m), b = ms[i] == -INFINITY ? 0.f : attn_ex2(ms[i] - m);
      L = L * a + ls[i] * b;
      acc = acc * a + os[i] * b;
      M = m;
    }
  }
  store1(reinterpret_cast<uint8_t*>(p.out) + (size_t)group * p.G * kAttnD * 2, g * kAttnD + tid, DTT, L > 0.f ? acc / L : 0.f);
}

template <int DTT>
int launch_stream(const CUtensorMap& tmK, const CUtensorMap& tmV, const AttnStreamParams& p, int grid, cudaStream_t stream) {
  static bool attr_set[64] = {};
  int dev = 0;
  MACO_CHECK_CUDA(cudaGetDevice(&dev));
  if (!attr_set[dev]) {
    MACO_CHECK_CUDA(cudaFuncSetAttribute(attn_stream_kernel<DTT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmem));
    attr_set[dev] = true;
  }
  attn_stream_kernel<DTT><<<grid, kStreamThreads, kStreamSmem, stream>>>(tmK, tmV, p);
  MACO_CHECK_CUDA(cudaGetLastError());
  if (p.chunks_per_head > 1) {                       // else a group is one chunk, and no share can end inside it
    cudaLaunchConfig_t cfg = {};
    const bool one_head = (long long)p.chunks_per_head * grid >= 4 * p.total;       // a group is four shares or more
    cfg.gridDim = dim3(p.groups, one_head ? p.G : 1); cfg.blockDim = dim3(128); cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    MACO_CHECK_CUDA(cudaLaunchKernelEx(&cfg, one_head ? attn_stream_merge_kernel<DTT, true> : attn_stream_merge_kernel<DTT, false>, p, grid));
  }
  return 0;
}

int check_and_fill(AttnParams& p, const void* q, const void* k, const void* v, void* out, float* scratch, int B,
                   int Hq, int Hkv, int S, int head_dim, int splits, int dtype, long long kv_batch_stride,
                   long long kv_head_stride, float scale) {
  if (head_dim != kAttnD) { maco_host::set_error("attention_decode: head_dim must be 128"); return -1; }
  if (Hkv <= 0 || Hq % Hkv != 0 || Hq / Hkv > kAttnMaxG) { maco_host::set_error("attention_decode: need 1..8 query heads per KV head"); return -1; }
  if (dtype != MACO_DT_BF16 && dtype != MACO_DT_F16) { maco_host::set_error("attention_decode: bf16 or fp16 only"); return -1; }
  if (splits < 1 || S < 1 || B < 1) { maco_host::set_error("attention_decode: empty problem"); return -1; }
  // the kernels read K / V rows and q with 16-byte vector loads and launch B * Hkv * splits CTAs
  if (((reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(q) |
        reinterpret_cast<uintptr_t>(out)) & 15) != 0) {
    maco_host::set_error("attention_decode: q, k, v and out must be 16-byte aligned");
    return -1;
  }
  if (kv_batch_stride % 8 != 0 || kv_head_stride % 8 != 0) {
    maco_host::set_error("attention_decode: KV batch and head strides must be multiples of 8 elements (16 bytes)");
    return -1;
  }
  if ((long long)B * Hkv * splits > 2147483647LL) { maco_host::set_error("attention_decode: B * Hkv * splits exceeds the grid limit"); return -1; }
  p.q = q; p.k = k; p.v = v; p.out = out; p.scratch = scratch; p.B = B; p.Hkv = Hkv; p.G = Hq / Hkv; p.S = S;
  p.splits = splits; p.dtype = dtype; p.kv_batch_stride = kv_batch_stride; p.kv_head_stride = kv_head_stride;
  p.scale = scale;
  return 0;
}

}  // namespace

extern "C" {

// Bytes of fp32 scratch the call needs.
unsigned long long maco_attention_decode_scratch_bytes(int B, int Hq, int Hkv, int splits) {
  const int G = Hq / (Hkv > 0 ? Hkv : 1);
  return (unsigned long long)B * Hkv * splits * (G * kAttnD + 2 * G) * sizeof(float);
}

int maco_attention_decode(const void* q, const void* k, const void* v, void* out, void* scratch, int B, int Hq, int Hkv,
                          int S, int head_dim, int splits, int dtype, long long kv_batch_stride,
                          long long kv_head_stride, float scale, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  AttnParams p;
  int rc = check_and_fill(p, q, k, v, out, reinterpret_cast<float*>(scratch), B, Hq, Hkv, S, head_dim, splits, dtype,
                          kv_batch_stride, kv_head_stride, scale);
  if (rc != 0) return rc;
  if (scratch == nullptr) { maco_host::set_error("attention_decode: scratch is null"); return -1; }
  attn_decode_kernel<<<B * Hkv * splits, 128, 0, stream>>>(p);
  attn_merge_kernel<<<B * Hkv, 128, 0, stream>>>(p);
  MACO_CHECK_CUDA(cudaGetLastError());
  return 0;
}

// Streaming form: scratch for 2 records per CTA.
unsigned long long maco_attention_stream_scratch_bytes(int G) {
  return (unsigned long long)maco_host::sm_count() * 2 * (G * kAttnD + 2 * G) * sizeof(float);
}

// Returns -2 when the caches cannot be addressed by a tensor map (use maco_attention_decode).
int maco_attention_decode_stream(const void* q, const void* k, const void* v, void* out, void* scratch, int B, int Hq, int Hkv, int S,
                                 int dtype, long long kv_batch_stride, long long kv_head_stride, float scale, void* stream_) {
  AttnParams c;
  int rc = check_and_fill(c, q, k, v, out, reinterpret_cast<float*>(scratch), B, Hq, Hkv, S, kAttnD, 1, dtype, kv_batch_stride, kv_head_stride, scale);
  if (rc != 0) return rc;
  CUtensorMap tmK, tmV;
  if (maco_host::encode_kv_tmap(&tmK, k, S, Hkv, B, kv_head_stride, kv_batch_stride) != 0 ||
      maco_host::encode_kv_tmap(&tmV, v, S, Hkv, B, kv_head_stride, kv_batch_stride) != 0) return -2;
  AttnStreamParams p;
  p.q = q; p.out = out; p.scratch = reinterpret_cast<float*>(scratch); p.status = maco_host::status_device_ptr();
  p.Hkv = Hkv; p.G = Hq / Hkv; p.S = S; p.chunks_per_head = (S + 127) / 128; p.groups = B * Hkv;
  p.total = (long long)p.groups * p.chunks_per_head; p.scale = scale;
  const int sms = maco_host::sm_count();
  const int grid = p.total < sms ? (int)p.total : sms;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  return dtype == MACO_DT_BF16 ? launch_stream<MACO_DT_BF16>(tmK, tmV, p, grid, stream) : launch_stream<MACO_DT_F16>(tmK, tmV, p, grid, stream);
}

}  // extern "C"

// ---- no-allocation variant ---------------------------------------------------------------------
// See maco_no_alloc.h for the contract. The scratch of the split-KV partials lives in this
// file-scope device array; the name below is only a host-side handle for it, so host code asks the
// runtime for the real device address once per device and hands that pointer to the kernels.
#include "maco_no_alloc.h"
#include <mutex>

static __device__ __align__(256) float g_static_attn_scratch[MACO_STATIC_SCRATCH_BYTES / sizeof(float)];

namespace {
std::mutex g_static_mu;
float* g_static_ptr[64] = {};

// Device address of the static scratch on the current device (looked up on first use).
int static_scratch_ptr(float** out) {
  int dev = 0;
  MACO_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) { maco_host::set_error("attention_decode_static: device index out of range"); return -1; }
  std::lock_guard<std::mutex> lk(g_static_mu);
  if (g_static_ptr[dev] == nullptr) {
    float* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_static_attn_scratch);
    if (e != cudaSuccess || ptr == nullptr) {
      maco_host::set_error(std::string("attention_decode_static: cudaGetSymbolAddress failed: ") + cudaGetErrorString(e));
      return -1;
    }
    g_static_ptr[dev] = ptr;
  }
  *out = g_static_ptr[dev];
  return 0;
}
}  // namespace

extern "C" int maco_attention_decode_static(const void* q, const void* k, const void* v, void* out, int B, int Hq,
                                            int Hkv, int S, int head_dim, int splits, int dtype,
                                            long long kv_batch_stride, long long kv_head_stride, float scale,
                                            void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  AttnParams p;
  int rc = check_and_fill(p, q, k, v, out, nullptr, B, Hq, Hkv, S, head_dim, splits, dtype, kv_batch_stride,
                          kv_head_stride, scale);
  if (rc != 0) return rc;
  const unsigned long long need = maco_attention_decode_scratch_bytes(B, Hq, Hkv, splits);
  if (need > MACO_STATIC_SCRATCH_BYTES) {
    char buf[200];
    snprintf(buf, sizeof buf,
             "attention_decode_static: needs %llu bytes of scratch, the built-in array holds %u; use fewer splits "
             "or maco_attention_decode with your own scratch", need, (unsigned)MACO_STATIC_SCRATCH_BYTES);
    maco_host::set_error(buf);
    return -3;
  }
  float* scratch = nullptr;
  rc = static_scratch_ptr(&scratch);
  if (rc != 0) return rc;
  p.scratch = scratch;
  attn_decode_kernel<<<B * Hkv * splits, 128, 0, stream>>>(p);
  attn_merge_kernel<<<B * Hkv, 128, 0, stream>>>(p);
  MACO_CHECK_CUDA(cudaGetLastError());
  return 0;
}
