// Bandwidth kernels around the sync round, sm_100a:
//   snapshot      copyToTensor            out = values                  (reference src/sharedtensor.c:442-444)
//   add / sub_add addFromTensor/pushUpdate values += d | values += a-b  (reference 338-343; one target instead of four)
//   table_scales  per-tensor energies and exponent codes over a flat arena (the reference's README lists
//                 "table sync" with per-tensor magnitudes as a TODO)
//   sample_sqerr  convergence probe for benchmarks and tests
//   delay         device-side pacing
//   snapshot_join values -> a new child's replica and -> the new link's mirror in one pass
//   tensor_*      tensor-scale frames (reference wire format) encoded/decoded on the device for TCP edges
// All are grid-stride kernels with 16-byte accesses sized to 148 SMs; none waits on anything.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "round.h"

namespace st {

namespace {

constexpr int kEwThreads = 256;

inline int ew_blocks(int64_t work_items, int per_sm = 8) {
  int64_t b = (work_items + kEwThreads - 1) / kEwThreads;
  int64_t cap = 148 * per_sm;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return int(b);
}

__device__ __forceinline__ float4 ldg_stream(const float4* p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

__device__ __forceinline__ void red_add_v4(float* p, float4 d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(d.x), "f"(d.y), "f"(d.z), "f"(d.w) : "memory");
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

// ---------------------------------------------------------------------------------------------
// snapshot, add / sub_add / add_scaled_bf16
//
// All of these are bound by HBM for large tensors and by calls and launches for small ones, so each is ONE launch: the
// ragged end is handled inside, the updates set the change marks themselves and the last CTA takes back the request for
// SMs (see GpuReplica::ask_for_sms).  A CTA takes one 4096-element tile at a time, four 16-byte accesses per thread in
// flight and eight CTAs per SM.  A user tensor that is not 16-byte aligned (a slice) costs four accesses where one would
// do, on the side that is read, where the L1 serves three of them; what is written or added leaves in whole vectors all the
// same.  (Element by element on both sides, 50 M elements took 117 us to add where aligned ones take 91.)
// ---------------------------------------------------------------------------------------------
namespace {

constexpr int kVecs = kTile / 4 / kEwThreads;  // 16-byte pieces of a thread
constexpr int kElems = 8;                      // single elements of a thread in flight

// What is left to do when a CTA's part of an update or of a snapshot is done.
__device__ __forceinline__ void finish(const UpdateMarks& m, int64_t n_tiles) {
  if (m.tile_state != nullptr) {
    // Marks after the data: the CTA's reductions come before the barrier, the barrier before the fence (which is
    // cumulative), the fence before the marks.
    __syncthreads();
    if (threadIdx.x < 32) {
      __threadfence();
      for (int64_t t = blockIdx.x + int64_t(threadIdx.x) * gridDim.x; t < n_tiles; t += 32 * int64_t(gridDim.x)) __stcg(m.tile_state + t, 1u);
    }
  }
  if (m.yield_word != nullptr && threadIdx.x == 0) {
    // (a counter that wraps: whatever it held before, one of the grid's CTAs takes the request back)
    if (atomicInc(m.ticket, gridDim.x - 1) >= gridDim.x - 1) *reinterpret_cast<volatile uint32_t*>(m.yield_word) = 0u;
  }
}

inline int tile_blocks(int64_t n, int per_sm = 8) {
  const int64_t tiles = (n + kTile - 1) / kTile;
  return int(tiles < 1 ? 1 : (tiles < 148 * per_sm ? tiles : 148 * per_sm));
}

struct Bf16x4 {
  uint32_t lo, hi;
};
__device__ __forceinline__ Bf16x4 to_bf16(float4 v) {
  __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
  return {*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi)};
}
__device__ __forceinline__ float4 from_bf16(uint2 raw) {
  const float2 a = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&raw.x)), b = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// These kernels follow each other and other small kernels closely: each may be launched while the one before it in the
// stream runs out, and waits for it before it touches memory.
__device__ __forceinline__ void wait_for_stream() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... P, class... A>
int launch_early(void (*kernel)(P...), int blocks, void* stream, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(kEwThreads);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute early{};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &early;
  cfg.numAttrs = 1;
  return int(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
}

// four consecutive elements from an address that is aligned for one
__device__ __forceinline__ float4 load4_any(const float* p) {
  float4 v;
  asm volatile("ld.global.f32 %0, [%4];\n\tld.global.f32 %1, [%4+4];\n\tld.global.f32 %2, [%4+8];\n\tld.global.f32 %3, [%4+12];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ uint2 load4_any(const __nv_bfloat16* p) {
  unsigned short a, b, c, d;
  asm volatile("ld.global.u16 %0, [%4];\n\tld.global.u16 %1, [%4+2];\n\tld.global.u16 %2, [%4+4];\n\tld.global.u16 %3, [%4+6];"
               : "=h"(a), "=h"(b), "=h"(c), "=h"(d)
               : "l"(p));
  return make_uint2(uint32_t(a) | (uint32_t(b) << 16), uint32_t(c) | (uint32_t(d) << 16));
}
__device__ __forceinline__ float4 load4(const float* p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

// Tiles are taken from the last to the first, the other way round than an update takes them.  A training loop pulls after it
// has pushed: the pull then begins with the values that are still in the L2, and the next push with those that the pull has
// read last.  For 50 M elements pushUpdate + copyToTensor take 174 us instead of 182, for 100 M 371 instead of 379; below some
// 20 M, where everything stays in the L2 anyway, it makes no difference.  (Hints that the other tensors are the first to leave
// the L2 add nothing to that, hints that the values are the last to leave take it away again.)
// VEC: the source is aligned.  The destination is (launch_snapshot moves both on to its first whole vector).
template <class T, bool VEC>
__global__ void __launch_bounds__(kEwThreads, 8) snapshot_kernel(const float* src, T* dst, int64_t n, int head, UpdateMarks m) {
  constexpr bool kBf16 = sizeof(T) == 2;
  const int64_t n_tiles = (n + kTile - 1) / kTile;
  wait_for_stream();
  for (int64_t turn = blockIdx.x; turn < n_tiles; turn += gridDim.x) {
    const int64_t tile = n_tiles - 1 - turn;
    if ((tile + 1) * kTile <= n) {
      const float* s4 = src + tile * kTile + threadIdx.x * 4;
      float4 v[kVecs];
#pragma unroll
      for (int i = 0; i < kVecs; i++) v[i] = VEC ? load4(s4 + i * 4 * kEwThreads) : load4_any(s4 + i * 4 * kEwThreads);
#pragma unroll
      for (int i = 0; i < kVecs; i++) {
        if constexpr (kBf16) {
          const Bf16x4 o = to_bf16(v[i]);
          __stcs(reinterpret_cast<uint2*>(dst + tile * kTile) + threadIdx.x + i * kEwThreads, make_uint2(o.lo, o.hi));
        } else {
          __stcs(reinterpret_cast<float4*>(dst + tile * kTile) + threadIdx.x + i * kEwThreads, v[i]);
        }
      }
    } else {
      const int left = int(min(int64_t(kTile), n - tile * kTile));
      for (int e0 = threadIdx.x; e0 < left; e0 += kElems * kEwThreads) {
        float v[kElems];
#pragma unroll
        for (int i = 0; i < kElems; i++)
          if (e0 + i * kEwThreads < left) v[i] = src[tile * kTile + e0 + i * kEwThreads];
#pragma unroll
        for (int i = 0; i < kElems; i++) {
          if (e0 + i * kEwThreads >= left) continue;
          if constexpr (kBf16) dst[tile * kTile + e0 + i * kEwThreads] = __float2bfloat16_rn(v[i]);
          else dst[tile * kTile + e0 + i * kEwThreads] = v[i];
        }
      }
    }
  }
  if (!VEC && blockIdx.x == 0 && int(threadIdx.x) < head) {  // the elements before the first whole vector
    const float x = src[int(threadIdx.x) - head];
    if constexpr (kBf16) dst[int(threadIdx.x) - head] = __float2bfloat16_rn(x);
    else dst[int(threadIdx.x) - head] = x;
  }
  finish(m, n_tiles);
}

enum Update { kAdd, kSubAdd, kScaledBf16 };
constexpr int update_ctas(int kind) { return kind == kSubAdd ? 5 : 8; }  // per SM: two operands take more registers

// values += a | values += a - b | values += alpha * a (bf16: the optimiser step of plain SGD fused with addFromTensor, so
// that bf16 training never materialises an fp32 delta)
// ALIGN: 2 = everything is aligned for vectors, 1 = the values are, 0 = not even those (never a replica's own)
template <int KIND, bool ATOMIC, int ALIGN>
__global__ void __launch_bounds__(kEwThreads, update_ctas(KIND)) update_kernel(float* values, const void* a_v, const float* b,
                                                               float alpha, int64_t n, UpdateMarks m) {
  const int64_t n_tiles = (n + kTile - 1) / kTile;
  wait_for_stream();
  for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int64_t base = tile * kTile;
    if (ALIGN > 0 && base + kTile <= n) {
      float4 d[kVecs];
      if constexpr (KIND == kScaledBf16) {
        const __nv_bfloat16* g = static_cast<const __nv_bfloat16*>(a_v) + base + threadIdx.x * 4;
        uint2 raw[kVecs];
#pragma unroll
        for (int i = 0; i < kVecs; i++)
          raw[i] = ALIGN == 2 ? __ldcs(reinterpret_cast<const uint2*>(g + i * 4 * kEwThreads)) : load4_any(g + i * 4 * kEwThreads);
#pragma unroll
        for (int i = 0; i < kVecs; i++) {
          d[i] = from_bf16(raw[i]);
          d[i].x *= alpha; d[i].y *= alpha; d[i].z *= alpha; d[i].w *= alpha;
        }
      } else {
        const float* a = static_cast<const float*>(a_v) + base + threadIdx.x * 4;
#pragma unroll
        for (int i = 0; i < kVecs; i++)
          d[i] = ALIGN == 2 ? ldg_stream(reinterpret_cast<const float4*>(a + i * 4 * kEwThreads)) : load4_any(a + i * 4 * kEwThreads);
        if constexpr (KIND == kSubAdd) {
#pragma unroll
          for (int i = 0; i < kVecs; i++) {
            const float* bp = b + base + (threadIdx.x + i * kEwThreads) * 4;
            const float4 o = ALIGN == 2 ? ldg_stream(reinterpret_cast<const float4*>(bp)) : load4_any(bp);
            d[i].x -= o.x; d[i].y -= o.y; d[i].z -= o.z; d[i].w -= o.w;
          }
        }
      }
#pragma unroll
      for (int i = 0; i < kVecs; i++) {
        float4* v4 = reinterpret_cast<float4*>(values + base) + threadIdx.x + i * kEwThreads;
        if (ATOMIC) {
          red_add_v4(reinterpret_cast<float*>(v4), d[i]);
        } else {
          float4 v = *v4;
          v.x += d[i].x; v.y += d[i].y; v.z += d[i].z; v.w += d[i].w;
          *v4 = v;
        }
      }
    } else {
      const int left = int(min(int64_t(kTile), n - base));
      for (int e0 = threadIdx.x; e0 < left; e0 += kElems * kEwThreads) {
        float d[kElems];
#pragma unroll
        for (int i = 0; i < kElems; i++) {
          const int e = e0 + i * kEwThreads;
          if (e >= left) continue;
          if constexpr (KIND == kScaledBf16) d[i] = alpha * __bfloat162float(static_cast<const __nv_bfloat16*>(a_v)[base + e]);
          else d[i] = static_cast<const float*>(a_v)[base + e];
        }
        if constexpr (KIND == kSubAdd) {
#pragma unroll
          for (int i = 0; i < kElems; i++)
            if (e0 + i * kEwThreads < left) d[i] -= b[base + e0 + i * kEwThreads];
        }
#pragma unroll
        for (int i = 0; i < kElems; i++) {
          const int e = e0 + i * kEwThreads;
          if (e >= left) continue;
          if (ATOMIC) atomicAdd(values + base + e, d[i]);
          else values[base + e] += d[i];
        }
      }
    }
  }
  finish(m, n_tiles);
}

template <int KIND>
int launch_update(float* values, const void* a, const float* b, float alpha, int64_t n, int atomic, const UpdateMarks& m, void* stream) {
  const bool src = (KIND == kScaledBf16 ? (reinterpret_cast<uintptr_t>(a) & 7) == 0 : aligned16(a)) && (KIND != kSubAdd || aligned16(b));
  const int align = !aligned16(values) ? 0 : (src ? 2 : 1);
  const auto kernel = atomic ? (align == 2 ? update_kernel<KIND, true, 2> : (align == 1 ? update_kernel<KIND, true, 1> : update_kernel<KIND, true, 0>))
                             : (align == 2 ? update_kernel<KIND, false, 2> : (align == 1 ? update_kernel<KIND, false, 1> : update_kernel<KIND, false, 0>));
  return launch_early(kernel, tile_blocks(n, update_ctas(KIND)), stream, values, a, b, alpha, n, m);
}

}  // namespace

template <class T>
static int launch_snapshot(const float* values, T* out, int64_t n, const UpdateMarks& m, void* stream) {
  // elements before `out` is aligned for four of them
  const int64_t head = int64_t((4 - reinterpret_cast<uintptr_t>(out) / sizeof(T) % 4) % 4);
  const int h = int(head < n ? head : n);
  const bool vec = h == 0 && aligned16(values);
  return launch_early(vec ? snapshot_kernel<T, true> : snapshot_kernel<T, false>, tile_blocks(n - h), stream, values + h, out + h, n - h, h, m);
}
int launch_snapshot_f32(const float* values, float* out, int64_t n, const UpdateMarks& m, void* stream) {
  return launch_snapshot(values, out, n, m, stream);
}
int launch_snapshot_bf16(const float* values, void* out, int64_t n, const UpdateMarks& m, void* stream) {
  return launch_snapshot(values, static_cast<__nv_bfloat16*>(out), n, m, stream);
}
int launch_add(float* values, const float* delta, int64_t n, int atomic, const UpdateMarks& m, void* stream) {
  return launch_update<kAdd>(values, delta, nullptr, 1.f, n, atomic, m, stream);
}
int launch_sub_add(float* values, const float* neu, const float* old, int64_t n, int atomic, const UpdateMarks& m, void* stream) {
  return launch_update<kSubAdd>(values, neu, old, 1.f, n, atomic, m, stream);
}
int launch_add_scaled_bf16(float* values, const void* g_bf16, float alpha, int64_t n, int atomic, const UpdateMarks& m, void* stream) {
  return launch_update<kScaledBf16>(values, g_bf16, nullptr, alpha, n, atomic, m, stream);
}

__global__ void fill_state_kernel(uint32_t* s, int n, uint32_t v) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) s[i] = v;
}
__global__ void set_word_kernel(uint32_t* w, uint32_t v) { *w = v; }
int launch_set_word(uint32_t* word, uint32_t value, void* stream) {
  set_word_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(word, value);
  return int(cudaGetLastError());
}
int launch_fill_state(uint32_t* tile_state, int n_tiles, uint32_t value, void* stream) {
  fill_state_kernel<<<(n_tiles + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(tile_state, n_tiles, value);
  return int(cudaGetLastError());
}

// ---------------------------------------------------------------------------------------------
// table_scales: two passes.  Pass 1: every CTA owns a contiguous chunk of one segment and writes one
// partial sum (double) into scratch.  Pass 2: one warp per segment adds that segment's partials in a
// fixed order (deterministic result) and derives the exponent code of the segment's RMS.
// ---------------------------------------------------------------------------------------------
constexpr int64_t kTsChunk = 1 << 16;  // elements per pass-1 CTA

int64_t table_scales_scratch_doubles(int n_seg, int64_t n_total) { return n_total / kTsChunk + 2 * int64_t(n_seg) + 2; }

// chunk c of the arena's chunk list: segment s covers chunks [first[s], first[s+1]).  A CTA walks over every
// gridDim.x-th chunk; a thread keeps four independent 16-byte loads in flight and four independent sums.
__global__ void __launch_bounds__(256) table_partial_kernel(const float* __restrict__ x, const int64_t* __restrict__ off, int n_seg,
                                                            const int64_t* __restrict__ first_chunk, double* __restrict__ partials,
                                                            int64_t max_chunks) {
  __shared__ double red[8];
  __shared__ int s_seg;
  int64_t n_chunks = first_chunk[n_seg];
  if (n_chunks > max_chunks) n_chunks = max_chunks;  // an inconsistent table never reaches past the scratch buffer
  for (int64_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
    if (threadIdx.x == 0) {
      int lo = 0, hi = n_seg - 1;  // last segment whose first chunk is <= c
      while (lo < hi) {
        int mid = (lo + hi + 1) / 2;
        if (first_chunk[mid] <= c) lo = mid; else hi = mid - 1;
      }
      s_seg = lo;
    }
    __syncthreads();
    const int seg = s_seg;
    const int64_t begin = off[seg] + (c - first_chunk[seg]) * kTsChunk;
    const int64_t end = min(begin + kTsChunk, off[seg + 1]);
    double acc = 0.0;
    // 16-byte loads over the aligned middle of the chunk, scalar loads at its ragged ends
    int64_t a0 = (begin + 3) & ~int64_t(3);
    if (a0 > end) a0 = end;
    const int64_t a1 = a0 + ((end - a0) & ~int64_t(3));
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
      for (int64_t i = begin + threadIdx.x; i < a0; i += 256) acc += double(x[i]) * double(x[i]);
      const float4* x4 = reinterpret_cast<const float4*>(x);
      const int64_t q1 = a1 / 4;
      int64_t i = a0 / 4 + threadIdx.x;
      double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
      for (; i + 768 < q1; i += 1024) {
        const float4 v0 = ldg_stream(x4 + i), v1 = ldg_stream(x4 + i + 256), v2 = ldg_stream(x4 + i + 512), v3 = ldg_stream(x4 + i + 768);
        s0 += (double(v0.x) * double(v0.x) + double(v0.y) * double(v0.y)) + (double(v0.z) * double(v0.z) + double(v0.w) * double(v0.w));
        s1 += (double(v1.x) * double(v1.x) + double(v1.y) * double(v1.y)) + (double(v1.z) * double(v1.z) + double(v1.w) * double(v1.w));
        s2 += (double(v2.x) * double(v2.x) + double(v2.y) * double(v2.y)) + (double(v2.z) * double(v2.z) + double(v2.w) * double(v2.w));
        s3 += (double(v3.x) * double(v3.x) + double(v3.y) * double(v3.y)) + (double(v3.z) * double(v3.z) + double(v3.w) * double(v3.w));
      }
      for (; i < q1; i += 256) {
        const float4 v = ldg_stream(x4 + i);
        s0 += (double(v.x) * double(v.x) + double(v.y) * double(v.y)) + (double(v.z) * double(v.z) + double(v.w) * double(v.w));
      }
      acc += (s0 + s1) + (s2 + s3);
      for (int64_t j = a1 + threadIdx.x; j < end; j += 256) acc += double(x[j]) * double(x[j]);
    } else {
      for (int64_t i = begin + threadIdx.x; i < end; i += 256) {
        float v = x[i];
        acc += double(v) * double(v);
      }
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < 8; w++) t += red[w];
      partials[c] = t;
    }
    __syncthreads();  // red and s_seg are reused by the next chunk
  }
}
__global__ void table_final_kernel(const int64_t* __restrict__ off, int n_seg, const int64_t* __restrict__ first_chunk,
                                   const double* __restrict__ partials, double* __restrict__ out_sumsq, int8_t* __restrict__ out_exp,
                                   int64_t max_chunks) {
  int seg = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (seg >= n_seg) return;
  const int lane = threadIdx.x & 31;
  double acc = 0.0;
  const int64_t c0 = first_chunk[seg], c1 = first_chunk[seg + 1];
  const bool consistent = c0 >= 0 && c0 <= c1 && c1 <= max_chunks;  // offsets that ascend and end where the caller said
  if (consistent)
    for (int64_t c = c0 + lane; c < c1; c += 32) acc += partials[c];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) {
    int64_t cnt = off[seg + 1] - off[seg];
    int e = -128;
    if (!consistent) {
      acc = __longlong_as_double(0x7ff8000000000000LL);  // NaN: the table contradicts n_total
    } else if (cnt > 0 && acc > 0.0) {
      double rms = sqrt(acc / double(cnt));
      int ex;
      frexp(rms, &ex);
      e = ex - 1;
      if (e < -126) e = -128;
      if (e > 127) e = 127;
    }
    out_sumsq[seg] = acc;
    out_exp[seg] = int8_t(e);
  }
}
__global__ void table_chunks_kernel(const int64_t* __restrict__ off, int n_seg, int64_t* __restrict__ first_chunk) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    int64_t c = 0;
    for (int s = 0; s < n_seg; s++) {
      first_chunk[s] = c;
      const int64_t len = off[s + 1] - off[s];
      c += len > 0 ? (len + kTsChunk - 1) / kTsChunk : 0;
    }
    first_chunk[n_seg] = c;
  }
}

int launch_table_scales(const float* x, const int64_t* seg_offsets_dev, int n_seg, int64_t n_total, double* scratch, double* out_sumsq,
                        int8_t* out_exp, void* stream_v) {
  cudaStream_t s = static_cast<cudaStream_t>(stream_v);
  // scratch layout: [first_chunk: n_seg+1 int64][partials: up to n_total/chunk + n_seg doubles]
  int64_t* first_chunk = reinterpret_cast<int64_t*>(scratch);
  double* partials = scratch + (n_seg + 1);
  const int64_t max_chunks = n_total / kTsChunk + n_seg;  // holds for offsets that ascend from 0 to n_total
  table_chunks_kernel<<<1, 32, 0, s>>>(seg_offsets_dev, n_seg, first_chunk);
  // the exact chunk count lives on the device: a grid of at most eight CTAs per SM walks over the chunks there are
  const int64_t grid = max_chunks < 148 * 8 ? (max_chunks < 1 ? 1 : max_chunks) : 148 * 8;
  table_partial_kernel<<<unsigned(grid), 256, 0, s>>>(x, seg_offsets_dev, n_seg, first_chunk, partials, max_chunks);
  table_final_kernel<<<(n_seg + 7) / 8, 256, 0, s>>>(seg_offsets_dev, n_seg, first_chunk, partials, out_sumsq, out_exp, max_chunks);
  return int(cudaGetLastError());
}

// ---------------------------------------------------------------------------------------------
// sample_sqerr / delay / snapshot_join
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) sample_sqerr_kernel(const float* __restrict__ a, int64_t stride_a, const float* __restrict__ b,
                                                           int64_t count, double* __restrict__ out) {
  double acc = 0.0;
  unsigned long long nan = 0;
  for (int64_t i = int64_t(blockIdx.x) * 256 + threadIdx.x; i < count; i += int64_t(gridDim.x) * 256) {
    float d = a[i * stride_a] - b[i];
    if (d != d) nan++;
    acc += double(d) * double(d);
  }
  for (int o = 16; o > 0; o >>= 1) {
    acc += __shfl_xor_sync(0xffffffffu, acc, o);
    nan += __shfl_xor_sync(0xffffffffu, nan, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(out, acc);
    if (nan) atomicAdd(reinterpret_cast<unsigned long long*>(out + 1), nan);
  }
}
int launch_sample_sqerr(const float* a, int64_t stride, const float* b, int64_t count, double* out, void* stream) {
  sample_sqerr_kernel<<<ew_blocks(count, 4), 256, 0, static_cast<cudaStream_t>(stream)>>>(a, stride, b, count, out);
  return int(cudaGetLastError());
}

// Convergence probe with a device time stamp: the sampled squared error of `a` against `b`, and when it is at or
// below `threshold` for the first time, the GPU's clock into *stamp (left alone once it is non-zero).  scratch:
// one double (the running sum, left at zero for the next launch) and one counter word behind it.
__global__ void __launch_bounds__(256) probe_converged_kernel(const float* __restrict__ a, int64_t stride_a, const float* __restrict__ b,
                                                              int64_t count, double threshold, double* __restrict__ scratch,
                                                              unsigned long long* __restrict__ stamp, double* __restrict__ last_err) {
  double acc = 0.0;
  for (int64_t i = int64_t(blockIdx.x) * 256 + threadIdx.x; i < count; i += int64_t(gridDim.x) * 256) {
    float d = a[i * stride_a] - b[i];
    acc += double(d) * double(d);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  __shared__ double part[8];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; w++) t += part[w];
    atomicAdd(scratch, t);
    __threadfence();
    unsigned int* counter = reinterpret_cast<unsigned int*>(scratch + 1);
    if (atomicAdd(counter, 1u) == gridDim.x - 1) {  // the last block: every partial sum is in
      const double total = atomicAdd(scratch, 0.0);
      *last_err = total;
      if (total <= threshold && *stamp == 0ull) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        *stamp = now;
      }
      *scratch = 0.0;
      *counter = 0u;
      __threadfence();
    }
  }
}
int launch_probe_converged(const float* a, int64_t stride, const float* b, int64_t count, double threshold, double* scratch,
                           uint64_t* stamp, double* last_err, void* stream) {
  probe_converged_kernel<<<ew_blocks(count, 2), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      a, stride, b, count, threshold, scratch, reinterpret_cast<unsigned long long*>(stamp), last_err);
  return int(cudaGetLastError());
}
// The GPU's clock into *out: launched behind an update it marks the moment the update had landed; launched alone and
// timed from the host it relates the GPU's clock to the host's.
__global__ void stamp_kernel(unsigned long long* out) {
  unsigned long long now;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
  *out = now;
}
int launch_stamp(uint64_t* out, void* stream) {
  stamp_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(reinterpret_cast<unsigned long long*>(out));
  return int(cudaGetLastError());
}

__global__ void delay_kernel(uint64_t ns) {
  uint64_t t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  // bounded by construction: the loop ends when the clock passes t0 + ns, and by an iteration cap
  for (uint64_t it = 0; it < (1ull << 32); it++) {
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (t - t0 >= ns) break;
    __nanosleep(200);
  }
}
int launch_delay(uint64_t ns, void* stream) {
  if (ns > 1000ull * 1000 * 1000) ns = 1000ull * 1000 * 1000;  // never longer than a second
  delay_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(ns);
  return int(cudaGetLastError());
}

__global__ void __launch_bounds__(kEwThreads) snapshot_join_kernel(const float4* __restrict__ values, float4* __restrict__ dst,
                                                                   float4* __restrict__ mirror, int64_t n4) {
  int64_t i = int64_t(blockIdx.x) * kEwThreads + threadIdx.x;
  const int64_t stride = int64_t(gridDim.x) * kEwThreads;
  for (; i < n4; i += stride) {
    float4 v = values[i];
    dst[i] = v;
    mirror[i] = v;
  }
}
int launch_snapshot_join(const float* values, float* dst_values, float* mirror, int64_t n_padded, void* stream) {
  int64_t n4 = n_padded / 4;
  snapshot_join_kernel<<<ew_blocks(n4), kEwThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const float4*>(values), reinterpret_cast<float4*>(dst_values), reinterpret_cast<float4*>(mirror), n4);
  return int(cudaGetLastError());
}

// ---------------------------------------------------------------------------------------------
// tensor-scale frames on the device (one scale for the whole tensor, 1 bit per element)
// ---------------------------------------------------------------------------------------------
// out2[0] = bits of max |v - k|, out2[1] = bits of max |v| (non-negative floats order like their bit patterns)
__global__ void __launch_bounds__(256) tensor_maxabs_kernel(const float* __restrict__ v, const float* __restrict__ k, int64_t n,
                                                            uint32_t* __restrict__ out2) {
  float mx = 0.f, mv = 0.f;
  for (int64_t i = int64_t(blockIdx.x) * 256 + threadIdx.x; i < n; i += int64_t(gridDim.x) * 256) {
    float a = v[i];
    mx = fmaxf(mx, fabsf(a - k[i]));
    mv = fmaxf(mv, fabsf(a));
  }
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    mv = fmaxf(mv, __shfl_xor_sync(0xffffffffu, mv, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(out2, __float_as_uint(mx));
    atomicMax(out2 + 1, __float_as_uint(mv));
  }
}
int launch_tensor_maxabs(const float* v, const float* k, int64_t n, uint32_t* out2, void* stream) {
  tensor_maxabs_kernel<<<ew_blocks(n, 4), 256, 0, static_cast<cudaStream_t>(stream)>>>(v, k, n, out2);
  return int(cudaGetLastError());
}
// words[i/32] bit i%32 = !(v-k > 0); k steps by -/+ scale.  n is padded by the caller to a multiple of 32
// with v = k = 0 beyond the valid range; `n_valid` stops the mirror update there.
__global__ void __launch_bounds__(256) tensor_encode_kernel(const float* __restrict__ v, float* __restrict__ k, int64_t n_valid, float scale,
                                                            uint32_t* __restrict__ words, int64_t n_words) {
  const int lane = threadIdx.x & 31;
  for (int64_t w = (int64_t(blockIdx.x) * 256 + threadIdx.x) >> 5; w < n_words; w += (int64_t(gridDim.x) * 256) >> 5) {
    int64_t i = w * 32 + lane;
    bool valid = i < n_valid;
    float kk = valid ? k[i] : 0.f;
    float x = valid ? v[i] - kk : 0.f;
    bool neg = valid && !(x > 0.f);
    uint32_t word = __ballot_sync(0xffffffffu, neg);
    if (valid && scale != 0.f) k[i] = kk + (neg ? -scale : scale);
    if (lane == 0) words[w] = word;
  }
}
int launch_tensor_encode(const float* v, float* k, int64_t n, float scale, uint32_t* words, void* stream) {
  int64_t n_words = (n + 31) / 32;
  tensor_encode_kernel<<<ew_blocks(n_words * 32, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(v, k, n, scale, words, n_words);
  return int(cudaGetLastError());
}
template <bool ATOMIC>
__global__ void __launch_bounds__(256) tensor_decode_kernel(const uint32_t* __restrict__ words, float scale, int64_t n, float* __restrict__ v,
                                                            float* __restrict__ k) {
  int64_t i = int64_t(blockIdx.x) * 256 + threadIdx.x;
  const int64_t stride = int64_t(gridDim.x) * 256;
  for (; i < n; i += stride) {
    float f = ((words[i >> 5] >> (i & 31)) & 1u) ? -scale : scale;
    if (ATOMIC) atomicAdd(v + i, f);
    else v[i] += f;
    if (k) k[i] += f;
  }
}
int launch_tensor_decode(const uint32_t* words, float scale, int64_t n, float* v, float* k, int atomic_v, void* stream) {
  if (scale == 0.f) return 0;
  if (atomic_v) tensor_decode_kernel<true><<<ew_blocks(n, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(words, scale, n, v, k);
  else tensor_decode_kernel<false><<<ew_blocks(n, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(words, scale, n, v, k);
  return int(cudaGetLastError());
}

}  // namespace st
