// Kernels over a table of tensors (see table.hpp).  A table of a model has a few large tensors and many small ones: a copy
// launch per tensor cost 2.1 ms of launches and gaps for the 148 tensors of GPT-2 small, whose bytes take 0.4 ms.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <stdexcept>
#include <string>

#include "table.hpp"

namespace st {

struct Chunk {
  int64_t arena;     // element of the arena
  uint32_t tensor;
  uint32_t count;    // elements
};
struct SumChunk {
  int64_t begin;     // elements of the arena
  uint32_t count;
  uint32_t segment;
};
struct SumSegment {
  uint32_t first, chunks;  // its chunks
  int64_t count;           // its elements
};

namespace {

constexpr int kThreads = 256;
constexpr uint32_t kChunk = 4096;     // a CTA's step: four 16-byte accesses per thread
constexpr int64_t kSumRange = 2048;   // the sums: elements of the arena that a CTA takes at least
constexpr int kSumLoads = 8;          // 16-byte loads of a thread in flight
constexpr int kSumCtasPerSm = 4;
constexpr int kSumCtas = 148 * kSumCtasPerSm;
constexpr int kPtrs = 256;            // tensors of one launch: their addresses travel as kernel parameters

struct Pointers {
  float* p[kPtrs];                    // less the tensor's offset, so that an arena element's number finds its tensor element
};

// Each of these kernels may be launched while the one before it in the stream runs out (which also is cheaper to issue, 2.4
// instead of 2.9 us), and waits for it before it touches anything that another one writes.
__device__ __forceinline__ void wait_for_stream() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... P, class... A>
cudaError_t launch_early(void (*kernel)(P...), int blocks, void* stream, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute early{};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &early;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

void ck(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw std::runtime_error(std::string("table of tensors: ") + what + ": " + cudaGetErrorString(e));
}

// ADD: arena += tensors (reductions at the L2), then the change marks of the arena tiles it touched, as an update does.
// Otherwise tensors = arena.  Every CTA takes every gridDim-th chunk, in arena order when it adds and from the end when it
// copies: a pull begins with what the push before it has left in the L2 (see snapshot_kernel; GPT-2 small, push and pull:
// 406 us instead of 415).
template <bool ADD>
__global__ void __launch_bounds__(kThreads, 8) table_kernel(float* __restrict__ arena, const Chunk* __restrict__ chunks, uint32_t n_chunks,
                                                            uint32_t first_tensor, const __grid_constant__ Pointers ptrs, UpdateMarks m) {
  wait_for_stream();
  for (uint32_t turn = blockIdx.x; turn < n_chunks; turn += gridDim.x) {
    const Chunk ch = chunks[ADD ? turn : n_chunks - 1 - turn];
    float* const t = ptrs.p[ch.tensor - first_tensor] + ch.arena;
    float* const a = arena + ch.arena;
    // Whole vectors on the side that is added to or written (the arena's chunks are aligned, a tensor may start anywhere);
    // the side that is read takes four accesses where it is not aligned with the other, three of which the L1 serves.
    const uint32_t head = ADD ? 0u : min(ch.count, uint32_t((4 - reinterpret_cast<uintptr_t>(t) / 4 % 4) % 4));
    const uint32_t n4 = (ch.count - head) / 4;
    const float* const src = (ADD ? t : a) + head;
    float* const dst = (ADD ? a : t) + head;
    const bool vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0;
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t at = threadIdx.x + i * kThreads;
      if (at >= n4) continue;
      if (vec) {
        v[i] = __ldcs(reinterpret_cast<const float4*>(src) + at);
      } else {
        const float* p = src + 4 * at;
        v[i] = make_float4(p[0], p[1], p[2], p[3]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint32_t at = threadIdx.x + i * kThreads;
      if (at >= n4) continue;
      if (ADD)
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(reinterpret_cast<float4*>(dst) + at), "f"(v[i].x), "f"(v[i].y), "f"(v[i].z),
                     "f"(v[i].w)
                     : "memory");
      else
        __stcs(reinterpret_cast<float4*>(dst) + at, v[i]);
    }
    // the elements before the first vector and behind the last
    const uint32_t e = threadIdx.x < head ? threadIdx.x : threadIdx.x + 4 * n4;
    if (threadIdx.x < ch.count - 4 * n4) {
      if (ADD) atomicAdd(a + e, t[e]);
      else t[e] = a[e];
    }
  }
  if (ADD && m.tile_state != nullptr) {
    __syncthreads();
    if (threadIdx.x < 32) {
      __threadfence();  // marks after the data
      for (uint32_t c = blockIdx.x + threadIdx.x * gridDim.x; c < n_chunks; c += 32 * gridDim.x) {
        const Chunk ch = chunks[c];
        __stcg(m.tile_state + ch.arena / kTile, 1u);
        __stcg(m.tile_state + (ch.arena + ch.count - 1) / kTile, 1u);
      }
    }
  }
  if (m.yield_word != nullptr && threadIdx.x == 0)
    if (atomicInc(m.ticket, gridDim.x - 1) >= gridDim.x - 1) *reinterpret_cast<volatile uint32_t*>(m.yield_word) = 0u;
}

// Sums of squares in double precision.  The arena is cut into equal ranges, one per CTA, and those into chunks where a
// segment ends: nobody waits for a last wave, and a CTA reduces over its threads once per chunk.  Whoever finishes a
// segment's last chunk adds the segment's partial sums up in their fixed order, so that the result does not depend on who
// that is, and writes it to the host.  One launch instead of three.
// Bound by HBM, which likes fewer CTAs with more loads each: 124 M elements are read in 78 us so, in 82 by eight CTAs per SM with
// four loads each.  Warp 0 sees to a finished chunk while the others have the next one's loads under way.
__global__ void __launch_bounds__(kThreads, kSumCtasPerSm) table_sums_kernel(const float* __restrict__ arena, const SumChunk* __restrict__ chunks,
                                                                 const uint32_t* __restrict__ first_chunk, const SumSegment* __restrict__ segments, double* __restrict__ partials,
                                                                 uint32_t* __restrict__ counters, double* __restrict__ out, int n_seg) {
  __shared__ double red[2][kThreads / 32];  // two chunks: the other warps may be one ahead of warp 0
  const bool aligned = (reinterpret_cast<uintptr_t>(arena) & 15) == 0;
  const uint32_t c0 = first_chunk[blockIdx.x], c1 = first_chunk[blockIdx.x + 1];
  wait_for_stream();
  for (uint32_t c = c0; c < c1; c++) {
    const SumChunk ch = chunks[c];
    double s0 = 0.0, s1 = 0.0;
    uint32_t at = 0;
    if (aligned) {
      const float4* x = reinterpret_cast<const float4*>(arena + ch.begin);  // (segments start on multiples of four)
      const uint32_t n4 = ch.count / 4;
      for (uint32_t i = threadIdx.x; i < n4; i += kSumLoads * kThreads) {
        float4 v[kSumLoads];
#pragma unroll
        for (int u = 0; u < kSumLoads; u++) v[u] = i + u * kThreads < n4 ? __ldcs(x + i + u * kThreads) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < kSumLoads; u++) {
          s0 += double(v[u].x) * double(v[u].x) + double(v[u].y) * double(v[u].y);
          s1 += double(v[u].z) * double(v[u].z) + double(v[u].w) * double(v[u].w);
        }
      }
      at = n4 * 4;
    }
    for (uint32_t i = at + threadIdx.x; i < ch.count; i += kThreads) s0 += double(arena[ch.begin + i]) * double(arena[ch.begin + i]);
    double acc = s0 + s1;
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    double* const mine = red[c & 1u];
    if ((threadIdx.x & 31) == 0) mine[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x >= 32) continue;
    const SumSegment sg = segments[ch.segment];
    uint32_t last = 0;
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < kThreads / 32; w++) t += mine[w];
      __stcg(partials + c, t);
      __threadfence();
      last = atomicAdd(counters + ch.segment, 1u) == sg.chunks - 1 ? 1u : 0u;
      if (last) __threadfence();  // the other chunks' partial sums come with the count that says they are there ...
    }
    if (__shfl_sync(0xffffffffu, last, 0)) {
      __syncwarp();               // ... for the whole warp: a shuffle orders no memory
      double t = 0.0;
      for (uint32_t i = threadIdx.x; i < sg.chunks; i += 32) t += __ldcg(partials + sg.first + i);
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (threadIdx.x == 0) {
        counters[ch.segment] = 0u;
        int e = -128;
        if (t > 0.0) {
          int ex;
          frexp(sqrt(t / double(sg.count)), &ex);
          e = ex - 1 < -126 ? -128 : min(ex - 1, 127);
        }
        out[ch.segment] = t;
        out[n_seg + ch.segment] = double(e);
      }
    }
  }
}

int blocks_for(uint32_t chunks) { return int(chunks < 148u * 8u ? chunks : 148u * 8u); }

struct OnDevice {
  int prev = -1;
  explicit OnDevice(int dev) {
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
    else prev = -1;
  }
  ~OnDevice() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

}  // namespace

TablePlan::TablePlan(int device, const std::vector<int64_t>& offsets, const std::vector<int64_t>& sizes)
    : device_(device), n_(int(sizes.size())), offsets_(offsets) {
  if (offsets.size() != sizes.size() + 1) throw std::invalid_argument("a table has one more offset than tensors");
  uint32_t n_chunks = 0;
  std::vector<SumChunk> sum_chunks;
  std::vector<SumSegment> segments;
  std::vector<uint32_t> sum_first{0};
  const int64_t range = std::max(kSumRange, ((offsets.back() + kSumCtas - 1) / kSumCtas + 1023) / 1024 * 1024);
  for (int k = 0; k < n_; k++) {
    if ((offsets[k] & 3) != 0 || sizes[k] < 0 || offsets[k + 1] < offsets[k] + sizes[k]) throw std::invalid_argument("offsets and sizes of a table contradict each other");
    first_chunk_.push_back(n_chunks);
    n_chunks += uint32_t((sizes[k] + kChunk - 1) / kChunk);
    const int64_t len = offsets[k + 1] - offsets[k];
    segments.push_back({uint32_t(sum_chunks.size()), 0u, len});
    for (int64_t at = offsets[k]; at < offsets[k + 1];) {
      const int64_t end = std::min(offsets[k + 1], (at / range + 1) * range);
      for (int64_t r = int64_t(sum_first.size()); r <= at / range; r++) sum_first.push_back(uint32_t(sum_chunks.size()));
      sum_chunks.push_back({at, uint32_t(end - at), uint32_t(k)});
      segments.back().chunks++;
      at = end;
    }
  }
  sum_first.push_back(uint32_t(sum_chunks.size()));
  n_sum_ctas_ = sum_chunks.empty() ? 0 : int(sum_first.size()) - 1;
  first_chunk_.push_back(n_chunks);
  // one block of device memory, laid out on the host and copied in one go
  auto padded = [](size_t v) { return (v + 255) / 256 * 256; };
  o_sum_ = padded(size_t(n_chunks) * sizeof(Chunk));
  o_seg_ = o_sum_ + padded(sum_chunks.size() * sizeof(SumChunk));
  o_fst_ = o_seg_ + padded(segments.size() * sizeof(SumSegment));
  o_cnt_ = o_fst_ + padded(sum_first.size() * 4);
  o_par_ = o_cnt_ + padded(size_t(n_) * 4);
  bytes_ = o_par_ + padded(sum_chunks.size() * 8) + 256;
  layout_.resize(o_par_);
  Chunk* c = reinterpret_cast<Chunk*>(layout_.data());
  for (int k = 0; k < n_; k++)
    for (int64_t at = 0; at < sizes[k]; at += kChunk) *c++ = {offsets[k] + at, uint32_t(k), uint32_t(std::min<int64_t>(kChunk, sizes[k] - at))};
  if (!sum_chunks.empty()) std::memcpy(layout_.data() + o_sum_, sum_chunks.data(), sum_chunks.size() * sizeof(SumChunk));
  if (!segments.empty()) std::memcpy(layout_.data() + o_seg_, segments.data(), segments.size() * sizeof(SumSegment));
  std::memcpy(layout_.data() + o_fst_, sum_first.data(), sum_first.size() * 4);
}

void TablePlan::bind(void* device_memory, void* pinned, void* stream) {
  OnDevice on(device_);
  uint8_t* d = static_cast<uint8_t*>(device_memory);
  ck(cudaMemcpyAsync(d, layout_.data(), layout_.size(), cudaMemcpyHostToDevice, static_cast<cudaStream_t>(stream)), "cudaMemcpyAsync");
  ck(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)), "cudaStreamSynchronize");  // (used from any stream from here on)
  std::vector<uint8_t>().swap(layout_);
  chunks_ = reinterpret_cast<Chunk*>(d);
  sum_chunks_ = reinterpret_cast<SumChunk*>(d + o_sum_);
  sum_segments_ = reinterpret_cast<SumSegment*>(d + o_seg_);
  sum_first_ = reinterpret_cast<uint32_t*>(d + o_fst_);
  counters_ = reinterpret_cast<uint32_t*>(d + o_cnt_);
  partials_ = reinterpret_cast<double*>(d + o_par_);
  host_ = static_cast<double*>(pinned);
}

TablePlan::~TablePlan() {
  if (chunks_ == nullptr) return;
  OnDevice on(device_);
  cudaDeviceSynchronize();  // kernels that use the memory may be under way on any stream
}

// The request for SMs is taken back by the last of several launches, the marks are set by each.
template <bool ADD>
static void launch_table(float* arena, const std::vector<uintptr_t>& ptrs, const std::vector<int64_t>& offsets, const Chunk* chunks,
                         const std::vector<uint32_t>& first_chunk, UpdateMarks m, void* stream) {
  const int n = int(ptrs.size());
  UpdateMarks inner = m;
  inner.yield_word = nullptr;
  const int launches = (n + kPtrs - 1) / kPtrs;
  for (int i = 0; i < launches; i++) {
    const int k0 = (ADD ? i : launches - 1 - i) * kPtrs, k1 = std::min(n, k0 + kPtrs);
    const bool last = i == launches - 1;
    Pointers p;
    for (int k = k0; k < k1; k++) p.p[k - k0] = reinterpret_cast<float*>(ptrs[k] - uintptr_t(offsets[k]) * 4);
    const uint32_t c0 = first_chunk[k0], count = first_chunk[k1] - c0;
    if (count == 0 && (!last || m.yield_word == nullptr)) continue;
    ck(launch_early(table_kernel<ADD>, count ? blocks_for(count) : 1, stream, arena, chunks + c0, count, uint32_t(k0), p, last ? m : inner), "kernel launch");
  }
}

void TablePlan::add(float* arena, const std::vector<uintptr_t>& ptrs, const UpdateMarks& m, void* stream) const {
  launch_table<true>(arena, ptrs, offsets_, chunks_, first_chunk_, m, stream);
}

void TablePlan::copy(const float* arena, const std::vector<uintptr_t>& ptrs, const UpdateMarks& m, void* stream) const {
  launch_table<false>(const_cast<float*>(arena), ptrs, offsets_, chunks_, first_chunk_, m, stream);
}

void TablePlan::start_scales(const float* arena, void* stream) {
  OnDevice on(device_);
  for (int k = 0; k < n_; k++) {  // (segments without elements)
    host_[k] = 0.0;
    host_[n_ + k] = -128.0;
  }
  if (n_sum_ctas_) {
    ck(launch_early(table_sums_kernel, n_sum_ctas_, stream, arena, sum_chunks_, sum_first_, sum_segments_, partials_, counters_, host_, n_), "kernel launch");
  }
}

const double* TablePlan::finish_scales(void* stream) {
  OnDevice on(device_);
  if (n_sum_ctas_) ck(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)), "cudaStreamSynchronize");
  return host_;
}

}  // namespace st
