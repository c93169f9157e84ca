// A table of tensors inside one shared arena: what is laid out once per table and the launches over it (host-visible, no
// CUDA syntax).  The tensors themselves stay where the caller has them: one kernel adds all of them into the arena, or
// fills all of them from it, and one kernel reads the arena for the per-tensor magnitudes.
#pragma once
#include <cstdint>
#include <mutex>
#include <vector>

#include "round.h"

namespace st {

class TablePlan {
 public:
  // Tensor k covers elements offsets[k] .. offsets[k] + sizes[k] - 1 of the arena; its segment ends where the next one
  // starts (offsets has one more entry, the arena's size).  Offsets are multiples of 4.
  TablePlan(int device, const std::vector<int64_t>& offsets, const std::vector<int64_t>& sizes);
  ~TablePlan();
  TablePlan(const TablePlan&) = delete;

  int tensors() const { return n_; }
  // The caller's memory for the layout (device) and the magnitudes (pinned), to be given to bind() before anything else.
  size_t device_bytes() const { return bytes_; }
  size_t pinned_bytes() const { return (size_t(n_) * 2 + 1) * 8; }
  void bind(void* device_memory, void* pinned, void* stream);
  // arena[k] += *ptrs[k], a reduction at the L2, for every tensor; *ptrs[k] = arena[k].  fp32 tensors of this device,
  // tensors() addresses.
  void add(float* arena, const std::vector<uintptr_t>& ptrs, const UpdateMarks& m, void* stream) const;
  void copy(const float* arena, const std::vector<uintptr_t>& ptrs, const UpdateMarks& m, void* stream) const;
  // Per segment the sum of squares and floor(log2(rms)) (-128: all zero) of `arena`: starts the kernel that reads them / waits
  // for the stream and returns the sums, then the exponents.  The lock is held from before the one until what the other
  // returned has been read.
  std::unique_lock<std::mutex> lock_scales() { return std::unique_lock<std::mutex>(mu_); }
  void start_scales(const float* arena, void* stream);
  const double* finish_scales(void* stream);

 private:
  int device_, n_;
  int n_sum_ctas_ = 0;
  std::vector<int64_t> offsets_;
  std::vector<uint8_t> layout_;         // what bind() copies
  size_t o_sum_ = 0, o_seg_ = 0, o_fst_ = 0, o_cnt_ = 0, o_par_ = 0, bytes_ = 0;
  struct Chunk* chunks_ = nullptr;      // pieces of at most 4096 elements of the tensors, in arena order
  std::vector<uint32_t> first_chunk_;   // of each tensor
  struct SumChunk* sum_chunks_ = nullptr;  // pieces of the segments, for the sums
  struct SumSegment* sum_segments_ = nullptr;
  uint32_t* sum_first_ = nullptr;       // the first chunk of each CTA, and their number
  double* partials_ = nullptr;
  uint32_t* counters_ = nullptr;        // chunks of a segment that are done (zero between launches)
  double* host_ = nullptr;              // pinned: sums, then exponents
  std::mutex mu_;                       // the magnitudes use partials_, counters_ and host_
};

}  // namespace st
