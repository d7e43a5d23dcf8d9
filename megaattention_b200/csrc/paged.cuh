// A paged step's page table and key lengths (step.cu reports them, meta_upload.cu puts them in place).
#pragma once
#include <cuda_runtime.h>

namespace ma {

// The step's page table (device) and key lengths (host, as they were checked) and where the plan
// has its own copies of them (lens null: no paged step; table null: lengths only).
struct PagedIn {
  const int* table;
  const int* lens;
  int* table_out;
  int* lens_out;
  long long pitch;
  int pitch_out, width, num_batch;
};

// visit(row, column) for this thread's share (first, first + step, ...) of a table.  Entries are counted
// in 32 bits, a table of more than 2^30 by groups of rows: with 64-bit divisions a call with a small
// table took 0.7 us longer (eight sequences of 700 keys 53.6 us for 52.8).
template <class F>
__device__ __forceinline__ void for_each_entry(int num_batch, int width, unsigned first, unsigned step, F visit) {
  const unsigned w = static_cast<unsigned>(width), rows = max(1u, (1u << 30) / w);
  for (unsigned b0 = 0; b0 < static_cast<unsigned>(num_batch); b0 += rows) {
    const unsigned n = min(rows, static_cast<unsigned>(num_batch) - b0) * w;
    for (unsigned i = first; i < n; i += step) visit(static_cast<int>(b0 + i / w), static_cast<int>(i % w));
  }
}

}  // namespace ma
