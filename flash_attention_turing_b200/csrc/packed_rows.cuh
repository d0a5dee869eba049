// Rows of a packed (varlen) output tensor that belong to no sequence: before cu_seqlens[0] and from cu_seqlens[b] on.  The
// kernels write every other row, so clearing these is all that is left of clearing the whole tensor beforehand.  That was a
// pass over O, dQ, dK and dV (strided ones for a packed dqkv): a training step of 64 texts, 24 k tokens, H16 D64, qkv packed,
// took 616 us with it and 508 without, one of 16 documents, 32 k tokens, Hq32 Hkv8 D128, 4006 and 3877.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

namespace fa {

struct PackedRows {
  __half* base;  // nullptr: nothing to clear
  int64_t row_stride, head_stride;
  int64_t total;  // rows of the tensor
  int heads, d;
  const int* cu_seqlens;
  int b;
};

namespace {

// Threads that take part in a clear.  The work follows the rows to clear, which may be nearly the whole of a buffer of fixed
// capacity, and not the sequences in it; two blocks per SM (of 148) store at the memory's rate.  With eight, a backward with nothing
// to clear took 79.2 instead of 78.4 us (64 texts of 64 tokens, H16 D64): every block that takes part reads the offsets first.
constexpr int kClearThreads = 256;
constexpr int kMaxClearBlocks = 2 * 148;

// Clears rows [first, last), 16 bytes per step and thread.  The row and the 16-byte unit within it advance by constants; with two
// divisions by the row length per store the forward's clear of 28672 rows, H16 D64, took 14 us longer (63.2 -> 49.0 us in all).
__device__ __forceinline__ void clear_rows(const PackedRows& t, int64_t first, int64_t last, uint32_t worker,
                                           uint32_t workers) {
  if (first >= last) return;
  const uint32_t unit_bits = t.d == 128 ? 4 : 3;  // d / 8 units of 16 bytes per head
  const uint32_t per_row = static_cast<uint32_t>(t.heads) << unit_bits;
  const uint32_t row_step = workers / per_row, unit_step = workers % per_row;
  int64_t row = first + worker / per_row;
  uint32_t unit = worker % per_row;
  while (row < last) {
    *reinterpret_cast<uint4*>(t.base + row * t.row_stride + (unit >> unit_bits) * t.head_stride +
                              (unit & ((1u << unit_bits) - 1)) * 8) = make_uint4(0, 0, 0, 0);
    row += row_step, unit += unit_step;
    if (unit >= per_row) unit -= per_row, ++row;
  }
}

// all: clear every row.  Once a wait has timed out the kernels that write the other rows return at once, and a caller that has
// not looked at the status word would find what the memory held before.
__device__ __forceinline__ void clear_unused_rows(const PackedRows& t, bool all, uint32_t worker, uint32_t workers) {
  const int first_used = t.cu_seqlens[0], end_used = t.cu_seqlens[t.b];
  const int64_t begin = min(t.total, all ? t.total : static_cast<int64_t>(max(first_used, 0)));
  const int64_t end = max(begin, min(t.total, static_cast<int64_t>(end_used)));
  clear_rows(t, 0, begin, worker, workers);
  clear_rows(t, end, t.total, worker, workers);
}

}  // namespace
}  // namespace fa
