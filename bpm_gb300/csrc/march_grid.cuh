// The whole march of a few fields in one cooperative launch (march_grid.cu).
#pragma once

#include "march.cuh"

namespace bpmgb {

constexpr int kGridCounterStride = 32;  // unsigned: a team's counter has a 128-byte line of its own
constexpr int kGridBlocks = 128;        // blocks per field, at most

struct GridMarchArgs {
  RowParams rp;      // of the group's first field
  ColParams cp;
  const float2* u0;  // (fields, ny, nx)
  int nz;
  unsigned* counter; // kGridCounterStride unsigned per field
  unsigned long long wait_ns;
  int* timeouts;     // the kernel's word of march_timeout_words
  unsigned starve;   // 0; the wait self-test: 1, an arrival that every gathering waits for in vain
};

// fields that can march at once on the current device, 0 where the grid has no such kernel
int grid_march_capacity(int nx, int ny);
// the march of nfields (<= capacity) fields on stream s
int grid_march_launch(int nx, int ny, const GridMarchArgs& a, int nfields, cudaStream_t s);
int grid_march_status(int clear, int* v);

}  // namespace bpmgb
