// Launch table of the large grids' z and inverse y passes (sns_stream.cu).
#pragma once

#include "sns_kernels.cuh"

namespace sns {

// One (N, precision), N = 256 and 512.
struct StreamOps {
  void (*init)();               // kernel attributes; call once per device before the first launch
  int (*blocks_per_sm)();       // resident CTAs
  // as Ops::yz_tma, which keeps the forward y pass; `part` (inverse y with a.clean): the map's boxes have part_rows rows, and
  // those without a row inside the sphere are not loaded
  void (*run)(const CUtensorMap& map, int axis, int dir, int variant, int part, TmaArgs a, const void* tw,
              const void* phase, Geom g, int grid, cudaStream_t st);
  int part_rows;
};

// nullptr for sizes whose passes run k_yz_tma
const StreamOps* stream_for(int n, int precision);
// this file's index-check record of the debug build, as bounds_record
int bounds_record_stream(long long* out3);

}  // namespace sns
