// Launch table of the fused forward-z + sweep pass (sns_p5.cu).
#pragma once

#include "sns_kernels.cuh"

namespace sns {

// One (N, precision), N = 256 and 512.
struct P5Ops {
  void (*init)();          // kernel attributes; call once per device before the first launch
  int (*grid)(int nsm);    // persistent CTAs
  int chunk_rows;          // box rows (z) of the map over the state
  // work: z-pencil map of the work fields (128 bytes x up to 256 rows); state: the same of
  // u[3], g[3] with chunk_rows rows; f_u: the field u_src is in it (0, or 3 for a state in
  // the g slots); `live` (nlive entries of my * ncb + cb) restricts the pass to those tiles,
  // null: all; np = 6: all six products (the unprojected nonlinear term, a.mode 2), else 5
  void (*run)(const CUtensorMap& work, const CUtensorMap& state, int np, int f_u, void* u, void* gbuf, void* rhs,
              const double* nyq_part, int nparts, const void* tw, const void* phase, SweepArgs a, int ncb,
              const int* live, int nlive, Geom g, int grid, int* err, cudaStream_t st);
};

// nullptr for sizes without this pass (forward z and the sweep run as two kernels)
const P5Ops* p5_for(int n, int precision);
// this file's index-check record of the debug build, as bounds_record
int bounds_record_p5(long long* out3);

}  // namespace sns
