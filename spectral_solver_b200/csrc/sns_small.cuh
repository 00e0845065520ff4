// Launch table of the small grids' stage kernels (sns_small.cu).
#pragma once

#include "sns_kernels.cuh"

namespace sns {

// One (N, precision).  Pointers are complex arrays of the handle's element type; all launches
// go to `st`.  `clean`: u is known to be zero outside the sphere, so its pencils there are
// neither written nor read.
struct SmallOps {
  int nparts;       // CTAs of `xpass`: Nyquist partial sums per field, DIAG pairs
  void (*init)();   // kernel attributes; call once per device before the first launch
  // inverse z of u[3] on both grids: work fields 2c, 2c + 1
  void (*zphase)(const void* u, void* work, const void* phase, const void* tw, double scale, int clean, Geom g,
                 cudaStream_t st);
  // inverse y of the first grid's fields (0, 2, 4; grids = 1) or of both grids'; the x pass to
  // the 10 product half spectra, [10][nparts] Nyquist sums in `part` (diag: nparts
  // (sum |u|^2 / 2, max |u|^2) pairs instead, work unchanged); forward y of the 10 fields
  void (*yinv)(void* work, const void* tw, int grids, int clean, Geom g, cudaStream_t st);
  void (*xpass)(void* work, const void* unyq, const void* phase, const void* tw, double scale, double* part, int diag,
                Geom g, cudaStream_t st);
  void (*yfwd)(void* work, const void* tw, Geom g, cudaStream_t st);
  // forward z, the sweep (prune: tiles outside the sphere are skipped) and, with emit, the
  // next stage's zphase
  void (*zsweep)(void* work, void* u, void* gbuf, void* rhs, const double* part, int nparts, const void* phase,
                 const void* tw, SweepArgs a, int prune, int emit, double scale, Geom g, cudaStream_t st);
  // FP64, N <= 64 (null otherwise): forward transform of a real field [z][y][x] to the full
  // complex layout through one half field of scratch; forward_init once per device before it
  void (*forward_init)();
  void (*forward)(const double* phys, void* work, void* full, const void* tw, Geom g, cudaStream_t st);
};

// nullptr for sizes without these kernels
const SmallOps* small_for(int n, int precision);
// this file's index-check record of the debug build, as bounds_record
int bounds_record_small(long long* out3);

}  // namespace sns
