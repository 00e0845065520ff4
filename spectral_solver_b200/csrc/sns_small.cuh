// Launch table of the small grids' stage kernels (sns_small.cu).
#pragma once

#include "sns_kernels.cuh"

namespace sns {

// One (N, precision).  Pointers are complex arrays of the handle's element type; all launches
// go to `st`.  `clean`: u is known to be zero outside the sphere, so its pencils there are
// neither written nor read.
struct SmallOps {
  int nparts;       // CTAs of `xpass`: Nyquist partial sums per field, DIAG pairs
  int rparts;       // CTAs of `xrot`: Nyquist partial sums per field
  void (*init)();   // kernel attributes; call once per device before the first launch
  // inverse z of u[3] on both grids: work fields 2c, 2c + 1; rot (the rotational form): of the
  // vorticity too, fields 6 + 2c, 7 + 2c
  void (*zphase)(const void* u, void* work, const void* phase, const void* tw, double scale, int clean, int rot,
                 Geom g, cudaStream_t st);
  // inverse y of the first 1, 2 or 4 groups of three fields (u plain, u shifted, vorticity plain,
  // vorticity shifted); the x pass to
  // the 10 product half spectra, [10][nparts] Nyquist sums in `part` (diag: nparts
  // (sum |u|^2 / 2, max |u|^2) pairs instead, work unchanged); the rotational
  // form's x pass (12 fields -> the 6 of u x omega, [6][rparts] sums); forward y of the first
  // `fields` (6, 10 or 12)
  void (*yinv)(void* work, const void* tw, int groups, int clean, Geom g, cudaStream_t st);
  void (*xpass)(void* work, const void* unyq, const void* phase, const void* tw, double scale, double* part, int diag,
                Geom g, cudaStream_t st);
  void (*xrot)(void* work, const void* unyq, const void* phase, const void* tw, double scale, double* part, Geom g,
               cudaStream_t st);
  void (*yfwd)(void* work, const void* tw, int fields, Geom g, cudaStream_t st);
  // forward z, the sweep (prune: tiles outside the sphere are skipped) and, with emit, the
  // next stage's zphase
  void (*zsweep)(void* work, void* u, void* gbuf, void* rhs, const double* part, int nparts, const void* phase,
                 const void* tw, SweepArgs a, int prune, int emit, int rot, double scale, Geom g, cudaStream_t st);
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
