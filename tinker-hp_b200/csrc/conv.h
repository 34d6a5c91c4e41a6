// conv.h -- interface of the three-kernel PME convolution (conv_dev.cuh).
#pragma once

#include "context.h"

namespace thp {
namespace conv {

// One system's arrays: the spread grid (zeroed once it has been read), the
// convolved grid, the influence function in the convolution's x order (row
// position R2 (k % R1) + k / R1 holds x frequency k), and the CG scalars.
struct Sys {
  void* in;
  void* out;
  const void* qfac;
  const CgScalars* cg;
  void* pot;  // real form: the convolved potential, one real per point
};

}  // namespace conv

// Whether cubic grids of n points per edge are covered, and n = r1 r2 (FP32,
// FP64 grids).
bool conv_split32(int n, int* r1, int* r2);
bool conv_split64(int n, int* r1, int* r2);
// The three launches for one system (many null) or for count systems of one
// grid length described in device memory.  check_stop: a system whose CG has
// stopped is skipped.  real: the spread grid holds one real per point (in the
// front of `in`) and so does the result (in `pot`; `out` is scratch).
cudaError_t launch_conv32(int n, const conv::Sys& one, const conv::Sys* many, int count, int check_stop, bool real,
                          cudaStream_t st);
cudaError_t launch_conv64(int n, const conv::Sys& one, const conv::Sys* many, int count, int check_stop, bool real,
                          cudaStream_t st);
// whether an n1 x n2 x n3 grid takes it
bool conv_covers(const int n[3], int mixed, int* r1, int* r2);

}  // namespace thp
