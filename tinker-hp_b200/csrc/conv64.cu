// conv64.cu -- the three-kernel convolution of FP64 grids (conv_dev.cuh).
namespace thp {
namespace conv {
using conv_real = double;
}
}  // namespace thp

#include "conv_dev.cuh"

namespace thp {

bool conv_split64(int n, int* r1, int* r2) { return conv::split_of<double>(n, r1, r2); }

cudaError_t launch_conv64(int n, const conv::Sys& one, const conv::Sys* many, int count, int check_stop, bool real,
                          cudaStream_t st) {
  return conv::launch_length<double>(n, one, many, count, check_stop, real, st);
}

}  // namespace thp
