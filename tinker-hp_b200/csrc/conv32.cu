// conv32.cu -- the three-kernel convolution of FP32 grids (conv_dev.cuh).
namespace thp {
namespace conv {
using conv_real = float;
}
}  // namespace thp

#include "conv_dev.cuh"

namespace thp {

bool conv_split32(int n, int* r1, int* r2) { return conv::split_of<float>(n, r1, r2); }

cudaError_t launch_conv32(int n, const conv::Sys& one, const conv::Sys* many, int count, int check_stop, bool real,
                          cudaStream_t st) {
  return conv::launch_length<float>(n, one, many, count, check_stop, real, st);
}

}  // namespace thp
