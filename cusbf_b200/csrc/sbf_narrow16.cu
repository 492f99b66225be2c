// sbf_narrow16.cu -- the tile kernels with strips of 16 windows, for small
// launches (see narrow_strip in sbf_kernels.cu).
#include "sbf_narrow.cuh"

namespace sbf {

const void* narrow16_kernel(int config, int which) { return narrow_kernel_of<16>(config, which); }

}  // namespace sbf
