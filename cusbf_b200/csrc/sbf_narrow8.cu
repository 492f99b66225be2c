// sbf_narrow8.cu -- the tile kernels with strips of 8 windows, for small
// launches (see narrow_strip in sbf_kernels.cu).
#include "sbf_narrow.cuh"

namespace sbf {

const void* narrow8_kernel(int config, int which) { return narrow_kernel_of<8>(config, which); }

}  // namespace sbf
