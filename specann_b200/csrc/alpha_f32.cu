// The FP32 instantiations of the alpha-solve kernel.
#include "alpha_launch.cuh"

namespace sa {

template int launch_alpha<float, int>(sa_handle*, const sa_alpha_params*);
template int launch_alpha<float, long long>(sa_handle*, const sa_alpha_params*);
template const void* alpha_kernel_of<float, int>(int);
template const void* alpha_kernel_of<float, long long>(int);

}  // namespace sa
