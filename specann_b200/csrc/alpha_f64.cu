// The FP64 instantiations of the alpha-solve kernel.
#include "alpha_launch.cuh"

namespace sa {

template int launch_alpha<double, int>(sa_handle*, const sa_alpha_params*);
template int launch_alpha<double, long long>(sa_handle*, const sa_alpha_params*);
template const void* alpha_kernel_of<double, int>(int);
template const void* alpha_kernel_of<double, long long>(int);

}  // namespace sa
