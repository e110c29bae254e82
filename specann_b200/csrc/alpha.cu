// Dispatch of the single-problem alpha solve to its instantiations (alpha_f32.cu, alpha_f64.cu).
#include "handle.cuh"

namespace sa {

template <typename T, typename RP>
int launch_alpha(sa_handle* h, const sa_alpha_params* p);
template <typename T, typename RP>
const void* alpha_kernel_of(int mode);

int alpha_solve_impl(sa_handle* h, const sa_alpha_params* p) {
  if (h->prec == 32) {
    return h->rp64 ? launch_alpha<float, long long>(h, p) : launch_alpha<float, int>(h, p);
  }
  return h->rp64 ? launch_alpha<double, long long>(h, p) : launch_alpha<double, int>(h, p);
}

const void* alpha_kernel_for(int prec, int rp64) {
  if (prec == 32) return rp64 ? alpha_kernel_of<float, long long>(0) : alpha_kernel_of<float, int>(0);
  return rp64 ? alpha_kernel_of<double, long long>(0) : alpha_kernel_of<double, int>(0);
}

}  // namespace sa
