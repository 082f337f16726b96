// Gradient kernel instantiations, la+lb+1 = 6, 7: one 512-thread CTA per SM
// (register budget of the __launch_bounds__ of grad_kernel); see
// grad_kernel.cuh.
#include "grad_kernel.cuh"

namespace mg {
GradFn grad_kernel_hi(int nab1, int ncd1) {
  switch (nab1) {
    case 6: return grad_fn_b<1, 6>(ncd1);
    case 7: return grad_fn_b<1, 7>(ncd1);
  }
  return nullptr;
}
}  // namespace mg
