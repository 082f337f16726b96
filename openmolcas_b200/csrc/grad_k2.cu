// Gradient kernel instantiations, la+lb+1 = 4, 5: one 512-thread CTA per SM
// (register budget of the __launch_bounds__ of grad_kernel); see
// grad_kernel.cuh.
#include "grad_kernel.cuh"

namespace mg {
GradFn grad_kernel_mid(int nab1, int ncd1) {
  switch (nab1) {
    case 4: return grad_fn_b<1, 4>(ncd1);
    case 5: return grad_fn_b<1, 5>(ncd1);
  }
  return nullptr;
}
}  // namespace mg
