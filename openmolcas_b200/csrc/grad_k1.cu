// Gradient kernel instantiations, la+lb+1 = 1..3: one 512-thread CTA per SM
// (register budget of the __launch_bounds__ of grad_kernel); see
// grad_kernel.cuh.
#include "grad_kernel.cuh"

namespace mg {
GradFn grad_kernel_lo(int nab1, int ncd1) {
  switch (nab1) {
    case 1: return grad_fn_b<1, 1>(ncd1);
    case 2: return grad_fn_b<1, 2>(ncd1);
    case 3: return grad_fn_b<1, 3>(ncd1);
  }
  return nullptr;
}
GradFn grad_kernel_m1(int nab1, int ncd1) {
  return nab1 <= 3 ? grad_kernel_lo(nab1, ncd1) : nab1 <= 5 ? grad_kernel_mid(nab1, ncd1) : grad_kernel_hi(nab1, ncd1);
}
}  // namespace mg
