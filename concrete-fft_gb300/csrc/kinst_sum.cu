// Instantiations: Fourier-domain product sums, every algorithm.
#include "c64_kernels.cuh"

namespace cfft {
template <int A>
static const void* pick_sum(bool reg_acc) {
  return reg_acc ? (const void*)u64_product_sum_kernel<A, kProdThreads, kSumRegAcc>
                 : (const void*)u64_product_sum_kernel<A, kProdThreads, 0>;
}
const void* u64_product_sum_kernel_ptr(int algo, bool reg_acc) {
  switch (algo) {
    case 0: return pick_sum<0>(reg_acc);
    case 1: return pick_sum<1>(reg_acc);
    case 2: return pick_sum<2>(reg_acc);
    case 3: return pick_sum<3>(reg_acc);
    case 4: return pick_sum<4>(reg_acc);
    case 5: return pick_sum<5>(reg_acc);
    case 6: return pick_sum<6>(reg_acc);
    case 7: return pick_sum<7>(reg_acc);
    default: return nullptr;
  }
}
}  // namespace cfft
