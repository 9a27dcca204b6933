// Instantiations: Fourier-domain product sums, every algorithm.
#include "c64_kernels.cuh"

namespace cfft {
template <int A, int E>
static const void* pick(bool reg_acc) {
  return reg_acc ? (const void*)u64_product_sum_kernel<A, E, kProdThreads, kSumRegAcc>
                 : (const void*)u64_product_sum_kernel<A, E, kProdThreads, 0>;
}
const void* u64_product_sum_kernel_ptr(int algo, bool reg_acc, bool few) {
  switch (algo) {
    case 0: return few ? pick<0, 0>(reg_acc) : pick<0, kAddsBatch>(reg_acc);
    case 1: return few ? pick<1, 0>(reg_acc) : pick<1, kAddsBatch>(reg_acc);
    case 2: return few ? pick<2, 0>(reg_acc) : pick<2, kAddsBatch>(reg_acc);
    case 3: return few ? pick<3, 0>(reg_acc) : pick<3, kAddsBatch>(reg_acc);
    case 4: return few ? pick<4, 0>(reg_acc) : pick<4, kAddsBatch>(reg_acc);
    case 5: return few ? pick<5, 0>(reg_acc) : pick<5, kAddsBatch>(reg_acc);
    case 6: return few ? pick<6, 0>(reg_acc) : pick<6, kAddsBatch>(reg_acc);
    case 7: return few ? pick<7, 0>(reg_acc) : pick<7, kAddsBatch>(reg_acc);
    default: return nullptr;
  }
}
}  // namespace cfft
