// Instantiations: operand preparation, every algorithm.
#include "c64_kernels.cuh"

namespace cfft {
template <int A, int E>
static const void* pick() {
  return (const void*)u64_prepare_kernel<A, E, kProdThreads>;
}
const void* u64_prepare_kernel_ptr(int algo, bool few) {
  switch (algo) {
    case 0: return few ? pick<0, 0>() : pick<0, kAddsBatch>();
    case 1: return few ? pick<1, 0>() : pick<1, kAddsBatch>();
    case 2: return few ? pick<2, 0>() : pick<2, kAddsBatch>();
    case 3: return few ? pick<3, 0>() : pick<3, kAddsBatch>();
    case 4: return few ? pick<4, 0>() : pick<4, kAddsBatch>();
    case 5: return few ? pick<5, 0>() : pick<5, kAddsBatch>();
    case 6: return few ? pick<6, 0>() : pick<6, kAddsBatch>();
    case 7: return few ? pick<7, 0>() : pick<7, kAddsBatch>();
    default: return nullptr;
  }
}
}  // namespace cfft
