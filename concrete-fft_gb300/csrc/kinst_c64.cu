// Instantiations: c64 shared-memory kernels, every algorithm.
#include "c64_kernels.cuh"
#include "split.cuh"

namespace cfft {
template <int A, int E>
static const void* pick(bool fwd) {
  return fwd ? (const void*)c64_smem_kernel<A, E, true> : (const void*)c64_smem_kernel<A, E, false>;
}
const void* c64_kernel(int algo, bool fwd, bool few) {
  switch (algo) {
    case 0: return few ? pick<0, 0>(fwd) : pick<0, kAddsBatch>(fwd);
    case 1: return few ? pick<1, 0>(fwd) : pick<1, kAddsBatch>(fwd);
    case 2: return few ? pick<2, 0>(fwd) : pick<2, kAddsBatch>(fwd);
    case 3: return few ? pick<3, 0>(fwd) : pick<3, kAddsBatch>(fwd);
    case 4: return few ? pick<4, 0>(fwd) : pick<4, kAddsBatch>(fwd);
    case 5: return few ? pick<5, 0>(fwd) : pick<5, kAddsBatch>(fwd);
    case 6: return few ? pick<6, 0>(fwd) : pick<6, kAddsBatch>(fwd);
    case 7: return few ? pick<7, 0>(fwd) : pick<7, kAddsBatch>(fwd);
    default: return nullptr;
  }
}
const void* c64_split_kernel_ptr(int algo, bool fwd, int ls, int mode, bool few) {
  switch (algo) {
    case 0: return split_ptr<0>(fwd, ls, mode, few);
    case 1: return split_ptr<1>(fwd, ls, mode, few);
    case 2: return split_ptr<2>(fwd, ls, mode, few);
    case 3: return split_ptr<3>(fwd, ls, mode, few);
    case 4: return split_ptr<4>(fwd, ls, mode, few);
    case 5: return split_ptr<5>(fwd, ls, mode, few);
    case 6: return split_ptr<6>(fwd, ls, mode, few);
    case 7: return split_ptr<7>(fwd, ls, mode, few);
    default: return nullptr;
  }
}
}  // namespace cfft
