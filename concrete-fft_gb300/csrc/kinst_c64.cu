// Instantiations: c64 shared-memory kernels, every algorithm.
#include "c64_kernels.cuh"
#include "split.cuh"

namespace cfft {
template <int A>
static const void* pick(bool fwd) {
  return fwd ? (const void*)c64_smem_kernel<A, true> : (const void*)c64_smem_kernel<A, false>;
}
const void* c64_kernel(int algo, bool fwd) {
  switch (algo) {
    case 0: return pick<0>(fwd);
    case 1: return pick<1>(fwd);
    case 2: return pick<2>(fwd);
    case 3: return pick<3>(fwd);
    case 4: return pick<4>(fwd);
    case 5: return pick<5>(fwd);
    case 6: return pick<6>(fwd);
    case 7: return pick<7>(fwd);
    default: return nullptr;
  }
}
const void* c64_split_kernel_ptr(int algo, bool fwd, int ls, int mode) {
  switch (algo) {
    case 0: return split_ptr<0>(fwd, ls, mode);
    case 1: return split_ptr<1>(fwd, ls, mode);
    case 2: return split_ptr<2>(fwd, ls, mode);
    case 3: return split_ptr<3>(fwd, ls, mode);
    case 4: return split_ptr<4>(fwd, ls, mode);
    case 5: return split_ptr<5>(fwd, ls, mode);
    case 6: return split_ptr<6>(fwd, ls, mode);
    case 7: return split_ptr<7>(fwd, ls, mode);
    default: return nullptr;
  }
}
}  // namespace cfft
