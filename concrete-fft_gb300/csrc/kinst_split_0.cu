// Split-transform kernels (split.cuh) of base algorithm 0 (Dif2).
#define CFFT_KERNEL_INSTANCE
#include "split.cuh"

namespace cfft {
template const void* split_ptr<0>(bool, int, int, bool);
}  // namespace cfft
