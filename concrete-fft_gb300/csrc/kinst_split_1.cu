// Split-transform kernels (split.cuh) of base algorithm 1 (Dit2).
#define CFFT_KERNEL_INSTANCE
#include "split.cuh"

namespace cfft {
template const void* split_ptr<1>(bool, int, int, bool);
}  // namespace cfft
