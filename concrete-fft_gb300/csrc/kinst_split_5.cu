// Split-transform kernels (split.cuh) of base algorithm 5 (Dit8).
#define CFFT_KERNEL_INSTANCE
#include "split.cuh"

namespace cfft {
template const void* split_ptr<5>(bool, int, int, bool);
}  // namespace cfft
