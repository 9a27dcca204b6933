// Split-transform kernels (split.cuh) of base algorithm 7 (Dit16).
#define CFFT_KERNEL_INSTANCE
#include "split.cuh"

namespace cfft {
template const void* split_ptr<7>(bool, int, int, bool);
}  // namespace cfft
