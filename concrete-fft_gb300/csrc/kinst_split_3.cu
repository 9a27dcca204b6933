// Split-transform kernels (split.cuh) of base algorithm 3 (Dit4).
#define CFFT_KERNEL_INSTANCE
#include "split.cuh"

namespace cfft {
template const void* split_ptr<3>(bool, int, int, bool);
}  // namespace cfft
