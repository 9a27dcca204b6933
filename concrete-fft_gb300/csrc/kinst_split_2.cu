// Split-transform kernels (split.cuh) of base algorithm 2 (Dif4).
#define CFFT_KERNEL_INSTANCE
#include "split.cuh"

namespace cfft {
template const void* split_ptr<2>(bool, int, int, bool);
}  // namespace cfft
