// Split-transform kernels (split.cuh) of base algorithm 6 (Dif16).
#define CFFT_KERNEL_INSTANCE
#include "split.cuh"

namespace cfft {
template const void* split_ptr<6>(bool, int, int, bool);
}  // namespace cfft
