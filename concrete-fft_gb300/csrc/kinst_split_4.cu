// Split-transform kernels (split.cuh) of base algorithm 4 (Dif8).
#define CFFT_KERNEL_INSTANCE
#include "split.cuh"

namespace cfft {
template const void* split_ptr<4>(bool, int, int, bool);
}  // namespace cfft
