// Cluster product kernels (split_product.cuh) of base algorithm 3 (Dit4).
#define CFFT_KERNEL_INSTANCE
#include "split_product.cuh"

namespace cfft {
template const void* split_product_ptr<3>(int, bool, bool);
template const void* split0_product_ptr<3>(int, int, bool);
template const void* split2_product_ptr<3>(int, int, int, bool);
}  // namespace cfft
