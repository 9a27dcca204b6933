// Cluster product kernels (split_product.cuh) of base algorithm 6 (Dif16).
#define CFFT_KERNEL_INSTANCE
#include "split_product.cuh"

namespace cfft {
template const void* split_product_ptr<6>(int, bool, bool);
template const void* split0_product_ptr<6>(int, int, bool);
template const void* split2_product_ptr<6>(int, int, int, bool);
}  // namespace cfft
