// FP64 instantiation of the whole-GPU form of the interior-point kernel (cxg_ipm.cuh): one
// large instance, cooperative launch, the root spread over every SM.
#define CXG_GRID_KERNELS
#define CXG_VEC_UNROLL "unroll 4"
#define CXG_UNROLLED_LEAF
#include "cxg_ipm.cuh"

namespace cxg {
CXG_IPM_GRID(, double)
}  // namespace cxg
