// FP64 GEMM kernels of the 32 x 32 CTA tile (4 warps of 16 x 16).
#include "dgemm_tile.cuh"

namespace uw12b {
const DgemmTile kTile32x32 = dgemm_detail::Ops<2, 2, 1, 2, 4, 5>::tile();
}  // namespace uw12b
