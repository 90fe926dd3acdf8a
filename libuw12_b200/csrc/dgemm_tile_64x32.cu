// FP64 GEMM kernels of the 64 x 32 CTA tile (4 warps of 32 x 16).
#include "dgemm_tile.cuh"

namespace uw12b {
const DgemmTile kTile64x32 = dgemm_detail::Ops<2, 2, 2, 2, 3, 4>::tile();
}  // namespace uw12b
