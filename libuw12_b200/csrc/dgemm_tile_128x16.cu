// FP64 GEMM kernels of the 128 x 16 CTA tile (4 warps of 32 x 16).
#include "dgemm_tile.cuh"

namespace uw12b {
const DgemmTile kTile128x16 = dgemm_detail::Ops<4, 1, 2, 2, 3, 3>::tile();
}  // namespace uw12b
