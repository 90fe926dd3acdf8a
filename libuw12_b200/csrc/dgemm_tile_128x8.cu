// FP64 GEMM kernels of the 128 x 8 CTA tile (4 warps of 32 x 8).
#include "dgemm_tile.cuh"

namespace uw12b {
const DgemmTile kTile128x8 = dgemm_detail::Ops<4, 1, 2, 1, 3, 3>::tile();
}  // namespace uw12b
