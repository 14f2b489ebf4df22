// Cell-staged star stencil launches (applies) for complex grids, stars and
// stars with one diagonal.
#include "gpw_star_cells_launch.cuh"

namespace gpw {

cudaError_t launch_cells_c128(const StencilArgs& a, const OpDesc& d, int nbatch, cudaStream_t st) {
  return d.slope ? cells_diagonal<double2>(a, d, nbatch, st) : cells_radius<double2, MODE_APPLY>(a, d, nbatch, st);
}

cudaError_t launch_cells_c64(const StencilArgs& a, const OpDesc& d, int nbatch, cudaStream_t st) {
  return d.slope ? cells_diagonal<float2>(a, d, nbatch, st) : cells_radius<float2, MODE_APPLY>(a, d, nbatch, st);
}

}  // namespace gpw
