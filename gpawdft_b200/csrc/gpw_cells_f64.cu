// Cell-staged star stencil launches for float64 grids.
#include "gpw_star_cells_launch.cuh"

namespace gpw {

cudaError_t launch_cells_f64(int mode, const StencilArgs& a, const OpDesc& d, int nbatch, cudaStream_t st) {
  return cells_real<double>(mode, a, d, nbatch, st);
}

}  // namespace gpw
