// Whole-row star stencil launches for float32 and complex64 grids.
#include "gpw_rows_launch.cuh"

namespace gpw {

cudaError_t launch_rows_f32(const OpDesc& d, int dtype, const StencilArgs& sa, int nbatch, cudaStream_t st) {
  if (dtype == GPW_F32)
    return rows_bulk_ok(sa, 4, nbatch) ? rows_radius<float, 4, true>(sa, d, nbatch, st)
                                       : rows_radius<float, 4, false>(sa, d, nbatch, st);
  return rows_bulk_ok(sa, 8, nbatch) ? rows_radius<float2, 4, true>(sa, d, nbatch, st)
                                     : rows_radius<float2, 4, false>(sa, d, nbatch, st);
}

}  // namespace gpw
