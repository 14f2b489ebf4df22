// Whole-row star stencil launches for float64 and complex128 grids, and the
// rule for which grids the kernel takes.
#include "gpw_rows_launch.cuh"

namespace gpw {

// Contiguous rows (the staged block is one run of memory) and a tile that
// fits: at most 256 points a row.
bool rows_ok(const OpDesc& d, int dtype, const StencilArgs& sa, int py) {
  if (!valid_dtype(dtype) || !d.star || d.R < 1 || d.R > 3 || sa.in == sa.out || !sa.out) return false;
  const GridView& v = sa.vin;
  for (int c = 0; c < 3; ++c)
    if (v.n[c] != sa.vout.n[c] || (sa.bc.periodic[c] && v.n[c] < d.R)) return false;
  if (v.s1 != v.n[2]) return false;
  const int es = (int)elt_size(dtype);
  if (dtype == GPW_C128 && (reinterpret_cast<uintptr_t>(sa.in) & 15u)) return false;
  if (py != 4 && !(py == 2 && dtype == GPW_C128)) return false;
  return rows_plan_for(es, d.R, py, es >= 16 && py >= 4 ? 192 : 256, d.R, v).G > 0;
}

bool rows_bulk_ok(const StencilArgs& sa, size_t es, int nbatch) {
  const GridView& v = sa.vin;
  return (reinterpret_cast<uintptr_t>(sa.in) & 15u) == 0 && (v.s1 * (int64_t)es) % 16 == 0 &&
         (v.s0 * (int64_t)es) % 16 == 0 && (nbatch == 1 || (v.sb * (int64_t)es) % 16 == 0);
}

cudaError_t launch_rows(const OpDesc& d, int dtype, const StencilArgs& sa, int nbatch, int py, cudaStream_t st) {
  if (!rows_ok(d, dtype, sa, py)) return cudaErrorInvalidValue;
  switch (dtype) {
    case GPW_F64:
      return rows_bulk_ok(sa, 8, nbatch) ? rows_radius<double, 4, true>(sa, d, nbatch, st)
                                         : rows_radius<double, 4, false>(sa, d, nbatch, st);
    case GPW_C128:
      return py == 2 ? rows_radius<double2, 2, true>(sa, d, nbatch, st)
                     : rows_radius<double2, 4, true>(sa, d, nbatch, st);
    case GPW_F32:
    case GPW_C64: return launch_rows_f32(d, dtype, sa, nbatch, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace gpw
