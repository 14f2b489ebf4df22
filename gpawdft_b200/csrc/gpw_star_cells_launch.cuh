// Launch of the cell-staged star stencil (gpw_star_cells.cuh): tile width,
// cell size and axis-0 chunking.  Included by gpw_cells_f64.cu,
// gpw_cells_f32.cu and gpw_cells_cpx.cu, which compile the element types in
// parallel.
#pragma once
#include <algorithm>
#include <mutex>

#include "gpw_internal.h"
#include "gpw_star_cells.cuh"
#include "gpw_tma_launch.cuh"

namespace gpw {

// Rows of 16-byte cells: every row of the input, and the wrap of a periodic
// row, on a 16-byte boundary.
inline bool cells16_ok(const StencilArgs& a, size_t es, int nbatch) {
  const GridView& v = a.vin;
  return (reinterpret_cast<uintptr_t>(a.in) & 15u) == 0 && (v.n[2] * es) % 16 == 0 && (v.s1 * (int64_t)es) % 16 == 0 &&
         (v.s0 * (int64_t)es) % 16 == 0 && (nbatch == 1 || (v.sb * (int64_t)es) % 16 == 0);
}

// Equal coefficients at +q and -q on every axis.
inline bool star_symmetric(const StarCoefs& sc, int R) {
  for (int q = 1; q <= R; ++q)
    if (sc.cx[R + q] != sc.cx[R - q] || sc.cy[R + q] != sc.cy[R - q] || sc.cz[R + q] != sc.cz[R - q]) return false;
  return true;
}

template <typename T, int R, int MODE, int TZ, int CELLB, int EPI, bool SYM, int SLOPE, int PY>
cudaError_t cells_run(StencilArgs a, const OpDesc& d, int nbatch, cudaStream_t st) {
  using C = CellsCfg<T, R, MODE, TZ, CELLB, PY>;
  auto kern = star_cells_kernel<T, R, MODE, TZ, CELLB, EPI, SYM, SLOPE, PY>;
  static std::once_flag once;
  static cudaError_t oe = cudaSuccess;
  static int per_sm = 1;
  std::call_once(once, [&] {
    oe = smem_optin_bytes(kern, C::smem);
    if (oe == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, C::NT, C::smem) != cudaSuccess)
      per_sm = 1;
  });
  if (oe != cudaSuccess) return oe;
  const GridView& v = a.vout;
  dim3 grid((v.n[2] + C::TZ - 1) / C::TZ, (v.n[1] + C::TY - 1) / C::TY, 1);
  a.nchunk = tma_model_chunks(v.n[0], (int64_t)grid.x * grid.y * nbatch, R, (int64_t)std::max(1, per_sm) * num_sms());
  grid.z = a.nchunk * nbatch;
  a.nblk_seg = grid.x * grid.y * a.nchunk;
  return launch_pdl(kern, grid, dim3(C::NT), C::smem, st, a, star_coefs_typed<typename EltTraits<T>::S>(d.sc));
}

template <typename T, int R, int MODE, int TZ, int CELLB, bool SYM, int SLOPE = 0, int PY = 2>
cudaError_t cells_term(const StencilArgs& a, const OpDesc& d, int nbatch, cudaStream_t st) {
  if constexpr (MODE == MODE_APPLY) {
    if (a.aux) return cells_run<T, R, MODE, TZ, CELLB, 2, SYM, SLOPE, PY>(a, d, nbatch, st);
    if (a.pot) return cells_run<T, R, MODE, TZ, CELLB, 1, SYM, SLOPE, PY>(a, d, nbatch, st);
  }
  return cells_run<T, R, MODE, TZ, CELLB, 0, SYM, SLOPE, PY>(a, d, nbatch, st);
}

template <typename T, int R, int MODE, int TZ, int PY>
cudaError_t cells_form(const StencilArgs& a, const OpDesc& d, int nbatch, cudaStream_t st) {
  constexpr int ES = (int)sizeof(T);
  if (ES < 16 && cells16_ok(a, ES, nbatch)) return cells_term<T, R, MODE, TZ, 16, true, 0, PY>(a, d, nbatch, st);
  return cells_term<T, R, MODE, TZ, ES, true, 0, PY>(a, d, nbatch, st);
}

// Applies of a star and one diagonal of axes 0 and 1 (OpDesc::slope).
template <typename T, int R, int SLOPE>
cudaError_t cells_slope(const StencilArgs& a, const OpDesc& d, int nbatch, cudaStream_t st) {
  return cells_term<T, R, MODE_APPLY, 32, (int)sizeof(T), true, SLOPE>(a, d, nbatch, st);
}
template <typename T>
cudaError_t cells_diagonal(const StencilArgs& a, const OpDesc& d, int nbatch, cudaStream_t st) {
  switch (d.R * d.slope) {
    case 1: return cells_slope<T, 1, 1>(a, d, nbatch, st);
    case 2: return cells_slope<T, 2, 1>(a, d, nbatch, st);
    case 3: return cells_slope<T, 3, 1>(a, d, nbatch, st);
    case -1: return cells_slope<T, 1, -1>(a, d, nbatch, st);
    case -2: return cells_slope<T, 2, -1>(a, d, nbatch, st);
    case -3: return cells_slope<T, 3, -1>(a, d, nbatch, st);
  }
  return cudaErrorInvalidValue;
}

// Tiles: 64 x 32 points for float32, 32 x 16 for complex128, else 32 x 32, with
// two rows a thread; for radius 1 and 3 (the stencils of GPAW's levels) also 48
// (complex128 24) points wide; and 32 wide with one row a thread for float32
// (32 x 32: narrow grids leave fewer lanes of it empty) and, of the 8-byte
// types, for radius 1 (more CTAs per SM) and 4 (no spills).  Of these the one
// with the least work -- staged cells, and twice its points (one row a thread:
// 1.6 times) -- of all its CTAs or, where they leave resident slots empty, of as
// many as there are slots.  us with the two-row tiles alone / with this choice:
// residuals of 796 x 61 x 32 x 19 float32, radius 3, 441 / 189, of 7 x 21 x 70 x 70
// 33 / 17, of 329 x 14 x 48 x 73 float64, radius 1, 134 / 110, a Laplacian of 70 x
// 24 x 72 x 37 complex64, radius 4, 174 / 125.
template <typename T, int R, int MODE>
cudaError_t cells_width(const StencilArgs& a, const OpDesc& d, int nbatch, cudaStream_t st) {
  constexpr int ES = (int)sizeof(T), TA = ES == 4 ? 64 : 32, TB = ES == 16 ? 24 : 48;
  constexpr bool ONE = ES == 4 || (ES == 8 && (R == 1 || R == 4)), WIDE = R == 1 || R == 3;
  // other stencils than Laplacians: one tile and cell size
  if (!star_symmetric(d.sc, R)) return cells_term<T, R, MODE, 32, ES, false, 0, ES == 4 ? 1 : 2>(a, d, nbatch, st);
  auto work = [&](auto cfg) {
    using C = decltype(cfg);
    const int64_t tiles = (int64_t)((a.vout.n[2] + C::TZ - 1) / C::TZ) * ((a.vout.n[1] + C::TY - 1) / C::TY);
    const int64_t ctas = tiles * nbatch * std::max(1, a.vout.n[0] / (2 * R + 2));
    return (double)std::max<int64_t>(ctas, 2LL * num_sms()) *
           (C::H * C::W + (C::PY == 1 ? 1.6 : 2.0) * C::TZ * C::TY);
  };
  const double wa = work(CellsCfg<T, R, MODE, TA, ES, 2>());
  double wb = 1e300, wc = 1e300;
  if constexpr (WIDE) wb = work(CellsCfg<T, R, MODE, TB, ES, 2>());
  if constexpr (ONE) wc = work(CellsCfg<T, R, MODE, 32, ES, 1>());
  if constexpr (ONE) {
    if (wc < wa && wc < wb) return cells_form<T, R, MODE, 32, 1>(a, d, nbatch, st);
  }
  if constexpr (WIDE) {
    if (wb < wa) return cells_form<T, R, MODE, TB, 2>(a, d, nbatch, st);
  }
  return cells_form<T, R, MODE, TA, 2>(a, d, nbatch, st);
}

template <typename T, int MODE>
cudaError_t cells_radius(const StencilArgs& a, const OpDesc& d, int nbatch, cudaStream_t st) {
  switch (d.R) {
    case 1: return cells_width<T, 1, MODE>(a, d, nbatch, st);
    case 2: return cells_width<T, 2, MODE>(a, d, nbatch, st);
    case 3: return cells_width<T, 3, MODE>(a, d, nbatch, st);
    case 4: return cells_width<T, 4, MODE>(a, d, nbatch, st);
  }
  return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t cells_real(int mode, const StencilArgs& a, const OpDesc& d, int nbatch, cudaStream_t st) {
  switch (mode) {
    case MODE_APPLY: return cells_radius<T, MODE_APPLY>(a, d, nbatch, st);
    case MODE_RESIDUAL: return cells_radius<T, MODE_RESIDUAL>(a, d, nbatch, st);
    case MODE_JACOBI: return cells_radius<T, MODE_JACOBI>(a, d, nbatch, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace gpw
