// Launch of the whole-row star stencil (gpw_rows.cuh) for one scalar type:
// tile height, shared memory and the (radius, rows per thread, copy form)
// dispatch.  Included by gpw_rows_f64.cu and gpw_rows_f32.cu, which compile
// the two in parallel.
#pragma once
#include <algorithm>
#include <mutex>

#include "gpw_internal.h"
#include "gpw_rows.cuh"

namespace gpw {

struct RowsPlan {
  int G, smem, nt;   // G = 0: does not fit
  int halo_off, stage_bytes;
};

// Thread groups of a tile: as many rows as the thread and shared-memory
// limits of two CTAs per SM (or one, when a single group needs it) allow, and
// among those the tile whose idle lanes, rows past the grid and staged halo
// rows (counted at a third of a computed row) cost least.
inline RowsPlan rows_plan_for(int es, int R, int py, int ntmax, int ry, const GridView& v) {
  RowsPlan best{};
  double bestc = 1e300;
  const int n1 = v.n[1], n2 = v.n[2], rb = (int)v.s1 * es;
  for (int G = 1; G * n2 <= ntmax && (G == 1 || (G - 1) * py < n1); ++G) {
    const int ty = G * py, h = ty + 2 * ry;
    RowsPlan p;
    p.G = G;
    p.halo_off = (h * rb + 15) / 16 * 16;
    p.stage_bytes = (p.halo_off + ty * 2 * R * es + 127) / 128 * 128;
    p.smem = ROWS_NS * p.stage_bytes + ROWS_NS * 8 + 128;
    p.nt = (G * n2 + 31) / 32 * 32;
    if (p.smem > (G == 1 ? 220 : 112) * 1024) break;
    const double c = (double)((n1 + ty - 1) / ty) * ((double)p.nt / n2 * py + 2 * ry / 3.0);
    if (c < bestc) {
      bestc = c;
      best = p;
    }
  }
  return best;
}

template <typename T, int R, int PY, bool BULK, bool HASX, bool EPI>
cudaError_t rows_run(const StencilArgs& sa, const OpDesc& d, int nbatch, bool has_y, bool has_z, cudaStream_t st) {
  using S = typename EltTraits<T>::S;
  const int ry = has_y ? R : 0;
  const RowsPlan p = rows_plan_for((int)sizeof(T), R, PY, RowsCfg<T, PY>::NT, ry, sa.vin);
  if (p.G < 1) return cudaErrorInvalidConfiguration;
  auto kern = star_rows_kernel<T, R, PY, BULK, HASX, EPI>;
  static std::once_flag once;
  static cudaError_t oe = cudaSuccess;
  std::call_once(once, [&] { oe = smem_optin_bytes(kern, 221 * 1024); });
  if (oe != cudaSuccess) return oe;
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, p.nt, p.smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  RowsArgs a{};
  a.in = sa.in;
  a.out = sa.out;
  a.vin = sa.vin;
  a.vout = sa.vout;
  a.bc = sa.bc;
  a.G = p.G;
  a.ty = p.G * PY;
  a.ry = ry;
  a.h = a.ty + 2 * ry;
  a.has_z = has_z ? 1 : 0;
  a.tiles = (sa.vin.n[1] + a.ty - 1) / a.ty;
  a.nb = nbatch;
  a.row_bytes = (int)(sa.vin.s1 * (int64_t)sizeof(T));
  a.halo_off = p.halo_off;
  a.stage_bytes = p.stage_bytes;
  a.halo2 = (!sa.bc.periodic[2] || (EltTraits<T>::cpx && sa.bc.use_phase)) ? 1 : 0;
  a.status = device_status_word();
  a.pot = sa.pot;
  a.aux = sa.aux;
  a.aux_scale = sa.aux_scale;
  // one CTA per resident slot, no share shorter than 2R + 2 planes
  const int64_t units = (int64_t)a.tiles * nbatch * sa.vin.n[0];
  const int64_t slots = (int64_t)per_sm * num_sms();
  const int64_t ctas = std::max<int64_t>(1, std::min<int64_t>(slots, units / (2 * R + 2)));
  return launch_pdl(kern, dim3((unsigned)ctas), dim3(p.nt), (size_t)p.smem, st, a, star_coefs_typed<S>(d.sc));
}

template <typename T, int R, int PY, bool BULK>
cudaError_t rows_form(const StencilArgs& sa, const OpDesc& d, int nbatch, cudaStream_t st) {
  bool hx = false, hy = false, hz = false;
  for (int i = 0; i <= 2 * R; ++i) {
    hx |= d.sc.cx[i] != 0.0;
    hy |= d.sc.cy[i] != 0.0;
    hz |= d.sc.cz[i] != 0.0;
  }
  if (sa.pot || sa.aux) return rows_run<T, R, PY, BULK, true, true>(sa, d, nbatch, hy, hz, st);
  if (hx) return rows_run<T, R, PY, BULK, true, false>(sa, d, nbatch, hy, hz, st);
  return rows_run<T, R, PY, BULK, false, false>(sa, d, nbatch, hy, hz, st);
}

template <typename T, int PY, bool BULK>
cudaError_t rows_radius(const StencilArgs& sa, const OpDesc& d, int nbatch, cudaStream_t st) {
  switch (d.R) {
    case 1: return rows_form<T, 1, PY, BULK>(sa, d, nbatch, st);
    case 2: return rows_form<T, 2, PY, BULK>(sa, d, nbatch, st);
    case 3: return rows_form<T, 3, PY, BULK>(sa, d, nbatch, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace gpw
