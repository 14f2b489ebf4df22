// Star stencil for grids that stay in L2: one thread per output column of a
// short run of axis-0 planes, every neighbour read straight from global
// memory (L1 / L2 hits), no staging.
//
// The marching kernels (gpw_star_cells.cuh, gpw_star_tma.cuh) read each value
// from memory once, which is what bounds large grids; on a small grid their
// march -- a chunk of planes, each a dependent load, wait and barrier -- is a
// serial chain that takes ~10 us whatever the grid, while the grid's 1 + 6R
// reads per point are L1 traffic a few SMs deep.  A launch here is as long as
// one or two memory latencies (~4 us; the V-cycles of a periodic 80^3 float64
// solve, 28 launches each: 296 -> 146 us with this kernel and the other small-
// grid ones).  Taken for the grids direct_bytes (gpw_launch.cu) names.
//
// An output's in-plane terms are one chain (centre, axis 1, axis 2), as
// c/bmgs/fd.c sums a plane; latency is hidden by the other threads.
#pragma once
#include "gpw_common.cuh"
#include "gpw_reduce.cuh"
#include "gpw_stencil.cuh"

namespace gpw {

constexpr int DIRECT_NT = 256;

template <typename T, int R, int MODE>
__global__ void __launch_bounds__(DIRECT_NT, (!EltTraits<T>::cpx && R <= 3 ? 4 : 1)) star_direct_kernel(const StencilArgs a,
                                                                const StarCoefsT<typename EltTraits<T>::S> k) {
  using S = typename EltTraits<T>::S;
  __shared__ double red[32];
  pdl_wait();
  const int b = blockIdx.z;
  if (a.active && !a.active[b]) return;
  const int n0 = a.vin.n[0], n1 = a.vin.n[1], n2 = a.vin.n[2];
  const int z0 = blockIdx.y * a.zchunk, z1 = min(n0, z0 + a.zchunk);
  const int idx = blockIdx.x * DIRECT_NT + threadIdx.x;
  const bool inside = idx < n1 * n2;
  double sumsq = 0.0;
  if (inside) {
    const int y = idx / n2, x = idx - y * n2;
    const bool phase = EltTraits<T>::cpx && a.bc.use_phase;
    // element offsets of the in-plane neighbours at distance q (below, above),
    // from the plane's start; ok / sd: inside or a periodic image, its side
    int ox[R][2], oy[R][2];
    unsigned okx = 0, oky = 0, imx = 0, imy = 0;  // bit 2 (q - 1) + above
#pragma unroll
    for (int q = 1; q <= R; ++q)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        int j, s;
        const unsigned bit = 1u << (2 * (q - 1) + u);
        if (wrap_axis(u ? x + q : x - q, n2, a.bc.periodic[2], j, s)) okx |= bit;
        if (s >= 0) imx |= bit;
        ox[q - 1][u] = y * (int)a.vin.s1 + j;
        if (wrap_axis(u ? y + q : y - q, n1, a.bc.periodic[1], j, s)) oky |= bit;
        if (s >= 0) imy |= bit;
        oy[q - 1][u] = j * (int)a.vin.s1 + x;
      }
    const T* in = static_cast<const T*>(a.in) + (int64_t)b * a.vin.sb;
    const int oc = y * (int)a.vin.s1 + x;
    // a neighbour: zero outside, times the phase of a periodic image
    auto image = [&](const T* p, bool ok, bool im, int axis, int u) {
      T v = ok ? *p : zero<T>();
      if (phase && im) v = phase_mul(a.bc.ph[axis][u ? 0 : 1], v);
      return v;
    };
    for (int o = z0; o < z1; ++o) {
      const T* pl = in + (int64_t)o * a.vin.s0;
      T zv[R][2];
#pragma unroll
      for (int q = 1; q <= R; ++q)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          int j, s;
          const bool ok = wrap_axis(u ? o + q : o - q, n0, a.bc.periodic[0], j, s);
          zv[q - 1][u] = image(in + (int64_t)j * a.vin.s0 + oc, ok, s >= 0, 0, u);
        }
      const T v = pl[oc];
      T part = scale((MODE == MODE_JACOBI) ? S(0) : (S)k.cc, v);
#pragma unroll
      for (int q = 1; q <= R; ++q) {
        const unsigned bd = 2 * (q - 1), bu = bd + 1;
        part = fmac((S)k.cy[R + q], image(pl + oy[q - 1][1], (oky >> bu) & 1u, (imy >> bu) & 1u, 1, 1), part);
        part = fmac((S)k.cy[R - q], image(pl + oy[q - 1][0], (oky >> bd) & 1u, (imy >> bd) & 1u, 1, 0), part);
      }
#pragma unroll
      for (int q = 1; q <= R; ++q) {
        const unsigned bd = 2 * (q - 1), bu = bd + 1;
        part = fmac((S)k.cz[R + q], image(pl + ox[q - 1][1], (okx >> bu) & 1u, (imx >> bu) & 1u, 2, 1), part);
        part = fmac((S)k.cz[R - q], image(pl + ox[q - 1][0], (okx >> bd) & 1u, (imx >> bd) & 1u, 2, 0), part);
      }
      if constexpr (MODE == MODE_APPLY) {
        if (a.pot)
          part = fmac(static_cast<const S*>(a.pot)[(int64_t)o * a.vout.s0 + (int64_t)y * a.vout.s1 + x], v, part);
      }
      T acc = zero<T>();
#pragma unroll
      for (int q = R; q >= 1; --q) acc = fmac((S)k.cx[R - q], zv[q - 1][0], acc);
      acc = add(acc, part);
#pragma unroll
      for (int q = 1; q <= R; ++q) acc = fmac((S)k.cx[R + q], zv[q - 1][1], acc);
      const int64_t oi = (int64_t)b * a.vout.sb + (int64_t)o * a.vout.s0 + (int64_t)y * a.vout.s1 + x;
      if constexpr (MODE == MODE_APPLY) {
        if (a.aux) acc = fmac((S)a.aux_scale, static_cast<const T*>(a.aux)[oi], acc);
        static_cast<T*>(a.out)[oi] = acc;
      } else {
        const T rho = static_cast<const T*>(a.rho)[(int64_t)b * a.vrho.sb + (int64_t)o * a.vrho.s0 +
                                                   (int64_t)y * a.vrho.s1 + x];
        if constexpr (MODE == MODE_RESIDUAL) {
          const T r = sub(acc, rho);
          if (a.out) static_cast<T*>(a.out)[oi] = r;
          sumsq += norm2(r);
        } else if constexpr (!EltTraits<T>::cpx) {
          const S w = (S)a.w;
          const S wc = w / (S)a.c0;
          static_cast<T*>(a.out)[oi] = (S(1) - w) * v + wc * (rho - acc);
        }
      }
    }
  }
  pdl_trigger();
  if constexpr (MODE == MODE_RESIDUAL) {
    if (!a.gsum.partial) return;  // residual without its norm
    const double tot = block_sum(sumsq, red);
    grid_sum_finish(a.gsum, b, blockIdx.x + gridDim.x * blockIdx.y, a.nblk_seg, tot, red);
  }
}

}  // namespace gpw
