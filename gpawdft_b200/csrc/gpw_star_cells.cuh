// Star stencil staged cell by cell: any boundary mix, element type, pitch and
// alignment, one register-blocked march along axis 0.
//
//  * A CTA owns a TZ x TY tile (axis 2 x axis 1) and stages each plane of it,
//    with its halo, by cp.async: a thread's cells sit at fixed places of the
//    box, so their in-plane source offset, validity and wrap sides are
//    computed once and a plane load is one cp.async per cell (16-byte cells
//    where rows are whole 16-byte units, else one element each).  Cells past
//    a zero boundary are zeroed once, periodic ones have wrapped sources, and
//    Bloch phases are a fix-up of the thread's own wrapped cells.
//  * A thread owns 16 bytes of adjacent axis-2 scalars (1 complex128, 2
//    complex64 or float64, 4 float32 elements) x PY (1 or 2) rows and reads shared
//    memory in 16-byte vectors at compile-time offsets.  Complex data is the
//    scalar stencil with axis-2 offsets doubled.
//  * One CTA barrier per plane: the load that refills a stage is issued after
//    the barrier that follows the stage's last read.  Potential, aux and rho
//    values are fetched a plane's computation ahead of their use.
//  * An arriving plane adds its in-plane sum and its axis-0 terms to 2R + 1
//    running sums; an output is complete R planes after its centre.  (The
//    sums rotate by register moves: renaming them, the loop unrolled 2R + 1
//    times, measured 9% slower for float64 and 4% faster for complex128.)
// Measured against the kernel it replaced (one element a cell, its address
// recomputed per plane, two barriers a plane), applies with a potential, R = 3:
// 48 x 95^3 float64 238 -> 216 us, 48 x 96^3 complex128 549 -> 536 us, 64 x 84 x
// 90 x 108 complex64 537 -> 423 us (3.0, 2.5 and 2.0 TB/s of compulsory bytes).
// What bounds it: latency, at 14 - 15 warps per SM (128 registers) that wait for
// shared memory and for their own arithmetic.  Of their rates complex128 uses
// 40% of shared memory's, 42% of the issue slots, 24% of float64's, complex64 44%
// and 50%; float64 on odd rows 56% and 45%, and 83% of the L1 with its one
// cp.async per element.
// Each output sums its terms in one fixed order (axis 0 below, centre and
// axis 1 plus axis 2, axis 0 above), the order of gpw_rows.cuh and
// gpw_star_tma.cuh.
#pragma once
#include "gpw_common.cuh"
#include "gpw_reduce.cuh"
#include "gpw_star_tma.cuh"
#include "gpw_stencil.cuh"

namespace gpw {

// TZ: tile width in elements; CELLB: bytes per staged cell; PY: rows a thread.
template <typename T, int R, int MODE, int TZ_, int CELLB, int PY_ = 2>
struct CellsCfg {
  using S = typename EltTraits<T>::S;
  static constexpr int ES = (int)sizeof(T), CS = EltTraits<T>::cpx ? 2 : 1;
  static constexpr int VEC = 16 / (int)sizeof(S);         // scalars per thread
  static constexpr int EPT = VEC / CS;                    // elements per thread
  static constexpr int TZ = TZ_, NTX = TZ / EPT, PY = PY_;
  static constexpr int NTY = 256 / NTX, NT = NTX * NTY, TY = NTY * PY;
  static constexpr int AL = 16 / ES;                      // elements per 16 bytes
  static constexpr int XL = (R + AL - 1) / AL * AL;       // halo columns, whole vectors
  static constexpr int W = TZ + 2 * XL, H = TY + 2 * R;   // staged box
  static constexpr int CPE = CELLB / ES, WC = W / CPE;    // elements per cell, cells per row
  static constexpr int NC = H * WC, NLD = (NC + NT - 1) / NT;
  static constexpr int JR = MODE == MODE_JACOBI ? R : 0;  // planes kept behind (the Jacobi centre)
  static constexpr int D = 3, NS = D + 1 + JR;            // planes in flight, stages
  static constexpr int STAGE = (H * W * ES + 127) / 128 * 128;
  static constexpr size_t smem = (size_t)NS * STAGE;
  // CTAs per SM the registers must allow
  static constexpr int MINB = R == 1 && PY == 1 ? (sizeof(S) == 4 ? 3 : 4) : 2;
};

// EPI: an apply with a potential (1: a.pot) or an aux term (2: a.aux, and
// a.pot where set); the term is fetched ahead, in 2 the potential is not.
// SYM: the coefficients at +q and -q are equal on every axis (a Laplacian):
// 3R + 1 coefficients stay in uniform registers, where 6R + 1 were loaded again
// on every plane.
// SLOPE: +-1 for a star and the diagonal (q, SLOPE q, 0) of axes 0 and 1,
// whose terms scatter with the axis-0 ones from the column of rows a thread
// holds anyway.  The centre, the largest term, comes after the in-plane
// ones, so that fewer partial sums of its size are rounded (60^2 x 84 normal
// values, R = 3: error against extended precision 1.3e-16; 1.8e-16 with the
// centre first, 2.3e-16 for the general kernel's order).
template <typename T, int R, int MODE, int TZ, int CELLB, int EPI, bool SYM, int SLOPE, int PY = 2>
__global__ void __launch_bounds__(CellsCfg<T, R, MODE, TZ, CELLB, PY>::NT, (CellsCfg<T, R, MODE, TZ, CELLB, PY>::MINB))
    star_cells_kernel(const StencilArgs a, const StarCoefsT<typename EltTraits<T>::S> k) {
  using C = CellsCfg<T, R, MODE, TZ, CELLB, PY>;
  using S = typename EltTraits<T>::S;
  constexpr int VEC = C::VEC, CS = C::CS, EPT = C::EPT, NR = 2 * R + 1, NS = C::NS, NT = C::NT;
  constexpr int WS = C::W * CS, XS = C::XL * CS;  // row pitch and halo in scalars
  using P = Pack<S, VEC>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[32];
  pdl_wait();

  const int b = blockIdx.z / a.nchunk, chunk = blockIdx.z - b * a.nchunk;
  if (a.active && !a.active[b]) return;
  const int x0 = blockIdx.x * TZ, y0 = blockIdx.y * C::TY;
  const int n0 = a.vout.n[0], n1 = a.vout.n[1], n2 = a.vout.n[2];
  const int z0 = (int)((int64_t)chunk * n0 / a.nchunk), z1 = (int)((int64_t)(chunk + 1) * n0 / a.nchunk);
  const T* in = static_cast<const T*>(a.in) + (int64_t)b * a.vin.sb;
  const int tid = threadIdx.x, tx = tid % C::NTX, ty = tid / C::NTX;
  const Boundary& bc = a.bc;
  const bool phase = EltTraits<T>::cpx && bc.use_phase;
  double sumsq = 0.0;

  // ---- this thread's cells: tid + k NT of the box.  Cells past a zero
  // boundary are never copied: they are zeroed once in every stage.
  unsigned off[C::NLD];              // bytes from the plane's start (cells_plane_ok)
  unsigned valid = 0, wrapped = 0;   // bit k: inside or an image; an image along axis 1 or 2
  unsigned char side[C::NLD];        // sides + 1: bits 0-1 axis 1, bits 2-3 axis 2
#pragma unroll
  for (int c = 0; c < C::NLD; ++c) {
    const int idx = tid + c * NT;
    const int r = idx / C::WC, q = (idx - r * C::WC) * C::CPE;
    int j1 = 0, j2 = 0, s1 = -1, s2 = -1;
    const bool ok = idx < C::NC && wrap_axis(y0 - R + r, n1, bc.periodic[1], j1, s1) &&
                    wrap_axis(x0 - C::XL + q, n2, bc.periodic[2], j2, s2);
    off[c] = ok ? (unsigned)((int64_t)j1 * a.vin.s1 + j2) * (unsigned)C::ES : 0u;
    if (ok) valid |= 1u << c;
    if (ok && (s1 >= 0 || s2 >= 0)) wrapped |= 1u << c;
    side[c] = (unsigned char)((s1 + 1) | ((s2 + 1) << 2));
    if (!ok && idx < C::NC)
      for (int st = 0; st < NS; ++st)
        for (int e = 0; e < CELLB / 4; ++e)
          reinterpret_cast<float*>(smem_raw + st * C::STAGE + idx * CELLB)[e] = 0.f;
  }
  const unsigned sbase = smem_u32(smem_raw) + tid * CELLB;
  // plane p into stage `slot`; a plane past a zero boundary is zeros
  auto load = [&](unsigned slot, int p) {
    int j0, s0;
    if (!wrap_axis(p, n0, bc.periodic[0], j0, s0)) {
#pragma unroll
      for (int c = 0; c < C::NLD; ++c)
        if ((valid >> c) & 1u)
          for (int e = 0; e < CELLB / 4; ++e)
            reinterpret_cast<float*>(smem_raw + slot * C::STAGE + (tid + c * NT) * CELLB)[e] = 0.f;
      return;
    }
    const char* base = reinterpret_cast<const char*>(in + (int64_t)j0 * a.vin.s0);
    const unsigned st = sbase + slot * C::STAGE;
#pragma unroll
    for (int c = 0; c < C::NLD; ++c)
      if ((valid >> c) & 1u) {
        if constexpr (CELLB == 16)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(st + c * NT * CELLB), "l"(base + off[c]));
        else
          asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(st + c * NT * CELLB), "l"(base + off[c]),
                       "n"(CELLB));
      }
  };
  // Bloch phases of this thread's periodic images, axis by axis as the
  // reference's chained halo copies apply them
  auto fix = [&](unsigned slot, int p) {
    if constexpr (EltTraits<T>::cpx) {
      int j0, s0;
      if (!wrap_axis(p, n0, bc.periodic[0], j0, s0)) return;
      const unsigned todo = s0 < 0 ? wrapped : valid;
      if (!todo) return;
      unsigned char* st = smem_raw + slot * C::STAGE + tid * CELLB;
#pragma unroll
      for (int c = 0; c < C::NLD; ++c) {
        if (!((todo >> c) & 1u)) continue;
        const int s1 = (side[c] & 3) - 1, s2 = ((side[c] >> 2) & 3) - 1;
#pragma unroll
        for (int e = 0; e < C::CPE; ++e) {
          T* cell = reinterpret_cast<T*>(st + c * NT * CELLB) + e;
          T val = *cell;
          if (s0 >= 0) val = phase_mul(bc.ph[0][s0], val);
          if (s1 >= 0) val = phase_mul(bc.ph[1][s1], val);
          if (s2 >= 0) val = phase_mul(bc.ph[2][s2], val);
          *cell = val;
        }
      }
    }
  };

  // ---- this thread's outputs
  const int x = x0 + EPT * tx, yb = ty * PY, y = y0 + yb;
  const int nx = min(EPT, n2 - x);                 // elements inside the grid (<= 0: none)
  const int rows = nx > 0 ? min(PY, n1 - y) : 0;   // rows inside the grid
  // VEC scalars of global memory at an element of a view: one 16-byte access
  // where every row of the view starts on one
  auto aligned = [](const void* p, const GridView& v) {
    return EPT == 1 || (((reinterpret_cast<uintptr_t>(p) | (uintptr_t)(v.s1 * C::ES) | (uintptr_t)(v.s0 * C::ES) |
                          (uintptr_t)(v.sb * C::ES)) & 15u) == 0);
  };
  const bool full = nx == EPT;
  const bool vst = full && aligned(a.out, a.vout);
  const bool vld = full && (MODE == MODE_APPLY ? aligned(a.aux, a.vout) : aligned(a.rho, a.vrho));
  auto gload = [&](const T* q) {
    const S* p = reinterpret_cast<const S*>(q);
    if (vld) return ldv<S, VEC>(p);
    P r;
#pragma unroll
    for (int e = 0; e < VEC; ++e) r.v[e] = e / CS < nx ? p[e] : S(0);
    return r;
  };
  // this thread's element of plane 0 (rho and aux: the epilogue's operand)
  const int64_t oel = (int64_t)y * a.vout.s1 + x;
  T* const out0 = a.out ? static_cast<T*>(a.out) + (int64_t)b * a.vout.sb + oel : nullptr;
  const T* ep0 = nullptr;
  int64_t eps0 = 0, eps1 = 0;
  if constexpr (MODE != MODE_APPLY) {
    ep0 = static_cast<const T*>(a.rho) + (int64_t)b * a.vrho.sb + (int64_t)y * a.vrho.s1 + x;
    eps0 = a.vrho.s0;
    eps1 = a.vrho.s1;
  } else if constexpr (EPI == 2) {
    if (a.aux) ep0 = static_cast<const T*>(a.aux) + (int64_t)b * a.vout.sb + oel;
    eps0 = a.vout.s0;
    eps1 = a.vout.s1;
  }
  const S* const pot0 = EPI != 0 && a.pot ? static_cast<const S*>(a.pot) + oel : nullptr;
  P acc[PY][NR];
#pragma unroll
  for (int j = 0; j < PY; ++j)
#pragma unroll
    for (int m = 0; m < NR; ++m)
#pragma unroll
      for (int e = 0; e < VEC; ++e) acc[j][m].v[e] = S(0);

  if (z0 < z1) {
    const int pfirst = z0 - R, nsteps = z1 - z0 + 2 * R;
#pragma unroll
    for (int s = 0; s < C::D; ++s) {
      if (s < nsteps) load(s, pfirst + s);
      cp_async_commit();
    }
    unsigned slot = 0, lslot = C::D % NS;  // the stage read, the stage refilled
    {
      for (int s = 0; s < nsteps; ++s) {
        const int p = pfirst + s, o = p - R;
        // this step's epilogue operands, fetched ahead of the wait
        P ep[PY];       // rho of output o, or (APPLY) aux of output o
        S pv[PY][EPT];  // the potential of plane p
        if constexpr (MODE != MODE_APPLY || EPI == 2) {
          if (ep0 && o >= z0) {
            const T* q = ep0 + (int64_t)o * eps0;
#pragma unroll
            for (int j = 0; j < PY; ++j)
              if (j < rows) ep[j] = gload(q + j * eps1);
          }
        }
        auto gpot = [&](int j, int e) {
          return j < rows && e < nx ? pot0[(int64_t)p * a.vout.s0 + j * a.vout.s1 + e] : S(0);
        };
        // (a halo plane has no potential of its own, and may lie outside the array)
        if constexpr (EPI == 1) {
          if (p >= z0 && p < z1) {
#pragma unroll
            for (int j = 0; j < PY; ++j)
#pragma unroll
              for (int e = 0; e < EPT; ++e) pv[j][e] = gpot(j, e);
          }
        }
        cp_async_wait<C::D - 1>();
        if (phase) fix(slot, p);
        __syncthreads();  // the plane is complete; every read of the stage refilled next is done
        if (s + C::D < nsteps) load(lslot, p + C::D);
        cp_async_commit();
        lslot = lslot + 1 == NS ? 0 : lslot + 1;

        const S* sl = reinterpret_cast<const S*>(smem_raw + slot * C::STAGE);
        const int cell = yb * WS + XS + VEC * tx;
        {
          P col[PY + 2 * R];
#pragma unroll
          for (int i = 0; i < PY + 2 * R; ++i) col[i] = ldv<S, VEC>(sl + cell + i * WS);
#pragma unroll
          for (int j = 0; j < PY; ++j) {
            const P c = col[j + R];
            {
              const S* row = sl + cell + (j + R) * WS;
              S nb[2 * XS + VEC];
#pragma unroll
              for (int q = 0; q < XS; q += VEC) {
                const P lo = ldv<S, VEC>(row - XS + q);
                const P hi = ldv<S, VEC>(row + VEC + q);
#pragma unroll
                for (int e = 0; e < VEC; ++e) {
                  nb[q + e] = lo.v[e];
                  nb[XS + VEC + q + e] = hi.v[e];
                }
              }
#pragma unroll
              for (int e = 0; e < VEC; ++e) nb[XS + e] = c.v[e];
              // the in-plane sum in two independent chains (centre and axis 1,
              // axis 2) joined at the end: half the dependent latency
              P part, pz;
#pragma unroll
              for (int e = 0; e < VEC; e += 2) {
                if constexpr (SLOPE != 0)
                  part.v[e] = part.v[e + 1] = S(0);
                else
                  mul_pair((MODE == MODE_JACOBI) ? S(0) : k.cc, c.v[e], c.v[e + 1], part.v[e], part.v[e + 1]);
                pz.v[e] = pz.v[e + 1] = S(0);
              }
#pragma unroll
              for (int q = 1; q <= R; ++q)
#pragma unroll
                for (int e = 0; e < VEC; e += 2) {
                  fma_pair(k.cy[R + q], col[j + R + q].v[e], col[j + R + q].v[e + 1], part.v[e], part.v[e + 1]);
                  fma_pair(k.cy[SYM ? R + q : R - q], col[j + R - q].v[e], col[j + R - q].v[e + 1], part.v[e], part.v[e + 1]);
                }
#pragma unroll
              for (int q = 1; q <= R; ++q)
#pragma unroll
                for (int e = 0; e < VEC; e += 2) {
                  constexpr int odd = CS == 1 ? 1 : 0;  // a real neighbour at odd distance is no aligned pair
                  if (odd && (q & 1)) {
#pragma unroll
                    for (int f = e; f < e + 2; ++f) {
                      pz.v[f] = fma(k.cz[R + q], nb[XS + f + q * CS], pz.v[f]);
                      pz.v[f] = fma(k.cz[SYM ? R + q : R - q], nb[XS + f - q * CS], pz.v[f]);
                    }
                  } else {
                    fma_pair(k.cz[R + q], nb[XS + e + q * CS], nb[XS + e + 1 + q * CS], pz.v[e], pz.v[e + 1]);
                    fma_pair(k.cz[SYM ? R + q : R - q], nb[XS + e - q * CS], nb[XS + e + 1 - q * CS], pz.v[e], pz.v[e + 1]);
                  }
                }
#pragma unroll
              for (int e = 0; e < VEC; e += 2) add_pair(pz.v[e], pz.v[e + 1], part.v[e], part.v[e + 1]);
              if constexpr (EPI == 1) {
#pragma unroll
                for (int e = 0; e < VEC; ++e) part.v[e] = fma(pv[j][e / CS], c.v[e], part.v[e]);
              } else if constexpr (EPI == 2) {
                if (pot0 && p >= z0 && p < z1) {
#pragma unroll
                  for (int e = 0; e < VEC; ++e) part.v[e] = fma(gpot(j, e / CS), c.v[e], part.v[e]);
                }
              }
              P& am = acc[j][R];
#pragma unroll
              for (int e = 0; e < VEC; e += 2) {
                add_pair(part.v[e], part.v[e + 1], am.v[e], am.v[e + 1]);
                if constexpr (SLOPE != 0) fma_pair(k.cc, c.v[e], c.v[e + 1], am.v[e], am.v[e + 1]);
              }
            }
            // scatter along axis 0: output plane p-R+m receives offset R-m
#pragma unroll
            for (int m = 0; m < NR; ++m)
              if (m != R) {
                P& am = acc[j][m];
#pragma unroll
                for (int e = 0; e < VEC; e += 2)
                  fma_pair(k.cx[SYM && m > R ? m : 2 * R - m], c.v[e], c.v[e + 1], am.v[e], am.v[e + 1]);
                if constexpr (SLOPE != 0) {
                  const P& d = col[j + R + SLOPE * (R - m)];
#pragma unroll
                  for (int e = 0; e < VEC; e += 2)
                    fma_pair(k.cd[SYM && m > R ? m : 2 * R - m], d.v[e], d.v[e + 1], am.v[e], am.v[e + 1]);
                }
              }
          }
        }
        // output plane o = p - R is complete
        if (o >= z0) {
          T* op = out0 + (int64_t)o * a.vout.s0;
#pragma unroll
          for (int j = 0; j < PY; ++j) {
            if (j < rows) {
              P r = acc[j][0];
              bool store = true;
              if constexpr (MODE == MODE_APPLY) {
                if (EPI == 2 && ep0) {
                  const S g = (S)a.aux_scale;
#pragma unroll
                  for (int e = 0; e < VEC; ++e) r.v[e] = fma(g, ep[j].v[e], r.v[e]);
                }
              } else if constexpr (MODE == MODE_RESIDUAL) {
                store = a.out != nullptr;
#pragma unroll
                for (int e = 0; e < VEC; ++e) {
                  r.v[e] = r.v[e] - ep[j].v[e];
                  if (e / CS < nx) sumsq += (double)r.v[e] * (double)r.v[e];
                }
              } else {
                // the centre value, R planes behind in the ring
                const S* osl = reinterpret_cast<const S*>(smem_raw + (slot >= R ? slot - R : slot + NS - R) * C::STAGE);
                const P cur = ldv<S, VEC>(osl + cell + (j + R) * WS);
                const S w = (S)a.w;
                const S wc = w / (S)a.c0;
#pragma unroll
                for (int e = 0; e < VEC; ++e) r.v[e] = (S(1) - w) * cur.v[e] + wc * (ep[j].v[e] - r.v[e]);
              }
              if (store) {
                S* q = reinterpret_cast<S*>(op + j * a.vout.s1);
                if (vst) {
                  stv<S, VEC>(q, r);
                } else {
#pragma unroll
                  for (int e = 0; e < VEC; ++e)
                    if (e / CS < nx) q[e] = r.v[e];
                }
              }
            }
          }
        }
#pragma unroll
        for (int j = 0; j < PY; ++j) {
#pragma unroll
          for (int m = 0; m < NR - 1; ++m) acc[j][m] = acc[j][m + 1];
#pragma unroll
          for (int e = 0; e < VEC; ++e) acc[j][NR - 1].v[e] = S(0);
        }
        slot = slot + 1 == NS ? 0 : slot + 1;
      }
    }
  }
  pdl_trigger();
  cp_async_wait<0>();
  if constexpr (MODE == MODE_RESIDUAL) {
    if (!a.gsum.partial) return;  // residual without its norm
    double tot = block_sum(sumsq, red);
    const int blk = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * chunk);
    grid_sum_finish(a.gsum, b, blk, a.nblk_seg, tot, red);
  }
}

}  // namespace gpw
