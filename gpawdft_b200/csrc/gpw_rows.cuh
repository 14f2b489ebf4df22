// Star stencil (apply) on whole rows: any boundary mix, element type and row
// alignment, rows of up to ROWS_NT points.
//
// The band stencils (Laplacians, gradients, kinetic + potential) of grids
// whose TY + 2R rows of one plane fit in shared memory a few times over.  A
// CTA owns TY = G PY whole rows of axis 1 and marches along axis 0.
//  * Rows of a plane are contiguous in memory, so the TY + 2R rows a tile
//    needs are one copy (three where they wrap around a periodic axis 1):
//    one cp.async.bulk of the block when rows are whole 16-byte units, else
//    element-wise cp.async over the same contiguous run -- no per-cell index
//    arithmetic either way, and no axis-2 halo at all.
//  * Threads are laid over the G x n2 columns of the tile without gaps, so a
//    row of 95 points wastes 1 of 96 lanes; each thread owns PY rows and
//    keeps 2R + 1 axis-0 sums per row in registers.
//  * The R columns past either end of a row: a periodic axis without phases
//    reads the other end of the row (an offset per thread), a zero axis and a
//    Bloch axis read a small halo block of the stage, zeros or the
//    phase-multiplied row ends, written one plane ahead.  So the inner loop
//    holds neither branches nor phases.
//  * One CTA barrier per plane; NS stages.  A stencil without terms along
//    axis 0 or 1 (a gradient) stages no halo planes or rows there.
//  * The grid is one CTA per resident slot; each takes an equal share of the
//    (tile, plane) units, so no last wave is partly empty.
// Measured: a gradient along axis 1 of 32 x 80 x 72 x 88 complex128, R = 3,
// 217 us on the fastest of the other kernels, 104 us here (5.0 TB/s, 77% of the
// copy rate).  With axis-0 terms its sums per row cost more than the cell-
// staged kernel's halo (kinetic + potential, 48 x 95^3 float64: 375 against
// 217 us).
// Terms are summed in the order of gpw_star_cells.cuh.
//
// Every mbarrier wait is bounded (GPW_ETIMEDOUT in the status word).
#pragma once
#include "gpw_star_tma.cuh"
#include "gpw_stencil.cuh"

namespace gpw {

constexpr int ROWS_NS = 4;    // stages of the ring

template <typename T, int PY>
struct RowsCfg {
  // threads per CTA, at two CTAs per SM (complex128 with 4 rows a thread
  // holds 112 registers of sums)
  static constexpr int NT = (sizeof(T) >= 16 && PY >= 4) ? 192 : 256;
};

struct RowsArgs {
  const void* in;
  void* out;
  GridView vin, vout;
  Boundary bc;
  int G, ty, h;          // thread groups, tile rows (G PY), staged rows (ty + 2 ry)
  int ry;                // axis-1 halo rows on each side: R, or 0 without axis-1 terms
  int has_z;             // axis-2 terms present
  int tiles;             // tiles along axis 1
  int nb;                // batch members
  int row_bytes;         // pitch of a staged row (the input's axis-1 stride)
  int halo_off;          // byte offset of the halo block in a stage
  int stage_bytes;
  int halo2;             // axis 2 reads the halo block (zero axis, or Bloch phases)
  int* status;
  const void* pot;
  const void* aux;
  double aux_scale;
};

// HASX: the stencil has terms along axis 0.
template <typename T, int R, int PY, bool BULK, bool HASX, bool EPI>
__global__ void __launch_bounds__(RowsCfg<T, PY>::NT, 2)
    star_rows_kernel(const RowsArgs a, const StarCoefsT<typename EltTraits<T>::S> k) {
  using S = typename EltTraits<T>::S;
  constexpr int NS = ROWS_NS, ES = (int)sizeof(T);
  constexpr int RX = HASX ? R : 0, NR = 2 * RX + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* ring = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + NS * a.stage_bytes);
  const int tid = threadIdx.x, nt = blockDim.x;
  const int n0 = a.vin.n[0], n1 = a.vin.n[1], n2 = a.vin.n[2];
  const Boundary& bc = a.bc;
  const bool per1 = bc.periodic[1] != 0;
  const bool phase = EltTraits<T>::cpx && bc.use_phase;
  const bool phase1 = phase && per1 && a.ry > 0, phase2 = phase && bc.periodic[2] && a.has_z;
  const int rb = a.row_bytes, h = a.h, ty = a.ty, ry = a.ry;
  bool timed_out = false;

  if (BULK && tid == 0) {
    for (int i = 0; i < NS; ++i) mbar_init(mbar_u32(&full[i]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  // the halo blocks of a zero axis 2 stay zero
  for (int i = tid; i < NS * ty * 2 * R; i += nt) {
    const int st = i / (ty * 2 * R), c = i - st * (ty * 2 * R);
    reinterpret_cast<T*>(ring + st * a.stage_bytes + a.halo_off)[c] = zero<T>();
  }
  __syncthreads();
  pdl_wait();

  // ---- this thread's column and rows; byte offsets from a stage's start
  const int g = tid / n2, x = tid - g * n2;
  const bool mine = g < a.G;
  const int yb = (mine ? g : 0) * PY;             // first row of the tile
  const int coff = (yb + ry) * rb + x * ES;       // its centre cell
  // axis-2 neighbours at distance q (0: below, 1: above) of the first output
  // row, and the step to the next row
  int zoff[R][2], zstep[R][2];
#pragma unroll
  for (int q = 1; q <= R; ++q)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int c = u ? x + q : x - q;
      zoff[q - 1][u] = (yb + ry) * rb + c * ES;
      zstep[q - 1][u] = rb;
      if (c < 0 || c >= n2) {
        if (!a.halo2) {  // periodic without phases
          zoff[q - 1][u] += (c < 0 ? n2 : -n2) * ES;
        } else {  // halo block: R columns below, then R above, of each tile row
          zoff[q - 1][u] = a.halo_off + (yb * 2 * R + (c < 0 ? c + R : R + c - n2)) * ES;
          zstep[q - 1][u] = 2 * R * ES;
        }
      }
    }

  // ---- units of this CTA: planes of tiles, tile-major
  const int64_t units = (int64_t)a.tiles * a.nb * n0;
  int64_t wu = (int64_t)blockIdx.x * units / gridDim.x;
  const int64_t wend = (int64_t)(blockIdx.x + 1) * units / gridDim.x;
  int gbase = 0;  // ring steps of the earlier segments
  while (wu < wend) {
    const int64_t col = wu / n0;
    const int z0 = (int)(wu - col * n0);
    const int z1 = (int)min((int64_t)n0, (int64_t)z0 + (wend - wu));
    wu += z1 - z0;
    const int b = (int)(col / a.tiles);
    const int y0 = (int)(col - (int64_t)b * a.tiles) * ty;
    const T* in = static_cast<const T*>(a.in) + (int64_t)b * a.vin.sb;
    const int pfirst = z0 - RX, nsteps = z1 - z0 + 2 * RX;
    // staged rows inside the grid (all of them where they wrap)
    const int rlo = per1 ? 0 : max(0, ry - y0), rhi = per1 ? h : min(h, n1 - y0 + ry);
    if (rlo > 0 || rhi < h) {
      // rows past a zero boundary: zeros in every stage (never copied into)
      const int w = rb / ES;
      for (int st = 0; st < NS; ++st) {
        T* s = reinterpret_cast<T*>(ring + st * a.stage_bytes);
        for (int i = tid; i < rlo * w; i += nt) s[i] = zero<T>();
        for (int i = rhi * w + tid; i < h * w; i += nt) s[i] = zero<T>();
      }
    }
    // this thread's rows inside the grid (0: none)
    const int rows = mine ? min(PY, n1 - y0 - yb) : 0;

    // the plane of step i into its stage; a plane past a zero boundary is
    // not copied (and not read)
    auto issue = [&](int i) {
      int j0, s0;
      const bool ok = wrap_axis(pfirst + i, n0, bc.periodic[0], j0, s0);
      const int slot = (gbase + i) % NS;
      unsigned char* st = ring + slot * a.stage_bytes;
      const T* pl = in + (int64_t)j0 * a.vin.s0;
      if (BULK && tid != 0) return;
      const unsigned bar = mbar_u32(&full[slot]);
      // (the last staged row without its pitch padding: the grid may end there)
      if (BULK) mbar_expect_tx(bar, ok ? (unsigned)((rhi - rlo) * rb) : 0u);
      if (ok) {
        for (int r = rlo; r < rhi;) {
          int j = (y0 - ry + r) % n1;
          j = j < 0 ? j + n1 : j;
          const int len = min(rhi - r, n1 - j);
          const T* src = pl + (int64_t)j * a.vin.s1;
          if constexpr (BULK) {
            bulk_load(smem_u32(st + r * rb), src, (unsigned)(len * rb), bar);
          } else {
            T* dst = reinterpret_cast<T*>(st + r * rb);
            const int cnt = (len - 1) * (rb / ES) + n2;
#pragma unroll 4
            for (int e = tid; e < cnt; e += nt) cp_async<ES>(dst + e, src + e, true);
          }
          r += len;
        }
      }
      if (!BULK) cp_async_commit();
    };
    // wait for the copies of step i's plane, then write its Bloch images: the
    // rows wrapped along axis 1 in place, the halo columns of axis 2
    auto land = [&](int i) {
      const int slot = (gbase + i) % NS;
      if constexpr (BULK) {
        if (!mbar_wait_bounded(mbar_u32(&full[slot]), (unsigned)(((gbase + i) / NS) & 1))) timed_out = true;
      } else {
        cp_async_wait<NS - 2>();
      }
      if constexpr (EltTraits<T>::cpx) {
        if (!(phase1 || phase2)) return;
        if (!BULK) __syncthreads();  // other threads' copies
        unsigned char* st = ring + slot * a.stage_bytes;
        if (phase1) {
          const int lw = max(0, ry - y0), uw = max(0, y0 + ty + ry - n1);
          for (int e = tid; e < (lw + uw) * n2; e += nt) {
            const int q = e / n2, c = e - q * n2;
            const int r = q < lw ? q : h - uw + (q - lw);
            T* p = reinterpret_cast<T*>(st + r * rb) + c;
            *p = phase_mul(bc.ph[1][q < lw ? 1 : 0], *p);
          }
        }
        if (phase2) {
          T* hb = reinterpret_cast<T*>(st + a.halo_off);
          for (int e = tid; e < ty * 2 * R; e += nt) {
            const int r = e / (2 * R), q = e - r * (2 * R);
            const T v = reinterpret_cast<const T*>(st + (r + ry) * rb)[q < R ? n2 - R + q : q - R];
            hb[e] = phase_mul(bc.ph[2][q < R ? 1 : 0], v);
          }
        }
        // order these writes before the copy that refills the stage
        if (BULK) asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      }
    };

    if (BULK) asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();  // the zero rows, and every read of the previous segment
#pragma unroll
    for (int i = 0; i < NS - 1; ++i) {
      if (i < nsteps) issue(i);
      else if (!BULK) cp_async_commit();
    }
    land(0);
    __syncthreads();

    T acc[PY][NR];
#pragma unroll
    for (int j = 0; j < PY; ++j)
#pragma unroll
      for (int m = 0; m < NR; ++m) acc[j][m] = zero<T>();
    T* const outp = static_cast<T*>(a.out) + (int64_t)b * a.vout.sb + (int64_t)(y0 + yb) * a.vout.s1 + x;

    for (int s = 0; s < nsteps; ++s) {
      // the stage read in step s - 1 is free: every thread has passed the
      // barrier at its end
      if (s + NS - 1 < nsteps) issue(s + NS - 1);
      else if (!BULK) cp_async_commit();
      const int p = pfirst + s;
      int j0, s0;
      const bool ok = wrap_axis(p, n0, bc.periodic[0], j0, s0);
      if (ok && rows > 0) {
        const unsigned char* st = ring + ((gbase + s) % NS) * a.stage_bytes;
        const unsigned char* cen = st + coff;
        T v[PY];
#pragma unroll
        for (int j = 0; j < PY; ++j) v[j] = *reinterpret_cast<const T*>(cen + j * rb);
        if (p >= z0 && p < z1) {
          T part[PY];
#pragma unroll
          for (int j = 0; j < PY; ++j) part[j] = scale((S)k.cc, v[j]);
          if (ry > 0) {
            T col[PY + 2 * R];
#pragma unroll
            for (int i = 0; i < PY + 2 * R; ++i)
              col[i] = (i >= R && i < PY + R) ? v[i - R] : *reinterpret_cast<const T*>(cen + (i - R) * rb);
#pragma unroll
            for (int j = 0; j < PY; ++j)
#pragma unroll
              for (int q = 1; q <= R; ++q) {
                part[j] = fmac((S)k.cy[R + q], col[j + R + q], part[j]);
                part[j] = fmac((S)k.cy[R - q], col[j + R - q], part[j]);
              }
          }
          if (a.has_z) {
#pragma unroll
            for (int j = 0; j < PY; ++j) {
              T pz = zero<T>();
#pragma unroll
              for (int q = 1; q <= R; ++q) {
                pz = fmac((S)k.cz[R + q], *reinterpret_cast<const T*>(st + zoff[q - 1][1] + j * zstep[q - 1][1]), pz);
                pz = fmac((S)k.cz[R - q], *reinterpret_cast<const T*>(st + zoff[q - 1][0] + j * zstep[q - 1][0]), pz);
              }
              part[j] = add(part[j], pz);
            }
          }
          if constexpr (EPI) {
            if (a.pot) {
              const S* pp = static_cast<const S*>(a.pot) + (int64_t)p * a.vout.s0 + (int64_t)(y0 + yb) * a.vout.s1 + x;
#pragma unroll
              for (int j = 0; j < PY; ++j)
                if (j < rows) part[j] = fmac(pp[j * a.vout.s1], v[j], part[j]);
            }
          }
#pragma unroll
          for (int j = 0; j < PY; ++j) acc[j][RX] = add(acc[j][RX], part[j]);
        } else if (EltTraits<T>::cpx && phase && s0 >= 0) {
#pragma unroll
          for (int j = 0; j < PY; ++j) v[j] = phase_mul(bc.ph[0][s0], v[j]);
        }
        if constexpr (HASX) {
          // output plane p - R + m takes this plane at offset R - m
#pragma unroll
          for (int j = 0; j < PY; ++j)
#pragma unroll
            for (int m = 0; m < NR; ++m)
              if (m != RX) acc[j][m] = fmac((S)k.cx[2 * R - m], v[j], acc[j][m]);
        }
      }
      const int o = p - RX;
      if (o >= z0) {
        T* op = outp + (int64_t)o * a.vout.s0;
#pragma unroll
        for (int j = 0; j < PY; ++j)
          if (j < rows) {
            T r = acc[j][0];
            if constexpr (EPI) {
              if (a.aux)
                r = fmac((S)a.aux_scale, static_cast<const T*>(a.aux)[op + j * a.vout.s1 - static_cast<T*>(a.out)], r);
            }
            op[j * a.vout.s1] = r;
          }
      }
#pragma unroll
      for (int j = 0; j < PY; ++j) {
#pragma unroll
        for (int m = 0; m < NR - 1; ++m) acc[j][m] = acc[j][m + 1];
        acc[j][NR - 1] = zero<T>();
      }
      if (s + 1 < nsteps) land(s + 1);
      __syncthreads();
    }
    gbase += nsteps;
  }
  pdl_trigger();
  if (!BULK) cp_async_wait<0>();
  if (timed_out && a.status) atomicExch(a.status, GPW_ETIMEDOUT);
}

}  // namespace gpw
