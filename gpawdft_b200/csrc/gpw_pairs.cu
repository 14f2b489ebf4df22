// The matrix of band-pair integrals, out[x][y] = sum_k conj(a_x[k]) b_y[k]
// (gpaw/grid_descriptor.py:263-319, the gemm with transa 'c' of :306): a
// contraction over the grid points with a short result, so K (the points) is
// split over the chip and the per-part results are summed in a fixed order.
//
// pair_mma_kernel: a warp owns MB x NB blocks of 8 x 8 pairs and a range of
// points, and accumulates them with float64 mma.sync m8n8k4 (there is no
// float64 tcgen05 form).  A fragment is one element per lane -- row lane / 4,
// point lane % 4 -- so lanes load their elements straight from global memory:
// 8 rows of four adjacent points a load, two steps in registers ahead of the
// one being multiplied, no shared memory.  Complex pairs take four real
// products into two accumulators.  All types are accumulated in float64.
// The warps of a CTA take adjacent tiles of the same points, so their common
// rows meet in L1.
//
// What bounds it: 48 x 48 complex128 pairs of 56^3 points (3.2 GFLOP on 270 MB)
// take 115 us, 28 TFLOP/s or about three quarters of the nominal float64 tensor
// rate, its eight warps per SM waiting for that pipe and, less, for operands
// (4.8 and 3.1 stall cycles an instruction in dependent and full pipes, 2.8 in
// loads); with the sum over parts and the caller's read of the result 164 - 177
// us.  One reduction per pair, which read every vector 48 times, took 1433 us.
#include <algorithm>

#include "gpw_internal.h"

namespace gpw {

constexpr int PM_WARPS = 4;   // warps per CTA
constexpr int PM_U = 2;       // k-steps (of 4 points) per register stage

struct PairArgs {
  const void *x, *y;
  int nx, ny;
  int64_t n;         // points per vector
  int tx, ty;        // warp tiles along x and y
  int kparts;        // ranges the points are split into
  int kw;            // warps of a CTA that share a tile (on kw ranges); 4 / kw tiles per CTA
  double* partial;   // [kparts][nx * ny * ncomp]
};

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

template <typename T> struct PairElt;
template <> struct PairElt<double> {
  static constexpr int NC = 1;
  static __device__ __forceinline__ void get(double v, double (&o)[1]) { o[0] = v; }
};
template <> struct PairElt<float> {
  static constexpr int NC = 1;
  static __device__ __forceinline__ void get(float v, double (&o)[1]) { o[0] = (double)v; }
};
template <> struct PairElt<double2> {
  static constexpr int NC = 2;
  static __device__ __forceinline__ void get(double2 v, double (&o)[2]) {
    o[0] = v.x;
    o[1] = v.y;
  }
};
template <> struct PairElt<float2> {
  static constexpr int NC = 2;
  static __device__ __forceinline__ void get(float2 v, double (&o)[2]) {
    o[0] = (double)v.x;
    o[1] = (double)v.y;
  }
};

template <typename T, int MB, int NB>
__global__ void __launch_bounds__(32 * PM_WARPS, 2) pair_mma_kernel(const PairArgs a) {
  using E = PairElt<T>;
  constexpr int NC = E::NC;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int tile = blockIdx.y * (PM_WARPS / a.kw) + w / a.kw;
  const int part = blockIdx.x * a.kw + w % a.kw;
  if (tile >= a.tx * a.ty || part >= a.kparts) return;
  const int x0 = (tile / a.ty) * 8 * MB, y0 = (tile % a.ty) * 8 * NB;
  // ranges in whole steps of 4 points
  const int64_t steps = (a.n + 3) / 4;
  const int64_t s0 = steps * part / a.kparts, s1 = steps * (part + 1) / a.kparts;
  const int row = lane >> 2, kl = lane & 3;
  const T* xp[MB];
  const T* yp[NB];
  bool xok[MB], yok[NB];
#pragma unroll
  for (int i = 0; i < MB; ++i) {
    xok[i] = x0 + 8 * i + row < a.nx;
    xp[i] = static_cast<const T*>(a.x) + (int64_t)(xok[i] ? x0 + 8 * i + row : 0) * a.n + kl;
  }
#pragma unroll
  for (int j = 0; j < NB; ++j) {
    yok[j] = y0 + 8 * j + row < a.ny;
    yp[j] = static_cast<const T*>(a.y) + (int64_t)(yok[j] ? y0 + 8 * j + row : 0) * a.n + kl;
  }
  double acc[MB][NB][NC][2];
#pragma unroll
  for (int i = 0; i < MB; ++i)
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
      for (int c = 0; c < NC; ++c) acc[i][j][c][0] = acc[i][j][c][1] = 0.0;

  T fx[2][PM_U][MB], fy[2][PM_U][NB];
  auto fetch = [&](int buf, int64_t s) {
#pragma unroll
    for (int u = 0; u < PM_U; ++u) {
      const int64_t k = 4 * (s + u);
      const bool ok = s + u < s1 && k + kl < a.n;
#pragma unroll
      for (int i = 0; i < MB; ++i) fx[buf][u][i] = ok && xok[i] ? __ldg(xp[i] + k) : zero<T>();
#pragma unroll
      for (int j = 0; j < NB; ++j) fy[buf][u][j] = ok && yok[j] ? __ldg(yp[j] + k) : zero<T>();
    }
  };
  auto multiply = [&](int buf) {
#pragma unroll
    for (int u = 0; u < PM_U; ++u) {
      double bx[NB][NC];
#pragma unroll
      for (int j = 0; j < NB; ++j) E::get(fy[buf][u][j], bx[j]);
#pragma unroll
      for (int i = 0; i < MB; ++i) {
        double ax[NC];
        E::get(fx[buf][u][i], ax);
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          dmma(acc[i][j][0], ax[0], bx[j][0]);
          if constexpr (NC == 2) {
            dmma(acc[i][j][0], ax[1], bx[j][1]);
            dmma(acc[i][j][1], ax[0], bx[j][1]);
            dmma(acc[i][j][1], -ax[1], bx[j][0]);
          }
        }
      }
    }
  };
  fetch(0, s0);
  for (int64_t s = s0; s < s1; s += 2 * PM_U) {
    fetch(1, s + PM_U);
    multiply(0);
    fetch(0, s + 2 * PM_U);
    multiply(1);
  }
  // accumulator element e of a lane: pair (row, 2 (lane % 4) + e) of the block
  double* p = a.partial + (int64_t)part * a.nx * a.ny * NC;
#pragma unroll
  for (int i = 0; i < MB; ++i)
#pragma unroll
    for (int j = 0; j < NB; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int px = x0 + 8 * i + row, py = y0 + 8 * j + 2 * kl + e;
        if (px < a.nx && py < a.ny) {
#pragma unroll
          for (int c = 0; c < NC; ++c) p[((int64_t)px * a.ny + py) * NC + c] = acc[i][j][c][e];
        }
      }
}

// out[v] = sum over the parts of partial[part][v], in order within 32
// groups of parts and then over the groups, carrying each addition's rounding
// error along (Knuth's two-sum): a plain sum of the ~300 parts was the largest
// error of the result.
struct PairSum {
  double s, c;
  __device__ __forceinline__ void add(double v) {
    const double t = __dadd_rn(s, v), bb = __dsub_rn(t, s);
    c = __dadd_rn(c, __dadd_rn(__dsub_rn(s, __dsub_rn(t, bb)), __dsub_rn(v, bb)));
    s = t;
  }
};

constexpr int PS_G = 32;  // groups of parts: a warp each (8 left the loads in a chain, 20 us)

__global__ void __launch_bounds__(32 * PS_G) pair_sum_kernel(int nv, int kparts, const double* __restrict__ partial,
                                                       double* __restrict__ out) {
  __shared__ PairSum red[PS_G][32];
  const int tx = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int v = blockIdx.x * 32 + tx;
  const int p0 = kparts * g / PS_G, p1 = kparts * (g + 1) / PS_G;
  PairSum s{0.0, 0.0};
  if (v < nv) {
#pragma unroll 8
    for (int p = p0; p < p1; ++p) s.add(__ldcg(partial + (int64_t)p * nv + v));
  }
  red[g][tx] = s;
  __syncthreads();
  if (g == 0 && v < nv) {
#pragma unroll
    for (int i = 1; i < PS_G; ++i) {
      s.add(red[i][tx].s);
      s.c += red[i][tx].c;
    }
    // (an infinite part leaves no error term)
    out[v] = isfinite(s.c) ? s.s + s.c : s.s;
  }
}

namespace {

// Blocks of 8 per warp tile (1 - 3) for nb blocks: the least padding, the
// widest of equals.
int pair_tile(int nb) {
  int best = 1, cost = 1 << 30;
  for (int t = 3; t >= 1; --t) {
    const int c = (nb + t - 1) / t * t;
    if (c < cost) {
      cost = c;
      best = t;
    }
  }
  return best;
}

struct PairPlan {
  int mb, nb, tx, ty, kw, kparts;
};

// Parts: about 8 warps per SM over all tiles, no range shorter than 64
// points.
PairPlan pair_plan(int64_t nx, int64_t ny, int64_t n) {
  PairPlan p;
  const int bx = (int)((nx + 7) / 8), by = (int)((ny + 7) / 8);
  p.mb = pair_tile(bx);
  p.nb = pair_tile(by);
  p.tx = (bx + p.mb - 1) / p.mb;
  p.ty = (by + p.nb - 1) / p.nb;
  const int64_t tiles = (int64_t)p.tx * p.ty;
  p.kw = tiles >= 4 ? 1 : (tiles >= 2 ? 2 : 4);
  const int64_t want = std::max<int64_t>(1, 8LL * num_sms() / tiles);
  p.kparts = (int)std::max<int64_t>(1, std::min<int64_t>(want, n / 64));
  return p;
}

template <typename T, int MB>
cudaError_t pair_launch_n(const PairPlan& p, const PairArgs& a, cudaStream_t st) {
  const int tpc = PM_WARPS / p.kw;
  const dim3 grid((p.kparts + p.kw - 1) / p.kw, (p.tx * p.ty + tpc - 1) / tpc);
  switch (p.nb) {
    case 1: pair_mma_kernel<T, MB, 1><<<grid, 32 * PM_WARPS, 0, st>>>(a); break;
    case 2: pair_mma_kernel<T, MB, 2><<<grid, 32 * PM_WARPS, 0, st>>>(a); break;
    default: pair_mma_kernel<T, MB, 3><<<grid, 32 * PM_WARPS, 0, st>>>(a); break;
  }
  return cudaGetLastError();
}

template <typename T>
cudaError_t pair_launch(const PairPlan& p, const PairArgs& a, cudaStream_t st) {
  switch (p.mb) {
    case 1: return pair_launch_n<T, 1>(p, a, st);
    case 2: return pair_launch_n<T, 2>(p, a, st);
    default: return pair_launch_n<T, 3>(p, a, st);
  }
}

}  // namespace

size_t pair_scratch_bytes(int dtype, int64_t nx, int64_t ny, int64_t n) {
  return (size_t)pair_plan(nx, ny, n).kparts * nx * ny * (is_complex(dtype) ? 2 : 1) * sizeof(double);
}

cudaError_t launch_pairs(int dtype, int64_t nx, int64_t ny, int64_t n, const void* x, const void* y, double* partial,
                         double* out, cudaStream_t st) {
  const PairPlan p = pair_plan(nx, ny, n);
  PairArgs a{x, y, (int)nx, (int)ny, n, p.tx, p.ty, p.kparts, p.kw, partial};
  cudaError_t e;
  switch (dtype) {
    case GPW_F64: e = pair_launch<double>(p, a, st); break;
    case GPW_F32: e = pair_launch<float>(p, a, st); break;
    case GPW_C128: e = pair_launch<double2>(p, a, st); break;
    case GPW_C64: e = pair_launch<float2>(p, a, st); break;
    default: return cudaErrorInvalidValue;
  }
  if (e != cudaSuccess) return e;
  const int nv = (int)(nx * ny * (is_complex(dtype) ? 2 : 1));
  pair_sum_kernel<<<(nv + 31) / 32, 32 * PS_G, 0, st>>>(nv, p.kparts, partial, out);
  return cudaGetLastError();
}

}  // namespace gpw
