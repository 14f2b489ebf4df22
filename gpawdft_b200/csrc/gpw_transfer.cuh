// Restriction and interpolation between a grid and its 2x coarser grid.
//
// Reference: c/transformers.c:54-123 fills a padded copy (c/bc.c, cfd = 0, so
// halo edges and corners are filled too) and then runs three separable 1D
// passes -- axis 2, then axis 1, then axis 0 -- each writing a transposed
// temporary (c/bmgs/restrict.c:137-154, c/bmgs/interpolate.c:141-168).
//
// Here one kernel does all three passes without temporaries in HBM: a CTA owns
// an (axis-1, axis-2) output tile and marches along axis 0.  Each input plane
// of the tile (with halo) is staged in shared memory by cp.async; the axis-2
// pass and the axis-1 pass run in shared memory; the axis-0 pass gathers from
// a per-thread register queue of the last planes' partial results.  One CTA
// barrier per step of the march.  Every 1D
// pass evaluates the reference's expression in the reference's order with
// unfused multiply / add, so results are bit-identical to the reference C.
//
// What bounds them (K = 6, float64): the restriction latency, at 15 warps per SM
// with 63% of the shared-memory rate and 48% of the issue slots in use, the
// interpolation issue (67%); the unfused arithmetic is 20% and 15% of float64's
// rate.  Two input planes a step and one barrier instead of one plane and a barrier
// per pass: K = 6, float64, restriction of 2 grids of 192^3 170 -> 59 us,
// interpolation of 2 grids of 95^3 63.5 -> 51 us (with the caller's host work).
//
// 1D rules (K = 2 nn taps; w = the reference's weight table):
//   restrict  out[i] = 0.5 * (a[c] + w1 (a[c+1] + a[c-1]) + w3 (a[c+3] + a[c-3]) + ...)
//             c = K - 1 + 2 i in padded coordinates   (c/bmgs/restrict.c:37-57)
//   interpolate, o = 2 i + e - skip0 (e = 0 or 1), c = K/2 - 1 + i:
//             e = 0: out[o] = a[c]
//             e = 1: out[o] = w1 (a[c] + a[c+1]) + w3 (a[c-1] + a[c+2]) + ...
//                                                     (c/bmgs/interpolate.c:31-64)
#pragma once
#include "gpw_common.cuh"

namespace gpw {

struct TransferArgs {
  const void* in;
  void* out;
  GridView vin, vout;
  Boundary bc;        // boundary of the input grid
  int pad0[3];        // low padding of the input (padded -> unpadded shift)
  int skip0[3];       // interpolation: skip of the first output per axis
  int zchunk, nchunk; // output planes of axis 0 per CTA
  const unsigned char* active;
  int subtract;       // interpolation: out = base - I(in) instead of out = I(in)
  const void* base;   // (the reference's phi -= I(e) into another buffer; must not alias out)
  GridView vbase;
  // K=2 restriction into a multigrid level: also write the level's first
  // weighted-Jacobi sweep from phi = 0, out2 = (w2 / c02) out (same view)
  void* out2;
  double w2, c02;
};

// Per-thread descriptors of a box's cells (H x W, NT threads, cell k of a
// thread = tid + k NT): the box origin in (axis 1, axis 2) is fixed for the
// CTA, so each cell's in-plane source offset, validity and wrap sides are
// computed once; loading a plane is then one cp.async per cell and the
// Bloch fix-up touches only wrapped cells.
template <typename T, int H, int W, int NT>
struct BoxLoader {
  static constexpr int NLD = (H * W + NT - 1) / NT;
  int off[NLD];            // j1 * s1 + j2
  unsigned valid = 0;      // bit k: cell k is inside the grid or a periodic image
  unsigned wrapped = 0;    // bit k: cell k is a periodic image along axis 1 or 2
  unsigned char side[NLD]; // wrap sides: bits 0-1 axis 1 (+1), bits 2-3 axis 2 (+1)

  __device__ __forceinline__ void init(const GridView& v, const Boundary& bc, int ys, int xs) {
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
#pragma unroll
    for (int k = 0; k < NLD; ++k) {
      const int idx = tid + k * NT;
      const int r = idx / W, c = idx - r * W;
      int j1 = 0, j2 = 0, s1 = -1, s2 = -1;
      const bool ok = idx < H * W && wrap_axis(ys + r, v.n[1], bc.periodic[1], j1, s1) &&
                      wrap_axis(xs + c, v.n[2], bc.periodic[2], j2, s2);
      off[k] = ok ? (int)((int64_t)j1 * v.s1 + j2) : 0;
      if (ok) valid |= 1u << k;
      if (ok && (s1 >= 0 || s2 >= 0)) wrapped |= 1u << k;
      side[k] = (unsigned char)((s1 + 1) | ((s2 + 1) << 2));
    }
  }

  // plane p into `slot` (row pitch W); zero-boundary cells read zeros
  __device__ __forceinline__ void load(T* slot, const T* in, const GridView& v, const Boundary& bc, int p) const {
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    int j0, s0;
    const bool ok0 = wrap_axis(p, v.n[0], bc.periodic[0], j0, s0);
    const T* base = in + (int64_t)j0 * v.s0;
#pragma unroll
    for (int k = 0; k < NLD; ++k) {
      const int idx = tid + k * NT;
      if ((H * W) % NT == 0 || idx < H * W) {
        const bool ok = ok0 && ((valid >> k) & 1u);
        cp_async<sizeof(T)>(slot + idx, ok ? base + off[k] : in, ok);
      }
    }
  }

  // Bloch phases of the periodic images, axis by axis as the reference's
  // chained halo copies apply them (each thread fixes its own copies)
  __device__ __forceinline__ void fix(T* slot, const GridView& v, const Boundary& bc, int p) const {
    if constexpr (EltTraits<T>::cpx) {
      const int tid = threadIdx.x + blockDim.x * threadIdx.y;
      int j0, s0;
      if (!wrap_axis(p, v.n[0], bc.periodic[0], j0, s0)) return;
      const unsigned todo = s0 >= 0 ? valid : wrapped;
#pragma unroll
      for (int k = 0; k < NLD; ++k) {
        if (!((todo >> k) & 1u)) continue;
        const int idx = tid + k * NT;
        const int s1 = (side[k] & 3) - 1, s2 = ((side[k] >> 2) & 3) - 1;
        T val = slot[idx];
        if (s0 >= 0) val = phase_mul(bc.ph[0][s0], val);
        if (s1 >= 0) val = phase_mul(bc.ph[1][s1], val);
        if (s2 >= 0) val = phase_mul(bc.ph[2][s2], val);
        slot[idx] = val;
      }
    }
  }
};

// unfused helpers for exact reference arithmetic
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double2 radd(double2 a, double2 b) {
  return make_double2(__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y));
}
// (packed: one instruction for both components, each rounded as the scalar one)
__device__ __forceinline__ float2 radd(float2 a, float2 b) {
  add_pair(b.x, b.y, a.x, a.y);
  return a;
}
__device__ __forceinline__ double rmul(double c, double a) { return __dmul_rn(c, a); }
__device__ __forceinline__ float rmul(float c, float a) { return __fmul_rn(c, a); }
__device__ __forceinline__ double2 rmul(double c, double2 a) {
  return make_double2(__dmul_rn(c, a.x), __dmul_rn(c, a.y));
}
__device__ __forceinline__ float2 rmul(float c, float2 a) {
  float2 r;
  mul_pair(c, a.x, a.y, r.x, r.y);
  return r;
}

// K = 2 rules: 0.5 * (a0 + 0.5 * (a1 + a_1))   (c/bmgs/restrict.c:38-39)
template <typename S>
__device__ __forceinline__ S r2(S am, S a0, S ap) {
  using C = typename EltTraits<S>::S;
  return rmul(C(0.5), radd(a0, rmul(C(0.5), radd(ap, am))));
}
// 0.5 * (a0 + a1)                 (c/bmgs/interpolate.c:33)
template <typename S>
__device__ __forceinline__ S i2h(S a0, S a1) {
  return rmul(typename EltTraits<S>::S(0.5), radd(a0, a1));
}

template <int K> struct TW;
template <> struct TW<2> { static __device__ __forceinline__ double w(int) { return 0.5; } };
template <> struct TW<4> {
  static __device__ __forceinline__ double w(int j) { return j == 0 ? 0.5625 : -0.0625; }
};
template <> struct TW<6> {
  static __device__ __forceinline__ double w(int j) {
    return j == 0 ? 0.58593750 : (j == 1 ? -0.09765625 : 0.01171875);
  }
};
template <> struct TW<8> {
  static __device__ __forceinline__ double w(int j) {
    return j == 0 ? 0.59814453125 : (j == 1 ? -0.11962890625 : (j == 2 ? 0.02392578125 : -0.00244140625));
  }
};

// restriction tap sum around a[c] with stride `st` (in elements)
template <int K, typename T>
__device__ __forceinline__ T restrict_1d(const T* a, int st) {
  using S = typename EltTraits<T>::S;
  if constexpr (K == 2) {
    // 0.5 * (aa[0] + 0.5 * (aa[1] + aa[-1]))
    return rmul(S(0.5), radd(a[0], rmul(S(0.5), radd(a[st], a[-st]))));
  } else {
    T s = a[0];
#pragma unroll
    for (int j = 0; j < K / 2; ++j) s = radd(s, rmul((S)TW<K>::w(j), radd(a[(2 * j + 1) * st], a[-(2 * j + 1) * st])));
    return rmul(S(0.5), s);
  }
}

// interpolation midpoint value between a[0] and a[st]
template <int K, typename T>
__device__ __forceinline__ T interp_mid(const T* a, int st) {
  using S = typename EltTraits<T>::S;
  if constexpr (K == 2) {
    return rmul(S(0.5), radd(a[0], a[st]));
  } else {
    T s = rmul((S)TW<K>::w(0), radd(a[0], a[st]));
#pragma unroll
    for (int j = 1; j < K / 2; ++j) s = radd(s, rmul((S)TW<K>::w(j), radd(a[-j * st], a[(1 + j) * st])));
    return s;
  }
}

// ------------------------------------------------------------------ restrict
// A step takes the two fine planes of one coarse plane: the axis-2 pass of
// step s (items of one staged row and MO adjacent outputs, the row's columns
// read once; consecutive lanes take consecutive rows, whose odd pitch meets
// no bank conflict) and the axis-1 / axis-0 pass of step s - 1 run between
// the same two barriers, on two axis-2 buffers.  Of the 2K - 1 planes of an
// output only the centre and the K at odd distance count, so a thread keeps
// the last K even and K / 2 odd planes.
template <typename T, int K>
struct RestrictCfg {
  // tile of coarse points, one axis-1 item a thread; 16-byte elements of the
  // wide stencils in half-width tiles (two CTAs per SM)
  static constexpr int OZ = (sizeof(T) >= 16 && K >= 4) ? 16 : 32, OY = 8, NT = OZ * OY;
  static constexpr int H = 2 * OY + 2 * K - 3;  // fine rows per plane tile
  static constexpr int W = 2 * OZ + 2 * K - 3;  // fine cols (odd)
  static constexpr int ZP = OZ + 1;             // axis-2 result pitch (odd)
  static constexpr int MO = 4, NSEG = OZ / MO;  // axis-2 outputs per item
  static constexpr int NS = 2;                  // stages of two planes
  static constexpr size_t smem = (size_t)(NS * 2 * H * W + 2 * 2 * H * ZP) * sizeof(T);
};

template <typename T, int K>
__global__ void __launch_bounds__(RestrictCfg<T, K>::NT, 2) restrict_kernel(const TransferArgs a) {
  using C = RestrictCfg<T, K>;
  using S = typename EltTraits<T>::S;
  constexpr int H = C::H, W = C::W, ZP = C::ZP, MO = C::MO, NS = C::NS, KH = K / 2, NT = C::NT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* ring = reinterpret_cast<T*>(smem_raw);   // NS stages of two planes
  T* zb = ring + NS * 2 * H * W;              // two buffers of two planes' axis-2 results

  const int b = blockIdx.z / a.nchunk, chunk = blockIdx.z - b * a.nchunk;
  if (a.active && !a.active[b]) return;
  const int X0 = blockIdx.x * C::OZ, Y0 = blockIdx.y * C::OY;
  const int I0 = chunk * a.zchunk, I1 = min(a.vout.n[0], I0 + a.zchunk);
  if (I0 >= I1) return;
  const T* in = static_cast<const T*>(a.in) + (int64_t)b * a.vin.sb;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + C::OZ * ty;
  // fine planes feeding outputs I0 .. I1-1: step s takes planes pfirst + 2s
  // and (not in the last step) pfirst + 2s + 1
  const int pfirst = 2 * I0 - a.pad0[0];
  const int nsteps = I1 - I0 + K - 1;
  const int Y = Y0 + ty, X = X0 + tx;
  const bool inside = Y < a.vout.n[1] && X < a.vout.n[2];

  BoxLoader<T, H, W, NT> ld;
  ld.init(a.vin, a.bc, 2 * Y0 - a.pad0[1], 2 * X0 - a.pad0[2]);
  auto load = [&](int s) {
    T* sl = ring + (s % NS) * 2 * H * W;
    ld.load(sl, in, a.vin, a.bc, pfirst + 2 * s);
    if (s + 1 < nsteps) ld.load(sl + H * W, in, a.vin, a.bc, pfirst + 2 * s + 1);
  };
  auto fix = [&](int s) {
    if (!a.bc.use_phase) return;
    T* sl = ring + (s % NS) * 2 * H * W;
    ld.fix(sl, a.vin, a.bc, pfirst + 2 * s);
    if (s + 1 < nsteps) ld.fix(sl + H * W, a.vin, a.bc, pfirst + 2 * s + 1);
  };
  T ev[K], od[KH];  // even planes 2(s-K+1) .. 2s, odd planes of the last K / 2 steps
#pragma unroll
  for (int i = 0; i < K; ++i) ev[i] = zero<T>();
#pragma unroll
  for (int i = 0; i < KH; ++i) od[i] = zero<T>();

#pragma unroll
  for (int s = 0; s < NS; ++s) {
    if (s < nsteps) load(s);
    cp_async_commit();
  }
  cp_async_wait<NS - 1>();
  fix(0);
  __syncthreads();
  for (int s = 0; s <= nsteps; ++s) {
    if (s < nsteps) {
      // axis-2 pass of both planes
      const T* sl = ring + (s % NS) * 2 * H * W;
      T* zs = zb + (s & 1) * 2 * H * ZP;
      const int items = (s + 1 < nsteps ? 2 : 1) * H * C::NSEG;
      for (int it = tid; it < items; it += NT) {
        const int q = it / H, r = it - q * H;          // q: plane, segment
        const int pl = q / C::NSEG, Ja = (q - pl * C::NSEG) * MO;
        const T* rp = sl + (pl * H + r) * W + 2 * Ja;
        T* zrow = zs + (pl * H + r) * ZP + Ja;
        T w[MO + K - 1];
#pragma unroll
        for (int t = 0; t < MO + K - 1; ++t) w[t] = rp[2 * t];
#pragma unroll
        for (int i = 0; i < MO; ++i) {
          T sum = rp[2 * i + K - 1];
#pragma unroll
          for (int j = 0; j < KH; ++j)
            sum = radd(sum, rmul((S)TW<K>::w(j), radd(w[i + KH + j], w[i + KH - 1 - j])));
          zrow[i] = rmul(S(0.5), sum);
        }
      }
    }
    if (s >= 1) {
      // axis-1 pass of step s - 1's planes, axis-0 sum of the output they complete
      const int u = s - 1;
      const T* zs = zb + (u & 1) * 2 * H * ZP + (2 * ty + K - 1) * ZP + tx;
#pragma unroll
      for (int i = 0; i < K - 1; ++i) ev[i] = ev[i + 1];
      ev[K - 1] = restrict_1d<K>(zs, ZP);
      const int t = u - (K - 1);
      if (t >= 0 && inside) {
        T sum = od[0];
#pragma unroll
        for (int j = 0; j < KH; ++j) sum = radd(sum, rmul((S)TW<K>::w(j), radd(ev[KH + j], ev[KH - 1 - j])));
        static_cast<T*>(a.out)[(int64_t)b * a.vout.sb + (int64_t)(I0 + t) * a.vout.s0 + (int64_t)Y * a.vout.s1 + X] =
            rmul(S(0.5), sum);
      }
#pragma unroll
      for (int i = 0; i < KH - 1; ++i) od[i] = od[i + 1];
      if (s < nsteps) od[KH - 1] = restrict_1d<K>(zs + H * ZP, ZP);
    }
    cp_async_wait<NS - 2>();
    if (s + 1 < nsteps) fix(s + 1);
    __syncthreads();
    if (s + NS < nsteps) load(s + NS);
    cp_async_commit();
  }
}

// ------------------------------------------------------------------ interpolate
// A step takes one coarse plane and yields two fine planes: the axis-2 pass
// of step s (an item is one staged row and one coarse column: its copy and
// its midpoint, from K values) and the axis-1 / axis-0 pass of step s - 1 run
// between the same two barriers.  A thread owns PY adjacent fine rows of one
// column, whose axis-1 pass reads K - 1 + PY / 2 values once, and keeps K
// axis-0 values of each.
template <typename T, int K, int PY_>
struct InterpCfg {
  static constexpr int OZ = 32, NTY = 8, NT = OZ * NTY;
  static constexpr int PY = PY_;  // rows per thread
  static constexpr int OY = NTY * PY, NM = PY / 2;
  static constexpr int H = OY / 2 + K - 1;     // coarse rows per plane tile
  static constexpr int W = OZ / 2 + K;         // coarse cols
  static constexpr int NS = 3;
  static constexpr size_t smem = (size_t)(NS * H * W + 2 * H * OZ) * sizeof(T);
};

template <typename T, int K, int PY>
__global__ void __launch_bounds__(InterpCfg<T, K, PY>::NT, (sizeof(T) * K >= 128 ? 1 : 2))
    interpolate_kernel(const TransferArgs a) {
  using C = InterpCfg<T, K, PY>;
  using S = typename EltTraits<T>::S;
  constexpr int H = C::H, W = C::W, NS = C::NS, NM = C::NM, OZ = C::OZ, NT = C::NT;
  constexpr int base = K / 2 - 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* ring = reinterpret_cast<T*>(smem_raw);
  T* zb = ring + NS * H * W;  // axis-2 results, two buffers of H x OZ

  const int b = blockIdx.z / a.nchunk, chunk = blockIdx.z - b * a.nchunk;
  if (a.active && !a.active[b]) return;
  const int X0 = blockIdx.x * OZ, Y0 = blockIdx.y * C::OY;
  const int O0 = chunk * a.zchunk, O1 = min(a.vout.n[0], O0 + a.zchunk);
  if (O0 >= O1) return;
  const T* in = static_cast<const T*>(a.in) + (int64_t)b * a.vin.sb;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + OZ * ty;
  // coarse index i of a fine output o: o + skip0 = 2 i + e, its centre the
  // unpadded coarse point base + i - pad0; X0 and Y0 are even, so the tile's
  // first outputs have i = X0 / 2, Y0 / 2 whatever the skip
  const int sk1 = a.skip0[1], sk2 = a.skip0[2];
  const int i0f = (O0 + a.skip0[0]) >> 1, i0l = (O1 - 1 + a.skip0[0]) >> 1;
  const int pfirst = base + i0f - a.pad0[0] - (K / 2 - 1);
  const int plast = base + i0l - a.pad0[0] + K / 2;
  const int nsteps = plast - pfirst + 1;
  const int oy = Y0 + PY * ty, ox = X0 + tx;
  const int rows = ox < a.vout.n[2] ? min(PY, a.vout.n[1] - oy) : 0;  // this thread's rows inside the grid

  T q[PY][K];
#pragma unroll
  for (int j = 0; j < PY; ++j)
#pragma unroll
    for (int i = 0; i < K; ++i) q[j][i] = zero<T>();
  T* outp = static_cast<T*>(a.out) + (int64_t)b * a.vout.sb + (int64_t)oy * a.vout.s1 + ox;
  const T* basep = a.subtract ? static_cast<const T*>(a.base) + (int64_t)b * a.vbase.sb + (int64_t)oy * a.vbase.s1 + ox
                              : nullptr;

  BoxLoader<T, H, W, NT> ld;
  ld.init(a.vin, a.bc, Y0 / 2 - a.pad0[1], X0 / 2 - a.pad0[2]);
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    if (s < nsteps) ld.load(ring + s * H * W, in, a.vin, a.bc, pfirst + s);
    cp_async_commit();
  }
  cp_async_wait<NS - 1>();
  if (a.bc.use_phase) ld.fix(ring, a.vin, a.bc, pfirst);
  __syncthreads();
  for (int s = 0; s <= nsteps; ++s) {
    if (s < nsteps) {
      // axis-2 pass: staged row r, coarse column li -> fine columns 2 li - skip
      // (the copy) and 2 li + 1 - skip (the midpoint) of the tile
      const T* sl = ring + (s % NS) * H * W;
      T* zs = zb + (s & 1) * H * OZ;
      for (int it = tid; it < H * (OZ / 2); it += NT) {
        const int r = it / (OZ / 2), li = it - r * (OZ / 2);
        const T* rp = sl + r * W + li;
        T v[K];
#pragma unroll
        for (int t = 0; t < K; ++t) v[t] = rp[t];
        T* zp = zs + r * OZ + 2 * li - sk2;
        if (2 * li - sk2 >= 0) zp[0] = v[base];
        zp[1] = interp_mid<K>(v + base, 1);
      }
      if (sk2)  // the copy at the tile's last column
        for (int r = tid; r < H; r += NT) zs[r * OZ + OZ - 1] = sl[r * W + OZ / 2 + base];
    }
    if (s >= 1) {
      const int p = pfirst + s - 1;
      const T* cp = zb + ((s - 1) & 1) * H * OZ + NM * ty * OZ + tx;
      T col[K - 1 + NM];
#pragma unroll
      for (int i = 0; i < K - 1 + NM; ++i) col[i] = cp[i * OZ];
      const int ic = p - base + a.pad0[0];  // i with its centre at p
      const int oe = 2 * ic - a.skip0[0], oo = 2 * (ic - K / 2) + 1 - a.skip0[0];
      const bool ste = oe >= O0 && oe < O1, sto = oo >= O0 && oo < O1 && s - 1 >= K - 1;
#pragma unroll
      for (int j = 0; j < PY; ++j) {
        // axis-1 pass: rows alternate between copies and midpoints, starting
        // with a copy (skip 0) or a midpoint (skip 1)
        const T mid = interp_mid<K>(col + base + (j >> 1), 1);
        T v;
        if ((j & 1) == 0)
          v = sk1 ? mid : col[base + (j >> 1)];
        else
          v = sk1 ? col[base + (j >> 1) + 1] : mid;
#pragma unroll
        for (int i = 0; i < K - 1; ++i) q[j][i] = q[j][i + 1];
        q[j][K - 1] = v;
        if (j < rows) {
          // plane p completes the even output centred at p and the odd one
          // whose last tap is p
          const int64_t oj = (int64_t)j * a.vout.s1, bj = (int64_t)j * a.vbase.s1;
          if (ste) outp[(int64_t)oe * a.vout.s0 + oj] = a.subtract ? sub(basep[(int64_t)oe * a.vbase.s0 + bj], v) : v;
          if (sto) {
            const T m = interp_mid<K>(q[j] + base, 1);
            outp[(int64_t)oo * a.vout.s0 + oj] = a.subtract ? sub(basep[(int64_t)oo * a.vbase.s0 + bj], m) : m;
          }
        }
      }
    }
    cp_async_wait<NS - 2>();
    if (a.bc.use_phase && s + 1 < nsteps) ld.fix(ring + ((s + 1) % NS) * H * W, a.vin, a.bc, pfirst + s + 1);
    __syncthreads();
    if (s + NS < nsteps) ld.load(ring + (s % NS) * H * W, in, a.vin, a.bc, pfirst + s + NS);
    cp_async_commit();
  }
}

}  // namespace gpw
