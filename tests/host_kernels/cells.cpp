// Walks every address that the cell-staged star stencil (gpw_star_cells.cuh)
// loads or stores outside its staged planes: each array lies between
// inaccessible pages, first against the upper one, then against the lower, so
// an access on either side of it ends the program.
#include <sys/mman.h>
#include <unistd.h>
#include <cstdio>
#include <utility>

#include "gpawdft_b200/csrc/gpw_star_cells.cuh"

namespace gpw {
alignas(128) unsigned char smem_raw[256 * 1024];
}
using namespace gpw;

// `bytes` between two inaccessible regions longer than any halo
struct Guarded {
  static constexpr size_t G = 1 << 22;
  char* map;
  size_t len, bytes;
  explicit Guarded(size_t b) : bytes(b) {
    const size_t pg = sysconf(_SC_PAGESIZE);
    len = (b + pg - 1) / pg * pg;
    map = (char*)mmap(nullptr, len + 2 * G, PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (map == MAP_FAILED || mprotect(map + G, len, PROT_READ | PROT_WRITE)) exit(3);
  }
  ~Guarded() { munmap(map, len + 2 * G); }
  void* at(bool high) const { return map + G + (high ? len - bytes : 0); }
};

template <typename T, int R, int MODE, int TZ, int CELLB, int EPI, int SLOPE, int PY = 2>
static void walk(int n0, int n1, int n2, int nb, int nchunk, bool pot, bool aux, bool periodic) {
  using C = CellsCfg<T, R, MODE, TZ, CELLB, PY>;
  using S = typename EltTraits<T>::S;
  const size_t pts = (size_t)n0 * n1 * n2;
  Guarded in(pts * nb * sizeof(T)), out(pts * nb * sizeof(T)), other(pts * nb * sizeof(T)), v(pts * sizeof(S));
  for (int high = 0; high < 2; ++high) {
    StencilArgs a{};
    a.in = in.at(high);
    a.out = out.at(high);
    a.rho = MODE == MODE_APPLY ? nullptr : other.at(high);
    a.aux = aux ? other.at(high) : nullptr;
    a.pot = pot ? v.at(high) : nullptr;
    const GridView g{{n0, n1, n2}, (int64_t)n1 * n2, n2, (int64_t)pts};
    a.vin = a.vout = a.vrho = g;
    for (int c = 0; c < 3; ++c) a.bc.periodic[c] = periodic;
    a.bc.use_phase = periodic;
    a.nchunk = nchunk;
    a.w = a.c0 = 1.0;
    gridDim = {(unsigned)(n2 + C::TZ - 1) / C::TZ, (unsigned)(n1 + C::TY - 1) / C::TY, (unsigned)(nchunk * nb)};
    blockDim = {(unsigned)C::NT, 1, 1};
    for (blockIdx.z = 0; blockIdx.z < gridDim.z; ++blockIdx.z)
      for (blockIdx.y = 0; blockIdx.y < gridDim.y; ++blockIdx.y)
        for (blockIdx.x = 0; blockIdx.x < gridDim.x; ++blockIdx.x)
          for (threadIdx.x = 0; threadIdx.x < blockDim.x; ++threadIdx.x)
            star_cells_kernel<T, R, MODE, TZ, CELLB, EPI, true, SLOPE, PY>(a, StarCoefsT<S>{});
  }
}

template <typename T, int R, int TZ, int CELLB, int SLOPE, int PY = 2>
static void applies(int n0, int n1, int n2, int nb, int nchunk, bool periodic) {
  walk<T, R, MODE_APPLY, TZ, CELLB, 0, SLOPE, PY>(n0, n1, n2, nb, nchunk, false, false, periodic);
  walk<T, R, MODE_APPLY, TZ, CELLB, 1, SLOPE, PY>(n0, n1, n2, nb, nchunk, true, false, periodic);
  walk<T, R, MODE_APPLY, TZ, CELLB, 2, SLOPE, PY>(n0, n1, n2, nb, nchunk, false, true, periodic);
  walk<T, R, MODE_APPLY, TZ, CELLB, 2, SLOPE, PY>(n0, n1, n2, nb, nchunk, true, true, periodic);
}

int main() {
  for (int periodic = 0; periodic < 2; ++periodic) {
    applies<double2, 3, 32, 16, 0>(9, 17, 33, 2, 1, periodic);
    applies<double2, 3, 32, 16, 1>(17, 21, 21, 2, 2, periodic);
    applies<double2, 1, 24, 16, -1>(8, 5, 25, 1, 2, periodic);
    applies<double, 3, 32, 8, 0>(17, 33, 31, 2, 2, periodic);
    applies<double, 2, 48, 16, 0>(12, 21, 50, 1, 2, periodic);
    applies<double, 4, 32, 8, 0>(3, 3, 3, 1, 1, periodic);
    applies<double, 4, 32, 16, 0, 1>(11, 17, 34, 1, 1, periodic);
    applies<float, 2, 32, 4, 0, 1>(13, 33, 37, 2, 2, periodic);
    applies<float2, 1, 32, 8, 0, 1>(9, 17, 31, 2, 2, periodic);
    walk<double, 3, MODE_RESIDUAL, 32, 8, 0, 0>(17, 33, 31, 2, 2, false, false, periodic);
    walk<double, 1, MODE_JACOBI, 48, 16, 0, 0>(9, 21, 50, 2, 2, false, false, periodic);
  }
  std::puts("in bounds");
  return 0;
}
