// march.cuh -- the fused x1 stage of a block of many columns: a CTA takes a
// tile of 32 neighbouring columns, a lane per column, and marches from the top
// level to the bottom in chunks of C levels, then back up.
//
// The CTA-per-column kernel (column.cuh) pays for parallelism inside a column:
// cyclic and parallel cyclic reduction instead of one elimination, a serial
// hydrostatic scan on one lane, phases that leave most lanes of the CTA idle.
// With thousands of columns the columns themselves are the parallelism, and
// the block elimination runs serially in a lane:
//   warps 0 .. C-1 share the levels of a chunk, in four phases:
//     1. the hydrostatic scan down to a level and its decomposition
//     2. reconstruction, two levels up: four cells of one variable at a time,
//        so that every limited slope and interface value is computed once
//     3. the Riemann problem at a face, three levels up
//     4. four levels up: flux divergence and sources added to du, |A| at the
//        cell's lower face and the Jacobian of the cell below
//     (column.cuh P1-P5a, the same expressions)
//   warps C and C + 1 eliminate the rows of the previous chunk downwards
//     (forward_backward.hpp:15-91 with the sweep reversed), a row each in
//     turn, so that one forms its row while the other finishes the row above:
//     with the rows scaled by twice the cell's volume over its lower face area,
//     b' = A_i + J_{i-1} = -b, c' = A_{i+1} - J_{i+1} = -c,
//     D_i = a_i - c'_i H_{i+1}, H_i = D_i^-1 b'_i,
//     g_i = D_i^-1 (r_i + c'_i g_{i+1}); 5x5 blocks by LU, with pivoting where
//     a pivot cancels
// H, g and what the update needs of du go to a scratch array laid out
// [tile][level][component][lane]; on the way up x_i = g_i + H_i x_{i-1}, then
// the species correction and the register update (forward_backward.hpp:93-137,
// implicit_hydro_tasks.cpp:152-160, 283).
//
// Rows of the block arrays run along x1, so the columns of a tile are strided
// in memory.  TMA moves them: a box of C levels x 32 columns x NV variables
// per request (a probe of the access pattern on w of 128x256x256: 5.9 TB/s,
// 3.0 TB/s with cp.async, 4.5 TB/s with loads and shared-memory stores).  A
// tensor map needs rows of a multiple of 16 bytes: for columns of an odd number
// of levels (g.bulk = 0) the map's rows are pairs of columns, and a request
// takes every second column of one variable from the 16-byte boundary below
// the chunk's first level, two levels more than the chunk.
//
// Measured against the CTA-per-column kernel (one launch, 128x256x256 moist,
// PPM + HLLC): FP32 fluxes 2.52 -> 1.16 ms, FP64 3.05 -> 1.63 ms; with 5x5
// blocks FP32 12.3 -> 3.1 ms.  What bounds it: a chunk is a chain of four
// barrier-separated phases of dependent FP64 and FP32 arithmetic (about 10k
// cycles for eight levels) that two CTAs per SM (shared memory) overlap: issue
// 46 %, DRAM 47 % busy; its traffic is the algorithmic bytes and 2 x 144 B per
// cell of scratch (18 doubles with three species).
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>

#include <type_traits>

#include "column.cuh"

namespace cb {

constexpr int kMarchCols = 32;  // columns per CTA
constexpr int kMarchUp = 4;     // levels per chunk of the way back up
// Fewest columns that march.  As long as every tile has an SM to itself (148
// tiles, 4736 columns) the march takes as long as for one: 128 levels of eight
// variables 121 us in FP32, 186 us in FP64, where the CTA-per-column kernel takes
// 38 and 46 ns a column.
constexpr int kMarchMinCols32 = 3400, kMarchMinCols64 = 4300;
// with 5x5 blocks one tile fills an SM: 128 levels 227 us a round of 148 tiles
// against 188 ns a column
constexpr int kMarchMinCols5 = 1200;
// Two tiles on an SM get in each other's way in FP64: 65x67 columns, 153 tiles,
// of 128 levels take 1172 us a step marching, 1092 with a CTA per column, and
// 69x70, 162 tiles, 1188 and 1171.  Outside these numbers of levels, where the
// other kernel is the slower one (16: 375 and 276 us), the line stays.
constexpr int kMarchMinCols64Pairs = 4800, kMarchPairsLo = 32, kMarchPairsHi = 150;
// Where shared memory holds one tile on an SM (six species but for even columns
// in FP32), 3x3 blocks march in rounds of 148 tiles, each of which has to pay
// for itself: so many sixteenths of the least columns, by the number of levels.
// Six species of 65 levels, 69x70 columns in two rounds: 893 us a step with a
// CTA per column, 1229 marching in FP32, 1270 and 1635 in FP64; 64x74 columns in
// one: 1043 and 858 in FP64.  Of 16 levels 69x70 columns take 492 and 434 us, of
// 160 levels 64x100 columns, in two rounds too, 2563 and 2281.
constexpr int march_round_16ths(int nx1, bool f32) {
  return nx1 < 32 ? 8 : (nx1 <= 128 ? (f32 ? 16 : 15) : 11);
}

// scratch per level of a tile with N x N blocks: H and g (a tile's levels
// contiguous); then du of the two transverse momenta (N = 3, whose solve
// leaves them), of the species, and (with species) the sum of the density
// increments.  The RK register u1 lies in the block's own array of it, in the
// same order of tiles, levels, components and lanes.
__host__ __device__ constexpr int march_h(int n) { return n * n + n; }
__host__ __device__ constexpr int march_nt(int n) { return n == 3 ? 2 : 0; }
__host__ __device__ constexpr int march_nd(int ny, int n) {
  return march_nt(n) + ny + (ny > 0 ? 1 : 0);
}

// tiles of bj x bk = 32 columns that cover nx2 x nx3 with the fewest tiles
struct MarchTile {
  int bj, bk, nj, nk;
};
inline MarchTile march_tile(int nx1, int nx2, int nx3) {
  MarchTile best{0, 0, 0, 0};
  // odd columns need a request per variable, k and parity of j, each to a
  // 128-byte boundary of shared memory
  for (int bj = 32; bj >= (nx1 % 2 ? 16 : 1); bj /= 2) {
    const int bk = kMarchCols / bj;
    const MarchTile t{bj, bk, (nx2 + bj - 1) / bj, (nx3 + bk - 1) / bk};
    if (!best.bj || (int64_t)t.nj * t.nk < (int64_t)best.nj * best.nk) best = t;
  }
  return best;
}

// lanes times levels of all tiles: doubles per component of scratch and u1
inline size_t march_cells(int nx1, int nx2, int nx3, int npanel) {
  const MarchTile t = march_tile(nx1, nx2, nx3);
  return (size_t)t.nj * t.nk * npanel * nx1 * kMarchCols;
}

// Shared memory of a tile, in doubles.  Levels are counted from the top (t = 0
// is the highest ghost cell).  w and du hold the chunk in hand; rings of a
// chunk and four levels hold the decomposed state q, the FP64 values that
// later phases need beside it (raw), and the face states wL, overwritten by
// the fluxes.
template <int NV, int C, typename R, int GEO, int N>
struct MarchSmem {
  static constexpr int RQ = C + 4, RP = 16, NC = kMarchCols, ny = NV - 5;
  // rows in the ring of |A|, J and the right-hand side: a chunk's, and the two
  // that the elimination still works on while the next chunk's are formed with
  // the two above them
  static constexpr int RR = C + 4, NRH = N + (GEO ? 2 : 1), NAJ = N * N + N * (N - 1);
  // raw: rho, p and, where q is rounded to FP32, v1 (GEO: all velocities)
  static constexpr int NR = sizeof(R) == 8 ? 2 : (GEO ? 5 : 3);
  static constexpr int rsz(int n) { return (n * (int)sizeof(R) + 7) / 8; }
  static constexpr int w = 0;                        // [NV][32][C], swizzled;
  static constexpr int wr = w;                       // in phases 2, 3: wR, [C][NV][32] R
  static constexpr int d = w + C * NV * NC;          // [NV][32][C], swizzled
  static constexpr int q = d + C * NV * NC;          // [RQ][NV][32] R
  static constexpr int raw = q + rsz(RQ * NV * NC);  // [RQ][NR][32]
  static constexpr int f = raw + RQ * NR * NC;       // [RQ][NV][32] R: wL, then F
  static constexpr int ps = f + rsz(RQ * NV * NC);   // [RP][32] face pressure
  static constexpr int gm = ps + RP * NC;            // [RQ][32] RovRd
  static constexpr int r = gm + RQ * NC;             // [RR][NRH][32] rhs, row geometry
  static constexpr int aj = r + RR * NRH * NC;       // [RR][NAJ][32] R: |A|, J
  static constexpr int hg = aj + rsz(RR * NAJ * NC);  // [NH][32] H, g of the last row
  static constexpr int NH = march_h(N);
  static constexpr int total1 = hg + NH * NC;
  // way back up: u and the species of w of four chunks, H and g of three, and x
  // of two
  static constexpr int UP = kMarchUp;
  // [4][NV][32][lev] u and [4][ny][32][lev] species first, then H, g and x
  static constexpr int hx(int lev) { return 4 * (NV + ny) * lev * NC; }
  static constexpr int nhx = 3 * UP * NH * NC + 2 * UP * N * NC;
  // columns of an odd number of levels keep two levels more of w and d each,
  // which shifts what follows, and of u and sp
  static constexpr int shift = 2 * NV * NC;
  static constexpr int total(bool odd) {
    const int a = total1 + (odd ? 2 * shift : 0), b = hx(odd ? UP + 2 : UP) + nhx;
    return a > b ? a : b;
  }
  // the levels' dx follow at `total`
  static constexpr size_t bytes(int nc1) { return sizeof(double) * ((size_t)total(nc1 % 2) + nc1); }
};

// levels per chunk: with 3x3 blocks eight in FP32, as far as two CTAs fit an SM
// with them (77x83x61 with eight and one CTA: 192 us, with four and two: 150);
// with 5x5 blocks four, whose six warps have the registers for the elimination
// (64x96x96 with eight levels: 524 bytes of spills, 1097 us a step; four: 1076)
template <typename R>
constexpr int march_chunk(int ny, int n, int odd) {
  return sizeof(R) == 4 && n == 3 && ny <= (odd ? 2 : 3) ? 8 : 4;
}

// barriers reached from the level warps' and the elimination warp's own loops
template <int ID, int NT>
__device__ __forceinline__ void march_sync() {
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(NT) : "memory");
}

template <int ID, int NT>
__device__ __forceinline__ void march_arrive() {
  asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(NT) : "memory");
}

struct MarchMaps {
  CUtensorMap w, du, u, sp;
};

__device__ __forceinline__ void march_tma_load(double *dst, const CUtensorMap *map, int x, int j,
                                               int k, int n, int pan, uint64_t *m) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(smem_addr(dst)),
      "l"(map), "r"(x), "r"(j), "r"(k), "r"(n), "r"(pan), "r"(smem_addr(m))
      : "memory");
}
__device__ __forceinline__ void march_tma_load2(double *dst, const CUtensorMap *map, int x, int y,
                                                uint64_t *m) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3}], [%4];" ::"r"(smem_addr(dst)),
      "l"(map), "r"(x), "r"(y), "r"(smem_addr(m))
      : "memory");
}
__device__ __forceinline__ void march_tma_store(const CUtensorMap *map, int x, int j, int k, int n,
                                                int pan, const double *src) {
  asm volatile(
      "cp.async.bulk.tensor.5d.global.shared::cta.tile.bulk_group "
      "[%0, {%1, %2, %3, %4, %5}], [%6];" ::"l"(map),
      "r"(x), "r"(j), "r"(k), "r"(n), "r"(pan), "r"(smem_addr(src))
      : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// place of (variable, column, level) in a box of 8 or 4 levels as TMA lays it
// out with the 64- or 32-byte swizzle: 16-byte pieces permuted so that a
// warp's reads of one level spread over the banks
template <int C>
__device__ __forceinline__ int march_box(int n, int c, int o) {
  if constexpr (C == 8) return (n * kMarchCols + c) * 8 + ((((o >> 1) ^ (c >> 1)) & 3) << 1) + (o & 1);
  else return (n * kMarchCols + c) * 4 + ((((o >> 1) ^ (c >> 2)) & 1) << 1) + (o & 1);
}

// Blocks of row t, scaled by twice the cell's volume over its lower face area:
// D x_i = v + b x_{i-1} + c x_{i+1}, from the rings of |A|, J (ajb) and the
// right-hand side (rb); at the walls (`bottom`, `top`) the ghost cell mirrors
// the boundary cell.  gw: gravity times the stage's time step
template <int N, int GEO, int RR, int NRH, int NAJ, typename R>
__device__ __forceinline__ void march_blocks(const R *ajb, const double *rb, int t, bool bottom,
                                             bool top, double gw, double (&D)[N][N],
                                             double (&b)[N][N], double (&c)[N][N], double (&v)[N]) {
  constexpr int NC = kMarchCols;
  // |A| at faces i and i + 1; J of cells i - 1, i and i + 1 (rows 1 ..)
  const R *ai = ajb + (t % RR) * NAJ * NC, *ap = ajb + ((t - 1) % RR) * NAJ * NC;
  const R *jm = ai + N * N * NC, *jc = ap + N * N * NC,
          *jp = ajb + ((t - 2) % RR) * NAJ * NC + N * N * NC;
  auto jrow = [](const R *j, int x, int y) {
    return x == 0 ? (y == 1 ? 1. : 0.) : (double)j[((x - 1) * N + y) * NC];
  };
  const double *ri = rb + (t % RR) * NRH * NC;
  const double dd = ri[N * NC];
  const double ra = GEO ? ri[(N + 1) * NC] : 1.;
#pragma unroll
  for (int x = 0; x < N; ++x) {
    v[x] = ri[x * NC];
#pragma unroll
    for (int y = 0; y < N; ++y) {
      const double am = ai[(N * x + y) * NC], au = ap[(N * x + y) * NC];
      if constexpr (GEO) {
        D[x][y] = am + au * ra + (ra - 1.) * jrow(jc, x, y);
        c[x][y] = (au - jrow(jp, x, y)) * ra;
      } else {
        D[x][y] = am + au;
        c[x][y] = x == 0 && y != 1 ? au : au - jrow(jp, x, y);
      }
      b[x][y] = x == 0 && y != 1 ? am : am + jrow(jm, x, y);
    }
    D[x][x] += dd;
  }
  const double ph = gw * dd;  // gravity over the row's scale
  D[1][0] -= ph;
  D[N - 1][1] -= ph;
  if (bottom) {
#pragma unroll
    for (int x = 0; x < N; ++x)
#pragma unroll
      for (int y = 0; y < N; ++y) {
        D[x][y] += y == 1 ? b[x][y] : -b[x][y];
        b[x][y] = 0.;
      }
  }
  if (top) {
#pragma unroll
    for (int x = 0; x < N; ++x)
#pragma unroll
      for (int y = 0; y < N; ++y) D[x][y] += y == 1 ? c[x][y] : -c[x][y];
  }
}

// D - c H and v + c g of the row above's H, g
template <int N>
__device__ __forceinline__ void march_above(const double *hg, double (&D)[N][N],
                                            const double (&c)[N][N], double (&v)[N]) {
  constexpr int NC = kMarchCols;
#pragma unroll
  for (int z = 0; z < N; ++z) {
    double hz[N];
#pragma unroll
    for (int y = 0; y < N; ++y) hz[y] = hg[(N * z + y) * NC];
    const double gz = hg[(N * N + z) * NC];
#pragma unroll
    for (int x = 0; x < N; ++x) {
#pragma unroll
      for (int y = 0; y < N; ++y) D[x][y] -= c[x][z] * hz[y];
      v[x] += c[x][z] * gz;
    }
  }
}

// magnitude of x for comparisons: the high word of |x|, whose differences of
// kPivotHigh are factors of 8
constexpr int kPivotHigh = 3 << 20;
__device__ __forceinline__ int high_word(double x) { return __double2hiint(x) & 0x7fffffff; }

// D = L U in place without pivoting, rp the pivots' reciprocals.
// Elimination does not feel a diagonal scaling, and at low Mach number or a
// vertical Courant number of a few D is a multiple of the identity with some
// |A| and flux differences (a host restatement of the recursion in 64 and 80
// bits: 60 to 1000 times closer than pivoting by the largest entry, as the rows
// differ in scale).  Beyond, pivots cancel: at Mach 1 and Courant number 300 it
// was up to 4e5 times further off.  False, and L U is not to be used, where a
// pivot is 8 times smaller or larger than the diagonal it came from, or not a
// number: the restatement is then as close as with pivoting throughout, and at
// Mach 0.05 no row of 10^4 fails up to Courant number 3, and 6 at 30.
__device__ __forceinline__ bool march_factor(double (&D)[5][5], double (&rp)[5]) {
  constexpr int N = 5;
  int od[N];  // the diagonal before elimination
#pragma unroll
  for (int q = 1; q < N; ++q) od[q] = high_word(D[q][q]);
#pragma unroll
  for (int q = 0; q < N; ++q) {
    rp[q] = Recip<double>(D[q][q]).r;
#pragma unroll
    for (int x = q + 1; x < N; ++x) {
      D[x][q] *= rp[q];
#pragma unroll
      for (int y = q + 1; y < N; ++y) D[x][y] -= D[x][q] * D[q][y];
    }
  }
  bool good = true;
#pragma unroll
  for (int q = 1; q < N; ++q)
    good &= (unsigned)(high_word(D[q][q]) - od[q] + kPivotHigh) < 2u * kPivotHigh;
  return good;
}

// h = (L U)^-1 [b v]: row-major D^-1 b, then D^-1 v
__device__ __forceinline__ void march_sweeps(const double (&D)[5][5], const double (&rp)[5],
                                             const double (&b)[5][5], const double (&v)[5],
                                             double (&h)[30]) {
  constexpr int N = 5;
#pragma unroll
  for (int y = 0; y <= N; ++y) {
    double r[N];
#pragma unroll
    for (int x = 0; x < N; ++x) {
      r[x] = y < N ? b[x][y < N ? y : 0] : v[x];
#pragma unroll
      for (int q = 0; q < x; ++q) r[x] -= D[x][q] * r[q];
    }
#pragma unroll
    for (int x = N - 1; x >= 0; --x) {
#pragma unroll
      for (int q = x + 1; q < N; ++q) r[x] -= D[x][q] * r[q];
      r[x] *= rp[x];
      h[y < N ? N * x + y : N * N + x] = r[x];
    }
  }
}

// The same by Gauss-Jordan elimination with partial pivoting, as inv(M<5>): the
// way out of march_factor, rare, so that its rows lie in local memory
static __device__ __noinline__ void march_pivoted(const double (&D)[5][5], const double (&b)[5][5],
                                           const double (&v)[5], double (&h)[30]) {
  constexpr int N = 5, NR = 2 * N + 1;
  double a[N][NR];
  for (int x = 0; x < N; ++x) {
    for (int y = 0; y < N; ++y) {
      a[x][y] = D[x][y];
      a[x][N + y] = b[x][y];
    }
    a[x][2 * N] = v[x];
  }
#pragma unroll 1
  for (int q = 0; q < N; ++q) {
    int p = q;
    for (int x = q + 1; x < N; ++x)
      if (fabs(a[x][q]) > fabs(a[p][q])) p = x;
    const double ip = 1. / a[p][q];
    for (int y = q; y < NR; ++y) {
      const double e = a[p][y] * ip;
      a[p][y] = a[q][y];
      a[q][y] = e;
    }
#pragma unroll 1
    for (int x = 0; x < N; ++x) {
      if (x == q) continue;
      const double f = a[x][q];
      for (int y = q; y < NR; ++y) a[x][y] -= f * a[q][y];
    }
  }
  for (int x = 0; x < N; ++x) {
    for (int y = 0; y < N; ++y) h[N * x + y] = a[x][N + y];
    h[N * N + x] = a[x][2 * N];
  }
}

// Row t from its blocks on, by either: H, g to hg and so.  For the warps of
// which some lane's march_factor fails
template <int GEO, int RR, int NRH, int NAJ, typename R>
__device__ __noinline__ void march_row_pivoted(const R *ajb, const double *rb, double *hg,
                                               double *so, int t, bool bottom, bool top,
                                               double gw) {
  constexpr int NC = kMarchCols;
  double D[5][5], A[5][5], b[5][5], c[5][5], v[5], rp[5], h[30];
  march_blocks<5, GEO, RR, NRH, NAJ>(ajb, rb, t, bottom, top, gw, D, b, c, v);
  if (!top) march_above<5>(hg, D, c, v);
#pragma unroll
  for (int x = 0; x < 5; ++x)
#pragma unroll
    for (int y = 0; y < 5; ++y) A[x][y] = D[x][y];
  if (march_factor(D, rp)) march_sweeps(D, rp, b, v, h);
  else march_pivoted(A, b, v, h);
  for (int e = 0; e < 30; ++e) {
    hg[e * NC] = h[e];
    so[e * NC] = h[e];
  }
}

template <int NY, int RECON, int RS, typename R, int GEO, int C, int N>
__global__ void __launch_bounds__((C + 2) * 32, N == 3 ? 2 : 1)
    k_x1march(Geom g, canoe_thermo_t th, Mix<R> mx, MarchTile tl,
              const __grid_constant__ MarchMaps maps,
              const double *__restrict__ w, const double *__restrict__ du, double *u, double *scr,
              double *u1,
              const double *__restrict__ dtp, Stage st, int stage) {
  using S = Slots<NY>;
  using P = MarchSmem<5 + NY, C, R, GEO, N>;
  constexpr int NV = S::NV, NC = kMarchCols, UP = kMarchUp;
  constexpr int ND = march_nd(NY, N), NT = march_nt(N), NH = P::NH;
  constexpr int RQ = P::RQ, RP = P::RP, NR = P::NR, RR = P::RR, NRH = P::NRH,
                NAJ = P::NAJ;
  constexpr bool PERT = sizeof(R) == 4;
  constexpr int NTP = C * 32, NTA = NTP + 64;
  extern __shared__ __align__(1024) double sm[];
  // w, du; of the way back up u and species (4 chunks), H and g (3)
  constexpr int MU = 2, MH = 6, NMB = 9;
  __shared__ __align__(8) uint64_t mbar[NMB];
  // bit q: a wait for barrier q gave up; of each barrier, 1 + the parity of the
  // phase armed last (0: none)
  __shared__ int lost_, armed[NMB];
  volatile int *const lost = &lost_;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nc1 = g.nc1, is = g.is, ie = g.ie;
  const bool bulk = g.bulk != 0;
  const bool leader = threadIdx.x == 0;

  // the tile's first column, and this lane's column within it: columns past
  // the block's edge repeat the last one inside and write nothing to u (their
  // scratch is their own)
  const int tj = blockIdx.x % tl.nj, tkp = blockIdx.x / tl.nj;
  const int pan = tkp / tl.nk;
  const int j0 = g.js + tj * tl.bj, k0 = g.ks + (tkp - pan * tl.nk) * tl.bk;
  const int j = min(j0 + lane % tl.bj, g.je), k = min(k0 + lane / tl.bj, g.ke);
  const int lc = (k - k0) * tl.bj + (j - j0);
  const bool on = lc == lane;
  const int64_t pbase = g.npanel > 1 ? (int64_t)pan * g.pstride : 0;
  const int64_t base = pbase + (int64_t)k * g.sk + (int64_t)j * nc1;
  // without boxes: the columns' first cells, and which columns are the tile's
  __shared__ int64_t colb[NC];
  const unsigned mine = __ballot_sync(~0u, on);
  if (threadIdx.x < NC) colb[threadIdx.x] = base;
  constexpr int WO = C + 2, UO = UP + 2;  // levels of a column in such a copy
  // parity of this column's first cell and of the step to the next variable:
  // where the 16-byte boundary lies
  const int par = (int)(base & 1), psv = (int)(g.sv & 1);
  // variables n0 .. n0 + nn - 1 of an array from level lo, by a warp; a box of
  // wl levels for each variable, k and parity of j, the even j's first
  auto pairs = [&](double *dst, const CUtensorMap *map, int n0, int nn, int lo, int wl, uint64_t *m) {
    for (int e = lane; e < nn * 2 * tl.bk; e += 32) {
      const int kk = e % tl.bk, pj = e / tl.bk % 2, n = e / (2 * tl.bk);
      const int row = (int)(pbase / nc1) + ((n0 + n) * g.nc3 + k0 + kk) * g.nc2 + j0 + pj;
      const int x = (row & 1) * nc1 + lo;
      march_tma_load2(dst + (n * NC + pj * (NC / 2) + kk * (tl.bj / 2)) * wl, map, x - (x & 1),
                      row >> 1, m);
    }
  };
  auto pcol = [&](int c) { return (c % tl.bj % 2) * (NC / 2) + c / tl.bj * (tl.bj / 2) + c % tl.bj / 2; };
  const int lp = bulk ? 0 : pcol(lc);
  double *scrh = scr + (int64_t)blockIdx.x * g.nx1 * NH * NC;  // H, g of the tile
  scr += (int64_t)gridDim.x * g.nx1 * NH * NC + (int64_t)blockIdx.x * g.nx1 * ND * NC;
  u1 += (int64_t)blockIdx.x * g.nx1 * NV * NC;
  const double grav = th.grav;
  const double wght = st.beta * dtp[0], idt = 1. / wght;
  double *wb = sm + P::w, *db = sm + P::d + (bulk ? 0 : P::shift);
  double *const sm2 = sm + (bulk ? 0 : 2 * P::shift);  // what follows w and d
  const int VS = NC * (bulk ? C : WO);  // doubles per variable of w, du
  double *rb = sm2 + P::r + lane;
  double *psr = sm2 + P::ps + lane, *gmr = sm2 + P::gm + lane, *rawb = sm2 + P::raw + lane;
  R *qb = reinterpret_cast<R *>(sm2 + P::q) + lane;
  R *fb = reinterpret_cast<R *>(sm2 + P::f) + lane;
  R *wrb = reinterpret_cast<R *>(sm + P::wr) + lane;
  R *ajb = reinterpret_cast<R *>(sm2 + P::aj) + lane;
  double *sdx = sm + P::total(!bulk);  // dx1f
  const int last_m = nc1 / C;  // rows lag the levels by four: t = nc1 ends them

  // The elimination warps, which have time to spare, wait for the copies; the
  // barrier that they then join hands the data to the level warps.  A bounded
  // wait that gave up is reported and sets `lost`, which other warps see behind
  // that barrier at the latest: the barrier whose phase is still open is not
  // armed again, no copy is issued to its buffer and nothing written to u.  The
  // tile runs its barriers out on whatever the buffers hold, gives the phases
  // still in flight a second bounded wait and leaves.
  bool ok = true;  // what this warp's own waits found
  auto wait = [&](int q, uint32_t parity) {
    if (ok && !mbar_wait(mbar + q, parity, q < MU ? g.polls : g.polls_up)) {
      ok = false;
      atomicOr(&lost_, 1 << q);
      if (g.err) atomicOr(g.err, (uint32_t)CANOE_EBIT_TIMEOUT);
    }
  };
  auto arm = [&](int q, uint32_t parity, uint32_t bytes) {
    armed[q] = 1 + (int)parity;
    mbar_expect_tx(mbar + q, bytes);
  };
  // w (q = 0) or du (1) of chunk m: w of levels lo .. lo + C - 1, du of the rows
  // that the chunk completes, four levels up.  A box is one request, by the
  // level warps' leader; the many of columns of odd levels are left to an
  // elimination warp (77x83x61: 429 -> 417 us a step).
  auto fetch = [&](int q, int m) {
    double *dst = q ? db : wb;
    const CUtensorMap *map = q ? &maps.du : &maps.w;
    const int lo = nc1 - C * (m + 1) + (q ? 4 : 0);
    if (lane == 0) {
      arm(q, m & 1, VS * NV * 8);
      if (bulk) march_tma_load(dst, map, lo, j0, k0, 0, pan, mbar + q);
    }
    if (!bulk) {
      __syncwarp();
      pairs(dst, map, 0, NV, lo, WO, mbar + q);
    }
  };
  if (leader) {
    *lost = 0;
    for (int q = 0; q < NMB; ++q) {
      armed[q] = 0;
      mbar_init(mbar + q, 1);
    }
    fence_mbar_init();
  }
  for (int i = threadIdx.x; i < nc1; i += NTA) sdx[i] = g.dx1f[i];
  __syncthreads();

  if (warp < C) {
    const int64_t nkj = (int64_t)g.nc3 * g.nc2;
    auto tab = [&](int t, int kk, int jj) { return g.shell[t * nkj + (int64_t)kk * g.nc2 + jj]; };
    double cosc = 0., sinc = 1., cth1 = 0.;
    if constexpr (GEO) {
      cosc = tab(kTabCosC, k, j);
      sinc = tab(kTabSinC, k, j);
      cth1 = tab(kTabCth1, k, j);
    }
    // place of level lo + o of this lane's column, in the even / odd variables
    const int pw0 = (par + nc1) & 1, pw1 = pw0 ^ psv;  // lo has nc1's parity
    auto at0 = [&](int o) { return bulk ? march_box<C>(0, lc, o) : lp * WO + o + pw0; };
    auto at1 = [&](int o) { return bulk ? march_box<C>(0, lc, o) : lp * WO + o + pw1; };
    const int a0 = at0(C - 1 - warp), a1 = at1(C - 1 - warp);  // this warp's level
    auto wrap = [](int s) { return s < 0 ? s + RQ : (s >= RQ ? s - RQ : s); };
    static_assert(RR == RQ, "rows and levels share their ring places");
    int bq = 0;  // ring place of the chunk's first level and row
    if (bulk && leader) fetch(0, 0);
    // `lost`, read behind one fetch for the next, whose buffer's last wait lies
    // before the barrier that opened this phase
    int gone = 0;
    if (warp == 0) {
      // face pressures from the top of the column up through the ghosts
      // (t = 2 is the face ie + 1)
      const double *w0 = w + base, *wp_ = w0 + S::IPR * g.sv;
      const double RdTv = wp_[ie] / w0[ie];
      double p = wp_[ie] * exp(grav * sdx[ie] / (2 * RdTv));
      const double gt = g.bc[1] == CANOE_BC_REFLECT ? -grav : grav;
      psr[2 * NC] = p;
#pragma unroll
      for (int t = 1; t <= NG; ++t) {
        p = p + gt * w0[ie + t] * sdx[ie + t];
        psr[((2 - t) & (RP - 1)) * NC] = p;
      }
    }
    march_sync<0, NTA>();
    for (int m = 0; m <= last_m; ++m) {
      const int t = m * C + warp;
      // ---- phase 1
      if (bulk && leader && !(gone & 2)) fetch(1, m);
      gone = *lost;
      if (t < nc1) {
        double wv[NV];
#pragma unroll
        for (int n = 0; n < NV; ++n) wv[n] = wb[n * VS + (n & 1 ? a1 : a0)];
        double a, b;  // psf(l), psf(l + 1)
        if (t <= 2) {
          a = psr[t * NC];
          b = psr[((t - 1) & (RP - 1)) * NC];
        } else {
          // psf(i) = psf(i+1) - grav rho(i) dx(i) from the top, in the
          // reference's order; every warp sums down from the last level of
          // the previous chunk
          const int t0 = m == 0 ? 2 : m * C - 1;
          a = psr[(t0 & (RP - 1)) * NC];
          b = a;
          for (int s = t0 + 1; s <= t; ++s) {
            const int i = nc1 - 1 - s;
            const double gg = i < is && g.bc[0] == CANOE_BC_REFLECT ? -grav : grav;
            const double x = gg * wb[at0(C - 1 - (s - m * C))];
            b = a;
            a = a - x * sdx[i];
          }
          psr[(t & (RP - 1)) * NC] = a;
        }
        const double pv = fabs(a - b) < 1.E-6 ? 0.5 * (a + b) : qdiv(a - b, log(qdiv(a, b)));
        double feps = 1.;
#pragma unroll
        for (int n = 1; n <= NY; ++n)
          if (n <= th.nvapor) feps += wv[n] * th.inv_mu_ratio_m1[n - 1];
        const double gmv = th.rd * feps;
        gmr[wrap(bq + warp) * NC] = gmv;
        R *qo = qb + wrap(bq + warp) * NV * NC;
        qo[0] = R(qdiv(wv[S::IPR], wv[0] * gmv));
        qo[S::IPR * NC] = R(wv[S::IPR] - pv);
#pragma unroll
        for (int n = 1; n < NV - 1; ++n) qo[n * NC] = R(wv[n]);
        double *ro = rawb + wrap(bq + warp) * NR * NC;
        ro[0] = wv[0];
        ro[NC] = wv[S::IPR];
        if constexpr (NR > 2) ro[2 * NC] = wv[S::IVX];
        if constexpr (NR > 3) {
          ro[3 * NC] = wv[S::IVY];
          ro[4 * NC] = wv[S::IVZ];
        }
      }
      march_sync<1, NTP>();
      // ---- phase 2: cells t - 2, by (variable, group of four cells)
      {
      // the warp's group of four cells and its first variable; its next ones
      // are four apart
      constexpr int SG = C / 4;
      const int e0 = 4 * (warp % SG), n0 = warp / SG;
      // q of the levels from two below the group's last cell to two above its
      // first
      const R *qp[8];
      R *fp[4];
#pragma unroll
      for (int y = 0; y < 8; ++y) qp[y] = qb + (wrap(bq + e0 - 4 + y) * NV + n0) * NC;
#pragma unroll
      for (int e = 0; e < 4; ++e) fp[e] = fb + (wrap(bq + e0 + e - 2) * NV + n0) * NC;
      R *hp = wrb + (e0 * NV + n0) * NC;
      const bool outflow = g.bc[0] == CANOE_BC_OUTFLOW || g.bc[1] == CANOE_BC_OUTFLOW;
#pragma unroll
      for (int it = 0; it < (NV + 3) / 4; ++it) {
        const int n = n0 + 4 * it;
        if (n >= NV) break;
        R qv[8];
#pragma unroll
        for (int y = 0; y < 8; ++y) qv[y] = qp[y][4 * it * NC];
        if (outflow && (n == 0 || n == S::IPR)) {
          // density and pressure of outflow ghosts take the transformed
          // values of the first / last interior cell
          // (change_to_temperature.cpp:114-127)
          for (int y = 0; y < 8; ++y) {
            int d = e0 - 4 + y;
            if (g.bc[0] == CANOE_BC_OUTFLOW) d = min(d, nc1 - 4 - m * C);
            if (g.bc[1] == CANOE_BC_OUTFLOW) d = max(d, 3 - m * C);
            if (d != e0 - 4 + y && d >= -4 && d < C) {
              const R v = qb[(wrap(bq + d) * NV + n) * NC];
#pragma unroll
              for (int z = 0; z < 8; ++z)
                if (z == y) qv[z] = v;
            }
          }
        }
        R lo[4], hi[4];
        if constexpr (RECON == CANOE_RECON_PPM) {
          R sl[6], fc[5];  // slopes of qv[1 .. 6]; faces below qv[1 .. 5]
#pragma unroll
          for (int y = 0; y < 6; ++y) sl[y] = ppm_slope(qv[y + 2], qv[y + 1], qv[y]);
#pragma unroll
          for (int y = 0; y < 5; ++y) fc[y] = ppm_face(qv[y + 2], qv[y + 1], sl[y + 1], sl[y]);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            lo[e] = fc[e + 1];
            hi[e] = fc[e];
            ppm_limit(qv[e + 2], lo[e], hi[e]);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            // cell of the group, kept inside is - 1 .. ie + 1
            const int c = max(min(nc1 - 1 - (m * C + e0 + e - 2), ie + 1), is - 1);
            plm_cell_nu(qv[e + 3], qv[e + 2], qv[e + 1], R(g.x1v[c - 1]), R(g.x1v[c]),
                        R(g.x1v[c + 1]), R(g.x1f[c]), R(g.x1f[c + 1]), lo[e], hi[e]);
          }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          fp[e][4 * it * NC] = lo[e];
          hp[(e * NV + 4 * it) * NC] = hi[e];
        }
      }
      }
      march_sync<1, NTP>();
      // ---- phase 3: face t - 3, between the cells t - 2 (left) and t - 3
      if (t >= 5 && t < nc1) {
        R *fo = fb + wrap(bq + warp - 3) * NV * NC;
        R wl[NV], wr[NV], fx[NV];
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          wl[n] = wrb[(warp * NV + n) * NC];
          wr[n] = fo[n * NC];
        }
        const double pf = psr[((t - 3) & (RP - 1)) * NC];
        const double gamma = qsqrt(gmr[wrap(bq + warp - 3) * NC] * gmr[wrap(bq + warp - 2) * NC]);
        if constexpr (PERT) {
          R pr = wr[S::IPR], pl = wl[S::IPR];
          if (R(pf) + pr < R(0)) pr = R(0);
          if (R(pf) + pl < R(0)) pl = R(0);
          wr[S::IPR] = pr;
          wl[S::IPR] = pl;
          wr[0] = qdiv(R(pf) + pr, wr[0] * R(gamma));
          wl[0] = qdiv(R(pf) + pl, wl[0] * R(gamma));
        } else {
          double pr = wr[S::IPR] + pf;
          if (pr < 0.) pr = pf;
          wr[S::IPR] = pr;
          wr[0] = qdiv(pr, wr[0] * gamma);
          double pl = wl[S::IPR] + pf;
          if (pl < 0.) pl = pf;
          wl[S::IPR] = pl;
          wl[0] = qdiv(pl, wl[0] * gamma);
        }
        if constexpr (GEO) {
          if constexpr (PERT) hllc_pert<R, NY, 0, true>(mx, wl, wr, R(pf), fx, R(cosc));
          else hllc<R, NY, 0, true>(mx, wl, wr, fx, R(cosc));
          const R ty = fx[S::IVY], tz = fx[S::IVZ];
          fx[S::IVY] = ty + tz * R(cth1);
          fx[S::IVZ] = tz + ty * R(cth1);
        } else if constexpr (PERT) {
          riemann_pert<R, NY, RS, 0>(mx, wl, wr, R(pf), fx);
        } else {
          riemann<R, NY, RS, 0>(mx, wl, wr, fx);
        }
#pragma unroll
        for (int n = 0; n < NV; ++n) fo[n * NC] = fx[n];
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // wR's place takes w
      march_sync<0, NTA>();
      // ---- phase 4: row i, level t - 4
      if (bulk && leader && !(gone & 1) && m < last_m) fetch(0, m + 1);
      gone = *lost;
      if (t >= 5 && t <= nc1) {
        const int i = nc1 - 1 - (t - 4);
        const double *rd = rawb + wrap(bq + warp - 3) * NR * NC;  // cell i - 1
        const double *ru = rawb + wrap(bq + warp - 4) * NR * NC;  // cell i
        const R *qd = qb + wrap(bq + warp - 3) * NV * NC, *qu = qb + wrap(bq + warp - 4) * NV * NC;
        if (i <= ie) {
          const R *flo = fb + wrap(bq + warp - 4) * NV * NC;
          const R *fhi = fb + wrap(bq + warp - 5) * NV * NC;
          const double rho = ru[0], v1 = NR > 2 ? ru[2 * NC] : (double)qu[S::IVX * NC];
          const double gsrc = wght * rho * grav;
          const double plo = psr[((t - 4) & (RP - 1)) * NC], phi = psr[((t - 5) & (RP - 1)) * NC];
          double dv[NV], dd, ra = 1.;  // diagonal of the scaled row, its area ratio
          if constexpr (GEO) {
            const double d2 = tab(kTabDx2A, k, j), d3 = tab(kTabDx3A, k, j);
            const double sc = sinc, cs = cosc;
            const double xv = g.x1v[i], df = sdx[i];
            const double a1m = d2 * d3 * g.x1f[i] * g.x1f[i] * sc;
            const double a1p = d2 * d3 * g.x1f[i + 1] * g.x1f[i + 1] * sc;
            const double vol = df * d2 * d3 * xv * xv * sc;
            const Recip<double> ivol(vol), ixv(xv), ia(a1m);
            const double a2m = xv * tab(kTabDx3AF2, k, j) * df;
            const double a2p = xv * tab(kTabDx3AF2, k, j + 1) * df;
            const double a3m = xv * tab(kTabDx2AF3, k, j) * df;
            const double a3p = xv * tab(kTabDx2AF3, k + 1, j) * df;
            const double v2 = NR > 3 ? ru[3 * NC] : (double)qu[S::IVY * NC];
            const double v3 = NR > 3 ? ru[4 * NC] : (double)qu[S::IVZ * NC];
            const double pr = ru[NC];
            const double v_2 = v2 + v3 * cs, v_3 = v3 + v2 * cs, sine2 = sc * sc;
            const double x_ov_rD =
                ivol.of(a2m * tab(kTabSinF2, k, j) - a2p * tab(kTabSinF2, k, j + 1));
            const double y_ov_rC =
                ivol.of(a3m * tab(kTabSinF3, k, j) - a3p * tab(kTabSinF3, k + 1, j));
            double csrc[3];
            csrc[0] = wght * ixv.of(2.0 * pr + rho * (v2 * v_2 + v3 * v_3));
            csrc[1] = wght * (-x_ov_rD * (pr + rho * v3 * v3 * sine2) - ixv.of(rho * v1 * v_2));
            csrc[2] = wght * (-y_ov_rC * (pr + rho * v2 * v2 * sine2) - ixv.of(rho * v1 * v_3));
#pragma unroll
            for (int n = 0; n < NV; ++n) {
              double dfl = a1p * (double)fhi[n * NC] - a1m * (double)flo[n * NC];
              if (PERT && n == S::IVX) dfl += a1p * phi - a1m * plo;
              double v = -ivol.of(wght * dfl);
              if (n == S::IVX) v += csrc[0];
              if (n == S::IVY) v += csrc[1];
              if (n == S::IVZ) v += csrc[2];
              if (n == S::IVX) v += gsrc;
              if (n == S::IPR) v += gsrc * v1;
              dv[n] = v;
            }
            dd = idt * ia.of(2. * vol);
            ra = ia.of(a1p);
          } else {
            const double idx = qdiv(1., sdx[i]);
#pragma unroll
            for (int n = 0; n < NV; ++n) {
              double d = ((double)fhi[n * NC] - (double)flo[n * NC]) * idx;
              if (PERT && n == S::IVX) d += (phi - plo) * idx;
              double v = -(wght * d);
              if (n == S::IVX) v += gsrc;
              if (n == S::IPR) v += gsrc * v1;
              dv[n] = v;
            }
            dd = idt * (2. * sdx[i]);
          }
#pragma unroll
          for (int n = 0; n < NV; ++n) dv[n] = db[n * VS + (n & 1 ? a1 : a0)] + dv[n];
          double dsum = dv[0];
#pragma unroll
          for (int n = 1; n <= NY; ++n) dsum += dv[n];
          double *ro = rb + wrap(bq + warp) * NRH * NC;
          ro[0] = dsum * dd;
          ro[NC] = dv[S::IVX] * dd;
          if constexpr (N == 5) {
            ro[2 * NC] = dv[S::IVY] * dd;
            ro[3 * NC] = dv[S::IVZ] * dd;
          }
          ro[(N - 1) * NC] = dv[S::IPR] * dd;
          ro[N * NC] = dd;
          if constexpr (GEO) ro[(N + 1) * NC] = ra;
          double *so = scr + (int64_t)(i - is) * ND * NC + lane;
#pragma unroll
          for (int n = 1; n <= NY; ++n) so[(NT + n - 1) * NC] = dv[n];
          if constexpr (NT > 0) {
            so[0] = dv[S::IVY];
            so[NC] = dv[S::IVZ];
          }
          if constexpr (NY > 0) so[(NT + NY) * NC] = dsum;
        }
        // |A| at face i and J of cell i - 1
        {
          const double gm1 = mx.gm1;
          // the FP32 path evaluates them in FP32: its velocities and mass
          // fractions are rounded in q already
          using W = typename std::conditional<GEO, double, R>::type;
          W wu[NV], wd[NV];
#pragma unroll
          for (int n = 1; n < NV - 1; ++n) {
            wd[n] = qd[n * NC];
            wu[n] = qu[n * NC];
          }
          wd[0] = W(rd[0]);
          wu[0] = W(ru[0]);
          wd[S::IPR] = W(rd[NC]);
          wu[S::IPR] = W(ru[NC]);
          if constexpr (GEO) {
            // velocities projected to the local frame, in FP64
            if constexpr (NR > 3) {
#pragma unroll
              for (int n = 0; n < 3; ++n) {
                wd[S::IVX + n] = rd[(2 + n) * NC];
                wu[S::IVX + n] = ru[(2 + n) * NC];
              }
            }
            wd[S::IVY] += wd[S::IVZ] * cosc;
            wu[S::IVY] += wu[S::IVZ] * cosc;
            wd[S::IVZ] *= sinc;
            wu[S::IVZ] *= sinc;
          }
          R *ao = ajb + wrap(bq + warp) * NAJ * NC;
          M<N> mt;
          jacobian<N, NY, R>(mt, gm1, wd);  // its first row is 0 1 0 ..
#pragma unroll
          for (int e = 0; e < N * (N - 1); ++e) ao[(N * N + e) * NC] = R(mt.a[1 + e / N][e % N]);
          abs_jacobian<N, NY, R>(mt, mx, gm1, wd, wu);
#pragma unroll
          for (int e = 0; e < N * N; ++e) ao[e * NC] = R(mt.a[e / N][e % N]);
        }
      }
      bq = wrap(bq + C);
      march_sync<0, NTA>();
    }
  } else {
    // ---- elimination of the rows of chunk m, while the level warps work on
    // chunk m + 1; this warp takes every second row
    const int e2 = warp - C;
    double *hg = sm2 + P::hg + lane;
    auto row = [&](int t) {
      if (t < 7 || t > nc1) return;  // rows ie .. is
      const int i = nc1 - 1 - (t - 4);
      double D[N][N], b[N][N], c[N][N], v[N];
      march_blocks<N, GEO, RR, NRH, NAJ>(ajb, rb, t, i == is, i == ie, grav * wght, D, b, c, v);
      if (i != ie) {
        // H, g of the row above, from the other warp
        if (e2 == 0) march_sync<2, 64>();
        else march_sync<3, 64>();
        march_above<N>(hg, D, c, v);
      }
      double h[NH];
      double *so = scrh + (int64_t)(i - is) * NH * NC + lane;
      auto keep = [&](double *to) {
#pragma unroll
        for (int e = 0; e < NH; ++e) to[e * NC] = h[e];
      };
      auto arrive = [&] {
        if (t >= nc1) return;
        if (e2 == 0) march_arrive<3, 64>();
        else march_arrive<2, 64>();
      };
      if constexpr (N == 3) {
        // adjugate over the determinant, as inv(M<3>)
        double K[3][3];
        K[0][0] = D[1][1] * D[2][2] - D[1][2] * D[2][1];
        K[1][0] = D[1][2] * D[2][0] - D[1][0] * D[2][2];
        K[2][0] = D[1][0] * D[2][1] - D[1][1] * D[2][0];
        K[0][1] = D[0][2] * D[2][1] - D[0][1] * D[2][2];
        K[1][1] = D[0][0] * D[2][2] - D[0][2] * D[2][0];
        K[2][1] = D[0][1] * D[2][0] - D[0][0] * D[2][1];
        K[0][2] = D[0][1] * D[1][2] - D[0][2] * D[1][1];
        K[1][2] = D[0][2] * D[1][0] - D[0][0] * D[1][2];
        K[2][2] = D[0][0] * D[1][1] - D[0][1] * D[1][0];
        const double id = Recip<double>(D[0][0] * K[0][0] + D[0][1] * K[1][0] + D[0][2] * K[2][0]).r;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
#pragma unroll
          for (int y = 0; y < 3; ++y)
            h[3 * x + y] = (K[x][0] * b[0][y] + K[x][1] * b[1][y] + K[x][2] * b[2][y]) * id;
          h[9 + x] = (K[x][0] * v[0] + K[x][1] * v[1] + K[x][2] * v[2]) * id;
        }
      } else {
        double rp[N];
        const bool good = march_factor(D, rp);
        march_sweeps(D, rp, b, v, h);
        if (!__all_sync(~0u, good)) {
          march_row_pivoted<GEO, RR, NRH, NAJ>(ajb, rb, hg, so, t, i == is, i == ie, grav * wght);
          __syncwarp();
          arrive();
          return;
        }
      }
      keep(hg);
      arrive();
      keep(so);
    };
    auto arrived = [&](int q, int m) {  // w (q = 0) or du (1) of chunk m
      if (e2 == q) wait(q, m & 1);
    };
    auto request = [&](int q, int m) {
      if (!bulk && e2 == q && __all_sync(~0u, ok)) fetch(q, m);
    };
    request(0, 0);
    arrived(0, 0);
    march_sync<0, NTA>();
    for (int m = -1; m <= last_m; ++m) {
      if (m < last_m) request(1, m + 1);
      if (m >= 0)
        for (int p = e2; p < C - 2; p += 2) row(m * C + p);
      // all but the chunk's last two rows are done before the next chunk's
      // rows are formed in their places
      if (m < last_m) {
        arrived(1, m + 1);
        march_sync<0, NTA>();  // phase 3 of chunk m + 1
        if (m + 2 <= last_m) request(0, m + 2);
      }
      if (m >= 0) row(m * C + C - 2 + e2);
      if (m < last_m) {
        if (m + 2 <= last_m) arrived(0, m + 2);
        march_sync<0, NTA>();  // phase 4 of chunk m + 1
      }
    }
  }

  // ---- way back up in chunks of four levels from 2 + 4 q (the first starts
  // in the ghost level is - 1: boxes start at even levels).  Phase q: the
  // elimination warp finds x of chunk q + 1, the level warps update chunk q,
  // chunk q - 1 is written out and chunk q + 2 fetched.
  asm volatile("fence.proxy.async;" ::: "memory");  // H, g and the buffers, before bulk copies
  march_sync<0, NTA>();
  // a tile that lost a copy on the way down does not go back up; no wait comes
  // between the two barriers, so that all warps read the same
  const bool down = *lost == 0;
  march_sync<0, NTA>();
  const int nq = down ? (ie - 2) / UP + 1 : -2;
  double *hb = sm + P::hx(bulk ? UP : UO), *xs = hb + 3 * UP * NH * NC + lane;
  const int UVS = NC * (bulk ? UP : UO), UC = UVS * NV, SC = UVS * NY;
  double *ub = sm, *spb = sm + 4 * UC;
  constexpr int HC = UP * NH * NC;
  // H and g of chunk q, by the lane 0 that waits for them
  auto fetch_h = [&](int q) {
    if (q >= nq || !ok) return;
    const int lo = 2 + UP * q, i0 = max(lo, is), n = min(lo + UP - 1, ie) - i0 + 1;
    arm(MH + q % 3, q / 3 & 1, n * NH * NC * 8);
    bulk_g2s(hb + (q % 3) * HC + (i0 - lo) * NH * NC, scrh + (int64_t)(i0 - is) * NH * NC,
             n * NH * NC * 8, mbar + MH + q % 3);
  };
  // u and the species of chunk q, by the whole warp that waits for them; what
  // the level warps read from scratch themselves starts towards L2
  auto fetch_u = [&](int q) {
    if (q >= nq || !(bulk ? ok : __all_sync(~0u, ok))) return;
    const int lo = 2 + UP * q, i0 = max(lo, is), n = min(lo + UP - 1, ie) - i0 + 1;
    uint64_t *mb = mbar + MU + (q & 3);
    double *du_ = ub + (q & 3) * UC, *ds = spb + (q & 3) * SC;
    if (lane == 0) {
      arm(MU + (q & 3), q >> 2 & 1, (UC + SC) * 8);
      if (bulk) {
        march_tma_load(du_, &maps.u, lo, j0, k0, 0, pan, mb);
        if constexpr (NY > 0) march_tma_load(ds, &maps.sp, lo, j0, k0, 1, pan, mb);
      }
      if constexpr (ND > 0)
        bulk_prefetch_l2(scr + (int64_t)(i0 - is) * ND * NC, n * ND * NC * 8);
      if (stage != 0) bulk_prefetch_l2(u1 + (int64_t)(i0 - is) * NV * NC, n * NV * NC * 8);
    }
    if (!bulk) {
      __syncwarp();
      pairs(du_, &maps.u, 0, NV, lo, UO, mb);
      pairs(ds, &maps.sp, 1, NY, lo, UO, mb);
    }
  };
  if (warp < C) {
    // C = 8: two warps per level, one for the densities, one for momenta and
    // energy; C = 4: a warp does both
    constexpr int HALVES = C / UP;
    const int lev = warp / HALVES, half = HALVES == 2 ? warp % 2 : -1;
    constexpr int N0 = NY > 0 ? 2 * NY + 2 : 1;  // values of the densities' half
    constexpr int N1 = NT + 4;                        // and of the momenta and energy
    constexpr int NL = HALVES == 2 ? (N0 > N1 ? N0 : N1) : N0 + N1;
    constexpr int OFF1 = HALVES == 2 ? 0 : N0;
    double cur[NL], nxt[NL];
    // scratch of the update: du and the sum of the densities, then u1
    auto load_scr = [&](int q, double *v) {
      const int i = 2 + UP * q + lev;
      if (q >= nq || i < is || i > ie) return;
      const double *si = scr + (int64_t)(i - is) * ND * NC + lane;
      const double *s1 = u1 + (int64_t)(i - is) * NV * NC + lane;
      if (half != 1) {
        constexpr int NM = N0 - NY - 1;  // du of the species and the sum
#pragma unroll
        for (int n = 0; n < NM; ++n) v[n] = si[(NT + n) * NC];
        if (stage != 0)
#pragma unroll
          for (int n = 0; n <= NY; ++n) v[NM + n] = s1[n * NC];
      }
      if (half != 0) {
#pragma unroll
        for (int n = 0; n < NT; ++n) v[OFF1 + n] = si[n * NC];
        if (stage != 0)
#pragma unroll
          for (int n = 0; n < 4; ++n) v[OFF1 + NT + n] = s1[(S::IVX + n) * NC];
      }
    };
    // places of this warp's level in the boxes of the even / odd variables (the
    // species' first is an odd one); without boxes a thread writes back one
    // level of one column, of every NTP / (UP * 32)-th variable
    const int b0 = bulk ? march_box<UP>(0, lane, lev) : lp * UO + lev + par;
    const int b1 = bulk ? b0 : lp * UO + lev + (par ^ psv);
    const int s0 = bulk ? march_box<UP>(0, lc, lev) : b1, s1 = bulk ? s0 : b0;
    constexpr int ZN = NTP / (UP * NC);
    const int ro = threadIdx.x % UP, rc = threadIdx.x / UP % NC, rn = threadIdx.x / (UP * NC);
    const int rp = bulk ? 0 : pcol(rc);
    load_scr(0, cur);
    for (int q = -1; q <= nq; ++q) {
      if (!bulk) {
        const int l = 2 + UP * (q - 1) + ro;
        if (q >= 1 && ((mine >> rc) & 1) && l >= is && l <= ie && !*lost) {
          const double *src = ub + ((q - 1) & 3) * UC + rp * UO + ro;
          const int64_t at = colb[rc] + l;
#pragma unroll
          for (int z = 0; z < (NV + ZN - 1) / ZN; ++z) {
            const int n = rn + z * ZN;
            if (n < NV) u[n * g.sv + at] = src[n * UVS + (int)((n * g.sv + colb[rc]) & 1)];
          }
        }
      }
      if (q >= 0) load_scr(q + 1, nxt);
      const int i = 2 + UP * q + lev;
      if (q >= 0 && q < nq && i >= is && i <= ie) {
        double *uc = ub + (q & 3) * UC;
        const double *xi = xs + (q & 1) * UP * N * NC + lev * N * NC;
        double *su = u1 + (int64_t)(i - is) * NV * NC + lane;
        // slots n0 .. n0 + NN - 1: their increments dv, and u1 as loaded (uold)
        auto update = [&](auto nn, int n0, const double *dv, const double *uold) {
          constexpr int NN = decltype(nn)::value;
          double uo[NN];
#pragma unroll
          for (int n = 0; n < NN; ++n) uo[n] = uc[(n0 + n) * UVS + ((n0 + n) & 1 ? b1 : b0)];
#pragma unroll
          for (int n = 0; n < NN; ++n) {
            if (stage == 0) su[(n0 + n) * NC] = uo[n];
            const double s = st.g1 * uo[n] + st.g2 * (stage == 0 ? uo[n] : uold[n]);
            if (on) uc[(n0 + n) * UVS + ((n0 + n) & 1 ? b1 : b0)] = s + dv[n];
          }
        };
        if (half != 1) {
          // species correction (forward_backward.hpp:101-124)
          double dv[NY + 1];
          const double x0 = xi[0];
          dv[0] = x0;
          if constexpr (NY > 0) {
            const double dens = x0 - cur[NY];
            const double *wc = spb + (q & 3) * SC;
#pragma unroll
            for (int n = 1; n <= NY; ++n) dv[n] = wc[(n - 1) * UVS + (n & 1 ? s0 : s1)];
#pragma unroll
            for (int n = 1; n <= NY; ++n) {
              dv[n] = cur[n - 1] + dens * dv[n];
              dv[0] -= dv[n];
            }
          }
          update(std::integral_constant<int, NY + 1>(), 0, dv, cur + (NY > 0 ? NY + 1 : 0));
        }
        if (half != 0) {
          const double *cm = cur + OFF1;
          const double dv[4] = {xi[NC], NT ? cm[0] : xi[2 * NC], NT ? cm[1] : xi[3 * NC],
                                xi[(N - 1) * NC]};
          update(std::integral_constant<int, 4>(), S::IVX, dv, cm + NT);
        }
      }
      if (q >= 0) {
#pragma unroll
        for (int z = 0; z < NL; ++z) cur[z] = nxt[z];
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      march_sync<0, NTA>();
    }
  } else if (warp == C + 1) {
    // the copies of u and the species
    fetch_u(0);
    int gone = 0;  // x of chunk q - 1 was lost in the phase before the last
    for (int q = -1; q <= nq; ++q) {
      if (lane == 0) {
        if (bulk && q >= 1 && ok && !gone)
          march_tma_store(&maps.u, 2 + UP * (q - 1), j0, k0, 0, pan, ub + ((q - 1) & 3) * UC);
        // chunk q - 2 has been read out: its place takes chunk q + 2
        asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
      }
      __syncwarp();
      fetch_u(q + 2);
      // for the level warps of the next phase
      if (q + 1 < nq) wait(MU + ((q + 1) & 3), ((q + 1) >> 2) & 1);
      gone = *lost;
      march_sync<0, NTA>();
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  } else {
    double x[N];
#pragma unroll
    for (int a = 0; a < N; ++a) x[a] = 0.;
    if (lane == 0)
      for (int q = 0; q < 3; ++q) fetch_h(q);
    for (int q = -1; q <= nq; ++q) {
      if (q + 1 < nq) {
        wait(MH + (q + 1) % 3, (q + 1) / 3 & 1);
        double *xo = xs + ((q + 1) & 1) * UP * N * NC;
        const double *hc = hb + (q + 1) % 3 * HC + lane;
#pragma unroll
        for (int o = 0; o < UP; ++o) {
          const int i = 2 + UP * (q + 1) + o;
          // (levels outside the column hold what the buffer held: not used)
          const bool in = i >= is && i <= ie;
          double y[N];
#pragma unroll
          for (int a = 0; a < N; ++a) y[a] = hc[(o * NH + N * N + a) * NC];
#pragma unroll
          for (int e = 0; e < N; ++e)
#pragma unroll
            for (int a = 0; a < N; ++a) y[a] += hc[(o * NH + N * a + e) * NC] * x[e];
#pragma unroll
          for (int a = 0; a < N; ++a) {
            x[a] = in ? y[a] : x[a];
            xo[(o * N + a) * NC] = x[a];
          }
        }
        __syncwarp();
        if (lane == 0) fetch_h(q + 4);
      }
      march_sync<0, NTA>();
    }
  }
  if (*lost)  // copies still in flight get a second bounded wait
    for (int q = 0; q < NMB; ++q)
      if (armed[q]) mbar_wait(mbar + q, armed[q] - 1);
}

// the tensor map encoder of the driver (null where there is none)
inline PFN_cuTensorMapEncodeTiled march_encoder() {
  static const PFN_cuTensorMapEncodeTiled f = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &r) != cudaSuccess ||
        r != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      p = nullptr;
    }
    return (PFN_cuTensorMapEncodeTiled)p;
  }();
  return f;
}

inline bool march_available() { return march_encoder() != nullptr; }

// launcher for one NY (instantiated in march_ny*.cu)
template <int NY, int N>
int run_x1march(const Geom &g, const canoe_thermo_t &th, int recon, int rs, int prec,
                const double *w, const double *du, double *u, const double *dtp, const Stage &s,
                int stage, cudaStream_t st) {
  const bool ppm = recon == CANOE_RECON_PPM, hllc = rs == CANOE_RSOLVER_HLLC;
  const bool f32 = prec == CANOE_FP32_PERTURBATION;
  const int npan = g.npanel > 1 ? g.npanel : 1;
  const MarchTile tl = march_tile(g.nx1, g.nx2, g.nx3);
  Geom gg = g;
  MarchMaps maps{};
  auto al16 = [](const void *p) { return ((uintptr_t)p & 15) == 0; };
  if (!(al16(w) && al16(du) && al16(u))) {
    set_error("the column march copies from 16-byte aligned arrays");
    return CANOE_ERR_ARG;
  }
  gg.bulk = g.nc1 % 2 == 0;
  // box of `lev` levels x the tile's columns x nn variables
  auto encode = [&](CUtensorMap &m, const double *p, int lev, int nn) {
    const cuuint64_t dim[5] = {(cuuint64_t)g.nc1, (cuuint64_t)g.nc2, (cuuint64_t)g.nc3,
                               (cuuint64_t)(5 + NY), (cuuint64_t)npan};
    const cuuint64_t pst = npan > 1 ? (cuuint64_t)g.pstride : (cuuint64_t)((5 + NY) * g.sv);
    const cuuint64_t str[4] = {(cuuint64_t)g.nc1 * 8, (cuuint64_t)g.sk * 8, (cuuint64_t)g.sv * 8,
                               pst * 8};
    const cuuint32_t box[5] = {(cuuint32_t)lev, (cuuint32_t)tl.bj, (cuuint32_t)tl.bk,
                               (cuuint32_t)nn, 1};
    const cuuint32_t one[5] = {1, 1, 1, 1, 1};
    if (gg.bulk)
      return march_encoder()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 5, const_cast<double *>(p), dim,
                             str, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             lev == 8 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    // rows of two columns (the array's last column, a ghost, may be left out)
    const cuuint64_t dim2[2] = {2 * (cuuint64_t)g.nc1, (cuuint64_t)npan * pst / g.nc1 / 2};
    const cuuint64_t str2[1] = {(cuuint64_t)g.nc1 * 16};
    const cuuint32_t box2[2] = {(cuuint32_t)lev + 2, (cuuint32_t)tl.bj / 2};
    return march_encoder()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<double *>(p), dim2,
                           str2, box2, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  auto go = [&](auto kern, const auto &mx, int C, size_t smem) -> int {
    if (!march_encoder() ||
        !(encode(maps.w, w, C, 5 + NY) && encode(maps.du, du, C, 5 + NY) &&
          encode(maps.u, u, kMarchUp, 5 + NY) && encode(maps.sp, w, kMarchUp, NY > 0 ? NY : 1))) {
      set_error("cuTensorMapEncodeTiled failed");
      return CANOE_ERR_CUDA;
    }
    if (int rc = ensure_smem((const void *)kern, smem)) return rc;
    kern<<<(unsigned)(tl.nj * tl.nk * npan), (C + 2) * 32, smem, st>>>(
        gg, th, mx, tl, maps, w, du, u, g.march, g.march_u1, dtp, s, stage);
    CB_CUDA(cudaGetLastError());
    return 0;
  };
#define CB_MK(RC, RSV, R, GEO)                                                        \
  (g.nc1 % 2 && march_chunk<R>(NY, N, 1) != march_chunk<R>(NY, N, 0)                          \
       ? go(k_x1march<NY, RC, RSV, R, GEO, march_chunk<R>(NY, N, 1), N>, make_mix<R>(th),   \
            march_chunk<R>(NY, N, 1),                                                      \
            MarchSmem<5 + NY, march_chunk<R>(NY, N, 1), R, GEO, N>::bytes(g.nc1))          \
       : go(k_x1march<NY, RC, RSV, R, GEO, march_chunk<R>(NY, N, 0), N>, make_mix<R>(th),   \
            march_chunk<R>(NY, N, 0),                                                      \
            MarchSmem<5 + NY, march_chunk<R>(NY, N, 0), R, GEO, N>::bytes(g.nc1)))
  if (g.shell) {
    if constexpr (NY == 0) {
      if (!hllc) {
        set_error("the cubed-sphere panel uses the HLLC solver");
        return CANOE_ERR_UNSUPPORTED;
      }
      if (ppm) return f32 ? CB_MK(3, 1, float, 1) : CB_MK(3, 1, double, 1);
      return f32 ? CB_MK(2, 1, float, 1) : CB_MK(2, 1, double, 1);
    } else {
      set_error("the cubed-sphere panel is dry");
      return CANOE_ERR_UNSUPPORTED;
    }
  }
  if (ppm) {
    if (hllc) return f32 ? CB_MK(3, 1, float, 0) : CB_MK(3, 1, double, 0);
    return f32 ? CB_MK(3, 0, float, 0) : CB_MK(3, 0, double, 0);
  }
  if (hllc) return f32 ? CB_MK(2, 1, float, 0) : CB_MK(2, 1, double, 0);
  return f32 ? CB_MK(2, 0, float, 0) : CB_MK(2, 0, double, 0);
#undef CB_MK
}

}  // namespace cb
