// column.cu -- dispatch of the x1 pencil kernel and of the column march over
// the species count.
#include <mutex>
#include <set>

#include "march.cuh"

namespace cb {

#define CB_DECL(NY)                                                                \
  extern template int run_x1col<NY>(const Geom &, const canoe_thermo_t &, int, int, \
                                    int, int, int, const double *, double *, double *, \
                                    double *, const double *, const Stage &, int,   \
                                    double *, cudaStream_t);
CB_DECL(0)
CB_DECL(1)
CB_DECL(2)
CB_DECL(3)
CB_DECL(6)
#undef CB_DECL
#define CB_DECL(NY, N)                                                                \
  extern template int run_x1march<NY, N>(const Geom &, const canoe_thermo_t &, int, int, \
                                         int, const double *, const double *, double *, \
                                         const double *, const Stage &, int, cudaStream_t);
#define CB_DECL2(NY) CB_DECL(NY, 3) CB_DECL(NY, 5)
CB_DECL2(0)
CB_DECL2(1)
CB_DECL2(2)
CB_DECL2(3)
CB_DECL2(6)
#undef CB_DECL2
#undef CB_DECL

// tiles of a march that shared memory lets an SM hold at once
template <int NY, typename R, int N, int GEO>
static int march_resident(int nc1, int per_sm, int reserved) {
  const size_t b = nc1 % 2 ? MarchSmem<5 + NY, march_chunk<R>(NY, N, 1), R, GEO, N>::bytes(nc1)
                           : MarchSmem<5 + NY, march_chunk<R>(NY, N, 0), R, GEO, N>::bytes(nc1);
  constexpr int kStatic = 1024;  // the kernel's barriers and column table
  return (int)(per_sm / (b + kStatic + reserved));
}

// whether the fused x1 stage of a block marches, its scratch granted
static bool march_serves(const Geom &g, const canoe_thermo_t &th, int flag, int prec) {
  const int64_t ncol = (int64_t)g.nx2 * g.nx3 * (g.npanel > 1 ? g.npanel : 1);
  const bool lines = line_solve_on(g, flag, 1) || line_solve_on(g, flag, 2);
  // what the march provides: the x1 solve between walls, on the hydrostatic
  // decomposition, with du initialised by an x2 pass
  if (!(flag & 1) || lines || g.bc[0] == CANOE_BC_PERIODIC || th.grav == 0. || !g.f2) return false;
  const int n = flag & 8 ? 5 : 3;
  const bool f32 = prec == CANOE_FP32_PERTURBATION;
  const int least = n == 5 ? kMarchMinCols5 : (f32 ? kMarchMinCols32 : kMarchMinCols64);
  if (ncol < least || !march_available()) return false;
  if (n == 3 && !g.shell) {
    const int sms = sm_count();
    int dev = 0, per_sm = 0, reserved = 0, resident = 0;
    if (sms < 1 || cudaGetDevice(&dev) ||
        cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) ||
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev)) {
      cudaGetLastError();
      return false;
    }
#define CB_RES(NY)                                                               \
  case NY:                                                                       \
    resident = f32 ? march_resident<NY, float, 3, 0>(g.nc1, per_sm, reserved)    \
                   : march_resident<NY, double, 3, 0>(g.nc1, per_sm, reserved);  \
    break;
    switch (th.ny) { CB_RES(0) CB_RES(1) CB_RES(2) CB_RES(3) CB_RES(6) }
#undef CB_RES
    if (resident < 1) return false;
    const MarchTile t = march_tile(g.nx1, g.nx2, g.nx3);
    const int64_t tiles = (int64_t)t.nj * t.nk;
    if (resident == 1) {
      const int64_t rounds = (tiles + sms - 1) / sms;
      // (columns so long that eight variables fill an SM too are the other
      // kernel's worst: 64x54 of 330 levels 2676 and 1265 us in FP32)
      if (th.ny > 3 && ncol * 16 < least * rounds * march_round_16ths(g.nx1, f32)) return false;
    } else if (!f32 && tiles > sms && g.nx1 >= kMarchPairsLo && g.nx1 <= kMarchPairsHi &&
               ncol < kMarchMinCols64Pairs) {
      return false;
    }
  }
  // columns too long for the CTA-per-column kernel stay refused there
  return sizeof(double) * col_smem(g.nv, g.nc1, g.nx1, n, 0, 1).total <= 227 * 1024;
}

// claims with scratch whose block has not stepped, which may be given back (not
// destroyed at exit: a host's blocks may go later than the library's statics)
static std::mutex claim_mu;
static std::set<MarchClaim *> &claims = *new std::set<MarchClaim *>;

static void claim_scratch(MarchClaim &c, size_t keep_free_one_in) {
  Geom &g = *c.g;
  const int n = c.flag & 8 ? 5 : 3;
  const size_t cells = march_cells(g.nx1, g.nx2, g.nx3, g.npanel > 1 ? g.npanel : 1);
  const size_t scr = cells * (march_h(n) + march_nd(c.th->ny, n)), reg = cells * (5 + c.th->ny);
  const bool own = reg > c.u1_doubles;  // ragged tiles of long columns: u1's array is too short
  const size_t bytes = (scr + (own ? reg : 0)) * sizeof(double);
  // the first step may be captured into a graph, where other modes refuse an
  // allocation
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  size_t left = 0, all = 0;
  double *p = nullptr;
  if (cudaMemGetInfo(&left, &all) != cudaSuccess || left < bytes + all / keep_free_one_in ||
      cudaMalloc(&p, bytes) != cudaSuccess) {
    cudaGetLastError();
    p = nullptr;
  }
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (p) {
    g.march = p;
    g.march_u1 = own ? p + scr : c.u1;
  }
}

static void drop_scratch(MarchClaim &c) {
  if (c.g && c.g->march) cudaFree(c.g->march);
  if (c.g) c.g->march = c.g->march_u1 = nullptr;
}

void march_create(MarchClaim &c, Geom *g, const canoe_thermo_t *th, int flag, int prec, double *u1,
                  size_t u1_doubles) {
  c.g = g;
  c.th = th;
  c.flag = flag;
  c.u1 = u1;
  c.u1_doubles = u1_doubles;
  cudaGetDevice(&c.dev);
  c.serves = march_serves(*g, *th, flag, prec);
  if (!c.serves) return;
  std::lock_guard<std::mutex> lk(claim_mu);
  claim_scratch(c, kMarchEager);
  if (g->march) claims.insert(&c);
}

bool march_allow(MarchClaim &c, bool on) {
  std::lock_guard<std::mutex> lk(claim_mu);
  if (c.decided) return false;
  c.allowed = on;
  if (!on) {
    claims.erase(&c);
    drop_scratch(c);
  }
  return true;
}

bool march_decide(MarchClaim &c) {
  if (!c.decided) {
    std::lock_guard<std::mutex> lk(claim_mu);
    claims.erase(&c);
    if (c.serves && c.allowed && !c.g->march) claim_scratch(c, kMarchReserve);
    c.decided = true;
  }
  return c.g->march != nullptr;
}

void march_destroy(MarchClaim &c) {
  std::lock_guard<std::mutex> lk(claim_mu);
  claims.erase(&c);
  drop_scratch(c);
}

cudaError_t block_malloc(void **p, size_t bytes) {
  const cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  int dev = -1;
  bool any = false;
  cudaGetLastError();
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> lk(claim_mu);
    for (auto it = claims.begin(); it != claims.end();) {
      if ((*it)->dev == dev) {
        drop_scratch(**it);
        any = true;
        it = claims.erase(it);
      } else {
        ++it;
      }
    }
  }
  return any ? cudaMalloc(p, bytes) : e;
}

template <int N>
static int launch_x1march(const Geom &g, const canoe_thermo_t &th, int recon, int rs, int prec,
                          const double *w, const double *du, double *u, const double *dtp,
                          const Stage &s, int stage, cudaStream_t st) {
  switch (th.ny) {
    case 0: return run_x1march<0, N>(g, th, recon, rs, prec, w, du, u, dtp, s, stage, st);
    case 1: return run_x1march<1, N>(g, th, recon, rs, prec, w, du, u, dtp, s, stage, st);
    case 2: return run_x1march<2, N>(g, th, recon, rs, prec, w, du, u, dtp, s, stage, st);
    case 3: return run_x1march<3, N>(g, th, recon, rs, prec, w, du, u, dtp, s, stage, st);
    case 6: return run_x1march<6, N>(g, th, recon, rs, prec, w, du, u, dtp, s, stage, st);
    default:
      set_error("unsupported number of mass-fraction slots");
      return CANOE_ERR_UNSUPPORTED;
  }
}

int launch_x1col(const Geom &g, const canoe_thermo_t &th, int recon, int rs, int flag,
                 int prec, int mode, const double *w, double *du, double *u, double *u1,
                 const double *dtp, const Stage &s, int stage, double *fo,
                 cudaStream_t st) {
  if ((flag & 1) && mode != kColFluxOnly && g.bc[0] == CANOE_BC_PERIODIC) {
    // the cyclic solve couples the two ends (periodic_forward_backward.hpp)
    if (g.bc[1] != CANOE_BC_PERIODIC) {
      set_error("periodic x1 needs both x1 boundaries periodic");
      return CANOE_ERR_ARG;
    }
    if (g.nx1 < 3) {
      set_error("the periodic implicit x1 solve needs at least 3 levels");
      return CANOE_ERR_ARG;
    }
  }
  if (mode == kColStep && g.march)
    return flag & 8 ? launch_x1march<5>(g, th, recon, rs, prec, w, du, u, dtp, s, stage, st)
                    : launch_x1march<3>(g, th, recon, rs, prec, w, du, u, dtp, s, stage, st);
  switch (th.ny) {
    case 0: return run_x1col<0>(g, th, recon, rs, flag, prec, mode, w, du, u, u1, dtp, s, stage, fo, st);
    case 1: return run_x1col<1>(g, th, recon, rs, flag, prec, mode, w, du, u, u1, dtp, s, stage, fo, st);
    case 2: return run_x1col<2>(g, th, recon, rs, flag, prec, mode, w, du, u, u1, dtp, s, stage, fo, st);
    case 3: return run_x1col<3>(g, th, recon, rs, flag, prec, mode, w, du, u, u1, dtp, s, stage, fo, st);
    case 6: return run_x1col<6>(g, th, recon, rs, flag, prec, mode, w, du, u, u1, dtp, s, stage, fo, st);
    default:
      set_error("unsupported number of mass-fraction slots");
      return CANOE_ERR_UNSUPPORTED;
  }
}

}  // namespace cb
