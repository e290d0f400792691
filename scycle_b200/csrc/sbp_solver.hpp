// Device-side SbpOps context and the multigrid-preconditioned CG solver.
#pragma once
#include <cuda_runtime.h>

#include <memory>
#include <type_traits>
#include <vector>

#include "sbp_dev.cuh"
#include "sbp_host.hpp"

namespace scy {

const char* last_error();
long long launch_count();
void profile_enable(int on);
int profile_collect(int level, int width, double* ms, long long* launches, double* bytes);

struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  DevBuf(DevBuf&& o) noexcept : p(o.p), bytes(o.bytes) {
    o.p = nullptr;
    o.bytes = 0;
  }
  DevBuf& operator=(DevBuf&& o) noexcept {
    if (this != &o) {
      release();
      p = o.p;
      bytes = o.bytes;
      o.p = nullptr;
      o.bytes = 0;
    }
    return *this;
  }
  ~DevBuf();
  int alloc(size_t b);
  void release();
  template <typename T>
  T* as() const {
    return static_cast<T*>(p);
  }
};

// Partial sums for the deterministic grid reductions.
struct Reducer {
  DevBuf partials, counter;
  int init(int max_blocks);
};

template <typename T>
struct LevelStore {
  int Ny = 0, Nz = 0;
  DevBuf tab[2][10];  // per direction: D, R3, R4, Q, R3T, R4T, w3, w4, Hd, Hinvd
  DevBuf fld[10];     // cy, cz, m3y, m3z, wy, wz, mu, qy, rz, dinv
  DevBuf sep1[6];     // cy1, m3y1, wz1 (Ny), cz1, m3z1, wy1 (Nz) when separable
  DevBuf comp[2];     // composed interior stencils Cy (Ny x 9) and CzT (9 x Nz)
  DevBuf comp10;      // class 0's middle entries along y (LevelDev::Cy10)
  DevBuf comp17[2];   // composed whole-operator stencils Cy17 (classes x Ny x 17), CzT17 (classes x 17 x Nz)
  DevBuf cls[2];      // line classes of the full form: ycls (Nz), zcls (Ny)
  DevBuf cross;       // the cross form's coefficient planes (LevelDev::cross)
  DevBuf fullw[2];    // the full form's outer weights wy1 (Nz), wz1 (Ny) when the interior is not separable
  LevelDev<T> dev{};
  // planes: the cross form's planes where another store of this level has them (and outlives this one)
  int init(const LevelHost& h, cudaStream_t s, const T* planes = nullptr);
};

struct Transfer {
  Interp1D iy, iz;
  std::vector<int> ylo, yhi, zlo, zhi;  // fine index range feeding each coarse index
};

struct TransferDev {
  DevBuf jy, wy0, wy1, jz, wz0, wz1, ylo, yhi, zlo, zhi;
};

struct ChebCoef {
  double c1, c2;
};

template <typename T>
struct Multigrid {
  struct Work {
    DevBuf v[5];  // x ping, x pong, d, b, r
  };
  int nlev = 0, nu = 2, ncoarse = 0;
  std::vector<std::unique_ptr<LevelStore<T>>> lev;
  std::vector<Work> work;
  std::vector<TransferDev> tr;
  std::vector<std::vector<ChebCoef>> cheb;
  std::vector<double> lambda;
  DevBuf coarse_inv;
  int init(const std::vector<LevelHost>& hosts, const std::vector<Transfer>& xfer, cudaStream_t s, const T* planes0);
  int setup_smoothers(const std::vector<LevelHost>& hosts, Reducer& red, double* dscal, cudaStream_t s);
  template <typename Tin>
  int vcycle(int l, const Tin* b_in, T** x_out, cudaStream_t s);
  int coarse_first() const;
  template <typename Tin>
  int coarse_cycle(int l, const Tin* b_in, T** x_out, cudaStream_t s);
};

int build_hierarchy(const scy_grid_desc& g, const std::vector<double>& y, const std::vector<double>& z,
                    const std::vector<double>& mu, const int bc[4], std::vector<LevelHost>& hosts,
                    std::vector<Transfer>& xfer);

struct FDPrecond;

// How much of a solve a call does.  norm_ready: scal[0] already holds (in
// stream order) the sum of squares of the rhs.  resid_ready (where corrects()):
// cg_r and scal[5] the residual of u and its sum of squares besides.  enqueue: launch the residual
// and the first iteration and return without reading anything; the scalars
// scal[0], [1], [5] then say whether that was enough.  first: resume such a
// solve, with its scal[0..5] as read.
struct SolvePart {
  int norm_ready = 0, resid_ready = 0, enqueue = 0;
  const double* first = nullptr;
};

struct SbpContext {
  SbpContext();
  ~SbpContext();
  scy_grid_desc desc{};
  std::vector<double> y, z, mu;
  int bc[4] = {0, 1, 0, 1};  // R, T, L, B
  cudaStream_t stream = nullptr;
  std::vector<LevelHost> hosts;
  std::vector<Transfer> xfer;
  std::unique_ptr<LevelStore<double>> fine;
  std::unique_ptr<Multigrid<double>> mg64;
  std::unique_ptr<Multigrid<float>> mg32;
  std::shared_ptr<FDPrecond> fd;  // shared by the instances of a batch with one operator
  int separable = 0;  // metrics and mu separable: fast diagonalisation is exact up to the mu3 column
  double sep_misfit = 0.0;  // separable operators: bound on the energy norm of I - K_sep^-1 K
  // The FP64 fast diagonalisation is close enough to the inverse for plain
  // defect correction: at 1/4 every pass gains a factor of four for certain
  // (measured: 1e-3 at 401 and 1e-2 at 33 rows of the stretched grids, where
  // the bound is 0.005 and 0.05).  Beyond it (a grid whose spacing changes by
  // half from one row to the next), and for operators that are not separable, CG.
  bool uses_fd(const scy_solve_opts& o) const {
    return o.precond == SCY_PC_FD || (o.precond == SCY_PC_AUTO && separable);
  }
  // A solve by defect correction (correct()).  It takes up to 1.6 times CG's
  // iterations (11 and 7 at 1e-12 on 33 rows that change by 1.4 each, in less
  // time), so a caller's small limit goes to CG: 32 passes, a factor of four
  // each for certain, gain 1e-19, which leaves six digits beyond the tightest
  // tolerance of this path for the norms' difference.
  static constexpr int kCorrectIts = 32;
  bool corrects(const scy_solve_opts& o) const {
    return uses_fd(o) && o.precision == SCY_PREC_FP64 && near_inverse() && !keeps_rounding(o.rtol) &&
           o.max_its >= kCorrectIts;
  }
  bool near_inverse() const { return separable && sep_misfit <= 0.25; }
  // Solves that keep the arithmetic of plain CG with whole sweep chains: those
  // asked for to near rounding and those of the single power-law driver
  // (keep_rounding), whose results are compared digit by digit with earlier
  // runs (replays of recorded step sequences; the viscous strain gVxz starts as
  // a difference of displacements that agree to rounding, so its first digits
  // are the solve's own rounding).  At 1e-13 the tolerance is a few hundred
  // roundings of the residual.  It is no matter of accuracy: power-law batches
  // solve by defect correction, and after 30 steps at 1e-12 on stretched grids
  // their gVxz is 3e-12 to 5e-12 from the oracle's replay, the single driver's
  // 7e-11 to 3e-10, a batch's by CG 1e-12 to 2e-11.
  int keep_rounding = 0;
  bool keeps_rounding(double rtol) const { return keep_rounding || rtol < 1e-13; }
  Reducer red;
  DevBuf scal;
  DevBuf cg_r, cg_p[2], cg_q, cg_z, cg_z32;

  int create(const scy_grid_desc& g);
  int rebuild();
  int apply(int op, const double* in, double* out);
  int set_rhs(const double* bcL, const double* bcR, const double* bcT, const double* bcB, double* rhs);
  int solve(const double* rhs, double* u, const scy_solve_opts& o, scy_solve_stats& st,
            const SolvePart& part = SolvePart());
  // whether a solve with these options can be enqueued (the fast
  // diagonalisation in FP64, tested every iteration by the recurrence)
  bool can_enqueue(const scy_solve_opts& o) const;
  int solve_noalloc(const double* rhs, double* u, const scy_solve_opts& o, scy_solve_stats& st);
  int change_bc(int R, int T, int L, int B);
  // r = rhs - A u with A u summed in double-double arithmetic (error-free
  // products and sums over the 33-point cross form) and rounded once, so r
  // is the true residual to rounding even where ||A|| ||u|| >> ||rhs||;
  // *rnorm2 (device or host pointer, may be NULL) gets ||r||^2 through the
  // context's reducer.  For defect correction of ill-conditioned solves.
  int residual_dd(const double* rhs, const double* u, double* r, double* rnorm2_host);
  DevBuf cross;  // cross-form planes of the fine level (built on first use)
  template <typename T>
  int ensure_mg(std::unique_ptr<Multigrid<T>>& mg);
  int ensure_fd();
  template <typename Tz, class PC>
  int pcg(PC&& pc, const double* rhs, double* u, const scy_solve_opts& o, scy_solve_stats& st, const SolvePart& part);
  template <class PC>
  int correct(PC&& pc, const double* rhs, double* u, const scy_solve_opts& o, scy_solve_stats& st,
              const SolvePart& part);
  int test_convergence(const double* h, const scy_solve_opts& o, double* u, double& tol, scy_solve_stats& st,
                       int* done);
  int read_convergence(const scy_solve_opts& o, double* u, double& tol, scy_solve_stats& st, int* done);
  int finish_solve(const double* rhs, double* u, const scy_solve_opts& o, double tol, scy_solve_stats& st);
};

}  // namespace scy
