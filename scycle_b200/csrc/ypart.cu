// Banded Cholesky solves along y of the fast-diagonalisation preconditioner,
// in segments of rows that run at the same time (FP64).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "common.cuh"
#include "fdiag.hpp"
#include "tma.cuh"

namespace scy {
namespace {

// After the z transform: for every z mode j and instance k the banded solve
// (Ky + lz_j My) x = t along y with the Cholesky factor L (L v = t, L^T x =
// v), in place in t (rows of Nzp values, instance k at rows k Ny ..).
//
// One chain is 2 Ny rows that depend on each other, so one thread per chain
// (b_ysolve_tma_kernel) takes 68 us at 401 rows however few chains there
// are.  Here the rows are cut into P segments of at most T: a segment only
// needs the last four rows of the one before (away from the closures L has
// four off-diagonals), and it needs them linearly.  So every segment is swept
// with nothing coming in; the true last rows are then carried from segment to
// segment (out = out_0 + M in, M the last four rows of G); and every row takes
// G in.  The same from the other end for L^T with its own table B and the
// first rows.
//
// A lone warp issues an instruction every five cycles or so when each needs
// the one before, so what counts is instructions a row: the segment's rows
// stay in registers (T is a template parameter, everything is unrolled), and a
// thread's coefficients (14 values a row: 1 / L_ii and L's four off-diagonals,
// G, B) lie one behind the other in shared memory, read 16 bytes at a time
// with constant offsets; the threads' tables are 2 mod 4 values apart, so no
// two lanes meet in a bank.  With the rows in shared memory and run-time
// strides the same sweeps took 330 to 770 cycles a row.
//
// A block owns MB modes: thread q of a group is (segment q / MB, mode q %
// MB).  Its tables come by bulk copy and stay for all instances the block
// takes, I at a time; blockDim.y groups work on different instances with
// barriers of their own.  Segments differ by a row: the shorter ones start
// with up to seven empty rows (zero coefficients and data).  The closures'
// four further off-diagonals ("wide": rows 5..8 of the first segment and the
// last four of the last) have a small table of their own.
//
// The wait for the copies is bounded; one that runs out sets status bit 4 of
// the group's instances and leaves t as it is.
struct YPartArgs {
  const double* tab;   // per mode block: [P * MB threads][T * 14 + 2]
  const double* wide;  // per mode block: [first / last segment][4 rows][4][MB]
  double* t;
  int Ny, Nzp, K, P, MB, base, extra;  // segments of base + 1 rows (the first `extra`) and of base rows
  unsigned* status;
  int polls, drop;
};
constexpr int kRow = 14, kMaxPad = 7, kMaxT = 48;

template <int T, int I>
__global__ void __launch_bounds__(384) ypart_kernel(const YPartArgs A) {
  constexpr int S = T * kRow + 2;
  extern __shared__ __align__(128) unsigned char yp_smem[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ double W[32 * 4];
  __shared__ int failed[16];
  const int P = A.P, MB = A.MB, PM = P * MB, Nzp = A.Nzp;
  const int q = threadIdx.x, grp = threadIdx.y, jb = blockIdx.x;
  double* const tab = reinterpret_cast<double*>(yp_smem);
  // per group and instance: the rows a segment passes on (as swept), and those it gets (true)
  double* const E = tab + (size_t)PM * S + (size_t)grp * I * 8 * PM;
  double* const Ein = E + I * 4 * PM;
  for (int i = grp * blockDim.x + q; i < 32 * MB; i += blockDim.x * blockDim.y) W[i] = A.wide[(size_t)jb * 32 * MB + i];
  if (q == 0) failed[grp] = 0;
  if (q == 0 && grp == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    // drop (a test hook): the copy is never issued, its wait runs out
    if (!A.drop) {
      const uint32_t bytes = (uint32_t)(PM * S) * 8u, part = (bytes / 8 + 15) / 16 * 16;
      mbar_expect_tx(&bar, bytes);
      const unsigned char* src = reinterpret_cast<const unsigned char*>(A.tab + (size_t)jb * PM * S);
      for (uint32_t at = 0; at < bytes; at += part)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         smem_u32(yp_smem + at)),
                     "l"(src + at), "r"(min(part, bytes - at)), "r"(smem_u32(&bar))
                     : "memory");
    }
  }
  // (the tables, laid out at set-up, ahead of the wait for the kernel that
  // makes t)
  chain_enter();
  __syncthreads();
  const bool act = q < PM;
  const int seg = act ? q / MB : 0, mode = act ? q % MB : 0;
  const int nr = seg < A.extra ? A.base + 1 : A.base, pad = T - nr;
  const int row0 = seg * A.base + min(seg, A.extra);
  const double* const c = tab + (size_t)(act ? q : 0) * S;
  const bool head = act && seg == 0, tail = act && seg == P - 1;
  double* const tcol = A.t + (long)(row0 - pad) * Nzp + jb * MB + mode;  // register row r is tcol[r * Nzp] (r >= pad)
  auto sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"((int)blockDim.x) : "memory"); };
  auto pair = [&](int r, int k) { return *reinterpret_cast<const double2*>(c + r * kRow + k); };
  // wide coefficients of register row r (rows 5..8 of the first segment, the last four of the last)
  auto wide_row = [&](int r) {
    return head && r - pad >= 5 && r - pad <= 8 ? r - pad - 5 : tail && r >= T - 4 ? 4 + r - (T - 4) : -1;
  };
  // lane c of four carries component c of (mode, instance) q / 4 over the segments: val = the segment's own
  // rows, coefficients its row of G or B; the true rows go to the next segment's Ein
  auto carry = [&](int first, int step, int crow0, int crow_step, int ck) {
    const int w = q >> 2, comp = q & 3, cm = w % MB, ci = w / MB;
    if (ci >= I) return;
    const unsigned mask = 0xfu << (threadIdx.x & 28);
    const double* e = E + (ci * 4 + comp) * PM + cm;
    double* ein = Ein + (ci * 4 + comp) * PM + cm;
    const double* cf = tab + (size_t)cm * S + (crow0 + crow_step * comp) * kRow + ck;
    double v = e[first * MB];
    ein[(first + step) * MB] = v;
    double xn = 0.0, g[4] = {0.0, 0.0, 0.0, 0.0};
    auto fetch = [&](int s) {
      const int pd = ck == 9 ? T - (s < A.extra ? A.base + 1 : A.base) : 0;  // B: from the first row that is not empty
      const double* p = cf + (size_t)s * MB * S + pd * kRow;
      xn = e[s * MB];
#pragma unroll
      for (int k = 0; k < 4; ++k) g[k] = p[k];
    };
    if (P > 2) fetch(first + step);
    for (int n = 1; n < P - 1; ++n) {
      const int s = first + n * step;
      const double e0 = __shfl_sync(mask, v, 0, 4), e1 = __shfl_sync(mask, v, 1, 4), e2 = __shfl_sync(mask, v, 2, 4),
                   e3 = __shfl_sync(mask, v, 3, 4);
      v = (fma(g[0], e0, xn) + g[1] * e1) + fma(g[2], e2, g[3] * e3);
      if (n + 2 < P) fetch(s + step);
      ein[(s + step) * MB] = v;
    }
  };
  const int stride = gridDim.y * blockDim.y * I;
  int k0 = (blockIdx.y * blockDim.y + grp) * I;
  for (; k0 < A.K; k0 += stride) {
    double x[I][T];
#pragma unroll
    for (int i = 0; i < I; ++i) {
      const double* src = tcol + (long)min(k0 + i, A.K - 1) * A.Ny * Nzp;
#pragma unroll
      for (int r = 0; r < T; ++r) x[i][r] = act && (r >= kMaxPad || r >= pad) ? src[(long)r * Nzp] : 0.0;
    }
    if (!mbar_wait(&bar, 0, A.polls)) failed[grp] = 1;
    sync();
    if (failed[grp]) break;
    // L v = t within the segment
    if (act) {
#pragma unroll
      for (int r = 0; r < T; ++r) {
        const double2 f01 = pair(r, 0), f23 = pair(r, 2);
        const double f4 = c[r * kRow + 4], f1d = f01.y * f01.x;
        const int wr = r >= 5 && (r <= 8 + kMaxPad || r >= T - 4) ? wide_row(r) : -1;
#pragma unroll
        for (int i = 0; i < I; ++i) {
          double s = x[i][r];
          if (r >= 4) s = fma(-f4, x[i][r - 4], s);
          if (r >= 3) s = fma(-f23.y, x[i][r - 3], s);
          if (r >= 2) s = fma(-f23.x, x[i][r - 2], s);
          if (r >= 5 && (r <= 8 + kMaxPad || r >= T - 4))
            if (wr >= 0) {
#pragma unroll
              for (int d = 0; d < 4; ++d)
                if (r >= 5 + d) s = fma(-W[(wr * 4 + d) * MB + mode], x[i][r - 5 - d], s);
            }
          s *= f01.x;
          x[i][r] = r >= 1 ? fma(-f1d, x[i][r - 1], s) : s;
        }
      }
#pragma unroll
      for (int i = 0; i < I; ++i)
#pragma unroll
        for (int d = 0; d < 4; ++d) E[(i * 4 + d) * PM + q] = x[i][T - 1 - d];
    }
    if (P > 1) {
      sync();
      carry(0, 1, T - 1, -1, 5);
      sync();
    }
    // v += G in, then L^T x = v within the segment
    if (act) {
      double e[I][4];
#pragma unroll
      for (int i = 0; i < I; ++i)
#pragma unroll
        for (int d = 0; d < 4; ++d) e[i][d] = seg > 0 ? Ein[(i * 4 + d) * PM + q] : 0.0;
#pragma unroll
      for (int r = T - 1; r >= 0; --r) {
        const double2 f01 = pair(r, 0), f23 = pair(r, 2), f4g0 = pair(r, 4), g12 = pair(r, 6);
        const double g3 = c[r * kRow + 8];
#pragma unroll
        for (int i = 0; i < I; ++i) {
          // x[r] holds v less what the rows below have taken off already
          x[i][r] += fma(f4g0.y, e[i][0], g12.x * e[i][1]) + fma(g12.y, e[i][2], g3 * e[i][3]);
        }
        if (r + 5 < T && (r <= 3 + kMaxPad || r >= T - 12)) {
#pragma unroll
          for (int d = 0; d < 4; ++d)
            if (r + 5 + d < T)
              if (const int wr = wide_row(r + 5 + d); wr >= 0) {
                const double w = W[(wr * 4 + d) * MB + mode];
#pragma unroll
                for (int i = 0; i < I; ++i) x[i][r] = fma(-w, x[i][r + 5 + d], x[i][r]);
              }
        }
#pragma unroll
        for (int i = 0; i < I; ++i) {
          const double v = x[i][r] * f01.x;
          x[i][r] = v;
          if (r >= 1) x[i][r - 1] = fma(-f01.y, v, x[i][r - 1]);
          if (r >= 2) x[i][r - 2] = fma(-f23.x, v, x[i][r - 2]);
          if (r >= 3) x[i][r - 3] = fma(-f23.y, v, x[i][r - 3]);
          if (r >= 4) x[i][r - 4] = fma(-f4g0.x, v, x[i][r - 4]);
        }
      }
#pragma unroll
      for (int i = 0; i < I; ++i)
#pragma unroll
        for (int r = 0; r < (4 + kMaxPad < T ? 4 + kMaxPad : T); ++r)
          if (r >= pad && r < pad + 4) E[(i * 4 + r - pad) * PM + q] = x[i][r];
    }
    if (P > 1) {
      sync();
      carry(P - 1, -1, 0, 1, 9);
      sync();
    }
    // x += B in, and out
    if (act) {
      double e[I][4];
#pragma unroll
      for (int i = 0; i < I; ++i)
#pragma unroll
        for (int d = 0; d < 4; ++d) e[i][d] = seg < P - 1 ? Ein[(i * 4 + d) * PM + q] : 0.0;
#pragma unroll
      for (int r = 0; r < T; ++r) {
        const double b0 = c[r * kRow + 9], b3 = c[r * kRow + 12];
        const double2 b12 = pair(r, 10);
#pragma unroll
        for (int i = 0; i < I; ++i) {
          const double v = x[i][r] + (fma(b0, e[i][0], b12.x * e[i][1]) + fma(b12.y, e[i][2], b3 * e[i][3]));
          if ((r >= kMaxPad || r >= pad) && k0 + i < A.K) tcol[((long)(k0 + i) * A.Ny + r) * Nzp] = v;
        }
      }
    }
  }
  if (k0 < A.K && q == 0) {
    for (int k = k0; k < A.K; k += stride)
      for (int i = 0; i < I && k + i < A.K; ++i) atomicOr(A.status + k + i, 4u);
  }
  // no block leaves while a copy into its shared memory may be in flight
  if (q == 0 && grp == 0 && !A.drop) mbar_wait(&bar, 0, 1 << 18);
  __syncthreads();
}

// The tables of mode j, segment sg (one thread each): the factor's entries
// within the segment, its rows' answer G to the four rows before it and B to
// the four rows after it.  L as YPart::plan takes it.
__global__ void __launch_bounds__(128) ypart_fill_kernel(const double* __restrict__ L, int Nz, int Ny, int T, int P,
                                                         int MB, int base, int extra, double* __restrict__ tab,
                                                         double* __restrict__ wide) {
  const int at = blockIdx.x * blockDim.x + threadIdx.x;
  if (at >= P * Nz) return;
  const int sg = at / Nz, j = at - sg * Nz, jb = j / MB, md = j % MB;
  const int r0 = sg * base + min(sg, extra), nr = sg < extra ? base + 1 : base, S = T * kRow + 2;
  auto lj = [&](int i, int k) { return L[((long)i * 9 + k) * Nz + j]; };
  double* c = tab + ((long)jb * P * MB + sg * MB + md) * S + (T - nr) * kRow;
  double* w = wide + (long)jb * 32 * MB + md;
  double col[kMaxT];
  for (int r = 0; r < nr; ++r) {
    // off-diagonals to rows of this segment (those to earlier ones are in G)
    for (int k = 0; k < 5; ++k) c[r * kRow + k] = r >= k ? lj(r0 + r, k) : 0.0;
    const int wr = sg == 0 && r >= 5 && r <= 8 ? r - 5 : sg == P - 1 && r >= nr - 4 ? 4 + r - (nr - 4) : -1;
    if (wr >= 0)
      for (int k = 5; k <= 8 && k <= r; ++k) w[(wr * 4 + k - 5) * MB] = lj(r0 + r, k);
  }
  // G: rows of this segment for a one in row r0 - 1 - d and no data
  if (sg > 0)
    for (int d = 0; d < 4; ++d)
      for (int r = 0; r < nr; ++r) {
        double sum = 0.0;
        for (int k = 1; k <= 8; ++k) {
          const int p = r - k;  // row of the segment; -1 - d is the incoming one
          const double v = p >= 0 ? col[p] : p == -1 - d ? 1.0 : 0.0;
          if (v != 0.0) sum = __dsub_rn(sum, __dmul_rn(lj(r0 + r, k), v));
        }
        col[r] = __dmul_rn(sum, lj(r0 + r, 0));
        c[r * kRow + 5 + d] = col[r];
      }
  // B: the same upwards for a one in row r0 + nr + d
  if (sg < P - 1)
    for (int d = 0; d < 4; ++d)
      for (int r = nr - 1; r >= 0; --r) {
        double sum = 0.0;
        for (int k = 1; k <= 8 && r0 + r + k < Ny; ++k) {
          const int p = r + k;
          const double v = p < nr ? col[p] : p == nr + d ? 1.0 : 0.0;
          if (v != 0.0) sum = __dsub_rn(sum, __dmul_rn(lj(r0 + p, k), v));
        }
        col[r] = __dmul_rn(sum, lj(r0 + r, 0));
        c[r * kRow + 9 + d] = col[r];
      }
}

int dev_smem_limit() { return 225 * 1024; }  // beside the static kilobyte

template <int T, int I>
int launch_one(const YPartArgs& A, size_t smem, int nb, int NG, cudaStream_t s, bool chain) {
  const int TP = (A.P * A.MB + 31) / 32 * 32;
  SCY_CUDA_TRY(cudaFuncSetAttribute(ypart_kernel<T, I>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    dev_smem_limit()));
  int per_sm = 0;
  SCY_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ypart_kernel<T, I>, TP * NG, smem));
  // as many blocks a mode block as are resident at once: each takes its
  // instances in turn with the tables it has loaded
  const int want = (A.K + NG * I - 1) / (NG * I), fit = std::max(1, per_sm * kNumSMs / nb);
  launch(chain, ypart_kernel<T, I>, dim3(nb, std::min(want, fit)), dim3(TP, NG), smem, s, A);
  SCY_LAUNCH_CHECK();
  return SCY_OK;
}

// (rows a thread; from 24 on two instances a thread spill, 40 bytes there to 1300
// at 48, and the autotuner times the forms with one beside them)
constexpr int kT[] = {8, 12, 16, 20, 24, 28, 32, 40, kMaxT};
}  // namespace

size_t YPart::smem_bytes(int shape) const {
  return (size_t)P * MB * (T * kRow + 2 + 8 * kShapeI[shape] * kShapeNG[shape]) * 8;
}
bool YPart::fits(int shape) const {
  const int TP = (P * MB + 31) / 32 * 32;
  return T > 0 && smem_bytes(shape) <= (size_t)dev_smem_limit() &&
         TP * kShapeNG[shape] <= 384 && 4 * MB * kShapeI[shape] <= TP;
}

void YPart::plan(const std::vector<double>& L, int Ny_, int Nz_, int Nzp_) {
  Ny = Ny_;
  Nz = Nz_;
  Nzp = Nzp_;
  // Segments: a row costs about 120 cycles in its three passes and a carry
  // about 80 each way, so T near 1.15 sqrt(Ny); no segment below eight rows, so
  // that the closures' wide rows (eight at either end) lie inside the first
  // and the last one.
  const double want = 1.15 * std::sqrt((double)Ny);
  int bestT = 0, bestP = 0;
  for (int t : kT) {
    const int p = (Ny + t - 1) / t;
    if ((p > 1 && Ny / p < 8) || t - Ny / p > kMaxPad) continue;
    if (!bestT || std::fabs(t - want) < std::fabs(bestT - want)) {
      bestT = t;
      bestP = p;
    }
  }
  P = bestP;
  T = bestT;
  // modes a block: four are one 32-byte sector of the transform's rows; the
  // tables (448 bytes a row) fit the shared memory up to about 480 rows, with
  // two modes to 960, with one to 1900
  for (MB = 4; MB >= 1 && T; MB /= 2)
    if (fits(0)) break;
  if (!T || MB < 1) {
    T = 0;
    return;
  }
  base = Ny / P;
  extra = Ny % P;
  auto row0 = [&](int sg) { return sg * base + std::min(sg, extra); };
  auto rows = [&](int sg) { return sg < extra ? base + 1 : base; };
  auto at = [&](int i, int k, int j) { return L[((size_t)i * 9 + k) * Nz + j]; };
  // the off-diagonals beyond the fourth must lie where the kernel looks for
  // them: within the first or the last segment, rows as in wide_row
  auto wide_row = [&](int sg, int r) {
    return sg == 0 && r >= 5 && r <= 8 ? r - 5 : sg == P - 1 && r >= rows(sg) - 4 ? 4 + r - (rows(sg) - 4) : -1;
  };
  for (int sg = 0; sg < P; ++sg)
    for (int r = 0; r < rows(sg); ++r)
      for (int k = 5; k <= 8 && k <= row0(sg) + r; ++k)
        for (int j = 0; j < Nz; ++j)
          if (at(row0(sg) + r, k, j) != 0.0 && (k > r || wide_row(sg, r) < 0)) {
            T = 0;
            return;
          }
  nb = (Nzp + MB - 1) / MB;
}

int YPart::fill(const double* L, cudaStream_t s) {
  const size_t S = T * kRow + 2, n = (size_t)nb * P * MB * S, nw = (size_t)nb * 32 * MB;
  DevBuf t;  // tab once it is laid out
  SCY_TRY(t.alloc(n * 8));
  SCY_TRY(wide.alloc(nw * 8));
  SCY_CUDA_TRY(cudaMemsetAsync(t.p, 0, n * 8, s));
  SCY_CUDA_TRY(cudaMemsetAsync(wide.p, 0, nw * 8, s));
  ypart_fill_kernel<<<(P * Nz + 127) / 128, 128, 0, s>>>(L, Nz, Ny, T, P, MB, base, extra, t.as<double>(),
                                                         wide.as<double>());
  SCY_LAUNCH_CHECK();
  SCY_CUDA_TRY(cudaStreamSynchronize(s));
  tab = std::move(t);
  return SCY_OK;
}

int YPart::solve(double* t, int K, int shape, unsigned* status, cudaStream_t s, bool chain, int polls, int drop) const {
  const YPartArgs A{tab.as<double>(), wide.as<double>(), t, Ny, Nzp, K, P, MB, base, extra, status, polls, drop};
  const int I = kShapeI[shape], NG = kShapeNG[shape];
  const size_t smem = smem_bytes(shape);
  switch (T) {
#define SCY_YP(TV) \
  case TV: return I == 1 ? launch_one<TV, 1>(A, smem, nb, NG, s, chain) : launch_one<TV, 2>(A, smem, nb, NG, s, chain)
    SCY_YP(8);
    SCY_YP(12);
    SCY_YP(16);
    SCY_YP(20);
    SCY_YP(24);
    SCY_YP(28);
    SCY_YP(32);
    SCY_YP(40);
    SCY_YP(48);
#undef SCY_YP
    default: break;
  }
  set_error("banded sweeps: no segment plan");
  return SCY_ERR_STATE;
}

}  // namespace scy
