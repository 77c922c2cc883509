// Poisson solve of Src/pdesolver.f90 + Src/mg.f90 + Src/sors.f90 as ONE
// persistent kernel: every V-cycle, every level, every red-black sweep, the
// residual-ratio exit test of sor_rb and the outer res/alpha < eps loop run on
// the device; the host sees a single launch.
//
// Two kernels with the same schedule and the same iterates, bit for bit:
// k_pdesolver_split (the second half of this file), on colour-split copies of
// the levels, for Dirichlet walls; k_pdesolver, the general one, on the
// caller's arrays, for periodic and Neumann planes, for solves without
// allocation, and where the split one does not apply (launch_split).
//
// Schedule (identical to the reference, one MPI rank):
//   for each V-cycle k: down leg sor_rb(level l, dig<0) + restriction,
//   coarsest sor_rb(dig=0) (up to 1e6 sweeps in cycle 1 until res <= eps,
//   4 afterwards) + prolongation, up leg sor_rb(dig>0) + prolongation.
//   sor_rb stops after 4 sweeps or when res/res_prev <= 0.6.
//
// Bit-exactness: node updates of one colour are independent, and every
// expression keeps the Fortran evaluation order (the file is compiled with
// --fmad=false), so the iterates equal the CPU oracle's.  The L1 residual is
// summed per block in a fixed tree and then over blocks in block order by
// every block, so all blocks take the same exit decision and the result is
// deterministic run to run.
//
// In the general kernel levels with few nodes (<= SMALL_NODES) are smoothed by
// block 0 alone with __syncthreads, avoiding grid-wide barriers on the tiny
// coarse grids.
//
// Periodic planes in y and z (bcnd 0) and the Neumann plane at x = 0
// (bcnd -2) run in a second instance of that kernel (GEN): the node rules of
// Src/sors.f90:113-125, the ghost-plane refresh after each colour
// (Src/sors.f90:157-231) and the restriction's periodic wraps
// (Src/mg.f90:314-805); the Dirichlet instance is unchanged.
#include <cooperative_groups.h>

#include "mgsplit.cuh"

namespace cg = cooperative_groups;

namespace lepic {

namespace {

constexpr int MG_MAX = 13;
constexpr int MG_BLOCK = 512;
constexpr long long SMALL_NODES = 20000;

struct MGLev {
  int n1, n2, n3;
  long long N1, N2;   // node extents n+3 in x, y
  long long R1, R2;   // rhs extents n+2
  double aw, ae, an, as, at, ab, ac;
  double *u;          // (n+3)^3
  double *b;          // (n+2)^3
  int *bc;            // (n+3)^3
  double *rf;         // (n+3)^3 fine residual scratch (levels that restrict)
  double *rp;         // (n1+2)(n2+2) residual plane r_pbc of the last z plane (GEN)
  __device__ long long g(int i, int j, int k) const { return i + N1 * (j + N2 * (long long)k); }
  __device__ long long r(int i, int j, int k) const { return i + R1 * (j + R2 * (long long)k); }
  __device__ long long nodes() const { return (long long)(n1 + 1) * (n2 + 1) * (n3 + 1); }
};

struct MGArgs {
  MGLev L[MG_MAX + 1];
  int ng, ncycl;
  int pbc, nmn;       // periodic planes in y and z; Neumann plane at x = 0 (GEN only)
  double alpha, eps, omega;
  double *partial;    // [gridDim.x]
  double *shared_d;   // [4]: small-level results
  int *out_i;         // [0] k, [1] status, [2..] iterations per level of last cycle
  double *out_d;      // [0] ktot, [1] res
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// deterministic block sum (fixed tree); result valid in all threads
__device__ double block_sum(double v, double *sh) {
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  int nw = blockDim.x >> 5;
  double t = (threadIdx.x < nw) ? sh[threadIdx.x] : 0.0;
  if (w == 0) t = warp_sum(t);
  if (threadIdx.x == 0) sh[32] = t;
  __syncthreads();
  double r = sh[32];
  __syncthreads();
  return r;
}

// Warps that share a loop: warp gw of nw (the whole grid or block 0).
struct Warps {
  int gw, nw;
};
__device__ __forceinline__ Warps grid_warps() {
  return {(int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), (int)((gridDim.x * blockDim.x) >> 5)};
}
__device__ __forceinline__ Warps block_warps() { return {(int)(threadIdx.x >> 5), (int)(blockDim.x >> 5)}; }

// The grid rows (j, k), j in [j0, j0 + nj), k in [k0, k0 + nk), dealt
// round-robin to the warps; body(j, k) runs on all 32 lanes of the warp, which
// split the row along i (coalesced, one 32-bit division per row).
template <class F>
__device__ __forceinline__ void for_rows(const Warps &w, int j0, int nj, int k0, int nk, F &&body) {
  const int rows = nj * nk;
  for (int r = w.gw; r < rows; r += w.nw) {
    const int kk = r / nj;
    body(j0 + (r - kk * nj), k0 + kk);
  }
}

// one colour of a red-black sweep
// colour 0 = red ((i+j+k) odd), 1 = black (Src/sors.f90:87-106, 249-267).
// GEN: Neumann nodes (-2) drop the west neighbour and take the east one
// twice; periodic nodes (0) on the last y or z plane are not updated.
template <bool GEN>
__device__ __forceinline__ void sweep_colour(const MGLev &L, double omega, int colour, const Warps &w) {
  const int lane = threadIdx.x & 31;
  const long long sy = L.N1, sz = L.N1 * L.N2;
  for_rows(w, 1, L.n2 + 1, 1, L.n3 + 1, [&](int j, int k) {
    int ks = (k % 2 == 0) ? 0 : 1;
    int is;
    if (colour == 0) is = (j % 2 == 0) ? 1 : 2;
    else is = (j % 2 == 0) ? 2 : 1;
    is = is + ks;
    if (is > 2) is = 1;
    for (int i = is + 2 * lane; i <= L.n1 + 1; i += 64) {
      long long q = L.g(i, j, k);
      const int bq = L.bc[q];
      if (bq > 0) continue;
      if (GEN) {
        if (bq == -2) {
          double tt = L.b[L.r(i, j, k)] - L.an * L.u[q + sy] - L.as * L.u[q - sy] - 2.0 * L.ae * L.u[q + 1] -
                      L.at * L.u[q + sz] - L.ab * L.u[q - sz];
          L.u[q] = (1.0 - omega) * L.u[q] + omega * tt / L.ac;
          continue;
        }
        if (bq == 0 && (k == L.n3 + 1 || j == L.n2 + 1)) continue;
      }
      double tt = L.b[L.r(i, j, k)] - L.aw * L.u[q - 1] - L.an * L.u[q + sy] - L.as * L.u[q - sy] -
                  L.ae * L.u[q + 1] - L.at * L.u[q + sz] - L.ab * L.u[q - sz];
      L.u[q] = (1.0 - omega) * L.u[q] + omega * tt / L.ac;
    }
  });
}

// Periodic ghost planes (Src/sors.f90:157-231), first phase: y ghosts of
// every z plane; second phase (after a barrier): z ghosts of every y row.
// A ghost is refreshed where the node next to it is periodic or Neumann.
__device__ __forceinline__ void ghosts_y(const MGLev &L, const Warps &w) {
  const int lane = threadIdx.x & 31;
  for_rows(w, 0, 1, 0, L.n3 + 3, [&](int, int k) {
    for (int i = lane; i <= L.n1 + 2; i += 32) {
      const int b1 = L.bc[L.g(i, 1, k)], bn = L.bc[L.g(i, L.n2 + 1, k)];
      if (b1 == 0 || b1 == -2) L.u[L.g(i, 0, k)] = L.u[L.g(i, L.n2, k)];
      if (bn == 0 || bn == -2) L.u[L.g(i, L.n2 + 1, k)] = L.u[L.g(i, 1, k)];
    }
  });
}
__device__ __forceinline__ void ghosts_z(const MGLev &L, const Warps &w) {
  const int lane = threadIdx.x & 31;
  for_rows(w, 0, L.n2 + 3, 0, 1, [&](int j, int) {
    for (int i = lane; i <= L.n1 + 2; i += 32) {
      const int b1 = L.bc[L.g(i, j, 1)], bm = L.bc[L.g(i, j, L.n3 + 1)];
      if (b1 == 0 || b1 == -2) L.u[L.g(i, j, 0)] = L.u[L.g(i, j, L.n3)];
      if (bm == 0 || bm == -2) L.u[L.g(i, j, L.n3 + 1)] = L.u[L.g(i, j, 1)];
    }
  });
}

// sum of |residual| over the plasma nodes of this thread's rows
__device__ __forceinline__ double residual_part(const MGLev &L, const Warps &w) {
  const int lane = threadIdx.x & 31;
  const long long sy = L.N1, sz = L.N1 * L.N2;
  double acc = 0.0;
  for_rows(w, 1, L.n2 + 1, 1, L.n3 + 1, [&](int j, int k) {
    for (int i = 1 + lane; i <= L.n1 + 1; i += 32) {
      long long q = L.g(i, j, k);
      if (L.bc[q] != -1) continue;
      double rij = L.b[L.r(i, j, k)] - (L.aw * L.u[q - 1] + L.an * L.u[q + sy] + L.as * L.u[q - sy] +
                                        L.ae * L.u[q + 1] + L.ac * L.u[q] + L.at * L.u[q + sz] +
                                        L.ab * L.u[q - sz]);
      acc += fabs(rij);
    }
  });
  return acc;
}

// Src/sors.f90:1-535, whole grid.  Returns res, ksor (uniform in all threads).
template <bool GEN>
__device__ void sor_rb(const MGArgs &a, const MGLev &L, int kmg, int dig, double eps_abs,
                       cg::grid_group &grid, double *sh, double &res_out, int &ksor_out) {
  const bool pbc = GEN && a.pbc;
  long long nr = 4;
  if (kmg == 1 && dig == 0) nr = 1000000;
  const double eta = 0.6;
  if (L.nodes() <= SMALL_NODES) {
    if (blockIdx.x == 0) {
      double res_s = 0.0, res = 0.0;
      int ksor = 0;
      const Warps w = block_warps();
      for (long long l = 1; l <= nr; ++l) {
        for (int colour = 0; colour < 2; ++colour) {
          sweep_colour<GEN>(L, a.omega, colour, w);
          __syncthreads();
          if (pbc) {
            ghosts_y(L, w);
            __syncthreads();
            ghosts_z(L, w);
            __syncthreads();
          }
        }
        res = block_sum(residual_part(L, w), sh);
        ksor++;
        bool stop = (dig == 0) ? (res <= eps_abs) : (res_s > 0.0 && (res / res_s) <= eta);
        if (stop) break;
        res_s = res;
      }
      if (threadIdx.x == 0) {
        a.shared_d[0] = res;
        a.shared_d[1] = (double)ksor;
      }
      __threadfence();
    }
    grid.sync();
    res_out = a.shared_d[0];
    ksor_out = (int)a.shared_d[1];
    grid.sync();  // everyone has read shared_d before it is reused
    return;
  }
  const Warps w = grid_warps();
  double res_s = 0.0, res = 0.0;
  int ksor = 0;
  for (long long l = 1; l <= nr; ++l) {
    for (int colour = 0; colour < 2; ++colour) {
      sweep_colour<GEN>(L, a.omega, colour, w);
      grid.sync();
      if (pbc) {
        ghosts_y(L, w);
        grid.sync();
        ghosts_z(L, w);
        grid.sync();
      }
    }
    double part = block_sum(residual_part(L, w), sh);
    if (threadIdx.x == 0) a.partial[blockIdx.x] = part;
    grid.sync();
    // every block sums the partials in the same fixed order
    double v = 0.0;
    if (threadIdx.x < 32) {
      for (int bI = threadIdx.x; bI < (int)gridDim.x; bI += 32) v += a.partial[bI];
      v = warp_sum(v);
      if (threadIdx.x == 0) sh[33] = v;
    }
    __syncthreads();
    res = sh[33];
    __syncthreads();
    ksor++;
    bool stop = (dig == 0) ? (res <= eps_abs) : (res_s > 0.0 && (res / res_s) <= eta);
    if (stop) break;
    res_s = res;
  }
  res_out = res;
  ksor_out = ksor;
}

// Src/mg.f90:808-847 (getres), Dirichlet form
__device__ __forceinline__ double getres(const MGLev &L, long long q, double urhs) {
  const long long sy = L.N1, sz = L.N1 * L.N2;
  double uij = L.u[q], un = L.u[q + sy], us = L.u[q - sy], ue = L.u[q + 1];
  double ut = L.u[q + sz], ub = L.u[q - sz], uw = L.u[q - 1];
  return urhs - (L.aw * uw + L.ae * ue + L.an * un + L.as * us + L.ac * uij + L.at * ut + L.ab * ub);
}

__device__ __forceinline__ int fmap(int ic, int ncell) {
  return ic == ncell / 2 + 2 ? ncell + 2 : (ic == 0 ? 0 : 2 * ic - 1);
}

// Src/mg.f90:248-805 (restriction), fine F -> coarse C
__device__ void restriction(const MGLev &F, const MGLev &C, cg::grid_group &grid) {
  const Warps w = grid_warps();
  const int lane = threadIdx.x & 31;
  for_rows(w, 1, F.n2 + 1, 1, F.n3 + 1, [&](int j, int k) {
    for (int i = 1 + lane; i <= F.n1 + 1; i += 32) {
      long long q = F.g(i, j, k);
      F.rf[q] = (F.bc[q] > 0) ? 0.0 : getres(F, q, F.b[F.r(i, j, k)]);
    }
  });
  grid.sync();
  const long long sy = F.N1, sz = F.N1 * F.N2;
  for_rows(w, 0, C.n2 + 3, 0, C.n3 + 3, [&](int j, int k) {
    for (int i = lane; i <= C.n1 + 2; i += 32) {
      long long qc = C.g(i, j, k);
      int bc2 = F.bc[F.g(fmap(i, F.n1), fmap(j, F.n2), fmap(k, F.n3))];
      C.bc[qc] = bc2;
      C.u[qc] = 0.0;
      if (i <= C.n1 + 1 && j <= C.n2 + 1 && k <= C.n3 + 1) {
        double re = 0.0;
        if (i >= 1 && j >= 1 && k >= 1 && bc2 <= 0) {
          long long q = F.g(2 * i - 1, 2 * j - 1, 2 * k - 1);
          const double *R = F.rf;
          double r000 = R[q];
          double rpp0 = R[q + 1 + sy], rp00 = R[q + 1], rpm0 = R[q + 1 - sy];
          double r0m0 = R[q - sy], rmm0 = R[q - 1 - sy], rm00 = R[q - 1];
          double rmp0 = R[q - 1 + sy], r0p0 = R[q + sy];
          double r00p = R[q + sz], rppp = R[q + 1 + sy + sz], rp0p = R[q + 1 + sz];
          double rpmp = R[q + 1 - sy + sz], r0mp = R[q - sy + sz];
          double rmmp = R[q - 1 - sy + sz], rm0p = R[q - 1 + sz];
          double rmpp = R[q - 1 + sy + sz], r0pp = R[q + sy + sz];
          double r00m = R[q - sz], rppm = R[q + 1 + sy - sz], rp0m = R[q + 1 - sz];
          double rpmm = R[q + 1 - sy - sz], r0mm = R[q - sy - sz];
          double rmmm = R[q - 1 - sy - sz], rm0m = R[q - 1 - sz];
          double rmpm = R[q - 1 + sy - sz], r0pm = R[q + sy - sz];
          re = (8.0 * r000 + 4.0 * (rp00 + rm00 + r0p0 + r0m0 + r00p + r00m) +
                2.0 * (rpp0 + rmp0 + rpm0 + rmm0 + rp0p + rm0p + r0pp + r0mp + rp0m + rm0m +
                       r0pm + r0mm) +
                rppp + rmpp + rpmp + rmmp + rppm + rmpm + rpmm + rmmm) /
               64.0;
        }
        C.b[C.r(i, j, k)] = re;
      }
    }
  });
  grid.sync();
}

// Src/mg.f90:808-847 (getres) with its Neumann form: on the plane ir = 1
// with flag_nmn the west term is dropped (aw = uw = 0) and ae doubled.
__device__ __forceinline__ double getres_n(const MGLev &L, long long q, double urhs, bool neumann) {
  const long long sy = L.N1, sz = L.N1 * L.N2;
  double uij = L.u[q], un = L.u[q + sy], us = L.u[q - sy], ue = L.u[q + 1];
  double ut = L.u[q + sz], ub = L.u[q - sz];
  double uw, aw = L.aw, ae = L.ae;
  if (neumann) {
    uw = 0.0;
    aw = 0.0;
    ae = 2.0 * ae;
  } else {
    uw = L.u[q - 1];
  }
  return urhs - (aw * uw + ae * ue + L.an * un + L.as * us + L.ac * uij + L.at * ut + L.ab * ub);
}

// Src/mg.f90:248-805 (restriction) with periodic planes in y and z and/or
// the Neumann plane.  (1) the fine residual of every node 1..n+1 (no wall
// mask: the gather tests the neighbours' bcnd as the reference does);
// (2) with periodic planes, the residual plane r_pbc of the last fine z plane
// as the reference's loop over coarse nodes leaves it (j outer, i inner, a
// later write replacing an earlier one: every fine node takes the value of
// the last coarse node that writes it); (3) the 27-point gather, where a
// neighbour at jr-1 = 0 takes the residual of its periodic image jr = n2 in
// the terms the reference wraps and one at kr-1 = 0 takes r_pbc.  Residuals
// outside 1..n+1 (a wrapped term at ir+1 = n1+2) are zero.
__device__ void restriction_gen(const MGArgs &a, const MGLev &F, const MGLev &C, cg::grid_group &grid) {
  const Warps w = grid_warps();
  const int lane = threadIdx.x & 31;
  const int n1 = F.n1, n2 = F.n2, m = F.n3;
  const bool nmn = a.nmn != 0, pbc = a.pbc != 0;
  for_rows(w, 1, n2 + 1, 1, m + 1, [&](int j, int k) {
    for (int i = 1 + lane; i <= n1 + 1; i += 32) {
      long long q = F.g(i, j, k);
      F.rf[q] = getres_n(F, q, F.b[F.r(i, j, k)], nmn && i == 1);
    }
  });
  grid.sync();
  auto G = [&](int x, int y, int z) -> double {
    if (x < 1 || x > n1 + 1 || y < 1 || y > n2 + 1 || z < 1 || z > m + 1) return 0.0;
    return F.rf[F.g(x, y, z)];
  };
  auto BC = [&](int x, int y, int z) -> int { return F.bc[F.g(x, y, z)]; };
  const long long RP1 = n1 + 2;
  if (pbc) {
    for_rows(w, 1, n2 + 1, 0, 1, [&](int b, int) {
      for (int x = 1 + lane; x <= n1 + 1; x += 32) {
        double v = 0.0;
        bool done = false;
        // coarse writers of (x, b): jr, ir odd within one node, latest first
        for (int jr = ((b + 1) & 1) ? b + 1 : b; jr >= b - 1 && !done; jr -= 2) {
          if (jr < 1 || jr > n2 + 1) continue;
          for (int ir = ((x + 1) & 1) ? x + 1 : x; ir >= x - 1 && !done; ir -= 2) {
            if (ir < 1 || ir > n1 + 1) continue;
            const int dx = x - ir, dy = b - jr;
            const bool le = BC(ir, jr, m + 1) <= 0;
            bool wr;
            if (dx == -1) wr = ir != 1 && (dy == -1 ? jr != 1 : (dy == 1 ? jr != n2 + 1 : true));
            else if (dx == 1) wr = ir != n1 + 1 && (dy == -1 ? jr != 1 : (dy == 1 ? jr != n2 + 1 : true));
            else wr = dy == -1 ? ((le ? ir != 1 : true) && jr != 1) : (dy == 1 ? jr != n2 + 1 : true);
            if (wr) {
              v = le ? F.rf[F.g(x, b, m)] : 0.0;
              done = true;
            }
          }
        }
        F.rp[x + RP1 * b] = v;
      }
    });
    grid.sync();
  }
  auto RP = [&](int x, int y) -> double { return pbc ? F.rp[x + RP1 * y] : 0.0; };
  for_rows(w, 0, C.n2 + 3, 0, C.n3 + 3, [&](int j, int k) {
    for (int i = lane; i <= C.n1 + 2; i += 32) {
      long long qc = C.g(i, j, k);
      int bc2 = F.bc[F.g(fmap(i, F.n1), fmap(j, F.n2), fmap(k, F.n3))];
      C.bc[qc] = bc2;
      C.u[qc] = 0.0;
      if (i > C.n1 + 1 || j > C.n2 + 1 || k > C.n3 + 1) continue;
      double re = 0.0;
      if (i >= 1 && j >= 1 && k >= 1 && bc2 <= 0) {
        const int ir = 2 * i - 1, jr = 2 * j - 1, kr = 2 * k - 1;
        const bool xl = ir != 1, xr = ir != n1 + 1, yl = jr != 1, yr = jr != n2 + 1, zr = kr != m + 1;
        const bool z0 = kr == 1;
        double r000 = G(ir, jr, kr);
        double rpp0 = (xr && yr && BC(ir + 1, jr + 1, kr) <= 0) ? G(ir + 1, jr + 1, kr) : 0.0;
        double rp00 = (xr && BC(ir + 1, jr, kr) <= 0) ? G(ir + 1, jr, kr) : 0.0;
        double rpm0 = 0.0;
        if (BC(ir + 1, jr - 1, kr) <= 0) {
          if (xr && yl) rpm0 = G(ir + 1, jr - 1, kr);
          else if (!yl) rpm0 = G(ir + 1, n2, kr);
        }
        double r0m0 = 0.0;
        if (BC(ir, jr - 1, kr) <= 0) r0m0 = yl ? G(ir, jr - 1, kr) : G(ir, n2, kr);
        double rmm0 = 0.0;
        if (BC(ir - 1, jr - 1, kr) <= 0 && xl) rmm0 = yl ? G(ir - 1, jr - 1, kr) : G(ir - 1, n2, kr);
        double rm00 = (xl && BC(ir - 1, jr, kr) <= 0) ? G(ir - 1, jr, kr) : 0.0;
        double rmp0 = (xl && yr && BC(ir - 1, jr + 1, kr) <= 0) ? G(ir - 1, jr + 1, kr) : 0.0;
        double r0p0 = (yr && BC(ir, jr + 1, kr) <= 0) ? G(ir, jr + 1, kr) : 0.0;
        double r00p = (zr && BC(ir, jr, kr + 1) <= 0) ? G(ir, jr, kr + 1) : 0.0;
        double rppp = (xr && yr && zr && BC(ir + 1, jr + 1, kr + 1) <= 0) ? G(ir + 1, jr + 1, kr + 1) : 0.0;
        double rp0p = (xr && zr && BC(ir + 1, jr, kr + 1) <= 0) ? G(ir + 1, jr, kr + 1) : 0.0;
        double rpmp = 0.0;
        if (BC(ir + 1, jr - 1, kr + 1) <= 0) {
          if (xr && yl && zr) rpmp = G(ir + 1, jr - 1, kr + 1);
          else if (!yl && zr) rpmp = G(ir + 1, n2, kr + 1);
        }
        double r0mp = 0.0;
        if (BC(ir, jr - 1, kr + 1) <= 0 && zr) r0mp = yl ? G(ir, jr - 1, kr + 1) : G(ir, n2, kr + 1);
        double rmmp = 0.0;
        if (BC(ir - 1, jr - 1, kr + 1) <= 0 && xl && zr)
          rmmp = yl ? G(ir - 1, jr - 1, kr + 1) : G(ir - 1, n2, kr + 1);
        double rm0p = (xl && zr && BC(ir - 1, jr, kr + 1) <= 0) ? G(ir - 1, jr, kr + 1) : 0.0;
        double rmpp = (xl && yr && zr && BC(ir - 1, jr + 1, kr + 1) <= 0) ? G(ir - 1, jr + 1, kr + 1) : 0.0;
        double r0pp = (yr && zr && BC(ir, jr + 1, kr + 1) <= 0) ? G(ir, jr + 1, kr + 1) : 0.0;
        double r00m = 0.0;
        if (BC(ir, jr, kr - 1) <= 0) r00m = z0 ? RP(ir, jr) : G(ir, jr, kr - 1);
        double rppm = 0.0;
        if (BC(ir + 1, jr + 1, kr - 1) <= 0 && xr && yr) rppm = z0 ? RP(ir + 1, jr + 1) : G(ir + 1, jr + 1, kr - 1);
        double rp0m = 0.0;
        if (BC(ir + 1, jr, kr - 1) <= 0 && xr) rp0m = z0 ? RP(ir + 1, jr) : G(ir + 1, jr, kr - 1);
        double rpmm = 0.0;
        if (BC(ir + 1, jr - 1, kr - 1) <= 0) {
          if (z0) rpmm = (xr && yl) ? RP(ir + 1, jr - 1) : 0.0;
          else if (yl) rpmm = xr ? G(ir + 1, jr - 1, kr - 1) : 0.0;
          else rpmm = G(ir + 1, n2, kr - 1);
        }
        double r0mm = 0.0;
        if (BC(ir, jr - 1, kr - 1) <= 0) {
          if (z0) r0mm = yl ? RP(ir, jr - 1) : 0.0;
          else r0mm = yl ? G(ir, jr - 1, kr - 1) : G(ir, n2, kr - 1);
        }
        double rmmm = 0.0;
        if (BC(ir - 1, jr - 1, kr - 1) <= 0 && xl) {
          if (z0) rmmm = yl ? RP(ir - 1, jr - 1) : 0.0;
          else rmmm = yl ? G(ir - 1, jr - 1, kr - 1) : G(ir - 1, n2, kr - 1);
        }
        double rm0m = 0.0;
        if (BC(ir - 1, jr, kr - 1) <= 0 && xl) rm0m = z0 ? RP(ir - 1, jr) : G(ir - 1, jr, kr - 1);
        double rmpm = 0.0;
        if (BC(ir - 1, jr + 1, kr - 1) <= 0 && xl && yr) rmpm = z0 ? RP(ir - 1, jr + 1) : G(ir - 1, jr + 1, kr - 1);
        double r0pm = 0.0;
        if (BC(ir, jr + 1, kr - 1) <= 0 && yr) r0pm = z0 ? RP(ir, jr + 1) : G(ir, jr + 1, kr - 1);
        re = (8.0 * r000 + 4.0 * (rp00 + rm00 + r0p0 + r0m0 + r00p + r00m) +
              2.0 * (rpp0 + rmp0 + rpm0 + rmm0 + rp0p + rm0p + r0pp + r0mp + rp0m + rm0m + r0pm + r0mm) +
              rppp + rmpp + rpmp + rmmp + rppm + rmpm + rpmm + rmmm) /
             64.0;
      }
      C.b[C.r(i, j, k)] = re;
    }
  });
  grid.sync();
}

// Src/mg.f90:849-939 (prolongation): coarse C added into fine F
__device__ void prolongation(const MGLev &F, const MGLev &C, cg::grid_group &grid) {
  const Warps w = grid_warps();
  const int lane = threadIdx.x & 31;
  const long long sy = F.N1, sz = F.N1 * F.N2;
  const long long cy = C.N1, cz = C.N1 * C.N2;
  for_rows(w, 1, C.n2 + 1, 1, C.n3 + 1, [&](int j, int k) {
    for (int i = 1 + lane; i <= C.n1 + 1; i += 32) {
      long long c = C.g(i, j, k);
      const double *E = C.u;
      double r000 = E[c], r0m0 = E[c - cy], rmm0 = E[c - 1 - cy], rm00 = E[c - 1];
      double r00m = E[c - cz], r0mm = E[c - cy - cz], rmmm = E[c - 1 - cy - cz], rm0m = E[c - 1 - cz];
      long long q = F.g(2 * i - 1, 2 * j - 1, 2 * k - 1);
      double *U = F.u;
      const int *B = F.bc;
      if (B[q] <= 0) U[q] = U[q] + r000;
      if (B[q - sy] <= 0) U[q - sy] = U[q - sy] + (r000 + r0m0) / 2.0;
      if (B[q - 1 - sy] <= 0) U[q - 1 - sy] = U[q - 1 - sy] + (r000 + r0m0 + rmm0 + rm00) / 4.0;
      if (B[q - 1] <= 0) U[q - 1] = U[q - 1] + (r000 + rm00) / 2.0;
      if (B[q - sz] <= 0) U[q - sz] = U[q - sz] + (r000 + r00m) / 2.0;
      if (B[q - sy - sz] <= 0) U[q - sy - sz] = U[q - sy - sz] + (r000 + r00m + r0mm + r0m0) / 4.0;
      if (B[q - 1 - sz] <= 0) U[q - 1 - sz] = U[q - 1 - sz] + (r000 + r00m + rm0m + rm00) / 4.0;
      if (B[q - 1 - sy - sz] <= 0)
        U[q - 1 - sy - sz] =
            U[q - 1 - sy - sz] + (r000 + r00m + rm0m + rm00 + r0m0 + r0mm + rmmm + rmm0) / 8.0;
    }
  });
  grid.sync();
}

template <bool GEN>
__global__ void __launch_bounds__(MG_BLOCK) k_pdesolver(const MGArgs *__restrict__ ap) {
  cg::grid_group grid = cg::this_grid();
  const MGArgs &a = *ap;
  __shared__ double sh[40];
  const int ng = a.ng;
  int k = 1;
  double res_s = 0.0, ktot = 0.0, r = 0.0;
  int status = 0;
  bool converged = false;
  while (!converged) {
    int iter[MG_MAX + 1];
    for (int i = 0; i <= MG_MAX; ++i) iter[i] = 0;
    const double eps_abs = a.alpha * a.eps;
    for (int ig = 1; ig <= 2 * ng - 1; ++ig) {
      int ksor = 0;
      if (ig < ng) {
        int il = ig;
        sor_rb<GEN>(a, a.L[il], k, ig - ng, eps_abs, grid, sh, r, ksor);
        iter[il] += ksor;
        if (GEN)
          restriction_gen(a, a.L[il], a.L[il + 1], grid);
        else
          restriction(a.L[il], a.L[il + 1], grid);
      } else if (ig == ng) {
        sor_rb<GEN>(a, a.L[ng], k, 0, eps_abs, grid, sh, r, ksor);
        iter[ng] += ksor;
        if (ng >= 2) prolongation(a.L[ng - 1], a.L[ng], grid);
      } else {
        int il = 2 * ng - ig;
        sor_rb<GEN>(a, a.L[il], k, ig - ng, eps_abs, grid, sh, r, ksor);
        iter[il] += ksor;
        if (il >= 2) prolongation(a.L[il - 1], a.L[il], grid);
      }
    }
    for (int i = 1; i <= ng; ++i) ktot = ktot + (double)(float)iter[i] / exp2((double)(2 * (i - 1)));
    r = r / a.alpha;
    if (k == 1) {
      res_s = r;
    } else if (fabs(r / res_s) > 10.0) {
      status = LEPIC_ERR_DIVERGED;
      converged = true;
    }
    if (r < a.eps || k == a.ncycl) converged = true;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      for (int i = 1; i <= ng; ++i) a.out_i[2 + i] = iter[i];
    }
    k = k + 1;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.out_i[0] = k;
    a.out_i[1] = status;
    a.out_d[0] = ktot;
    a.out_d[1] = r;
  }
}

// ------------------------------------------------ colour-split Dirichlet solve
// The same schedule and the same node arithmetic on colour-split levels
// (mgsplit.cuh), for Dirichlet walls.  What it changes is how many grid
// barriers a sweep costs and what a phase reads:
//   * a sweep is two phases, red and black, and no third one for its residual:
//     the black nodes' share is summed in the black phase (their neighbours
//     are final there) and the red nodes' share in the next sweep's red phase,
//     which writes its new values into a second buffer that is dropped when
//     the residual ends the smoothing;
//   * a residual that nothing reads (that of the fourth sweep, but for the
//     last smoothing of a cycle) is not computed;
//   * the levels that fit the shared memory of one SM are smoothed there by
//     block 0.
// Measured against the general kernel: 128^3 with electrodes, cold, to 1e-10
// 13.8 -> 4.06 ms (13 cycles; a red or black phase of level 1 takes 8 us for
// the 52 MB it moves through L2, one of a small level 2 to 3 us with its
// barrier); in the step loop 40x24x32 1.17 -> 0.43 ms, 96^3 4.5 -> 0.94 ms.
// What bounds it is latency, of L2 on the finest level and of barriers and
// dependent FP64 operations below: at 128^3 19.2 GB go through L2 at 4.8 TB/s,
// 15 % of what it can do, the SMs issue 16 % of the time with their 16 warps
// and the FP64 pipe is 11 % busy.
// 512 threads: with 768 and 1024 the phases spill (128^3: 4.8 and 5.8 ms when
// 512 took 4.4).
constexpr int SP_BLOCK = 512;
// elements per colour up to which one cluster solves faster than the grid
// (cold solves by the grid and by a cluster: 32x24x32, 17,000, 577 and 505 us;
// 40x32x40, 33,100, 676 and 616; 48x40x32, 39,100, 683 and 684; 40x40x48,
// 48,200, 705 and 713; 48^3, 67,600, 778 and 859; 56^3, 1102 and 1438)
constexpr long long SP_SMALL = 40000;
static_assert(MG_MAX == mgs::LEVELS, "the shared memory of their descriptors");

struct SPArgs {
  mgs::Lev<double> L[MG_MAX + 2];   // levels 1..ng; after them level ls + 1 with its arrays on the grid
  unsigned oc[MG_MAX + 1];          // levels ls+1..ng: byte offset of their arrays on chip
  unsigned ol;                      // and of the level descriptors
  int ng, ls, ncycl;
  double alpha, eps, omega;
  double *u;                  // the caller's grid arrays
  const double *b;
  const int *bc;
  double *partial;            // [2][gridDim.x]
  int *out_i;
  double *out_d;
  double *host;               // pinned host memory for k, status, ktot, res (or null)
  GridBarrier barrier;
};

extern __shared__ __align__(16) unsigned char sp_smem[];

// the descriptors, copied to shared memory by every block: read from the
// kernel's parameters level by level they cost microseconds of constant-cache
// misses per smoothing call
__device__ __forceinline__ const mgs::Lev<double> &lev(const SPArgs &a, int l) {
  return reinterpret_cast<const mgs::Lev<double> *>(sp_smem + a.ol)[l - 1];
}

// deterministic sum over the team of one value per thread in two steps: each
// caller's share into slot `set` before a barrier, the total after it (every
// warp adds the shares up in the same order)
template <bool GRID>
__device__ __forceinline__ void share(double v, int set, double *sh, double *partial) {
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  v = warp_sum(v);
  if (!GRID) {
    if (lane == 0) sh[32 * set + wp] = v;
    return;
  }
  if (lane == 0) sh[wp] = v;
  __syncthreads();
  if (wp == 0) {
    v = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
    v = warp_sum(v);
    if (lane == 0) partial[set * gridDim.x + blockIdx.x] = v;
  }
}
template <bool GRID>
__device__ __forceinline__ double total(int set, const double *sh, const double *partial) {
  const int lane = threadIdx.x & 31;
  double v = 0.0;
  if (GRID) {
    for (int q = lane; q < (int)gridDim.x; q += 32) v += partial[set * gridDim.x + q];
  } else {
    v = lane < (int)(blockDim.x >> 5) ? sh[32 * set + lane] : 0.0;
  }
  return warp_sum(v);
}

// level l on the grid / on chip (block 0)
template <bool GRID>
__device__ __forceinline__ const mgs::Lev<double> &level_of(const SPArgs &a, int l) {
  return lev(a, GRID && l == a.ls + 1 ? a.ng + 1 : l);
}
// the red half of a level's residual: below level 1 it lies in the red buffer
// that is not current (walls and ghosts are 0 in both)
__device__ __forceinline__ double *residual_red(const mgs::Lev<double> &L, int cur) {
  return L.rf[mgs::RED] ? L.rf[mgs::RED] : L.red[cur ^ 1];
}

// Src/sors.f90:1-535: up to four sweeps (the coarsest level of the first
// cycle: until res <= eps_abs), ended early when a sweep's residual is at
// most 0.6 of the one before; cur: the current red buffer.  The residual of
// sweep l - 1 is known after the red phase of sweep l.  Returns the last
// sweep's residual when need_res, the sweeps done in ksor.  started: the
// restriction has done the first sweep's red phase.
template <bool GRID, class Sync>
__device__ __forceinline__ double smooth(const SPArgs &a, int level, int &cur, bool first, int dig, bool need_res,
                                         bool started, Sync &grid, double *sh, int &ksor) {
  using namespace mgs;
  const Lev<double> &L = level_of<GRID>(a, level);
  const Team w = GRID ? grid_team() : block_team();
  const double om = a.omega, eps_abs = a.alpha * a.eps;
  const int nr = (first && dig == 0) ? 1000000 : 4;
  auto barrier = [&]() {
    if (GRID)
      grid.sync();
    else
      __syncthreads();
  };
  double res = 0.0, part = 0.0;
  bool stopped = false;
  ksor = nr;
  for (int l = 1; l <= nr; ++l) {
    if (l == 1 && started) {
      cur ^= 1;   // taken back below: the values stand in the current buffer
    } else if (l == 1) {
      colour_phase<double, 2, RED, DO_RELAX, !GRID>(L, L.red[cur], L.red[cur ^ 1], L.black, om, w);
      barrier();
    } else {
      part += colour_phase<double, 2, RED, DO_RELAX | DO_RES, !GRID>(L, L.red[cur], L.red[cur ^ 1], L.black, om, w);
      share<GRID>(part, l & 1, sh, a.partial);
      barrier();
      if (dig == 0) {
        res = total<GRID>(l & 1, sh, a.partial);
        stopped = res <= eps_abs;
        if (l % SWEEPS_PER_BEAT == 0) {
          if (!GRID)
            grid.beat();
          else if (grid.dead())
            stopped = true;
        }
      } else if (l >= 3) {
        const double before = l == 3 ? total<GRID>((l - 1) & 1, sh, a.partial) : res;
        res = total<GRID>(l & 1, sh, a.partial);
        stopped = before > 0.0 && res / before <= 0.6;
      }
      if (stopped) {
        ksor = l - 1;
        break;
      }
    }
    cur ^= 1;
    if (l < nr || need_res)
      part = colour_phase<double, 2, BLACK, DO_RELAX | DO_RES, !GRID>(L, L.black, L.black, L.red[cur], om, w);
    else
      colour_phase<double, 2, BLACK, DO_RELAX, !GRID>(L, L.black, L.black, L.red[cur], om, w);
    barrier();
  }
  if (need_res && !stopped) {
    part += colour_phase<double, 2, RED, DO_RES, !GRID>(L, L.red[cur], nullptr, L.black, om, w);
    share<GRID>(part, 1, sh, a.partial);   // sweep 4 (l = 5)
    barrier();
    res = total<GRID>(1, sh, a.partial);
  }
  return res;
}

// the residual of a level weighted onto the next one
template <bool GRID, class Sync>
__device__ __forceinline__ void restrict_level(const SPArgs &a, int level, int cur, bool masks, Sync &grid) {
  using namespace mgs;
  const Lev<double> &F = level_of<GRID>(a, level), &C = level_of<GRID>(a, level + 1);
  double *R = residual_red(F, cur);
  const Team w = GRID ? grid_team() : block_team();
  residual_colour<double, 2, RED, !GRID>(F, F.red[cur], F.black, R, w);
  residual_colour<double, 2, BLACK, !GRID>(F, F.black, F.red[cur], F.rf[BLACK], w);
  if (GRID)
    grid.sync();
  else
    __syncthreads();
  restrict_to<double, !GRID>(F, C, R, F.rf[BLACK], masks, true, a.omega, w);
  if (GRID)
    grid.sync();
  else
    __syncthreads();
}

// the part of a V-cycle on the levels on chip, by block 0
template <class Sync>
__device__ __forceinline__ void chip_cycle(const SPArgs &a, bool first, int *iter, Sync &grid, double *sh) {
  using namespace mgs;
  const int top = a.ls + 1, ng = a.ng, t0 = threadIdx.x, bd = blockDim.x;
  int cur[MG_MAX + 1];
  const Lev<double> &X = level_of<true>(a, top);
  {
    // two elements per thread and turn, every load before the first store
    const Lev<double> &L = level_of<false>(a, top);
    for (int e = 2 * t0; e < L.len; e += 2 * bd) {
      const Vec<double, 2> b0 = ldv<double, 2>(X.b[0] + e), b1 = ldv<double, 2>(X.b[1] + e),
                           r0 = ldv<double, 2>(X.red[0] + e);   // the first red phase is done
      const unsigned short m = first ? *reinterpret_cast<const unsigned short *>(X.m + e) : 0;
      const Vec<double, 2> zero = {{0.0, 0.0}};
      stv<double, 2>(L.b[0] + e, b0);
      stv<double, 2>(L.b[1] + e, b1);
      stv<double, 2>(L.red[0] + e, r0);
      stv<double, 2>(L.black + e, zero);
      if (first || e < L.HN || e >= L.HN * (L.n3 + 2)) stv<double, 2>(L.red[1] + e, zero);   // planes no red phase writes
      if (first) {
        *reinterpret_cast<unsigned short *>(L.m + e) = m;
        if (L.rf[BLACK]) stv<double, 2>(L.rf[BLACK] + e, zero);
      }
    }
    __syncthreads();
  }
  // down to the coarsest level and up again (one call site per step: the
  // loops keep their registers)
  const int mid = ng - top;
  for (int g = 0; g <= 2 * mid; ++g) {
    const int l = g <= mid ? top + g : ng - (g - mid);
    if (g <= mid) cur[l] = 0;
    if (g > mid) {
      const Lev<double> &F = level_of<false>(a, l), &C = level_of<false>(a, l + 1);
      prolong_to<double, true>(F, C, F.red[cur[l]], F.red[cur[l] ^ 1], C.red[cur[l + 1]], block_team());
      __syncthreads();
    }
    int k = 0;
    smooth<false>(a, l, cur[l], first, g <= mid ? l - ng : ng - l, false, g <= mid, grid, sh, k);
    iter[l] += k;
    if (g < mid) restrict_level<false>(a, l, cur[l], first, grid);
  }
  const Lev<double> &L = level_of<false>(a, top);
  for (int e = 2 * t0; e < L.len; e += 2 * bd) {
    stv<double, 2>(X.red[0] + e, ldv<double, 2>(L.red[cur[top]] + e));
    stv<double, 2>(X.black + e, ldv<double, 2>(L.black + e));
  }
}

// the caller's grids into the split arrays of level 1 and back
__device__ __noinline__ void split_in(const SPArgs &a) {
  using namespace mgs;
  const Lev<double> &L = lev(a, 1);
  const long long N1 = L.n1 + 3, R1 = L.n1 + 2, R2 = L.n2 + 2;
  const int last = L.n1 + 2;
  elements(L, grid_team(), [&](int e, int ii, int j, int k) {
    // the row's nodes i = 2 ii and 2 ii + 1: one of each colour
    const long long q = 2 * ii + N1 * (j + (long long)L.N2 * k), qb = 2 * ii + R1 * (j + R2 * (long long)k);
    const bool jk = j >= 1 && k >= 1 && j <= L.n2 + 1 && k <= L.n3 + 1;
    const int odd = (j + k + 1) & 1;   // the colour of i odd is RED when j + k is even
    unsigned m = 0;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int i = 2 * ii + x, c = x ? odd ^ 1 : odd;
      double u = 0.0, b = 0.0;
      unsigned bits = x ? MB_ODD : 0;
      if (i <= last) {
        u = a.u[q + x];
        const int bc = a.bc[q + x];
        if (bc <= 0) bits |= MB_FREE;
        if (jk && i >= 1 && i <= L.n1 + 1) {
          b = a.b[qb + x];
          bits |= (bc <= 0 ? MB_UPD : 0) | (bc == -1 ? MB_PLASMA : 0);
        }
      }
      m |= MB(c, bits);
      L.b[c][e] = b;
      if (L.rf[c]) L.rf[c][e] = 0.0;
      (c == RED ? L.red[0] : L.black)[e] = u;
      if (c == RED) L.red[1][e] = u;
    }
    L.m[e] = (unsigned char)m;
  });
}
__device__ __noinline__ void split_out(const SPArgs &a, int cur) {
  using namespace mgs;
  const Lev<double> &L = lev(a, 1);
  const double *red = L.red[cur];
  elements(L, grid_team(), [&](int e, int ii, int j, int k) {
    const unsigned m = L.m[e];
    const int odd = (j + k + 1) & 1;
    double *u = a.u + 2 * ii + (long long)(L.n1 + 3) * (j + (long long)L.N2 * k);
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int c = x ? odd ^ 1 : odd;
      if (m & MB(c, MB_FREE)) u[x] = c == RED ? red[e] : L.black[e];
    }
  });
}

template <class Sync>
__global__ void __launch_bounds__(SP_BLOCK, 1) k_pdesolver_split(const __grid_constant__ SPArgs a) {
  using namespace mgs;
  Sync grid(a.barrier);
  __shared__ double sh[64];
  const int ng = a.ng, ls = a.ls, down = ls < ng ? ls : ng - 1;   // down: the last grid level restricted from
  unsigned curs = 0;   // bit l: the current red buffer of grid level l
  {
    const int words = (int)(sizeof(Lev<double>) / 4) * (ng + 1);
    const unsigned *from = reinterpret_cast<const unsigned *>(a.L + 1);
    for (int q = threadIdx.x; q < words; q += blockDim.x) reinterpret_cast<unsigned *>(sp_smem + a.ol)[q] = from[q];
    __syncthreads();
    // the levels on chip: their arrays in this block's shared memory
    const int l = ls + 1 + threadIdx.x;
    if (l <= ng) {
      Lev<double> &L = const_cast<Lev<double> &>(lev(a, l));
      double *p = reinterpret_cast<double *>(sp_smem + a.oc[l]);
      const int n = L.len;
      L.red[0] = p;
      L.red[1] = p + n;
      L.black = p + 2 * n;
      L.b[0] = p + 3 * n;
      L.b[1] = p + 4 * n;
      L.rf[BLACK] = l == ng ? nullptr : p + 5 * n;
      L.m = reinterpret_cast<unsigned char *>(p + (l == ng ? 5 : 6) * n);
    }
  }
  __syncthreads();
  split_in(a);
  grid.sync();
  double res_s = 0.0, ktot = 0.0, r = 0.0;
  int status = 0, k = 1;
  bool converged = false;
  while (!converged && !grid.dead()) {
    const bool first = k == 1;
    int iter[MG_MAX + 1];
    for (int i = 0; i <= MG_MAX; ++i) iter[i] = 0;
    // grid levels down, the coarsest level or the levels on chip, grid levels
    // up (one call site per step)
    const int mid = down + 1;
    for (int g = 1; g <= 2 * down + 1; ++g) {
      if (g == mid && ls < ng) {
        if (blockIdx.x == 0 && !grid.dead()) chip_cycle(a, first, iter, grid, sh);
        grid.sync();
        continue;
      }
      const int l = g <= mid ? g : 2 * mid - g;
      int cur = (curs >> l) & 1, ks = 0;
      if (g > mid) {
        const Lev<double> &F = level_of<true>(a, l), &C = level_of<true>(a, l + 1);
        prolong_to<double>(F, C, F.red[cur], F.red[cur ^ 1], C.red[(curs >> (l + 1)) & 1], grid_team());
        grid.sync();
      }
      r = smooth<true>(a, l, cur, first, g <= mid ? l - ng : ng - l, g == 2 * down + 1, g > 1 && g <= mid, grid, sh,
                       ks);
      iter[l] += ks;
      curs = (curs & ~(1u << l)) | ((unsigned)cur << l);
      if (g < mid) {
        restrict_level<true>(a, l, cur, first, grid);
        curs &= ~(2u << l);   // level l + 1 starts in its first buffer
      }
    }
    for (int i = 1; i <= ng; ++i) ktot = ktot + (double)(float)iter[i] / exp2((double)(2 * (i - 1)));
    r = r / a.alpha;
    if (first) {
      res_s = r;
    } else if (fabs(r / res_s) > 10.0) {
      status = LEPIC_ERR_DIVERGED;
      converged = true;
    }
    if (r < a.eps || k == a.ncycl) converged = true;
    if (blockIdx.x == 0 && threadIdx.x == 0)
      for (int i = 1; i <= ng; ++i) a.out_i[2 + i] = iter[i];
    k = k + 1;
  }
  if (!grid.dead()) split_out(a, (curs >> 1) & 1);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.out_i[0] = k;
    a.out_i[1] = status;
    a.out_d[0] = ktot;
    a.out_d[1] = r;
    if (a.host) {
      a.host[0] = k;
      a.host[1] = status;
      a.host[2] = ktot;
      a.host[3] = r;
    }
  }
  grid.leave(a.out_i + 1, a.host ? a.host + 1 : nullptr);
}

// the solve's results to the host: waits for the stream, returns the status
int solve_results(const int *out_i, const double *out_d, int *k_out, double *ktot_out, double *res_out,
                  cudaStream_t s) {
  int hi[2];
  double hd[2];
  LEPIC_CUDA(cudaMemcpyAsync(hi, out_i, sizeof(hi), cudaMemcpyDeviceToHost, s));
  LEPIC_CUDA(cudaMemcpyAsync(hd, out_d, sizeof(hd), cudaMemcpyDeviceToHost, s));
  LEPIC_CUDA(cudaStreamSynchronize(s));
  if (k_out) *k_out = hi[0];
  if (ktot_out) *ktot_out = hd[0];
  if (res_out) *res_out = hd[1];
  return hi[1];
}

// The split solve's arrays and launch; LEPIC_OK with launched = false where it
// does not apply (a level with too many nodes for its 32-bit element numbers,
// coefficients out of div_by's range, no device memory for its copies: 32
// bytes per grid node, against 12 of the general kernel): the caller takes the
// general kernel.
int launch_split(const int n[3], const double h[3], double *u, const double *b, const int *bcnd, int ncycl,
                 double eps, double omega, int ng, double eps0, int *out_i, double *out_d, double *host,
                 cudaStream_t s, bool &launched, unsigned rounds) {
  using Lev = mgs::Lev<double>;
  launched = false;
  if (Lev::elements(n[0], n[1], n[2]) >= 2130000000LL) return LEPIC_OK;
  SPArgs A;
  memset(&A, 0, sizeof(A));
  A.ng = ng;
  A.ncycl = ncycl;
  A.eps = eps;
  A.omega = omega;
  A.u = u;
  A.b = b;
  A.bc = bcnd;
  A.out_i = out_i;
  A.out_d = out_d;
  A.host = host;
  A.barrier = grid_barrier(rounds);
  if (!A.barrier.line) return LEPIC_ERR_CUDA;
  for (int l = 1; l <= ng; ++l) {
    Lev &L = A.L[l];
    L.shape(n[0] >> (l - 1), n[1] >> (l - 1), n[2] >> (l - 1));
    double hl[3];
    for (int q = 0; q < 3; ++q) hl[q] = h[q] * (double)(1 << (l - 1));
    L.aw = eps0 / (hl[0] * hl[0]);
    L.an = eps0 / (hl[1] * hl[1]);
    L.at = eps0 / (hl[2] * hl[2]);
    L.ac = -(L.an + L.an + L.aw + L.aw + L.at + L.at);
    L.rac = 1.0 / L.ac;
  }
  if (!(fabs(A.L[1].ac) < 1e100 && fabs(A.L[ng].ac) > 1e-100)) return LEPIC_OK;   // div_by's range
  // the levels that fit on chip (level 1 stays on the grid): per element two
  // red and one black value, b of both, the black residual, one byte
  size_t csm = 0;
  A.ls = ng;
  for (int l = ng; l >= 2; --l) {
    const size_t need = ((size_t)A.L[l].len * (8 * (l == ng ? 5 : 6) + 1) + 15) & ~(size_t)15;
    if (csm + need > mgs::CHIP) break;
    A.oc[l] = (unsigned)csm;
    csm += need;
    A.ls = l - 1;
  }
  A.ol = (unsigned)csm;
  csm += sizeof(Lev) * (ng + 1);
  if (A.ls < ng) A.L[ng + 1] = A.L[A.ls + 1];
  for (int l = 1; l <= A.ls + 1 && l <= ng; ++l) {
    Lev &L = A.L[l <= A.ls ? l : ng + 1];
    // one allocation per level: red twice, black, b twice, and on the levels
    // that restrict the residual (its red half in the spare red buffer but
    // on level 1, whose walls are not 0)
    const size_t n8 = (size_t)L.len;
    const bool restricts = l <= A.ls && l < ng;
    const int halves = 5 + (restricts ? (l == 1 ? 2 : 1) : 0);
    char nm[32];
    snprintf(nm, sizeof nm, "mgs_%d", l);
    double *p = (double *)scratch(nm, (sizeof(double) * halves + 1) * n8);
    if (!p) {
      cudaGetLastError();
      scratch_drop("mgs_");   // the general kernel may need what the other levels took
      return LEPIC_OK;
    }
    L.red[0] = p;
    L.red[1] = p + n8;
    L.black = p + 2 * n8;
    L.b[0] = p + 3 * n8;
    L.b[1] = p + 4 * n8;
    if (restricts) {
      L.rf[mgs::BLACK] = p + 5 * n8;
      if (l == 1) L.rf[mgs::RED] = p + 6 * n8;
    }
    L.m = reinterpret_cast<unsigned char *>(p + halves * n8);
  }
  A.alpha = residual_scale(n, A.L[1].ac);
  const int blocks = ctx().sms;
  A.partial = (double *)scratch("mgs_partial", sizeof(double) * 2 * blocks);
  if (!A.partial) return LEPIC_ERR_CUDA;
  void *args[] = {&A};
  int tm = timer_start("pdesolver_f64", s);
  LEPIC_CUDA(mgs::launch_solve((const void *)k_pdesolver_split<mgs::GridSync>,
                               (const void *)k_pdesolver_split<mgs::ClusterSync>, args, A.L[1].len, SP_SMALL, SP_BLOCK,
                               csm, blocks, s));
  timer_stop(tm, s);
  launched = true;
  return LEPIC_OK;
}

}  // namespace

int launch_pdesolver(const Dims &d, const double h[3], double *u, const double *b, const int *bcnd,
                     int ncycl, double eps, double omega, int ng, double eps0, int *k_out,
                     double *ktot_out, double *res_out, cudaStream_t s, int pbc, int nmn, unsigned rounds) {
  if (ng < 1 || ng > MG_MAX) return LEPIC_ERR_ARG;
  const bool gen = pbc || nmn;
  int n[3] = {d.n1, d.n2, d.n3};
  for (int a = 0; a < 3; ++a)
    if (n[a] % (1 << (ng - 1))) return LEPIC_ERR_ARG;
  Ctx &c = ctx();
  int *out_i = (int *)scratch("mg_out_i", sizeof(int) * (MG_MAX + 4));
  double *out_d = (double *)scratch("mg_out_d", sizeof(double) * 2);
  if (!out_i || !out_d) return LEPIC_ERR_CUDA;
  bool launched = false;
  double *host = gen ? nullptr : result_block();
  if (!gen)
    if (int rc = launch_split(n, h, u, b, bcnd, ncycl, eps, omega, ng, eps0, out_i, out_d, host, s, launched, rounds))
      return rc;
  if (launched && host) {
    LEPIC_CUDA(cudaStreamSynchronize(s));
    if (k_out) *k_out = (int)host[0];
    if (ktot_out) *ktot_out = host[2];
    if (res_out) *res_out = host[3];
    return (int)host[1];
  }
  if (launched) return solve_results(out_i, out_d, k_out, ktot_out, res_out, s);
  MGArgs A;
  memset(&A, 0, sizeof(A));
  A.ng = ng;
  A.ncycl = ncycl;
  A.eps = eps;
  A.omega = omega;
  A.pbc = pbc ? 1 : 0;
  A.nmn = nmn ? 1 : 0;
  char nm[32];
  for (int l = 1; l <= ng; ++l) {
    MGLev &L = A.L[l];
    L.n1 = n[0] >> (l - 1);
    L.n2 = n[1] >> (l - 1);
    L.n3 = n[2] >> (l - 1);
    L.N1 = L.n1 + 3;
    L.N2 = L.n2 + 3;
    L.R1 = L.n1 + 2;
    L.R2 = L.n2 + 2;
    double hl[3];
    for (int q = 0; q < 3; ++q) hl[q] = h[q] * (double)(1 << (l - 1));
    L.aw = eps0 / (hl[0] * hl[0]);
    L.ae = L.aw;
    L.an = eps0 / (hl[1] * hl[1]);
    L.as = L.an;
    L.at = eps0 / (hl[2] * hl[2]);
    L.ab = L.at;
    L.ac = -(L.an + L.as + L.aw + L.ae + L.at + L.ab);
    long long nn = (long long)(L.n1 + 3) * (L.n2 + 3) * (L.n3 + 3);
    long long nr = (long long)(L.n1 + 2) * (L.n2 + 2) * (L.n3 + 2);
    if (l == 1) {
      L.u = u;
      L.b = const_cast<double *>(b);
      L.bc = const_cast<int *>(bcnd);
    } else {
      snprintf(nm, sizeof nm, "mg_e%d", l);
      L.u = (double *)scratch(nm, sizeof(double) * nn);
      snprintf(nm, sizeof nm, "mg_r%d", l);
      L.b = (double *)scratch(nm, sizeof(double) * nr);
      snprintf(nm, sizeof nm, "mg_bc%d", l);
      L.bc = (int *)scratch(nm, sizeof(int) * nn);
      if (!L.u || !L.b || !L.bc) return LEPIC_ERR_CUDA;
    }
    if (l < ng) {
      snprintf(nm, sizeof nm, "mg_rf%d", l);
      L.rf = (double *)scratch(nm, sizeof(double) * nn);
      if (!L.rf) return LEPIC_ERR_CUDA;
      LEPIC_CUDA(cudaMemsetAsync(L.rf, 0, sizeof(double) * nn, s));
      if (gen) {
        snprintf(nm, sizeof nm, "mg_rp%d", l);
        L.rp = (double *)scratch(nm, sizeof(double) * (size_t)(L.n1 + 2) * (L.n2 + 2));
        if (!L.rp) return LEPIC_ERR_CUDA;
      }
    }
  }
  double ac = A.L[1].ac;
  A.alpha = residual_scale(n, ac);
  void *kern = gen ? (void *)k_pdesolver<true> : (void *)k_pdesolver<false>;
  int occ = 0;
  LEPIC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, MG_BLOCK, 0));
  if (occ < 1) return LEPIC_ERR_CUDA;
  int blocks = c.sms * (occ < 2 ? occ : 2);
  A.partial = (double *)scratch("mg_partial", sizeof(double) * blocks);
  A.shared_d = (double *)scratch("mg_shared", sizeof(double) * 4);
  A.out_i = out_i;
  A.out_d = out_d;
  if (!A.partial || !A.shared_d) return LEPIC_ERR_CUDA;
  MGArgs *dA = (MGArgs *)scratch("mg_args", sizeof(MGArgs));
  if (!dA) return LEPIC_ERR_CUDA;
  LEPIC_CUDA(cudaMemcpyAsync(dA, &A, sizeof(MGArgs), cudaMemcpyHostToDevice, s));
  void *args[] = {&dA};
  int tm = timer_start("pdesolver_f64", s);
  LEPIC_CUDA(cudaLaunchCooperativeKernel(kern, dim3(blocks), dim3(MG_BLOCK), args, 0, s));
  timer_stop(tm, s);
  return solve_results(out_i, out_d, k_out, ktot_out, res_out, s);
}

}  // namespace lepic

// ---------------------------------------------------------------------------
// Allocation-free variant of the Poisson solve.
//
// Some callers cannot call cudaMalloc once their time loop runs: a Fortran
// driver (or a framework such as PyTorch) that owns the device memory through
// its own pool hands every buffer in and forbids allocations inside the loop,
// because cudaMalloc synchronises the whole device and fails once the pool has
// claimed the memory.  lepic_dev_pdesolver_noalloc runs the same cooperative
// kernel as lepic_dev_pdesolver, but carves all of its scratch (the level
// arrays e, r, bcnd and the fine residuals of levels 2..ng, the block partial
// sums, the argument block and the outputs) out of one file-scope device array
// of MG_NOALLOC_BYTES bytes, which every GPU that loads the library holds until
// the process exits.  The caller still passes u, b and bcnd.
// ---------------------------------------------------------------------------
namespace lepic {
namespace {

constexpr size_t MG_NOALLOC_BYTES = 8u << 20;  // 8 MiB: grids up to 64^3 cells
static __device__ __align__(256) unsigned char g_mg_noalloc_scratch[MG_NOALLOC_BYTES];

constexpr int MG_NOALLOC_MAX_DEVICES = 64;
unsigned char *g_noalloc_ptr[MG_NOALLOC_MAX_DEVICES] = {nullptr};

inline size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

}  // namespace

}  // namespace lepic

extern "C" int lepic_dev_pdesolver_noalloc(const lepic_grid_t *g, double *u, const double *b,
                                           int ncycl, double eps, double omega, int ng,
                                           const lepic_phys_t *P, int *k_out, double *ktot_out,
                                           double *res_out, void *stream) {
  using namespace lepic;
  if (!g || !P) return LEPIC_ERR_ARG;
  if (P->flag_pbc || P->flag_nmn) return LEPIC_ERR_UNSUPPORTED;
  if (ng < 1 || ng > MG_MAX) return LEPIC_ERR_ARG;
  const int n[3] = {g->n[0], g->n[1], g->n[2]};
  for (int a = 0; a < 3; ++a)
    if (n[a] < 1 || n[a] % (1 << (ng - 1))) return LEPIC_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  int dev = 0;
  LEPIC_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= MG_NOALLOC_MAX_DEVICES) return LEPIC_ERR_ARG;
  // Set-up, once per device with that device current: the host-side name of
  // the __device__ array is not a device address, so look the address up.
  if (!g_noalloc_ptr[dev]) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_mg_noalloc_scratch);
    if (e != cudaSuccess) return cuda_status(e, "cudaGetSymbolAddress(g_mg_noalloc_scratch)");
    g_noalloc_ptr[dev] = (unsigned char *)p;
  }
  unsigned char *base = g_noalloc_ptr[dev];
  int sms = 0, occ = 0;
  LEPIC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  LEPIC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_pdesolver<false>, MG_BLOCK, 0));
  if (occ < 1 || sms < 1) return LEPIC_ERR_CUDA;
  const int blocks = sms * (occ < 2 ? occ : 2);

  MGArgs A;
  memset(&A, 0, sizeof(A));
  A.ng = ng;
  A.ncycl = ncycl;
  A.eps = eps;
  A.omega = omega;
  // carve the scratch array; rf regions are recorded to be zeroed
  size_t off = 0;
  auto carve = [&](size_t bytes) -> unsigned char * {
    size_t at = off;
    off = align256(off + bytes);
    return off <= MG_NOALLOC_BYTES ? base + at : nullptr;
  };
  MGArgs *dA = (MGArgs *)carve(sizeof(MGArgs));
  A.partial = (double *)carve(sizeof(double) * blocks);
  A.shared_d = (double *)carve(sizeof(double) * 4);
  A.out_i = (int *)carve(sizeof(int) * (MG_MAX + 4));
  A.out_d = (double *)carve(sizeof(double) * 2);
  double *rf_ptr[MG_MAX + 1] = {nullptr};
  size_t rf_bytes[MG_MAX + 1] = {0};
  bool fits = dA && A.partial && A.shared_d && A.out_i && A.out_d;
  for (int l = 1; l <= ng && fits; ++l) {
    MGLev &L = A.L[l];
    L.n1 = n[0] >> (l - 1);
    L.n2 = n[1] >> (l - 1);
    L.n3 = n[2] >> (l - 1);
    L.N1 = L.n1 + 3;
    L.N2 = L.n2 + 3;
    L.R1 = L.n1 + 2;
    L.R2 = L.n2 + 2;
    double hl[3];
    for (int q = 0; q < 3; ++q) hl[q] = g->h[q] * (double)(1 << (l - 1));
    L.aw = P->eps0 / (hl[0] * hl[0]);
    L.ae = L.aw;
    L.an = P->eps0 / (hl[1] * hl[1]);
    L.as = L.an;
    L.at = P->eps0 / (hl[2] * hl[2]);
    L.ab = L.at;
    L.ac = -(L.an + L.as + L.aw + L.ae + L.at + L.ab);
    const size_t nn = (size_t)(L.n1 + 3) * (L.n2 + 3) * (L.n3 + 3);
    const size_t nr = (size_t)(L.n1 + 2) * (L.n2 + 2) * (L.n3 + 2);
    if (l == 1) {
      L.u = u;
      L.b = const_cast<double *>(b);
      L.bc = const_cast<int *>(g->bcnd);
    } else {
      L.u = (double *)carve(sizeof(double) * nn);
      L.b = (double *)carve(sizeof(double) * nr);
      L.bc = (int *)carve(sizeof(int) * nn);
      fits = fits && L.u && L.b && L.bc;
    }
    if (l < ng) {
      L.rf = (double *)carve(sizeof(double) * nn);
      rf_ptr[l] = L.rf;
      rf_bytes[l] = sizeof(double) * nn;
      fits = fits && L.rf;
    }
  }
  if (!fits) {
    fprintf(stderr,
            "lepic_dev_pdesolver_noalloc: a %dx%dx%d grid with %d levels needs more than the %zu "
            "bytes of static scratch (grids up to 64^3 cells fit); use lepic_dev_pdesolver\n",
            n[0], n[1], n[2], ng, MG_NOALLOC_BYTES);
    return LEPIC_ERR_SCRATCH_LIMIT;
  }
  A.alpha = residual_scale(n, A.L[1].ac);
  // the shared array keeps the previous call's contents: clear the fine
  // residual arrays whose ghost entries the restriction may read
  for (int l = 1; l < ng; ++l) LEPIC_CUDA(cudaMemsetAsync(rf_ptr[l], 0, rf_bytes[l], s));
  LEPIC_CUDA(cudaMemcpyAsync(dA, &A, sizeof(MGArgs), cudaMemcpyHostToDevice, s));
  void *args[] = {&dA};
  LEPIC_CUDA(cudaLaunchCooperativeKernel((void *)k_pdesolver<false>, dim3(blocks), dim3(MG_BLOCK), args, 0, s));
  return solve_results(A.out_i, A.out_d, k_out, ktot_out, res_out, s);
}
