// Mixed-precision Poisson solve: FP32 multigrid V-cycles inside an FP64
// iterative-refinement loop, as one persistent cooperative kernel.
//
//   repeat:  r = b - A u          (FP64, plasma nodes; L1 norm -> exit test
//                                   res/alpha < eps of Src/pdesolver.f90:91-111)
//            A e = r  approx.     (one FP32 V-cycle, zero initial guess)
//            u = u + e            (FP64)
//
// The operators are the reference's (Src/mg.h, Src/sors.f90 red-black SOR,
// Src/mg.f90 27-point full-weighting restriction and trilinear
// prolongation), evaluated in FP32 on the correction; only the residual and
// the accumulation of u are FP64, so u converges to the FP64 solution while
// the V-cycle moves half the bytes.
//
// All levels are colour-split (mgsplit.cuh): a red or black phase reads and
// writes only what it needs, 16 bytes per load, and finds walls and parity in
// one byte per element.  What bounds a solve is the number of grid phases
// (2 to 3 us for one of a small level with its barrier) and, on large grids,
// the values moved through L2 and HBM (256^3: 41.8 GB through HBM, 0.58 of the
// measured copy bandwidth, and 101 GB through L2).  A refinement therefore has
// as few phases as its schedule allows:
//   * u and b are held as colour-split FP64 copies for the solve, so the FP64
//     residual is one phase of vector loads, which also does the first
//     sweep's red phase (from a zero correction it needs no neighbours);
//     likewise the restriction for the coarser levels;
//   * the last pre-sweep's black phase writes the black nodes' residual;
//   * the last sweep of level 1 adds its values to u.
// Coarse levels that fit the shared memory of one SM run there in block 0.
// Measured against 32x8x8-node tiles staged by TMA (17 phases of about 22 us a
// refinement at 128^3): 256^3 with electrodes cold 40 -> 11.1 ms (18
// refinements); in the step loop 128^3 1.53 -> 0.58 ms (4), 48x80x112 0.72 ->
// 0.34 ms, 32^3 0.38 -> 0.20 ms.
#include <cstring>

#include "mgsplit.cuh"

namespace lepic {

namespace {

using mgs::BLACK;
using mgs::MB;
using mgs::MB_FREE;
using mgs::MB_ODD;
using mgs::MB_PLASMA;
using mgs::MB_UPD;
using mgs::RED;
using mgs::Team;
using Lev = mgs::Lev<float>;

constexpr int XM_MAX = mgs::LEVELS;   // multigrid levels
// threads per block: twice as many, at half the registers, on grids whose
// finest level moves through HBM (cold solves with electrodes, 512 and 1024
// threads: 128^3 2.37 and 2.80 ms, 160^3 9.42 and 10.34, 192^3 6.19 and 6.32,
// 208^3 13.10 and 12.79, 224^3 25.8 and 25.0, 256^3 11.63 and 11.17)
constexpr int XM_BLOCK = 512, XM_BLOCK_LARGE = 1024;
constexpr long long XM_LARGE = 4300000;   // elements per colour from which it takes those: between 192^3 and 208^3
constexpr int XV = 4;           // elements per 16-byte load
// elements per colour up to which one cluster solves faster than the grid
// (cold solves by the grid and by a cluster: 32^3, 24,500, 328 and 296 us;
// 40x32x32, 29,400, 306 and 277; 40x32x40, 36,100, 321 and 329; 48x40x32,
// 42,100, 356 and 380; 48x40x48, 61,400, 368 and 384; 56^3, 640 and 789)
constexpr long long XM_SMALL = 35000;

struct XArgs {
  Lev L[XM_MAX + 2];          // levels 1..ng; after them level ls + 1 with its arrays on the grid
  unsigned oc[XM_MAX + 1];    // levels ls+1..ng: byte offset of their arrays on chip
  unsigned ol;                // and of the level descriptors
  int ng, ls;                 // levels 1..ls on the grid, ls+1..ng in block 0's shared memory
  int max_refine, nu_fine_pre, nu_fine_post, nu_pre, nu_post, coarse_sweeps;
  float omega;
  double aw, an, at, ac;      // FP64 finest coefficients (ae = aw, as = an, ab = at)
  double *u;                  // the caller's grid arrays
  const double *b;
  const int *bcnd;
  double *us[2], *bs[2];      // their colour-split copies
  double alpha, eps;
  double *partial;            // [2][gridDim.x]
  int *out_i;      // [0] refinement iterations, [1] status
  double *out_d;   // [0] res/alpha, [1] first res/alpha
  double *host;    // pinned host memory for refinements, status, res/alpha (or null)
  GridBarrier barrier;
};

extern __shared__ __align__(16) unsigned char xm_smem[];

// level l on the grid / on chip: its descriptor in shared memory
template <bool GRID>
__device__ __forceinline__ const Lev &level_of(const XArgs &a, int l) {
  return reinterpret_cast<const Lev *>(xm_smem + a.ol)[(GRID && l == a.ls + 1 ? a.ng + 1 : l) - 1];
}

template <bool GRID>
__device__ __forceinline__ Team team() {
  return GRID ? mgs::grid_team() : mgs::block_team();
}
template <bool GRID, class Sync>
__device__ __forceinline__ void barrier(Sync &grid) {
  if (GRID)
    grid.sync();
  else
    __syncthreads();
}

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// deterministic grid-wide sum of one value per thread, ending at a grid
// barrier.  The block partials alternate between two halves of a.partial
// (parity), so one barrier suffices: a half is rewritten two sums later.
template <class Sync>
__device__ __forceinline__ double grid_sum(const XArgs &a, double v, int parity, Sync &grid, double *sh) {
  double *part = a.partial + (parity & 1) * gridDim.x;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  v = wsum(v);
  if (lane == 0) sh[wp] = v;
  __syncthreads();
  if (wp == 0) {
    v = wsum(lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0);
    if (lane == 0) part[blockIdx.x] = v;
  }
  grid.sync();
  double s = 0.0;
  for (int q = lane; q < (int)gridDim.x; q += 32) s += part[q];   // every warp, in the same order
  return wsum(s);
}

// ------------------------------------------------------------ level 1, FP64
// One colour of the FP64 residual b - A u, as the FP32 right-hand side of the
// V-cycle; START: red also takes the first sweep's red phase from a zero
// correction.  Returns this thread's share of the L1 norm over the plasma
// nodes (bcnd = -1).
template <int COLOUR>
__device__ __forceinline__ double residual_f64(const XArgs &a, const Lev &L, bool start, const Team &w) {
  const int e1 = L.HN * (L.n3 + 2), H = L.H, HN = L.HN, step = 2 * w.n;
  const double aw = a.aw, an = a.an, at = a.at, ac = a.ac;
  const double *S = a.us[COLOUR], *O = a.us[COLOUR ^ 1], *B = a.bs[COLOUR];
  const float om = a.omega;
  double acc = 0.0;
#pragma unroll 1
  for (int e = HN + 2 * w.id; e < e1; e += step) {
    mgs::Pts<double, 2> p;
    mgs::load_pts<double, 2, COLOUR>(p, e, H, HN, S, O, B, L.m);
    const bool odd = (p.m & MB_ODD) != 0;
    mgs::Vec<float, 2> rv, sv;
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const double uw = odd ? p.x.v[v] : (v == 0 ? p.e : p.x.v[0]);
      const double ue = odd ? (v == 1 ? p.e : p.x.v[1]) : p.x.v[v];
      const double r = p.r.v[v] - (aw * uw + an * p.n.v[v] + an * p.s.v[v] + aw * ue + ac * p.c.v[v] +
                                   at * p.t.v[v] + at * p.b.v[v]);
      if (p.m & (MB_PLASMA << (8 * v))) acc += fabs(r);
      const bool upd = (p.m & (MB_UPD << (8 * v))) != 0;
      rv.v[v] = upd ? (float)r : 0.f;
      sv.v[v] = upd && start ? mgs::first_red(L, (float)r, om) : 0.f;
    }
    mgs::stv<float, 2>(L.b[COLOUR] + e, rv);
    if (COLOUR == RED) mgs::stv<float, 2>(L.red[0] + e, sv);
    if (COLOUR == BLACK && !start) mgs::stv<float, 2>(L.black + e, sv);
  }
  return acc;
}

// the caller's grids into the split copies, the node bytes and zero ghosts of
// level 1 (ghost nodes are never prolonged to: their correction stays 0)
__device__ __noinline__ void split_in(const XArgs &a) {
  const Lev &L = level_of<true>(a, 1);
  const long long N1 = L.n1 + 3, R1 = L.n1 + 2, R2 = L.n2 + 2;
  const int last = L.n1 + 2;
  mgs::elements(L, mgs::grid_team(), [&](int e, int ii, int j, int k) {
    // the row's nodes i = 2 ii and 2 ii + 1: one of each colour
    const long long q = 2 * ii + N1 * (j + (long long)L.N2 * k), qb = 2 * ii + R1 * (j + R2 * (long long)k);
    const bool jk = j >= 1 && k >= 1 && j <= L.n2 + 1 && k <= L.n3 + 1;
    const int odd = (j + k + 1) & 1;   // the colour of i odd
    unsigned m = 0;
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int i = 2 * ii + x, c = x ? odd ^ 1 : odd;
      double u = 0.0, b = 0.0;
      unsigned bits = x ? MB_ODD : 0;
      if (i <= last) {
        u = a.u[q + x];
        if (jk && i >= 1 && i <= L.n1 + 1) {
          const int bc = a.bcnd[q + x];
          b = a.b[qb + x];
          bits |= (bc <= 0 ? MB_UPD | MB_FREE : 0) | (bc == -1 ? MB_PLASMA : 0);
        }
      }
      m |= MB(c, bits);
      a.us[c][e] = u;
      a.bs[c][e] = b;
    }
    L.m[e] = (unsigned char)m;
    L.red[0][e] = L.black[e] = 0.f;
    if (L.rf[RED]) L.rf[RED][e] = L.rf[BLACK][e] = 0.f;
  });
}
__device__ __noinline__ void split_out(const XArgs &a) {
  const Lev &L = level_of<true>(a, 1);
  mgs::elements(L, mgs::grid_team(), [&](int e, int ii, int j, int k) {
    const unsigned m = L.m[e];
    const int odd = (j + k + 1) & 1;
    double *u = a.u + 2 * ii + (long long)(L.n1 + 3) * (j + (long long)L.N2 * k);
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int c = x ? odd ^ 1 : odd;
      if (m & MB(c, MB_UPD)) u[x] = a.us[c][e];
    }
  });
}

// ------------------------------------------------------------ FP32 V-cycle
// nu sweeps of a level.  started: the first red phase is done and black is 0
// (not written yet); rf: the last black phase also writes the black residual;
// addu: the last sweep adds its values to u.
template <bool GRID, class Sync>
__device__ __forceinline__ void sweeps(const XArgs &a, const Lev &L, int nu, bool started, bool rf, bool addu,
                                       Sync &grid) {
  using namespace mgs;
  const Team w = team<GRID>();
  const float om = a.omega;
  for (int s = 0; s < nu; ++s) {
    const bool last = s == nu - 1, add = GRID && addu && last;
    if (s % SWEEPS_PER_BEAT == SWEEPS_PER_BEAT - 1) {
      if (!GRID)
        grid.beat();
      else if (grid.dead())
        break;
    }
    if (s > 0 || !started) {
      if (add)
        colour_phase<float, XV, mgs::RED, DO_RELAX | DO_ADDU, !GRID>(L, L.red[0], L.red[0], L.black, om, w, nullptr,
                                                              a.us[mgs::RED]);
      else
        colour_phase<float, XV, mgs::RED, DO_RELAX, !GRID>(L, L.red[0], L.red[0], L.black, om, w);
      barrier<GRID>(grid);
    }
    if (s == 0 && started) {
      if (last && rf)
        colour_phase<float, XV, mgs::BLACK, DO_RELAX | DO_RF | ZERO, !GRID>(L, L.black, L.black, L.red[0], om, w,
                                                                     L.rf[mgs::BLACK]);
      else
        colour_phase<float, XV, mgs::BLACK, DO_RELAX | ZERO, !GRID>(L, L.black, L.black, L.red[0], om, w);
    } else if (last && rf) {
      colour_phase<float, XV, mgs::BLACK, DO_RELAX | DO_RF, !GRID>(L, L.black, L.black, L.red[0], om, w, L.rf[mgs::BLACK]);
    } else if (add) {
      colour_phase<float, XV, mgs::BLACK, DO_RELAX | DO_ADDU, !GRID>(L, L.black, L.black, L.red[0], om, w, nullptr,
                                                              a.us[mgs::BLACK]);
    } else {
      colour_phase<float, XV, mgs::BLACK, DO_RELAX, !GRID>(L, L.black, L.black, L.red[0], om, w);
    }
    barrier<GRID>(grid);
  }
}

// the residual of level l (its black half already written when it has been
// swept) weighted onto level l + 1, whose first red phase is done with it
template <bool GRID, class Sync>
__device__ __forceinline__ void restrict_level(const XArgs &a, int l, bool swept, bool masks, Sync &grid) {
  using namespace mgs;
  const Team w = team<GRID>();
  const Lev &F = level_of<GRID>(a, l), &C = level_of<GRID>(a, l + 1);
  residual_colour<float, XV, mgs::RED, !GRID>(F, F.red[0], F.black, F.rf[mgs::RED], w);
  if (!swept) residual_colour<float, XV, mgs::BLACK, !GRID>(F, F.black, F.red[0], F.rf[mgs::BLACK], w);
  barrier<GRID>(grid);
  // (a level that is not swept on the way down starts from 0)
  restrict_to<float, !GRID>(F, C, F.rf[mgs::RED], F.rf[mgs::BLACK], masks, (l + 1 == a.ng ? a.coarse_sweeps : a.nu_pre) > 0,
                     a.omega, w);
  barrier<GRID>(grid);
}

// the sweeps of level l on the way down (or the coarsest level's)
template <bool GRID, class Sync>
__device__ __forceinline__ void down_sweeps(const XArgs &a, int l, bool started, Sync &grid) {
  const bool coarsest = l == a.ng;
  const int nu = coarsest ? a.coarse_sweeps : (l == 1 ? a.nu_fine_pre : a.nu_pre);
  sweeps<GRID>(a, level_of<GRID>(a, l), nu, started, !coarsest, coarsest && a.ng == 1, grid);
}

// the part of a V-cycle on the levels on chip, by block 0
template <class Sync>
__device__ __forceinline__ void chip_cycle(const XArgs &a, bool first, Sync &grid) {
  using namespace mgs;
  const int top = a.ls + 1, ng = a.ng, t0 = threadIdx.x, bd = blockDim.x;
  const Lev &X = level_of<true>(a, top), &T = level_of<false>(a, top);
  // four elements per thread and turn, every load before the first store
  for (int e = XV * t0; e < T.len; e += XV * bd) {
    const Vec<float, XV> b0 = ldv<float, XV>(X.b[0] + e), b1 = ldv<float, XV>(X.b[1] + e),
                         r0 = ldv<float, XV>(X.red[0] + e);
    const unsigned m = first ? *reinterpret_cast<const unsigned *>(X.m + e) : 0u;
    const Vec<float, XV> zero = {{0.f, 0.f, 0.f, 0.f}};
    stv<float, XV>(T.b[0] + e, b0);
    stv<float, XV>(T.b[1] + e, b1);
    stv<float, XV>(T.red[0] + e, r0);
    stv<float, XV>(T.black + e, zero);
    if (first) {
      *reinterpret_cast<unsigned *>(T.m + e) = m;
      if (T.rf[mgs::RED]) {
        stv<float, XV>(T.rf[mgs::RED] + e, zero);
        stv<float, XV>(T.rf[mgs::BLACK] + e, zero);
      }
    }
  }
  __syncthreads();
  const int mid = ng - top;
  for (int g = 0; g <= 2 * mid; ++g) {
    const int l = g <= mid ? top + g : ng - (g - mid);
    if (g <= mid) {
      down_sweeps<false>(a, l, true, grid);
      if (g < mid) restrict_level<false>(a, l, a.nu_pre > 0, first, grid);
    } else {
      const Lev &F = level_of<false>(a, l), &C = level_of<false>(a, l + 1);
      prolong_to<float, true>(F, C, F.red[0], nullptr, C.red[0], block_team());
      __syncthreads();
      sweeps<false>(a, F, a.nu_post, false, false, false, grid);
    }
  }
  for (int e = XV * t0; e < T.len; e += XV * bd) {
    stv<float, XV>(X.red[0] + e, ldv<float, XV>(T.red[0] + e));
    stv<float, XV>(X.black + e, ldv<float, XV>(T.black + e));
  }
}

// u += e on the non-wall nodes of level 1 (when no sweep of level 1 did it)
__device__ __noinline__ void add_u(const XArgs &a) {
  const Lev &L = level_of<true>(a, 1);
  const Team w = mgs::grid_team();
  for (int e = w.id; e < L.len; e += w.n) {
    const unsigned m = L.m[e];
    if (m & MB(RED, MB_UPD)) a.us[RED][e] += (double)L.red[0][e];
    if (m & MB(BLACK, MB_UPD)) a.us[BLACK][e] += (double)L.black[e];
  }
}

template <class Sync, int BLOCK>
__global__ void __launch_bounds__(BLOCK, 1) k_refine_mixed(const __grid_constant__ XArgs a) {
  Sync grid(a.barrier);
  __shared__ double sh[32];
  const int ng = a.ng, ls = a.ls, down = ls < ng ? ls : ng - 1;   // down: the last grid level restricted from
  {
    // the level descriptors in shared memory (read from the kernel's
    // parameters level by level they cost microseconds of constant-cache
    // misses per phase), those on chip with their arrays there
    const int words = (int)(sizeof(Lev) / 4) * (ng + 1);
    const unsigned *from = reinterpret_cast<const unsigned *>(a.L + 1);
    for (int q = threadIdx.x; q < words; q += blockDim.x) reinterpret_cast<unsigned *>(xm_smem + a.ol)[q] = from[q];
    __syncthreads();
    const int l = ls + 1 + threadIdx.x;
    if (l <= ng) {
      Lev &L = const_cast<Lev &>(level_of<false>(a, l));
      float *p = reinterpret_cast<float *>(xm_smem + a.oc[l]);
      const int n = L.len;
      L.red[0] = p;
      L.black = p + n;
      L.b[0] = p + 2 * n;
      L.b[1] = p + 3 * n;
      if (l < ng) {
        L.rf[0] = p + 4 * n;
        L.rf[1] = p + 5 * n;
      }
      L.m = reinterpret_cast<unsigned char *>(p + (l < ng ? 6 : 4) * n);
    }
    __syncthreads();
  }
  split_in(a);
  grid.sync();
  double res = 0.0, res0 = -1.0;
  int it = 0, status = 0;
  // the residual does the first red phase of level 1, unless there is none or
  // (one level, one sweep) it is the phase that adds to u
  const bool start1 = ng == 1 ? a.coarse_sweeps > 1 : a.nu_fine_pre > 0;
  for (;;) {
    const Lev &L1 = level_of<true>(a, 1);
    double acc = residual_f64<RED>(a, L1, start1, mgs::grid_team());
    acc += residual_f64<BLACK>(a, L1, start1, mgs::grid_team());
    res = grid_sum(a, acc, it, grid, sh) / a.alpha;
    if (res0 < 0.0) res0 = res;
    if (grid.dead() || res < a.eps) break;
    if (it >= a.max_refine) {
      status = LEPIC_ERR_NOT_CONVERGED;
      break;
    }
    if (it > 0 && res > 10.0 * res0) {
      status = LEPIC_ERR_DIVERGED;
      break;
    }
    // FP32 V-cycle on the correction: grid levels down, the coarsest level or
    // the levels on chip, grid levels up
    const bool first = it == 0;
    const int mid = down + 1;
    bool added = false;
    for (int g = 1; g <= 2 * down + 1; ++g) {
      if (g == mid && ls < ng) {
        if (blockIdx.x == 0 && !grid.dead()) chip_cycle(a, first, grid);
        grid.sync();
        continue;
      }
      const int l = g <= mid ? g : 2 * mid - g;
      if (g <= mid) {
        down_sweeps<true>(a, l, l > 1 || start1, grid);
        added = added || (ng == 1 && a.coarse_sweeps > 0);
        if (g < mid) restrict_level<true>(a, l, (l == 1 ? a.nu_fine_pre : a.nu_pre) > 0, first, grid);
      } else {
        const Lev &F = level_of<true>(a, l), &C = level_of<true>(a, l + 1);
        mgs::prolong_to<float>(F, C, F.red[0], nullptr, C.red[0], mgs::grid_team());
        grid.sync();
        const int nu = l == 1 ? a.nu_fine_post : a.nu_post;
        sweeps<true>(a, F, nu, false, false, l == 1, grid);
        added = added || (l == 1 && nu > 0);
      }
    }
    if (!added) {
      add_u(a);
      grid.sync();
    }
    ++it;
  }
  if (!grid.dead()) split_out(a);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.out_i[0] = it;
    a.out_i[1] = status;
    a.out_d[0] = res;
    a.out_d[1] = res0;
    if (a.host) {
      a.host[0] = it;
      a.host[1] = status;
      a.host[2] = res;
    }
  }
  grid.leave(a.out_i + 1, a.host ? a.host + 1 : nullptr);
}

}  // namespace

// the status of the last solve (not converged, diverged) into the device
// error word, for a caller that does not wait for the solve
__global__ void k_solve_status(const int *out_i, int *err) {
  if (out_i[1] != 0) raise_err(err, out_i[1], out_i[0]);
}

// The barrier's give-up by itself: two blocks, of which one waits for the
// other, which leaves without having arrived.
__global__ void k_wait_selftest(GridBarrier barrier, int *out_i) {
  mgs::GridSync grid(barrier);
  __syncthreads();
  if (blockIdx.x == 0) grid.sync();
  grid.leave(out_i + 1, nullptr);
}
constexpr long long ROUND_NS = 900000;   // a round of looks takes 0.95 ms

// A solve without device memory for the split copies (30 bytes per grid node):
// FP64 cycles by the general kernel (12), to the same residual; the cycles
// count as refinements.
static int solve_without_copies(const Dims &d, const double h[3], double *u, const double *b, const int *bcnd,
                                double eps, double omega, int ng, double eps0, int max_refine, int *iters,
                                double *res_out, cudaStream_t s) {
  cudaGetLastError();
  scratch_drop("xm_");
  if (max_refine < 1) return LEPIC_ERR_CUDA;
  int k = 0;
  double ktot = 0.0, res = 0.0;
  int rc = launch_pdesolver(d, h, u, b, bcnd, max_refine, eps, omega, ng, eps0, &k, &ktot, &res, s);
  if (rc == LEPIC_ERR_CUDA) return rc;
  if (rc == LEPIC_OK && !(res < eps)) rc = LEPIC_ERR_NOT_CONVERGED;
  const int hi[2] = {k - 1, rc};
  int *out_i = (int *)scratch("xm_out_i", sizeof(int) * 4);
  double *out_d = (double *)scratch("xm_out_d", sizeof(double) * 2);
  if (!out_i || !out_d) return LEPIC_ERR_CUDA;
  LEPIC_CUDA(cudaMemcpyAsync(out_i, hi, sizeof(hi), cudaMemcpyHostToDevice, s));
  LEPIC_CUDA(cudaMemcpyAsync(out_d, &res, sizeof(double), cudaMemcpyHostToDevice, s));
  if (!iters && !res_out) {
    k_solve_status<<<1, 1, 0, s>>>(out_i, ctx().d_err);
    LEPIC_CUDA(cudaGetLastError());
    return LEPIC_OK;
  }
  if (iters) *iters = hi[0];
  if (res_out) *res_out = res;
  return rc;
}

int launch_pdesolver_mixed(const Dims &d, const double h[3], double *u, const double *b, const int *bcnd,
                           double eps, double omega, int ng, double eps0, int max_refine, int nu_fine_pre,
                           int nu_fine_post, int nu_pre, int nu_post, int coarse_sweeps, int *iters,
                           double *res_out, cudaStream_t s, unsigned rounds) {
  if (ng < 1 || ng > XM_MAX) return LEPIC_ERR_ARG;
  const int n[3] = {d.n1, d.n2, d.n3};
  for (int q = 0; q < 3; ++q)
    if (n[q] % (1 << (ng - 1))) return LEPIC_ERR_ARG;
  Ctx &c = ctx();
  XArgs A;
  memset(&A, 0, sizeof(A));
  A.ng = ng;
  A.max_refine = max_refine;
  A.nu_fine_pre = nu_fine_pre;
  A.nu_fine_post = nu_fine_post;
  A.nu_pre = nu_pre;
  A.nu_post = nu_post;
  A.coarse_sweeps = coarse_sweeps;
  A.omega = (float)omega;
  A.u = u;
  A.b = b;
  A.bcnd = bcnd;
  A.eps = eps;
  A.barrier = grid_barrier(rounds);
  if (!A.barrier.line) return LEPIC_ERR_CUDA;
  if (Lev::elements(n[0], n[1], n[2]) >= 2130000000LL) return LEPIC_ERR_UNSUPPORTED;   // 32-bit element numbers
  // shapes and coefficients per level (Src/mg.h)
  for (int l = 1; l <= ng; ++l) {
    double hl[3];
    for (int q = 0; q < 3; ++q) hl[q] = h[q] * (double)(1 << (l - 1));
    const double aw = eps0 / (hl[0] * hl[0]), an = eps0 / (hl[1] * hl[1]), at = eps0 / (hl[2] * hl[2]);
    const double ac = -(an + an + aw + aw + at + at);
    if (l == 1) {
      A.aw = aw;
      A.an = an;
      A.at = at;
      A.ac = ac;
    }
    Lev &L = A.L[l];
    L.shape(n[0] >> (l - 1), n[1] >> (l - 1), n[2] >> (l - 1));
    L.aw = (float)aw;
    L.an = (float)an;
    L.at = (float)at;
    L.ac = (float)ac;
    L.rac = 1.f / L.ac;
  }
  // the coarse levels that fit on chip (level 1 stays on the grid): per
  // element red, black, b of both, on the levels that restrict the residual
  // of both, one byte
  size_t csm = 0;
  A.ls = ng;
  for (int l = ng; l >= 2; --l) {
    const size_t need = ((size_t)A.L[l].len * (4 * (l < ng ? 6 : 4) + 1) + 15) & ~(size_t)15;
    if (csm + need > mgs::CHIP) break;
    A.oc[l] = (unsigned)csm;
    csm += need;
    A.ls = l - 1;
  }
  A.ol = (unsigned)csm;
  csm += sizeof(Lev) * (ng + 1);
  if (A.ls < ng) A.L[ng + 1] = A.L[A.ls + 1];
  char nm[32];
  for (int l = 1; l <= A.ls + 1 && l <= ng; ++l) {
    Lev &L = A.L[l <= A.ls ? l : ng + 1];
    const size_t len = (size_t)L.len;
    const bool restricts = l <= A.ls && l < ng;
    const int halves = restricts ? 6 : 4;
    snprintf(nm, sizeof nm, "xm_%d", l);
    float *p = (float *)scratch(nm, (sizeof(float) * halves + 1) * len);
    if (!p)
      return solve_without_copies(d, h, u, b, bcnd, eps, omega, ng, eps0, max_refine, iters, res_out, s);
    L.red[0] = p;
    L.black = p + len;
    L.b[0] = p + 2 * len;
    L.b[1] = p + 3 * len;
    if (restricts) {
      L.rf[0] = p + 4 * len;
      L.rf[1] = p + 5 * len;
    }
    L.m = reinterpret_cast<unsigned char *>(p + halves * len);
  }
  {
    const size_t len = (size_t)A.L[1].len;
    double *p = (double *)scratch("xm_f64", sizeof(double) * 4 * len);
    if (!p)
      return solve_without_copies(d, h, u, b, bcnd, eps, omega, ng, eps0, max_refine, iters, res_out, s);
    for (int q = 0; q < 2; ++q) {
      A.us[q] = p + q * len;
      A.bs[q] = p + (2 + q) * len;
    }
  }
  A.alpha = residual_scale(n, A.ac);
  const int blocks = c.sms;
  A.partial = (double *)scratch("xm_partial", sizeof(double) * 2 * blocks);
  A.out_i = (int *)scratch("xm_out_i", sizeof(int) * 4);
  A.out_d = (double *)scratch("xm_out_d", sizeof(double) * 2);
  if (!A.partial || !A.out_i || !A.out_d) return LEPIC_ERR_CUDA;
  const bool wait = iters || res_out;
  A.host = wait ? result_block() : nullptr;
  void *args[] = {&A};
  int tm = timer_start("pdesolver_mixed", s);
  const bool large = A.L[1].len >= XM_LARGE;
  LEPIC_CUDA(mgs::launch_solve(large ? (const void *)k_refine_mixed<mgs::GridSync, XM_BLOCK_LARGE>
                                     : (const void *)k_refine_mixed<mgs::GridSync, XM_BLOCK>,
                               (const void *)k_refine_mixed<mgs::ClusterSync, XM_BLOCK>, args, A.L[1].len, XM_SMALL,
                               large ? XM_BLOCK_LARGE : XM_BLOCK, csm, blocks, s));
  timer_stop(tm, s);
  if (!wait) {
    // no wait: the solve's status goes to the device error word
    k_solve_status<<<1, 1, 0, s>>>(A.out_i, ctx().d_err);
    LEPIC_CUDA(cudaGetLastError());
    return LEPIC_OK;
  }
  if (A.host) {
    LEPIC_CUDA(cudaStreamSynchronize(s));
    if (iters) *iters = (int)A.host[0];
    if (res_out) *res_out = A.host[2];
    return (int)A.host[1];
  }
  int hi[4];
  double hd[2];
  LEPIC_CUDA(cudaMemcpyAsync(hi, A.out_i, sizeof(hi), cudaMemcpyDeviceToHost, s));
  LEPIC_CUDA(cudaMemcpyAsync(hd, A.out_d, sizeof(hd), cudaMemcpyDeviceToHost, s));
  LEPIC_CUDA(cudaStreamSynchronize(s));
  if (iters) *iters = hi[0];
  if (res_out) *res_out = hd[0];
  return hi[1];
}

int pdesolver_mixed_stats(int *iters, double *res, cudaStream_t s) {
  if (!iters || !res) return LEPIC_ERR_ARG;
  const int *oi = (const int *)scratch("xm_out_i", sizeof(int) * 4);
  const double *od = (const double *)scratch("xm_out_d", sizeof(double) * 2);
  if (!oi || !od) return LEPIC_ERR_CUDA;
  LEPIC_CUDA(cudaMemcpyAsync(iters, oi, sizeof(int), cudaMemcpyDeviceToHost, s));
  LEPIC_CUDA(cudaMemcpyAsync(res, od, sizeof(double), cudaMemcpyDeviceToHost, s));
  return LEPIC_OK;
}

}  // namespace lepic

extern "C" int lepic_dev_wait_selftest(long long limit_ns, void *stream) {
  if (limit_ns <= 0 || limit_ns > 2000000000LL) return LEPIC_ERR_ARG;
  const cudaStream_t s = (cudaStream_t)stream;
  const lepic::GridBarrier barrier = lepic::grid_barrier((unsigned)((limit_ns + lepic::ROUND_NS - 1) / lepic::ROUND_NS));
  int *out_i = (int *)lepic::scratch("wait_out_i", sizeof(int) * 2);
  if (!barrier.line || !out_i) return LEPIC_ERR_CUDA;
  LEPIC_CUDA(cudaMemsetAsync(out_i, 0, sizeof(int) * 2, s));
  lepic::k_wait_selftest<<<2, 32, 0, s>>>(barrier, out_i);
  lepic::k_solve_status<<<1, 1, 0, s>>>(out_i, lepic::ctx().d_err);
  LEPIC_CUDA(cudaGetLastError());
  return LEPIC_OK;
}

extern "C" int lepic_dev_pdesolver_mixed_stats(int *iters, double *res, void *stream) {
  return lepic::pdesolver_mixed_stats(iters, res, (cudaStream_t)stream);
}

extern "C" int lepic_dev_pdesolver_mixed(const lepic_grid_t *g, double *u, const double *b, double eps,
                                         double omega, int ng, const lepic_phys_t *P, int max_refine,
                                         int nu_fine_pre, int nu_fine_post, int nu_pre, int nu_post,
                                         int coarse_sweeps, int *iters, double *res, void *stream) {
  if (!g || !P) return LEPIC_ERR_ARG;
  if (P->flag_pbc || P->flag_nmn) return LEPIC_ERR_UNSUPPORTED;
  if (nu_fine_pre < 0 || nu_fine_post < 0 || nu_pre < 0 || nu_post < 0 || coarse_sweeps < 0 || max_refine < 0)
    return LEPIC_ERR_ARG;
  return lepic::launch_pdesolver_mixed(lepic::Dims(g->n), g->h, u, b, g->bcnd, eps, omega, ng, P->eps0,
                                       max_refine, nu_fine_pre, nu_fine_post, nu_pre, nu_post, coarse_sweeps,
                                       iters, res, (cudaStream_t)stream);
}
