// Colour-split multigrid levels: the red nodes ((i+j+k) odd) and the black
// ones of a level live in two arrays of their own, so that a red or black
// relaxation reads and writes whole cache lines of what it needs (in the
// natural order each colour is every other value of a line, and both colours'
// phases move all of them).
//
// Node (i, j, k), 0 <= i <= n+2 etc., of colour c (0 red, 1 black) is element
//   e = (i >> 1) + H (j + N2 k)
// of that colour's arrays; all nodes of one colour in a row (j, k) have i of
// one parity s, and in terms of e the six neighbours, all of the other
// colour, are
//   west e - 1 + s, east e + s, south/north e -+ H, below/above e -+ H N2.
// A byte per element holds what the loops ask about its red and its black
// node (MB_*), the parity s among it, so a relaxation needs no coordinates at all: it runs over the
// elements of the planes k = 1..n3+1 (whose neighbours are all inside the
// arrays), every load issued before the byte is looked at, V consecutive
// elements per thread with vector loads.
//
// The red values have two buffers: a red phase reads one and writes the
// other, so that it can compute the residual of the finished sweep and the
// next sweep's red values in one pass; when the residual ends the smoothing
// the written buffer is simply not taken.
#pragma once

#include <type_traits>

#include "lepic_internal.cuh"

namespace lepic {
namespace mgs {

// the red node's four bits, the black node's in the upper half (MB(COLOUR, bit))
enum : unsigned {
  MB_UPD = 1,      // inside 1..n+1 and not a wall: relaxed
  MB_PLASMA = 2,   // inside 1..n+1 and bcnd = -1: counted in the residual norm
  MB_ODD = 4,      // s: parity of i
  MB_FREE = 8      // not a wall (ghost nodes included): prolonged to
};
__host__ __device__ constexpr unsigned MB(int colour, unsigned bit) { return bit << (4 * colour); }

// x / d for 0 <= x < 2^31 by a multiplication (d > 0): with m = ceil(2^p / d),
// p = 31 + ceil(log2 d), x m exceeds x 2^p / d by x (m d - 2^p) / d, less than
// 2^p / d
struct Div {
  unsigned long long m;
  int p, d;
  void set(int dd) {
    d = dd;
    int l = 0;
    while ((1LL << l) < dd) ++l;
    p = 31 + l;
    m = ((1ULL << p) + (unsigned)dd - 1) / (unsigned)dd;
  }
  __host__ __device__ int div(int x) const { return (int)(((unsigned long long)(unsigned)x * m) >> p); }
};

template <class T>
struct Lev {
  static constexpr int VW = 16 / sizeof(T);   // elements of a 16-byte load
  int n1, n2, n3;
  int H, N2, N3;            // row pitch in elements (a multiple of VW), rows per plane, planes
  int HN, len;              // H N2, elements per colour
  Div dH, dN2;
  T aw, an, at, ac;         // ae = aw, as = an, ab = at (Src/mg.h)
  T rac;                    // 1 / ac, correctly rounded
  T *red[2], *black;
  T *b[2];
  T *rf[2];                 // residual (levels that restrict)
  unsigned char *m;
  __host__ __device__ int node(int i, int j, int k) const { return (i >> 1) + H * (j + N2 * k); }
  __host__ void shape(int a, int bb, int c) {
    n1 = a;
    n2 = bb;
    n3 = c;
    H = row(a);
    N2 = n2 + 3;
    N3 = n3 + 3;
    HN = H * N2;
    len = HN * N3;
    dH.set(H);
    dN2.set(N2);
  }
  static int row(int a) { return (((a + 2) >> 1) + VW) & ~(VW - 1); }
  // elements of one colour's array of an a x bb x c level
  static long long elements(int a, int bb, int c) { return (long long)row(a) * (bb + 3) * (c + 3); }
};

// The barrier between two phases of the levels on the grid: of all blocks of a
// cooperative launch, or, for small grids, of one cluster of CLUSTER blocks
// (0.3 us by itself, the cooperative groups' barrier of the grid 1.2).
// The grid's barrier is a word of its own per launch (grid_barrier()): each
// block adds 1, block 0 what takes the word to its top bit flipped and the
// count back to 0, and the blocks watch that bit.  Unlike the cooperative
// groups' barrier nothing waits for the addition's result, and the read that
// sees the bit is the acquire (with relaxed reads and a fence behind them the
// mixed solve of 48x40x56 took 468 us instead of 421).  Solves at 128^3: FP64
// 4.32 -> 4.07 ms, mixed 613 -> 582 us; at 256^3 mixed 12.4 -> 11.2 ms.
//
// The blocks are co-resident (cooperative launch) and a phase takes
// milliseconds at most, but for block 0's on the levels on chip, which may
// smooth the coarsest one a million times: it counts its sweeps there in a
// second word (beat).  A wait therefore lasts as long as anything moves,
// arrivals or beats; where nothing has for BARRIER_ROUNDS rounds of looks (about
// a second; counted in looks, since a process that shares the device may stop
// this one for any time), the block gives up: it neither arrives nor
// waits at any barrier any more, ends its cycle on what the level arrays hold
// and leaves phi alone; the others no longer get past a barrier and do the
// same.  The last block to leave then clears the word, whose count the missing
// arrivals have left anywhere, for the launch that has it next, and makes
// LEPIC_ERR_TIMEOUT the solve's status.
constexpr unsigned BARRIER_LOOKS = 1u << 12;
constexpr int SWEEPS_PER_BEAT = 256;
struct GridSync {
  enum { WORD = 0, BEAT = 1, LEFT = 2, SPARE = 4 };   // of the launch's line
  struct State {
    unsigned *line, phase;
    bool dead;
    unsigned rounds, moved, idle;   // the limit; what had moved after the last round, rounds without any since
  };
  static __device__ __forceinline__ State &state() {
    __shared__ State s;
    return s;
  }
  static __device__ __forceinline__ unsigned look(const unsigned *w) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(w) : "memory");
    return v;
  }
  // (the bit cannot flip before this block has arrived once)
  __device__ explicit GridSync(const GridBarrier &g) {
    if (threadIdx.x == 0) state() = {g.line, look(g.line + WORD) & 0x80000000u, false, g.rounds, 0, 0};
  }
  // looks at `word` until its top bit differs from phase's, BARRIER_LOOKS
  // times at most: what is left of them (a loop of its own instructions: with
  // the compiler's, the rest of the wait costs every barrier of a solve 1 %)
  static __device__ __forceinline__ unsigned watch(const unsigned *word, unsigned phase) {
    unsigned left;
    asm volatile(
        "{\n .reg .pred p;\n .reg .b32 v, n;\n mov.u32 n, %3;\n"
        "LOOK%=:\n ld.acquire.gpu.global.u32 v, [%1];\n xor.b32 v, v, %2;\n setp.lt.s32 p, v, 0;\n"
        " @p bra SEEN%=;\n sub.u32 n, n, 1;\n setp.ne.u32 p, n, 0;\n @p bra LOOK%=;\n"
        "SEEN%=:\n mov.u32 %0, n;\n}\n"
        : "=r"(left)
        : "l"(word), "r"(phase), "n"(BARRIER_LOOKS)
        : "memory");
    return left;
  }
  // after a round of looks: nothing has moved for too long
  static __device__ __forceinline__ bool give_up(State &s) {
    const unsigned moved = look(s.line + WORD) + look(s.line + BEAT);
    s.idle = moved != s.moved ? 0 : s.idle + 1;
    s.moved = moved;
    if (s.idle < s.rounds) return false;
    s.dead = true;
    s.line += SPARE;   // its arrivals go there from now on (a test before each would delay the living ones')
    return true;
  }
  __device__ __forceinline__ void sync() {
    __syncthreads();
    if (threadIdx.x == 0) {
      State &s = state();
      const unsigned add = blockIdx.x == 0 ? 0x80000000u - (gridDim.x - 1) : 1u;
      asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(s.line + WORD), "r"(add) : "memory");
      if (!s.dead)
        while (!watch(s.line + WORD, s.phase) && !give_up(s)) {
        }
      s.phase ^= 0x80000000u;
    }
    __syncthreads();
  }
  // this block has given up (the same for all of its threads between barriers)
  __device__ __forceinline__ bool dead() const { return state().dead; }
  // the end of the kernel: every block calls it once.  status, host: where
  // block 0 has put the solve's status (host may be null).
  __device__ __forceinline__ void leave(int *status, double *host) {
    __syncthreads();
    if (threadIdx.x != 0) return;
    const State &s = state();
    const unsigned mine = s.dead ? 0x10001u : 1u;   // the blocks that left, and of them those that had given up
    __threadfence();
    unsigned *const line = s.dead ? s.line - SPARE : s.line;
    const unsigned left = atomicAdd(line + LEFT, mine) + mine;
    if ((left & 0xffffu) != gridDim.x) return;
    __threadfence();
    line[LEFT] = 0;
    if (left >> 16) {
      line[WORD] = 0;
      *status = LEPIC_ERR_TIMEOUT;
      if (host) *host = LEPIC_ERR_TIMEOUT;
    }
  }
  // block 0 on the levels on chip: the others' wait goes on
  __device__ __forceinline__ void beat() {
    if (threadIdx.x == 0) asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(state().line + BEAT));
  }
};
struct ClusterSync {
  __device__ explicit ClusterSync(const GridBarrier &) {}
  __device__ __forceinline__ bool dead() const { return false; }
  __device__ __forceinline__ void leave(int *, double *) {}
  __device__ __forceinline__ void beat() {}
  __device__ __forceinline__ void sync() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
  }
};
constexpr int CLUSTER = 16;

// threads that share a loop
struct Team {
  int id, n;
};
__device__ __forceinline__ Team grid_team() {
  return {(int)(blockIdx.x * blockDim.x + threadIdx.x), (int)(gridDim.x * blockDim.x)};
}
__device__ __forceinline__ Team block_team() { return {(int)threadIdx.x, (int)blockDim.x}; }

template <class T, int V>
struct alignas(sizeof(T) * V) Vec {
  T v[V];
};
template <class T, int V>
__device__ __forceinline__ Vec<T, V> ldv(const T *p) {
  return *reinterpret_cast<const Vec<T, V> *>(p);
}
template <class T, int V>
__device__ __forceinline__ void stv(T *p, const Vec<T, V> &x) {
  *reinterpret_cast<Vec<T, V> *>(p) = x;
}

// A pointer into the block's dynamic shared memory, as one that the compiler
// knows to point there (32-bit addresses and shared loads instead of generic
// ones; the levels' descriptors hold generic pointers for both kinds).  The
// levels on chip keep half the issue slots of their SM and three quarters of
// its shared-memory pipe busy (48x80x112, FP32): a solve of 32^3 takes 196 us
// instead of 202 (mixed), of 16x16x24 252 instead of 258 (FP64).
template <bool CHIP, class P>
__device__ __forceinline__ P *place(P *p) {
  if constexpr (CHIP) {
    extern __shared__ __align__(16) unsigned char mgs_smem[];
    return reinterpret_cast<P *>(mgs_smem + ((unsigned)__cvta_generic_to_shared(p) -
                                             (unsigned)__cvta_generic_to_shared(mgs_smem)));
  } else {
    return p;
  }
}

enum { RED = 0, BLACK = 1 };
// what a colour's phase does: relax its nodes (ZERO: from 0, not read), add up
// the residual norm, write the residual out, add the relaxed values to an
// FP64 solution
enum { DO_RELAX = 1, DO_RES = 2, DO_RF = 4, DO_ADDU = 8, ZERO = 16 };

// What a phase reads for V consecutive elements: the elements themselves, the
// six neighbours and the byte (the x neighbours: the other colour's elements
// at the same place and one more, before or after them).
template <class T, int V>
struct Pts {
  Vec<T, V> x, n, s, t, b, c, r;
  T e;
  unsigned m;   // the V bytes, shifted to this colour's bits
};
template <class T, int V, int COLOUR, bool SELF = true>
__device__ __forceinline__ void load_pts(Pts<T, V> &p, int e, int H, int HN, const T *S, const T *O, const T *B,
                                         const unsigned char *M) {
  static_assert(V == 2 || V == 4, "");
  if (V == 2)
    p.m = *reinterpret_cast<const unsigned short *>(M + e) >> (4 * COLOUR);
  else
    p.m = *reinterpret_cast<const unsigned *>(M + e) >> (4 * COLOUR);
  const T *o = O + e;
  p.x = ldv<T, V>(o);
  p.n = ldv<T, V>(o + H);
  p.s = ldv<T, V>(o - H);
  p.t = ldv<T, V>(o + HN);
  p.b = ldv<T, V>(o - HN);
  if (SELF) p.c = ldv<T, V>(S + e);
  p.r = ldv<T, V>(B + e);
  const T lo = o[-1], hi = o[V];
  p.e = (p.m & MB_ODD) ? hi : lo;
}

// One colour of a red-black sweep (Src/sors.f90:87-106, 249-267) over the
// team's elements: reads S (the colour's values) and O (the other colour's),
// writes D (S itself for black).  DO_RES adds up |residual| over the plasma
// nodes, with the relaxed value when COLOUR is BLACK (its sweep ends with
// it) and with the value read when it is RED (the sweep before this one ends
// with it).  The expressions keep the Fortran order.  (A thread's next
// elements loaded before the current ones are worked on was slower: twice the
// registers, spilled at 512 threads.)
template <class T, int V, int COLOUR, int WHAT, bool CHIP = false>
__device__ __forceinline__ T colour_phase(const Lev<T> &L, const T *S_, T *D_, const T *O_, T omega, const Team &w,
                                          T *R_ = nullptr, double *U = nullptr) {
  const int e1 = L.HN * (L.n3 + 2), H = L.H, HN = L.HN, step = V * w.n;
  const T aw = L.aw, an = L.an, at = L.at, ac = L.ac, rac = L.rac;
  const T *S = place<CHIP>(S_), *O = place<CHIP>(O_), *B = place<CHIP>(L.b[COLOUR]);
  T *D = WHAT & DO_RELAX ? place<CHIP>(D_) : nullptr, *R = WHAT & DO_RF ? place<CHIP>(R_) : nullptr;
  const unsigned char *M = place<CHIP>(L.m);
  T acc = T(0);
#pragma unroll 1
  for (int e = HN + V * w.id; e < e1; e += step) {
    Pts<T, V> p;
    load_pts<T, V, COLOUR, !(WHAT & ZERO)>(p, e, H, HN, S, O, B, M);
    const bool odd = (p.m & MB_ODD) != 0;
    Vec<T, V> dv, rv;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const T uw = odd ? p.x.v[v] : (v == 0 ? p.e : p.x.v[v > 0 ? v - 1 : 0]);
      const T ue = odd ? (v == V - 1 ? p.e : p.x.v[v < V - 1 ? v + 1 : V - 1]) : p.x.v[v];
      const T u0 = (WHAT & ZERO) ? T(0) : p.c.v[v];
      const bool upd = (p.m & (MB_UPD << (8 * v))) != 0;
      T u = u0;
      if (WHAT & DO_RELAX) {
        const T tt = p.r.v[v] - aw * uw - an * p.n.v[v] - an * p.s.v[v] - aw * ue - at * p.t.v[v] - at * p.b.v[v];
        if constexpr (std::is_same_v<T, double>)
          u = (1.0 - omega) * u0 + div_by(omega * tt, ac, rac);
        else
          u = (WHAT & ZERO) ? omega * tt * rac : (1.f - omega) * u0 + omega * tt * rac;
        u = upd ? u : u0;
        dv.v[v] = u;
      }
      if (WHAT & (DO_RES | DO_RF)) {
        const T ur = COLOUR == BLACK ? u : u0;
        const T rij = p.r.v[v] - (aw * uw + an * p.n.v[v] + an * p.s.v[v] + aw * ue + ac * ur + at * p.t.v[v] +
                                  at * p.b.v[v]);
        if ((WHAT & DO_RES) && (p.m & (MB_PLASMA << (8 * v)))) acc += rij < T(0) ? -rij : rij;
        if (WHAT & DO_RF) rv.v[v] = upd ? rij : T(0);
      }
    }
    if (WHAT & DO_RELAX) stv<T, V>(D + e, dv);
    if (WHAT & DO_RF) stv<T, V>(R + e, rv);
    if (WHAT & DO_ADDU) {
#pragma unroll
      for (int v = 0; v < V; v += 2) {
        Vec<double, 2> uu = ldv<double, 2>(U + e + v);
        if (p.m & (MB_UPD << (8 * v))) uu.v[0] += (double)dv.v[v];
        if (p.m & (MB_UPD << (8 * v + 8))) uu.v[1] += (double)dv.v[v + 1];
        stv<double, 2>(U + e + v, uu);
      }
    }
  }
  return acc;
}

// residual of every node of a colour (Src/mg.f90:808-847, its order of
// terms), 0 on walls
template <class T, int V, int COLOUR, bool CHIP = false>
__device__ __forceinline__ void residual_colour(const Lev<T> &L, const T *S_, const T *O_, T *R_, const Team &w) {
  const int e1 = L.HN * (L.n3 + 2), H = L.H, HN = L.HN, step = V * w.n;
  const T aw = L.aw, an = L.an, at = L.at, ac = L.ac;
  const T *S = place<CHIP>(S_), *O = place<CHIP>(O_), *B = place<CHIP>(L.b[COLOUR]);
  T *R = place<CHIP>(R_);
  const unsigned char *M = place<CHIP>(L.m);
#pragma unroll 1
  for (int e = HN + V * w.id; e < e1; e += step) {
    Pts<T, V> p;
    load_pts<T, V, COLOUR>(p, e, H, HN, S, O, B, M);
    const bool odd = (p.m & MB_ODD) != 0;
    Vec<T, V> rv;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const T uw = odd ? p.x.v[v] : (v == 0 ? p.e : p.x.v[v > 0 ? v - 1 : 0]);
      const T ue = odd ? (v == V - 1 ? p.e : p.x.v[v < V - 1 ? v + 1 : V - 1]) : p.x.v[v];
      const T r = p.r.v[v] - (aw * uw + aw * ue + an * p.n.v[v] + an * p.s.v[v] + ac * p.c.v[v] + at * p.t.v[v] +
                              at * p.b.v[v]);
      rv.v[v] = (p.m & (MB_UPD << (8 * v))) ? r : T(0);
    }
    stv<T, V>(R + e, rv);
  }
}

// fine node of a coarse one per axis (Src/mg.f90:429-436)
__device__ __forceinline__ int fine_of(int ic, int ncell_fine) {
  return ic == ncell_fine / 2 + 2 ? ncell_fine + 2 : (ic == 0 ? 0 : 2 * ic - 1);
}

// a red node's value after the first red phase of a sweep that starts from 0
// (the relaxation's own arithmetic with every neighbour 0)
template <class T>
__device__ __forceinline__ T first_red(const Lev<T> &L, T b, T omega) {
  if constexpr (std::is_same_v<T, double>)
    return (1.0 - omega) * 0.0 + div_by(omega * b, L.ac, L.rac);
  else
    return omega * b * L.rac;
}

// The elements of a level, its whole arrays, over the team's threads:
// body(e, ii, j, k) for e = ii + H (j + N2 k), of both colours.  (A row per
// warp needs no division but leaves a third of the lanes idle: a row of 129
// nodes has 66 elements.)
template <class T, class F>
__device__ __forceinline__ void elements(const Lev<T> &L, const Team &w, F &&body) {
  for (int e = w.id; e < L.len; e += w.n) {
    const int r = L.dH.div(e), k = L.dN2.div(r), j = r - k * L.N2;
    body(e, e - r * L.H, j, k);
  }
}

// 27-point full weighting (Src/mg.f90:696-702) of F's residual (R, K: its red
// and black halves, an even / odd number of unit steps from a coarse node's
// twin) onto C's right-hand side, C's correction cleared; masks: C's node bytes as well
// (they stay the same for a whole solve).  start: the red values as the first sweep's red
// phase leaves them (every neighbour is 0 there), so that the sweep begins
// with its black phase.
template <class T, bool CHIP = false>
__device__ __forceinline__ void restrict_to(const Lev<T> &F, const Lev<T> &C, const T *R_, const T *K_, bool masks,
                                            bool start, T omega, const Team &w) {
  const int H = F.H, HN = F.HN;
  const T *R = place<CHIP>(R_), *K = place<CHIP>(K_);
  T *cb[2] = {place<CHIP>(C.b[RED]), place<CHIP>(C.b[BLACK])}, *cr = place<CHIP>(C.red[0]), *ck = place<CHIP>(C.black);
  unsigned char *cm = place<CHIP>(C.m);
  elements(C, w, [&](int e, int ii, int j, int k) {
    unsigned m = 0;
    if (masks) {
      for (int c = 0; c < 2; ++c) {
        const int s = (c + 1 + j + k) & 1, i = 2 * ii + s;
        unsigned b = s ? MB_ODD : 0;
        if (i <= C.n1 + 2) {
          const int fi = fine_of(i, F.n1), fj = fine_of(j, F.n2), fk = fine_of(k, F.n3);
          const unsigned fm = F.m[F.node(fi, fj, fk)] >> (4 * ((fi + fj + fk + 1) & 1));
          b |= fm & MB_FREE;
          if (i >= 1 && j >= 1 && k >= 1 && i <= C.n1 + 1 && j <= C.n2 + 1 && k <= C.n3 + 1)
            b |= fm & (MB_UPD | MB_PLASMA);
        }
        m |= MB(c, b);
      }
      cm[e] = (unsigned char)m;
      if (C.rf[RED]) C.rf[RED][e] = T(0);
      if (C.rf[BLACK]) C.rf[BLACK][e] = T(0);
    } else {
      m = cm[e];
    }
    ck[e] = T(0);
    // the planes no red phase writes, in both buffers (a ghost that is not a
    // wall is prolonged to)
    if (C.red[1] && (masks || k == 0 || k == C.n3 + 2)) C.red[1][e] = T(0);
    const int q0 = H * ((2 * j - 1) + F.N2 * (2 * k - 1));
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int i = 2 * ii + ((c + 1 + j + k) & 1);
      T re = T(0);
      if (m & MB(c, MB_UPD)) {
        const int q = (i - 1) + q0;
        re = (T(8) * R[q] + T(4) * (K[q + 1] + K[q] + K[q + H] + K[q - H] + K[q + HN] + K[q - HN]) +
              T(2) * (R[q + 1 + H] + R[q + H] + R[q + 1 - H] + R[q - H] + R[q + 1 + HN] + R[q + HN] +
                      R[q + H + HN] + R[q - H + HN] + R[q + 1 - HN] + R[q - HN] + R[q + H - HN] + R[q - H - HN]) +
              K[q + 1 + H + HN] + K[q + H + HN] + K[q + 1 - H + HN] + K[q - H + HN] + K[q + 1 + H - HN] +
              K[q + H - HN] + K[q + 1 - H - HN] + K[q - H - HN]) /
             T(64);
      }
      cb[c][e] = re;
      if (c == RED) cr[e] = start && (m & MB(c, MB_UPD)) ? first_red(C, re, omega) : T(0);
    }
  });
}

// Trilinear prolongation (Src/mg.f90:849-939): C's correction added to F's
// nodes 0..n+1 that are not walls; rF, rC: the current red buffers.  A fine
// node sits on a coarse one or between two, four or eight (its upper corner
// first, in the reference's order of terms); which, is the same for a whole
// row of one colour.  rO: the other red buffer (or null), whose plane k = 0 no
// red phase writes.  A thread takes two elements of a row, ii and ii + 1 (ii
// even): their nodes 2 ii .. 2 ii + 3 lie between the coarse columns ii .. ii + 2.
// Every load is issued before the bytes are looked at.
template <class T, bool CHIP = false>
__device__ __forceinline__ void prolong_to(const Lev<T> &F, const Lev<T> &C, T *rF_, T *rO, const T *rC_,
                                           const Team &w) {
  const T *bC = place<CHIP>(C.black), *rC = place<CHIP>(rC_);
  T *rF = place<CHIP>(rF_), *bF = place<CHIP>(F.black);
  const unsigned char *M = place<CHIP>(F.m);
  const int H = C.H, HN = C.HN, last = F.n1 + 1;
#pragma unroll 1
  for (int e = 2 * w.id; e < F.len; e += 2 * w.n) {
    const int r = F.dH.div(e), k = F.dN2.div(r), j = r - k * F.N2, ii = e - r * F.H;
    if (2 * ii > last || j > F.n2 + 1 || k > F.n3 + 1) continue;
    const unsigned m = *reinterpret_cast<const unsigned short *>(M + e);
    Vec<T, 2> vr = ldv<T, 2>(rF + e), vb = ldv<T, 2>(bF + e);
    // the corner (ii + 1, cj, ck) of the first element's even node; the node
    // one step from another is of the other colour
    const int cj = (j >> 1) + 1, ck = (k >> 1) + 1;
    const bool y = !(j & 1), z = !(k & 1);              // between coarse nodes along the axis
    const int u = (ii >> 1) + H * (cj + C.N2 * ck);
    const bool odd = (ii + 1 + cj + ck) & 1;
    const T *P = odd ? rC : bC, *Q = odd ? bC : rC;     // the corner's colour and the other
    // columns ii, ii + 1 and ii + 2 of the up to four coarse rows: element
    // ii / 2 of Q, ii / 2 of P, ii / 2 + 1 of Q (rows one step away: P and Q
    // change places)
    T a0[3], a1[3], a2[3], a3[3];
    const bool more = 2 * ii + 2 <= last;               // the second element has nodes to prolong to
    auto row = [&](T (&a)[3], const T *p, const T *q, int at) {
      a[0] = q[at];
      a[1] = p[at];
      a[2] = more ? q[at + 1] : T(0);
    };
    row(a0, P, Q, u);
    if (z) row(a1, Q, P, u - HN);
    if (y) row(a2, Q, P, u - H);
    if (y && z) row(a3, P, Q, u - H - HN);
    const int s = (1 + j + k) & 1;                      // red's parity of i; black's is the other
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      // corner column v + 1, the lower column v
      T on, be;                                         // for the colour with i odd / even
      if (y && z) {
        on = (a0[v + 1] + a1[v + 1] + a3[v + 1] + a2[v + 1]) / T(4);
        be = (a0[v + 1] + a1[v + 1] + a1[v] + a0[v] + a2[v + 1] + a3[v + 1] + a3[v] + a2[v]) / T(8);
      } else if (z) {
        on = (a0[v + 1] + a1[v + 1]) / T(2);
        be = (a0[v + 1] + a1[v + 1] + a1[v] + a0[v]) / T(4);
      } else if (y) {
        on = (a0[v + 1] + a2[v + 1]) / T(2);
        be = (a0[v + 1] + a2[v + 1] + a2[v] + a0[v]) / T(4);
      } else {
        on = a0[v + 1];
        be = (a0[v + 1] + a0[v]) / T(2);
      }
      const int i = 2 * (ii + v);
      const bool in0 = i <= last, in1 = i + 1 <= last;  // i even, i odd
      const unsigned mv = m >> (8 * v);
      if ((mv & MB(RED, MB_FREE)) && (s ? in1 : in0)) vr.v[v] = vr.v[v] + (s ? on : be);
      if ((mv & MB(BLACK, MB_FREE)) && (s ? in0 : in1)) vb.v[v] = vb.v[v] + (s ? be : on);
    }
    stv<T, 2>(rF + e, vr);
    stv<T, 2>(bF + e, vb);
    if (rO && k == 0) stv<T, 2>(rO + e, vr);
  }
}

// Launch of a solve: `one` (its ClusterSync instance) as one cluster when the
// finest level has at most `small` elements per colour and such a cluster
// fits the device, else `all` (GridSync) cooperatively on every SM.  A
// kernel's limit on dynamic shared memory is the same at every launch, the most
// one takes: with each launch's own, two threads that solve on different grids
// lower each other's between setting it and the launch.
constexpr size_t CHIP = 227000;   // for the levels on chip: 16^3 and below
constexpr int LEVELS = 13;        // multigrid levels at most
constexpr size_t SMEM_MOST = CHIP + sizeof(Lev<double>) * (LEVELS + 1);
static_assert(SMEM_MOST + 2048 <= 232448, "beside the kernels' static shared memory");
inline cudaError_t launch_solve(const void *all, const void *one, void **args, long long elements, long long small,
                                int threads, size_t smem, int sms, cudaStream_t s) {
  cudaError_t e = cudaSuccess;
  if (elements <= small) {
    e = cudaFuncSetAttribute(one, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(one, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MOST);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CLUSTER;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(CLUSTER);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = at;
    c.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, one, &c) == cudaSuccess && n >= 1) return cudaLaunchKernelExC(&c, one, args);
    cudaGetLastError();
  }
  e = cudaFuncSetAttribute(all, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MOST);
  if (e != cudaSuccess) return e;
  return cudaLaunchCooperativeKernel(all, dim3(sms), dim3(threads), args, smem, s);
}

}  // namespace mgs
}  // namespace lepic
