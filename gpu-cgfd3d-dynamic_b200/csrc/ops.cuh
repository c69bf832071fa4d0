// ops.cuh -- finite-difference operators of the MacCormack/DRP scheme
// (src/forward/fd_t.h:9-140, tables in src/forward/fd_t.cu:64-110) as
// sm_100a device functions, plus the argument blocks of the stage kernels.
#pragma once
#include <cuda_runtime.h>

#include "../../include/cgfd.h"
#include "common.h"

namespace cgfd {

// one-sided 5-point DRP derivative, forward (F = 1: offsets -1..3) or
// backward (F = 0: offsets -3..1)
constexpr real kC1 = RL(-0.291647047), kC2 = RL(-0.666745142), kC3 = RL(1.250117713),
               kC4 = RL(-0.333411808), kC5 = RL(0.041686285);
// 2-point and 3-point one-sided operators (MAC22, MAC24)
constexpr real kB1 = RL(-7.0) / RL(6.0), kB2 = RL(8.0) / RL(6.0), kB3 = RL(-1.0) / RL(6.0);
// one-sided traction-image weights at split nodes
constexpr real kA0 = RL(1.2500392377), kA1 = RL(1.5417647610), kA2 = RL(-0.3334118088),
               kA3 = RL(0.0416862855);

__device__ __forceinline__ real mac22(const real *p, long s, int f) {
  return f ? (__ldg(p + s) - __ldg(p)) : (__ldg(p) - __ldg(p - s));
}
__device__ __forceinline__ real mac24(const real *p, long s, int f) {
  return f ? (kB1 * __ldg(p) + kB2 * __ldg(p + s) + kB3 * __ldg(p + 2 * s))
           : -(kB1 * __ldg(p) + kB2 * __ldg(p - s) + kB3 * __ldg(p - 2 * s));
}
// DRP on register values v[-3..3] centred at v
__device__ __forceinline__ real drp_v(const real *v, int f) {
  return f ? (kC1 * v[-1] + kC2 * v[0] + kC3 * v[1] + kC4 * v[2] + kC5 * v[3])
           : -(kC1 * v[1] + kC2 * v[0] + kC3 * v[-1] + kC4 * v[-2] + kC5 * v[-3]);
}

__device__ __forceinline__ void mv3(const real *__restrict__ m, const real *v, real *o) {
  o[0] = __ldg(m + 0) * v[0] + __ldg(m + 1) * v[1] + __ldg(m + 2) * v[2];
  o[1] = __ldg(m + 3) * v[0] + __ldg(m + 4) * v[1] + __ldg(m + 5) * v[2];
  o[2] = __ldg(m + 6) * v[0] + __ldg(m + 7) * v[1] + __ldg(m + 8) * v[2];
}

// level slots
enum { LP = 0, LA = 1, LB = 2, LE = 3 };
// RK mode of a stage = its index.  The classical RK4 step
//   u1 = u0 + dt/2 k1, u2 = u0 + dt/2 k2, u3 = u0 + dt k3,
//   u(n+1) = u0 + dt/6 (k1 + 2 k2 + 2 k3 + k4)
// is formed without an accumulator that every stage reads and writes: with
// V = u0 + (u1 - u0)/2 + (u2 - u0), known when the second stage ends,
//   u(n+1) = u3 + 2/3 (V - u3) + dt/6 k4
// is the same sum.  So only the second stage writes the fourth level (V)
// and only the last one reads it (u(n+1) takes its place), 156 values per
// point and step instead of 192.  Each value is written as a level plus
// small increments, so that a stored level is rounded once: five roundings
// of a level reach u(n+1), weighted 1/3, 2/3, 1/3 (u1, u2, u3), 2/3 (V) and
// 1, against four of weight 1 in the accumulator (measured on a hilly box
// without a fault, 12 steps: relative L2 error against 64 bits 1.4e-7, with
// the accumulator 2.0e-7).  Step with the accumulator -> so: 9.76 -> 8.65 ms
// on 300x600x240 with its read-backs, 2.75 -> 2.44 on 200x300x160, 0.565 ->
// 0.515 on 100x160x80.
enum { RK_FIRST = 0, RK_SECOND = 1, RK_THIRD = 2, RK_LAST = 3 };

// does a stage of this mode read the time-n level?
__host__ __device__ constexpr bool rk_reads_pre(int mode) { return mode == RK_SECOND || mode == RK_THIRD; }
// next stage input from the level it starts from (u0) and its increment
__device__ __forceinline__ real rk_out(real u0, real inc) { return u0 + inc; }
// V of the second stage: cur = u1, inc = u2 - u0
__device__ __forceinline__ real rk_v(real u0, real cur, real inc) { return u0 + (RL(0.5) * (cur - u0) + inc); }
// u(n+1) of the last stage: cur = u3, inc = dt/6 k4
__device__ __forceinline__ real rk_end(real v, real cur, real inc) { return cur + (RL(2.0) / RL(3.0) * (v - cur) + inc); }

// block of the volume kernels: kTileX x kTileY points of one z row.  128
// threads rather than 256: an SM refills in smaller pieces, the last wave is
// shorter (interior launch of 30.0 M points at the 1000 W cap 1.058 -> 1.018
// ms, 8 against 4 blocks per SM, the same 64 registers).
constexpr int kTileX = 32, kTileY = 4;

// a box of interior points (inclusive bounds) covered by one launch;
// blocks [first, next box's first) belong to it
struct VolBox {
  int i0, i1, j0, j1, k0, k1;
  int nbx, nby, first;
  int kind;
};
constexpr int kMaxBoxes = 48;

struct VolArgs {
  Grid g;
  int nbox, nblocks;
  int ychunk;                  // interior kernel: y tiles per chunk (z marches within a chunk)
  VolBox box[kMaxBoxes];
  const real *cur, *pre;
  real *out, *end;            // next-stage level (null at the last stage), E
  const real *coef, *free_mat;   // packed metric and medium (coef_group, coef_row, coef_jac)
  real ca, cb;
  int isfree;
  int nfault;
  // 1: the launch leaves the fault planes x = i0 within each fault's split
  // box grown by 3 nodes (welded nodes too; ghost-inclusive J0, J1, K0, K1
  // in fdef) to a later one, so that it reads nothing the stage's first
  // fault kernels write and may run beside them; outside that box no tap of
  // a plane point reaches a split node
  int defer_i0;
  int fi0[MAXF];
  int fdef[MAXF][4];
  const uint8_t *fflag[MAXF];
  PmlFaceDev pml[6];           // indexed 2*dim + side; `on` = 0 when absent
};

// operator triple N (4 x direction + 2 y + z) of the kernels that hold every
// kind; each is defined in a unit of its own
template <int N>
void launch_volume_all_n(const VolArgs &a, int mode, cudaStream_t st);

struct FaultArgs {
  Grid g;
  FaultDev F;
  const real *wcur, *wpre;
  real *wout, *wend;
  const real *coef, *free_mat;   // packed metric and medium (coef_group, coef_row, coef_jac)
  // fault wavefield levels [9][2 sides][ny*nz]: stage input, time-n level,
  // next-stage output (null at the last stage), fourth level (V, then n+1)
  const real *fc, *fp;
  real *fo, *fe;
  int idir, jdir, kdir;
  int mode;
  real ca, cb, rkb, dt;
  int isfree, imethod;
  int j0, k0, nj, nk;          // launch box of split nodes (interior indices)
  // welded nodes whose fault fields a stage reads (the split box grown by
  // the 3-node stencil reach, or the whole plane without split nodes)
  int wj0, wk0, wnj, wnk;
  Ctl *ctl;
  // tractions J e_a . sigma of the stage input at x = i0-6..i0-1, i0+1..i0+6
  // over the split box grown by 3 nodes in j and k: [12][9][tnk][tnj],
  // components T1 (e_xi), T2 (e_eta), T3 (e_zeta); T2 and T3 only for
  // |x - i0| <= 3.  tj0 / tk0: ghost-inclusive j / k of element (0, 0).
  real *trac;
  int tj0, tk0, tnj, tnk;
};

struct StationArgs {
  Grid g;
  StationDev st;
  const real *w;
  const real *fout[MAXF];
  long ns;
  Ctl *ctl;
};

// exponential sponge on the end-of-step level: masks E[nx | ny | nz]
// (ghost-inclusive index), blocks of ghost-inclusive inclusive bounds
// i1 i2 j1 j2 k1 k2, first[b] = points of the blocks before b
struct SpongeArgs {
  Grid g;
  real *w;
  const real *E;
  int nblk;
  int blk[6][6];
  long first[7];
};

// peak ground motion of the free surface: end-of-step and time-n levels,
// peaks [15][nj][ni] and displacement [3][nj][ni] at interior (i, j)
struct PeakArgs {
  Grid g;
  const real *wend, *wpre;
  real *pg, *dis;
  real dt;
  Ctl *ctl;
  int max_rec;
};

}  // namespace cgfd
