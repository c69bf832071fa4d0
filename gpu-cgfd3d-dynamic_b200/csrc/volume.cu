// volume.cu -- fused volume stage kernels.
//
// One RK stage of every grid point outside the split-node slabs of the
// faults: right-hand side of the velocity-stress system and the stage's
// Runge-Kutta update in one pass.
//   * interior stencil   sv_curv_col_el_iso_rhs_inner_gpu
//                        (src/forward/sv_curv_col_el_iso_gpu.cu:232-388)
//   * traction image     sv_curv_col_el_iso_rhs_timg_z2_gpu  (:399-600)
//   * velocity below the free surface
//                        sv_curv_col_el_iso_rhs_vlow_z2_gpu  (:607-747)
//   * CFS-PML correction and auxiliary-field RHS
//                        sv_curv_col_el_iso_rhs_cfspml_gpu   (:825-1290)
//   * RK stage update    wav_update / wav_update_end (src/forward/wav_t.cu:219-234)
//                        and the PML auxiliary updates of drv_rk_curv_col.cu:329-568
// The reference runs these as 9-10 launches per stage plus three full
// read-modify-write sweeps of the wavefield for the RK update.  Here the
// domain is cut into boxes: the interior box (no PML, no surface rows) runs
// k_volume<INTERIOR>, whose code holds no boundary logic; slabs that one
// direction's PML faces reach run k_volume<FACE_X/Y/Z>; PML edges, corners
// and the bottom ring run k_volume<EDGE>; the four rows under the free
// surface run k_volume<TOP> away from the PML columns and k_volume<SHELL>
// in them; the fault planes' welded points next to split nodes run
// k_volume<PLANE> after the first fault kernels.  On small grids
// k_volume_all runs all boundary boxes in one launch.  Each stage reads the
// input level (stencil taps come from L1/L2), the metric and the medium
// once and writes the output levels once; each thread asks L2 early for
// the lines it reads last (prefetch), and interior threads for the next z
// row's DRAM misses.
//
// A level stores the nine components of a point in two 16-byte groups and
// one real (Grid::w), so a stencil tap is three loads: x taps are
// immediate offsets from the point's three pointers, y / z taps share two
// int offset tables, the centre sample is loaded once for all three
// directions.  The RHS is built direction by direction, so a PML face of
// normal d reuses direction d's contribution.
//
// Roofline: algorithmic traffic per point and step is 156 floats = 624 B
// (21+9, 30+18, 30+9, 30+9 floats over the 4 stages), 140 on aligned grids.
// In practice large grids also meet the 1000 W limit and the interior kernel
// the L1 data pipe (13 taps of 36 bytes a point), small ones latency.
#include <cuda_runtime.h>

#include "ops.cuh"

namespace cgfd {

namespace {

constexpr int BX = kTileX, BY = kTileY;

// conservative traction J * (e . sigma_row) at point q for metric row DIR
// (0: xi, 1: eta, 2: zeta), all three stress rows (xx,xy,xz), (xy,yy,yz),
// (xz,yz,zz)
template <int DIR, bool AL>
__device__ __forceinline__ void ctrac3(const Grid &g, const real *__restrict__ w, const real *__restrict__ cf,
                                       long q, real t[3]) {
  const real4 e = coef_group(cf, g.scmp, AL ? DIR / 2 : DIR, q);
  const real J = coef_jac(cf, q);
  const real sxx = __ldg(w + g.w(TXX, q)), sxy = __ldg(w + g.w(TXY, q));
  const real4 s4 = __ldg(reinterpret_cast<const real4 *>(w + 4 * g.scmp) + q);   // Tyy Tzz Tyz Txz
  const real syy = s4.x, szz = s4.y, syz = s4.z, sxz = s4.w;
  if (AL && DIR == 0) {
    t[0] = J * (e.x * sxx); t[1] = J * (e.x * sxy); t[2] = J * (e.x * sxz);
  } else if (AL && DIR == 1) {
    t[0] = J * (e.y * sxy); t[1] = J * (e.y * syy); t[2] = J * (e.y * syz);
  } else {
    t[0] = J * (e.x * sxx + e.y * sxy + e.z * sxz);
    t[1] = J * (e.x * sxy + e.y * syy + e.z * syz);
    t[2] = J * (e.x * sxz + e.y * syz + e.z * szz);
  }
}

// The point's three groups within one level: pointers to the point itself,
// from which x taps are immediate offsets, and the level's arrays with the
// point number, so that a y or z tap's address is one 32-bit multiply-add
// from an array base that the whole block shares instead of a 64-bit sum per
// thread (184 -> 146 integer instructions per interior point; 240x400x133
// interior launch 236 -> 232 us).  Point numbers fit 32 bits: a level of 2^32
// points would be 155 GB.
struct Taps {
  const real4 *__restrict__ a;  // Vx Vy Vz Txx
  const real4 *__restrict__ b;  // Tyy Tzz Tyz Txz
  const real *__restrict__ t;   // Txy
  const real4 *a0, *b0;
  const real *t0;
  unsigned p;
};
__device__ __forceinline__ Taps taps_at(const real *w, long sc, unsigned p) {
  Taps T;
  T.a0 = reinterpret_cast<const real4 *>(w);
  T.b0 = reinterpret_cast<const real4 *>(w + 4 * sc);
  T.t0 = w + 8 * sc;
  T.p = p;
  T.a = T.a0 + p;
  T.b = T.b0 + p;
  T.t = T.t0 + p;
  return T;
}
// Nine components of a point as they lie in memory: the pairs (Vx Vy) (Vz
// Txx) (Tyy Tzz) (Tyz Txz) and Txy.  The stencil sums run on pairs: on
// sm_100 one fma.rn.f32x2 does two multiply-adds, each rounded as the
// scalar one, so the 27 derivatives of a point take 75 instructions instead
// of 135 (interior launch of 30.0 M points with waves everywhere, where the
// GPU sits at its 1000 W cap: 1.089 -> 1.058 ms).  At 64 registers 17 of the 64
// interior instantiations spill 4-16 bytes, 7 of them the aligned ones of
// stage 2, which writes two levels.
#ifdef CGFD_FP64
typedef double2 real2;
__device__ __forceinline__ real2 mul2(real c, real2 x) { return make_double2(c * x.x, c * x.y); }
__device__ __forceinline__ real2 fma2(real c, real2 x, real2 y) { return make_double2(fma(c, x.x, y.x), fma(c, x.y, y.y)); }
__device__ __forceinline__ void split2(real2 v, real &x, real &y) { x = v.x; y = v.y; }
__device__ __forceinline__ void ldg4(const real4 *q, real2 &x, real2 &y) {
  x = ::__ldg(reinterpret_cast<const double2 *>(q));
  y = ::__ldg(reinterpret_cast<const double2 *>(q) + 1);
}
#else
typedef unsigned long long real2;
__device__ __forceinline__ real2 pack2(real x, real y) {
  real2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void split2(real2 v, real &x, real &y) { asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ real2 mul2(real c, real2 x) {
  real2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(c, c)), "l"(x));
  return r;
}
__device__ __forceinline__ real2 fma2(real c, real2 x, real2 y) {
  real2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pack2(c, c)), "l"(x), "l"(y));
  return r;
}
__device__ __forceinline__ void ldg4(const real4 *q, real2 &x, real2 &y) {
  const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2 *>(q));
  x = v.x;
  y = v.y;
}
#endif
struct V9 {
  real2 p[4];
  real t;
};
__device__ __forceinline__ void unpack9(const V9 &v, real d[9]) {
#pragma unroll
  for (int n = 0; n < 4; n++) split2(v.p[n], d[2 * n], d[2 * n + 1]);
  d[8] = v.t;
}
__device__ __forceinline__ V9 mul9(real c, const V9 &x) {
  V9 r;
#pragma unroll
  for (int n = 0; n < 4; n++) r.p[n] = mul2(c, x.p[n]);
  r.t = c * x.t;
  return r;
}
__device__ __forceinline__ V9 fma9(real c, const V9 &x, const V9 &y) {
  V9 r;
#pragma unroll
  for (int n = 0; n < 4; n++) r.p[n] = fma2(c, x.p[n], y.p[n]);
  r.t = fma(c, x.t, y.t);
  return r;
}
// the nine components of the point o points away; X: a tap along x
template <bool X>
__device__ __forceinline__ V9 tap9(const Taps &T, int o) {
  V9 v;
  ldg4(X ? T.a + o : (T.a0 + o) + T.p, v.p[0], v.p[1]);
  ldg4(X ? T.b + o : (T.b0 + o) + T.p, v.p[2], v.p[3]);
  v.t = __ldg(X ? T.t + o : (T.t0 + o) + T.p);
  return v;
}

template <int F>
__device__ __forceinline__ real wdrp(int n) {
  return F ? (n == 0 ? kC1 : n == 1 ? kC2 : n == 2 ? kC3 : n == 3 ? kC4 : kC5)
           : (n == 0 ? -kC5 : n == 1 ? -kC4 : n == 2 ? -kC3 : n == 3 ? -kC2 : -kC1);
}

template <int F>
__device__ __forceinline__ void tap_offsets(int s, int off[4]) {
  if (F) { off[0] = -s; off[1] = s; off[2] = 2 * s; off[3] = 3 * s; }
  else { off[0] = -3 * s; off[1] = -2 * s; off[2] = -s; off[3] = s; }
}

// Aligned grids (AL): the metric rows of directions x and y have one entry
// each, (xi_x 0 0) and (0 eta_y 0), as under a stretched topography above a
// vertical fault.  direction-DIR part of the RHS from the nine derivatives
// D[c] along it and e, its metric row
template <int DIR, bool AL>
__device__ __forceinline__ void rhs_dir(const real D[9], const real e[3], real lam, real mu, real l2m,
                                        real slw, real r[9]) {
  if (AL && DIR == 0) {
    r[VX] = slw * (e[0] * D[TXX]); r[VY] = slw * (e[0] * D[TXY]); r[VZ] = slw * (e[0] * D[TXZ]);
    r[TXX] = l2m * e[0] * D[VX]; r[TYY] = r[TZZ] = lam * (e[0] * D[VX]);
    r[TXY] = mu * (e[0] * D[VY]); r[TXZ] = mu * (e[0] * D[VZ]); r[TYZ] = 0.f;
    return;
  }
  if (AL && DIR == 1) {
    r[VX] = slw * (e[1] * D[TXY]); r[VY] = slw * (e[1] * D[TYY]); r[VZ] = slw * (e[1] * D[TYZ]);
    r[TYY] = l2m * e[1] * D[VY]; r[TXX] = r[TZZ] = lam * (e[1] * D[VY]);
    r[TXY] = mu * (e[1] * D[VX]); r[TYZ] = mu * (e[1] * D[VZ]); r[TXZ] = 0.f;
    return;
  }
  r[VX] = slw * (e[0] * D[TXX] + e[1] * D[TXY] + e[2] * D[TXZ]);
  r[VY] = slw * (e[0] * D[TXY] + e[1] * D[TYY] + e[2] * D[TYZ]);
  r[VZ] = slw * (e[0] * D[TXZ] + e[1] * D[TYZ] + e[2] * D[TZZ]);
  r[TXX] = l2m * e[0] * D[VX] + lam * (e[1] * D[VY] + e[2] * D[VZ]);
  r[TYY] = l2m * e[1] * D[VY] + lam * (e[0] * D[VX] + e[2] * D[VZ]);
  r[TZZ] = l2m * e[2] * D[VZ] + lam * (e[0] * D[VX] + e[1] * D[VY]);
  r[TXY] = mu * (e[1] * D[VX] + e[0] * D[VY]);
  r[TXZ] = mu * (e[2] * D[VX] + e[0] * D[VZ]);
  r[TYZ] = mu * (e[2] * D[VY] + e[1] * D[VZ]);
}

// one-sided DRP derivatives of the nine components in table order (F:
// offsets -1, 0, 1, 2, 3; B: -3, -2, -1, 0, 1), the centre sample v0 known;
// off[n] are the offsets of the other four taps
template <int F, bool X>
__device__ __forceinline__ void derivs(const Taps &T, const V9 &v0, const int off[4], real D[9]) {
  V9 r = mul9(wdrp<F>(0), tap9<X>(T, off[0]));
  if (F) r = fma9(wdrp<F>(1), v0, r);
  r = fma9(wdrp<F>(F ? 2 : 1), tap9<X>(T, off[1]), r);
  r = fma9(wdrp<F>(F ? 3 : 2), tap9<X>(T, off[2]), r);
  if (!F) r = fma9(wdrp<F>(3), v0, r);
  unpack9(fma9(wdrp<F>(4), tap9<X>(T, off[3]), r), D);
}

// Accumulate one direction's derivatives straight into the strain rates
// E = (xx, yy, zz, yz, xz, xy), the shear ones as the sums dV_b/dx_c +
// dV_c/dx_b that Hooke's law needs, and the momentum sums
// s_r = sum_a e_a . d(sigma_row r)/dxi_a.
template <int DIR, bool AL>
__device__ __forceinline__ void accumulate(const real D[9], const real ea[3], real E[6], real s[3]) {
  if (AL && DIR == 0) {
    E[0] += ea[0] * D[VX]; E[4] += ea[0] * D[VZ]; E[5] += ea[0] * D[VY];
    s[0] += ea[0] * D[TXX]; s[1] += ea[0] * D[TXY]; s[2] += ea[0] * D[TXZ];
    return;
  }
  if (AL && DIR == 1) {
    E[1] += ea[1] * D[VY]; E[3] += ea[1] * D[VZ]; E[5] += ea[1] * D[VX];
    s[0] += ea[1] * D[TXY]; s[1] += ea[1] * D[TYY]; s[2] += ea[1] * D[TYZ];
    return;
  }
  E[0] += ea[0] * D[VX];
  E[1] += ea[1] * D[VY];
  E[2] += ea[2] * D[VZ];
  E[3] += ea[2] * D[VY]; E[3] += ea[1] * D[VZ];
  E[4] += ea[2] * D[VX]; E[4] += ea[0] * D[VZ];
  E[5] += ea[1] * D[VX]; E[5] += ea[0] * D[VY];
  s[0] += ea[0] * D[TXX];
  s[1] += ea[1] * D[TYY];
  s[2] += ea[2] * D[TZZ];
  s[1] += ea[2] * D[TYZ]; s[2] += ea[1] * D[TYZ];
  s[0] += ea[2] * D[TXZ]; s[2] += ea[0] * D[TXZ];
  s[0] += ea[1] * D[TXY]; s[1] += ea[0] * D[TXY];
}
template <int F, int DIR, bool AL>
__device__ __forceinline__ void acc_dir(const Taps &T, const V9 &v0, const int off[4], const real ea[3],
                                        real E[6], real s[3]) {
  real D[9];
  derivs<F, DIR == 0>(T, v0, off, D);
  accumulate<DIR, AL>(D, ea, E, s);
}
// rates of the nine components from the accumulated sums
__device__ __forceinline__ void rates(const real E[6], const real s[3], real lam, real mu, real slw, real h[9]) {
  const real l2m = lam + 2.0f * mu;
  h[VX] = slw * s[0]; h[VY] = slw * s[1]; h[VZ] = slw * s[2];
  h[TXX] = l2m * E[0] + lam * (E[1] + E[2]);
  h[TYY] = l2m * E[1] + lam * (E[0] + E[2]);
  h[TZZ] = l2m * E[2] + lam * (E[0] + E[1]);
  h[TYZ] = mu * E[3]; h[TXZ] = mu * E[4]; h[TXY] = mu * E[5];
}

// the nine components of point p of a level in the grouped layout with
// sc points per component (read-only data through the non-coherent path)
__device__ __forceinline__ void ld9(const real *w, long sc, unsigned p, real v[9], bool ro) {
  const real4 *A = reinterpret_cast<const real4 *>(w) + p, *B = reinterpret_cast<const real4 *>(w + 4 * sc) + p;
  const real4 x = ro ? __ldg(A) : *A, y = ro ? __ldg(B) : *B;
  v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
  v[8] = ro ? __ldg((w + 8 * sc) + p) : (w + 8 * sc)[p];
}
// the nine components of point p of level w
__device__ __forceinline__ void st9(real *w, long sc, unsigned p, const real v[9]) {
  reinterpret_cast<real4 *>(w)[p] = make_real4(v[0], v[1], v[2], v[3]);
  reinterpret_cast<real4 *>(w + 4 * sc)[p] = make_real4(v[4], v[5], v[6], v[7]);
  (w + 8 * sc)[p] = v[8];
}

// RK stage update (see RK_FIRST in ops.cuh) of nine components at point p of
// levels with sc points per component: cur holds the stage input's values,
// h their rates.  All reads of the levels are issued before the first
// store: the compiler cannot prove that the levels do not alias, and
// interleaved load / store pairs would cost one memory round trip per
// component.
template <int MODE>
__device__ __forceinline__ void rk_point(const real *pre, real *out, real *end, long sc, unsigned p, real ca, real cb,
                                         const real cur[9], const real h[9]) {
  real r[9];
  if (MODE == RK_FIRST) {
#pragma unroll
    for (int c = 0; c < 9; c++) r[c] = rk_out(cur[c], ca * h[c]);
    st9(out, sc, p, r);
  } else if (MODE == RK_LAST) {
    real v[9];
    ld9(end, sc, p, v, false);
#pragma unroll
    for (int c = 0; c < 9; c++) r[c] = rk_end(v[c], cur[c], cb * h[c]);
    st9(end, sc, p, r);
  } else {
    real u0[9];
    ld9(pre, sc, p, u0, true);
#pragma unroll
    for (int c = 0; c < 9; c++) r[c] = rk_out(u0[c], ca * h[c]);
    st9(out, sc, p, r);
    if (MODE == RK_SECOND) {
#pragma unroll
      for (int c = 0; c < 9; c++) r[c] = rk_v(u0[c], cur[c], ca * h[c]);
      st9(end, sc, p, r);
    }
  }
}
// L2 prefetch of the lines of point p of a level
__device__ __forceinline__ void prefetch9(const real *w, long sc, unsigned p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const real4 *>(w) + p));
  asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const real4 *>(w + 4 * sc) + p));
  asm volatile("prefetch.global.L2 [%0];" ::"l"((w + 8 * sc) + p));
}
// L2 prefetch of the auxiliary-field lines that pml_face reads at (I, J, K)
template <int MODE>
__device__ __forceinline__ void pml_prefetch(const PmlFaceDev &P, int I, int J, int K) {
  const int li = I - P.i1, lj = J - P.j1, lk = K - P.k1;
  if (li < 0 || li >= P.fni || lj < 0 || lj >= P.fnj || lk < 0 || lk >= P.fnk) return;
  const unsigned pa = li + (lj + lk * P.fnj) * P.fni;
  const long sz = P.siz;
  const real *lv[3] = { P.acur, rk_reads_pre(MODE) ? P.apre : nullptr, MODE == RK_LAST ? P.aend : nullptr };
#pragma unroll
  for (int l = 0; l < 3; l++) {
    if (!lv[l]) continue;
    prefetch9(lv[l], sz, pa);
  }
}

// PML face P (normal d) at this point: add its correction to corr and
// advance its auxiliary fields (stored like a wavefield level, grouped,
// with P.siz points per component)
template <int MODE>
__device__ __forceinline__ void pml_face(const VolArgs &a, const PmlFaceDev &P, int d, int I, int J, int K,
                                         const real r[9], const real D[9], const real e2[3], real lam,
                                         real mu, real l2m, bool surf, long fidx, real corr[9]) {
  const int li = I - P.i1, lj = J - P.j1, lk = K - P.k1;
  if (li < 0 || li >= P.fni || lj < 0 || lj >= P.fnj || lk < 0 || lk >= P.fnk) return;
  const int layer = d == 0 ? li : (d == 1 ? lj : lk);
  const real cA = __ldg(P.A + layer), cB = __ldg(P.B + layer), cD = __ldg(P.D + layer);
  const unsigned pa = li + (lj + lk * P.fnj) * P.fni;
  real ac[9], ar[9];
  ld9(P.acur, P.siz, pa, ac, true);
#pragma unroll
  for (int c = 0; c < 9; c++) {
    corr[c] += (cB - 1.0f) * r[c] - cB * ac[c];
    ar[c] = cD * r[c] - cA * ac[c];
  }
  if (surf) {
    // free-surface coupling of the x / y faces: the d-derivative of the
    // surface-converted dz velocity gradient
    const real *X = a.free_mat + (long)(d == 0 ? 0 : 1) * a.g.ny * a.g.nx * 9 + fidx;
    const real dd[3] = { D[VX], D[VY], D[VZ] };
    real z[3];
    mv3(X, dd, z);
    real q[9];
    q[TXX] = l2m * (e2[0] * z[0]) + lam * (e2[1] * z[1] + e2[2] * z[2]);
    q[TYY] = l2m * (e2[1] * z[1]) + lam * (e2[0] * z[0] + e2[2] * z[2]);
    q[TZZ] = l2m * (e2[2] * z[2]) + lam * (e2[0] * z[0] + e2[1] * z[1]);
    q[TXY] = mu * (e2[1] * z[0] + e2[0] * z[1]);
    q[TXZ] = mu * (e2[2] * z[0] + e2[0] * z[2]);
    q[TYZ] = mu * (e2[2] * z[1] + e2[1] * z[2]);
#pragma unroll
    for (int c = TXX; c <= TXY; c++) { corr[c] += (cB - 1.0f) * q[c]; ar[c] += cD * q[c]; }
  }
  rk_point<MODE>(P.apre, P.aout, P.aend, P.siz, pa, a.ca, a.cb, ac, ar);
}

// RK stage update of the wavefield at p
template <int MODE>
__device__ __forceinline__ void rk_update(const VolArgs &a, unsigned p, const real v0[9], const real h[9]) {
  rk_point<MODE>(a.pre, a.out, a.end, a.g.scmp, p, a.ca, a.cb, v0, h);
}

// kernel kinds: the interior box (no boundary logic), slabs that only PML
// faces of one direction reach (x, y or z), the generic shell (the rows
// under the free surface, with any PML faces), and the PML edges and
// corners away from the free surface (the shell's code without the
// free-surface logic, which keeps it in registers)
enum { INTERIOR = 0, SHELL = 1, FACE_X = 2, FACE_Y = 3, FACE_Z = 4, EDGE = 5, PLANE = 6, TOP = 7 };
// PLANE: the interior kernel's code on packed boxes: the fault planes
// x = i0 inside the interior box, when the interior launch defers them.
// TOP: the shell's code without the PML faces, for the rows under the free
// surface away from every PML face (fewer live values than the shell)

// block -> box of a launch's list (sorted by first block)
__device__ __forceinline__ int box_of_block(const VolArgs &a) {
  int lo = 0, hi = a.nbox - 1;
#pragma unroll 1
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if ((int)blockIdx.x >= a.box[mid].first) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}
// block -> point of box b; boxes with a narrow x extent (PML x slabs) pack
// their points densely instead of leaving most of a 32-wide row idle
__device__ __forceinline__ bool locate(const VolArgs &a, int b, int &i, int &j, int &k) {
  const VolBox &B = a.box[b];
  const int bid = blockIdx.x - B.first;
  const int ni = B.i1 - B.i0 + 1, nj = B.j1 - B.j0 + 1;
  if (B.nbx == 0) {
    // packed: flat index over the (x, y) rectangle of one z row
    const int t = (bid % B.nby) * (BX * BY) + threadIdx.y * BX + threadIdx.x;
    k = B.k0 + bid / B.nby;
    if (t >= ni * nj) return false;
    i = B.i0 + t % ni;
    j = B.j0 + t / ni;
    return true;
  }
  const int bx = bid % B.nbx, rem = bid / B.nbx, by = rem % B.nby, bz = rem / B.nby;
  i = B.i0 + bx * BX + threadIdx.x;
  j = B.j0 + by * BY + threadIdx.y;
  k = B.k0 + bz;
  return i <= B.i1 && j <= B.j1;
}

// interior box (one box): 3-D grid (x tiles, y tiles of one chunk, z rows x
// chunks).  The blocks of one y chunk of a.ychunk tiles march up z before
// the next chunk starts, so the planes a z window touches stay in L2 (a
// whole xy plane per z row would need more than the 126 MB L2 holds).
[[maybe_unused]] __device__ __forceinline__ bool locate_interior(const VolArgs &a, int &i, int &j, int &k) {
  const VolBox &B = a.box[0];
  const int nkb = B.k1 - B.k0 + 1;
  const int chunk = blockIdx.z / nkb, bz = blockIdx.z - chunk * nkb;
  const int by = chunk * a.ychunk + blockIdx.y;
  i = B.i0 + blockIdx.x * BX + threadIdx.x;
  j = B.j0 + by * BY + threadIdx.y;
  k = B.k0 + bz;
  return i <= B.i1 && j <= B.j1;
}

// points that another kernel updates: the split-node slabs (i0-3..i0+3 of
// unwelded nodes) belong to the fault kernels; with defer_i0 the fault
// planes go to a later launch
__device__ __forceinline__ bool other_kernels_point(const VolArgs &a, int I, int J, int K) {
  for (int f = 0; f < a.nfault; f++) {
    const int d = I - a.fi0[f];
    if (d < -3 || d > 3) continue;
    if (d == 0 && a.defer_i0 && J >= a.fdef[f][0] && J <= a.fdef[f][1] && K >= a.fdef[f][2] &&
        K <= a.fdef[f][3])
      return true;
    if (__ldg(a.fflag[f] + J + (long)K * a.g.ny) & FL_SPLIT) return true;
  }
  return false;
}

#ifndef CGFD_PREFETCH
#define CGFD_PREFETCH 1
#endif
// interior kernel: z rows ahead whose DRAM misses each thread prefetches
// (0: none)
#ifndef CGFD_AHEAD
#define CGFD_AHEAD 1
#endif

// resident blocks per SM asked of the compiler, per kernel kind (register
// budget 65536 / (128 x blocks))
#ifndef CGFD_LB_INTERIOR
#define CGFD_LB_INTERIOR 8
#endif
#ifndef CGFD_LB_TOP
#define CGFD_LB_TOP 6
#endif
#ifndef CGFD_LB_SHELL
#define CGFD_LB_SHELL 6
#endif
#ifndef CGFD_LB_FACE
#define CGFD_LB_FACE 6
#endif

// one RK stage of one point
template <int ID, int JD, int KD, int MODE, int KIND, bool AL>
__device__ __forceinline__ void volume_point(const VolArgs &a, int i, int j, int k) {
  static_assert(KIND >= INTERIOR && KIND <= TOP, "kernel kind");
  const Grid &g = a.g;
  const long sc = g.scmp;
  const int I = i + NG, J = j + NG, K = k + NG;
  const unsigned sy = (unsigned)g.sy, sz = (unsigned)g.sz;
  const unsigned p = (I + g.xoff) + J * sy + K * sz;
  if (other_kernels_point(a, I, J, K)) return;
#if CGFD_PREFETCH
  // the RK update reads the time-n level (in the last stage V) at its end:
  // ask L2 for its lines now, so that those reads wait on L2, not DRAM
  if (MODE != RK_FIRST) prefetch9(MODE == RK_LAST ? a.end : a.pre, sc, p);
#if CGFD_AHEAD > 0
  if (KIND == INTERIOR) {
    // the DRAM misses of the block CGFD_AHEAD z rows up: the newest stencil
    // plane of the stage input and its coefficients (that block runs soon
    // after this one: blocks march up z within a y chunk)
    const int kc = K + CGFD_AHEAD, kn = kc + (KD ? 3 : 1);
    if (kn < g.nz) prefetch9(a.cur, sc, p + (kn - K) * sz);
    if (kc < g.nz) {
#pragma unroll
      for (int n = 0; n < (AL ? 2 : 3); n++)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const real4 *>(a.coef + sc + 4 * n * sc) + (p + CGFD_AHEAD * sz)));
    }
  }
#endif
  // likewise the auxiliary fields of the PML faces this point lies in
  if (KIND != INTERIOR && KIND != PLANE && KIND != TOP) {
#pragma unroll
    for (int f = 0; f < 6; f++) {
      if (KIND >= FACE_X && KIND <= FACE_Z && f / 2 != KIND - FACE_X) continue;
      if (a.pml[f].on) pml_prefetch<MODE>(a.pml[f], I, J, K);
    }
  }
#endif
  const Taps w = taps_at(a.cur, sc, p);
  const V9 c0 = tap9<true>(w, 0);
  real v0[9];
  unpack9(c0, v0);
  // the metric rows and the medium
  const real4 g0 = coef_group(a.coef, sc, 0, p), g1 = coef_group(a.coef, sc, 1, p);
  const real4 r0 = AL ? make_real4(g0.x, 0.f, 0.f, g0.z) : g0;
  const real4 r1 = AL ? make_real4(0.f, g0.y, 0.f, g0.w) : g1;
  const real4 r2 = AL ? g1 : coef_group(a.coef, sc, 2, p);
  const real e[3][3] = { { r0.x, r0.y, r0.z }, { r1.x, r1.y, r1.z }, { r2.x, r2.y, r2.z } };
  const real lam = r0.w, mu = r1.w, slw = r2.w;
  const real l2m = lam + 2.0f * mu;
  int ox[4], oy[4], oz[4];
  tap_offsets<ID>(1, ox);
  tap_offsets<JD>((int)g.sy, oy);
  tap_offsets<KD>((int)g.sz, oz);

  real h[9];
  if (KIND == INTERIOR || KIND == PLANE) {
    real E[6] = { 0.f, 0.f, 0.f, 0.f, 0.f, 0.f };
    real s[3] = { 0.f, 0.f, 0.f };
    acc_dir<ID, 0, AL>(w, c0, ox, e[0], E, s);
    acc_dir<JD, 1, AL>(w, c0, oy, e[1], E, s);
    acc_dir<KD, 2, AL>(w, c0, oz, e[2], E, s);
    rates(E, s, lam, mu, slw, h);
    rk_update<MODE>(a, p, v0, h);
    return;
  }

  if constexpr (KIND >= FACE_X && KIND <= FACE_Z) {
    // one PML direction FD: the other two directions accumulate like the
    // interior, direction FD is kept apart for the face's correction and
    // auxiliary update
    constexpr int FD = KIND - FACE_X;
    constexpr int FF = FD == 0 ? ID : (FD == 1 ? JD : KD);
    real E[6] = { 0.f, 0.f, 0.f, 0.f, 0.f, 0.f };
    real s[3] = { 0.f, 0.f, 0.f };
    if (FD != 0) acc_dir<ID, 0, AL>(w, c0, ox, e[0], E, s);
    if (FD != 1) acc_dir<JD, 1, AL>(w, c0, oy, e[1], E, s);
    if (FD != 2) acc_dir<KD, 2, AL>(w, c0, oz, e[2], E, s);
    real D[9], r[9], corr[9];
    derivs<FF, FD == 0>(w, c0, FD == 0 ? ox : (FD == 1 ? oy : oz), D);
    rhs_dir<FD, AL>(D, e[FD], lam, mu, l2m, slw, r);
    rates(E, s, lam, mu, slw, h);
#pragma unroll
    for (int c = 0; c < 9; c++) h[c] += r[c];
#pragma unroll
    for (int c = 0; c < 9; c++) corr[c] = 0.f;
    if (a.pml[2 * FD].on) pml_face<MODE>(a, a.pml[2 * FD], FD, I, J, K, r, D, e[2], lam, mu, l2m, false, 0, corr);
    if (a.pml[2 * FD + 1].on) pml_face<MODE>(a, a.pml[2 * FD + 1], FD, I, J, K, r, D, e[2], lam, mu, l2m, false, 0, corr);
#pragma unroll
    for (int c = 0; c < 9; c++) h[c] += corr[c];
    rk_update<MODE>(a, p, v0, h);
    return;
  }

  // ---- shell and edges: PML edges and corners, rows under the free surface
  const int nk2 = g.nk + NG - 1;
  const bool top = (KIND == SHELL || KIND == TOP) && a.isfree && K >= nk2 - 3;
  const bool surfrow = (KIND == SHELL || KIND == TOP) && a.isfree && K == nk2;
  constexpr bool pml = KIND != TOP;
  const long fidx = ((long)J * g.nx + I) * 9;
  real corr[9], r[9], D[9], dvx[3], dvy[3];
#pragma unroll
  for (int c = 0; c < 9; c++) corr[c] = 0.f;
  // x
  derivs<ID, true>(w, c0, ox, D);
  dvx[0] = D[VX]; dvx[1] = D[VY]; dvx[2] = D[VZ];
  rhs_dir<0, AL>(D, e[0], lam, mu, l2m, slw, r);
#pragma unroll
  for (int c = 0; c < 9; c++) h[c] = r[c];
  if (pml && a.pml[0].on) pml_face<MODE>(a, a.pml[0], 0, I, J, K, r, D, e[2], lam, mu, l2m, surfrow, fidx, corr);
  if (pml && a.pml[1].on) pml_face<MODE>(a, a.pml[1], 0, I, J, K, r, D, e[2], lam, mu, l2m, surfrow, fidx, corr);
  // y
  derivs<JD, false>(w, c0, oy, D);
  dvy[0] = D[VX]; dvy[1] = D[VY]; dvy[2] = D[VZ];
  rhs_dir<1, AL>(D, e[1], lam, mu, l2m, slw, r);
#pragma unroll
  for (int c = 0; c < 9; c++) h[c] += r[c];
  if (pml && a.pml[2].on) pml_face<MODE>(a, a.pml[2], 1, I, J, K, r, D, e[2], lam, mu, l2m, surfrow, fidx, corr);
  if (pml && a.pml[3].on) pml_face<MODE>(a, a.pml[3], 1, I, J, K, r, D, e[2], lam, mu, l2m, surfrow, fidx, corr);
  // z
  derivs<KD, false>(w, c0, oz, D);
  rhs_dir<2, AL>(D, e[2], lam, mu, l2m, slw, r);
  if (pml && a.pml[4].on) pml_face<MODE>(a, a.pml[4], 2, I, J, K, r, D, e[2], lam, mu, l2m, false, fidx, corr);
  if (pml && a.pml[5].on) pml_face<MODE>(a, a.pml[5], 2, I, J, K, r, D, e[2], lam, mu, l2m, false, fidx, corr);
  if (top && K >= nk2 - 2) {
    // velocity below the surface: the z part of the velocity gradient comes
    // from the conversion matrices (surface) or from 2nd / 4th order
    // one-sided differences (one / two rows below)
    const long sz = g.sz;
    real dz[3];
    if (K == nk2) {
      const real *X = a.free_mat + fidx;
      const real *Y = X + (long)g.ny * g.nx * 9;
      real o1[3], o2[3];
      mv3(X, dvx, o1); mv3(Y, dvy, o2);
      dz[0] = o1[0] + o2[0]; dz[1] = o1[1] + o2[1]; dz[2] = o1[2] + o2[2];
    } else if (K == nk2 - 1) {
      // velocities are components 0-2 of the first group: stride 4 floats
      const real *v = a.cur + 4 * (long)p;
      dz[0] = mac22(v + VX, 4 * sz, KD); dz[1] = mac22(v + VY, 4 * sz, KD); dz[2] = mac22(v + VZ, 4 * sz, KD);
    } else {
      const real *v = a.cur + 4 * (long)p;
      dz[0] = mac24(v + VX, 4 * sz, KD); dz[1] = mac24(v + VY, 4 * sz, KD); dz[2] = mac24(v + VZ, 4 * sz, KD);
    }
    real Dz[9], rz[9];
#pragma unroll
    for (int c = 0; c < 9; c++) Dz[c] = 0.f;
    Dz[VX] = dz[0]; Dz[VY] = dz[1]; Dz[VZ] = dz[2];
    rhs_dir<2, AL>(Dz, e[2], lam, mu, l2m, slw, rz);
#pragma unroll
    for (int c = TXX; c <= TXY; c++) h[c] += rz[c];
#pragma unroll
    for (int c = VX; c <= VZ; c++) h[c] += r[c];
  } else {
#pragma unroll
    for (int c = 0; c < 9; c++) h[c] += r[c];
  }
  if (top && K >= nk2 - (KD ? 3 : 1)) {
    // traction image on the momentum equation in the top rows
    const real *cur = a.cur;
    const long sy = g.sy;
    const real sj = slw / coef_jac(a.coef, p);
    // per tap the three traction rows at once; each row's sum over the
    // taps keeps the order of the coefficient table
    real dx[3] = { 0.f, 0.f, 0.f }, dy[3] = { 0.f, 0.f, 0.f }, dzz[3] = { 0.f, 0.f, 0.f };
    real t[3];
#pragma unroll
    for (int n = 0; n < 5; n++) {
      ctrac3<0, AL>(g, cur, a.coef, p + (ID ? n - 1 : n - 3), t);
#pragma unroll
      for (int rr = 0; rr < 3; rr++) dx[rr] += wdrp<ID>(n) * t[rr];
    }
#pragma unroll
    for (int n = 0; n < 5; n++) {
      ctrac3<1, AL>(g, cur, a.coef, p + (JD ? n - 1 : n - 3) * sy, t);
#pragma unroll
      for (int rr = 0; rr < 3; rr++) dy[rr] += wdrp<JD>(n) * t[rr];
    }
#pragma unroll
    for (int n = 0; n < 5; n++) {
      const int kk = K + (KD ? n - 1 : n - 3);
      if (kk == nk2) {
        t[0] = t[1] = t[2] = 0.f;
      } else {
        ctrac3<2, AL>(g, cur, a.coef, g.at(I, J, kk < nk2 ? kk : 2 * nk2 - kk), t);
        if (kk > nk2) { t[0] = -t[0]; t[1] = -t[1]; t[2] = -t[2]; }
      }
#pragma unroll
      for (int rr = 0; rr < 3; rr++) dzz[rr] += wdrp<KD>(n) * t[rr];
    }
#pragma unroll
    for (int rr = 0; rr < 3; rr++) h[VX + rr] = (dx[rr] + dy[rr] + dzz[rr]) * sj;
  }
#pragma unroll
  for (int c = 0; c < 9; c++) h[c] += corr[c];
  rk_update<MODE>(a, p, v0, h);
}

template <int ID, int JD, int KD, int MODE, int KIND, bool AL>
__global__ void __launch_bounds__(BX * BY, KIND == INTERIOR || KIND == PLANE ? CGFD_LB_INTERIOR
                                         : (KIND == SHELL || KIND == EDGE ? CGFD_LB_SHELL
                                                                          : (KIND == TOP ? CGFD_LB_TOP : CGFD_LB_FACE)))
    k_volume(const __grid_constant__ VolArgs a) {
  int i, j, k;
  if (KIND == INTERIOR ? !locate_interior(a, i, j, k) : !locate(a, box_of_block(a), i, j, k)) return;
  volume_point<ID, JD, KD, MODE, KIND, AL>(a, i, j, k);
}

#ifndef CGFD_LB_ALL
#define CGFD_LB_ALL 6
#endif
// every kind in one launch, each block the kind of its box (merge_points in
// api.cu says when).  6 blocks per SM as the boundary kinds have them alone;
// 5: 105 us per step of 36x56x32 and 419 of 101x163x77, 8: 116 and 433, 6: 107
// and 420.  One register budget (80) for seven bodies: every instantiation
// spills, 4-132 bytes on aligned grids and 36-196 on others, the second
// stage's the most.
template <int ID, int JD, int KD, int MODE, bool AL>
__global__ void __launch_bounds__(BX * BY, CGFD_LB_ALL) k_volume_all(const __grid_constant__ VolArgs a) {
  const int b = box_of_block(a);
  int i, j, k;
  if (!locate(a, b, i, j, k)) return;
  switch (a.box[b].kind) {
    case INTERIOR: volume_point<ID, JD, KD, MODE, INTERIOR, AL>(a, i, j, k); break;
    case FACE_X: volume_point<ID, JD, KD, MODE, FACE_X, AL>(a, i, j, k); break;
    case FACE_Y: volume_point<ID, JD, KD, MODE, FACE_Y, AL>(a, i, j, k); break;
    case FACE_Z: volume_point<ID, JD, KD, MODE, FACE_Z, AL>(a, i, j, k); break;
    case EDGE: volume_point<ID, JD, KD, MODE, EDGE, AL>(a, i, j, k); break;
    case TOP: volume_point<ID, JD, KD, MODE, TOP, AL>(a, i, j, k); break;
    default: volume_point<ID, JD, KD, MODE, SHELL, AL>(a, i, j, k); break;
  }
}

template <int ID, int JD, int KD, bool AL>
void launch_all(const VolArgs &a, int mode, cudaStream_t st) {
  const dim3 blk(BX, BY, 1);
  if (mode == RK_FIRST) k_volume_all<ID, JD, KD, RK_FIRST, AL><<<a.nblocks, blk, 0, st>>>(a);
  else if (mode == RK_SECOND) k_volume_all<ID, JD, KD, RK_SECOND, AL><<<a.nblocks, blk, 0, st>>>(a);
  else if (mode == RK_THIRD) k_volume_all<ID, JD, KD, RK_THIRD, AL><<<a.nblocks, blk, 0, st>>>(a);
  else k_volume_all<ID, JD, KD, RK_LAST, AL><<<a.nblocks, blk, 0, st>>>(a);
}

template <int ID, int JD, int KD, int KIND, bool AL>
void launch4(const VolArgs &a, int mode, cudaStream_t st) {
  if (a.nbox == 0) return;
  const dim3 blk(BX, BY, 1);
  dim3 grd(a.nblocks);
  if (KIND == INTERIOR) {
    const VolBox &B = a.box[0];
    const int nchunks = (B.nby + a.ychunk - 1) / a.ychunk;
    grd = dim3(B.nbx, a.ychunk, (B.k1 - B.k0 + 1) * nchunks);
  }
  if (mode == RK_FIRST) k_volume<ID, JD, KD, RK_FIRST, KIND, AL><<<grd, blk, 0, st>>>(a);
  else if (mode == RK_SECOND) k_volume<ID, JD, KD, RK_SECOND, KIND, AL><<<grd, blk, 0, st>>>(a);
  else if (mode == RK_THIRD) k_volume<ID, JD, KD, RK_THIRD, KIND, AL><<<grd, blk, 0, st>>>(a);
  else k_volume<ID, JD, KD, RK_LAST, KIND, AL><<<grd, blk, 0, st>>>(a);
}

template <int KIND, bool AL>
void launch_dirs(const VolArgs &a, int idir, int jdir, int kdir, int mode, cudaStream_t st) {
  switch (idir * 4 + jdir * 2 + kdir) {
    case 0: launch4<0, 0, 0, KIND, AL>(a, mode, st); break;
    case 1: launch4<0, 0, 1, KIND, AL>(a, mode, st); break;
    case 2: launch4<0, 1, 0, KIND, AL>(a, mode, st); break;
    case 3: launch4<0, 1, 1, KIND, AL>(a, mode, st); break;
    case 4: launch4<1, 0, 0, KIND, AL>(a, mode, st); break;
    case 5: launch4<1, 0, 1, KIND, AL>(a, mode, st); break;
    case 6: launch4<1, 1, 0, KIND, AL>(a, mode, st); break;
    default: launch4<1, 1, 1, KIND, AL>(a, mode, st); break;
  }
}
// Aligned grids take the kernels without the four off-axis metric entries:
// 32 bytes of metric and medium per point and stage instead of 48, 12 metric
// products fewer per direction x and y.  Step, general -> aligned: 300x600x240
// 7.69 -> 7.55 ms, 200x300x160 2.07 -> 1.98, 100x160x80 421 -> 408 us, 101x163x77
// 394 -> 384, sponge 120x180x90 362 -> 353.
template <int KIND>
void launch_kind(const VolArgs &a, int idir, int jdir, int kdir, int mode, cudaStream_t st) {
#ifndef CGFD_FP64
  if (a.g.al) return launch_dirs<KIND, true>(a, idir, jdir, kdir, mode, st);
#endif
  launch_dirs<KIND, false>(a, idir, jdir, kdir, mode, st);
}

}  // namespace

// This file is compiled once per kernel kind (CGFD_VOLUME_KIND = 0..7, set
// by the build) so that the 64 instantiations of each kind (32 in the double
// build, which has no aligned ones) build in parallel, and once per operator
// triple for the kernels that hold every kind (8..15); unit 0 also holds the
// host helpers.
#ifndef CGFD_VOLUME_KIND
#define CGFD_VOLUME_KIND 0
#endif

#if CGFD_VOLUME_KIND == 0
// append n boxes (interior indices, inclusive) of one kind to a launch's
// list; with pack, boxes at most 24 points wide are packed (nbx = 0); the
// interior kernel's 3-D grid needs the tiled layout (pack = false).  False
// when the list is full.
bool volume_boxes(VolArgs &a, int kind, const int (*boxes)[6], int n, bool pack) {
  for (int q = 0; q < n; q++) {
    const int *b = boxes[q];
    if (b[1] < b[0] || b[3] < b[2] || b[5] < b[4]) continue;
    if (a.nbox >= kMaxBoxes) return false;
    VolBox &B = a.box[a.nbox++];
    B.i0 = b[0]; B.i1 = b[1]; B.j0 = b[2]; B.j1 = b[3]; B.k0 = b[4]; B.k1 = b[5];
    B.kind = kind;
    B.first = a.nblocks;
    const int ni = b[1] - b[0] + 1, nj = b[3] - b[2] + 1, nk = b[5] - b[4] + 1;
    if (pack && ni <= 24) {
      B.nbx = 0;
      B.nby = (ni * nj + BX * BY - 1) / (BX * BY);
      a.nblocks += B.nby * nk;
    } else {
      B.nbx = (ni + BX - 1) / BX;
      B.nby = (nj + BY - 1) / BY;
      a.nblocks += B.nbx * B.nby * nk;
    }
  }
  return true;
}

void launch_volume_all(const VolArgs &a, int idir, int jdir, int kdir, int mode, cudaStream_t st) {
  if (a.nbox == 0) return;
  switch (idir * 4 + jdir * 2 + kdir) {
    case 0: launch_volume_all_n<0>(a, mode, st); break;
    case 1: launch_volume_all_n<1>(a, mode, st); break;
    case 2: launch_volume_all_n<2>(a, mode, st); break;
    case 3: launch_volume_all_n<3>(a, mode, st); break;
    case 4: launch_volume_all_n<4>(a, mode, st); break;
    case 5: launch_volume_all_n<5>(a, mode, st); break;
    case 6: launch_volume_all_n<6>(a, mode, st); break;
    default: launch_volume_all_n<7>(a, mode, st); break;
  }
}

void launch_volume_interior(const VolArgs &a, int idir, int jdir, int kdir, int mode, cudaStream_t st) {
  launch_kind<INTERIOR>(a, idir, jdir, kdir, mode, st);
}
// the first group of an aligned grid, (xi_x eta_y lambda mu), of every point
// from the general rows 0 and 1
__global__ void __launch_bounds__(256) k_align(const real4 *__restrict__ rows, real4 *__restrict__ out, long sc) {
  const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= sc) return;
  const real4 r0 = rows[p], r1 = rows[sc + p];
  out[p] = make_real4(r0.x, r1.y, r0.w, r1.w);
}
void launch_align(const real *rows, real *out, long sc, cudaStream_t st) {
  k_align<<<(unsigned)((sc + 255) / 256), 256, 0, st>>>(reinterpret_cast<const real4 *>(rows), reinterpret_cast<real4 *>(out), sc);
}
#elif CGFD_VOLUME_KIND == 1
void launch_volume_shell(const VolArgs &a, int idir, int jdir, int kdir, int mode, cudaStream_t st) {
  launch_kind<SHELL>(a, idir, jdir, kdir, mode, st);
}
#elif CGFD_VOLUME_KIND == 2
void launch_volume_face_x(const VolArgs &a, int idir, int jdir, int kdir, int mode, cudaStream_t st) {
  launch_kind<FACE_X>(a, idir, jdir, kdir, mode, st);
}
#elif CGFD_VOLUME_KIND == 3
void launch_volume_face_y(const VolArgs &a, int idir, int jdir, int kdir, int mode, cudaStream_t st) {
  launch_kind<FACE_Y>(a, idir, jdir, kdir, mode, st);
}
#elif CGFD_VOLUME_KIND == 4
void launch_volume_face_z(const VolArgs &a, int idir, int jdir, int kdir, int mode, cudaStream_t st) {
  launch_kind<FACE_Z>(a, idir, jdir, kdir, mode, st);
}
#elif CGFD_VOLUME_KIND == 5
void launch_volume_edge(const VolArgs &a, int idir, int jdir, int kdir, int mode, cudaStream_t st) {
  launch_kind<EDGE>(a, idir, jdir, kdir, mode, st);
}
#elif CGFD_VOLUME_KIND == 6
void launch_volume_plane(const VolArgs &a, int idir, int jdir, int kdir, int mode, cudaStream_t st) {
  launch_kind<PLANE>(a, idir, jdir, kdir, mode, st);
}
#elif CGFD_VOLUME_KIND == 7
void launch_volume_top(const VolArgs &a, int idir, int jdir, int kdir, int mode, cudaStream_t st) {
  launch_kind<TOP>(a, idir, jdir, kdir, mode, st);
}
#else
template <>
void launch_volume_all_n<CGFD_VOLUME_KIND - 8>(const VolArgs &a, int mode, cudaStream_t st) {
  constexpr int N = CGFD_VOLUME_KIND - 8;
#ifndef CGFD_FP64
  if (a.g.al) return launch_all<N / 4, N / 2 % 2, N % 2, true>(a, mode, st);
#endif
  launch_all<N / 4, N / 2 % 2, N % 2, false>(a, mode, st);
}
#endif

}  // namespace cgfd
