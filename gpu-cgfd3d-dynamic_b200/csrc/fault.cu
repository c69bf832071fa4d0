// fault.cu -- split-node fault kernels.
//
// Per RK stage the reference launches, per fault, wave2fault, the trial
// traction + slip-weakening friction kernel, fault2wave, the fault velocity
// RHS, the fault stress RHS (forward or backward variant), two fault RK
// updates, fault2wave again and the stage traction update, each as its own
// kernel (src/forward/drv_rk_curv_col.cu:277-588).  Here that becomes three
// kernels over the fault plane:
//
//   k_fault_pre     welded nodes: fault wavefield from the volume at i0
//                   (wave2fault_gpu, src/forward/transform.cu:101-212);
//                   tractions J e . sigma of the stage input at the volume
//                   points i0-6..i0+6 around the split box, once each, into a
//                   per-fault scratch array read by the next two kernels
//   k_fault_split   split nodes, six threads each, in one pass:
//                   T1 traction image, trial traction and linear
//                   slip-weakening friction (trial_slipweakening_gpu,
//                   src/forward/trial_slipweakening.cu:92-388), stage
//                   traction output (fault_var_stage_update_gpu,
//                   fault_wav_t.cu:291-316), split-node velocity RHS
//                   (sv_curv_col_el_iso_fault_gpu.cu:323-429) and its RK
//                   update; then the velocity gradients of both sides and the
//                   fault traction rates with their RK update (..._stress_F_gpu
//                   :432-1159 / _B_gpu :1162-1879, split nodes), the
//                   split-node volume point of the output level from the
//                   fault fields (fault2wave_gpu, transform.cu:293-376) and,
//                   after the last stage, slip / slip rate / rupture time
//                   (fault_var_update_gpu, fault_wav_t.cu:198-264)
//   k_fault_slab    the volume points i0-3..i0+3 (not i0), one thread each:
//                   velocity RHS with the traction image through the fault
//                   (sv_curv_col_el_iso_rhs_fault_velo_gpu,
//                   src/forward/sv_curv_col_el_iso_fault_gpu.cu:192-322),
//                   stress RHS with the fault's one-sided operators
//                   (..._stress_F_gpu / _B_gpu, volume points) and the RK
//                   update of all nine components in whole 16-byte groups
//
// The volume stage kernel skips i0-3..i0+3 of split nodes, so these kernels
// own those points' RK update.  The slab and traction kernels give each
// (node, x offset) its own thread with the x offset fastest: the fault plane
// is a constant-x plane, so a warp over nodes alone would touch one cache
// line per thread on every volume access.
#include <cuda_runtime.h>

#include "ops.cuh"

namespace cgfd {

namespace {

__device__ __forceinline__ long fidx(int c, int m, long ns, long nd) { return ((long)c * 2 + m) * ns + nd; }

// J * (e_d . sigma) at point q, 3 components (d: 0 xi, 1 eta, 2 zeta)
__device__ __forceinline__ void trac3(const Grid &g, const real *__restrict__ w, const real *__restrict__ cf,
                                      long q, int d, real t[3]) {
  const long sc = g.scmp;
  const real J = coef_jac(cf, q);
  const real4 e = coef_row(g, cf, d, q);
  const real ex = e.x, ey = e.y, ez = e.z;
  // Txx ends the first 16-byte group, Tyy Tzz Tyz Txz are the second
  const real sxx = __ldg(w + g.w(TXX, q));
  const real4 s4 = __ldg(reinterpret_cast<const real4 *>(w + 4 * sc) + q);
  const real syy = s4.x, szz = s4.y, syz = s4.z, sxz = s4.w, sxy = __ldg(w + g.w(TXY, q));
  t[0] = J * (ex * sxx + ey * sxy + ez * sxz);
  t[1] = J * (ex * sxy + ey * syy + ez * syz);
  t[2] = J * (ex * sxz + ey * syz + ez * szz);
}

// odd extension of a 7-point line about its entry nf (3..6, the free
// surface): v[nf] = 0 and v[nf + l] = -v[nf - l] beyond it.  Fixed indices
// in every case keep the line in registers.
__device__ __forceinline__ void odd_image(real v[7], int nf) {
  switch (nf) {
    case 3: v[3] = 0.f; v[4] = -v[2]; v[5] = -v[1]; v[6] = -v[0]; break;
    case 4: v[4] = 0.f; v[5] = -v[3]; v[6] = -v[2]; break;
    case 5: v[5] = 0.f; v[6] = -v[4]; break;
    default: v[6] = 0.f; break;
  }
}

// RK stage update (see RK_FIRST in ops.cuh) of one value: u0 the time-n
// level's (in the last stage V), cur the stage input's, h its rate; returns
// the value written to the next stage's input (in the last stage time n+1)
__device__ __forceinline__ real rk_put(int mode, real ca, real cb, real u0, real cur, real h, real *out, real *end) {
  if (mode == RK_LAST) {
    const real r = rk_end(u0, cur, cb * h);
    *end = r;
    return r;
  }
  const real r = rk_out(mode == RK_FIRST ? cur : u0, ca * h);
  *out = r;
  if (mode == RK_SECOND) *end = rk_v(u0, cur, ca * h);
  return r;
}

// Programmatic dependent launch: a kernel launched with launch_after() may
// start before the one ahead of it in its stream has ended (in an ordinary
// launch both instructions do nothing).  after_previous()
// waits for that one's end (and its writes), let_next_start() lets the next
// one's blocks in.  The split-node kernel reads its node's own values while
// the first fault kernel runs, the slab kernel forms its stress right-hand
// sides (which need nothing of the split kernel) beside the split kernel.
// Step: two faults 44x64x32 173 -> 165 us (direct launches 205 -> 177),
// 60x120x64 243 -> 235, 100x160x80 404 -> 392, 300x600x240 the same.
__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// The operators of ops.cuh by plain loads, for what the kernel ahead writes:
// the compiler may move a read-only (non-coherent) load above the wait for it
__device__ __forceinline__ real drp_co(const real *p, long s, int f) {
  if (!f) s = -s;
  const real t = kC1 * p[-s] + kC2 * p[0] + kC3 * p[s] + kC4 * p[2 * s] + kC5 * p[3 * s];
  return f ? t : -t;
}
__device__ __forceinline__ real mac22_co(const real *p, long s, int f) { return f ? p[s] - p[0] : p[0] - p[-s]; }
__device__ __forceinline__ real mac24_co(const real *p, long s, int f) {
  if (!f) s = -s;
  const real t = kB1 * p[0] + kB2 * p[s] + kB3 * p[2 * s];
  return f ? t : -t;
}

// slot of x offset d (-6..-1, 1..6) in the traction scratch
__device__ __forceinline__ int trac_slot(int d) { return d < 0 ? d + 6 : d + 5; }

// split-node volume point from the fault fields (fault2wave_gpu,
// transform.cu:293-376): velocity = mean of the two sides, stress from the
// traction vectors [T1 | mean T2 | mean T3] through the inverse metric.
// V, T2, T3: the node's values of one component and side, [3 side + component]
// entries `st` apart.
__device__ __forceinline__ void split_to_volume(const Grid &g, const real *__restrict__ cf, int i0, int J, int K,
                                                const real *V, const real *T2, const real *T3, int st, const real T1[3],
                                                real *wt) {
  const long sc = g.scmp;
  const long p0 = g.at(i0, J, K);
  real mt[3][3];   // columns e_xi, e_eta, e_zeta
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const real4 e = coef_row(g, cf, c, p0);
    mt[0][c] = e.x; mt[1][c] = e.y; mt[2][c] = e.z;
  }
  const real rj = 1.0f / coef_jac(cf, p0);
  real tr[3][3];
#pragma unroll
  for (int r = 0; r < 3; r++) {
    tr[r][0] = T1[r];
    tr[r][1] = (T2[r * st] + T2[(3 + r) * st]) * 0.5f;
    tr[r][2] = (T3[r * st] + T3[(3 + r) * st]) * 0.5f;
  }
  const real c00 = mt[1][1] * mt[2][2] - mt[2][1] * mt[1][2], c01 = mt[2][1] * mt[0][2] - mt[0][1] * mt[2][2];
  const real c02 = mt[0][1] * mt[1][2] - mt[0][2] * mt[1][1], c10 = mt[1][2] * mt[2][0] - mt[1][0] * mt[2][2];
  const real c11 = mt[0][0] * mt[2][2] - mt[2][0] * mt[0][2], c12 = mt[1][0] * mt[0][2] - mt[0][0] * mt[1][2];
  const real c20 = mt[1][0] * mt[2][1] - mt[1][1] * mt[2][0], c21 = mt[2][0] * mt[0][1] - mt[0][0] * mt[2][1];
  const real c22 = mt[0][0] * mt[1][1] - mt[0][1] * mt[1][0];
  const real id = 1.0f / (c00 * mt[0][0] + c01 * mt[1][0] + c02 * mt[2][0]);
  const real mi[3][3] = { { c00 * id, c01 * id, c02 * id }, { c10 * id, c11 * id, c12 * id }, { c20 * id, c21 * id, c22 * id } };
  real sg[3][3];
#pragma unroll
  for (int r = 0; r < 3; r++)
#pragma unroll
    for (int c = 0; c < 3; c++) sg[r][c] = (tr[r][0] * mi[0][c] + tr[r][1] * mi[1][c] + tr[r][2] * mi[2][c]) * rj;
  real u[3];
#pragma unroll
  for (int c = 0; c < 3; c++) u[c] = (V[c * st] + V[(3 + c) * st]) * 0.5f;
  reinterpret_cast<real4 *>(wt)[p0] = make_real4(u[0], u[1], u[2], sg[0][0]);
  // the reference's fault2wave_gpu receives Tyz and Txz in swapped
  // positions (transform.cu:281-289 vs :293-300); kept for parity
  reinterpret_cast<real4 *>(wt + 4 * sc)[p0] =
      make_real4(sg[1][1], sg[2][2], (sg[0][2] + sg[2][0]) * 0.5f, (sg[1][2] + sg[2][1]) * 0.5f);
  wt[g.w(TXY, p0)] = (sg[0][1] + sg[1][0]) * 0.5f;
}

}  // namespace

// ---------------------------------------------------------------------------
// welded node t of the box wj0.., wk0..
__device__ __forceinline__ void weld_node(const FaultArgs &a, long t) {
  const Grid &g = a.g;
  if (t >= (long)a.wnj * a.wnk) return;
  const int k = a.wk0 + (int)(t / a.wnj), j = a.wj0 + (int)(t % a.wnj);
  const int J = j + NG, K = k + NG;
  const long ns = (long)g.ny * g.nz, nd = J + (long)K * g.ny;
  if (a.F.flag[nd] & FL_SPLIT) return;
  const long p = g.at(a.F.i0, J, K);
  const real *w = a.wcur;
  real t2[3], t3[3];
  trac3(g, w, a.coef, p, 1, t2);
  trac3(g, w, a.coef, p, 2, t3);
  real *f = const_cast<real *>(a.fc);
#pragma unroll
  for (int m = 0; m < 2; m++) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      f[fidx(FVX + c, m, ns, nd)] = w[g.w(VX + c, p)];
      f[fidx(FT2X + c, m, ns, nd)] = t2[c];
      f[fidx(FT3X + c, m, ns, nd)] = t3[c];
    }
  }
}

// ---------------------------------------------------------------------------
// tractions of the stage input around the split box, one thread per
// (node, x offset), x offset fastest so that a warp reads contiguous x runs:
// T1 = J e_xi . sigma at x = i0+-1..6, T2 = J e_eta . sigma and
// T3 = J e_zeta . sigma at x = i0+-1..3.  The trial, friction and slab
// velocity kernels read them from here instead of recomputing each one
// (10 loads) for every tap.  Layout [9][tnk][tnj][12], x offset fastest.
__device__ __forceinline__ void trac_item(const FaultArgs &a, long t) {
  const Grid &g = a.g;
  const long node = t / 12;
  if (node >= (long)a.tnj * a.tnk) return;
  const int slot = (int)(t - node * 12);
  const int d = slot < 6 ? slot - 6 : slot - 5;
  const int kk = (int)(node / a.tnj), jj = (int)(node - (long)kk * a.tnj);
  const long pl = (long)a.tnj * a.tnk * 12;
  const long q = g.at(a.F.i0 + d, a.tj0 + jj, a.tk0 + kk);
  real *tp = a.trac + node * 12 + slot;
  real v[3];
  trac3(g, a.wcur, a.coef, q, 0, v);
  tp[0] = v[0]; tp[pl] = v[1]; tp[2 * pl] = v[2];
  if (d >= -3 && d <= 3) {
    trac3(g, a.wcur, a.coef, q, 1, v);
    tp[3 * pl] = v[0]; tp[4 * pl] = v[1]; tp[5 * pl] = v[2];
    trac3(g, a.wcur, a.coef, q, 2, v);
    tp[6 * pl] = v[0]; tp[7 * pl] = v[1]; tp[8 * pl] = v[2];
  }
}

// x offset from the fault of slab slot y = 0..5: -3, -2, -1, 1, 2, 3
__device__ __forceinline__ int slab_offset(int y) { return y < 3 ? y - 3 : y - 2; }

// slab work item t over the split box, six per node with the x offset
// fastest (a warp reads runs of contiguous x): node (j, k), offset s
__device__ __forceinline__ bool slab_item(const FaultArgs &a, long t, int &j, int &k, int &s) {
  const long node = t / 6;
  if (node >= (long)a.nj * a.nk) return false;
  const int r = (int)(t - node * 6);
  k = a.k0 + (int)(node / a.nj);
  j = a.j0 + (int)(node - (long)(k - a.k0) * a.nj);
  s = slab_offset(r);
  return true;
}

// ---------------------------------------------------------------------------
// velocity RHS at the six volume points i0-3..i0+3 (not i0) of split nodes,
// one thread per point, one warp per (slab offset, row of 32 nodes)
// (sv_curv_col_el_iso_rhs_fault_velo_gpu, :192-322)
__device__ __forceinline__ void slab_velocity(const FaultArgs &a, int j, int k, int s, real hv3[3]) {
  const Grid &g = a.g;
  const int J = j + NG, K = k + NG;
  const long ns = (long)g.ny * g.nz, nd = J + (long)K * g.ny;
  const FaultDev &F = a.F;
  const int i0 = F.i0;
  const int km = g.nk - (k + 1);
  const bool surf = a.isfree && km <= 3;
  const int nf = km + 3;
  const long q = g.at(i0 + s, J, K);
  const long pl = (long)a.tnj * a.tnk * 12, row = (long)a.tnj * 12;
  const real *tr = a.trac + ((long)(K - a.tk0) * a.tnj + (J - a.tj0)) * 12;

  // T1 along x through this point: this side's volume points, the split
  // node's T1 at the fault, and beyond it the odd extension through the
  // split node (traction image)
  real v1[7][3];
#pragma unroll
  for (int l = -3; l <= 3; l++) {
    const int x = s + l;
    if (x == 0) {
#pragma unroll
      for (int c = 0; c < 3; c++) v1[l + 3][c] = F.scal[(FS_T1X + c) * ns + nd];
    } else if ((x < 0) == (s < 0)) {
#pragma unroll
      for (int c = 0; c < 3; c++) v1[l + 3][c] = tr[c * pl + trac_slot(x)];
    } else {
#pragma unroll
      for (int c = 0; c < 3; c++) v1[l + 3][c] = 0.f;
    }
  }
  real hv[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    real v[7];
#pragma unroll
    for (int l = 0; l < 7; l++) v[l] = v1[l][c];
    if (s == -2) { v[6] = 2.f * v[5] - v[4]; }
    if (s == -1) { v[5] = 2.f * v[4] - v[3]; v[6] = 2.f * v[4] - v[2]; }
    if (s == 1) { v[0] = 2.f * v[2] - v[4]; v[1] = 2.f * v[2] - v[3]; }
    if (s == 2) { v[0] = 2.f * v[1] - v[2]; }
    hv[c] = drp_v(v + 3, a.idir);
  }

  // y and z lines of T2 = J e_eta . sigma and T3 = J e_zeta . sigma
  const real *t2 = tr + 3 * pl + trac_slot(s), *t3 = t2 + 3 * pl;
  const real rr = coef_row(g, a.coef, 2, q).w / coef_jac(a.coef, q);
#pragma unroll
  for (int c = 0; c < 3; c++) {
    real y[7], z[7];
#pragma unroll
    for (int l = 0; l < 7; l++) {
      y[l] = t2[c * pl + (l - 3) * 12];
      z[l] = t3[c * pl + (l - 3) * row];
    }
    if (surf) {
      odd_image(z, nf);
    }
    hv3[c] = (hv[c] + drp_v(y + 3, a.jdir) + drp_v(z + 3, a.kdir)) * rr;
  }
}

// component c (0 x, 1 y, 2 z) of a 16-byte group
__device__ __forceinline__ real cmp3(const real4 &v, int c) { return c == 0 ? v.x : (c == 1 ? v.y : v.z); }

// drp, mac24 and mac22 (same weights, same order of the sums) of the three
// velocity components along stride st (in groups) from whole 16-byte groups
// (Vx Vy Vz Txx) of one level, direction f
__device__ __forceinline__ void vel_drp(const real4 *__restrict__ p, long st, int f, real o[3]) {
  if (f) {
    const real4 a = __ldg(p - st), b = __ldg(p), c = __ldg(p + st), d = __ldg(p + 2 * st), e = __ldg(p + 3 * st);
#pragma unroll
    for (int n = 0; n < 3; n++)
      o[n] = kC1 * cmp3(a, n) + kC2 * cmp3(b, n) + kC3 * cmp3(c, n) + kC4 * cmp3(d, n) + kC5 * cmp3(e, n);
  } else {
    const real4 a = __ldg(p + st), b = __ldg(p), c = __ldg(p - st), d = __ldg(p - 2 * st), e = __ldg(p - 3 * st);
#pragma unroll
    for (int n = 0; n < 3; n++)
      o[n] = -(kC1 * cmp3(a, n) + kC2 * cmp3(b, n) + kC3 * cmp3(c, n) + kC4 * cmp3(d, n) + kC5 * cmp3(e, n));
  }
}
__device__ __forceinline__ void vel_mac24(const real4 *__restrict__ p, long st, int f, real o[3]) {
  const real4 b = __ldg(p), c = __ldg(f ? p + st : p - st), d = __ldg(f ? p + 2 * st : p - 2 * st);
#pragma unroll
  for (int n = 0; n < 3; n++) {
    const real t = kB1 * cmp3(b, n) + kB2 * cmp3(c, n) + kB3 * cmp3(d, n);
    o[n] = f ? t : -t;
  }
}
__device__ __forceinline__ void vel_mac22(const real4 *__restrict__ p, long st, int f, real o[3]) {
  const real4 b = __ldg(p), c = __ldg(f ? p + st : p - st);
#pragma unroll
  for (int n = 0; n < 3; n++) o[n] = f ? cmp3(c, n) - cmp3(b, n) : cmp3(b, n) - cmp3(c, n);
}

// ---------------------------------------------------------------------------
// stress RHS and RK update at the six volume points i0-3..i0+3 (not i0) of
// split nodes, one thread per point, x offset fastest
// (sv_curv_col_el_iso_rhs_fault_stress_F_gpu :432-1159 / _B_gpu :1162-1879,
// volume points)
__device__ __forceinline__ void slab_stress(const FaultArgs &a, int j, int k, int s, real h[6]) {
  const Grid &g = a.g;
  const int J = j + NG, K = k + NG;
  const long ns = (long)g.ny * g.nz, nd = J + (long)K * g.ny;
  const int i0 = a.F.i0;
  const real *w = a.wcur;
  const int km = g.nk - (k + 1);
  const bool fwd = a.idir == 1;
  const bool top = a.isfree && km == 0;
  // fault velocity of this side, input level
  real fV[3];
  const int m = s < 0 ? 0 : 1;
#pragma unroll
  for (int c = 0; c < 3; c++) fV[c] = a.fc[fidx(FVX + c, m, ns, nd)];
  const long q = g.at(i0 + s, J, K);
  // the velocity taps as whole 16-byte groups (Vx Vy Vz Txx): one load per
  // tap for all three components
  const real4 *V = reinterpret_cast<const real4 *>(w) + q;
  const real4 v0 = __ldg(V);
  real dx[3], dy[3], dz[3];
  if (fwd) {
    // forward operators; points left of the fault see the minus side
    if (s == 3) vel_drp(V, 1, 1, dx);
    else if (s == 2) vel_mac24(V, 1, 1, dx);
    else if (s == 1) vel_mac22(V, 1, 1, dx);
    else if (s == -1) {
#pragma unroll
      for (int c = 0; c < 3; c++) dx[c] = fV[c] - cmp3(v0, c);
    } else if (s == -2) {
      const real4 v1 = __ldg(V + 1);
#pragma unroll
      for (int c = 0; c < 3; c++) dx[c] = kB1 * cmp3(v0, c) + kB2 * cmp3(v1, c) + kB3 * fV[c];
    } else {
      const real4 vm = __ldg(V - 1), v1 = __ldg(V + 1), v2 = __ldg(V + 2);
#pragma unroll
      for (int c = 0; c < 3; c++)
        dx[c] = kC1 * cmp3(vm, c) + kC2 * cmp3(v0, c) + kC3 * cmp3(v1, c) + kC4 * cmp3(v2, c) + kC5 * fV[c];
    }
  } else {
    if (s == -3) vel_drp(V, 1, 0, dx);
    else if (s == -2) vel_mac24(V, 1, 0, dx);
    else if (s == -1) vel_mac22(V, 1, 0, dx);
    else if (s == 1) {
#pragma unroll
      for (int c = 0; c < 3; c++) dx[c] = cmp3(v0, c) - fV[c];
    } else if (s == 2) {
      const real4 vm = __ldg(V - 1);
#pragma unroll
      for (int c = 0; c < 3; c++) dx[c] = -(kB3 * fV[c] + kB2 * cmp3(vm, c) + kB1 * cmp3(v0, c));
    } else {
      const real4 vm2 = __ldg(V - 2), vm = __ldg(V - 1), v1 = __ldg(V + 1);
#pragma unroll
      for (int c = 0; c < 3; c++)
        dx[c] = -(kC5 * fV[c] + kC4 * cmp3(vm2, c) + kC3 * cmp3(vm, c) + kC2 * cmp3(v0, c) + kC1 * cmp3(v1, c));
    }
  }
  vel_drp(V, g.sy, a.jdir, dy);
  if (a.isfree && km == 1) vel_mac22(V, g.sz, a.kdir, dz);
  else if (a.isfree && km == 2) vel_mac24(V, g.sz, a.kdir, dz);
  else vel_drp(V, g.sz, a.kdir, dz);
  if (top) {
    const real *X = a.free_mat + ((long)J * g.nx + (i0 + s)) * 9;
    const real *Y = X + (long)g.ny * g.nx * 9;
    real o1[3], o2[3];
    mv3(X, dx, o1); mv3(Y, dy, o2);
#pragma unroll
    for (int c = 0; c < 3; c++) dz[c] = o1[c] + o2[c];
  }
  const real4 r0 = coef_row(g, a.coef, 0, q), r1 = coef_row(g, a.coef, 1, q), r2 = coef_row(g, a.coef, 2, q);
  const real e[3][3] = { { r0.x, r0.y, r0.z }, { r1.x, r1.y, r1.z }, { r2.x, r2.y, r2.z } };
  const real lam = r0.w, mu = r1.w;
  const real l2m = lam + 2.0f * mu;
  real G[3][3];
#pragma unroll
  for (int b = 0; b < 3; b++)
#pragma unroll
    for (int c = 0; c < 3; c++) G[c][b] = e[0][b] * dx[c] + e[1][b] * dy[c] + e[2][b] * dz[c];
  h[0] = l2m * G[0][0] + lam * (G[1][1] + G[2][2]);
  h[1] = l2m * G[1][1] + lam * (G[0][0] + G[2][2]);
  h[2] = l2m * G[2][2] + lam * (G[0][0] + G[1][1]);
  h[3] = mu * (G[1][2] + G[2][1]);   // Tyz
  h[4] = mu * (G[0][2] + G[2][0]);   // Txz
  h[5] = mu * (G[0][1] + G[1][0]);   // Txy
}

// ---------------------------------------------------------------------------
// row c of a 3x3 matrix times a vector held in shared memory, entries `st`
// apart
__device__ __forceinline__ real row3(const real *__restrict__ m, int c, const real *v, int st) {
  return __ldg(m + 3 * c) * v[0] + __ldg(m + 3 * c + 1) * v[st] + __ldg(m + 3 * c + 2) * v[2 * st];
}

// split nodes: trial traction and linear slip-weakening friction
// (trial_slipweakening_gpu), the stage traction output, the refresh of the
// stage input's split-node volume point, the split-node velocity RHS with
// its RK update; velocity gradients of both sides (continuity matrices or
// traction rate, free-surface rows), fault traction rates and their RK
// update, the split-node volume point of the output level, and after the
// last stage slip / slip rate / rupture time
// (sv_curv_col_el_iso_rhs_fault_stress_F_gpu :432-1159 / _B_gpu :1162-1879,
// split nodes; fault2wave_gpu; fault_var_update_gpu).
//
// A block is 32 nodes of one row by six warps, one per side and component:
// a lane holds one of the node's six velocities, T2 and T3, and the warps
// meet through shared memory where a component needs the others (the
// friction law, which every warp evaluates for itself, and the 3x3
// matrices, of which each warp reads its row).  The kernel is bound by the
// latency of its dependent loads: with one thread per node, 154 registers and
// a chain of a hundred loads, a launch of 3200 nodes took 26.9 us on 25 of
// the 148 SMs.
__global__ void __launch_bounds__(192) k_fault_split(const FaultArgs a) {
  enum { S_R = 0, S_VP, S_V, S_T2, S_T3, S_SY, S_SZ, S_SX, S_NV, S_N2, S_N3, S_N };
  __shared__ real sh[S_N][6][32];
  const Grid &g = a.g;
  const FaultDev &F = a.F;
  const int tx = threadIdx.x, q = threadIdx.y, m = q / 3, c = q - 3 * m;
  const int j = a.j0 + blockIdx.x * 32 + tx, k = a.k0 + blockIdx.y;
  const int J = j + NG, K = k + NG;
  const long ns = (long)g.ny * g.nz, nd = J + (long)K * g.ny, ny = g.ny;
  const uint8_t fl = j < a.j0 + a.nj ? F.flag[nd] : 0;
  const bool act = fl & FL_SPLIT;
  const int i0 = F.i0, mode = a.mode;
  const int km = g.nk - (k + 1);
  const bool fwd = a.idir == 1, top = a.isfree && km == 0;
  const long p0 = g.at(i0, J, K);
  const real *cf = a.coef;
  // entries of this node: side and component e / of side s, component 0 (the
  // components follow 32 apart)
  auto S = [&](int n, int e) -> real & { return sh[n][e][tx]; };
  const int sg = 2 * m - 1;
  real x1 = 0.f, x2 = 0.f, x3 = 0.f, dy2 = 0.f, dz3 = 0.f;
  real jac0 = 0.f, rho0 = 0.f, rho1 = 0.f, slip = 0.f, mus = 0.f, mud = 0.f, Dc = 1.f, C0 = 0.f;
  real T0[3] = { 0.f, 0.f, 0.f }, dt1[3] = { 0.f, 0.f, 0.f };
  real4 exi = make_real4(1.f, 0.f, 0.f, 0.f);
  const long oV = fidx(FVX + c, m, ns, nd), o2 = fidx(FT2X + c, m, ns, nd), o3 = fidx(FT3X + c, m, ns, nd);
  real uV = 0.f, u2 = 0.f, u3 = 0.f;       // what the RK updates start from
  real cV = 0.f, c2 = 0.f, c3 = 0.f;       // stage input
  if (act) {
    // what the friction law reads of this node
    jac0 = coef_jac(cf, p0);
    exi = coef_row(g, cf, 0, p0);
    rho0 = F.scal[FS_RHO0 * ns + nd]; rho1 = F.scal[FS_RHO1 * ns + nd];
    slip = F.out[CGFD_FAULT_SLIP * ns + nd];
    mus = F.scal[FS_MUS * ns + nd]; mud = F.scal[FS_MUD * ns + nd];
    Dc = F.scal[FS_DC * ns + nd]; C0 = F.scal[FS_C0 * ns + nd];
#pragma unroll
    for (int n = 0; n < 3; n++) T0[n] = F.scal[(FS_T0X + n) * ns + nd];
    if (a.imethod == 2 && (fl & FL_GRID)) {
#pragma unroll
      for (int n = 0; n < 3; n++) dt1[n] = F.scal[(FS_HT1X + n) * ns + nd];
    }
    if (mode != RK_FIRST) {
      const real *l = mode == RK_LAST ? a.fe : a.fp;
      uV = l[oV]; u2 = l[o2]; u3 = l[o3];
    }
  }
  // so far nothing that the stage's first fault kernel writes has been read
  after_previous();
  let_next_start();
  if (act) {
    // T1 = J e_xi . sigma at this side's i0+-1..3
    const long pl = (long)a.tnj * a.tnk * 12;
    const real *tr = a.trac + ((long)(K - a.tk0) * a.tnj + (J - a.tj0)) * 12 + c * pl;
    x1 = tr[trac_slot(sg)]; x2 = tr[trac_slot(2 * sg)]; x3 = tr[trac_slot(3 * sg)];
    // along-fault derivatives of the fault tractions and velocity
    const real *t2 = a.fc + o2, *t3 = a.fc + o3, *v = a.fc + oV;
    dy2 = (fl & FL_RUPY) ? mac22_co(t2, 1, a.jdir) : drp_co(t2, 1, a.jdir);
    if (a.isfree && km <= 3) {
      // traction image of T3 about the free surface
      real l[7];
#pragma unroll
      for (int n = 0; n < 7; n++) l[n] = t3[(long)(n - 3) * ny];
      odd_image(l, km + 3);
      dz3 = drp_v(l + 3, a.kdir);
    } else {
      dz3 = (fl & FL_RUPZ) ? mac22_co(t3, ny, a.kdir) : drp_co(t3, ny, a.kdir);
    }
    S(S_SY, q) = (fl & FL_RUPY) ? mac22_co(v, 1, a.jdir) : drp_co(v, 1, a.jdir);
    real dz;
    if (a.isfree && km == 1) dz = mac22_co(v, ny, a.kdir);
    else if (a.isfree && km == 2) dz = mac24_co(v, ny, a.kdir);
    else dz = (fl & FL_RUPZ) ? mac22_co(v, ny, a.kdir) : drp_co(v, ny, a.kdir);
    S(S_SZ, q) = dz;
    cV = *v; c2 = *t2; c3 = *t3;
    S(S_VP, q) = mode == RK_FIRST ? cV : (mode == RK_LAST ? a.fp[oV] : uV);
    S(S_V, q) = cV; S(S_T2, q) = c2; S(S_T3, q) = c3;
    const real img = kA1 * x1 + kA2 * x2 + kA3 * x3;
    S(S_R, q) = 0.5f * ((real)sg * img + (dy2 + dz3));
  }
  __syncthreads();

  real T1s[3] = { 0.f, 0.f, 0.f };
  if (act) {
    // trial traction from the velocity jump of time level n and friction
    const real M0 = 0.5f * jac0 * rho0, M1 = 0.5f * jac0 * rho1;
    real Tr[3];
#pragma unroll
    for (int n = 0; n < 3; n++) {
      const real dV = S(S_VP, 3 + n) - S(S_VP, n);
      Tr[n] = 2.0f * (M0 * M1 * dV / a.dt + M0 * S(S_R, 3 + n) - M1 * S(S_R, n)) / (kA0 * (M0 + M1));
    }
    real vn[3] = { exi.x, exi.y, exi.z };
    const real vn0 = sqrt(vn[0] * vn[0] + vn[1] * vn[1] + vn[2] * vn[2]);
    const real jacvec = jac0 * vn0;
    vn[0] /= vn0; vn[1] /= vn0; vn[2] /= vn0;
    real Tl[3];
#pragma unroll
    for (int n = 0; n < 3; n++) Tl[n] = Tr[n] / jacvec + T0[n];
    const real Tn0 = Tl[0] * vn[0] + Tl[1] * vn[1] + Tl[2] * vn[2];
    const real Ts[3] = { Tl[0] - vn[0] * Tn0, Tl[1] - vn[1] * Tn0, Tl[2] - vn[2] * Tn0 };
    const real Ts0 = sqrt(Ts[0] * Ts[0] + Ts[1] * Ts[1] + Ts[2] * Ts[2]);
    bool change = false;
    real Tau_n = Tn0;
    if (Tn0 >= 0.f) { Tau_n = 0.f; change = true; }     // the fault cannot open
    const real fr = slip <= Dc ? mus - (mus - mud) * slip / Dc : mud;
    const real Tau_c = -fr * Tau_n + C0;
    real Tau_s = Ts0;
    if (Ts0 >= Tau_c) { Tau_s = Tau_c; change = true; }
    real Tau[3];
    if (change) {
      const real r = fabs(Ts0) < RL(1e-1) ? 0.f : Tau_s / Ts0;
#pragma unroll
      for (int n = 0; n < 3; n++) { Tau[n] = Tau_n * vn[n] + r * Ts[n]; T1s[n] = (Tau[n] - T0[n]) * jacvec; }
    } else {
#pragma unroll
      for (int n = 0; n < 3; n++) { Tau[n] = Tl[n]; T1s[n] = Tr[n]; }
    }
    if (q == 0) {
#pragma unroll
      for (int n = 0; n < 3; n++) F.scal[(FS_T1X + n) * ns + nd] = T1s[n];
    } else if (q == 1) {
      // the stage input level sees the new split-node traction before the
      // volume kernel reads it (drv_rk_curv_col.cu:285, fault2wave on
      // w_cur); no fault kernel reads the volume at i0
      split_to_volume(g, cf, i0, J, K, &S(S_V, 0), &S(S_T2, 0), &S(S_T3, 0), 32, T1s, const_cast<real *>(a.wcur));
    } else if (q == 2) {
      const real s1[3] = { F.scal[FS_S1X * ns + nd], F.scal[FS_S1Y * ns + nd], F.scal[FS_S1Z * ns + nd] };
      const real s2[3] = { F.scal[FS_S2X * ns + nd], F.scal[FS_S2Y * ns + nd], F.scal[FS_S2Z * ns + nd] };
      const real t[3] = { Tau_n, Tau[0] * s1[0] + Tau[1] * s1[1] + Tau[2] * s1[2],
                          Tau[0] * s2[0] + Tau[1] * s2[1] + Tau[2] * s2[2] };
      // Tn, Ts1, Ts2 follow one another
      real o[3] = { 0.f, 0.f, 0.f };
      if (mode != RK_FIRST) {
#pragma unroll
        for (int n = 0; n < 3; n++) o[n] = F.out[(CGFD_FAULT_TN + n) * ns + nd];
      }
#pragma unroll
      for (int n = 0; n < 3; n++) F.out[(CGFD_FAULT_TN + n) * ns + nd] = mode == RK_FIRST ? a.rkb * t[n] : o[n] + a.rkb * t[n];
    }
    // split-node velocity RHS and RK update (the output levels only: the
    // velocity taps of this stage read the input level)
    const real rr = 1.0f / ((m ? rho1 : rho0) * jac0);
    const real T1c = c == 0 ? T1s[0] : (c == 1 ? T1s[1] : T1s[2]);
    const real dx = m == 0 ? (kA0 * T1c - kA1 * x1 - kA2 * x2 - kA3 * x3) : (-kA0 * T1c + kA1 * x1 + kA2 * x2 + kA3 * x3);
    S(S_NV, q) = rk_put(mode, a.ca, a.cb, uV, cV, (dx + dy2 + dz3) * rr, a.fo + oV, a.fe + oV);

    // normal velocity derivative of this side
    const int me = 3 * m, ot = 3 - me;
    real sx;
    if (a.imethod == 1 && m == (fwd ? 1 : 0)) {
      // its one-sided difference
      const real *w = a.wcur;
      sx = fwd ? w[g.w(VX + c, g.at(i0 + 1, J, K))] - cV : cV - w[g.w(VX + c, g.at(i0 - 1, J, K))];
    } else if (a.imethod == 1) {
      // continuity of the traction rate across the fault, from the other
      // side's one-sided difference
      const real4 w1 = __ldg(reinterpret_cast<const real4 *>(a.wcur) + g.at(fwd ? i0 + 1 : i0 - 1, J, K));
      const real wv[3] = { w1.x, w1.y, w1.z };
      real d[3];
#pragma unroll
      for (int n = 0; n < 3; n++) d[n] = fwd ? wv[n] - S(S_V, ot + n) : S(S_V, ot + n) - wv[n];
      if (!top) {
        auto M = [&](int id) { return F.mat + ((long)id * ns + nd) * 9; };
        const int b = fwd ? FM_P2M1 : FM_M2P1;
        sx = row3(M(b), c, d, 1) + row3(M(b + 1), c, &S(S_SY, ot), 32) + row3(M(b + 2), c, &S(S_SZ, ot), 32) -
             row3(M(b + 3), c, &S(S_SY, me), 32) - row3(M(b + 4), c, &S(S_SZ, me), 32);
      } else {
        auto FM = [&](int id) { return F.fmat + ((long)id * ny + J) * 9; };
        const int b = fwd ? FF_P2M1 : FF_M2P1;
        sx = row3(FM(b), c, d, 1) + row3(FM(b + 1), c, &S(S_SY, ot), 32) - row3(FM(b + 2), c, &S(S_SY, me), 32);
      }
    } else if (!top) {
      // from the traction rate
      auto M = [&](int id) { return F.mat + ((long)id * ns + nd) * 9; };
      const int b = m ? FM_T1VXPLUS : FM_T1VXMIN;
      sx = row3(M(b), c, dt1, 1) - row3(M(b + 1), c, &S(S_SY, me), 32) - row3(M(b + 2), c, &S(S_SZ, me), 32);
    } else {
      auto FM = [&](int id) { return F.fmat + ((long)id * ny + J) * 9; };
      const int b = m ? FF_T1VXPLUS : FF_T1VXMIN;
      sx = row3(FM(b), c, dt1, 1) - row3(FM(b + 1), c, &S(S_SY, me), 32);
    }
    S(S_SX, q) = sx;
  }
  __syncthreads();

  // fault traction rates and RK update of T2, T3
  if (act) {
    const int me = 3 * m;
    real z[3];
    if (top) {
      // split nodes on the free surface: traction-free top as well
      const real *A = F.fmat + ((long)(m ? FF_VX2VZ2 : FF_VX2VZ1) * ny + J) * 9, *B = A + ny * 9;
#pragma unroll
      for (int n = 0; n < 3; n++) z[n] = row3(A, n, &S(S_SX, me), 32) + row3(B, n, &S(S_SY, me), 32);
    } else {
#pragma unroll
      for (int n = 0; n < 3; n++) z[n] = S(S_SZ, me + n);
    }
    const real *D2 = F.mat + ((long)(m ? FM_D21_2 : FM_D21_1) * ns + nd) * 9, *D3 = D2 + 27 * ns;
    const real h2 = row3(D2, c, &S(S_SX, me), 32) + row3(D2 + 9 * ns, c, &S(S_SY, me), 32) + row3(D2 + 18 * ns, c, z, 1);
    const real h3 = row3(D3, c, &S(S_SX, me), 32) + row3(D3 + 9 * ns, c, &S(S_SY, me), 32) + row3(D3 + 18 * ns, c, z, 1);
    S(S_N2, q) = rk_put(mode, a.ca, a.cb, u2, c2, h2, a.fo + o2, a.fe + o2);
    S(S_N3, q) = rk_put(mode, a.ca, a.cb, u3, c3, h3, a.fo + o3, a.fe + o3);
  }
  __syncthreads();
  if (!act) return;

  if (q == 0) {
    // the split-node volume point of the output level
    split_to_volume(g, cf, i0, J, K, &S(S_NV, 0), &S(S_N2, 0), &S(S_N3, 0), 32, T1s, mode == RK_LAST ? a.wend : a.wout);
  } else if (mode == RK_LAST && q == 1) {
    // end of step: slip rate, slip, peak slip rate, rupture time
    real s1[3], s2[3], dV[3];
#pragma unroll
    for (int n = 0; n < 3; n++) {
      s1[n] = F.scal[(FS_S1X + n) * ns + nd];
      s2[n] = F.scal[(FS_S2X + n) * ns + nd];
      dV[n] = S(S_NV, 3 + n) - S(S_NV, n);
    }
    const real Vs1 = dV[0] * s1[0] + dV[1] * s1[1] + dV[2] * s1[2];
    const real Vs2 = dV[0] * s2[0] + dV[1] * s2[1] + dV[2] * s2[2];
    const real Vs = sqrt(Vs2 * Vs2 + Vs1 * Vs1);
    real *o = F.out;
    const real l0 = slip, l1 = o[CGFD_FAULT_SLIP1 * ns + nd], l2 = o[CGFD_FAULT_SLIP2 * ns + nd];
    const real pk = o[CGFD_FAULT_PEAK_VS * ns + nd];
    o[CGFD_FAULT_VS * ns + nd] = Vs;
    o[CGFD_FAULT_VS1 * ns + nd] = Vs1;
    o[CGFD_FAULT_VS2 * ns + nd] = Vs2;
    o[CGFD_FAULT_SLIP * ns + nd] = l0 + Vs * a.dt;
    o[CGFD_FAULT_SLIP1 * ns + nd] = l1 + Vs1 * a.dt;
    o[CGFD_FAULT_SLIP2 * ns + nd] = l2 + Vs2 * a.dt;
    if (Vs > pk) o[CGFD_FAULT_PEAK_VS * ns + nd] = Vs;
    if (!(fl & FL_T0SET) && Vs > RL(1e-3)) {
      o[CGFD_FAULT_INIT_T0 * ns + nd] = (a.ctl->it + 1) * a.dt;
      F.flag[nd] = fl | FL_T0SET;
    }
    if (!isfinite(Vs)) atomicOr(&a.ctl->err, 1);
  } else if (mode == RK_LAST && q == 2) {
    // traction rate of the step
    real mt[3];
#pragma unroll
    for (int n = 0; n < 3; n++) mt[n] = F.scal[(FS_MT1X + n) * ns + nd];
#pragma unroll
    for (int n = 0; n < 3; n++) {
      F.scal[(FS_HT1X + n) * ns + nd] = (T1s[n] - mt[n]) / a.dt;
      F.scal[(FS_MT1X + n) * ns + nd] = T1s[n];
    }
  }
}

// the six volume points i0-3..i0+3 (not i0) of split nodes, x offset fastest:
// velocity RHS (traction image through the fault) and stress RHS (the
// fault's one-sided x operators), then the RK update with whole-group stores.
// Two threads a point, one per RHS: the two read nothing of one another, and
// the launch is as long as one thread's chain of loads where the fault does
// not fill the GPU.  The halves meet in shared memory because the first
// 16-byte group holds three velocities and Txx: the first half then updates
// that group, the second (Tyy Tzz Tyz Txz) and Txy; each has asked for the
// levels its update starts from before its RHS.
constexpr int kSlabPoints = 96;
__global__ void __launch_bounds__(2 * kSlabPoints) k_fault_slab(const FaultArgs a) {
  __shared__ real sh[9][kSlabPoints];
  const Grid &g = a.g;
  const int tx = threadIdx.x, half = threadIdx.y, mode = a.mode;
  int j = 0, k = 0, s = 1;
  bool act = slab_item(a, (long)blockIdx.x * kSlabPoints + tx, j, k, s);
  act = act && (a.F.flag[(j + NG) + (long)(k + NG) * g.ny] & FL_SPLIT);
  const long sc = g.scmp, q = act ? g.at(a.F.i0 + s, j + NG, k + NG) : 0;
  const long o4 = half ? 4 * sc + 4 * q : 4 * q, o1 = 8 * sc + q;
  real4 cur = make_real4(0.f, 0.f, 0.f, 0.f), u0 = cur;
  real cur1 = 0.f, u1 = 0.f;
  if (act) {
    const real *l = mode == RK_LAST ? a.wend : a.wpre;
    if (mode != RK_THIRD) cur = *reinterpret_cast<const real4 *>(a.wcur + o4);
    if (mode != RK_FIRST) u0 = *reinterpret_cast<const real4 *>(l + o4);
    if (half) {
      if (mode != RK_THIRD) cur1 = a.wcur[o1];
      if (mode != RK_FIRST) u1 = l[o1];
      real h[6];
      slab_stress(a, j, k, s, h);
#pragma unroll
      for (int n = 0; n < 6; n++) sh[3 + n][tx] = h[n];
    } else {
      // T1 of the split node is the split kernel's
      after_previous();
      real h[3];
      slab_velocity(a, j, k, s, h);
#pragma unroll
      for (int n = 0; n < 3; n++) sh[n][tx] = h[n];
    }
  }
  // no kernel behind this one may take the split kernel's end for granted
  // before this one ends
  after_previous();
  __syncthreads();
  if (!act) return;
  const int n0 = 4 * half;
  const real h[4] = { sh[n0][tx], sh[n0 + 1][tx], sh[n0 + 2][tx], sh[n0 + 3][tx] };
  if (mode == RK_LAST) {
    *reinterpret_cast<real4 *>(a.wend + o4) =
        make_real4(rk_end(u0.x, cur.x, a.cb * h[0]), rk_end(u0.y, cur.y, a.cb * h[1]),
                   rk_end(u0.z, cur.z, a.cb * h[2]), rk_end(u0.w, cur.w, a.cb * h[3]));
    if (half) a.wend[o1] = rk_end(u1, cur1, a.cb * sh[8][tx]);
    return;
  }
  const real4 b = mode == RK_FIRST ? cur : u0;
  *reinterpret_cast<real4 *>(a.wout + o4) = make_real4(rk_out(b.x, a.ca * h[0]), rk_out(b.y, a.ca * h[1]),
                                                       rk_out(b.z, a.ca * h[2]), rk_out(b.w, a.ca * h[3]));
  if (half) a.wout[o1] = rk_out(mode == RK_FIRST ? cur1 : u1, a.ca * sh[8][tx]);
  if (mode == RK_SECOND) {
    *reinterpret_cast<real4 *>(a.wend + o4) =
        make_real4(rk_v(u0.x, cur.x, a.ca * h[0]), rk_v(u0.y, cur.y, a.ca * h[1]),
                   rk_v(u0.z, cur.z, a.ca * h[2]), rk_v(u0.w, cur.w, a.ca * h[3]));
    if (half) a.wend[o1] = rk_v(u1, cur1, a.ca * sh[8][tx]);
  }
}

// ---------------------------------------------------------------------------
// stations and fault stations of the current level (io_recv_keep,
// io_funcs.cu:428-469, including its use of corner 5 in place of corner 4;
// io_fault_recv_keep, io_funcs.cu:2313-2351)
__device__ __forceinline__ void record_item(const StationArgs &a, int t) {
  const int rec = a.ctl->nrec;
  const StationDev &S = a.st;
  if (rec >= S.max_rec) return;
  if (t < S.n * 9) {
    const int n = t / 9, c = t % 9;
    const long *ixp = S.idx + (long)n * 8;
    const real Lx2 = S.w[3 * n], Ly2 = S.w[3 * n + 1], Lz2 = S.w[3 * n + 2];
    const real Lx1 = 1.0f - Lx2, Ly1 = 1.0f - Ly2, Lz1 = 1.0f - Lz2;
    // component c of the level: points 4 floats apart in the grouped
    // arrays, 1 real apart for Txy
    const real *v = a.w + a.g.w(c, 0);
    const int u4 = wstep(c);
    const long ix[8] = { u4 * ixp[0], u4 * ixp[1], u4 * ixp[2], u4 * ixp[3],
                         u4 * ixp[4], u4 * ixp[5], u4 * ixp[6], u4 * ixp[7] };
    const real b0 = v[ix[0]], b1 = v[ix[1]], b2 = v[ix[2]], b3 = v[ix[3]];
    const real b5 = v[ix[5]], b6 = v[ix[6]], b7 = v[ix[7]];
    const real r = b0 * Lx1 * Ly1 * Lz1 + b1 * Lx2 * Ly1 * Lz1 + b2 * Lx1 * Ly2 * Lz1 + b3 * Lx2 * Ly2 * Lz1 +
                    b5 * Lx1 * Ly1 * Lz2 + b5 * Lx2 * Ly1 * Lz2 + b6 * Lx1 * Ly2 * Lz2 + b7 * Lx2 * Ly2 * Lz2;
    S.seis[(long)t * S.max_rec + rec] = r;
    if (!isfinite(r)) atomicOr(&a.ctl->err, 1);
  } else if (t < S.n * 9 + S.nf * 9) {
    const int u = t - S.n * 9, n = u / 9, c = u % 9;
    const real *o = a.fout[S.fid[n]] + (long)c * a.ns;
    const int *ix = S.fidx + 4 * n;
    const real Ly2 = S.fw[2 * n], Lz2 = S.fw[2 * n + 1], Ly1 = 1.0f - Ly2, Lz1 = 1.0f - Lz2;
    S.fseis[(long)u * S.max_rec + rec] = o[ix[0]] * Ly1 * Lz1 + o[ix[1]] * Ly2 * Lz1 + o[ix[2]] * Ly1 * Lz2 + o[ix[3]] * Ly2 * Lz2;
  }
}

__global__ void __launch_bounds__(128) k_record(const __grid_constant__ StationArgs a) {
  record_item(a, blockIdx.x * blockDim.x + threadIdx.x);
}

// what a stage's split-node kernel needs first, in one launch (the three
// parts read the stage input and write apart from one another): blocks of
// welded nodes, of tractions, and in a step's first stage of station
// samples, which precede everything that changes the sampled level and the
// fault output.  Small grids are bound by the number of dependent launches:
// a kernel of 4 us each for the two fault parts and 5 us for the stations
// before, 5 us together.
__global__ void __launch_bounds__(192) k_fault_pre(const __grid_constant__ FaultArgs a, const __grid_constant__ StationArgs st,
                                                   int nweld, int ntrac) {
  let_next_start();
  const int b = blockIdx.x;
  if (b < nweld) weld_node(a, (long)b * 192 + threadIdx.x);
  else if (b < nweld + ntrac) trac_item(a, (long)(b - nweld) * 192 + threadIdx.x);
  else record_item(st, (b - nweld - ntrac) * 192 + threadIdx.x);
}

__global__ void k_advance(Ctl *c, int max_rec) {
  c->it += 1;
  if (c->nrec < max_rec) c->nrec += 1;
}

// ---------------------------------------------------------------------------
// first part of a stage: welded nodes, tractions (and, with st, the
// stations), then trial traction and friction (which also refreshes the
// stage input at i0, read by the volume kernels); returns the number of
// launches
namespace {
// a launch that may overlap the end of the kernel ahead of it in the stream
template <class... P, class... Q>
void launch_after(void (*k)(P...), dim3 grid, dim3 block, cudaStream_t st, const Q &...args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.stream = st;
  cfg.attrs = &at; cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k, args...);
}
}  // namespace

int launch_fault_pre(const FaultArgs &a, const StationArgs *rec, cudaStream_t st) {
  const bool split = a.nj > 0 && a.nk > 0;
  const int nweld = (int)(((long)a.wnj * a.wnk + 191) / 192);
  const int ntrac = split ? (int)(((long)a.tnj * a.tnk * 12 + 191) / 192) : 0;
  const int nrec = rec ? ((rec->st.n + rec->st.nf) * 9 + 191) / 192 : 0;
  const StationArgs none{};
  k_fault_pre<<<nweld + ntrac + nrec, 192, 0, st>>>(a, rec ? *rec : none, nweld, ntrac);
  if (!split) return 1;
  const dim3 blk(32, 6), grd((a.nj + 31) / 32, a.nk);
  launch_after(k_fault_split, grd, blk, st, a);
  return 2;
}

// second part: the slab points around the split nodes; independent of the
// volume kernels of the same stage (disjoint outputs, shared read-only input).
// behind_fault: the operation ahead in the stream is a fault kernel, whose end
// the launch may overlap; behind an event wait or a timing event it is an
// ordinary launch
int launch_fault_post(const FaultArgs &a, bool behind_fault, cudaStream_t st) {
  if (a.nj <= 0 || a.nk <= 0) return 0;
  const long nslab = (long)a.nj * a.nk * 6;
  const dim3 grd((unsigned)((nslab + kSlabPoints - 1) / kSlabPoints)), blk(kSlabPoints, 2);
  if (behind_fault) launch_after(k_fault_slab, grd, blk, st, a);
  else k_fault_slab<<<grd, blk, 0, st>>>(a);
  return 1;
}

void launch_record(const StationArgs &a, cudaStream_t st) {
  const int n = (a.st.n + a.st.nf) * 9;
  if (n > 0 && a.st.max_rec > 0) k_record<<<(n + 127) / 128, 128, 0, st>>>(a);
}

void launch_advance(Ctl *c, int max_rec, cudaStream_t st) { k_advance<<<1, 1, 0, st>>>(c, max_rec); }

namespace {
// the interior nodes of the fault output fields [nf][ny*nz] into a
// contiguous [nf][nk][nj] array, so that one copy brings them to the host
__global__ void k_fault_gather(const real *__restrict__ out, real *__restrict__ dst, int nf, int nj, int nk,
                               int ny, long ns) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long n = (long)nj * nk;
  if (t >= n * nf) return;
  const int q = (int)(t / n);
  const long r = t - q * n;
  const int k = (int)(r / nj), j = (int)(r - (long)k * nj);
  dst[t] = __ldg(out + q * ns + (j + NG) + (long)(k + NG) * ny);
}
}  // namespace

void launch_fault_gather(const real *out, real *dst, int nf, const Grid &g, cudaStream_t st) {
  const long n = (long)nf * g.nj * g.nk;
  k_fault_gather<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, dst, nf, g.nj, g.nk, g.ny, (long)g.ny * g.nz);
}

}  // namespace cgfd
