// fs_filament.cu -- filament mechanics, approximate Jacobian and Broyden
// update of the implicit BDF2 step, FP64 on sm_100a.
//
//   k_initial_guess      Filament::initialGuess (Filament.hpp:227-237, Bead.hpp:202-217); with
//                        start order 2 the first bead extrapolated to second order (fs_start.cu)
//   k_assign_forces      Filament::unRobotArmify (Filament.hpp:489-505) +
//                        Fcm::assign_filament_data's Y = fmod(Xs, L) (FCMfunctions.cpp:882-918)
//                        and, in CTAs of its own, setZeroForcesTorques, applyElasticTorques, applyConstraintForcesTorques,
//                        applyExternalForcesTorques (Filament.hpp:271-402), one thread per bead
//                        adding its links' terms in the reference's order
//   k_jacobian_rows, k_jacobian_factor
//                        buildApproximateJacobian with BlockC/D/E/F (Filament.hpp:803-1120) as a
//                        block tridiagonal matrix, factored (two warps per filament)
//   k_error_check        ErrorCheckFCM + dexpinv (MobilityConstraints.cpp:109-143, 447-770)
//   k_tri_apply          filamentJsolver::solve (FilamentJacobianSolver.hpp:49-73): J0^-1 b from
//                        the factors, then the bad-Broyden history corrections
//   k_broyden_cols       history update of main.cpp:640-663 (with a learned diagonal; else k_tri_apply)
//   k_update / k_step    Filament::update (Filament.hpp:425-452), Filament::step (:455-478); with
//                        tension order 1 the tensions extrapolated linearly after lambda_extrap_step
#include <algorithm>
#include "fs_internal.cuh"

namespace {

struct Q {
  double s, v[3];
};

__device__ __forceinline__ Q qload(const double *a) {
  Q q;
  q.s = a[0];
  q.v[0] = a[1];
  q.v[1] = a[2];
  q.v[2] = a[3];
  return q;
}
__device__ __forceinline__ void qstore(const Q &q, double *a) {
  a[0] = q.s;
  a[1] = q.v[0];
  a[2] = q.v[1];
  a[3] = q.v[2];
}
__device__ __forceinline__ double dot3(const double *a, const double *b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
__device__ __forceinline__ void cross3(const double *a, const double *b, double *c) {
  double c0 = a[1] * b[2] - a[2] * b[1], c1 = a[2] * b[0] - a[0] * b[2], c2 = a[0] * b[1] - a[1] * b[0];
  c[0] = c0;
  c[1] = c1;
  c[2] = c2;
}
__device__ __forceinline__ double norm3(const double *a) { return sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]); }

// expmInPlace (UnitQuaternion.hpp:227-242): q <- (cos(t/2), sin(t/2)/t v) * q
__device__ Q q_expm(Q q, const double *v) {
  double theta = norm3(v);
  if (theta > 1.e-12) {
    double tmp = sin(theta * .5) / theta;
    Q p;
    p.s = cos(theta * .5);
    p.v[0] = tmp * v[0];
    p.v[1] = tmp * v[1];
    p.v[2] = tmp * v[2];
    double scal_tmp = q.s * p.s - dot3(q.v, p.v);
    double t[3];
    cross3(p.v, q.v, t);
    Q r;
    for (int d = 0; d < 3; ++d) r.v[d] = q.s * p.v[d] + p.s * q.v[d] + t[d];
    r.s = scal_tmp;
    return r;
  }
  return q;
}

// tangent / normal / binormal (UnitQuaternion.hpp:341-378)
__device__ __forceinline__ void q_tangent(const Q &q, double *v) {
  double q22 = 2 * q.v[1] * q.v[1], q33 = 2 * q.v[2] * q.v[2];
  v[0] = (1 - q22 - q33);
  v[1] = 2 * (q.v[0] * q.v[1] + q.s * q.v[2]);
  v[2] = 2 * (q.v[0] * q.v[2] - q.s * q.v[1]);
}
__device__ __forceinline__ void q_normal(const Q &q, double *v) {
  double q11 = 2 * q.v[0] * q.v[0], q33 = 2 * q.v[2] * q.v[2];
  v[0] = 2 * (q.v[0] * q.v[1] - q.s * q.v[2]);
  v[1] = (1 - q11 - q33);
  v[2] = 2 * (q.v[1] * q.v[2] + q.s * q.v[0]);
}
__device__ __forceinline__ void q_binormal(const Q &q, double *v) {
  double q11 = 2 * q.v[0] * q.v[0], q22 = 2 * q.v[1] * q.v[1];
  v[0] = 2 * (q.v[0] * q.v[2] + q.s * q.v[1]);
  v[1] = 2 * (q.v[1] * q.v[2] - q.s * q.v[0]);
  v[2] = (1 - q11 - q22);
}
// RotateVector (UnitQuaternion.hpp:323-338)
__device__ void q_rotate(const Q &q, double *v) {
  double vx = v[0], vy = v[1], vz = v[2];
  const double *e = q.v;
  double s = q.s;
  double q11 = 2 * e[0] * e[0], q22 = 2 * e[1] * e[1], q33 = 2 * e[2] * e[2];
  v[0] = (1 - q22 - q33) * vx + 2 * (e[0] * e[1] - s * e[2]) * vy + 2 * (e[0] * e[2] + s * e[1]) * vz;
  v[1] = 2 * (e[0] * e[1] + s * e[2]) * vx + (1 - q11 - q33) * vy + 2 * (e[1] * e[2] - s * e[0]) * vz;
  v[2] = 2 * (e[0] * e[2] - s * e[1]) * vx + 2 * (e[1] * e[2] + s * e[0]) * vy + (1 - q11 - q22) * vz;
}
// assignMidPointOf (UnitQuaternion.hpp:472-489) with quaSquareRootTimInPlace (:411-421)
__device__ Q q_midpoint(const Q &p1, const Q &p2) {
  Q m;
  m.s = p2.s * p1.s + dot3(p2.v, p1.v);
  double cr[3];
  cross3(p2.v, p1.v, cr);
  for (int d = 0; d < 3; ++d) m.v[d] = -p2.s * p1.v[d] + p1.s * p2.v[d] - cr[d];
  if (m.s < -.9999999999999) {
    m.s = 0.;
    m.v[0] = 0.;
    m.v[1] = 0.;
    m.v[2] = 1.;
  } else {
    m.s = sqrt(0.5 * (m.s + 1.));
    for (int d = 0; d < 3; ++d) m.v[d] /= (2. * m.s);
  }
  double scal_tmp = m.s * p1.s - dot3(m.v, p1.v);
  double t[3];
  cross3(m.v, p1.v, t);
  Q o;
  for (int d = 0; d < 3; ++d) o.v[d] = m.s * p1.v[d] + p1.s * m.v[d] + t[d];
  o.s = scal_tmp;
  return o;
}

// dexpinv (MobilityConstraints.cpp:109-143)
__device__ void dexpinv(const double *u, const double *w, double *out) {
  double tmp = norm3(u);
  double cuw[3];
  cross3(u, w, cuw);
  if (tmp >= 1.e-12) {
    double tmp2 = tmp / sin(.5 * tmp);
    tmp2 *= cos(.5 * tmp);
    tmp = .5 * tmp2 - 1.;
    double nu = norm3(u);
    double un[3] = {u[0] / nu, u[1] / nu, u[2] / nu};
    double c1[3], c2[3];
    cross3(un, w, c1);
    cross3(un, c1, c2);
    for (int d = 0; d < 3; ++d) {
      out[d] = w[d] - .5 * cuw[d];
      out[d] -= tmp * c2[d];
    }
  } else {
    tmp = 1. / 12;
    double c2[3];
    cross3(u, cuw, c2);
    for (int d = 0; d < 3; ++d) {
      out[d] = w[d] - .5 * cuw[d];
      out[d] += tmp * c2[d];
    }
  }
}

struct FilConsts {
  double L[3];
  double dt, dl, mu, tol;
  double gravity[3], st[3];
  int impl_euler_steps, lambda_extrap_step;
  // swimming drive: time of the forces (nt dt), per-filament parameters or null
  double tt, swim_curvature;
  int swim_sperm_decay;
  const double *swim;
};

// Strain twist of link i of filament f (nw beads) at time k.tt
// (applyElasticTorques, Filament.hpp:297-326): component 0 is the constant
// STRAINTWISTZ; components 1 and 2 are set on every link by the swimming drive,
// Beta facPref cos(k s - w t + phase) and Alpha facPref sin(...), so they are
// zero for a filament without a drive.
__device__ void link_strain_twist(const FilConsts &k, int f, int nw, int i, double *st) {
  st[0] = k.st[0];
  st[1] = 0.0;
  st[2] = 0.0;
  if (!k.swim) return;
  const double *sw = k.swim + 5 * f;
  const double dL = k.dl, L_filament = (nw - 1) * dL, L_filament_long = nw * dL;
  const double T0 = (k.swim_curvature / L_filament_long);
  const double sarc = dL * i + .5 * dL;
  double facPref;
  if (k.swim_sperm_decay) {
    if (sarc > L_filament / 2.0)
      facPref = T0 * 2.0 * (L_filament - sarc) / L_filament;
    else
      facPref = T0;
  } else {
    facPref = T0 * (L_filament - sarc) / L_filament;
  }
  const double arg = sw[3] * sarc - sw[4] * k.tt + sw[2];
  st[1] = sw[1] * facPref * cos(arg);
  st[2] = sw[0] * facPref * sin(arg);
}

// ---- per-bead / per-filament kernels -----------------------------------------
// order 2 with a history of two steps (*hist_ok == 2): the first bead from
// 3X - 3Xt + Xtt, rounded as written (fs_start.cu); otherwise the reference's 2X - Xt
__global__ void k_initial_guess(int np, const int *__restrict__ seg_id, const double *__restrict__ X,
                                const double *__restrict__ Xt, const double *__restrict__ U,
                                const double *__restrict__ Ut, const double *__restrict__ q, double *__restrict__ Xs,
                                double *__restrict__ Us, double *__restrict__ qs, int order,
                                const double *__restrict__ Xtt, const int *__restrict__ hist_ok) {
  FS_AFTER_PREVIOUS();
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= np) return;
  if (seg_id[b] == 0) {
    if (order == 2 && *hist_ok >= 2)
      for (int d = 0; d < 3; ++d)
        Xs[3 * b + d] =
            __dadd_rn(__dsub_rn(__dmul_rn(3., X[3 * b + d]), __dmul_rn(3., Xt[3 * b + d])), Xtt[3 * b + d]);
    else
      for (int d = 0; d < 3; ++d) Xs[3 * b + d] = 2. * X[3 * b + d] - Xt[3 * b + d];
  }
  double us[3];
  for (int d = 0; d < 3; ++d) us[d] = 2. * U[3 * b + d] - Ut[3 * b + d];
  for (int d = 0; d < 3; ++d) Us[3 * b + d] = us[d];
  qstore(q_expm(qload(q + 4 * b), us), qs + 4 * b);
}

// One warp per filament, beads in chunks of 32: the lanes form their beads'
// tangents in parallel, then every lane runs the running sum of
// Filament::unRobotArmify (Filament.hpp:489-505) over the chunk in bead order
// (tangents broadcast by shuffles; the same additions in the same order as one
// thread walking the filament) and keeps its own bead's position; the
// fmod(X, L) of assign_filament_data runs per lane.
__device__ __forceinline__ void unrobot_assign(int block, int nfil, const int *__restrict__ fil_start,
                                               const double *__restrict__ qs, double *__restrict__ Xs,
                                               double *__restrict__ Y, const FilConsts &k) {
  const int f = block * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (f >= nfil) return;  // warp-uniform
  const int b0 = fil_start[f], b1 = fil_start[f + 1];
  const double half = 0.5 * k.dl;
  double Xsum[3] = {Xs[3 * b0], Xs[3 * b0 + 1], Xs[3 * b0 + 2]};
  double t1[3] = {0.0, 0.0, 0.0};
  for (int c0 = b0; c0 < b1; c0 += 32) {
    const int b = c0 + lane, nb = min(32, b1 - c0);
    double t[3] = {0.0, 0.0, 0.0}, mine[3] = {0.0, 0.0, 0.0};
    if (b < b1) q_tangent(qload(qs + 4 * b), t);
    for (int i = 0; i < nb; ++i) {  // warp-uniform trip count
      double t2[3];
      for (int d = 0; d < 3; ++d) t2[d] = __shfl_sync(0xffffffffu, t[d], i);
      if (c0 + i > b0)
        for (int d = 0; d < 3; ++d) Xsum[d] += (t1[d] + t2[d]) * half;
      for (int d = 0; d < 3; ++d) t1[d] = t2[d];
      if (lane == i)
        for (int d = 0; d < 3; ++d) mine[d] = Xsum[d];
    }
    if (b < b1) {
      for (int d = 0; d < 3; ++d) {
        if (b > b0) Xs[3 * b + d] = mine[d];
        Y[3 * b + d] = fmod(mine[d], k.L[d]);
      }
    }
  }
}

// elastic torque of link (i, i+1) (Filament.hpp:297-340), before the +/- to the beads
__device__ void elastic_link(const double *qi_, const double *qj_, double oneOverDL, double kap, double cmod,
                             const double *st, double *vtmp) {
  Q qi = qload(qi_), qj = qload(qj_);
  Q qm = q_midpoint(qi, qj);
  Q q2 = qj;
  q2.s -= qi.s;
  for (int d = 0; d < 3; ++d) q2.v[d] -= qi.v[d];
  q2.s *= oneOverDL;
  for (int d = 0; d < 3; ++d) q2.v[d] *= oneOverDL;
  double tt[3];
  cross3(q2.v, qm.v, tt);
  double nv[3];
  for (int d = 0; d < 3; ++d) nv[d] = -q2.s * qm.v[d] + qm.s * q2.v[d] + tt[d];
  for (int d = 0; d < 3; ++d) vtmp[d] = 2. * nv[d] - st[d];
  vtmp[0] *= cmod;
  vtmp[1] *= kap;
  vtmp[2] *= kap;
  q_rotate(qm, vtmp);
}

// Positions (CTAs below ublocks, a warp per filament) and forces (the others, a thread per
// bead): neither reads what the other writes
__global__ void __launch_bounds__(128) k_assign_forces(int ublocks, int nfil, int np, const int *__restrict__ fil_id,
                                                       const int *__restrict__ seg_id,
                                                       const int *__restrict__ fil_start,
                                                       const double *__restrict__ qs, const double *__restrict__ lam,
                                                       const double *__restrict__ kap,
                                                       const double *__restrict__ cmod, double *__restrict__ Xs,
                                                       double *__restrict__ Y, double *__restrict__ F,
                                                       double *__restrict__ TAU, FilConsts k) {
  FS_AFTER_PREVIOUS();
  if ((int)blockIdx.x < ublocks) {
    unrobot_assign(blockIdx.x, nfil, fil_start, qs, Xs, Y, k);
    return;
  }
  const int b = (blockIdx.x - ublocks) * blockDim.x + threadIdx.x;
  if (b >= np) return;
  const int f = fil_id[b], i = seg_id[b];
  const int nw = fil_start[f + 1] - fil_start[f];
  const int l0 = fil_start[f] - f;
  const double oneOverDL = 1. / k.dl;
  double tau[3] = {0.0, 0.0, 0.0}, fo[3] = {0.0, 0.0, 0.0}, v[3], st[3];
  // elastic: link i-1 subtracts, link i adds (link order of Filament.hpp:297)
  if (i >= 1) {
    link_strain_twist(k, f, nw, i - 1, st);
    elastic_link(qs + 4 * (b - 1), qs + 4 * b, oneOverDL, kap[f], cmod[f], st, v);
    for (int d = 0; d < 3; ++d) tau[d] -= v[d];
  }
  if (i < nw - 1) {
    link_strain_twist(k, f, nw, i, st);
    elastic_link(qs + 4 * b, qs + 4 * (b + 1), oneOverDL, kap[f], cmod[f], st, v);
    for (int d = 0; d < 3; ++d) tau[d] += v[d];
  }
  // constraint forces and torques (Filament.hpp:351-368)
  const double fac = -.5 * k.dl;
  double t[3], c2[3];
  q_tangent(qload(qs + 4 * b), t);
  if (i >= 1) {
    const double *lm = lam + 3 * (l0 + i - 1);
    for (int d = 0; d < 3; ++d) fo[d] += lm[d];
    cross3(t, lm, c2);
    for (int d = 0; d < 3; ++d) tau[d] += fac * c2[d];
  }
  if (i < nw - 1) {
    const double *lm = lam + 3 * (l0 + i);
    for (int d = 0; d < 3; ++d) fo[d] -= lm[d];
    cross3(t, lm, c2);
    for (int d = 0; d < 3; ++d) tau[d] += fac * c2[d];
  }
  for (int d = 0; d < 3; ++d) {
    F[3 * b + d] = fo[d] + k.gravity[d];
    TAU[3 * b + d] = tau[d];
  }
}

// Spring links (spring_links::apply_spring_link_forces, spring_link_functions.cpp:24-45),
// after the filaments' own forces (main.cpp:354-357): per link, the minimum-image
// displacement of its beads (VecPeriodicX, :139-145) and a Hookean force along it,
// + on the first bead and - on the second. One thread per bead adds its links in
// link order, the order of the reference's sequential loop.
__global__ void k_spring_forces(int np, const int *__restrict__ off, const int *__restrict__ ent,
                                const int *__restrict__ beads, const double *__restrict__ Xs, double ks, double l0,
                                FilConsts k, double *__restrict__ F) {
  FS_AFTER_PREVIOUS();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= np) return;
  double f[3] = {F[3 * b], F[3 * b + 1], F[3 * b + 2]};
  for (int e = off[b]; e < off[b + 1]; ++e) {
    const int l = ent[e] >> 1, second = ent[e] & 1;
    const int bn = beads[2 * l], bm = beads[2 * l + 1];
    double disp[3];
    for (int d = 0; d < 3; ++d) {
      disp[d] = Xs[3 * bn + d] - Xs[3 * bm + d];
      disp[d] = disp[d] - k.L[d] * floor(disp[d] / k.L[d] + 0.5);
    }
    const double dist = sqrt(disp[0] * disp[0] + disp[1] * disp[1] + disp[2] * disp[2]);
    const double mag = ks * (dist - l0);
    for (int d = 0; d < 3; ++d) {
      const double sf = -mag * disp[d] / dist;
      if (second)
        f[d] -= sf;
      else
        f[d] += sf;
    }
  }
  for (int d = 0; d < 3; ++d) F[3 * b + d] = f[d];
}

// ---- Jacobian ------------------------------------------------------------------
struct M3 {
  double m[9];
};
__device__ __forceinline__ M3 rcross(const double *x) {
  M3 r;
  r.m[0] = 0.;
  r.m[1] = x[2];
  r.m[2] = -x[1];
  r.m[3] = -x[2];
  r.m[4] = 0.;
  r.m[5] = x[0];
  r.m[6] = x[1];
  r.m[7] = -x[0];
  r.m[8] = 0.;
  return r;
}
__device__ __forceinline__ M3 mt(const M3 &a) {
  M3 r;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) r.m[3 * i + j] = a.m[3 * j + i];
  return r;
}
__device__ M3 mmul(const M3 &a, const M3 &b) {
  M3 r;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      double acc = 0.0;
      for (int kk = 0; kk < 3; ++kk) acc += a.m[3 * i + kk] * b.m[3 * kk + j];
      r.m[3 * i + j] = acc;
    }
  return r;
}
__device__ __forceinline__ M3 madd(M3 a, const M3 &b) {
  for (int i = 0; i < 9; ++i) a.m[i] += b.m[i];
  return a;
}
__device__ __forceinline__ M3 msub(M3 a, const M3 &b) {
  for (int i = 0; i < 9; ++i) a.m[i] -= b.m[i];
  return a;
}
__device__ __forceinline__ M3 msc(M3 a, double s) {
  for (int i = 0; i < 9; ++i) a.m[i] *= s;
  return a;
}
__device__ __forceinline__ M3 outer(const double *a, const double *b) {
  M3 r;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) r.m[3 * i + j] = a[i] * b[j];
  return r;
}
__device__ M3 blockE_diag(const M3 &dOmega, const M3 &LieMat, const M3 &OmegaMat, const double *Us, double dt) {
  double ov[3];
  for (int i = 0; i < 3; ++i) ov[i] = OmegaMat.m[3 * i] * Us[0] + OmegaMat.m[3 * i + 1] * Us[1] + OmegaMat.m[3 * i + 2] * Us[2];
  M3 inner = msub(dOmega, msc(madd(OmegaMat, mmul(LieMat, dOmega)), 0.5));
  M3 corr = madd(madd(rcross(ov), mmul(LieMat, OmegaMat)), mmul(mmul(LieMat, LieMat), dOmega));
  inner = madd(inner, msc(corr, 1. / 12.));
  return msc(inner, -2 * dt / 3.);
}
__device__ M3 blockE_off(const M3 &dOmega, const M3 &LieMat, double dt) {
  M3 inner = msub(dOmega, msc(mmul(LieMat, dOmega), 0.5));
  inner = madd(inner, msc(mmul(mmul(LieMat, LieMat), dOmega), 1. / 12.));
  return msc(inner, -2 * dt / 3.);
}
__device__ __forceinline__ void frame(const double *qa, double *t, double *n, double *b) {
  Q q = qload(qa);
  q_tangent(q, t);
  q_normal(q, n);
  q_binormal(q, b);
}
// store of a 3x3 block at column c0 of a 3 x 9 row (row-major)
__device__ __forceinline__ void put3(double *J, int c0, const M3 &a) {
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) J[9 * i + c0 + j] = a.m[3 * i + j];
}

// the three BlockE blocks of bead row k (Filament.hpp:958-1089), stored into the 3 x 9
// row J: columns of bead k - 1 (not for the first bead), k, k + 1 (not for the last)
__device__ void blockE_row(int k, int nw, const double *qs, const double *Us, const double *TAU, const double *lam,
                           double rad_k, double myC, double myKAP, const double *ST, double DL, double dt, double MU,
                           double *J) {
  const double PI = FS_PI;
  double t[3], nn[3], b[3], tp1[3], np1[3], bp1[3], tm1[3], nm1[3], bm1[3];
  const double Tfac = 1 / (8 * PI * MU * (rad_k * rad_k * rad_k));
  const M3 LieMat = mt(rcross(Us + 3 * k));
  const double tT[3] = {Tfac * TAU[3 * k], Tfac * TAU[3 * k + 1], Tfac * TAU[3 * k + 2]};
  const M3 OmegaMat = rcross(tT);
  frame(qs + 4 * k, t, nn, b);
  if (k == 0) {
    frame(qs + 4, tp1, np1, bp1);
    M3 ConstraintPart = mmul(msc(rcross(lam), -0.5 * DL), rcross(t));
    double beta = -ST[2] + 0.5 * (np1[0] * b[0] + np1[1] * b[1] + np1[2] * b[2] - nn[0] * bp1[0] - nn[1] * bp1[1] - nn[2] * bp1[2]) / DL;
    double CP[3] = {b[1] * np1[2] - b[2] * np1[1] - nn[1] * bp1[2] + nn[2] * bp1[1],
                    b[2] * np1[0] - b[0] * np1[2] - nn[2] * bp1[0] + nn[0] * bp1[2],
                    b[0] * np1[1] - b[1] * np1[0] - nn[0] * bp1[1] + nn[1] * bp1[0]};
    double ttp[3] = {t[0] + tp1[0], t[1] + tp1[1], t[2] + tp1[2]};
    M3 EP = msc(madd(msc(outer(ttp, CP), 0.5 / DL), msc(rcross(t), beta)), 0.5 * myC);
    EP = madd(EP, msc(msub(msc(mmul(rcross(tp1), rcross(t)), 1. / DL),
                           msc(madd(msc(rcross(nn), ST[0]), msc(rcross(b), ST[1])), 0.5)),
                      0.5 * myKAP));
    M3 dOmega = msc(madd(EP, ConstraintPart), Tfac);
    put3(J, 3, blockE_diag(dOmega, LieMat, OmegaMat, Us, dt));
    EP = msc(msub(msc(rcross(tp1), beta), msc(outer(ttp, CP), 0.5 / DL)), 0.5 * myC);
    EP = madd(EP, msc(msub(msc(mmul(mt(rcross(t)), rcross(tp1)), 1. / DL),
                           msc(madd(msc(rcross(np1), ST[0]), msc(rcross(bp1), ST[1])), 0.5)),
                      0.5 * myKAP));
    dOmega = msc(EP, Tfac);
    put3(J, 6, blockE_off(dOmega, LieMat, dt));
    return;
  }
  if (k == nw - 1) {
    frame(qs + 4 * (k - 1), tm1, nm1, bm1);
    M3 ConstraintPart = mmul(msc(rcross(lam + 3 * (k - 1)), -0.5 * DL), rcross(t));
    double beta = -ST[2] + 0.5 * (nn[0] * bm1[0] + nn[1] * bm1[1] + nn[2] * bm1[2] - nm1[0] * b[0] - nm1[1] * b[1] - nm1[2] * b[2]) / DL;
    double CPm[3] = {bm1[1] * nn[2] - bm1[2] * nn[1] - nm1[1] * b[2] + nm1[2] * b[1],
                     bm1[2] * nn[0] - bm1[0] * nn[2] - nm1[2] * b[0] + nm1[0] * b[2],
                     bm1[0] * nn[1] - bm1[1] * nn[0] - nm1[0] * b[1] + nm1[1] * b[0]};
    double ttm[3] = {t[0] + tm1[0], t[1] + tm1[1], t[2] + tm1[2]};
    M3 EP = msc(msub(msc(rcross(t), beta), msc(outer(ttm, CPm), 0.5 / DL)), -0.5 * myC);
    EP = msub(EP, msc(msub(msc(mmul(mt(rcross(tm1)), rcross(t)), 1. / DL),
                           msc(madd(msc(rcross(nn), ST[0]), msc(rcross(b), ST[1])), 0.5)),
                      0.5 * myKAP));
    M3 dOmega = msc(madd(EP, ConstraintPart), Tfac);
    put3(J, 3, blockE_diag(dOmega, LieMat, OmegaMat, Us + 3 * k, dt));
    EP = msc(msub(msc(rcross(tm1), beta), msc(outer(ttm, CPm), 0.5 / DL)), -0.5 * myC);
    EP = msub(EP, msc(msub(msc(mmul(rcross(t), rcross(tm1)), 1. / DL),
                           msc(madd(msc(rcross(nm1), ST[0]), msc(rcross(bm1), ST[1])), 0.5)),
                      0.5 * myKAP));
    dOmega = msc(EP, Tfac);
    put3(J, 0, blockE_off(dOmega, LieMat, dt));
    return;
  }
  frame(qs + 4 * (k - 1), tm1, nm1, bm1);
  frame(qs + 4 * (k + 1), tp1, np1, bp1);
  double lamvec[3] = {lam[3 * (k - 1)] + lam[3 * k], lam[3 * (k - 1) + 1] + lam[3 * k + 1], lam[3 * (k - 1) + 2] + lam[3 * k + 2]};
  M3 ConstraintPart = mmul(msc(rcross(lamvec), -0.5 * DL), rcross(t));
  double beta = -ST[2] + 0.5 * (np1[0] * b[0] + np1[1] * b[1] + np1[2] * b[2] - nn[0] * bp1[0] - nn[1] * bp1[1] - nn[2] * bp1[2]) / DL;
  double CPk[3] = {b[1] * np1[2] - b[2] * np1[1] - nn[1] * bp1[2] + nn[2] * bp1[1],
                   b[2] * np1[0] - b[0] * np1[2] - nn[2] * bp1[0] + nn[0] * bp1[2],
                   b[0] * np1[1] - b[1] * np1[0] - nn[0] * bp1[1] + nn[1] * bp1[0]};
  double tp[3] = {t[0] + tp1[0], t[1] + tp1[1], t[2] + tp1[2]};
  double tm[3] = {t[0] + tm1[0], t[1] + tm1[1], t[2] + tm1[2]};
  M3 EP = msc(madd(msc(outer(tp, CPk), 0.5 / DL), msc(rcross(t), beta)), 0.5 * myC);
  EP = madd(EP, msc(msub(msc(mmul(rcross(tp1), rcross(t)), 1. / DL),
                         msc(madd(msc(rcross(nn), ST[0]), msc(rcross(b), ST[1])), 0.5)),
                    0.5 * myKAP));
  // the k-1 side beta, with the k+1 side CrossPart kept (Filament.hpp:1068-1070)
  beta = -ST[2] + 0.5 * (nn[0] * bm1[0] + nn[1] * bm1[1] + nn[2] * bm1[2] - nm1[0] * b[0] - nm1[1] * b[1] - nm1[2] * b[2]) / DL;
  EP = msub(EP, msc(msub(msc(rcross(t), beta), msc(outer(tm, CPk), 0.5 / DL)), 0.5 * myC));
  EP = msub(EP, msc(msub(msc(mmul(mt(rcross(tm1)), rcross(t)), 1. / DL),
                         msc(madd(msc(rcross(nn), ST[0]), msc(rcross(b), ST[1])), 0.5)),
                    0.5 * myKAP));
  M3 dOmega = msc(madd(ConstraintPart, EP), Tfac);
  put3(J, 3, blockE_diag(dOmega, LieMat, OmegaMat, Us + 3 * k, dt));
  EP = msc(msub(msc(rcross(tm1), beta), msc(outer(tm, CPk), 0.5 / DL)), -0.5 * myC);
  EP = msub(EP, msc(msub(msc(mmul(rcross(t), rcross(tm1)), 1. / DL),
                         msc(madd(msc(rcross(nm1), ST[0]), msc(rcross(bm1), ST[1])), 0.5)),
                    0.5 * myKAP));
  dOmega = msc(EP, Tfac);
  put3(J, 0, blockE_off(dOmega, LieMat, dt));
  // right block with the k-1 side beta (Filament.hpp:1083)
  EP = msc(msub(msc(rcross(tp1), beta), msc(outer(tp, CPk), 0.5 / DL)), 0.5 * myC);
  EP = madd(EP, msc(msub(msc(mmul(mt(rcross(t)), rcross(tp1)), 1. / DL),
                         msc(madd(msc(rcross(np1), ST[0]), msc(rcross(bp1), ST[1])), 0.5)),
                    0.5 * myKAP));
  dOmega = msc(EP, Tfac);
  put3(J, 6, blockE_off(dOmega, LieMat, dt));
}

// ---- approximate Jacobian as a block tridiagonal matrix ----------------------------
//
// With columns [X0 (3) | U (3nw) | lambda (3nw-3)] and rows [first-bead
// position (3) | constraints (3nw-3) | Lie updates (3nw)], the reference's J
// (Filament.hpp:803-867) is
//     J = [ I  0  P  ]    P  = (temp/dt) [I 0 ... 0]
//         [ 0  C  D' ]    C  = BlockC(DL/2), D' = 10 BlockD/dt (block bidiagonal, scalar blocks)
//         [ 0  E  F' ]    E  = BlockE (block tridiagonal), F' = BlockF/dt (block bidiagonal)
// C's rows are running sums along the filament (row r: fac c_0 + 2 fac sum_{1<=q<=r} c_q +
// fac c_{r+1}, c_q = cross(u_q, t_q)), so the difference of two successive constraint rows
// is fac (c_r + c_{r+1}) and D' becomes block tridiagonal: with the unknowns (u_k, lambda_k)
// and the rows (Lie update k, constraint k - constraint k-1) of a bead taken together, J
// is block tridiagonal with 6 x 6 blocks,
//     A_k z_{k-1} + B_k z_k + G_k z_{k+1} = r_k
// (the last bead has no lambda: its second half is the identity). It is factored once per
// build, from both ends towards the bead in the middle (mid = nw / 2), two chains at a
// time: with Dk = B_k - A_k W_{k-1} before the middle, B_k - G_k W_{k+1} after it and both
// in it, each bead keeps 108 doubles: Dk^-1, W_k = Dk^-1 times the block towards the middle
// (in the middle: G) and T_k = Dk^-1 times the block it came from (in the middle: A). An
// application runs the chains y_k = Dk^-1 r_k - T_k y_before inwards and z_k = y_k - W_k
// z_inner outwards. Linear in the filament's length, where the 3nw x 3nw inverse of the
// Schur complement of D' is cubic to build and quadratic to apply; against J solved in 80
// bits over filaments of 2 to 48 beads (dt 1e-3 to 0.3, moduli 0.1 to 100, ah 0.6 to 1.6)
// it is within 2e-14, the Schur complement within 1e-13.
#define FS_MAX_NW 48
constexpr int TRI = 108;     // doubles of a bead's factors: D^-1, W, T (6 x 6 row-major each)
constexpr int TRI_ROW = 39;  // doubles of a bead's row: E (3 x 9), F'(k,k) (9), tangent (3)
constexpr int TRI_APPLY_WARPS = 2;  // filaments per CTA of k_tri_apply

// D' blocks of a row (BlockD(nt), Filament.hpp:912-949), of the radii of its bead and the next
__device__ __forceinline__ double tri_dd(int nt, const FilConsts &k, double rad) {
  double facn = -2. * k.dt / (18. * FS_PI * k.mu * rad);
  if (nt <= k.impl_euler_steps) facn *= (3. / 2.);
  return 10. * facn / k.dt;
}
__device__ __forceinline__ double tri_ee(int nt, const FilConsts &k, double rad_next) {
  double facu = 2. * k.dt / (18. * FS_PI * k.mu * rad_next);
  if (nt <= k.impl_euler_steps) facu *= (3. / 2.);
  return 10. * facu / k.dt;
}
// entry (i, c) of the matrix u -> cross(u, t)
__device__ __forceinline__ double cross_entry(const double *t, int i, int c) {
  if (i == c) return 0.0;
  const double v = t[3 - i - c];
  return (i + 1) % 3 == c ? v : -v;
}

// Bead rows of J, a thread per bead: the E row and F' block (that of bead k is F'(k,k) and,
// a function of bead k alone, also F'(k,k-1)) and the tangent, as rows[entry][bead]. Bound by
// the FP64 instructions of blockE_row, a few warps per SM at its registers.
__global__ void __launch_bounds__(128) k_jacobian_rows(int np, const int *__restrict__ fil_id,
                                                       const int *__restrict__ fil_start,
                                                       const double *__restrict__ qs, const double *__restrict__ Us,
                                                       const double *__restrict__ TAU, const double *__restrict__ lam,
                                                       const double *__restrict__ kap, const double *__restrict__ cmod,
                                                       double *__restrict__ rows, FilConsts k, double a, double ah,
                                                       const int *__restrict__ keep) {
  FS_AFTER_PREVIOUS();
  if (keep && *keep) return;  // the previous step's J0 stays (fs_set_broyden_memory)
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= np) return;
  const int f = fil_id[g], b0 = fil_start[f], nw = fil_start[f + 1] - b0, kk = g - b0;
  if (nw < 2) return;  // J0 is the identity
  const double *q_f = qs + 4 * b0, *Us_f = Us + 3 * b0;
  const double rad = kk == 0 ? ah : a;
  // this->myStrainTwist as applyElasticTorques(nt) left it: its last link (nw >= 2 here)
  double stj[3], E[27], tv[3];
  link_strain_twist(k, f, nw, nw - 2, stj);
#pragma unroll
  for (int e = 0; e < 27; ++e) E[e] = 0.0;
  blockE_row(kk, nw, q_f, Us_f, TAU + 3 * b0, lam + 3 * (b0 - f), rad, cmod[f], kap[f], stj, k.dl, k.dt, k.mu, E);
  for (int i = 0; i < 3; ++i) E[9 * i + 3 + i] += 1.;  // BlockE's identity (Filament.hpp:1092-1094)
#pragma unroll
  for (int e = 0; e < 27; ++e) rows[(size_t)e * np + g] = E[e];
  // BlockF / dt (Filament.hpp:1099-1120)
  const double fac2 = k.dt * k.dl / (24 * FS_PI * k.mu * (rad * rad * rad));
  q_tangent(qload(q_f + 4 * kk), tv);
  const M3 tmat = mt(rcross(tv)), umat = rcross(Us_f + 3 * kk);
  const M3 F =
      msc(madd(msub(tmat, msc(mmul(umat, tmat), 0.5)), msc(mmul(mmul(umat, umat), tmat), 1. / 12.)), fac2 / k.dt);
#pragma unroll
  for (int e = 0; e < 9; ++e) rows[(size_t)(27 + e) * np + g] = F.m[e];
#pragma unroll
  for (int d = 0; d < 3; ++d) rows[(size_t)(36 + d) * np + g] = tv[d];
}

// Column c (0..5) of block A_k (which = -1), B_k (0) or G_k (+1); E: the bead's row, dd, ee
// the D' entries of its constraint row, ddp, eep of the row before (0 where absent; dd = 1
// and ee = 0 for the last bead, whose lambda is held at 0)
__device__ __forceinline__ void tri_column(double v[6], int which, int c, const double *E, bool last, double fac,
                                           double dd, double ee, double ddp, double eep) {
  const int c3 = c % 3;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double top, bot;  // rows i (Lie) and 3 + i (constraint)
    if (c < 3) {
      top = E[9 * i + 3 * which + 3 + c3];
      bot = last || which < 0 ? 0.0 : fac * cross_entry(E + TRI_ROW * which + 36, i, c3);
    } else {
      top = which > 0 || (which == 0 && last) ? 0.0 : E[27 + 3 * i + c3];
      bot = i != c3 ? 0.0 : which < 0 ? -ddp : which > 0 ? ee : dd - eep;
    }
    v[i] = top;
    v[3 + i] = bot;
  }
}

// The two chains of a filament, a warp each (then the middle bead by the first): 24 lanes
// hold the columns of [Dk | I | towards | from] and run a Gauss-Jordan elimination of Dk on
// them, pivot rows in place. Bound by the latency of that chain (search, reciprocal and
// update of six pivots, each on the one before) and, with several filaments per SM, by its
// instructions. 1,024 filaments of 32 beads, both kernels: 72 us, against 850 us for the Schur
// complement's assembly and inverse (a warp per filament over all its beads, no second
// chain: 110 us; 4,096 filaments 400 us, with two chains 208 us).
__global__ void __launch_bounds__(64) k_jacobian_factor(int np, const int *__restrict__ fil_start,
                                                        const double *__restrict__ rows, double *__restrict__ tri,
                                                        int nt, FilConsts k, double a, double ah,
                                                        int *__restrict__ flags, const int *__restrict__ keep) {
  FS_AFTER_PREVIOUS();
  extern __shared__ __align__(16) double tri_smem[];
  if (keep && *keep) return;
  const int f = blockIdx.x, tid = threadIdx.x, lane = tid & 31, side = tid >> 5;
  const int b0 = fil_start[f], nw = fil_start[f + 1] - b0, nl = nw - 1, mid = nw / 2;
  if (nw < 2) return;  // J0 is the identity
  double *bead = tri_smem + 72;  // W of the two chains' last bead first
  for (int e = tid; e < TRI_ROW * nw; e += 64) {
    const int r = e / nw, kk = e - r * nw;
    bead[TRI_ROW * kk + r] = rows[(size_t)r * np + b0 + kk];
  }
  __syncthreads();
  const double fac = 0.5 * k.dl, dd_a = tri_dd(nt, k, a), dd_h = tri_dd(nt, k, ah), ee_a = tri_ee(nt, k, a);
  const int part = lane / 6, c = lane % 6;  // 0 D, 1 identity, 2 towards, 3 from (lanes 24.. idle)
  double *out = tri + (size_t)TRI * b0;
  bool singular = false;
  const int steps = side == 0 ? mid + 1 : nl - mid;
  for (int s = 0; s < steps; ++s) {
    const int kk = side == 0 ? s : nl - s;
    if (kk == mid) __syncthreads();  // the second chain is done; it waits below
    const double *E = bead + TRI_ROW * kk;
    const bool last = kk == nl;
    const double dd = last ? 1.0 : kk == 0 ? dd_h : dd_a, ee = kk < nl - 1 ? ee_a : 0.0;
    const double ddp = kk == 0 || last ? 0.0 : kk == 1 ? dd_h : dd_a, eep = kk > 0 && !last ? ee_a : 0.0;
    const int dir = side == 0 ? 1 : -1;
    double v[6];
    if (part == 1 || part > 3) {
#pragma unroll
      for (int i = 0; i < 6; ++i) v[i] = part == 1 && i == c ? 1.0 : 0.0;
    } else {
      const int which = part == 0 ? 0 : part == 2 ? dir : -dir;
      if ((which < 0 && kk == 0) || (which > 0 && last)) {
#pragma unroll
        for (int i = 0; i < 6; ++i) v[i] = 0.0;
      } else {
        tri_column(v, which, c, E, last, fac, dd, ee, ddp, eep);
      }
    }
    if (part == 0) {
      if (kk > 0 && kk <= mid) {  // D -= A W_{k-1}
        double w[6];
#pragma unroll
        for (int l = 0; l < 6; ++l) w[l] = tri_smem[6 * l + c];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          v[i] -= (E[9 * i] * w[0] + E[9 * i + 1] * w[1] + E[9 * i + 2] * w[2]) +
                  (E[27 + 3 * i] * w[3] + E[28 + 3 * i] * w[4] + E[29 + 3 * i] * w[5]);
          v[3 + i] += ddp * w[3 + i];
        }
      }
      if (kk < nl && kk >= mid) {  // D -= G W_{k+1}
        double w[6];
        const double *t = E + TRI_ROW + 36;
#pragma unroll
        for (int l = 0; l < 6; ++l) w[l] = tri_smem[36 + 6 * l + c];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          v[i] -= E[9 * i + 6] * w[0] + E[9 * i + 7] * w[1] + E[9 * i + 8] * w[2];
          v[3 + i] -= fac * (w[(i + 1) % 3] * t[(i + 2) % 3] - w[(i + 2) % 3] * t[(i + 1) % 3]) + ee * w[3 + i];
        }
      }
    }
    unsigned used = 0, pos = 0;  // pivot rows taken; the column each register row served
#pragma unroll
    for (int j = 0; j < 6; ++j) {
      double col[6];
#pragma unroll
      for (int i = 0; i < 6; ++i) col[i] = __shfl_sync(0xffffffffu, v[i], j);
      // the largest remaining entry, to the 17 leading bits of its significand
      unsigned key[6];
#pragma unroll
      for (int i = 0; i < 6; ++i)
        key[i] = (used >> i) & 1u ? 0u : (((unsigned)__double2hiint(col[i]) & 0x7ffffff8u) | (unsigned)i);
      const int pr = max(max(max(key[0], key[1]), max(key[2], key[3])), max(key[4], key[5])) & 7u;
      used |= 1u << pr;
      pos |= (unsigned)j << (4 * pr);
      const bool h0 = pr & 1, h1 = pr & 2, h2 = pr & 4;
      const double piv = h2 ? (h0 ? col[5] : col[4]) : h1 ? (h0 ? col[3] : col[2]) : (h0 ? col[1] : col[0]);
      double x = h2 ? (h0 ? v[5] : v[4]) : h1 ? (h0 ? v[3] : v[2]) : (h0 ? v[1] : v[0]);
      singular |= !(fabs(piv) > 0.0);
      x *= 1.0 / piv;
#pragma unroll
      for (int i = 0; i < 6; ++i) v[i] = pr == i ? x : v[i] - col[i] * x;
    }
    __syncwarp();  // the W before is no longer read
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const int j = (pos >> (4 * i)) & 7u;
      if (part >= 1 && part <= 3) out[(size_t)TRI * kk + 36 * (part - 1) + 6 * j + c] = v[i];
      if (part == 2) tri_smem[36 * side + 6 * j + c] = v[i];
    }
    __syncwarp();
  }
  if (side == 1) __syncthreads();
  if (singular && lane == 0) atomicOr(&flags[FLAG_PIVOT], 1);
}

// v -= M (v of lanes src .. src + 5): one link of a chain, lane row i of M's six
__device__ __forceinline__ double tri_link(double g, const double *row, double v, int src) {
  const double2 t0 = *reinterpret_cast<const double2 *>(row), t1 = *reinterpret_cast<const double2 *>(row + 2),
                t2 = *reinterpret_cast<const double2 *>(row + 4);
  const double v0 = __shfl_sync(0xffffffffu, v, src), v1 = __shfl_sync(0xffffffffu, v, src + 1),
               v2 = __shfl_sync(0xffffffffu, v, src + 2), v3 = __shfl_sync(0xffffffffu, v, src + 3),
               v4 = __shfl_sync(0xffffffffu, v, src + 4), v5 = __shfl_sync(0xffffffffu, v, src + 5);
  return (g - (t0.x * v0 + t0.y * v1 + t1.x * v2)) - (t1.y * v3 + t2.x * v4 + t2.y * v5);
}

// J0^-1 b for one filament of nw >= 2 beads, by one warp and in place. b (shared): 6nw entries
// [first-bead position rows | constraint rows | Lie rows], then [X0 | U | lambda/dt]. wt
// (shared, 16-byte aligned): 72nw doubles; y (shared): 6nw.
__device__ __forceinline__ void tri_apply(int nw, const double *__restrict__ tri, double *b, double *wt, double *y,
                                          double dt, double pcoef) {
  const int lane = threadIdx.x & 31, nl = nw - 1, m = 3 * nw, mid = nw / 2;
  const unsigned dst = (unsigned)__cvta_generic_to_shared(wt);
  for (int e = lane; e < 36 * nw; e += 32) {  // W and T arrive while the lanes form y_k = Dk^-1 r_k
    const int kk = e / 36, j = e - 36 * kk;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * e),
                 "l"(tri + (size_t)TRI * kk + 36 + 2 * j)
                 : "memory");
  }
  const double *b1 = b + 3, *b2 = b + m;
#pragma unroll 3
  for (int e = lane; e < 6 * nw; e += 32) {
    const int kk = e / 6, i = e - 6 * kk;
    const double2 *d = reinterpret_cast<const double2 *>(tri + (size_t)TRI * kk + 6 * i);
    const double2 d0 = d[0], d1 = d[1], d2 = d[2];
    double r[3] = {0.0, 0.0, 0.0};
    if (kk < nl)
      for (int c = 0; c < 3; ++c) r[c] = kk > 0 ? b1[3 * kk + c] - b1[3 * kk - 3 + c] : b1[c];
    y[e] = (d0.x * b2[3 * kk] + d0.y * b2[3 * kk + 1] + d1.x * b2[3 * kk + 2]) + (d1.y * r[0] + d2.x * r[1] + d2.y * r[2]);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncwarp();
  // lanes 0..5: the chain from the first bead; 8..13: from the last (other lanes follow along)
  const bool down = lane & 8;
  const int src = down ? 8 : 0, i = (lane & 7) < 6 ? lane & 7 : 0;
  const bool mine = lane < 16 && (lane & 7) < 6;
  double v = y[6 * (down ? nl : 0) + i];
  for (int s = 1; s < mid; ++s) {  // inwards
    const int kk = down ? nl - s : s;
    const bool on = !down || kk > mid;
    const double u = tri_link(y[6 * kk + i], wt + 72 * kk + 36 + 6 * i, v, src);
    if (on) v = u;
    if (on && mine) y[6 * kk + i] = v;
  }
  {  // the middle: T_m of the first chain, W_m of the second
    double u = tri_link(0.0, wt + 72 * mid + (down ? 0 : 36) + 6 * i, v, src);
    if (down && mid == nl) u = 0.0;
    const double o = __shfl_xor_sync(0xffffffffu, u, 8);
    v = y[6 * mid + i] + (down ? o + u : u + o);
    __syncwarp();
    if (mine && !down) y[6 * mid + i] = v;
  }
  for (int s = 1; s <= mid; ++s) {  // outwards
    const int kk = down ? (mid + s < nl ? mid + s : nl) : mid - s;
    const bool on = !down || mid + s <= nl;
    const double u = tri_link(y[6 * kk + i], wt + 72 * kk + 6 * i, v, src);
    if (on) v = u;
    if (on && mine) y[6 * kk + i] = v;
  }
  __syncwarp();
  for (int e = lane; e < m; e += 32) {
    const int kk = e / 3, d = e - 3 * kk;
    b[3 + e] = y[6 * kk + d];
    if (kk < nl) b[3 + m + e] = y[6 * kk + 3 + d] / dt;  // the reference's 1/dt rows (Filament.hpp:863-865)
  }
  if (lane < 3) b[lane] -= pcoef * y[3 + lane];
  __syncwarp();
}
__host__ __device__ constexpr int tri_apply_doubles(int nw) { return (72 + 6 + 6) * nw; }

// x_f = J0_f^-1 b_f (one bead: the identity), then x += sum_i C_i dots_i
// (FilamentJacobianSolver.hpp:49-73); a warp per filament. With upd given x is not written: b is
// dE, and columns ncol of Cnew and Dnew are (C's columns below ncol are what is read). Bound by the latency of the two
// chains (a shuffle and two dependent products per bead) and the factors' load before them.
// With the dots before it, 1,024 filaments of 32 beads and 6 columns: 33 us (the columns one
// load after another: 42); 4,096 filaments 97 us (132).
__global__ void __launch_bounds__(32 * TRI_APPLY_WARPS) k_tri_apply(
    int nfil, const int *__restrict__ fil_start, const double *__restrict__ tri, const double *__restrict__ b,
    double *__restrict__ x, const double *__restrict__ C, const double *__restrict__ dots, int iter,
    const int *__restrict__ iter_d, const int *__restrict__ off_d, size_t n6, double dt, double pcoef, int max_nw,
    const double *__restrict__ upd, const double *__restrict__ nrm, double *Cnew, double *Dnew) {
  FS_AFTER_PREVIOUS();
  extern __shared__ __align__(16) double tri_smem[];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int f = blockIdx.x * TRI_APPLY_WARPS + wl;
  if (f >= nfil) return;  // warp-uniform; no block barrier below
  const int b0 = fil_start[f], nw = fil_start[f + 1] - b0, s0 = 6 * b0, n = 6 * nw;
  double *wt = tri_smem + (size_t)wl * tri_apply_doubles(max_nw), *bb = wt + 72 * max_nw, *y = bb + 6 * max_nw;
  for (int r = lane; r < n; r += 32) bb[r] = b[s0 + r];
  __syncwarp();
  if (nw >= 2) tri_apply(nw, tri + (size_t)TRI * b0, bb, wt, y, dt, pcoef);
  const int ncol = (iter_d ? *iter_d : iter) + (off_d ? *off_d : 0);
  // three entries a lane and four columns at a time: twelve loads in flight
  for (int r0 = lane; r0 < n; r0 += 96) {
    double v[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) v[j] = r0 + 32 * j < n ? bb[r0 + 32 * j] : 0.0;
    for (int i0 = 0; i0 < ncol; i0 += 4) {
      double w[4][3], d[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        d[u] = i0 + u < ncol ? dots[i0 + u] : 0.0;
#pragma unroll
        for (int j = 0; j < 3; ++j)
          w[u][j] = i0 + u < ncol && r0 + 32 * j < n ? C[(size_t)(i0 + u) * n6 + s0 + r0 + 32 * j] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (i0 + u < ncol)
#pragma unroll
          for (int j = 0; j < 3; ++j) v[j] += w[u][j] * d[u];
    }
    if (upd) {  // the history's next column, as k_broyden_cols forms it
      const double nn = nrm[0];
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (r0 + 32 * j < n) {
          const size_t r = s0 + r0 + 32 * j;
          double t = v[j] * (-1. / nn);
          t -= upd[r] / nn;
          Cnew[(size_t)ncol * n6 + r] = t;
          Dnew[(size_t)ncol * n6 + r] = b[r] / nn;
        }
    } else {
#pragma unroll
      for (int j = 0; j < 3; ++j)
        if (r0 + 32 * j < n) x[s0 + r0 + 32 * j] = v[j];
    }
  }
}

// explicit inverse of filament f's J0 (with the 1/dt rows), one column per CTA (test access)
__global__ void __launch_bounds__(32) k_tri_inverse(int nw, const double *__restrict__ tri, double dt, double pcoef,
                                                    double *__restrict__ out) {
  FS_AFTER_PREVIOUS();
  extern __shared__ __align__(16) double tri_smem[];
  double *bb = tri_smem + 72 * nw, *y = bb + 6 * nw;
  const int n = 6 * nw, e = blockIdx.x, lane = threadIdx.x;
  for (int r = lane; r < n; r += 32) bb[r] = (r == e) ? 1.0 : 0.0;
  __syncwarp();
  if (nw >= 2) tri_apply(nw, tri, bb, tri_smem, y, dt, pcoef);
  for (int r = lane; r < n; r += 32) out[(size_t)r * n + e] = bb[r];
}

// ---- error check ---------------------------------------------------------------
__global__ void k_error_check(int np, const int *__restrict__ fil_id, const int *__restrict__ seg_id,
                              const int *__restrict__ fil_start, const double *__restrict__ Xs,
                              const double *__restrict__ X, const double *__restrict__ Xt,
                              const double *__restrict__ Us, const double *__restrict__ U,
                              const double *__restrict__ V, const double *__restrict__ W, double *__restrict__ err,
                              int nt, FilConsts k, int *__restrict__ flags, unsigned long long *__restrict__ maxbits) {
  FS_AFTER_PREVIOUS();
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  bool over = false, nonfin = false, expl = false;
  double mx = 0.0;
  if (b < np) {
    const int f = fil_id[b], i = seg_id[b];
    const int b0 = fil_start[f], nw = fil_start[f + 1] - b0;
    const int s0 = 6 * b0;
    double dv[3];
    dexpinv(Us + 3 * b, W + 3 * b, dv);
    const double fourthirds = 4. / 3., onethird = 1. / 3., twothirdsDt = k.dt * 2. / 3.;
    for (int d = 0; d < 3; ++d) {
      double e1, e2;
      if (nt <= k.impl_euler_steps) {
        e1 = Xs[3 * b + d] - X[3 * b + d] - k.dt * V[3 * b + d];
        e2 = Us[3 * b + d] - k.dt * dv[d];
      } else {
        e1 = Xs[3 * b + d] - fourthirds * X[3 * b + d] + onethird * Xt[3 * b + d] - twothirdsDt * V[3 * b + d];
        e2 = Us[3 * b + d] - onethird * U[3 * b + d] - twothirdsDt * dv[d];
      }
      err[s0 + 3 * i + d] = e1;
      err[s0 + 3 * nw + 3 * i + d] = e2;
      over |= (fabs(e1) > k.tol) || (fabs(e2) > k.tol);
      nonfin |= !isfinite(e1) || !isfinite(e2);
      expl |= (fabs(e1) > 1e6) || (fabs(e2) > 1e6);
      mx = fmax(mx, fmax(fabs(e1), fabs(e2)));
    }
  }
  const unsigned full = 0xffffffffu;
  if (__any_sync(full, over) && (threadIdx.x & 31) == 0) atomicOr(&flags[FLAG_CHECK], 1);
  if (__any_sync(full, nonfin) && (threadIdx.x & 31) == 0) atomicOr(&flags[FLAG_NONFINITE], 1);
  if (__any_sync(full, expl) && (threadIdx.x & 31) == 0) atomicOr(&flags[FLAG_EXPLODE], 1);
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(full, mx, o));
  if ((threadIdx.x & 31) == 0 && maxbits) atomicMax(maxbits, fs_dbits(mx));
}

// ---- Broyden ---------------------------------------------------------------------
#define RED_THREADS 256
#define RED_BLOCKS 296

// partial dot products D_i . b for i < iter (iter_d ? *iter_d : iter), plus the
// columns carried from earlier steps (off_d ? *off_d : 0, fs_start.cu): each of the
// RED_BLOCKS blocks sums a fixed strided slice of every column, so the partials
// (and the fixed-order final sums) do not depend on how many columns there are
__global__ void __launch_bounds__(RED_THREADS) k_dots(const double *__restrict__ D, const double *__restrict__ b,
                                                       size_t n6, int iter, const int *__restrict__ iter_d,
                                                       const int *__restrict__ off_d, double *__restrict__ partial) {
  FS_AFTER_PREVIOUS();
  // columns in groups of DOT_COLS: a thread reads b[k] once per group and keeps
  // the group's loads in flight together; each column's sum runs in the same
  // order as one column at a time (k ascending per thread, then the shuffle
  // tree, then the warps in order), so the partials are bitwise those
  constexpr int DOT_COLS = 16;
  __shared__ double sh[DOT_COLS][RED_THREADS / 32];
  const int ncol = (iter_d ? *iter_d : iter) + (off_d ? *off_d : 0);
  for (int i0 = 0; i0 < ncol; i0 += DOT_COLS) {
    double acc[DOT_COLS];
#pragma unroll
    for (int j = 0; j < DOT_COLS; ++j) acc[j] = 0.0;
    for (size_t k = (size_t)blockIdx.x * RED_THREADS + threadIdx.x; k < n6; k += (size_t)gridDim.x * RED_THREADS) {
      const double bk = b[k];
#pragma unroll
      for (int j = 0; j < DOT_COLS; ++j)
        if (i0 + j < ncol) acc[j] += D[(size_t)(i0 + j) * n6 + k] * bk;
    }
#pragma unroll
    for (int j = 0; j < DOT_COLS; ++j) {
      double a = acc[j];
      for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
      if ((threadIdx.x & 31) == 0) sh[j][threadIdx.x >> 5] = a;
    }
    __syncthreads();
    if (threadIdx.x < DOT_COLS && i0 + (int)threadIdx.x < ncol) {
      const int j = threadIdx.x;
      double s = 0.0;
      for (int w = 0; w < RED_THREADS / 32; ++w) s += sh[j][w];
      partial[(size_t)(i0 + j) * gridDim.x + blockIdx.x] = s;
    }
    __syncthreads();
  }
}

// fixed-order final sums: one warp per output
__global__ void k_reduce_rows(const double *__restrict__ partial, int nparts, int nrows, double *__restrict__ out,
                              int do_sqrt, const int *__restrict__ nrows_d, const int *__restrict__ off_d) {
  FS_AFTER_PREVIOUS();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= (nrows_d ? *nrows_d : nrows) + (off_d ? *off_d : 0)) return;
  double acc = 0.0;
  for (int p = lane; p < nparts; p += 32) acc += partial[(size_t)row * nparts + p];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) out[row] = do_sqrt ? sqrt(acc) : acc;
}

// dE = newerr - err and per-block sums of dE^2
__global__ void __launch_bounds__(RED_THREADS) k_diff_sq(const double *__restrict__ ne, const double *__restrict__ e,
                                                          double *__restrict__ dE, size_t n6,
                                                          double *__restrict__ partial) {
  FS_AFTER_PREVIOUS();
  __shared__ double sh[RED_THREADS / 32];
  double acc = 0.0;
  for (size_t k = (size_t)blockIdx.x * RED_THREADS + threadIdx.x; k < n6; k += (size_t)gridDim.x * RED_THREADS) {
    double d = ne[k] - e[k];
    dE[k] = d;
    acc += d * d;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < RED_THREADS / 32; ++w) s += sh[w];
    partial[blockIdx.x] = s;
  }
}

// The same sums for short vectors, a CTA per column, in one launch: out[i] = D_i . b, or with
// e given D_i . (b - e); then the last CTA also writes dE = b - e and *norm = |dE|.
__global__ void __launch_bounds__(1024) k_dots_small(const double *__restrict__ D, const double *__restrict__ b,
                                                     const double *__restrict__ e, double *__restrict__ dE, int n6,
                                                     int iter, const int *__restrict__ iter_d,
                                                     const int *__restrict__ off_d, double *__restrict__ out,
                                                     double *__restrict__ norm) {
  FS_AFTER_PREVIOUS();
  __shared__ double sh[32];
  const int ncol = (iter_d ? *iter_d : iter) + (off_d ? *off_d : 0), tid = threadIdx.x;
  const bool diff = e && blockIdx.x == gridDim.x - 1;
  if (!diff && (int)blockIdx.x >= ncol) return;
  const double *col = D + (size_t)blockIdx.x * n6;
  double acc = 0.0;
#pragma unroll 4
  for (int k = tid; k < n6; k += 1024) {
    const double v = e ? b[k] - e[k] : b[k];
    if (diff) dE[k] = v;
    acc += (diff ? v : col[k]) * v;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((tid & 31) == 0) sh[tid >> 5] = acc;
  __syncthreads();
  if (tid < 32) {
    acc = sh[tid];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (tid == 0) {
      if (diff) *norm = sqrt(acc);
      else out[blockIdx.x] = acc;
    }
  }
}

// C_iter = -tmp/|dE| - upd/|dE|, D_iter = dE/|dE| (main.cpp:657-661)
// column iter (iter_d ? *iter_d : iter) of the history, after the columns carried
// from earlier steps (off_d ? *off_d : 0)
__global__ void k_broyden_cols(const double *__restrict__ tmp, const double *__restrict__ upd,
                               const double *__restrict__ dE, const double *__restrict__ nrm, size_t n6,
                               double *__restrict__ Cmat, double *__restrict__ Dmat, int iter,
                               const int *__restrict__ iter_d, const int *__restrict__ off_d) {
  FS_AFTER_PREVIOUS();
  size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n6) return;
  const size_t col = (size_t)((iter_d ? *iter_d : iter) + (off_d ? *off_d : 0)) * n6;
  double *__restrict__ Ccol = Cmat + col;
  double *__restrict__ Dcol = Dmat + col;
  const double n = nrm[0];
  double t = tmp[k] * (-1. / n);
  t -= upd[k] / n;
  Ccol[k] = t;
  Dcol[k] = dE[k] / n;
}

// ---- update / step ----------------------------------------------------------------
__global__ void k_update(int np, const int *__restrict__ fil_id, const int *__restrict__ seg_id,
                         const int *__restrict__ fil_start, const double *__restrict__ u, double *__restrict__ Xs,
                         double *__restrict__ Us, const double *__restrict__ q, double *__restrict__ qs,
                         double *__restrict__ lam) {
  FS_AFTER_PREVIOUS();
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= np) return;
  const int f = fil_id[b], i = seg_id[b];
  const int b0 = fil_start[f], nw = fil_start[f + 1] - b0, l0 = b0 - f;
  const int s = 6 * b0;
  double us[3];
  if (i == 0) {
    for (int d = 0; d < 3; ++d) {
      Xs[3 * b + d] -= u[s + d];
      us[d] = Us[3 * b + d] - u[s + 3 + d];
    }
  } else {
    for (int d = 0; d < 3; ++d) us[d] = Us[3 * b + d] - u[s + 6 + 3 * (i - 1) + d];
  }
  for (int d = 0; d < 3; ++d) Us[3 * b + d] = us[d];
  qstore(q_expm(qload(q + 4 * b), us), qs + 4 * b);
  if (i < nw - 1)
    for (int d = 0; d < 3; ++d) lam[3 * (l0 + i) + d] -= u[s + 3 * nw + 3 + 3 * i + d];
}

__global__ void k_step(int np, int nlink, double *__restrict__ X, double *__restrict__ Xs, double *__restrict__ Xt,
                       double *__restrict__ U, double *__restrict__ Us, double *__restrict__ Ut,
                       double *__restrict__ q, double *__restrict__ qt, double *__restrict__ lam,
                       double *__restrict__ lam1, double *__restrict__ lam2, int nt, int ex, int tension_order) {
  FS_AFTER_PREVIOUS();
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < np) {
    const int b = t;
    double uu[3];
    for (int d = 0; d < 3; ++d) {
      Xt[3 * b + d] = X[3 * b + d];
      X[3 * b + d] = Xs[3 * b + d];
      Ut[3 * b + d] = U[3 * b + d];
      uu[d] = Us[3 * b + d];
      U[3 * b + d] = uu[d];
    }
    Q qq = qload(q + 4 * b);
    qstore(qq, qt + 4 * b);
    qstore(q_expm(qq, uu), q + 4 * b);
  }
  if (t < 3 * nlink) {
    const int kk = t;
    if (nt > ex && tension_order == 2) {
      double lamtmp = 3 * lam[kk] - 3 * lam1[kk] + lam2[kk];
      lam2[kk] = lam1[kk];
      lam1[kk] = lam[kk];
      lam[kk] = lamtmp;
    } else if (nt >= ex) {  // the reference: at nt == ex only; tension order 1 from then on
      double lamtmp = 2. * lam[kk] - lam1[kk];
      lam2[kk] = lam1[kk];
      lam1[kk] = lam[kk];
      lam[kk] = lamtmp;
    } else {
      lam1[kk] = lam[kk];
    }
  }
}

FilConsts make_fconsts(const fs_ctx *c) {
  FilConsts k;
  for (int d = 0; d < 3; ++d) {
    k.L[d] = c->L[d];
    k.gravity[d] = c->p.gravity[d];
    k.st[d] = c->p.strain_twist[d];
  }
  k.dt = c->p.dt;
  k.dl = c->p.dl;
  k.mu = c->p.mu;
  k.tol = c->p.tol;
  k.impl_euler_steps = c->p.impl_euler_steps;
  k.lambda_extrap_step = c->p.lambda_extrap_step;
  k.tt = 0.0;
  k.swim_curvature = c->swim_curvature;
  k.swim_sperm_decay = c->swim_sperm_decay;
  k.swim = c->swim;
  return k;
}

}  // namespace

fs_status fil_initial_guess(fs_ctx *c) {
  if (!c->have_state) return FS_ERR_STATE;
  ProfScope ps(c, FS_STAGE_UPDATE);
  const int order = (c->start_order == 2 && c->hist_Xtt) ? 2 : 1;
  fs_launch(k_initial_guess, fs_blocks(c->np, 256), 256, 0, c->stream, c->np, c->seg_id, c->X, c->Xt, c->U, c->Ut,
            c->q, c->Xs, c->Us, c->qs, order, c->hist_Xtt, c->hist_ok);
  FS_LAUNCH_CHECK();
  return FS_OK;
}

fs_status fil_forces(fs_ctx *c, int nt) {
  if (!c->have_state) return FS_ERR_STATE;
  ProfScope ps(c, FS_STAGE_FORCES);
  FilConsts k = make_fconsts(c);
  k.tt = nt * c->p.dt;  // double tt = nt*dt (Filament.hpp:295)
  const int ublocks = fs_blocks(c->nfil, 4);
  fs_launch(k_assign_forces, ublocks + fs_blocks(c->np, 128), 128, 0, c->stream, ublocks, c->nfil, c->np, c->fil_id,
            c->seg_id, c->fil_start, c->qs, c->lam, c->kap, c->cc, c->Xs, c->Y, c->F, c->TAU, k);
  FS_LAUNCH_CHECK();
  if (c->nspring > 0) {
    fs_launch(k_spring_forces, fs_blocks(c->np, 256), 256, 0, c->stream, c->np, c->spring_off, c->spring_ent,
              c->spring_beads, c->Xs, c->spring_k, c->spring_l0, k, c->F);
    FS_LAUNCH_CHECK();
  }
  return FS_OK;
}

// keep (device, or null): nonzero leaves the previous J0 in place
fs_status fil_jacobian_build(fs_ctx *c, int nt, const int *keep) {
  if (!c->have_state) return FS_ERR_STATE;
  ProfScope ps(c, FS_STAGE_JACOBIAN);
  FilConsts k = make_fconsts(c);
  k.tt = nt * c->p.dt;
  if (c->np == 0) return FS_OK;
  double *rows = c->jtri + (size_t)TRI * c->np;
  fs_launch(k_jacobian_rows, fs_blocks(c->np, 128), 128, 0, c->stream, c->np, c->fil_id, c->fil_start, c->qs, c->Us,
            c->TAU, c->lam, c->kap, c->cc, rows, k, c->p.a, c->p.ah, keep);
  FS_LAUNCH_CHECK();
  // a plain launch: its CTAs all fit at once, and placed while the rows' kernel still fills some
  // of the SMs they crowd the others (1,024 filaments of 32 beads: 104 us for both, 72 so)
  k_jacobian_factor<<<c->nfil, 64, sizeof(double) * (72 + TRI_ROW * c->max_nw), c->stream>>>(
      c->np, c->fil_start, rows, c->jtri, nt, k, c->p.a, c->p.ah, c->flags, keep);
  FS_LAUNCH_CHECK();
  return FS_OK;
}

fs_status fil_jacobian_prepare(fs_ctx *c) {
  if (c->max_nw > FS_MAX_NW) return FS_ERR_INVALID_ARG;
  FS_CUDA(cudaFuncSetAttribute(k_tri_apply, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(sizeof(double) * TRI_APPLY_WARPS * tri_apply_doubles(FS_MAX_NW))));
  return FS_OK;
}

size_t fil_jacobian_doubles(int np) { return (size_t)(TRI + TRI_ROW) * np; }

// P's coefficient (temp / dt, Filament.hpp:820-830)
static double tri_pcoef(const fs_ctx *c) { return (c->p.dt / (9 * FS_PI * c->p.mu * c->p.ah)) / c->p.dt; }

fs_status fil_jacobian_inverse(fs_ctx *c, int f, double *out_d) {
  const int b0 = c->fil_start_h[f], nw = c->fil_start_h[f + 1] - b0, n = 6 * nw;
  fs_launch(k_tri_inverse, n, 32, sizeof(double) * tri_apply_doubles(nw), c->stream, nw, c->jtri + (size_t)TRI * b0,
            c->p.dt, tri_pcoef(c), out_d);
  FS_LAUNCH_CHECK();
  return FS_OK;
}

fs_status fil_error_check(fs_ctx *c, const double *V, const double *W, double *err, int nt) {
  if (!c->have_state) return FS_ERR_STATE;
  ProfScope ps(c, FS_STAGE_ERROR_CHECK);
  FilConsts k = make_fconsts(c);
  FS_CUDA(cudaMemsetAsync(c->flags, 0, sizeof(int) * 3, c->stream));  // check, nonfinite, explode
  FS_CUDA(cudaMemsetAsync(c->maxerr_bits, 0, sizeof(unsigned long long), c->stream));
  fs_launch(k_error_check, fs_blocks(c->np, 256), 256, 0, c->stream, c->np, c->fil_id, c->seg_id, c->fil_start, c->Xs,
            c->X, c->Xt, c->Us, c->U, V, W, err, nt, k, c->flags, c->maxerr_bits);
  FS_LAUNCH_CHECK();
  return FS_OK;
}

// iter_d (graph capture): the history length is read on the device; off_d: the
// columns carried from earlier steps before it (fs_set_broyden_memory), or none
// Vectors up to this long: a CTA per column. With the application of 6 columns: 480 beads 17.3
// us, against 21.0 for blocks of partial sums and their reduction; 4,096 beads 19.8 (21.4);
// 8,192 beads 25.7 (22.4).
constexpr size_t DOTS_SMALL = 24576;

// dots[i] = D_i . b; with e given D_i . dE, dE = b - e and c->scalars[0] = |dE|
static fs_status broyden_dots(fs_ctx *c, const double *b, const double *e, int iter, const int *iter_d,
                              const int *off_d) {
  const size_t n6 = (size_t)6 * c->np;
  // rows launched: a bound on the device count (with the memory on, callers pass
  // iter 0 and no iter_d: the count is the carried and current columns, off_d)
  const int base = iter_d ? c->p.broyden_maxiter : iter;
  const int rows = off_d ? c->p.broyden_maxiter + c->bmem_cols + base : base;
  if (n6 <= DOTS_SMALL) {
    if (rows == 0 && !e) return FS_OK;
    fs_launch(k_dots_small, rows + (e ? 1 : 0), 1024, 0, c->stream, c->Dmat, b, e, c->dE, (int)n6, iter, iter_d, off_d,
              c->dots, c->scalars);
    FS_LAUNCH_CHECK();
    return FS_OK;
  }
  if (e) {
    fs_launch(k_diff_sq, RED_BLOCKS, RED_THREADS, 0, c->stream, b, e, c->dE, n6, c->partials);
    FS_LAUNCH_CHECK();
    fs_launch(k_reduce_rows, 1, 32, 0, c->stream, c->partials, RED_BLOCKS, 1, c->scalars, 1, nullptr, nullptr);
    FS_LAUNCH_CHECK();
  }
  if (rows == 0) return FS_OK;
  fs_launch(k_dots, RED_BLOCKS, RED_THREADS, 0, c->stream, c->Dmat, e ? c->dE : b, n6, iter, iter_d, off_d,
            c->partials);
  FS_LAUNCH_CHECK();
  fs_launch(k_reduce_rows, fs_blocks(rows, 8), 256, 0, c->stream, c->partials, RED_BLOCKS, iter, c->dots, 0, iter_d,
            off_d);
  FS_LAUNCH_CHECK();
  return FS_OK;
}

// x = J0^-1 b + C dots, or with upd given the history's next column
static fs_status tri_apply_launch(fs_ctx *c, const double *b, double *x, const double *upd, int iter,
                                  const int *iter_d, const int *off_d) {
  fs_launch(k_tri_apply, fs_blocks(c->nfil, TRI_APPLY_WARPS), 32 * TRI_APPLY_WARPS,
            sizeof(double) * TRI_APPLY_WARPS * tri_apply_doubles(c->max_nw), c->stream, c->nfil, c->fil_start,
            c->jtri, b, x, c->Cmat, c->dots, iter, iter_d, off_d, (size_t)6 * c->np, c->p.dt, tri_pcoef(c), c->max_nw,
            upd, c->scalars, c->Cmat, c->Dmat);
  FS_LAUNCH_CHECK();
  return FS_OK;
}

fs_status fil_broyden_apply(fs_ctx *c, const double *b, double *x, int iter, const int *iter_d, const int *off_d) {
  if (!c->have_state) return FS_ERR_STATE;
  ProfScope ps(c, FS_STAGE_BROYDEN);
  FS_TRY(broyden_dots(c, b, nullptr, iter, iter_d, off_d));
  FS_TRY(tri_apply_launch(c, b, x, nullptr, iter, iter_d, off_d));
  return learn_diag_apply(c, b, x);  // learned initial inverse-Jacobian diagonal, when on
}

// main.cpp:641-663 with the current err/newerr/upd: history column `iter`
fs_status fil_broyden_update(fs_ctx *c, int iter, const int *iter_d, const int *off_d) {
  ProfScope ps(c, FS_STAGE_BROYDEN);
  FS_TRY(broyden_dots(c, c->newerr, c->err, iter, iter_d, off_d));
  if (!learn_diag_on(c)) return tri_apply_launch(c, c->dE, c->tmp, c->upd, iter, iter_d, off_d);
  FS_TRY(tri_apply_launch(c, c->dE, c->tmp, nullptr, iter, iter_d, off_d));
  FS_TRY(learn_diag_apply(c, c->dE, c->tmp));
  const size_t n6 = (size_t)6 * c->np;
  fs_launch(k_broyden_cols, fs_blocks((long long)n6, 256), 256, 0, c->stream, c->tmp, c->upd, c->dE, c->scalars, n6,
            c->Cmat, c->Dmat, iter, iter_d, off_d);
  FS_LAUNCH_CHECK();
  return FS_OK;
}

fs_status fil_state_update(fs_ctx *c, const double *upd) {
  if (!c->have_state) return FS_ERR_STATE;
  ProfScope ps(c, FS_STAGE_UPDATE);
  fs_launch(k_update, fs_blocks(c->np, 256), 256, 0, c->stream, c->np, c->fil_id, c->seg_id, c->fil_start, upd, c->Xs,
            c->Us, c->q, c->qs, c->lam);
  FS_LAUNCH_CHECK();
  return FS_OK;
}

fs_status fil_step(fs_ctx *c, int nt) {
  if (!c->have_state) return FS_ERR_STATE;
  ProfScope ps(c, FS_STAGE_UPDATE);
  int n = c->np > 3 * c->nlink ? c->np : 3 * c->nlink;
  fs_launch(k_step, fs_blocks(n, 256), 256, 0, c->stream, c->np, c->nlink, c->X, c->Xs, c->Xt, c->U, c->Us, c->Ut,
            c->q, c->qt, c->lam, c->lam1, c->lam2, nt, c->p.lambda_extrap_step, c->tension_order == 1 ? 1 : 2);
  FS_LAUNCH_CHECK();
  return FS_OK;
}

fs_status fil_max_abs_err(fs_ctx *c, const double *err, double *out_h) {
  (void)err;
  unsigned long long bits;
  FS_CUDA(cudaMemcpyAsync(&bits, c->maxerr_bits, sizeof bits, cudaMemcpyDeviceToHost, c->stream));
  FS_CUDA(cudaStreamSynchronize(c->stream));
  memcpy(out_h, &bits, sizeof bits);
  return FS_OK;
}
