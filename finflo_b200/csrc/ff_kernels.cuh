// sm_100a kernels of the FINFLO per-iteration hot path (FP64).
//
// Launch shapes:
//   k_state / k_fin / k_time3_copr ...  element-wise, one thread per cell
//   k_patch_*                         one grid row per boundary patch
//   k_grad                            one thread per cell incl. ghost layer 1
//   k_residual                        32x4x4-cell tiles, all three face
//                                     directions fused, face fluxes staged
//                                     in shared memory, residual written once
//   k_sweep_coef + k_lusgs_sweep      coefficient pass into the skewed sweep
//                                     layout, then a cooperative persistent
//                                     kernel marching the i+j+k hyperplanes
//                                     with a bounded grid barrier
//   k_flow_coef + k_flow_sweep        the same sweep as a wavefront of warps
//                                     (the default, ff_flow.cuh)
#pragma once
#include "ff_device.cuh"
#include <cooperative_groups.h>

namespace ff {

constexpr int TI = 32, TJ = 4, TK = 4;   // residual tile
#ifndef RES_MIN_CTAS
#define RES_MIN_CTAS 4                    // residual threads per SM the register budget aims at, / 128
#endif
constexpr int NCOEF = 13;                 // LU-SGS coefficients per cell

// ---------------------------------------------------------------------------
// STATIM: PDTOP state.f:1690, PERFGA state.f:159, CONSVA base3c.f:489, and the
// laminar TURBDI (ADJUIN res3c.f:9447: EPS2 = 1, VIST = 0 on interior cells).
struct StateV {
  double P, drdp, ro, vis, drdh, cp, ch, c, e, u, v, w;
};

FF_DI StateV state_eval(const DevBlock& b, const ff_params& p, size_t n) {
  StateV s;
  double pd = b.a[FF_PDIFF][n], T = b.a[FF_TEMP][n];
  s.u = b.a[FF_U][n]; s.v = b.a[FF_V][n]; s.w = b.a[FF_W][n];
  const double rk = p.iturb < 3 ? 0. : b.a[FF_RK][n];
  s.P = pd + p.frspre;
  const double gm1 = p.gamma - 1., cp2 = p.gamma / gm1 * p.rgas;
  double trgs = T * p.rgas;
  s.drdp = 1. / trgs;
  s.ro = s.P * s.drdp;
  s.vis = p.visu0 * T * sqrt(T) / (T + p.tsu0);
  double e = trgs / gm1;
  s.drdh = -s.ro / e / p.gamma;
  double rkin = (s.u * s.u + s.v * s.v + s.w * s.w) * .5;
  if (p.iturb < 3) {
    s.c = sqrt(dmax(1. / (s.drdh / s.ro + s.drdp), 1.0));
  } else {   // CONSVA two-equation branch: k in the sound speed and E
    double ypro = 1. / s.ro;
    double xturb = 1. + (2. / 3.) * rk * ypro * s.drdp;
    s.c = sqrt(dmax(xturb / (s.drdh * ypro + s.drdp), 1.0));
  }
  s.cp = cp2;
  s.ch = s.vis * cp2 / p.pr;
  s.e = p.iturb < 3 ? (e + rkin) * s.ro : (e + rkin) * s.ro + rk;
  return s;
}

FF_DI void state_store(const DevBlock& b, size_t n, const StateV& s) {
  b.a[FF_P][n] = s.P;
  b.a[FF_DRDP][n] = s.drdp;
  b.a[FF_RO][n] = s.ro;
  b.a[FF_VIS][n] = s.vis;
  b.a[FF_DRDH][n] = s.drdh;
  b.a[FF_CP][n] = s.cp;
  b.a[FF_CH][n] = s.ch;
  b.a[FF_C][n] = s.c;
  b.a[FF_E][n] = s.e;
  b.a[FF_RM][n] = s.ro * s.u;
  b.a[FF_RN][n] = s.ro * s.v;
  b.a[FF_RW][n] = s.ro * s.w;
}
// one cell of the equation of state
FF_DI void state_cell(const DevBlock& b, const ff_params& p, size_t n, bool interior) {
  state_store(b, n, state_eval(b, p, n));
  if (p.iturb < 3 && interior) {   // with two equations TURBEQ, not ADJUIN, sets EPS2 and VIST
    b.a[FF_EPS2][n] = 1.0;
    b.a[FF_VIST][n] = 0.0;
  }
}

__global__ void k_state(DevBlock b, ff_params p) {
  size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= (size_t)b.ntot) return;
  int i = (int)(n % b.is), j = (int)((n / b.is) % (b.jmax + 4)), k = (int)(n / b.il);
  state_cell(b, p, n, i >= 2 && i < b.imax + 2 && j >= 2 && j < b.jmax + 2 && k >= 2 && k < b.kmax + 2);
}

// Face description of a patch: direction, sign, normal stride, interior layer.
struct FaceG { int dir, idir, s, layer; };
FF_DI FaceG face_g(const DevBlock& b, int iface) {
  FaceG f;
  f.dir = (iface - 1) % 3 + 1;
  f.idir = iface <= 3 ? 1 : -1;
  f.s = f.dir == 1 ? 1 : (f.dir == 2 ? b.is : b.il);
  int mx = f.dir == 1 ? b.imax : (f.dir == 2 ? b.jmax : b.kmax);
  f.layer = iface <= 3 ? 1 : mx;
  return f;
}
FF_DI size_t face_cell(const DevBlock& b, const FaceG& f, int a, int c) {
  if (f.dir == 1) return ix(b, f.layer, a, c);
  if (f.dir == 2) return ix(b, a, f.layer, c);
  return ix(b, a, c, f.layer);
}

// Patch-cell iteration: blockIdx.y = patch, x covers r1 x r2.
#define FF_PATCH_LOOP(b)                                                       \
  const ff_patch& pa = (b).patch[blockIdx.y];                                  \
  int n1 = pa.r1b - pa.r1a + 1, n2 = pa.r2b - pa.r2a + 1;                      \
  int t = blockIdx.x * blockDim.x + threadIdx.x;                               \
  if (t >= n1 * n2) return;                                                    \
  int pa1 = pa.r1a + t % n1, pa2 = pa.r2a + t / n1;                            \
  FaceG fg = face_g((b), pa.iface);                                            \
  int ls = fg.idir * fg.s;                                                     \
  (void)ls;                                                                    \
  size_t L = face_cell((b), fg, pa1, pa2);

// The patch kernels below read everything a cell needs before the first
// store: a slot's store may alias the next slot's load as far as the compiler
// knows, so load-store pairs in turn cost one L2 round trip each (k_reflec
// 10.8, k_mir 12.1, k_refcor 12.0, k_refcen 8.6 and k_inlet_outlet 7.7 us a
// launch on a 16x8x8 block; 6.3, 4.4, 3.7, 4.9 and 6.0 us now).

// REFLEC turb3.f:5294: solid walls (viscous, wall at rest) and the inlet
// pressure extrapolation.  mode 0: REFLEC; mode 1: re-evaluate the equation of
// state in the two ghost cells first (the second STATIM pass).
FF_DI void reflec_cell(const DevBlock& b, const ff_params& p, const ff_patch& pa, size_t L, int ls, int mode) {
  size_t LB = L - ls, LT = L + ls, LC = L - 2 * ls;
  bool wall = pa.ityp >= 7 && pa.ityp <= 10;
  if (!wall && pa.ityp != FF_BC_INL) return;
  double* P = b.a[FF_P]; double* PD = b.a[FF_PDIFF];
  double *T = b.a[FF_TEMP], *RO = b.a[FF_RO];
  const double pl = P[L], pdl = PD[L];
  StateV sB, sC;
  if (mode == 1) { sB = state_eval(b, p, LB); sC = state_eval(b, p, LC); }
  if (pa.ityp == FF_BC_INL) {
    if (mode == 1) { state_store(b, LB, sB); state_store(b, LC, sC); }
    P[LB] = pl; PD[LB] = pdl; P[LC] = pl; PD[LC] = pdl;
    return;
  }
  const double tl = T[L], vis = b.a[FF_VIS][L], ch = b.a[FF_CH][L], cc = b.a[FF_C][L], drdp = b.a[FF_DRDP][L];
  const double drdh = b.a[FF_DRDH][L], u = -b.a[FF_U][L], v = -b.a[FF_V][L], w = -b.a[FF_W][L], rol = RO[L];
  const double plt = P[LT], pdlt = PD[LT], e = b.a[FF_E][L];
  double rk = 0., re = 0., ret = 0.;
  if (p.iturb >= 3) { rk = b.a[FF_RK][L]; re = b.a[FF_REPS][L]; ret = b.a[FF_REPS][LT]; }
  if (mode == 1) { state_store(b, LB, sB); state_store(b, LC, sC); }
  int ihfl = pa.iheat == 1 ? 1 : 0;
  double tsurf = pa.iheat == 1 ? pa.bount : 0.0;
  double tb = (1 - ihfl) * tl + ihfl * (2. * tsurf - tl);
  tb = dmax(dmin(tb, p.tuplim), p.tlolim);
  T[LB] = tb; T[LC] = tb;
  b.a[FF_VIS][LB] = vis; b.a[FF_CH][LB] = ch; b.a[FF_C][LB] = cc;
  b.a[FF_DRDP][LB] = drdp; b.a[FF_DRDH][LB] = drdh;
  b.a[FF_U][LB] = u; b.a[FF_V][LB] = v; b.a[FF_W][LB] = w;
  b.a[FF_U][LC] = u; b.a[FF_V][LC] = v; b.a[FF_W][LC] = w;
  double ro = dmax(0.001 * p.frsden, rol);
  double pb = dmax(0.001 * p.frspre, 2. * pl - plt);
  double pdb = dmax(-0.999 * p.frspre, 2. * pdl - pdlt);
  RO[LB] = ro; RO[LC] = ro; P[LB] = pb; P[LC] = pb; PD[LB] = pdb; PD[LC] = pdb;
  b.a[FF_EPS2][LB] = 1.; b.a[FF_VIST][LB] = 0.; b.a[FF_EPS2][LC] = 1.; b.a[FF_VIST][LC] = 0.;
  b.a[FF_RM][LB] = ro * u; b.a[FF_RN][LB] = ro * v; b.a[FF_RW][LB] = ro * w;
  b.a[FF_RM][LC] = ro * u; b.a[FF_RN][LC] = ro * v; b.a[FF_RW][LC] = ro * w;
  b.a[FF_E][LB] = e; b.a[FF_E][LC] = e;
  if (p.iturb >= 3) {   // turb3.f:5646-5658 (ITURB = 6)
    b.a[FF_RK][LB] = -rk;
    b.a[FF_REPS][LB] = dmax(0., 2. * re - ret);
  }
}

// mode 2: both passes, for blocks whose patches touch no cell of one another
// (BlockCtx::patch_own): a cell's two ghosts are then this thread's alone.
__global__ void k_reflec(DevBlock b, ff_params p, int mode) {
  FF_PATCH_LOOP(b)
  if (mode != 1) reflec_cell(b, p, pa, L, ls, 0);
  if (mode != 0) reflec_cell(b, p, pa, L, ls, 1);
}

// REFCEN turb3.f:5881: linear extrapolation into the first wall ghost.
__global__ void k_refcen(DevBlock b, ff_params p) {
  FF_PATCH_LOOP(b)
  if (pa.ityp < 7 || pa.ityp > 10) return;
  size_t LB = L - ls, LT = L + ls;
  const int sl[12] = {FF_RO, FF_P, FF_PDIFF, FF_E, FF_U, FF_V, FF_W, FF_RM, FF_RN, FF_RW, FF_RK, FF_REPS};
  const double lim[3] = {0.001 * p.frsden, 0.001 * p.frspre, -0.999 * p.frspre};
  const int nv = p.iturb >= 3 ? 12 : 10;   // turb3.f:6013-6027
  double x[12];
#pragma unroll
  for (int q = 0; q < 12; q++)
    if (q < nv) x[q] = 2. * b.a[sl[q]][L] - b.a[sl[q]][LT];
#pragma unroll
  for (int q = 0; q < 12; q++)
    if (q < nv) b.a[sl[q]][LB] = q < 3 ? dmax(lim[q], x[q]) : (q == 10 ? dmax(p.rklim, x[q]) : (q == 11 ? dmax(p.epslim, x[q]) : x[q]));
}

// INLET base3c.f:9223 (INLOUT 4) and OUTLET base3c.f:9595 (INLOUT 2, 3): the
// level-1 ghost update FLUCYC does before the fluxes (res3c.f:7730-7834).
__global__ void k_inlet_outlet(DevBlock b, ff_params p, int icycle) {
  FF_PATCH_LOOP(b)
  bool inl = pa.ityp == FF_BC_INL && pa.ibtype == 4;
  bool out = pa.ityp == FF_BC_OUT && (pa.ibtype == 2 || pa.ibtype == 3);
  if (!inl && !out) return;
  size_t II = L, IM1 = L - ls, IM2 = IM1 - ls;
  size_t IF1 = fg.idir == 1 ? II : II + fg.s;
  double *U = b.a[FF_U], *V = b.a[FF_V], *W = b.a[FF_W], *T = b.a[FF_TEMP], *RO = b.a[FF_RO];
  double *P = b.a[FF_P], *PD = b.a[FF_PDIFF], *E = b.a[FF_E], *RM = b.a[FF_RM], *RN = b.a[FF_RN];
  double *RW = b.a[FF_RW], *EPS2 = b.a[FF_EPS2], *VIST = b.a[FF_VIST], *VIS = b.a[FF_VIS];
  if (inl) {
    const double dpkoe = P[II], dpdif = PD[II], eps2 = EPS2[II], vist = VIST[II];
    const double r1 = icycle == 1 ? pa.bounr : RO[IM1], r2 = RO[IM2];
    EPS2[IM1] = eps2; EPS2[IM2] = eps2;
    VIST[IM1] = vist; VIST[IM2] = vist;
    double rm = pa.bounu * pa.bounr, rn = pa.bounv * pa.bounr, rw = pa.bounw * pa.bounr;
    RM[IM1] = rm; RN[IM1] = rn; RW[IM1] = rw; RM[IM2] = rm; RN[IM2] = rn; RW[IM2] = rw;
    if (icycle == 1) RO[IM1] = pa.bounr;
    T[IM1] = pa.bount; T[IM2] = pa.bount;
    P[IM1] = dpkoe; P[IM2] = dpkoe; PD[IM1] = dpdif; PD[IM2] = dpdif;
    double e = p.rgas / (p.gamma - 1.) * pa.bount;
    double u1 = rm / r1, v1 = rn / r1, w1 = rw / r1, u2 = rm / r2, v2 = rn / r2, w2 = rw / r2;
    U[IM1] = u1; V[IM1] = v1; W[IM1] = w1; U[IM2] = u2; V[IM2] = v2; W[IM2] = w2;
    double e1 = r1 * (e + .5 * (u1 * u1 + v1 * v1 + w1 * w1));
    double e2 = r2 * (e + .5 * (u2 * u2 + v2 * v2 + w2 * w2));
    if (p.iturb >= 3) {   // base3c.f:9534-9541
      b.a[FF_RK][IM1] = pa.bounrk; b.a[FF_RK][IM2] = pa.bounrk;
      b.a[FF_REPS][IM1] = pa.bounep; b.a[FF_REPS][IM2] = pa.bounep;
      e1 = e1 + pa.bounrk;
      e2 = e2 + pa.bounrk;
    }
    E[IM1] = e1; E[IM2] = e2;
    return;
  }
  // FLUCYC's local TURLIM (res3c.f:7750); FLXCYC passes the real one
  const double turlim = p.iturb >= 3 ? p.turlim : 1.e-6;
  double rk3 = pa.ibtype == 2 ? 0.7 : 1.0, rk4 = pa.ibtype == 2 ? 0.3 : 0.0;
  const double a11 = b.a[FF_A1XA + 4 * (fg.dir - 1)][IF1], a12 = b.a[FF_A1YA + 4 * (fg.dir - 1)][IF1],
               a13 = b.a[FF_A1ZA + 4 * (fg.dir - 1)][IF1];
  const double ui = U[II], vi = V[II], wi = W[II], um = U[IM1], vm = V[IM1], wm = W[IM1], ti = T[II];
  const double roi = RO[II], ro1 = RO[IM1], ro2 = RO[IM2], vis2 = VIS[IM2], e2i = EPS2[II], vti = VIST[II];
  double rk = 0., re = 0., e1 = 0., e2 = 0.;
  if (p.iturb >= 3) { rk = b.a[FF_RK][II]; re = b.a[FF_REPS][II]; e1 = E[IM1]; e2 = E[IM2]; }
  double a21, a22, a23, a31, a32, a33;
  surfvects(a11, a12, a13, a21, a22, a23, a31, a32, a33);
  double veloc = .5 * (a11 * (ui + pa.bounu) + a12 * (vi + pa.bounv) + a13 * (wi + pa.bounw));
  P[IM1] = pa.bounp; P[IM2] = pa.bounp; PD[IM1] = pa.bounpd; PD[IM2] = pa.bounpd;
  double eps2 = dmin(e2i, turlim), vist = dmin(vti, turlim * vis2);
  EPS2[IM1] = eps2; EPS2[IM2] = eps2; VIST[IM1] = vist; VIST[IM2] = vist;
  if (-veloc * fg.idir > 0.) {
    double u = roi * ui / ro1, v = vi, w = wi;
    U[IM1] = u; U[IM2] = u; V[IM1] = v; V[IM2] = v; W[IM1] = w; W[IM2] = w;
    T[IM1] = ti; T[IM2] = ti;
    RM[IM1] = ro1 * u; RM[IM2] = ro2 * u;
    RN[IM1] = ro1 * v; RN[IM2] = ro2 * v;
    RW[IM1] = ro1 * w; RW[IM2] = ro2 * w;
  } else {
    double velc1 = a11 * ui + a12 * vi + a13 * wi;
    double velc2 = a21 * pa.bounu + a22 * pa.bounv + a23 * pa.bounw;
    double velc3 = a31 * pa.bounu + a32 * pa.bounv + a33 * pa.bounw;
    double uu = a11 * velc1 + a21 * velc2 + a31 * velc3;
    double vv = a12 * velc1 + a22 * velc2 + a32 * velc3;
    double ww = a13 * velc1 + a23 * velc2 + a33 * velc3;
    double u = rk3 * um + rk4 * uu, v = rk3 * vm + rk4 * vv, w = rk3 * wm + rk4 * ww;
    U[IM1] = u; U[IM2] = u; V[IM1] = v; V[IM2] = v; W[IM1] = w; W[IM2] = w;
    T[IM1] = pa.bount; T[IM2] = pa.bount;
    RO[IM1] = pa.bounr; RO[IM2] = pa.bounr;
  }
  if (p.iturb >= 3 && -veloc * fg.idir > 0.) {   // base3c.f:10134-10146
    b.a[FF_RK][IM1] = rk; b.a[FF_RK][IM2] = rk;
    b.a[FF_REPS][IM1] = re; b.a[FF_REPS][IM2] = re;
    E[IM1] = e1 + rk;
    E[IM2] = e2 + rk;
  }
}

// MIR ns3c.f:9003 -> MIRROR gluebm.f:3911 for symmetry patches.
FF_DI void mir_cells(const DevBlock& b) {
  FF_PATCH_LOOP(b)
  if (pa.ityp != FF_BC_MIR) return;
  (void)ls;
  int kdir = fg.idir == 1 ? -1 : 1, koff = fg.idir == 1 ? 0 : 1;
  size_t IC1 = L, IT = IC1 + (size_t)koff * fg.s;
  size_t IT1 = IC1 + kdir * fg.s, IT2 = IC1 + 2 * kdir * fg.s, IC2 = IC1 - kdir * fg.s;
  double nx = b.a[FF_A1XA + 4 * (fg.dir - 1)][IT];
  double ny = b.a[FF_A1YA + 4 * (fg.dir - 1)][IT];
  double nz = b.a[FF_A1ZA + 4 * (fg.dir - 1)][IT];
  double a11 = -2. * nx * nx + 1.0, a12 = -2. * nx * ny, a13 = -2. * nx * nz;
  double a22 = -2. * ny * ny + 1.0, a23 = -2. * ny * nz, a33 = -2. * nz * nz + 1.0;
  double *U = b.a[FF_U], *V = b.a[FF_V], *W = b.a[FF_W];
  double u1 = U[IC1], v1 = V[IC1], w1 = W[IC1], u2 = U[IC2], v2 = V[IC2], w2 = W[IC2];
  const int sc[8] = {FF_TEMP, FF_E, FF_P, FF_PDIFF, FF_EPS2, FF_VIST, FF_RK, FF_REPS};
  double q1[8], q2[8];
#pragma unroll
  for (int s = 0; s < 8; s++) { q1[s] = b.a[sc[s]][IC1]; q2[s] = b.a[sc[s]][IC2]; }
  U[IT1] = a11 * u1 + a12 * v1 + a13 * w1;
  V[IT1] = a12 * u1 + a22 * v1 + a23 * w1;
  W[IT1] = a13 * u1 + a23 * v1 + a33 * w1;
  U[IT2] = a11 * u2 + a12 * v2 + a13 * w2;
  V[IT2] = a12 * u2 + a22 * v2 + a23 * w2;
  W[IT2] = a13 * u2 + a23 * v2 + a33 * w2;
#pragma unroll
  for (int s = 0; s < 8; s++) { b.a[sc[s]][IT1] = q1[s]; b.a[sc[s]][IT2] = q2[s]; }
}

// REFCOR turb3.f:6040: ghost cells with two or three ghost indices copy the
// interior edge/corner cell next to them.  One thread per cell of the twelve
// edge bars (2 x 2 ghost cells across, the corners at their ends included),
// 16 (IMAX + JMAX + KMAX + 12) threads; a corner belongs to three bars, which
// write it the same value.
__host__ __device__ inline int refcor_threads(int imax, int jmax, int kmax) {
  return 16 * (imax + jmax + kmax + 12);
}
FF_DI void refcor_cells(const DevBlock& b) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int mx[3] = {b.imax, b.jmax, b.kmax};
  int d = 0;
  for (; d < 3; d++) {
    const int len = 16 * (mx[d] + 4);
    if (t < len) break;
    t -= len;
  }
  if (d == 3) return;
  auto ghost = [&](int q, int n) { return q < 2 ? q - 1 : n + q - 1; };   // 0..3 -> -1, 0, n + 1, n + 2
  int c[3];
  c[d] = t / 16 - 1;
  c[(d + 1) % 3] = ghost(t & 3, mx[(d + 1) % 3]);
  c[(d + 2) % 3] = ghost((t >> 2) & 3, mx[(d + 2) % 3]);
  int in[3];
#pragma unroll
  for (int q = 0; q < 3; q++) in[q] = max(1, min(mx[q], c[q]));
  const size_t n = ix(b, c[0], c[1], c[2]), src = ix(b, in[0], in[1], in[2]);
  const int sl[20] = {FF_RO, FF_RM, FF_RN, FF_RW, FF_E, FF_U, FF_V, FF_W, FF_P, FF_PDIFF,
                      FF_EPS2, FF_VIST, FF_TEMP, FF_VIS, FF_CH, FF_C, FF_DRDP, FF_DRDH, FF_RK, FF_REPS};
  double x[20];
#pragma unroll
  for (int s = 0; s < 20; s++) x[s] = b.a[sl[s]][src];
#pragma unroll
  for (int s = 0; s < 20; s++) b.a[sl[s]][n] = x[s];
}

__global__ void k_mir(DevBlock b) { mir_cells(b); }
__global__ void k_refcor(DevBlock b) { refcor_cells(b); }
// Both in one launch, for blocks whose patches touch no cell of one another:
// MIR writes face ghosts and REFCOR edge and corner ghosts, both from interior
// cells.  blockIdx.y past the patches: REFCOR.
__global__ void k_refcor_mir(DevBlock b, int npatch) {
  if ((int)blockIdx.y < npatch) mir_cells(b);
  else refcor_cells(b);
}

// DERFUN turb3.f:2476 + TEMDER turb3.f:3456 (IDERI = 1) of one cell; returns STRAIN.
FF_DI double grad_cell(const DevBlock& b, int level, int K, size_t L) {
  const int IS = b.is, IL = b.il;
  const double *U = b.a[FF_U], *V = b.a[FF_V], *W = b.a[FF_W], *T = b.a[FF_TEMP];
  const double *A1 = b.a[FF_A1], *A2 = b.a[FF_A2], *A3 = b.a[FF_A3];
  const double *D1 = b.a[FF_D1], *D2 = b.a[FF_D2], *D3 = b.a[FF_D3];
  double q[4][6];   // face-weighted values of u,v,w,T on the 6 faces (m/p per dir)
  double aa[6];     // areas: 1m,1p,2m,2p,3m,3p
  const double* Dd[3] = {D1, D2, D3};
  const double* Ad[3] = {A1, A2, A3};
  const int st[3] = {1, IS, IL};
  const double* F[4] = {U, V, W, T};
#pragma unroll
  for (int d = 0; d < 3; d++) {
#pragma unroll
    for (int side = 0; side < 2; side++) {
      size_t nb = side == 0 ? L - st[d] : L + st[d];
      const double dl = Dd[d][L];
      const double dd = dl + Dd[d][nb], w1 = 2.0 * quot(dl, dd, rcp(dd)), w2 = 2.0 - w1;
      aa[2 * d + side] = side == 0 ? Ad[d][L] : Ad[d][L + st[d]];
#pragma unroll
      for (int v = 0; v < 4; v++) q[v][2 * d + side] = w2 * F[v][L] + w1 * F[v][nb];
    }
  }
  double pvol = .5 * rcp(b.a[FF_VOL][L]);
  double g[3][3];   // g[v][x] = d(u_v)/dx_x
#pragma unroll
  for (int x = 0; x < 3; x++) {
    const double* N1 = b.a[FF_A1XA + x];
    const double* N2 = b.a[FF_A2XA + x];
    const double* N3 = b.a[FF_A3XA + x];
    double n3p = N3[L + IL], n3m = N3[L], n2p = N2[L + IS], n2m = N2[L], n1p = N1[L + 1], n1m = N1[L];
#pragma unroll
    for (int v = 0; v < 3; v++)
      g[v][x] = pvol * (n3p * (aa[5] * q[v][5]) - n3m * (aa[4] * q[v][4]) + n2p * (aa[3] * q[v][3])
                        - n2m * (aa[2] * q[v][2]) + n1p * (aa[1] * q[v][1]) - n1m * (aa[0] * q[v][0]));
    bool tk = !(level == 1 && (K == 0 || K == b.kmax + 1) && b.kmax <= 1);
    if (tk)
      b.a[FF_DTDX + x][L] = pvol * (aa[5] * n3p * q[3][5] - aa[4] * n3m * q[3][4] + aa[3] * n2p * q[3][3]
                                    - aa[2] * n2m * q[3][2] + aa[1] * n1p * q[3][1] - aa[0] * n1m * q[3][0]);
  }
  double w12 = .5 * (g[0][1] - g[1][0]), w13 = .5 * (g[0][2] - g[2][0]), w23 = .5 * (g[1][2] - g[2][1]);
  b.a[FF_W12][L] = w12; b.a[FF_W13][L] = w13; b.a[FF_W23][L] = w23;
  b.a[FF_OHMI][L] = 2. * sqrt(w12 * w12 + w13 * w13 + w23 * w23);
  double s11 = g[0][0], s22 = g[1][1], s33 = g[2][2];
  double s12 = .5 * (g[0][1] + g[1][0]), s13 = .5 * (g[0][2] + g[2][0]), s23 = .5 * (g[1][2] + g[2][1]);
  b.a[FF_S11][L] = s11; b.a[FF_S12][L] = s12; b.a[FF_S13][L] = s13;
  b.a[FF_S22][L] = s22; b.a[FF_S23][L] = s23; b.a[FF_S33][L] = s33;
  double stn = s11 * s11 + 2. * s12 * s12 + 2. * s13 * s13 + s22 * s22 + 2. * s23 * s23 + s33 * s33;
  const double strain = sqrt(2. * stn);
  b.a[FF_STRAIN][L] = strain;
  return strain;
}

// DERFUN + TEMDER on the interior and, on level 1, the first ghost layer
// (laminar; k_pre_ke does it for k-omega).
__global__ void k_grad(DevBlock b, int level) {
  int lo = level == 1 ? 0 : 1, hi = level == 1 ? 1 : 0;
  int ni = b.imax + hi - lo + 1, nj = b.jmax + hi - lo + 1, nk = b.kmax + hi - lo + 1;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ni * nj * nk) return;
  int I = lo + t % ni, J = lo + (t / ni) % nj, K = lo + t / (ni * nj);
  grad_cell(b, level, K, ix(b, I, J, K));
}

// FLUXBL base3c.f:4085 (IDIFF = 1) for the face between M = L-S and L; the
// result is the viscous part of the face flux (FRO untouched).
// Face geometry both viscous face fluxes (FLUXBL, FLKEBL) read: the
// interpolation weights from the cell thicknesses D1..D3, the unit vector s
// between the two cell centres with its length and reciprocal, and the face's
// unit normal and area.  Computed once per face.
struct FaceGeom {
  double w1, w2, sx, sy, sz, slen, rslen, nx, ny, nz, area;
};

FF_DI FaceGeom face_geom(const DevBlock& b, size_t L, int S, int dir) {
#define LD(s, n) __ldg(b.a[s] + (n))
  FaceGeom g;
  const size_t M = L - S;
  const double* D = b.a[FF_D1 + dir - 1];
  const double dl = __ldg(D + L);
  g.w1 = 2.0 * (dl * rcp(dl + __ldg(D + M)));
  g.w2 = 2.0 - g.w1;
  double sx = LD(FF_XC, L) - LD(FF_XC, M), sy = LD(FF_YC, L) - LD(FF_YC, M), sz = LD(FF_ZC, L) - LD(FF_ZC, M);
  double rs_;
  sqrt_rsq(dmax(sx * sx + sy * sy + sz * sz, 1.e-300), g.slen, rs_);
  g.slen += 1.e-21;
  g.rslen = rcp(g.slen);
  g.sx = sx * g.rslen; g.sy = sy * g.rslen; g.sz = sz * g.rslen;
  const int ao = 4 * (dir - 1);
  g.nx = LD(FF_A1XA + ao, L); g.ny = LD(FF_A1YA + ao, L); g.nz = LD(FF_A1ZA + ao, L);
  g.area = LD(FF_A1 + ao, L);
#undef LD
  return g;
}

FF_DI void visc_flux(const DevBlock& b, const ff_params& p, size_t L, int S, int dir, const FaceGeom& g,
                     double f[5]) {
  size_t M = L - S;
  const double w1 = g.w1, w2 = g.w2;
  double w1p = .5 * w1, w2p = .5 * w2;
#define LD(s, n) __ldg(b.a[s] + (n))
  double s11l = LD(FF_S11, L), s11m = LD(FF_S11, M), s22l = LD(FF_S22, L), s22m = LD(FF_S22, M);
  double s33l = LD(FF_S33, L), s33m = LD(FF_S33, M), s12l = LD(FF_S12, L), s12m = LD(FF_S12, M);
  double s13l = LD(FF_S13, L), s13m = LD(FF_S13, M), s23l = LD(FF_S23, L), s23m = LD(FF_S23, M);
  double w12l = LD(FF_W12, L), w12m = LD(FF_W12, M), w13l = LD(FF_W13, L), w13m = LD(FF_W13, M);
  double w23l = LD(FF_W23, L), w23m = LD(FF_W23, M);
  double dudx = w2p * s11l + w1p * s11m, dvdy = w2p * s22l + w1p * s22m, dwdz = w2p * s33l + w1p * s33m;
  double dudy = w2p * (s12l + w12l) + w1p * (s12m + w12m);
  double dudz = w2p * (s13l + w13l) + w1p * (s13m + w13m);
  double dvdx = w2p * (s12l - w12l) + w1p * (s12m - w12m);
  double dvdz = w2p * (s23l + w23l) + w1p * (s23m + w23m);
  double dwdx = w2p * (s13l - w13l) + w1p * (s13m - w13m);
  double dwdy = w2p * (s23l - w23l) + w1p * (s23m - w23m);
  double s11i = w2 * s11l + w1 * s11m, s12i = w2 * s12l + w1 * s12m, s13i = w2 * s13l + w1 * s13m;
  double s22i = w2 * s22l + w1 * s22m, s23i = w2 * s23l + w1 * s23m, s33i = w2 * s33l + w1 * s33m;
  double dtdxi = w2p * LD(FF_DTDX, L) + w1p * LD(FF_DTDX, M);
  double dtdyi = w2p * LD(FF_DTDY, L) + w1p * LD(FF_DTDY, M);
  double dtdzi = w2p * LD(FF_DTDZ, L) + w1p * LD(FF_DTDZ, M);
  const double sxi = g.sx, syi = g.sy, szi = g.sz, rslen = g.rslen;
  const double nx = g.nx, ny = g.ny, nz = g.nz, area = g.area;
  double alfa = sxi * nx + syi * ny + szi * nz;
  double surf = 0.5 * area * (LD(FF_EPS2, L) * LD(FF_VIS, L) + LD(FF_EPS2, M) * LD(FF_VIS, M));
  const double rprt = rcp(p.prt);
  double surfe = 0.5 * area * (LD(FF_CP, L) * LD(FF_VIST, L) * rprt + LD(FF_CH, L)
                               + LD(FF_CP, M) * LD(FF_VIST, M) * rprt + LD(FF_CH, M));
  double ul = LD(FF_U, L), um = LD(FF_U, M), vl = LD(FF_V, L), vm = LD(FF_V, M), wl = LD(FF_W, L), wm = LD(FF_W, M);
  double duvwsj = nx * (dudx * sxi + dudy * syi + dudz * szi) + ny * (dvdx * sxi + dvdy * syi + dvdz * szi)
                + nz * (dwdx * sxi + dwdy * syi + dwdz * szi);
  double f2 = nx * s11i + ny * s12i + nz * s13i;
  double f3 = nx * s12i + ny * s22i + nz * s23i;
  double f4 = nx * s13i + ny * s23i + nz * s33i;
  if (alfa > 0.) {
    double adotu = nx * (ul - um) + ny * (vl - vm) + nz * (wl - wm);
    double cc = adotu * rslen - duvwsj;
    f2 = alfa * ((ul - um) * rslen - (sxi * dudx + syi * dudy + szi * dudz)) + sxi * cc + f2;
    f3 = alfa * ((vl - vm) * rslen - (sxi * dvdx + syi * dvdy + szi * dvdz)) + syi * cc + f3;
    f4 = alfa * ((wl - wm) * rslen - (sxi * dwdx + syi * dwdy + szi * dwdz)) + szi * cc + f4;
  }
  const double R23 = .6666667;
  double dv = dudx + dvdy + dwdz;
  f2 = surf * (f2 - R23 * nx * dv);
  f3 = surf * (f3 - R23 * ny * dv);
  f4 = surf * (f4 - R23 * nz * dv);
  double f5 = .5 * ((ul + um) * f2 + (vl + vm) * f3 + (wl + wm) * f4) + surfe * (dtdxi * nx + dtdyi * ny + dtdzi * nz);
  if (alfa > 0.)
    f5 = surfe * alfa * ((LD(FF_TEMP, L) - LD(FF_TEMP, M)) * rslen - sxi * dtdxi - syi * dtdyi - szi * dtdzi) + f5;
#undef LD
  f[0] = 0.; f[1] = -f2; f[2] = -f3; f[3] = -f4; f[4] = -f5;
}

FF_DI void visc_flux(const DevBlock& b, const ff_params& p, size_t L, int S, int dir, double f[5]) {
  visc_flux(b, p, L, S, dir, face_geom(b, L, S, dir), f);
}

// FLUXDO base3c.f:3677 (thin layer, IDIFF = 1): the viscous flux on coarse
// levels and whenever FULLNS is off (T = float for a coarse face pass in
// FP32).
template <typename T>
FF_DI void visc_flux_thin(const DevBlock& b, const ff_params& p, size_t L, int S, int dir, T f[5], T fe0 = T(0.)) {
#define LD(s, n) T(__ldg(b.a[s] + (n)))
  size_t M = L - S;
  const int ao = 4 * (dir - 1);
  T area = LD(FF_A1 + ao, L);
  T nx = LD(FF_A1XA + ao, L), ny = LD(FF_A1YA + ao, L), nz = LD(FF_A1ZA + ao, L);
  T surg = -area * (area / (LD(FF_VOL, L) + LD(FF_VOL, M)));
  T surf = surg * (LD(FF_EPS2, L) * LD(FF_VIS, L) + LD(FF_EPS2, M) * LD(FF_VIS, M));
  const T prt = T(p.prt);
  T surfe = surg * (LD(FF_CP, L) * LD(FF_VIST, L) / prt + LD(FF_CH, L)
                    + LD(FF_CP, M) * LD(FF_VIST, M) / prt + LD(FF_CH, M));
  T ul = LD(FF_U, L), um = LD(FF_U, M), vl = LD(FF_V, L), vm = LD(FF_V, M), wl = LD(FF_W, L), wm = LD(FF_W, M);
  T duc = T(.333333) * (nx * (ul - um) + ny * (vl - vm) + nz * (wl - wm));
  T f2 = surf * (ul - um + nx * duc);
  T f3 = surf * (vl - vm + ny * duc);
  T f4 = surf * (wl - wm + nz * duc);
  T f5 = T(.5) * ((ul + um) * f2 + (vl + vm) * f3 + (wl + wm) * f4);
  f[0] = T(0.); f[1] = f2; f[2] = f3; f[3] = f4;
  f[4] = fe0 + f5 + surfe * (LD(FF_TEMP, L) - LD(FF_TEMP, M));
#undef LD
}

// BOTSKE base3c.f:6147 wall-face flux (laminar, TURCOR false as FLUCYC passes
// it, wall at rest).  II = interior cell at the wall.
template <typename T>
FF_DI void wall_flux(const DevBlock& b, const ff_params& p, size_t II, int S, int idir, int dir,
                     int iheat, int intem, T f[5]) {
#define LD(s, n) T(__ldg(b.a[s] + (n)))
  T rc1 = intem == 6 ? T(1.) : T(1.5), rc2 = rc1 - T(1.);
  const T prs = T(p.pr) / T(p.prt), ymr = T(.166666667), eps = T(1.e-3);
  int lstrid = S * idir;
  size_t II2 = II + lstrid, IF1 = idir == 1 ? II : II + S;
  int ihfl = (iheat == 2 || iheat >= 12) ? 1 : 0;
  int iht = (iheat == 0 || iheat == 15) ? 0 : 1;
  const int ao = 4 * (dir - 1);
  T a_f = LD(FF_A1 + ao, IF1);
  T dist = (a_f + LD(FF_A1 + ao, IF1 + lstrid)) / LD(FF_VOL, II);
  T surg = -dist * ymr;
  T visb = dmax(T(0.01) * T(p.frsvis), rc1 * LD(FF_VIS, II) - rc2 * LD(FF_VIS, II2));
  T chsb = dmax(eps, rc1 * LD(FF_CH, II) - rc2 * LD(FF_CH, II2));
  // PB = YP1*PB1 + YP4*PB4 (base3c.f:6304-6315, 6487): the extrapolated
  // pressure, or its difference from FRSPRE for KT (IFLUX=7)
  T pb1 = p.flux == FF_FLUX_KT
              ? dmax(T(-.99) * T(p.frspre), rc1 * LD(FF_PDIFF, II) - rc2 * LD(FF_PDIFF, II2))
              : dmax(T(0.01) * T(p.frspre), rc1 * LD(FF_P, II) - rc2 * LD(FF_P, II2));
  T surf = surg * visb;
  T surfe = surg * (prs * T(0.) / visb + T(1.)) * chsb;
  T tempb = dmax(T(0.01) * T(p.frstem), rc1 * LD(FF_TEMP, II) - rc2 * LD(FF_TEMP, II2));
  T tsurf = iheat == 3 ? tempb : T(p.frstem);
  T cvii = T(iht * idir) * (T(9.000) * LD(FF_TEMP, II) - T(1.000) * LD(FF_TEMP, II2) - T(8.) * tsurf);
  T uvii = T(idir) * (T(9.000) * LD(FF_U, II) - T(1.000) * LD(FF_U, II2));
  T vvii = T(idir) * (T(9.000) * LD(FF_V, II) - T(1.000) * LD(FF_V, II2));
  T wvii = T(idir) * (T(9.000) * LD(FF_W, II) - T(1.000) * LD(FF_W, II2));
  T ax = LD(FF_A1XA + ao, IF1), ay = LD(FF_A1YA + ao, IF1), az = LD(FF_A1ZA + ao, IF1);
  T duc = T(.33333) * (ay * vvii + az * wvii + ax * uvii);
  T f2v = surf * (uvii + ax * duc);
  T f3v = surf * (vvii + ay * duc);
  T f4v = surf * (wvii + az * duc);
  T f5v = T(1 - ihfl) * surfe * cvii;
  f[0] = T(0.);
  f[1] = a_f * (ax * pb1 + f2v);
  f[2] = a_f * (ay * pb1 + f3v);
  f[3] = a_f * (az * pb1 + f4v);
  f[4] = a_f * f5v;
#undef LD
}

// Flux of one face (dir, cell L on the high side, normal index m).
// FLUXVL base3c.f:1733-1961 (IFLUX=0) at one face: van Leer flux-vector
// splitting of the MUSCL-extrapolated conservative variables qc[v][m]
// (v = RO, RM, RN, RW, E; cells I-2S..I+S), perfect gas, added to f.
// wps: FLUXWP base3c.f:1967-2195 (IFLUX=2), the wave/particle split of the
// subsonic momentum and energy fluxes (base3c.f:2118-2125, 2156-2163).
FF_DI void vl_flux(const double qc[5][4], double nx, double ny, double nz, double area, int intem,
                   const ff_params& p, bool wps, double f[5]) {
  const double gamma = p.gamma, gm1 = gamma - 1., ygm = 1. / gamma;
  double ip[5], im[5];
#pragma unroll
  for (int v = 0; v < 5; v++) xxtrap(qc[v][0], qc[v][1], qc[v][2], qc[v][3], intem, ip[v], im[v]);
  double ppi = (gamma - 1.) * (ip[4] - .5 / ip[0] * (ip[1] * ip[1] + ip[2] * ip[2] + ip[3] * ip[3]));
  double pmi = (gamma - 1.) * (im[4] - .5 / im[0] * (im[1] * im[1] + im[2] * im[2] + im[3] * im[3]));
  ip[0] = dmax(0.001 * p.frsden, ip[0]);
  ppi = dmax(0.001 * p.frspre, ppi);
  im[0] = dmax(0.001 * p.frsden, im[0]);
  pmi = dmax(0.001 * p.frspre, pmi);
  double a21, a22, a23, a31, a32, a33;
  surfvects(nx, ny, nz, a21, a22, a23, a31, a32, a33);
  const double rip0 = nx * ip[1] + ny * ip[2] + nz * ip[3], rip1 = a21 * ip[1] + a22 * ip[2] + a23 * ip[3],
               rip2 = a31 * ip[1] + a32 * ip[2] + a33 * ip[3];
  const double rim0 = nx * im[1] + ny * im[2] + nz * im[3], rim1 = a21 * im[1] + a22 * im[2] + a23 * im[3],
               rim2 = a31 * im[1] + a32 * im[2] + a33 * im[3];
  double fm[5], fp[5];
  {  // F- from the right state
    const double ypro = 1. / ip[0], u = ypro * rip0, v = ypro * rip1, w = ypro * rip2;
    const double pp = dmax(0.01, ppi), c = sqrt(gamma * pp * ypro), rma = u / c;
    if (rma < -1.) {
      fm[0] = area * rip0; fm[1] = area * (rip0 * u + pp); fm[2] = area * rip0 * v;
      fm[3] = area * rip0 * w; fm[4] = area * u * (ip[4] + pp);
    } else if (rma < 1.) {
      const double h = .5 * (rma - 1.), f1 = -area * ip[0] * c * (h * h);
      fm[0] = f1; fm[2] = f1 * v; fm[3] = f1 * w;
      if (wps) {
        const double rma2 = .25 * ((rma - 1.) * (rma - 1.)) * (2. + rma);
        fm[1] = f1 * u + area * pp * rma2;
        fm[4] = f1 * ip[4] * ypro + area * u * pp * rma2;
      } else {
        fm[1] = f1 * (gm1 * u - 2. * c) * ygm;
        fm[4] = f1 * (ip[4] + pp) * ypro;
      }
    } else {
      fm[0] = fm[1] = fm[2] = fm[3] = fm[4] = 0.;
    }
  }
  {  // F+ from the left state
    const double ypro = 1. / im[0], u = ypro * rim0, v = ypro * rim1, w = ypro * rim2;
    const double pm = dmax(0.01, pmi), c = sqrt(gamma * pm * ypro), rma = u / c;
    if (rma > 1.) {
      fp[0] = area * rim0; fp[1] = area * (rim0 * u + pm); fp[2] = area * rim0 * v;
      fp[3] = area * rim0 * w; fp[4] = area * u * (im[4] + pm);
    } else if (rma > -1.) {
      const double h = .5 * (rma + 1.), f1 = +area * im[0] * c * (h * h);
      fp[0] = f1; fp[2] = f1 * v; fp[3] = f1 * w;
      if (wps) {
        const double rma2 = .25 * ((rma + 1.) * (rma + 1.)) * (2. - rma);
        fp[1] = f1 * u + area * pm * rma2;
        fp[4] = f1 * im[4] * ypro + area * u * pm * rma2;
      } else {
        fp[1] = f1 * (gm1 * u + 2. * c) * ygm;
        fp[4] = f1 * (im[4] + pm) * ypro;
      }
    } else {
      fp[0] = fp[1] = fp[2] = fp[3] = fp[4] = 0.;
    }
  }
  const double f2 = fp[1] + fm[1], f3 = fp[2] + fm[2], f4 = fp[3] + fm[3];
  f[0] = fm[0] + fp[0] + f[0];
  f[1] = nx * f2 + a21 * f3 + a31 * f4 + f[1];
  f[2] = ny * f2 + a22 * f3 + a32 * f4 + f[2];
  f[3] = nz * f2 + a23 * f3 + a33 * f4 + f[3];
  f[4] = fm[4] + fp[4] + f[4];
}

#include "ff_fluxes.cuh"

// JAMESON base3c.f:2827-3019 (IPRESC = 0) at face L (cells L-S | L): the
// pressure sensors of the two cells (second differences of PDIFF), EPS2 =
// RJK2 * their max, EPS4 = max(0, RJK4 - EPS2), SCALEJ averaged to the face;
// the second- and fourth-difference dissipation of RO, RM, RN, RW, E taken
// off f.  Added to Roe's flux on the finest level when RJK2 or RJK4 > 0
// (FLUCYC res3c.f:7899-7906, RESIKE 6955-6962); k and omega keep theirs.
FF_DI void jst_flux(const DevBlock& b, const ff_params& p, size_t L, int S, double* f) {
  const double* PD = b.a[FF_PDIFF];
  const double pd0 = __ldg(PD + L - 2 * S), pd1 = __ldg(PD + L - S), pd2 = __ldg(PD + L), pd3 = __ldg(PD + L + S);
  const double fp4 = 4. * p.frspre;
  const double pres1 = fabs(pd2 - 2. * pd1 + pd0) / (pd2 + 2. * pd1 + pd0 + fp4);
  const double pres2 = fabs(pd3 - 2. * pd2 + pd1) / (pd3 + 2. * pd2 + pd1 + fp4);
  const double eps2 = p.rjk2 * dmax(pres1, pres2), eps4 = dmax(0., p.rjk4 - eps2);
  const double rlami = .5 * (__ldg(b.a[FF_SCALEJ] + L) + __ldg(b.a[FF_SCALEJ] + L - S));
  const int sl[5] = {FF_RO, FF_RM, FF_RN, FF_RW, FF_E};
#pragma unroll
  for (int v = 0; v < 5; v++) {
    const double* q = b.a[sl[v]];
    const double q0 = __ldg(q + L - 2 * S), q1 = __ldg(q + L - S), q2 = __ldg(q + L), q3 = __ldg(q + L + S);
    f[v] = -(rlami * (eps2 * (q2 - q1) - eps4 * (q3 - 3. * q2 + 3. * q1 - q0))) + f[v];
  }
}

// SCALARD base3c.f:6-78 (IPRESC = 0, no grid rotation): SCALEJ of cells
// 0..MAX+1 in each direction, |(U,V,W) . mean face vectors| + C * the mean
// face areas; the JAMESON dissipation scale.
__global__ void k_scalard(DevBlock b) {
  const int ni = b.imax + 2, nj = b.jmax + 2;
  const long n = (long)ni * nj * (b.kmax + 2);
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int I = t % ni, J = (t / ni) % nj, K = t / ((long)ni * nj);
  const size_t kk = ix(b, I, J, K), is = b.is, il = b.il;
#define LD(s, n) __ldg(b.a[s] + (n))
  const double a1 = LD(FF_A1, kk), a1p = LD(FF_A1, kk + 1), a2 = LD(FF_A2, kk), a2p = LD(FF_A2, kk + is);
  const double a3 = LD(FF_A3, kk), a3p = LD(FF_A3, kk + il);
  const double a1k = .5 * (a1 + a1p), a2k = .5 * (a2 + a2p), a3k = .5 * (a3 + a3p);
  const double a1xk = .5 * (LD(FF_A1XA, kk) * a1 + LD(FF_A1XA, kk + 1) * a1p);
  const double a1yk = .5 * (LD(FF_A1YA, kk) * a1 + LD(FF_A1YA, kk + 1) * a1p);
  const double a1zk = .5 * (LD(FF_A1ZA, kk) * a1 + LD(FF_A1ZA, kk + 1) * a1p);
  const double a2xk = .5 * (LD(FF_A2XA, kk) * a2 + LD(FF_A2XA, kk + is) * a2p);
  const double a2yk = .5 * (LD(FF_A2YA, kk) * a2 + LD(FF_A2YA, kk + is) * a2p);
  const double a2zk = .5 * (LD(FF_A2ZA, kk) * a2 + LD(FF_A2ZA, kk + is) * a2p);
  const double a3xk = .5 * (LD(FF_A3XA, kk) * a3 + LD(FF_A3XA, kk + il) * a3p);
  const double a3yk = .5 * (LD(FF_A3YA, kk) * a3 + LD(FF_A3YA, kk + il) * a3p);
  const double a3zk = .5 * (LD(FF_A3ZA, kk) * a3 + LD(FF_A3ZA, kk + il) * a3p);
  const double u = LD(FF_U, kk), v = LD(FF_V, kk), w = LD(FF_W, kk);
  const double ucii = a1xk * u + a1yk * v + a1zk * w, vcii = a2xk * u + a2yk * v + a2zk * w;
  const double wcii = a3xk * u + a3yk * v + a3zk * w;
  b.a[FF_SCALEJ][kk] = sqrt(ucii * ucii + vcii * vcii + wcii * wcii) + (a1k + a2k + a3k) * LD(FF_C, kk);
#undef LD
}

// sq (optional): RO, U, V, W, P of cell L in a staged stencil, variable v
// at sq[v * vs], the cells along the face normal es apart.  T = float: a
// coarse level's face in FP32 (loads converted, fluxes in FP32).
// ALT = false compiles out the selectable variants (the other IFLUX schemes,
// XXTRAA, JAMESON) for the residual kernels of the plain Roe/XXTRAP case:
// their code would raise the register count of every face.
template <typename T, bool ALT = true>
FF_DI void face_flux(const DevBlock& b, const ff_params& p, int dir, size_t L, int m, int t1, int t2,
                     int level, T f[5], const double* sq = nullptr, int es = 0, int vs = 0) {
  const int S = dir == 1 ? 1 : (dir == 2 ? b.is : b.il);
  const int nmax = dir == 1 ? b.imax : (dir == 2 ? b.jmax : b.kmax);
  int intem = dir == 1 ? p.interi : (dir == 2 ? p.interj : p.interk);
  if (level > 1) intem = p.coarse_inter;
  // wall face?  (BOTSKE overwrites, res3c.f:8092)
  if (m == 1 || m == nmax + 1) {
    int iface = m == 1 ? dir : dir + 3;
    for (int ip = 0; ip < b.npatch; ip++) {
      const ff_patch& pa = b.patch[ip];
      if (pa.iface != iface || pa.ityp < 8 || pa.ityp > 10) continue;
      if (t1 < pa.r1a || t1 > pa.r1b || t2 < pa.r2a || t2 > pa.r2b) continue;
      int idir = m == 1 ? 1 : -1;
      size_t II = m == 1 ? L : L - S;
      wall_flux(b, p, II, S, idir, dir, pa.iheat, intem, f);
      return;
    }
  }
  const int idi = dir == 1 ? p.idi1 : (dir == 2 ? p.idi2 : p.idi3);
  if (m <= min(idi, nmax + 1)) {   // SINVIS base3c.f:3876: viscous faces
    bool full = false;
    if constexpr (sizeof(T) == sizeof(double)) {
      if (level == 1 && p.fullns) { visc_flux(b, p, L, S, dir, f); full = true; }
    }
    if (!full) visc_flux_thin(b, p, L, S, dir, f);
  } else {
    f[0] = f[1] = f[2] = f[3] = f[4] = T(0.);
  }
  const int ao = 4 * (dir - 1);
  if constexpr (ALT && sizeof(T) == sizeof(double)) {
    if (p.flux != FF_FLUX_ROE) {   // the other IFLUX schemes (FLUCYC res3c.f:7890-7990)
      alt_flux<5>(b, p, dir, L, S, intem, 1, f);
      return;
    }
  }
  T q[5][4];
  const int sl[5] = {FF_RO, FF_U, FF_V, FF_W, FF_P};
  if (sq) {
#pragma unroll
    for (int v = 0; v < 5; v++) {
      const double* a = sq + v * vs;
      q[v][0] = T(a[-2 * es]); q[v][1] = T(a[-es]); q[v][2] = T(a[0]); q[v][3] = T(a[es]);
    }
  } else {
#pragma unroll
    for (int v = 0; v < 5; v++) {
      const double* a = b.a[sl[v]];
      q[v][0] = T(__ldg(a + L - 2 * S)); q[v][1] = T(__ldg(a + L - S)); q[v][2] = T(__ldg(a + L));
      q[v][3] = T(__ldg(a + L + S));
    }
  }
  size_t L2 = dir == 3 ? L : L - S;
  T cr[4] = {T(__ldg(b.a[FF_DRDP] + L)), T(__ldg(b.a[FF_DRDH] + L)), q[0][2], q[4][2]};
  // RO and P of cell L2 (L itself for k faces) are in the stencil
  T cl[4] = {T(__ldg(b.a[FF_DRDP] + L2)), T(__ldg(b.a[FF_DRDH] + L2)), dir == 3 ? q[0][2] : q[0][1],
             dir == 3 ? q[4][2] : q[4][1]};
  if constexpr (ALT && sizeof(T) == sizeof(double)) {
    if (p.xxtral) {   // XXTRAA over the cells' extents along the normal
      const double* D = b.a[FF_D1 + dir - 1];
      const double dd[4] = {__ldg(D + L - 2 * S), __ldg(D + L - S), __ldg(D + L), __ldg(D + L + S)};
      roe_flux<double, true>(q, __ldg(b.a[FF_A1XA + ao] + L), __ldg(b.a[FF_A1YA + ao] + L),
                             __ldg(b.a[FF_A1ZA + ao] + L), __ldg(b.a[FF_A1 + ao] + L), intem, p, __ldg(b.a[FF_C] + L),
                             __ldg(b.a[FF_C] + L - S), cr, cl, f, dd);
    } else {
      roe_flux(q, __ldg(b.a[FF_A1XA + ao] + L), __ldg(b.a[FF_A1YA + ao] + L), __ldg(b.a[FF_A1ZA + ao] + L),
               __ldg(b.a[FF_A1 + ao] + L), intem, p, __ldg(b.a[FF_C] + L), __ldg(b.a[FF_C] + L - S), cr, cl, f);
    }
    if (level == 1 && (p.rjk2 > 0. || p.rjk4 > 0.)) jst_flux(b, p, L, S, f);
    return;
  }
  roe_flux(q, T(__ldg(b.a[FF_A1XA + ao] + L)), T(__ldg(b.a[FF_A1YA + ao] + L)), T(__ldg(b.a[FF_A1ZA + ao] + L)),
           T(__ldg(b.a[FF_A1 + ao] + L)), intem, p, T(__ldg(b.a[FF_C] + L)), T(__ldg(b.a[FF_C] + L - S)), cr, cl, f);
}

// RESIDU: fused k, i, j face fluxes and SWEEP res3c.f:992 for a 32x4x4 tile.
// NT threads per CTA (128, 256 or 512): each thread sums the faces of
// CPT = 512 / NT cells of the 32x4x4 tile (a k column of CPT cells); the
// register budget gives RES_MIN_CTAS * 128 threads per SM at every NT.
template <int NT>
__global__ void __launch_bounds__(NT, RES_MIN_CTAS * 128 / NT) k_residual(DevBlock b, ff_params p, int level) {
  constexpr int CPT = TI * TJ * TK / NT;
  constexpr int NF = TI * (TJ + 1) * TK, NC = TI * TJ * TK;
  // one direction's faces (at most 640) x 5, then the cells' running sums
  // (in shared memory, not registers: the face flux needs the registers)
  extern __shared__ double res_smem[];
  double(*sF)[NF] = reinterpret_cast<double(*)[NF]>(res_smem);
  double(*sAcc)[NC] = reinterpret_cast<double(*)[NC]>(res_smem + 5 * NF);
  const int tid = threadIdx.x;
  const int i0 = blockIdx.x * TI, j0 = blockIdx.y * TJ, k0 = blockIdx.z * TK;
  const int ci = tid % TI, cj = (tid / TI) % TJ, ck0 = (tid / (TI * TJ)) * CPT;
#pragma unroll
  for (int c = 0; c < CPT; c++)
#pragma unroll
    for (int v = 0; v < 5; v++) sAcc[v][ci + TI * (cj + TJ * (ck0 + c))] = 0.;
  // the directions in SWEEP order (k, i, j; res3c.f:355); one call site of the
  // face flux keeps a single copy of its code in the instruction stream
#pragma unroll 1
  for (int pass = 0; pass < 3; pass++) {
    const int dir = pass == 0 ? 3 : pass;   // k, i, j
    const int ni = TI + (dir == 1), nj = TJ + (dir == 2), nk = TK + (dir == 3);
    for (int f = tid; f < ni * nj * nk; f += blockDim.x) {
      const int fi = f % ni, fj = (f / ni) % nj, fk = f / (ni * nj);
      const int I = i0 + fi + 1, J = j0 + fj + 1, K = k0 + fk + 1;
      if (I > b.imax + (dir == 1) || J > b.jmax + (dir == 2) || K > b.kmax + (dir == 3)) continue;
      const int m = dir == 1 ? I : (dir == 2 ? J : K);
      const int t1 = dir == 1 ? J : I, t2 = dir == 3 ? J : K;
      double fl[5];
      face_flux(b, p, dir, ix(b, I, J, K), m, t1, t2, level, fl);
#pragma unroll
      for (int v = 0; v < 5; v++) sF[v][f] = fl[v];
    }
    __syncthreads();
    const int fs = dir == 1 ? 1 : (dir == 2 ? ni : ni * nj);   // low face -> high face of a cell
#pragma unroll
    for (int c = 0; c < CPT; c++) {
      const int f0 = ci + ni * (cj + nj * (ck0 + c));
      const int I = i0 + ci + 1, J = j0 + cj + 1, K = k0 + ck0 + c + 1;
      if (I > b.imax || J > b.jmax || K > b.kmax) continue;
      const int ca = ci + TI * (cj + TJ * (ck0 + c));
      if (pass < 2) {
#pragma unroll
        for (int v = 0; v < 5; v++) sAcc[v][ca] = sAcc[v][ca] - (sF[v][f0 + fs] - sF[v][f0]);
      } else {   // last direction, then 1/VOL (SWEEP IDO = 1)
        const size_t n = ix(b, I, J, K);
        const double rv = 1. / __ldg(b.a[FF_VOL] + n);
#pragma unroll
        for (int v = 0; v < 5; v++) b.a[FF_DRO + v][n] = (sAcc[v][ca] - (sF[v][f0 + fs] - sF[v][f0])) * rv;
      }
    }
    __syncthreads();
  }
}

// Sum of squares (RESL2 res3c.f:8920) of the five residuals into out[0..4].
__global__ void k_resl2(DevBlock b, double* out) {
  __shared__ double red[5][8];
  double s[5] = {0, 0, 0, 0, 0};
  int n_int = b.imax * b.jmax * b.kmax;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n_int; t += gridDim.x * blockDim.x) {
    int I = t % b.imax + 1, J = (t / b.imax) % b.jmax + 1, K = t / (b.imax * b.jmax) + 1;
    size_t n = ix(b, I, J, K);
#pragma unroll
    for (int v = 0; v < 5; v++) { double d = b.a[FF_DRO + v][n]; s[v] += d * d; }
  }
#pragma unroll
  for (int v = 0; v < 5; v++) {
    double x = s[v];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31) == 0) red[v][threadIdx.x >> 5] = x;
  }
  __syncthreads();
  if (threadIdx.x < 5) {
    double x = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) x += red[threadIdx.x][w];
    atomicAdd(out + threadIdx.x, x);
  }
}

// What TIME3 divides by that is the same for all cells, inverted once.
struct TimeConst {
  double rcfl, rdiff, prt;   // 1 / CFL of the level, 1 / CDIFF, PR / PRT
};

// TIME3 base3c.f:79 (interior cell I, J, K at kk): the local time step.
FF_DI double time3_cell(const DevBlock& b, const ff_params& p, const TimeConst& tc, int I, int J, int K, size_t kk) {
  const int IS = b.is, IL = b.il;
#define LD(s, n) __ldg(b.a[s] + (n))
  double a1 = LD(FF_A1, kk), a1p = LD(FF_A1, kk + 1), a2 = LD(FF_A2, kk), a2p = LD(FF_A2, kk + IS);
  double a3 = LD(FF_A3, kk), a3p = LD(FF_A3, kk + IL);
  double zz = 0.;
  if (p.idi1 != 0 && I <= min(p.idi1, b.imax)) zz = .5 * (a1 + a1p);
  if (p.idi2 != 0 && J <= min(p.idi2, b.jmax)) zz = dmax(.5 * (a2 + a2p), zz);
  if (p.idi3 != 0 && K <= min(p.idi3, b.kmax)) zz = dmax(.5 * (a3 + a3p), zz);
  double ro = b.a[FF_RO][kk], u = b.a[FF_U][kk], v = b.a[FF_V][kk], w = b.a[FF_W][kk];
  double c = b.a[FF_C][kk], P = b.a[FF_P][kk];
  double pvol = rcp(LD(FF_VOL, kk)), ypro = rcp(ro + 1.e-10);
  double a1k = .5 * (a1 + a1p), a2k = .5 * (a2 + a2p), a3k = .5 * (a3 + a3p);
  double ucii = .5 * (LD(FF_A1XA, kk) * a1 + LD(FF_A1XA, kk + 1) * a1p) * u
              + .5 * (LD(FF_A1YA, kk) * a1 + LD(FF_A1YA, kk + 1) * a1p) * v
              + .5 * (LD(FF_A1ZA, kk) * a1 + LD(FF_A1ZA, kk + 1) * a1p) * w;
  double vcii = .5 * (LD(FF_A2XA, kk) * a2 + LD(FF_A2XA, kk + IS) * a2p) * u
              + .5 * (LD(FF_A2YA, kk) * a2 + LD(FF_A2YA, kk + IS) * a2p) * v
              + .5 * (LD(FF_A2ZA, kk) * a2 + LD(FF_A2ZA, kk + IS) * a2p) * w;
  double wcii = .5 * (LD(FF_A3XA, kk) * a3 + LD(FF_A3XA, kk + IL) * a3p) * u
              + .5 * (LD(FF_A3YA, kk) * a3 + LD(FF_A3YA, kk + IL) * a3p) * v
              + .5 * (LD(FF_A3ZA, kk) * a3 + LD(FF_A3ZA, kk + IL) * a3p) * w;
#undef LD
  double ar, rar;
  sqrt_rsq(dmax(a1k * a1k + a2k * a2k + a3k * a3k, 1.e-300), ar, rar);
  double b1 = pvol * (fabs(ucii) + fabs(vcii) + fabs(wcii) + c * ar) * tc.rcfl;
  double rnum = zz * zz * (pvol * pvol) * ypro;
  double tt = rnum * (b.a[FF_VIS][kk] + tc.prt * b.a[FF_VIST][kk]) * tc.rdiff;
  double b11 = dmax(b1, 2. * tt * p.pvisc);
  double denlow = 1. + dmax(0., (p.frspre - 2. * P) * rcp_any(P));   // infinite for P = 0
  double denmax = 1. + dmax(0., (ro - 2. * p.frsden) * ypro) * 5.;
  double dtl = rcp_any(b11 * dmax(denlow, denmax));
  if (p.timel) dtl = dtl * p.dt / (1.5 * dtl + p.dt);   // TIMEL dual time step, base3c.f:206-215
  return dtl;
}

// LOCDT imps3.f:784 + COPR imps3.f:891: the residual of cell kk times the time
// step in primitive increments.
FF_DI void copr_cell(const DevBlock& b, double dtl, size_t kk, double x[5]) {
  double dri = dtl * b.a[FF_DRO][kk], dmi = dtl * b.a[FF_DM][kk], dni = dtl * b.a[FF_DN][kk];
  double dwi = dtl * b.a[FF_DW][kk], dre = dtl * b.a[FF_DE][kk];
  double ro = b.a[FF_RO][kk], u = b.a[FF_U][kk], v = b.a[FF_V][kk], w = b.a[FF_W][kk], c = b.a[FF_C][kk];
  double yp = rcp(ro), drodh = b.a[FF_DRDH][kk], drodp = b.a[FF_DRDP][kk];
  double beta = .5 * (u * u + v * v + w * w);
  double dkin = u * dmi + v * dni + w * dwi;
  double hi = yp * (b.a[FF_E][kk] + b.a[FF_P][kk]);
  double dei = dre - (hi - 2 * beta) * dri - dkin;
  double dpi = c * c * (dri - drodh * yp * dei);
  x[0] = (dri - drodp * dpi) * rcp(drodh);
  x[1] = yp * (-u * dri + dmi);
  x[2] = yp * (-v * dri + dni);
  x[3] = yp * (-w * dri + dwi);
  x[4] = dpi;
}

// TIME3 + LOCDT + COPR in place (the sweeps that work on DRO..DE; the warp
// wavefront takes them in k_flow_coef).  mode 1: TIME3 only (the two-equation
// path converts in k_locdtk_imsoko_coprke).
__global__ void k_time3_copr(DevBlock b, ff_params p, TimeConst tc, int mode = 0) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= b.imax * b.jmax * b.kmax) return;
  int I = t % b.imax + 1, J = (t / b.imax) % b.jmax + 1, K = t / (b.imax * b.jmax) + 1;
  const size_t kk = ix(b, I, J, K);
  const double dtl = time3_cell(b, p, tc, I, J, K, kk);
  if (mode == 1) { b.a[FF_DTL][kk] = dtl; return; }
  double x[5];
  copr_cell(b, dtl, kk, x);
  b.a[FF_DTL][kk] = dtl;
#pragma unroll
  for (int v = 0; v < 5; v++) b.a[FF_DRO + v][kk] = x[v];
}

// LU-SGS coefficients of one interior cell (PREDGS imps4.f:388-470 for
// upper=1, CORRGS imps4.f:120-200 + DIAGGS imps4.f:604 for upper=0): the
// split eigenvalue coefficients x[d][0..2] of the face the cell's product in
// direction d crosses, DT1 = THETA*DTL, the scalings SCINV / SCINP and the
// diagonal factor of the lower sweep.
struct CellCoef {
  double x[3][3], dt1, scinv, scinp, fdiag;
};

FF_DI void lusgs_cell_coef(const DevBlock& b, const ff_params& p, int I, int J, int K, int upper, CellCoef& cc) {
  const int IS = b.is, IL = b.il;
  size_t N = ix(b, I, J, K);
#define LD(s, n) __ldg(b.a[s] + (n))
  double u = LD(FF_U, N), v = LD(FF_V, N), w = LD(FF_W, N), c = LD(FF_C, N), ro = LD(FF_RO, N);
  double vol = LD(FF_VOL, N), mu = LD(FF_VIST, N) + LD(FF_VIS, N);
  const int st[3] = {1, IS, IL};
  const int idi[3] = {p.idi1, p.idi2, p.idi3};
  const int idx[3] = {I, J, K};
  double xa[3], rmax_lo[3];
  for (int d = 0; d < 3; d++) {
    const int ao = 4 * d;
    size_t fN = upper ? N : N + st[d];          // face normal used for the eigenvalue
    size_t nb = upper ? N - st[d] : N + st[d];  // cell across that face
    double ff = 2.;
    if (upper && idx[d] == 1) ff = 4.;
    if (idx[d] > idi[d]) ff = 0.;
    double rl1 = LD(FF_A1XA + ao, fN) * u + LD(FF_A1YA + ao, fN) * v + LD(FF_A1ZA + ao, fN) * w;
    double rnum = (vol + LD(FF_VOL, nb)) * (ro + LD(FF_RO, nb));
    double tt = (ff * 2.) * LD(FF_A1 + ao, N) / rnum * (mu + LD(FF_VIST, nb) + LD(FF_VIS, nb));
    double rmax = fabs(rl1) + c;
    double sg = upper ? -1. : 1.;
    cc.x[d][0] = (rl1 + sg * rmax) * .5 + sg * tt;
    cc.x[d][1] = (rl1 + c + sg * rmax) * .5 + sg * tt;
    cc.x[d][2] = (rl1 - c + sg * rmax) * .5 + sg * tt;
    xa[d] = rmax + tt;
    // SCINP uses the spectral radius of the eigenvalue face in both sweeps
    rmax_lo[d] = fabs(rl1) + c;
  }
  double dt1 = p.theta * LD(FF_DTL, N);
  double a1 = LD(FF_A1, N), a2 = LD(FF_A2, N), a3 = LD(FF_A3, N);
  double a1p = LD(FF_A1, N + 1), a2p = LD(FF_A2, N + IS), a3p = LD(FF_A3, N + IL);
  cc.dt1 = dt1;
  cc.scinv = upper ? 1. / (vol + dt1 * (xa[0] * a1 + xa[1] * a2 + xa[2] * a3))
                   : 1. / (vol + dt1 * (xa[0] * a1p + xa[1] * a2p + xa[2] * a3p));
  cc.scinp = 1. / (vol + dt1 * (rmax_lo[0] * a1 + rmax_lo[1] * a2 + rmax_lo[2] * a3));
  cc.fdiag = 1.;
  if (!upper) {   // DIAGGS imps4.f:614-660
    double r[6];
    for (int d = 0; d < 3; d++) {
      const int ao = 4 * d;
      size_t fp = N + st[d];
      r[2 * d] = fabs(LD(FF_A1XA + ao, N) * u + LD(FF_A1YA + ao, N) * v + LD(FF_A1ZA + ao, N) * w) + c;
      r[2 * d + 1] = fabs(LD(FF_A1XA + ao, fp) * u + LD(FF_A1YA + ao, fp) * v + LD(FF_A1ZA + ao, fp) * w) + c;
    }
    double sc = .5 * (a1 * r[0] + a1p * r[1] + a2 * r[2] + a2p * r[3] + a3 * r[4] + a3p * r[5]);
    cc.fdiag = 1. + p.theta * LD(FF_DTL, N) / vol * sc;
  }
#undef LD
}

// Coefficients in the storage layout, coef[c*ntot + n], c = xi(3) xj(3)
// xk(3) dt1 scinv scinp fdiag (the allocation-free stage's sweep).
template <typename CT>
__global__ void k_lusgs_coef(DevBlock b, ff_params p, CT* coef, int upper) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= b.imax * b.jmax * b.kmax) return;
  int I = t % b.imax + 1, J = (t / b.imax) % b.jmax + 1, K = t / (b.imax * b.jmax) + 1;
  CellCoef cc;
  lusgs_cell_coef(b, p, I, J, K, upper, cc);
  size_t nt = b.ntot, N = ix(b, I, J, K);
  for (int d = 0; d < 3; d++)
    for (int e = 0; e < 3; e++) coef[(3 * d + e) * nt + N] = (CT)cc.x[d][e];
  coef[9 * nt + N] = (CT)cc.dt1;
  coef[10 * nt + N] = (CT)cc.scinv;
  coef[11 * nt + N] = (CT)cc.scinp;
  coef[12 * nt + N] = (CT)cc.fdiag;
}

// The static part of one sweep's layout (see sw_index): the unit normals
// of the three products' faces, the areas and the volume -- the metrics
// only, written once per block.
template <typename CT>
__global__ void k_sweep_static(DevBlock b, CT* sw, int upper) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t row = (size_t)(b.imax + b.jmax - 1) * b.jmax;
  if (t >= row * b.kmax) return;
  const int K = (int)(t / row) + 1;
  const int r = (int)(t % row), J = r % b.jmax + 1, I = r / b.jmax + 2 - J;
  if (I < 1 || I > b.imax) return;
  const size_t ns = sw_size(b.imax, b.jmax, b.kmax), S = sw_index(b, I, J, K);
  const size_t N = ix(b, I, J, K);
  const int IS = b.is, IL = b.il;
  const int st[3] = {1, IS, IL};
  sw[SW_VOL * ns + S] = (CT)__ldg(b.a[FF_VOL] + N);
  sw[SW_A1 * ns + S] = (CT)__ldg(b.a[FF_A1] + (upper ? N + 1 : N));
  sw[SW_A2 * ns + S] = (CT)__ldg(b.a[FF_A2] + (upper ? N + IS : N));
  sw[SW_A3 * ns + S] = (CT)__ldg(b.a[FF_A3] + (upper ? N + IL : N));
  for (int d = 0; d < 3; d++) {
    const int ao = 4 * d;
    size_t fN = upper ? N : N + st[d];   // the face the product in direction d crosses
    sw[(SW_F + 3 * d + 0) * ns + S] = (CT)__ldg(b.a[FF_A1XA + ao] + fN);
    sw[(SW_F + 3 * d + 1) * ns + S] = (CT)__ldg(b.a[FF_A1YA + ao] + fN);
    sw[(SW_F + 3 * d + 2) * ns + S] = (CT)__ldg(b.a[FF_A1ZA + ao] + fN);
  }
}

// The state-dependent part of one sweep's layout (see sw_index; the static
// part is k_sweep_static's), and for the first sweep (upper = 1) the
// right-hand side DRO..DE(,DRK,DEPS) copied into dwp in the same layout and
// type.
template <typename CT>
__global__ void k_sweep_coef(DevBlock b, ff_params p, CT* sw, CT* dwp, int upper) {
  // one thread per slot of the sweep layout, in slot order, so that the
  // ~50 stores of a warp are contiguous; slots outside the block (I < 1 or
  // I > IMAX on a diagonal) have no cell
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t row = (size_t)(b.imax + b.jmax - 1) * b.jmax;
  if (t >= row * b.kmax) return;
  const int K = (int)(t / row) + 1;
  const int r = (int)(t % row), J = r % b.jmax + 1, I = r / b.jmax + 2 - J;
  if (I < 1 || I > b.imax) return;
  CellCoef cc;
  lusgs_cell_coef(b, p, I, J, K, upper, cc);
  const size_t ns = sw_size(b.imax, b.jmax, b.kmax), S = sw_index(b, I, J, K);
  const size_t N = ix(b, I, J, K);
  sw[SW_DT1 * ns + S] = (CT)cc.dt1;
  sw[SW_SCINV * ns + S] = (CT)cc.scinv;
  sw[SW_SCINP * ns + S] = (CT)cc.scinp;
  sw[SW_FD * ns + S] = (CT)cc.fdiag;
  CT ro = (CT)__ldg(b.a[FF_RO] + N), c = (CT)__ldg(b.a[FF_C] + N);
  sw[SW_RO * ns + S] = ro;
  CT ypro = CT(1) / ro;
  sw[(SW_SC + 0) * ns + S] = ypro;
  sw[(SW_SC + 1) * ns + S] = ro * c;
  sw[(SW_SC + 2) * ns + S] = (CT(.5) * ypro) / c;
  if (p.iturb >= 3) {
    CT rk = (CT)__ldg(b.a[FF_RK] + N), drdp = (CT)__ldg(b.a[FF_DRDP] + N), drdh = (CT)__ldg(b.a[FF_DRDH] + N);
    sw[(SW_SC + 3) * ns + S] = CT(.667) * rk * (ypro * ypro) * drdh;
    sw[(SW_SC + 4) * ns + S] = CT(1) / (CT(1) + CT(.667) * rk * ypro * drdp);
  }
  for (int d = 0; d < 3; d++)
    for (int e = 0; e < 3; e++) sw[(SW_L + 3 * d + e) * ns + S] = (CT)cc.x[d][e];
  if (upper) {
    const int nv = p.iturb >= 3 ? 7 : 5;
    for (int v = 0; v < nv; v++) dwp[v * ns + S] = (CT)b.a[FF_DRO + v][N];
  }
}

// The increments back from the sweep layout into DRO..DE(,DRK,DEPS).
template <typename CT>
__global__ void k_sweep_out(DevBlock b, const CT* __restrict__ dwp, int nv) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= b.imax * b.jmax * b.kmax) return;
  int I = t % b.imax + 1, J = (t / b.imax) % b.jmax + 1, K = t / (b.imax * b.jmax) + 1;
  const size_t ns = sw_size(b.imax, b.jmax, b.kmax), S = sw_index(b, I, J, K);
  const size_t N = ix(b, I, J, K);
  for (int v = 0; v < nv; v++) b.a[FF_DRO + v][N] = (double)dwp[v * ns + S];
}

// One LU-SGS sweep as i+j+k hyperplanes (cooperative, persistent).  The
// triangular system is the reference's (PREDGS: neighbours i+1, j+1, k+1 with
// the reference's dropped i+1 coupling in row J = JMAX, imps4.f:547-559;
// CORRGS: i-1, j-1, k-1), so the result equals its slab-by-slab order.
// dw: increment arrays (5 x ntot) of type CT; read through L2 (__ldcg)
// because other blocks write them during the sweep.
template <typename CT, int NV>
__global__ void k_lusgs_sweep_basic(DevBlock b, const CT* __restrict__ coef, CT* dw, int upper,
                                    unsigned* bar, int* err) {
  const int IMAX = b.imax, JMAX = b.jmax, KMAX = b.kmax, IS = b.is, IL = b.il;
  const size_t nt = b.ntot;
  const int nthreads = gridDim.x * blockDim.x;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nplanes = IMAX + JMAX + KMAX - 2;
  for (int s = 0; s < nplanes; s++) {
    int m = upper ? IMAX + JMAX + KMAX - s : 3 + s;
    int klo = max(1, m - IMAX - JMAX), khi = min(KMAX, m - 2);
    int npairs = (khi - klo + 1) * JMAX;
    for (int q = tid; q < npairs; q += nthreads) {
      int K = klo + q / JMAX, J = q % JMAX + 1, I = m - J - K;
      if (I < 1 || I > IMAX) continue;
      size_t N = ix(b, I, J, K);
      CT dt1 = coef[9 * nt + N];
      CT vol = (CT)__ldg(b.a[FF_VOL] + N);
      CT cd[NV];
      CT fd = upper ? CT(1) : coef[12 * nt + N];
#pragma unroll
      for (int v = 0; v < NV; v++) cd[v] = __ldcg(dw + v * nt + N) * fd;
      // the three neighbours: k first (reference order), then i and j
      CT ck[NV], yd[NV], bd[NV];
#pragma unroll
      for (int v = 0; v < NV; v++) { ck[v] = 0; yd[v] = 0; bd[v] = 0; }
      const int st[3] = {1, IS, IL};
      // PREDGS drops the i+1 coupling of row J = JMAX unless bit 2 of upper
      // (predgs_full) asks for it; PRKEGS does not drop it
      const bool has[3] = {upper ? (I < IMAX && (NV == 7 || J < JMAX || (upper & 2))) : (I > 1), upper ? (J < JMAX) : (J > 1),
                           upper ? (K < KMAX) : (K > 1)};
#pragma unroll
      for (int d = 2; d >= 0; d--) {
        if (!has[d]) continue;
        size_t nb = upper ? N + st[d] : N - st[d];
        size_t fN = upper ? nb : N;              // shared face
        const int ao = 4 * d;
        CT x[NV];
#pragma unroll
        for (int v = 0; v < NV; v++) x[v] = __ldcg(dw + v * nt + nb);
        CT out[NV];
        nb_product<CT, NV>(out, x, b, nb, (CT)__ldg(b.a[FF_C] + nb), (CT)__ldg(b.a[FF_RO] + nb),
                           (CT)__ldg(b.a[FF_A1XA + ao] + fN), (CT)__ldg(b.a[FF_A1YA + ao] + fN),
                           (CT)__ldg(b.a[FF_A1ZA + ao] + fN), coef[(3 * d) * nt + nb],
                           coef[(3 * d + 1) * nt + nb], coef[(3 * d + 2) * nt + nb]);
        CT* dst = d == 2 ? ck : (d == 0 ? yd : bd);
#pragma unroll
        for (int v = 0; v < NV; v++) dst[v] = out[v];
      }
      CT a3 = (CT)__ldg(b.a[FF_A3] + (upper ? N + IL : N));
      CT a1 = (CT)__ldg(b.a[FF_A1] + (upper ? N + 1 : N));
      CT a2 = (CT)__ldg(b.a[FF_A2] + (upper ? N + IS : N));
      CT scinv = coef[10 * nt + N], scinp = coef[11 * nt + N];
      CT res[NV];
#pragma unroll
      for (int v = 0; v < NV; v++) {
        CT x = upper ? (-dt1 * a3 * ck[v] + vol * cd[v]) : (dt1 * a3 * ck[v] + vol * cd[v]);
        x = upper ? x - dt1 * (a1 * yd[v] + a2 * bd[v]) : x + dt1 * (a1 * yd[v] + a2 * bd[v]);
        res[v] = x * (v == 4 ? scinp : scinv);
      }
#pragma unroll
      for (int v = 0; v < NV; v++) __stcg(dw + v * nt + N, res[v]);
    }
    if (!grid_barrier(bar, bar + 1, gridDim.x, err)) return;
  }
}

// The hyperplane sweep on the sweep layout (k_sweep_coef): the cells of a
// plane with one K and consecutive J are consecutive in sw and dwp, so each
// warp's loads are coalesced.  Each cell pulls the products of its three
// upstream neighbours from their increments and their precomputed frames,
// scalars and eigenvalue coefficients.
template <typename CT, int NV>
__global__ void k_lusgs_sweep(DevBlock b, const CT* __restrict__ sw, CT* dwp, int upper, unsigned* bar, int* err) {
  const int IMAX = b.imax, JMAX = b.jmax, KMAX = b.kmax;
  const int W = IMAX + JMAX - 1;
  const size_t ns = sw_size(IMAX, JMAX, KMAX);
  const int nthreads = gridDim.x * blockDim.x;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nplanes = IMAX + JMAX + KMAX - 2;
  const long off[3] = {JMAX, JMAX + 1, (long)W * JMAX};
  for (int s = 0; s < nplanes; s++) {
    const int m = upper ? IMAX + JMAX + KMAX - s : 3 + s;
    const int klo = max(1, m - IMAX - JMAX), khi = min(KMAX, m - 2);
    const int npairs = (khi - klo + 1) * JMAX;
    for (int q = tid; q < npairs; q += nthreads) {
      const int K = klo + q / JMAX, J = q % JMAX + 1, I = m - J - K;
      if (I < 1 || I > IMAX) continue;
      const size_t S = ((size_t)(K - 1) * W + (m - K - 2)) * JMAX + (J - 1);
      // PREDGS drops the i+1 coupling of row J = JMAX unless bit 2 of upper
      // (predgs_full) asks for it; PRKEGS does not drop it
      const bool has[3] = {upper ? (I < IMAX && (NV == 7 || J < JMAX || (upper & 2))) : (I > 1), upper ? (J < JMAX) : (J > 1),
                           upper ? (K < KMAX) : (K > 1)};
      CT ck[NV], yd[NV], bd[NV];
#pragma unroll
      for (int d = 2; d >= 0; d--) {   // k first (reference order), then i and j
        CT* dst = d == 2 ? ck : (d == 0 ? yd : bd);
        if (!has[d]) {
#pragma unroll
          for (int v = 0; v < NV; v++) dst[v] = CT(0);
          continue;
        }
        const size_t nb = upper ? S + off[d] : S - off[d];
        CT x[NV], f[3], sc[5], l[3];
#pragma unroll
        for (int v = 0; v < NV; v++) x[v] = __ldcg(dwp + v * ns + nb);
#pragma unroll
        for (int c = 0; c < 3; c++) f[c] = __ldg(sw + (SW_F + 3 * d + c) * ns + nb);
#pragma unroll
        for (int c = 0; c < (NV == 7 ? 5 : 3); c++) sc[c] = __ldg(sw + (SW_SC + c) * ns + nb);
#pragma unroll
        for (int e = 0; e < 3; e++) l[e] = __ldg(sw + (SW_L + 3 * d + e) * ns + nb);
        nb_product_pre<CT, NV>(dst, x, f, sc, NV == 7 ? __ldg(sw + SW_RO * ns + nb) : CT(0), l[0], l[1], l[2]);
      }
      const CT dt1 = __ldg(sw + SW_DT1 * ns + S), vol = __ldg(sw + SW_VOL * ns + S);
      const CT fd = upper ? CT(1) : __ldg(sw + SW_FD * ns + S);
      const CT a1 = __ldg(sw + SW_A1 * ns + S), a2 = __ldg(sw + SW_A2 * ns + S), a3 = __ldg(sw + SW_A3 * ns + S);
      const CT scinv = __ldg(sw + SW_SCINV * ns + S), scinp = __ldg(sw + SW_SCINP * ns + S);
#pragma unroll
      for (int v = 0; v < NV; v++) {
        CT cd = __ldcg(dwp + v * ns + S) * fd;
        CT x = upper ? (-dt1 * a3 * ck[v] + vol * cd) : (dt1 * a3 * ck[v] + vol * cd);
        x = upper ? x - dt1 * (a1 * yd[v] + a2 * bd[v]) : x + dt1 * (a1 * yd[v] + a2 * bd[v]);
        __stcg(dwp + v * ns + S, x * (v == 4 ? scinp : scinv));
      }
    }
    if (!grid_barrier(bar, bar + 1, gridDim.x, err)) return;
  }
}

// DRO/CP (imps3.f:483), FIN res3c.f:1077, the limits of CYCLES
// (ns3c.f:1553-1596: UPLIM/LOLIM res3c.f:3314-3401, PDTOP, LOLIMP), the
// interior *OLD copies of SUBIN and the max|dp| monitor (DROMXX, IDRXX=6).
// state: the equation of state of the new values in the same pass (where it comes next).
__global__ void k_fin(DevBlock b, ff_params p, unsigned long long* dromax_bits, int divide_cp, int state) {
  size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double amax = 0.;
  if (n < (size_t)b.ntot) {
    int i = (int)(n % b.is), j = (int)((n / b.is) % (b.jmax + 4)), k = (int)(n / b.il);
    bool kin = k >= 2 && k < b.kmax + 2, jin = j >= 2 && j < b.jmax + 2;
    bool interior = kin && jin && i >= 2 && i < b.imax + 2;
    double T = b.a[FF_TEMP][n], U = b.a[FF_U][n], V = b.a[FF_V][n], W = b.a[FF_W][n], PD = b.a[FF_PDIFF][n];
    const bool sst = p.iturb >= 3;
    double rk = 0., re = 0.;
    if (sst) { rk = b.a[FF_RK][n]; re = b.a[FF_REPS][n]; }
    if (interior) {
      double dt = b.a[FF_DRO][n], dm = b.a[FF_DM][n], dn = b.a[FF_DN][n], dw = b.a[FF_DW][n], de = b.a[FF_DE][n];
      const double told = b.a[FF_TOLD][n], uold = b.a[FF_UOLD][n], vold = b.a[FF_VOLD][n], wold = b.a[FF_WOLD][n],
                   pold = b.a[FF_POLD][n];
      double drk = 0., deps = 0., rkold = 0., epold = 0.;
      if (sst) { drk = b.a[FF_DRK][n]; deps = b.a[FF_DEPS][n]; rkold = b.a[FF_RKOLD][n]; epold = b.a[FF_EPSOLD][n]; }
      if (divide_cp) {
        const double cp = b.a[FF_CP][n], ro = sst ? b.a[FF_RO][n] : 0.;
        dt = dt / cp;
        b.a[FF_DRO][n] = dt;
        if (sst) {   // imps3.f:488-492
          drk = drk * ro; deps = deps * ro;
          b.a[FF_DRK][n] = drk; b.a[FF_DEPS][n] = deps;
        }
      }
      if (sst) {   // FIN res3c.f:1190-1198
        rk = rkold + drk / (1. + fabs(drk) / (.45 * rkold));
        re = epold + deps / (1. + fabs(deps) / (.90 * epold));
      }
      T = told + dt;
      U = uold + dm;
      V = vold + dn;
      W = wold + dw;
      PD = pold + de;
      amax = fabs(de);
    }
    if (kin && jin) {   // UPLIM range: interior k-planes, interior rows
      T = dmin(T, p.tuplim); U = dmin(U, 5000.); V = dmin(V, 5000.); W = dmin(W, 5000.);
    }
    T = dmax(T, p.tlolim); U = dmax(U, -5000.); V = dmax(V, -5000.); W = dmax(W, -5000.);
    double P = PD + p.frspre;
    double prelim = dmin(0., P - 0.01 * p.frspre);
    P = P - prelim; PD = PD - prelim;
    b.a[FF_TEMP][n] = T; b.a[FF_U][n] = U; b.a[FF_V][n] = V; b.a[FF_W][n] = W;
    b.a[FF_PDIFF][n] = PD; b.a[FF_P][n] = P;
    if (sst) {   // LOLIM of RK and REPS over every cell (FIN, then CYCLES)
      b.a[FF_RK][n] = dmax(rk, p.rklim);
      b.a[FF_REPS][n] = dmax(re, p.epslim);
    }
    if (interior) {
      b.a[FF_TOLD][n] = T; b.a[FF_UOLD][n] = U; b.a[FF_VOLD][n] = V; b.a[FF_WOLD][n] = W;
      b.a[FF_POLD][n] = PD;
    }
    if (state) state_cell(b, p, n, interior);
  }
  for (int o = 16; o > 0; o >>= 1) amax = dmax(amax, __shfl_down_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0 && amax > 0.) atomicMax(dromax_bits, (unsigned long long)__double_as_longlong(amax));
}

// Standalone DRO/CP that ends IMPS (imps3.f:483) when it is called as a stage.
__global__ void k_fin_divide(DevBlock b, int sst) {
  size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= (size_t)b.ntot) return;
  int i = (int)(n % b.is), j = (int)((n / b.is) % (b.jmax + 4)), k = (int)(n / b.il);
  if (i >= 2 && i < b.imax + 2 && j >= 2 && j < b.jmax + 2 && k >= 2 && k < b.kmax + 2) {
    b.a[FF_DRO][n] = b.a[FF_DRO][n] / b.a[FF_CP][n];
    if (sst) {   // imps3.f:488-492
      b.a[FF_DRK][n] = b.a[FF_DRK][n] * b.a[FF_RO][n];
      b.a[FF_DEPS][n] = b.a[FF_DEPS][n] * b.a[FF_RO][n];
    }
  }
}

// ---------------------------------------------------------------------------
// Multigrid transfers (FAS V-cycle of CYCLES ns3c.f:1607-2170)
// ---------------------------------------------------------------------------

// TRANSF multi.f:156: volume-weighted restriction of TEMP,U,V,W,PDIFF,EPS2,
// VIST and of the residuals (into P2H) for coarse cells 0..MAX+1, and the
// interior *OLD copies.
// One thread a coarse cell, ghosts included, the outer ring in the same pass:
// a face ghost of the second layer takes what the first layer gets along the
// face normal (computed again), other second-layer cells are not used on
// coarse levels and left alone; the forcing terms of all ghosts are zero.
// forced: ADDRES of the finer level (its DRO += P2H) first, as k_forcing does;
// only the interior, whose 8 children are this thread's.
__global__ void k_transf(DevBlock f, DevBlock c, int sst, int forced) {
  size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= (size_t)c.ntot) return;
  int I = (int)(n % c.is) - 1, J = (int)((n / c.is) % (c.jmax + 4)) - 1, K = (int)(n / c.il) - 1;
  const bool interior = I >= 1 && I <= c.imax && J >= 1 && J <= c.jmax && K >= 1 && K <= c.kmax;
  if (!interior) {
#pragma unroll
    for (int v = 0; v < 5; v++) c.a[FF_ROP2H + v][n] = 0.;
    if (sst) { c.a[FF_RKP2H][n] = 0.; c.a[FF_EPP2H][n] = 0.; }
    const int second = (I == -1 || I == c.imax + 2) + (J == -1 || J == c.jmax + 2) + (K == -1 || K == c.kmax + 2);
    if (second > 1) return;
    I = max(0, min(c.imax + 1, I)); J = max(0, min(c.jmax + 1, J)); K = max(0, min(c.kmax + 1, K));
  }
  size_t ijk = ix(f, 2 * I - 1, 2 * J - 1, 2 * K - 1);
  size_t o[8] = {ijk + f.is + 1, ijk, ijk + 1, ijk + f.is,
                 ijk + f.is + 1 + f.il, ijk + f.il, ijk + 1 + f.il, ijk + f.is + f.il};
  const double* VOL = f.a[FF_VOL];
  double vv[8];
#pragma unroll
  for (int q = 0; q < 8; q++) vv[q] = VOL[o[q]];
  double pvol = 1. / c.a[FF_VOL][ix(c, I, J, K)];
  auto mean = [&](int slot) {
    const double* X = f.a[slot];
    double s = 0.;
#pragma unroll
    for (int q = 0; q < 8; q++) s += vv[q] * X[o[q]];
    return s * pvol;
  };
  const int vs[7] = {FF_TEMP, FF_U, FF_V, FF_W, FF_PDIFF, FF_EPS2, FF_VIST};
  double x[9];
#pragma unroll
  for (int v = 0; v < 7; v++) x[v] = mean(vs[v]);
  if (sst) { x[7] = mean(FF_RK); x[8] = mean(FF_REPS); }   // TRANKE multi.f:434
#pragma unroll
  for (int v = 0; v < 7; v++) c.a[vs[v]][n] = x[v];
  if (sst) { c.a[FF_RK][n] = x[7]; c.a[FF_REPS][n] = x[8]; }
  if (!interior) return;
  c.a[FF_TOLD][n] = x[0];
  c.a[FF_UOLD][n] = x[1];
  c.a[FF_VOLD][n] = x[2];
  c.a[FF_WOLD][n] = x[3];
  c.a[FF_POLD][n] = x[4];
  if (sst) { c.a[FF_RKOLD][n] = x[7]; c.a[FF_EPSOLD][n] = x[8]; }
  const int rs[7] = {FF_DRO, FF_DM, FF_DN, FF_DW, FF_DE, FF_DRK, FF_DEPS};
  const int ps[7] = {FF_ROP2H, FF_RMP2H, FF_RNP2H, FF_RWP2H, FF_EP2H, FF_RKP2H, FF_EPP2H};
#pragma unroll
  for (int v = 0; v < 7; v++) {
    if (v >= 5 && !sst) break;
    double r[8], s = 0.;
#pragma unroll
    for (int q = 0; q < 8; q++) r[q] = f.a[rs[v]][o[q]];
    if (forced) {
      double* P2 = f.a[ps[v]];
#pragma unroll
      for (int q = 0; q < 8; q++) r[q] = P2[o[q]] + r[q];
#pragma unroll
      for (int q = 0; q < 8; q++) f.a[rs[v]][o[q]] = r[q];
    }
#pragma unroll
    for (int q = 0; q < 8; q++) s += vv[q] * r[q];
    c.a[ps[v]][n] = s * pvol;
  }
}

// FORCFU multi.f:1609 (mode 0: P2H -= R) and ADDRES multi.f:1686 (mode 1:
// R = P2H + R), every cell of the level.
__global__ void k_forcing(DevBlock b, int mode, int sst) {
  size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= (size_t)b.ntot) return;
  const int ps[7] = {FF_ROP2H, FF_RMP2H, FF_RNP2H, FF_RWP2H, FF_EP2H, FF_RKP2H, FF_EPP2H};
  const int nv = sst ? 7 : 5;
#pragma unroll
  for (int v = 0; v < 7; v++) {
    if (v >= nv) break;
    double* P2 = b.a[ps[v]];
    double* R = b.a[FF_DRO + v];
    const double r = R[n];
    double q = P2[n];
    if (mode != 1) P2[n] = q = q - r;
    if (mode != 0) R[n] = q + r;
  }
}

// INTERT multi.f:2051 -> INTERO 2007: damped injection of the coarse k and
// omega corrections (CMGK, CMGEPS) into the fine interior.
FF_DI void intert_cell(const DevBlock& c, const DevBlock& f, const ff_params& p, size_t N, size_t F) {
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const double cc1 = q == 0 ? p.cmgk : p.cmgeps, cc2 = cc1 + 1.E-7;
    double drok = c.a[q == 0 ? FF_RK : FF_REPS][N] - c.a[q == 0 ? FF_RKOLD : FF_EPSOLD][N];
    double* R = f.a[q == 0 ? FF_RK : FF_REPS];
    double r = R[F];
    R[F] = r + cc1 * r * drok / (cc2 * r + fabs(drok));
  }
}

// INTERP multi.f:1763: inject the coarse correction into the 8 children.
FF_DI void interp_cell(const DevBlock& c, const DevBlock& f, size_t N, size_t F) {
  const double dp = c.a[FF_PDIFF][N] - c.a[FF_POLD][N], dt = c.a[FF_TEMP][N] - c.a[FF_TOLD][N];
  const double du = c.a[FF_U][N] - c.a[FF_UOLD][N], dv = c.a[FF_V][N] - c.a[FF_VOLD][N];
  const double dw = c.a[FF_W][N] - c.a[FF_WOLD][N];
  const double t = f.a[FF_TEMP][F], u = f.a[FF_U][F], v = f.a[FF_V][F], w = f.a[FF_W][F], P = f.a[FF_P][F],
               pd = f.a[FF_PDIFF][F];
  f.a[FF_TEMP][F] = t + dt;
  f.a[FF_U][F] = u + du;
  f.a[FF_V][F] = v + dv;
  f.a[FF_W][F] = w + dw;
  f.a[FF_P][F] = P + dp;
  f.a[FF_PDIFF][F] = pd + dp;
}

// FIN on a coarse level (update = 1: UPLIM/LOLIM TEMP, LOLIMP, no PDTOP,
// ns3c.f:1935-1990) and the limits after INTERP (update = 0, ns3c.f:2059-2125:
// LOLIMP; the two-equation branch also limits TEMP, RK and REPS).
// update 2: the division by CP (and RO) of k_fin_divide in the same pass.
// STATE: see k_fin; a template parameter, because its registers cost the pass
// without it a fifth (80x48x40 cells 8.8 -> 10.8 us).
template <bool STATE>
FF_DI void fin_coarse_cell(const DevBlock& b, const ff_params& p, size_t n, bool kin, bool jin, bool interior, int update) {
  const bool sst = p.iturb >= 3;
  double T = b.a[FF_TEMP][n];
  if (update && interior) {
    double dt = b.a[FF_DRO][n];
    if (update == 2) b.a[FF_DRO][n] = dt = dt / b.a[FF_CP][n];
    T = b.a[FF_TOLD][n] + dt;
    b.a[FF_U][n] = b.a[FF_UOLD][n] + b.a[FF_DM][n];
    b.a[FF_V][n] = b.a[FF_VOLD][n] + b.a[FF_DN][n];
    b.a[FF_W][n] = b.a[FF_WOLD][n] + b.a[FF_DW][n];
    b.a[FF_PDIFF][n] = b.a[FF_POLD][n] + b.a[FF_DE][n];
    if (sst) {   // FIN res3c.f:1190-1198
      double drk = b.a[FF_DRK][n], deps = b.a[FF_DEPS][n];
      if (update == 2) {   // imps3.f:488-492
        const double ro = b.a[FF_RO][n];
        b.a[FF_DRK][n] = drk = drk * ro;
        b.a[FF_DEPS][n] = deps = deps * ro;
      }
      double rkold = b.a[FF_RKOLD][n], epold = b.a[FF_EPSOLD][n];
      b.a[FF_RK][n] = rkold + drk / (1. + fabs(drk) / (.45 * rkold));
      b.a[FF_REPS][n] = epold + deps / (1. + fabs(deps) / (.90 * epold));
    }
  }
  if (sst) {   // LOLIM of RK, REPS over every cell (FIN; after INTERP, CYCLES)
    b.a[FF_RK][n] = dmax(b.a[FF_RK][n], p.rklim);
    b.a[FF_REPS][n] = dmax(b.a[FF_REPS][n], p.epslim);
  }
  // TEMP limits after a coarse FIN, and after INTERP on the two-equation branch
  if (update || sst) {
    if (kin && jin) T = dmin(T, p.tuplim);
    T = dmax(T, p.tlolim);
    b.a[FF_TEMP][n] = T;
  }
  double P = b.a[FF_P][n];
  double prelim = dmin(0., P - 0.01 * p.frspre);
  b.a[FF_P][n] = P - prelim;
  b.a[FF_PDIFF][n] = b.a[FF_PDIFF][n] - prelim;
  if (STATE) state_cell(b, p, n, interior);
}

template <bool STATE>
__global__ void k_fin_coarse(DevBlock b, ff_params p, int update) {
  size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= (size_t)b.ntot) return;
  int i = (int)(n % b.is), j = (int)((n / b.is) % (b.jmax + 4)), k = (int)(n / b.il);
  bool kin = k >= 2 && k < b.kmax + 2, jin = j >= 2 && j < b.jmax + 2;
  fin_coarse_cell<STATE>(b, p, n, kin, jin, kin && jin && i >= 2 && i < b.imax + 2, update);
}

// INTERP, INTERT and the limits of k_fin_coarse over the finer level in one
// pass: each cell depends on itself and its parent only.
__global__ void k_prolong(DevBlock c, DevBlock f, ff_params p) {
  size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= (size_t)f.ntot) return;
  int I = (int)(n % f.is) - 1, J = (int)((n / f.is) % (f.jmax + 4)) - 1, K = (int)(n / f.il) - 1;
  const bool kin = K >= 1 && K <= f.kmax, jin = J >= 1 && J <= f.jmax;
  const bool interior = kin && jin && I >= 1 && I <= f.imax;
  if (interior) {
    const size_t N = ix(c, (I + 1) / 2, (J + 1) / 2, (K + 1) / 2);
    interp_cell(c, f, N, n);
    if (p.iturb >= 3) intert_cell(c, f, p, N, n);
  }
  fin_coarse_cell<false>(f, p, n, kin, jin, interior, 0);
}

// CONNEC ns3c.f:8605 (EXPTOT/IMPVO2 gluebm.f:6819/6964) for aligned 1:1
// patches of all blocks in one launch: blockIdx.y = connection item; the two
// interior layers of the source block fill the two ghost layers of the
// destination patch (TEMP,U,V,W,E,EPS2,VIST,CH,P,PDIFF,RK,REPS, as BOUNDI passes).
struct ConnItem { int dst, src; ff_patch pa; };

// The donor face cell (ad, cd) of receiver patch point (a, c) of a 1:1
// connection in orientation ICON(14) = pa.iori: the donor's export order
// (second in-face index fastest on odd faces, first on even faces; EXPVOL
// gluebm.f:6115-6136), the receiver's import order (first index fastest on
// odd faces, second on even; IMPVO2 7040-7080) and PERMUT's turn of the
// receiver sequence (gluebm.f:4868).
FF_DI void conn_donor(const ff_patch& pa, int a, int c, int& ad, int& cd) {
  const int n1 = pa.r1b - pa.r1a + 1, n2 = pa.r2b - pa.r2a + 1;
  const bool rodd = pa.iface & 1, dodd = pa.nface & 1;
  const int P = rodd ? n1 : n2, Q = rodd ? n2 : n1;
  const int x = rodd ? a - pa.r1a + 1 : c - pa.r2a + 1;
  const int y = rodd ? c - pa.r2a + 1 : a - pa.r1a + 1;
  int u, v;
  switch (pa.iori & 3) {
    case 1: u = Q + 1 - y; v = x; break;
    case 2: u = P + 1 - x; v = Q + 1 - y; break;
    case 3: u = y; v = P + 1 - x; break;
    default: u = x; v = y;
  }
  if (dodd) { cd = pa.n2a + u - 1; ad = pa.n1a + v - 1; }
  else { ad = pa.n1a + u - 1; cd = pa.n2a + v - 1; }
}

__global__ void k_connec(const DevBlock* __restrict__ blocks, const ConnItem* __restrict__ items) {
  const ConnItem& it = items[blockIdx.y];
  const ff_patch& pa = it.pa;
  int n1 = pa.r1b - pa.r1a + 1, n2 = pa.r2b - pa.r2a + 1;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n1 * n2) return;
  int a = pa.r1a + t % n1, c = pa.r2a + t / n1;
  const DevBlock& d = blocks[it.dst];
  const DevBlock& s = blocks[it.src];
  FaceG fd = face_g(d, pa.iface), fs = face_g(s, pa.nface);
  int ad, cd;
  conn_donor(pa, a, c, ad, cd);
  size_t L = face_cell(d, fd, a, c);
  size_t S = face_cell(s, fs, ad, cd);
  const int vs[12] = {FF_TEMP, FF_U, FF_V, FF_W, FF_E, FF_EPS2, FF_VIST, FF_CH, FF_P, FF_PDIFF, FF_RK, FF_REPS};
  int lsd = fd.idir * fd.s, lss = fs.idir * fs.s;
  double x[2][12];
#pragma unroll
  for (int g = 0; g < 2; g++)
#pragma unroll
    for (int v = 0; v < 12; v++) x[g][v] = s.a[vs[v]][S + g * lss];
#pragma unroll
  for (int g = 0; g < 2; g++)
#pragma unroll
    for (int v = 0; v < 12; v++) d.a[vs[v]][L - (g + 1) * lsd] = x[g][v];
}

// Halo pack (mode 0, from the source block) / unpack (mode 1, into the
// destination's ghost layers) of remote 1:1 patches; blockIdx.y = item.
struct HaloItem { int blk, mode; long long offset; ff_patch pa; };

__global__ void k_halo(const DevBlock* __restrict__ blocks, const HaloItem* __restrict__ items,
                       int mode, double* __restrict__ sbuf, const double* __restrict__ rbuf) {
  const HaloItem& it = items[blockIdx.y];
  if (it.mode != mode) return;
  const ff_patch& pa = it.pa;
  int n1 = pa.r1b - pa.r1a + 1, n2 = pa.r2b - pa.r2a + 1, n = n1 * n2;
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  int a = t % n1, c = t / n1;
  const DevBlock& b = blocks[it.blk];
  const int vs[12] = {FF_TEMP, FF_U, FF_V, FF_W, FF_E, FF_EPS2, FF_VIST, FF_CH, FF_P, FF_PDIFF, FF_RK, FF_REPS};
  if (mode == 0) {
    FaceG fs = face_g(b, pa.nface);
    int ad, cd;
    conn_donor(pa, a + pa.r1a, c + pa.r2a, ad, cd);
    size_t S = face_cell(b, fs, ad, cd);
    int lss = fs.idir * fs.s;
    double* o = sbuf + it.offset;
#pragma unroll
    for (int g = 0; g < 2; g++)
#pragma unroll
      for (int v = 0; v < 12; v++) o[(size_t)(g * 12 + v) * n + t] = b.a[vs[v]][S + g * lss];
  } else {
    FaceG fd = face_g(b, pa.iface);
    size_t L = face_cell(b, fd, a + pa.r1a, c + pa.r2a);
    int lsd = fd.idir * fd.s;
    const double* o = rbuf + it.offset;
#pragma unroll
    for (int g = 0; g < 2; g++)
#pragma unroll
      for (int v = 0; v < 12; v++) b.a[vs[v]][L - (g + 1) * lsd] = o[(size_t)(g * 12 + v) * n + t];
  }
}

// SUBIN ns3c.f:9742: the *OLD copies of the interior cells.
__global__ void k_subin_copy(DevBlock b) {
  size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= (size_t)b.ntot) return;
  int i = (int)(n % b.is), j = (int)((n / b.is) % (b.jmax + 4)), k = (int)(n / b.il);
  if (!(i >= 2 && i < b.imax + 2 && j >= 2 && j < b.jmax + 2 && k >= 2 && k < b.kmax + 2)) return;
  b.a[FF_TOLD][n] = b.a[FF_TEMP][n];
  b.a[FF_UOLD][n] = b.a[FF_U][n];
  b.a[FF_VOLD][n] = b.a[FF_V][n];
  b.a[FF_WOLD][n] = b.a[FF_W][n];
  b.a[FF_POLD][n] = b.a[FF_PDIFF][n];
}

// max |DE| over the interior (DROMXX, IDRXX = 6) into dm_bits.
__global__ void k_maxabs_de(DevBlock b, unsigned long long* dm_bits) {
  double amax = 0.;
  int ncell = b.imax * b.jmax * b.kmax;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ncell; t += gridDim.x * blockDim.x) {
    int I = t % b.imax + 1, J = (t / b.imax) % b.jmax + 1, K = t / (b.imax * b.jmax) + 1;
    amax = dmax(amax, fabs(b.a[FF_DE][ix(b, I, J, K)]));
  }
  for (int o = 16; o > 0; o >>= 1) amax = dmax(amax, __shfl_down_sync(0xffffffffu, amax, o));
  if ((threadIdx.x & 31) == 0 && amax > 0.) atomicMax(dm_bits, (unsigned long long)__double_as_longlong(amax));
}

// TIMDER res3c.f:3014 / TIMDKE res3c.f:3062 on the interior cells: the
// second-order physical-time derivative of TIMEL added to the residual,
// PDT * (-1.5 VOL (Q - Q2) + 0.5 VOL (Q2 - Q3)) with PDT = 1 / (VOL DT).
template <int NV>
__global__ void k_timder(DevBlock b, ff_params p) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= b.imax * b.jmax * b.kmax) return;
  int I = t % b.imax + 1, J = (t / b.imax) % b.jmax + 1, K = t / (b.imax * b.jmax) + 1;
  const size_t n = ix(b, I, J, K);
  const int sq[7] = {FF_RO, FF_RM, FF_RN, FF_RW, FF_E, FF_RK, FF_REPS};
  const double vol = b.a[FF_VOL][n], pdt = 1. / (vol * p.dt);
#pragma unroll
  for (int v = 0; v < NV; v++) {
    const double q = b.a[sq[v]][n], q2 = b.a[FF_ROLE2 + v][n], q3 = b.a[FF_ROLE3 + v][n];
    b.a[FF_DRO + v][n] = b.a[FF_DRO + v][n] + pdt * (-1.5 * vol * (q - q2) + 0.5 * vol * (q2 - q3));
  }
}

// STARTI res3c.f:3175 (mode 0: both old time levels = the state, every
// cell) and NEWTIM ns3c.f:9420 with R1 = 1 (mode 1: level n-1 <- level n,
// level n <- the state, interior cells).
__global__ void k_time_levels(DevBlock b, int nv, int mode) {
  const int sq[7] = {FF_RO, FF_RM, FF_RN, FF_RW, FF_E, FF_RK, FF_REPS};
  if (mode == 0) {
    size_t n = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= (size_t)b.ntot) return;
    for (int v = 0; v < nv; v++) {
      const double q = b.a[sq[v]][n];
      b.a[FF_ROLE3 + v][n] = q;
      b.a[FF_ROLE2 + v][n] = q;
    }
    return;
  }
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= b.imax * b.jmax * b.kmax) return;
  int I = t % b.imax + 1, J = (t / b.imax) % b.jmax + 1, K = t / (b.imax * b.jmax) + 1;
  const size_t n = ix(b, I, J, K);
  for (int v = 0; v < nv; v++) {
    b.a[FF_ROLE3 + v][n] = b.a[FF_ROLE2 + v][n];
    b.a[FF_ROLE2 + v][n] = b.a[sq[v]][n];
  }
}

#include "ff_sst.cuh"

}  // namespace ff

// Staged values per thread of the pipelined sweep: sweep data + right-hand side
constexpr int LSTAGE = SW_N + 7;

FF_DI void cp_async_ca(void* smem, const double* g) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(g) : "memory");
}
FF_DI void cp_async_ca(void* smem, const float* g) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(g) : "memory");
}
FF_DI void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Start the copy of one cell's sweep data into the thread's stage slots
// (stride = threads per CTA).
template <typename CT, int NV>
FF_DI void lines_stage(CT* stg, int stride, const CT* __restrict__ sw, const CT* dwp, size_t ns, size_t S,
                       int upper) {
#pragma unroll
  for (int c = 0; c < SW_N; c++) {
    if (c == SW_FD && upper) continue;
    if (NV == 5 && (c == SW_RO || c == SW_SC + 3 || c == SW_SC + 4)) continue;
    cp_async_ca(stg + c * stride, sw + c * ns + S);
  }
#pragma unroll
  for (int v = 0; v < NV; v++) cp_async_ca(stg + (SW_N + v) * stride, dwp + v * ns + S);
}

#include "ff_pipe.cuh"
#include "ff_flow.cuh"
#include "ff_ddadi.cuh"
