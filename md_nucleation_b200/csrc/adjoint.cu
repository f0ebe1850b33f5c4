/*
 * adjoint.cu -- the gradient harness (no counterpart in the reference):
 * dJ/dtheta of an ion-vapor objective over a window of MD steps of one
 * replica, by the discrete adjoint of the engine's velocity Verlet step.
 *
 * Forward: the engine advances the window (FP32 pair terms, FP64
 * integration) and the replica's in-domain atoms are gathered every K steps
 * (checkpoints).  Backward: every segment is recomputed in FP64 from its
 * checkpoint at once, one cluster each, keeping x_t, the taper weights with
 * their gradients, the count term's derivatives and the SHAKE multipliers of
 * each step; then one cluster runs, last
 * segment first, the adjoint of
 *   (1) v_a = v + c F          (2) y = x + dt v_a          (3) x' = SHAKE(y; x)
 *   (4) v_b = v_a + (x' - y)/dt (5) F' = F(x'; theta)      (6) v' = v_b + c F'
 * (MD::verlet, src/verlet.cpp:20-39, with the SHAKE step of src/shake.cpp:6-92
 * and the velocity correction the engine applies) backwards through it:
 *   - (5): the transposed force Jacobian applied to the force adjoint:
 *     analytic for the pair terms (LJ, LJ + Coulomb, Born-Mayer-Huggins), the
 *     taper weights w(|x - c_ion|) of the vapor atoms included with their
 *     dependence on the ion centre; forward-mode (dual number) products for
 *     the bonded terms, whose force Jacobians are symmetric (F = -grad U);
 *   - (3): the adjoint of the converged projection x' = y + sum_k g_k D_k r_k
 *     (r_k the constraint vector at the step's start): G^T mu = rho solved per
 *     group of constraints that share atoms, lambda_y = lambda - sum_k mu_k
 *     B_k^T, plus the g_k D_k dr_k terms into the previous positions.
 *
 * What bounds it: a step is a few ten thousand FP64 pair products between two
 * points where all CTAs meet.  So nothing is scattered: a warp takes an atom
 * and sums over its row of partners (each pair evaluated from both sides), a
 * bonded term's forces go to rows of their own that the atoms' owners read,
 * and a warp takes a constraint group with everything that happens to its
 * atoms between two force products.  A step has two cluster barriers.  492
 * atoms, 25 thousand pairs: a reverse step takes 26 us, a recomputed one 21,
 * most of it the latency of FP64 chains.  (With FP64 atomics per pair, 150
 * thousand on 1,476 addresses, 164 us, of which the atomics 130, and 127.)
 * Parameter derivatives are summed per warp and row of parameters, then in
 * shared memory; the sums agree between runs up to FP64 rounding order.
 */
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <set>
#include <type_traits>
#include <vector>

#include "mdn.h"
#include "mdn_types.h"

__attribute__((visibility("hidden"))) int mdn_error(int code, const char* msg);
__attribute__((visibility("hidden"))) unsigned mdn_internal_quirks(const mdn_handle* h);
int mdn_snapshot_device(const RepParams* dP, const RepDyn* dD, const int* d_iblob, int R, const double* ion_x,
                        const double* ion_v, const double* slab_x, const double* slab_v, const double* vslab_x,
                        const double* vslab_v, long long* d_offset, int* d_type, double* d_x, double* d_v,
                        long long d_capacity, cudaStream_t stream);
__attribute__((visibility("hidden"))) void mdn_snapshot_args(const mdn_handle* h, SnapshotArgs* s);

namespace {

constexpr int ADJ_THREADS = 512;
constexpr int ADJ_CLUSTER = 16; /* CTAs of a reverse sweep: 21.6 ms for the 400 steps above, 8 took 27.7 */
constexpr int MAX_PARAMS = 512;
constexpr int SHAKE_SWEEPS = 1000;

enum PairKind : unsigned char { PK_GI = 0, PK_GV, PK_VI, PK_VV, PK_ION_LJC, PK_ION_BMH };

/* ------------------------------------------------------------------------- */
/* dual numbers: value and one tangent                                         */
/* ------------------------------------------------------------------------- */
struct Dual {
  double v, d;
};
__device__ __forceinline__ Dual mk(double v, double d = 0.0) { return {v, d}; }
__device__ __forceinline__ Dual operator+(Dual a, Dual b) { return {a.v + b.v, a.d + b.d}; }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) { return {a.v - b.v, a.d - b.d}; }
__device__ __forceinline__ Dual operator-(Dual a) { return {-a.v, -a.d}; }
__device__ __forceinline__ Dual operator*(Dual a, Dual b) { return {a.v * b.v, a.d * b.v + a.v * b.d}; }
__device__ __forceinline__ Dual operator/(Dual a, Dual b) {
  return {a.v / b.v, (a.d * b.v - a.v * b.d) / (b.v * b.v)};
}
__device__ __forceinline__ Dual operator*(double a, Dual b) { return {a * b.v, a * b.d}; }
__device__ __forceinline__ Dual operator*(Dual a, double b) { return {a.v * b, a.d * b}; }
__device__ __forceinline__ Dual operator-(double a, Dual b) { return {a - b.v, -b.d}; }
__device__ __forceinline__ Dual operator/(double a, Dual b) { return {a / b.v, -a * b.d / (b.v * b.v)}; }
__device__ __forceinline__ Dual dsqrt(Dual a) {
  double s = sqrt(a.v);
  return {s, a.d / (2.0 * s)};
}
__device__ __forceinline__ Dual dacos(Dual a) { return {acos(a.v), -a.d / sqrt(1.0 - a.v * a.v)}; }
__device__ __forceinline__ double dsqrt(double a) { return sqrt(a); }
__device__ __forceinline__ double dacos(double a) { return acos(a); }
__device__ __forceinline__ bool gt0(Dual a) { return a.v > 0; }
__device__ __forceinline__ bool gt0(double a) { return a > 0; }

/* bonded forces, the engine's / reference's expressions
 * (src/potential/compute_AMBER.cpp:52-253), on atoms in fixed slots */
template <class T>
__device__ void bond_t(const T (*X)[3], const double* co, T (*f)[3]) {
  T dx = X[0][0] - X[1][0], dy = X[0][1] - X[1][1], dz = X[0][2] - X[1][2];
  T rsq = dx * dx + dy * dy + dz * dz;
  T r = dsqrt(rsq);
  T dr = r - T{co[1]};
  T rk = co[0] * dr;
  T fb = -2.0 * rk / r;
  f[0][0] = fb * dx; f[0][1] = fb * dy; f[0][2] = fb * dz;
  f[1][0] = -(fb * dx); f[1][1] = -(fb * dy); f[1][2] = -(fb * dz);
}

template <class T>
__device__ void angle_t(const T (*X)[3], const double* co, T (*f)[3]) {
  T dx1 = X[0][0] - X[1][0], dy1 = X[0][1] - X[1][1], dz1 = X[0][2] - X[1][2];
  T rsq1 = dx1 * dx1 + dy1 * dy1 + dz1 * dz1;
  T r1 = dsqrt(rsq1);
  T dx2 = X[2][0] - X[1][0], dy2 = X[2][1] - X[1][1], dz2 = X[2][2] - X[1][2];
  T rsq2 = dx2 * dx2 + dy2 * dy2 + dz2 * dz2;
  T r2 = dsqrt(rsq2);
  T C = dx1 * dx2 + dy1 * dy2 + dz1 * dz2;
  C = C / (r1 * r2);
  T Cs = 1.0 / dsqrt(1.0 - C * C);
  T dtheta = dacos(C) - T{co[1]};
  T tk = co[0] * dtheta;
  T a = -2.0 * tk * Cs;
  T a11 = a * C / rsq1;
  T a12 = -a / (r1 * r2);
  T a22 = a * C / rsq2;
  T f1[3] = {a11 * dx1 + a12 * dx2, a11 * dy1 + a12 * dy2, a11 * dz1 + a12 * dz2};
  T f3[3] = {a22 * dx2 + a12 * dx1, a22 * dy2 + a12 * dy1, a22 * dz2 + a12 * dz1};
  for (int q = 0; q < 3; q++) {
    f[0][q] = f1[q];
    f[1][q] = -(f1[q] + f3[q]);
    f[2][q] = f3[q];
  }
}

template <class T>
__device__ void dihedral_t(const T (*X)[3], const double* co, int multi, T (*f)[3]) {
  T vb1x = X[0][0] - X[1][0], vb1y = X[0][1] - X[1][1], vb1z = X[0][2] - X[1][2];
  T vb2x = X[2][0] - X[1][0], vb2y = X[2][1] - X[1][1], vb2z = X[2][2] - X[1][2];
  T vb2xm = -vb2x, vb2ym = -vb2y, vb2zm = -vb2z;
  T vb3x = X[3][0] - X[2][0], vb3y = X[3][1] - X[2][1], vb3z = X[3][2] - X[2][2];
  T ax = vb1y * vb2zm - vb1z * vb2ym;
  T ay = vb1z * vb2xm - vb1x * vb2zm;
  T az = vb1x * vb2ym - vb1y * vb2xm;
  T bx = vb3y * vb2zm - vb3z * vb2ym;
  T by = vb3z * vb2xm - vb3x * vb2zm;
  T bz = vb3x * vb2ym - vb3y * vb2xm;
  T rasq = ax * ax + ay * ay + az * az;
  T rbsq = bx * bx + by * by + bz * bz;
  T rgsq = vb2xm * vb2xm + vb2ym * vb2ym + vb2zm * vb2zm;
  T rg = dsqrt(rgsq);
  T rginv{0.0}, ra2inv{0.0}, rb2inv{0.0};
  if (gt0(rg)) rginv = 1.0 / rg;
  if (gt0(rasq)) ra2inv = 1.0 / rasq;
  if (gt0(rbsq)) rb2inv = 1.0 / rbsq;
  T rabinv = dsqrt(ra2inv * rb2inv);
  T c = (ax * bx + ay * by + az * bz) * rabinv;
  T s = rg * rabinv * (ax * vb3x + ay * vb3y + az * vb3z);
  T df{0.0};
  for (int JJ = 0; JJ < multi; JJ++) {
    const int J5 = JJ * 5;
    T p_{1.0}, df1{0.0}, ddf1{0.0};
    for (int loop = 0; loop < co[J5 + 1]; loop++) {
      ddf1 = p_ * c - df1 * s;
      df1 = p_ * s + df1 * c;
      p_ = ddf1;
    }
    p_ = p_ * co[J5 + 3] + df1 * co[J5 + 4];
    df1 = df1 * co[J5 + 3] - ddf1 * co[J5 + 4];
    df1 = df1 * (-co[J5 + 1]);
    if (co[1] == 0) df1 = T{0.0}; /* term 0's periodicity tested for every term (compute_AMBER.cpp:199) */
    df = df + (-co[J5]) * df1;
  }
  T fg = vb1x * vb2xm + vb1y * vb2ym + vb1z * vb2zm;
  T hg = vb3x * vb2xm + vb3y * vb2ym + vb3z * vb2zm;
  T fga = fg * ra2inv * rginv;
  T hgb = hg * rb2inv * rginv;
  T gaa = -ra2inv * rg;
  T gbb = rb2inv * rg;
  T dtf[3] = {gaa * ax, gaa * ay, gaa * az};
  T dtg[3] = {fga * ax - hgb * bx, fga * ay - hgb * by, fga * az - hgb * bz};
  T dth[3] = {gbb * bx, gbb * by, gbb * bz};
  for (int q = 0; q < 3; q++) {
    T s2 = df * dtg[q];
    T f1 = df * dtf[q];
    T f4 = df * dth[q];
    f[0][q] = f1;
    f[1][q] = s2 - f1;
    f[2][q] = -s2 - f4;
    f[3][q] = f4;
  }
}

/* Born-Mayer-Huggins (Tosi-Fumi NaCl, src/potential/BMHFT/potentialBMHFT.hpp:21-39):
 * c0 = A b, c1 = 6 C, c2 = 8 D (kcal/mol units), c3 = sigma, c4 = 1/rho */
__constant__ double kBornD[2][2][5] = {
    {{25.4435 * 3.1546 / 4.184, 6. * 101.1719 / 4.184, 8. * 48.1771 / 4.184, 2.340, 3.1546},
     {20.3548 * 3.1546 / 4.184, 6. * 674.4793 / 4.184, 8. * 837.077 / 4.184, 2.755, 3.1546}},
    {{20.3548 * 3.1546 / 4.184, 6. * 674.4793 / 4.184, 8. * 837.077 / 4.184, 2.755, 3.1546},
     {15.2661 * 3.1546 / 4.184, 6. * 6985.6786 / 4.184, 8. * 14031.5785 / 4.184, 3.170, 3.1546}}};

/* ------------------------------------------------------------------------- */
/* the dense system of the window                                              */
/* ------------------------------------------------------------------------- */
struct Unit {
  int na, nc;     /* atoms (<= 8), constraints (<= 3) */
  int atom[8];
  int cons[3];
  int ci[3], cj[3]; /* the constraints' atoms as places in atom[] */
  double d2[3];     /* squared lengths */
  double cf[3][3];  /* d s_k / d l_l = cf[k][l] r_l (s_k the bond vector, l_l the multiplier) */
};
constexpr int kPrimary = 8; /* this side of the pair counts its parameter derivatives */

struct Sys {
  int N, n_ion, nt;
  const int* type;       /* [N] */
  const double* q;       /* [N] charges at s = 1 */
  const double* mass;    /* [N] */
  const double* c;       /* [N] kick coefficient 0.5 dt 4.184e-4 / m */
  const unsigned char* vapor; /* [N] 1 for vapor atoms (taper weights) */
  const double* A;       /* [nt*nt] */
  const double* B;
  const double* ieps;    /* [nt*nt] 1 / pair eps, 1 / pair sigma (for the derivatives) */
  const double* isig;
  const int* pidx;       /* [nt*nt] parameter base index (eps; sigma = +1), -1 */
  const int* bmh;        /* [N] Born-Mayer-Huggins row of ion atoms */
  int n_bonds, n_angles, n_dih;
  const int* bonds;      /* [3*n] i, j, type */
  const int* angles;     /* [4*n] */
  const int* dih;        /* [5*n] */
  const double* bond_c;  /* [2*types] */
  const double* angle_c;
  const double* dih_c;   /* [15*types] */
  const int* dih_multi;
  int n_cons, n_colors;
  const int* cons;       /* [3*n] i, j, bond type (length = bond_c[2*type+1]) */
  const int* cons_color;
  const int* cons_nb_off; /* CSR: constraints sharing an atom with constraint k */
  const int* cons_nb;
  int n_cons_nb;          /* entries of cons_nb */
  /* pairs by atom, from both sides: the partners of atom i are row[row_off[i]
   * .. row_off[i + 1]), x the partner, y its kind and kPrimary */
  const int* row_off;
  const int2* row;
  const int* row_order;   /* [N] atoms, longest rows first */
  /* bonded terms by atom: rows tb_off[i] .. tb_off[i + 1] of Buf::tb act on
   * atom i; tb_at[4 t + a] is the row of term t's a-th atom */
  const int* tb_off;
  const int* tb_at;
  /* what one warp carries from one force product to the next: a group of
   * constraints that share atoms, or up to 8 unconstrained atoms; n_units = 0
   * when a group has more than three constraints (shake / shake_adjoint) */
  int n_units;
  const Unit* units;
  double ri2, RI2, rcenter, overlap;
  double ion_msum, qqrd2e, dt;
  double efield[3];
  int efield_on, vcorr;
  int n_vmol, a_v, vmol_first; /* in-domain vapor molecules: atoms vmol_first + m*a_v + a */
  double vmol_mass;
  double R0, W, w_energy, w_count, inv_n;
  int n_params;           /* the last one is the charge scale */
};

struct Buf {
  double* X;     /* [(K+1)*3N] positions of the segment */
  double* V;     /* [3N] velocities and forces of the segment's current step */
  double* F;     /* [3N] (the recompute alone uses them) */
  double* gam;   /* [K*n_cons] converged SHAKE multipliers of each step */
  double* lx;    /* [3N] adjoint of x, carried across segments */
  double* lv;    /* [3N] adjoint of v */
  double* lf;    /* [3N] adjoint of F */
  double* xb;    /* [3N] accumulates the adjoint of the previous positions */
  double* w;     /* [(K+1)*N] taper weights of each step of the segment */
  double* dw;    /* [(K+1)*3N] their gradients */
  double* mg;    /* [(K+1)*3*(n_vmol+1)] count term: d/d(centre of vapor molecule m), then minus their sum */
  double* tb;    /* [rows*3] bonded terms' forces (or products) */
  double* part;  /* [ADJ_CLUSTER*3] the CTAs' shares of the weights' pull on the ion centre */
  double* mu;    /* [n_cons] */
  double* grad;  /* [n_params] */
  int* flag;     /* [2] SHAKE convergence scratch, status */
};

__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double s = 0;
  if (threadIdx.x < 32) {
    s = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) red[32] = s;
  }
  __syncthreads();
  s = red[32];
  __syncthreads();
  return s;
}

/* The reverse sweep runs on a cluster of CTAs: its loops are split over all
 * the cluster's threads, its phases are separated by cluster barriers, and
 * global data that other CTAs wrote in the same launch are read from L2
 * (__ldcg), since the L1 caches are not coherent.  A kernel launched without
 * a cluster is a cluster of one CTA (the recompute). */
namespace cg = cooperative_groups;
__device__ __forceinline__ int ctid() { return (int)(cg::this_cluster().block_rank() * blockDim.x + threadIdx.x); }
__device__ __forceinline__ int cnthr() { return (int)(cg::this_cluster().num_blocks() * blockDim.x); }
__device__ __forceinline__ void csync() {
  cg::cluster_group cl = cg::this_cluster();
  if (cl.num_blocks() > 1) {
    __threadfence();
    cl.sync();
  } else {
    __syncthreads();
  }
}

/* three sums over the block, the same in every thread; red >= 67 doubles */
__device__ void block_sum3(double* v, double* red) {
#pragma unroll
  for (int k = 0; k < 3; k++)
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0)
    for (int k = 0; k < 3; k++) red[4 * w + k] = v[k];
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0;
    for (int q = 0; q < nw; q++) t += red[4 * q + threadIdx.x];
    red[64 + threadIdx.x] = t;
  }
  __syncthreads();
  for (int k = 0; k < 3; k++) v[k] = red[64 + k];
  __syncthreads();
}

/* this warp among the cluster's, the CTAs in turn */
__device__ __forceinline__ int cwarp() {
  return (int)((threadIdx.x >> 5) * cg::this_cluster().num_blocks() + cg::this_cluster().block_rank());
}
__device__ __forceinline__ int cnwarps() { return cnthr() >> 5; }

/* ion centre of x (mass-weighted) into cent[0..2]; x was written by the whole
 * cluster */
__device__ void ion_centre(const Sys& S, const double* x, double* cent, double* red) {
  double v[3] = {0, 0, 0};
  for (int i = threadIdx.x; i < S.n_ion; i += blockDim.x)
    for (int k = 0; k < 3; k++) v[k] += __ldcg(x + 3 * i + k) * S.mass[i];
  block_sum3(v, red);
  if (threadIdx.x < 3) cent[threadIdx.x] = v[threadIdx.x] / S.ion_msum;
  __syncthreads();
}

/* taper weight of atom i and its gradient (src/verlet.cpp:109-134) */
__device__ __forceinline__ double weight_of(const Sys& S, const double* x, const double* cent, int i, double* g) {
  g[0] = g[1] = g[2] = 0;
  if (!S.vapor[i]) return 1;
  const double a = 3.141592653589793 / S.overlap * 0.5;
  double dx = __ldcg(x + 3 * i) - cent[0], dy = __ldcg(x + 3 * i + 1) - cent[1], dz = __ldcg(x + 3 * i + 2) - cent[2];
  double r2 = dx * dx + dy * dy + dz * dz;
  if (r2 < S.ri2) return 1;
  if (r2 > S.RI2) return 0;
  double r = sqrt(r2);
  double C = cos(a * (r - S.rcenter));
  double dwdr = -2.0 * C * sin(a * (r - S.rcenter)) * a;
  g[0] = dwdr * dx / r;
  g[1] = dwdr * dy / r;
  g[2] = dwdr * dz / r;
  return C * C;
}

/* What the reverse sweep needs of the positions x of step t besides x: the
 * weights and the count term's derivatives.  Every CTA of the cluster makes
 * all of it for itself in its own shared memory (sw: the weights) and the
 * first one keeps it; returns this thread's share of the count term. */
__device__ double place_terms(const Sys& S, const Buf& B, const double* x, int t, double* cent, double* sw,
                              double* red) {
  const bool lead = cg::this_cluster().block_rank() == 0;
  ion_centre(S, x, cent, red);
  for (int i = threadIdx.x; i < S.N; i += blockDim.x) {
    double g[3];
    const double w = weight_of(S, x, cent, i, g);
    sw[i] = w;
    if (lead) {
      B.w[(size_t)t * S.N + i] = w;
      for (int k = 0; k < 3; k++) B.dw[(size_t)t * 3 * S.N + 3 * i + k] = g[k];
    }
  }
  double jp = 0;
  if (lead && S.w_count != 0) {
    double C[3] = {0, 0, 0};
    double* const mg = B.mg + (size_t)t * 3 * (S.n_vmol + 1);
    for (int m = threadIdx.x; m < S.n_vmol; m += blockDim.x) {
      const int a0 = S.vmol_first + m * S.a_v;
      double cm[3] = {0, 0, 0};
      for (int a = 0; a < S.a_v; a++)
        for (int q = 0; q < 3; q++) cm[q] += __ldcg(x + 3 * (a0 + a) + q) * S.mass[a0 + a];
      for (int q = 0; q < 3; q++) cm[q] /= S.vmol_mass;
      double dv[3] = {cm[0] - cent[0], cm[1] - cent[1], cm[2] - cent[2]};
      double rho = sqrt(dv[0] * dv[0] + dv[1] * dv[1] + dv[2] * dv[2]);
      double sgm = 1.0 / (1.0 + exp((rho - S.R0) / S.W));
      jp += S.w_count * sgm;
      double dSdrho = -sgm * (1.0 - sgm) / S.W * S.w_count * S.inv_n;
      for (int q = 0; q < 3; q++) {
        const double c = dSdrho * dv[q] / rho;
        mg[3 * m + q] = c;
        C[q] += c;
      }
    }
    block_sum3(C, red);
    if (threadIdx.x < 3) mg[3 * S.n_vmol + threadIdx.x] = -C[threadIdx.x];
  }
  __syncthreads();
  return jp;
}

/* force factor f(u) and df/du of one pair (u = r^2), parameter derivatives
 * of f (d eps, d sigma, d s at s = 1) */
struct PairEval {
  double f, fp, fe, fs_sig, fq;
  double a7, b4; /* the two LJ terms of f */
  int p;  /* parameter base, -1 */
};

__device__ __forceinline__ PairEval eval_pair(const Sys& S, int i, int j, int kind, double u) {
  PairEval o;
  o.p = -1;
  o.fe = o.fs_sig = o.fq = o.a7 = o.b4 = 0;
  const int tt = S.type[i] * S.nt + S.type[j];
  const double ui = 1.0 / u;
  double f = 0, fp = 0;
  if (kind == PK_ION_BMH) {
    const double* cB = kBornD[S.bmh[i]][S.bmh[j]];
    double r = sqrt(u);
    double e = exp(cB[4] * (cB[3] - r));
    double qq = S.qqrd2e * S.q[i] * S.q[j];
    const double u3 = ui * ui * ui, u4 = u3 * ui;
    double g = cB[4] * cB[0] * r * e - cB[1] * u3 - cB[2] * u4 + qq / r;
    double gp = cB[4] * cB[0] * e * (1.0 - cB[4] * r) + (6.0 * cB[1] * u3 + 8.0 * cB[2] * u4 ) / r - qq * ui;
    f = g * ui;
    double dfdr = gp * ui - 2.0 * g * ui / r;
    fp = dfdr / (2.0 * r);
    o.fq = 2.0 * qq * ui / r; /* Coulomb scales as s^2 */
  } else {
    const double u2 = ui * ui, u4 = u2 * u2, u7 = u4 * u2 * ui;
    const double a7 = S.A[tt] * u7, b4 = S.B[tt] * u4;
    f = a7 - b4;
    fp = (4.0 * b4 - 7.0 * a7) * ui;
    o.a7 = a7;
    o.b4 = b4;
    if (kind == PK_GI || kind == PK_VI) {
      o.p = S.pidx[tt];
      if (o.p >= 0) {
        o.fe = f * S.ieps[tt];
        o.fs_sig = (12.0 * a7 - 6.0 * b4) * S.isig[tt];
      }
    }
    if (kind == PK_VI || kind == PK_VV || kind == PK_ION_LJC) {
      const double fc = S.qqrd2e * S.q[i] * S.q[j] * ui * sqrt(ui);
      f += fc;
      fp += -1.5 * fc * ui;
      if (kind == PK_VI) o.fq = fc;
      else if (kind == PK_ION_LJC) o.fq = 2.0 * fc;
    }
  }
  o.f = f;
  o.fp = fp;
  return o;
}

__device__ __forceinline__ double warp_sum_dd(double v) {
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
  return v;
}

/* 32 bonded terms 32 k .. of x into their rows of B.tb: their forces, or with
 * lam the products of their Jacobians (symmetric: F = -grad U) with lam by
 * forward mode */
template <class T>
__device__ __forceinline__ void bonded_rows(const Sys& S, const Buf& B, const double* x, const double* lam, int k) {
  constexpr bool dual = !std::is_same<T, double>::value;
  const int nb = S.n_bonds, na = S.n_angles, nd = S.n_dih;
  /* the long terms first; the rows are numbered bonds, angles, dihedrals */
  int t = 32 * k + (int)(threadIdx.x & 31);
  if (t >= nb + na + nd) return;
  t = t < nd ? nb + na + t : t < nd + na ? nb + t - nd : t - nd - na;
  int n;
  T X[4][3], f[4][3];
  const int* r;
  if (t < nb) { r = S.bonds + 3 * t; n = 2; }
  else if (t < nb + na) { r = S.angles + 4 * (t - nb); n = 3; }
  else { r = S.dih + 5 * (t - nb - na); n = 4; }
#pragma unroll
  for (int a = 0; a < 4; a++) {
    if (a >= n) break;
#pragma unroll
    for (int q = 0; q < 3; q++) {
      if constexpr (dual) X[a][q] = mk(__ldcg(x + 3 * r[a] + q), __ldcg(lam + 3 * r[a] + q));
      else X[a][q] = __ldcg(x + 3 * r[a] + q);
    }
  }
  if (n == 2) bond_t<T>(X, S.bond_c + 2 * r[2], f);
  else if (n == 3) angle_t<T>(X, S.angle_c + 2 * r[3], f);
  else dihedral_t<T>(X, S.dih_c + 15 * r[4], S.dih_multi[r[4]], f);
#pragma unroll
  for (int a = 0; a < 4; a++) {
    if (a >= n) break;
    double* const row = B.tb + 3 * (size_t)S.tb_at[4 * t + a];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      if constexpr (dual) row[q] = f[a][q].d;
      else row[q] = f[a][q];
    }
  }
}

/* the bonded terms' rows of component q of atom i, summed */
__device__ __forceinline__ double bonded_sum(const Sys& S, const Buf& B, int i, int q) {
  const int e1 = S.tb_off[i + 1];
  double t = 0;
#pragma unroll 16
  for (int e = S.tb_off[i]; e < e1; e++) t += __ldcg(B.tb + 3 * (size_t)e + q);
  return t;
}

/* The warp items of a force evaluation (or product), the CTA's own: bonded
 * terms by 32 (dual, and longest), then atoms, longest rows first.  Items are
 * dealt to the CTAs in turn and taken by the warps from a counter. */
template <class Bonded, class Row>
__device__ __forceinline__ void force_queue(const Sys& S, int* next, Bonded&& bonded, Row&& row) {
  const int nbk = (S.n_bonds + S.n_angles + S.n_dih + 31) >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cg::this_cluster().block_rank(), C = (int)cg::this_cluster().num_blocks();
  for (;;) {
    int it = 0;
    if (lane == 0) it = atomicAdd(next, 1);
    it = rank + __shfl_sync(0xffffffffu, it, 0) * C;
    if (it >= nbk + S.N) break;
    if (it < nbk) bonded(it);
    else row(S.row_order[it - nbk]);
    __syncwarp();
  }
}

/* pair forces on every atom into F (the bonded terms into B.tb); returns the
 * thread's share of the window's ion-vapor energy */
__device__ double force_rows(const Sys& S, const Buf& B, const double* x, const double* sw, double* F, int* next) {
  const int lane = threadIdx.x & 31;
  double jp = 0;
  force_queue(S, next, [&](int k) { bonded_rows<double>(S, B, x, nullptr, k); },
              [&](int i) {
                const double xi[3] = {__ldcg(x + 3 * i), __ldcg(x + 3 * i + 1), __ldcg(x + 3 * i + 2)};
                double a[3] = {0, 0, 0};
                for (int e = S.row_off[i] + lane; e < S.row_off[i + 1]; e += 32) {
                  const int2 pr = S.row[e];
                  const int j = pr.x, kind = pr.y & 7;
                  const double d0 = xi[0] - __ldcg(x + 3 * j), d1 = xi[1] - __ldcg(x + 3 * j + 1),
                               d2 = xi[2] - __ldcg(x + 3 * j + 2);
                  const double u = d0 * d0 + d1 * d1 + d2 * d2;
                  const PairEval ev = eval_pair(S, i, j, kind, u);
                  double g = ev.f;
                  if (kind == PK_VI || kind == PK_VV) g *= sw[i] * sw[j];
                  a[0] += g * d0;
                  a[1] += g * d1;
                  a[2] += g * d2;
                  /* U = u (a7 / 12 - b4 / 6) + u fc, fq = fc */
                  if (kind == PK_VI && (pr.y & kPrimary))
                    jp += S.w_energy * u * (ev.a7 * (1.0 / 12.0) - ev.b4 * (1.0 / 6.0) + ev.fq);
                }
                for (int k = 0; k < 3; k++) a[k] = warp_sum_dd(a[k]);
                if (lane < 3) {
                  double t = lane == 0 ? a[0] : lane == 1 ? a[1] : a[2];
                  if (S.efield_on && i < S.n_ion) t += 5.55e-5 * S.q[i] * S.efield[lane];
                  F[3 * i + lane] = t;
                }
              });
  return jp;
}

/* lx += J_F(x)^T lam (+ the objective's gradient when obj), the bonded terms'
 * products into B.tb, grad += (dF/dtheta)^T lam (+ the objective's); the
 * CTA's share of the weights' pull on the ion centre into B.part.  xs, ls: x
 * and lam in shared memory, or x and lam themselves where they do not fit.
 * qsum: the lane's share of the charge scale's derivative. */
template <bool STAGED>
__device__ __forceinline__ double at_of(const double* p, int q) {
  if (STAGED) return p[q];
  return __ldcg(p + q);
}
template <bool STAGED>
__device__ void vjp_rows(const Sys& S, const Buf& B, const double* x, int t, const double* xs, const double* ls,
                         bool obj, double* sgrad, double* spart, double& qsum, int* next) {
  const int lane = threadIdx.x & 31;
  const unsigned FULL = 0xffffffffu;
  const double* const w = B.w + (size_t)t * S.N;
  const double* const dw = B.dw + (size_t)t * 3 * S.N;
  const double* const mg = B.mg + (size_t)t * 3 * (S.n_vmol + 1);
  double pull = 0; /* lanes 0..2: component of the share */
  force_queue(
      S, next, [&](int k) { bonded_rows<Dual>(S, B, x, B.lf, k); },
      [&](int i) {
        double xi[3], li[3], a[3] = {0, 0, 0}, om = 0;
        for (int q = 0; q < 3; q++) {
          xi[q] = at_of<STAGED>(xs, 3 * i + q);
          li[q] = at_of<STAGED>(ls, 3 * i + q);
        }
        const int e1 = S.row_off[i + 1];
        const double wi = w[i];
        const bool vap = S.vapor[i] != 0;
        for (int e0 = S.row_off[i]; e0 < e1; e0 += 32) {
          int p = -1;
          double pe = 0, ps = 0;
          if (e0 + lane < e1) {
            const int2 pr = S.row[e0 + lane];
            const int j = pr.x, kind = pr.y & 7;
            const bool primary = (pr.y & kPrimary) != 0;
            double d[3], m[3];
            for (int q = 0; q < 3; q++) {
              d[q] = xi[q] - at_of<STAGED>(xs, 3 * j + q);
              m[q] = li[q] - at_of<STAGED>(ls, 3 * j + q);
            }
            const double u = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
            const PairEval ev = eval_pair(S, i, j, kind, u);
            const double dm = d[0] * m[0] + d[1] * m[1] + d[2] * m[2];
            double W = 1;
            if (kind == PK_VI || kind == PK_VV) {
              const double wj = w[j];
              W = wi * wj;
              if (vap) om += wj * (ev.f * dm);
            }
            const double cm = W * ev.f;
            double cd = W * (2.0 * ev.fp * dm);
            if (primary) {
              if (ev.p >= 0) {
                p = ev.p;
                pe = W * ev.fe * dm;
                ps = W * ev.fs_sig * dm;
              }
              qsum += W * ev.fq * dm;
            }
            if (obj && kind == PK_VI && S.w_energy != 0) {
              /* dU/du = -(a7 - b4 + fc) / 2 with fc = fq, U as in force_rows */
              const double sc = S.w_energy * S.inv_n;
              cd += sc * (ev.b4 - ev.a7 - ev.fq);
              if (primary) {
                if (p >= 0) {
                  const int tt = S.type[i] * S.nt + S.type[j];
                  pe += sc * u * (ev.a7 * (1.0 / 12.0) - ev.b4 * (1.0 / 6.0)) * S.ieps[tt];
                  ps += sc * u * (ev.a7 - ev.b4) * S.isig[tt];
                }
                qsum += sc * u * ev.fq;
              }
            }
            for (int q = 0; q < 3; q++) a[q] += cm * m[q] + cd * d[q];
          }
          /* parameter rows present in the warp, one after another */
          for (unsigned todo = __ballot_sync(FULL, p >= 0); todo;) {
            const int r = __shfl_sync(FULL, p, __ffs(todo) - 1);
            const double se = warp_sum_dd(p == r ? pe : 0.0), ss = warp_sum_dd(p == r ? ps : 0.0);
            if (lane == 0) {
              atomicAdd(&sgrad[r], se);
              atomicAdd(&sgrad[r + 1], ss);
            }
            todo &= ~__ballot_sync(FULL, p == r);
          }
        }
        for (int q = 0; q < 3; q++) a[q] = warp_sum_dd(a[q]);
        if (vap) om = warp_sum_dd(om);
        if (lane < 3) {
          double v = lane == 0 ? a[0] : lane == 1 ? a[1] : a[2];
          if (vap) {
            const double g = om * dw[3 * i + lane];
            v += g;
            pull += g;
            if (obj && S.w_count != 0)
              v += S.mass[i] / S.vmol_mass * mg[3 * ((i - S.vmol_first) / S.a_v) + lane];
          }
          if (S.efield_on && i < S.n_ion) qsum += 5.55e-5 * S.q[i] * S.efield[lane] * li[lane];
          B.lx[3 * i + lane] = __ldcg(B.lx + 3 * i + lane) + v;
        }
      });
  if (lane < 3) spart[3 * (threadIdx.x >> 5) + lane] = pull;
  __syncthreads();
  if (threadIdx.x < 3) {
    double v = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) v += spart[3 * k + threadIdx.x];
    B.part[3 * cg::this_cluster().block_rank() + threadIdx.x] = v;
  }
}

/* SHAKE of every constraint of y against the reference positions xr,
 * colour by colour; gam receives the accumulated multipliers */
__device__ void shake(const Sys& S, const Buf& B, double* y, const double* xr, double* gam) {
  for (int k = threadIdx.x; k < S.n_cons; k += blockDim.x) gam[k] = 0;
  __syncthreads();
  for (int sweep = 0; sweep < SHAKE_SWEEPS; sweep++) {
    for (int col = 0; col < S.n_colors; col++) {
      for (int k = threadIdx.x; k < S.n_cons; k += blockDim.x) {
        if (S.cons_color[k] != col) continue;
        const int i = S.cons[3 * k], j = S.cons[3 * k + 1];
        const double dk = S.bond_c[2 * S.cons[3 * k + 2] + 1];
        const double mi = S.mass[i], mj = S.mass[j];
        double r[3], s[3];
        for (int q = 0; q < 3; q++) {
          r[q] = xr[3 * i + q] - xr[3 * j + q];
          s[q] = y[3 * i + q] - y[3 * j + q];
        }
        double s2 = s[0] * s[0] + s[1] * s[1] + s[2] * s[2];
        double dot = r[0] * s[0] + r[1] * s[1] + r[2] * s[2];
        double minv = 1 / mi + 1 / mj;
        if (dot < 1e-10) dot = 1e-10;
        double g = (dk * dk - s2) / (2 * minv * dot);
        gam[k] += g;
        for (int q = 0; q < 3; q++) {
          y[3 * i + q] += r[q] * g / mi;
          y[3 * j + q] -= r[q] * g / mj;
        }
      }
      __syncthreads();
    }
    if (threadIdx.x == 0) B.flag[0] = 1;
    __syncthreads();
    for (int k = threadIdx.x; k < S.n_cons; k += blockDim.x) {
      const int i = S.cons[3 * k], j = S.cons[3 * k + 1];
      const double dk = S.bond_c[2 * S.cons[3 * k + 2] + 1];
      double s2 = 0;
      for (int q = 0; q < 3; q++) {
        double d = y[3 * i + q] - y[3 * j + q];
        s2 += d * d;
      }
      double dr = s2 - dk * dk;
      if (!(dr * dr <= 1e-20)) B.flag[0] = 0;
    }
    __syncthreads();
    const int conv = B.flag[0];
    __syncthreads();
    if (conv) return;
  }
  if (threadIdx.x == 0) B.flag[1] |= MDN_ST_SHAKE_NOCONV;
  __syncthreads();
}

/* adjoint of the converged projection x = y + sum_k g_k D_k r_k:
 * lam (adjoint of x) -> lam_y written into lam, and the g_k D_k dr_k terms
 * added into xb (adjoint of the reference positions xr) */
__device__ void shake_adjoint(const Sys& S, const Buf& B, const double* x, const double* xr, const double* gam,
                              double* lam, double* xb, double* sc) {
  /* the constraints are few: the first CTA of the cluster solves them with
   * block barriers (x-bar, which the other CTAs added to, read from L2), the
   * others wait at the cluster barrier below */
  if (S.n_cons > 0 && cg::this_cluster().block_rank() == 0) {
    /* G_{kl} = s_k . r_l * coef(k, l); G^T mu = rho, rho_l = r_l . (lam_i/m_i - lam_j/m_j) */
    for (int k = (int)threadIdx.x; k < S.n_cons; k += (int)blockDim.x) B.mu[k] = 0;
    __syncthreads();
    auto G = [&](int k, int l) {
      const int ik = S.cons[3 * k], jk = S.cons[3 * k + 1], il = S.cons[3 * l], jl = S.cons[3 * l + 1];
      double coef = 0;
      if (il == ik) coef += 1.0 / S.mass[il];
      if (jl == ik) coef -= 1.0 / S.mass[jl];
      if (il == jk) coef -= 1.0 / S.mass[il];
      if (jl == jk) coef += 1.0 / S.mass[jl];
      if (coef == 0) return 0.0;
      double sr = 0;
      for (int q = 0; q < 3; q++)
        sr += (x[3 * ik + q] - x[3 * jk + q]) * (xr[3 * il + q] - xr[3 * jl + q]);
      return sr * coef;
    };
    /* what the sweeps reuse, once per step into shared memory (sc): rho_l,
     * G_ll and G_kl of each neighbour entry */
    double* const srho = sc;
    double* const sdiag = sc + S.n_cons;
    double* const snb = sc + 2 * S.n_cons;
    for (int l = (int)threadIdx.x; l < S.n_cons; l += (int)blockDim.x) {
      const int il = S.cons[3 * l], jl = S.cons[3 * l + 1];
      double rho = 0;
      for (int q = 0; q < 3; q++) {
        double rl = xr[3 * il + q] - xr[3 * jl + q];
        rho += rl * (__ldcg(lam + 3 * il + q) / S.mass[il] - __ldcg(lam + 3 * jl + q) / S.mass[jl]);
      }
      srho[l] = rho;
      sdiag[l] = G(l, l);
      for (int e = S.cons_nb_off[l]; e < S.cons_nb_off[l + 1]; e++) snb[e] = G(S.cons_nb[e], l);
    }
    __syncthreads();
    for (int sweep = 0; sweep < SHAKE_SWEEPS; sweep++) {
      if ((int)threadIdx.x == 0) B.flag[0] = 1;
      __syncthreads();
      for (int col = 0; col < S.n_colors; col++) {
        for (int l = (int)threadIdx.x; l < S.n_cons; l += (int)blockDim.x) {
          if (S.cons_color[l] != col) continue;
          double acc = srho[l];
          for (int e = S.cons_nb_off[l]; e < S.cons_nb_off[l + 1]; e++) acc -= snb[e] * B.mu[S.cons_nb[e]];
          double nm = acc / sdiag[l];
          if (fabs(nm - B.mu[l]) > 1e-13 * (fabs(nm) + 1e-300)) B.flag[0] = 0;
          B.mu[l] = nm;
        }
        __syncthreads();
      }
      const int conv = B.flag[0];
      __syncthreads();
      if (conv) break;
    }
    /* lam_y = lam - sum_k mu_k B_k^T (B_k: +s_k at i_k, -s_k at j_k) */
    for (int k = (int)threadIdx.x; k < S.n_cons; k += (int)blockDim.x) {
      const int i = S.cons[3 * k], j = S.cons[3 * k + 1];
      const double mk_ = B.mu[k];
      for (int q = 0; q < 3; q++) {
        double sk = x[3 * i + q] - x[3 * j + q];
        atomicAdd(&lam[3 * i + q], -mk_ * sk);
        atomicAdd(&lam[3 * j + q], mk_ * sk);
      }
    }
    __syncthreads();
    /* g_l D_l dr_l: r_l = xr_i - xr_j */
    for (int l = (int)threadIdx.x; l < S.n_cons; l += (int)blockDim.x) {
      const int i = S.cons[3 * l], j = S.cons[3 * l + 1];
      for (int q = 0; q < 3; q++) {
        double t = gam[l] * (__ldcg(lam + 3 * i + q) / S.mass[i] - __ldcg(lam + 3 * j + q) / S.mass[j]);
        atomicAdd(&xb[3 * i + q], t);
        atomicAdd(&xb[3 * j + q], -t);
      }
    }
    __syncthreads();
  }
  csync();
}

/* The values of one component of a unit's constraints in every lane of its
 * warp: lane 3 a + q holds component q of the unit's atom a */
__device__ __forceinline__ double comp(double v, int a, int q) { return __shfl_sync(0xffffffffu, v, 3 * a + q); }

/* A d = b for up to three unknowns (identity rows past n), Cramer's rule;
 * false when A is singular (a constraint given twice) */
__device__ __forceinline__ bool solve3(const double (*A)[3], const double* b, double* d) {
  const double c00 = A[1][1] * A[2][2] - A[1][2] * A[2][1];
  const double c01 = A[1][0] * A[2][2] - A[1][2] * A[2][0];
  const double c02 = A[1][0] * A[2][1] - A[1][1] * A[2][0];
  const double det = A[0][0] * c00 - A[0][1] * c01 + A[0][2] * c02;
  if (!(fabs(det) > 1e-300)) return false;
  const double inv = 1.0 / det;
  const double e12 = b[1] * A[2][2] - A[1][2] * b[2], e11 = b[1] * A[2][1] - A[1][1] * b[2],
               e10 = A[1][0] * b[2] - b[1] * A[2][0];
  d[0] = (b[0] * c00 - A[0][1] * e12 + A[0][2] * e11) * inv;
  d[1] = (A[0][0] * e12 - b[0] * c01 + A[0][2] * e10) * inv;
  d[2] = (-A[0][0] * e11 - A[0][1] * e10 + b[0] * c02) * inv;
  return true;
}

/* a unit's constraints in registers */
struct UnitCons {
  int nc, ci[3], cj[3];
  double cf[3][3];
  __device__ __forceinline__ explicit UnitCons(const Unit& U) : nc(U.nc) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      ci[k] = U.ci[k];
      cj[k] = U.cj[k];
#pragma unroll
      for (int l = 0; l < 3; l++) cf[k][l] = U.cf[k][l];
    }
  }
};
__device__ __forceinline__ double pick(const double* v, int q) { return q == 0 ? v[0] : q == 1 ? v[1] : v[2]; }

/* Newton's method on a unit's constraints: y (this lane's component, im its
 * atom's inverse mass) moves along the reference bond vectors of xr; gam: the
 * multipliers.  One step past the sweeps' criterion, (|s|^2 - d^2)^2 <= 1e-20
 * A^4, which brings the residuals to rounding.  After 50 steps, or with a
 * singular system, the sweeps from the start, as for larger groups (shake);
 * false when they reach their cap. */
__device__ __forceinline__ bool unit_shake(const UnitCons& U, const double* d2, double im, double& y, double xr,
                                           double* gam) {
  const int lane = threadIdx.x & 31, a = lane / 3, q = lane - 3 * a;
  double r[3][3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    gam[k] = 0;
    if (k >= U.nc) continue;
#pragma unroll
    for (int c = 0; c < 3; c++) r[k][c] = comp(xr, U.ci[k], c) - comp(xr, U.cj[k], c);
  }
  const double y0 = y;
  bool done = false;
  for (int it = 0; it < 50; it++) {
    double A[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}}, b[3] = {0, 0, 0}, d[3];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      if (k >= U.nc) continue;
      double sk[3];
#pragma unroll
      for (int c = 0; c < 3; c++) sk[c] = comp(y, U.ci[k], c) - comp(y, U.cj[k], c);
      b[k] = d2[k] - (sk[0] * sk[0] + sk[1] * sk[1] + sk[2] * sk[2]);
      if (!(b[k] * b[k] <= 1e-20)) ok = false;
#pragma unroll
      for (int l = 0; l < 3; l++)
        if (l < U.nc) A[k][l] = 2.0 * (sk[0] * r[l][0] + sk[1] * r[l][1] + sk[2] * r[l][2]) * U.cf[k][l];
    }
    if (ok && done) return true;
    done = ok;
    if (!solve3(A, b, d)) break;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      if (k >= U.nc) continue;
      gam[k] += d[k];
      const double rq = d[k] * pick(r[k], q) * im;
      if (a == U.ci[k]) y += rq;
      if (a == U.cj[k]) y -= rq;
    }
  }
  y = y0;
  gam[0] = gam[1] = gam[2] = 0;
  for (int sweep = 0; sweep < SHAKE_SWEEPS; sweep++) {
    bool ok = true;
    for (int pass = 0; pass < 2; pass++) /* the sweep, then the residuals */
#pragma unroll
      for (int k = 0; k < 3; k++) {
        if (k >= U.nc) continue;
        double s2 = 0, dot = 0;
#pragma unroll
        for (int c = 0; c < 3; c++) {
          const double s = comp(y, U.ci[k], c) - comp(y, U.cj[k], c);
          s2 += s * s;
          dot += s * r[k][c];
        }
        const double res = d2[k] - s2;
        if (pass == 1) {
          if (!(res * res <= 1e-20)) ok = false;
          continue;
        }
        if (dot < 1e-10) dot = 1e-10;
        const double g = res / (2 * U.cf[k][k] * dot);
        gam[k] += g;
        const double rq = g * pick(r[k], q) * im;
        if (a == U.ci[k]) y += rq;
        if (a == U.cj[k]) y -= rq;
      }
    if (ok) return true;
  }
  return false;
}

/* Adjoint of a unit's converged projection x = y + sum_k g_k D_k r_k: lam
 * (this lane's component of the adjoint of x) becomes that of y; returns what
 * goes into the adjoint of the reference positions xr */
__device__ __forceinline__ double unit_shake_adjoint(const UnitCons& U, double im, double x, double xr,
                                                     const double* gam, double& lam) {
  const int lane = threadIdx.x & 31, a = lane / 3, q = lane - 3 * a;
  double sk[3][3], A[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}}, rho[3] = {0, 0, 0}, mu[3];
  const double lm = lam * im;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    if (k >= U.nc) continue;
#pragma unroll
    for (int c = 0; c < 3; c++) sk[k][c] = comp(x, U.ci[k], c) - comp(x, U.cj[k], c);
  }
#pragma unroll
  for (int l = 0; l < 3; l++) {
    if (l >= U.nc) continue;
    double r[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      r[c] = comp(xr, U.ci[l], c) - comp(xr, U.cj[l], c);
      rho[l] += r[c] * (comp(lm, U.ci[l], c) - comp(lm, U.cj[l], c));
    }
#pragma unroll
    for (int k = 0; k < 3; k++)
      if (k < U.nc) A[l][k] = (sk[k][0] * r[0] + sk[k][1] * r[1] + sk[k][2] * r[2]) * U.cf[k][l];
  }
  if (!solve3(A, rho, mu)) {
    /* the sweeps of shake_adjoint */
    mu[0] = mu[1] = mu[2] = 0;
    bool ok = false;
    for (int sweep = 0; sweep < SHAKE_SWEEPS && !ok; sweep++) {
      ok = true;
#pragma unroll
      for (int l = 0; l < 3; l++) {
        if (l >= U.nc) continue;
        double acc = rho[l];
#pragma unroll
        for (int k = 0; k < 3; k++)
          if (k != l && k < U.nc) acc -= A[l][k] * mu[k];
        const double nm = acc / A[l][l];
        if (fabs(nm - mu[l]) > 1e-13 * (fabs(nm) + 1e-300)) ok = false;
        mu[l] = nm;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 3; k++) {
    if (k >= U.nc) continue;
    const double s = mu[k] * pick(sk[k], q);
    if (a == U.ci[k]) lam -= s;
    if (a == U.cj[k]) lam += s;
  }
  const double ly = lam * im;
  double xb = 0;
#pragma unroll
  for (int l = 0; l < 3; l++) {
    if (l >= U.nc) continue;
    double d[3];
#pragma unroll
    for (int c = 0; c < 3; c++) d[c] = comp(ly, U.ci[l], c) - comp(ly, U.cj[l], c);
    const double t = gam[l] * pick(d, q);
    if (a == U.ci[l]) xb += t;
    if (a == U.cj[l]) xb -= t;
  }
  return xb;
}

/* Every segment's recompute at once, one cluster each: cluster s starts from
 * checkpoint s (cpx, cpv) and writes its segment's positions, multipliers,
 * weights and count-term derivatives.  first: the window's first segment
 * takes the start forces that the state holds (f0; zero on a replica that was
 * never stepped, since the reference evaluates no force before the first
 * kick), the others evaluate F(x_0).  A step is: kick, kick, drift and
 * constraints by units | everything that depends on the new positions.
 * Jseg[CTA] = its share of the segment's objective sum, flags[2 s + 1] the
 * SHAKE status.  sw_smem = 0: the weights do not fit shared memory (one CTA
 * per segment then). */
__global__ void __launch_bounds__(ADJ_THREADS, 1) adjoint_recompute(Sys S, Buf B, int K, long long n_steps,
                                                                    const double* cpx, const double* cpv,
                                                                    const double* f0, double* Jseg, int sw_smem) {
  __shared__ double red[72];
  __shared__ double cent[3];
  __shared__ int next;
  extern __shared__ double csh[];
  const int s = (int)(blockIdx.x / cg::this_cluster().num_blocks());
  const int n3 = 3 * S.N, lane = threadIdx.x & 31;
  const int Ks = (int)min((long long)K, n_steps - (long long)s * K);
  Buf b = B;
  b.X += (size_t)s * (K + 1) * n3;
  b.V += (size_t)s * n3;
  b.F += (size_t)s * n3;
  b.gam += (size_t)s * K * max(S.n_cons, 1);
  b.w += (size_t)s * (K + 1) * S.N;
  b.dw += (size_t)s * (K + 1) * n3;
  b.mg += (size_t)s * (K + 1) * 3 * (S.n_vmol + 1);
  b.tb += (size_t)s * 12 * max(1, S.n_bonds + S.n_angles + S.n_dih);
  b.flag += 2 * s;
  for (int q = ctid(); q < n3; q += cnthr()) {
    b.X[q] = cpx[(size_t)s * n3 + q];
    b.V[q] = cpv[(size_t)s * n3 + q];
    if (s == 0) b.F[q] = f0[q];
  }
  if (ctid() == 0) b.flag[1] = 0;
  double jacc = 0;
  for (int t = 0; t <= Ks; t++) {
    double* const x1 = b.X + (size_t)t * n3;
    if (t > 0) {
      const double* const x0 = x1 - n3;
      double* const gam = b.gam + (size_t)(t - 1) * S.n_cons;
      const bool bonded = t > 1 || s > 0; /* F holds the pair forces alone */
      for (int u = cwarp(); u < S.n_units; u += cnwarps()) {
        const Unit& U = S.units[u];
        const bool on = lane < 3 * U.na;
        const int i = U.atom[on ? lane / 3 : 0], q = 3 * i + lane % 3;
        double xo = 0, va = 0, y = 0, g[3], d2[3] = {U.d2[0], U.d2[1], U.d2[2]};
        const UnitCons uc(U);
        const double im = on ? 1.0 / S.mass[i] : 0.0;
        if (on) {
          const double c = S.c[i], f = __ldcg(b.F + q) + (bonded ? bonded_sum(S, b, i, lane % 3) : 0.0);
          va = __ldcg(b.V + q);
          if (t > 1) va += c * f;
          va += c * f;
          xo = __ldcg(x0 + q);
          y = xo + S.dt * va;
        }
        const double yd = y;
        if (uc.nc > 0) {
          if (!unit_shake(uc, d2, im, y, xo, g) && lane == 0) b.flag[1] = MDN_ST_SHAKE_NOCONV;
          if (S.vcorr) va += (y - yd) / S.dt;
          if (lane < uc.nc) gam[U.cons[lane]] = pick(g, lane);
        }
        if (on) {
          x1[q] = y;
          b.V[q] = va;
        }
      }
      if (S.n_units == 0) { /* one CTA */
        for (int q = threadIdx.x; q < n3; q += blockDim.x) {
          const int i = q / 3;
          const double f = b.F[q] + (bonded ? bonded_sum(S, b, i, q - 3 * i) : 0.0);
          double va = b.V[q];
          if (t > 1) va += S.c[i] * f;
          va += S.c[i] * f;
          b.V[q] = va;
          x1[q] = x0[q] + S.dt * va;
        }
        __syncthreads();
        shake(S, b, x1, x0, gam);
        if (S.vcorr)
          for (int q = threadIdx.x; q < n3; q += blockDim.x) {
            double y = x0[q] + S.dt * b.V[q];
            b.V[q] += (x1[q] - y) / S.dt;
          }
      }
    }
    if (threadIdx.x == 0) next = 0;
    csync();
    double* const sw = sw_smem ? csh : b.w + (size_t)t * S.N;
    const double jc = place_terms(S, b, x1, t, cent, sw, red);
    double je = 0;
    if (t > 0 || s > 0) je = force_rows(S, b, x1, sw, b.F, &next);
    if (t > 0) jacc += jc + je;
    csync();
  }
  jacc = block_sum(jacc, red);
  if (threadIdx.x == 0) Jseg[blockIdx.x] = jacc;
}

/* The reverse sweep of one segment over its recomputed trajectory (B
 * pointing at it), last step first, on one cluster; the adjoints of x, v, F
 * carry over from the segment after it.  A step is: the force product by
 * atoms | by units, what remains of the product (bonded rows, the weights'
 * pull on the ion centre), the adjoints of the constraints, the drift and
 * the first kick, and of the second kick of the step before it.  f0_theta = 1
 * on the first segment when its start forces came from a force evaluation at
 * x_0, whose parameter dependence then enters the gradient.  STAGED: x and
 * the force adjoint fit shared memory. */
template <bool STAGED>
__global__ void __launch_bounds__(ADJ_THREADS, 1) adjoint_segment(Sys S, Buf B, int K, int first, int f0_theta) {
  __shared__ double sgrad[MAX_PARAMS];
  __shared__ double spart[3 * (ADJ_THREADS / 32)];
  __shared__ double red[40];
  __shared__ int next;
  extern __shared__ double csh[]; /* x and lam when staged, then 2 n_cons + n_cons_nb doubles for shake_adjoint */
  const int n3 = 3 * S.N, lane = threadIdx.x & 31;
  double* const xs = csh;
  double* const ls = csh + n3;
  const bool vc = S.n_cons > 0 && S.vcorr;
  double qsum = 0;
  for (int p = threadIdx.x; p < S.n_params; p += blockDim.x) sgrad[p] = 0;
  /* (6) of the segment's last step: F-bar += c V-bar */
  for (int q = ctid(); q < n3; q += cnthr()) B.lf[q] = __ldcg(B.lf + q) + S.c[q / 3] * __ldcg(B.lv + q);
  csync();
  for (int t = K; t >= 0; t--) {
    if (t == 0 && !(first && f0_theta)) break;
    const double* x1 = B.X + (size_t)t * n3;
    /* objective at x_t and (5): x-bar += J^T F-bar; at t = 0 only for the
     * parameters of F(x_0) */
    if (threadIdx.x == 0) next = 0;
    if (STAGED)
      for (int q = threadIdx.x; q < n3; q += blockDim.x) {
        xs[q] = x1[q];
        ls[q] = __ldcg(B.lf + q);
      }
    __syncthreads();
    vjp_rows<STAGED>(S, B, x1, t, STAGED ? xs : x1, STAGED ? ls : B.lf, t > 0, sgrad, spart, qsum, &next);
    csync();
    if (t == 0) break;
    const double* x0 = x1 - n3;
    const double* const gam = B.gam + (size_t)(t - 1) * S.n_cons;
    const double* const mg = B.mg + (size_t)t * 3 * (S.n_vmol + 1) + 3 * S.n_vmol;
    double pull[3];
#pragma unroll
    for (int k = 0; k < 3; k++)
      pull[k] = mg[k] - warp_sum_dd(lane < (int)cg::this_cluster().num_blocks() ? __ldcg(B.part + 3 * lane + k) : 0.0);
    /* what the force product leaves to the owner of component q of atom i */
    auto rest = [&](int i, int k) {
      double v = bonded_sum(S, B, i, k);
      if (i < S.n_ion) v += S.mass[i] / S.ion_msum * (k == 0 ? pull[0] : k == 1 ? pull[1] : pull[2]);
      return v;
    };
    /* (2) y = x + dt v_a; (1) v_a = v + c F; (6) of the step before */
    auto carry = [&](int q, double ly, double xb, double lv) {
      const double lva = lv + S.dt * ly, cl = S.c[q / 3] * lva;
      B.lx[q] = ly + xb;
      B.lv[q] = lva;
      B.lf[q] = t > 1 ? cl + cl : cl;
    };
    for (int u = cwarp(); u < S.n_units; u += cnwarps()) {
      const Unit& U = S.units[u];
      const bool on = lane < 3 * U.na;
      const int k = lane % 3, i = U.atom[on ? lane / 3 : 0], q = 3 * i + k;
      double lam = 0, lv = 0, xb = 0, g[3] = {0, 0, 0};
      const UnitCons uc(U);
      const double im = on ? 1.0 / S.mass[i] : 0.0, xq = on ? x1[q] : 0.0, xo = on ? x0[q] : 0.0;
#pragma unroll
      for (int c = 0; c < 3; c++)
        if (c < uc.nc) g[c] = gam[U.cons[c]];
      if (on) {
        lv = __ldcg(B.lv + q);
        /* (4): v_b = v_a + (x_t - y)/dt */
        lam = __ldcg(B.lx + q) + rest(i, k) + (vc ? lv / S.dt : 0.0);
      }
      if (uc.nc > 0) xb = unit_shake_adjoint(uc, im, xq, xo, g, lam);
      if (on) carry(q, vc ? lam - lv / S.dt : lam, xb, lv);
    }
    if (S.n_units == 0) {
      for (int q = ctid(); q < n3; q += cnthr()) {
        B.lx[q] = __ldcg(B.lx + q) + rest(q / 3, q % 3) + (vc ? B.lv[q] / S.dt : 0.0);
        B.xb[q] = 0;
      }
      csync();
      shake_adjoint(S, B, x1, x0, gam, B.lx, B.xb, STAGED ? csh + 2 * n3 : csh);
      for (int q = ctid(); q < n3; q += cnthr()) {
        const double lv = B.lv[q], ly = __ldcg(B.lx + q);
        carry(q, vc ? ly - lv / S.dt : ly, __ldcg(B.xb + q), lv);
      }
    }
    csync();
  }
  qsum = block_sum(qsum, red);
  if (threadIdx.x == 0) sgrad[S.n_params - 1] += qsum;
  __syncthreads();
  /* the CTAs' shares of the gradient */
  for (int p = threadIdx.x; p < S.n_params; p += blockDim.x)
    if (sgrad[p] != 0) atomicAdd(B.grad + p, sgrad[p]);
}

/* ------------------------------------------------------------------------- */
/* host side                                                                   */
/* ------------------------------------------------------------------------- */
int err(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  return mdn_error(code, buf);
}

struct ParamRow {
  int kind, ta, tb;
};

/* the parameter rows of a descriptor, in the documented order */
std::vector<ParamRow> param_rows(const mdn_replica_desc* d) {
  std::set<int> gt, it, vt;
  for (int i = 0; i < d->gas.n_atoms; i++) gt.insert(d->gas.type[i]);
  for (int i = 0; i < d->ion.n_atoms; i++) it.insert(d->ion.type[i]);
  for (int i = 0; i < d->vapor.n_atoms; i++) vt.insert(d->vapor.type[i]);
  std::vector<ParamRow> rows;
  if (d->interactions & MDN_I_GI)
    for (int g : gt)
      for (int i : it) rows.push_back({0, g, i});
  if (d->interactions & MDN_I_VI)
    for (int v : vt)
      for (int i : it) rows.push_back({1, v, i});
  rows.push_back({2, 0, 0});
  return rows;
}

/* device memory of the call, listed in owned; a failed allocation is a null
 * there, and its error is not left for a later call to read */
void* dalloc(size_t bytes, std::vector<void*>& owned) {
  void* p = nullptr;
  if (cudaMalloc(&p, bytes) != cudaSuccess) {
    cudaGetLastError();
    p = nullptr;
  }
  owned.push_back(p);
  return p;
}

template <class T>
T* dput(const std::vector<T>& v, std::vector<void*>& owned) {
  T* const p = (T*)dalloc(sizeof(T) * std::max<size_t>(v.size(), 1), owned);
  if (p && !v.empty()) cudaMemcpy(p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice);
  return p;
}

template <class T>
T* dzero(size_t n, std::vector<void*>& owned) {
  T* const p = (T*)dalloc(sizeof(T) * std::max<size_t>(n, 1), owned);
  if (p) cudaMemset(p, 0, sizeof(T) * std::max<size_t>(n, 1));
  return p;
}

}  // namespace

extern "C" int mdn_adjoint_params(const mdn_replica_desc* d, int* n_params, int* rows, int capacity) {
  if (!d || !n_params) return err(MDN_ERR_ARG, "mdn_adjoint_params: null argument");
  std::vector<ParamRow> r = param_rows(d);
  *n_params = 2 * (int)(r.size() - 1) + 1;
  if (rows)
    for (int k = 0; k < (int)r.size() && k < capacity; k++) {
      rows[3 * k] = r[k].kind;
      rows[3 * k + 1] = r[k].ta;
      rows[3 * k + 2] = r[k].tb;
    }
  return MDN_OK;
}

extern "C" int mdn_adjoint(mdn_handle* h, const mdn_replica_desc* d, const mdn_adjoint_spec* spec, double* J,
                           double* grad, double* ms) {
  if (!h || !d || !spec || !J || !grad) return err(MDN_ERR_ARG, "mdn_adjoint: null argument");
  SnapshotArgs sa;
  mdn_snapshot_args(h, &sa);
  if (sa.R != 1) return err(MDN_ERR_ARG, "mdn_adjoint needs a handle with one replica (it has %d)", sa.R);
  if (spec->n_steps <= 0 || spec->checkpoint_every <= 0)
    return err(MDN_ERR_ARG, "mdn_adjoint: n_steps and checkpoint_every must be positive");
  if (d->nvt_mode != MDN_NVT_OFF) return err(MDN_ERR_ARG, "mdn_adjoint: the thermostat must be off");
  if (d->interactions & MDN_I_GG) return err(MDN_ERR_ARG, "mdn_adjoint: gg is not available");
  if (spec->count_width <= 0) return err(MDN_ERR_ARG, "mdn_adjoint: count_width must be positive");
  cudaSetDevice(sa.dev);
  const unsigned quirks = mdn_internal_quirks(h);
  mdn_replica_info info;
  int rc = mdn_replica_info_get(h, 0, &info);
  if (rc) return rc;
  if ((long long)info.loop_pair + spec->n_steps > info.loop_update)
    return err(MDN_ERR_ARG,
               "mdn_adjoint: the window of %lld steps crosses the rebuild after %d more steps; shorten it or "
               "raise the margin",
               spec->n_steps, info.loop_update - info.loop_pair);
  /* ---- the state at the window start and the dense atom order (the order
   * of the snapshot gather: ion, in-domain gas molecules, in-domain vapor) */
  const int ni = info.n_ion, ag = info.gas_atoms, av = info.vapor_atoms, ng = info.n_gas, nv = info.n_vapor;
  const size_t nm = 1 + (size_t)ng + nv;
  std::vector<double> ion_x(3 * ni), ion_v(3 * ni), ion_f(3 * ni), mol_x(3 * nm), mol_v(3 * nm);
  std::vector<unsigned char> region(nm);
  std::vector<double> gx(3 * (size_t)ng * ag), gvv(gx.size()), gf(gx.size());
  std::vector<double> vx(3 * (size_t)nv * av), vvv(vx.size()), vf(vx.size()), vw((size_t)nv * av);
  mdn_state st;
  memset(&st, 0, sizeof st);
  st.ion_x = ion_x.data(); st.ion_v = ion_v.data(); st.ion_f = ion_f.data();
  st.mol_x = mol_x.data(); st.mol_v = mol_v.data(); st.region = region.data();
  st.gas_ax = gx.data(); st.gas_av = gvv.data(); st.gas_af = gf.data();
  st.vap_ax = vx.data(); st.vap_av = vvv.data(); st.vap_af = vf.data(); st.vap_w = vw.data();
  if ((rc = mdn_download_state(h, 0, &st))) return rc;
  std::vector<int> gin, vin;
  for (int q = 0; q < ng; q++)
    if (region[1 + q]) gin.push_back(q);
  for (int q = 0; q < nv; q++)
    if (region[1 + ng + q]) vin.push_back(q);
  const int N = ni + (int)gin.size() * ag + (int)vin.size() * av;
  const int gas0 = ni, vap0 = ni + (int)gin.size() * ag;
  std::vector<int> gslot(ng, -1), vslot(nv, -1);
  for (size_t k = 0; k < gin.size(); k++) gslot[gin[k]] = (int)k;
  for (size_t k = 0; k < vin.size(); k++) vslot[vin[k]] = (int)k;
  std::vector<double> x0(3 * (size_t)N), v0(3 * (size_t)N);
  std::vector<int> type(N);
  std::vector<double> q(N), mass(N), cc(N);
  std::vector<unsigned char> isvap(N, 0);
  std::vector<int> bmh(N, 0);
  auto put = [&](int a, const double* xs, const double* vs, int t, double qa) {
    for (int k = 0; k < 3; k++) {
      x0[3 * a + k] = xs[k];
      v0[3 * a + k] = vs[k];
    }
    type[a] = t;
    q[a] = qa;
    mass[a] = d->atom_mass[t];
    cc[a] = 0.5 * d->dt * 4.184e-4 / d->atom_mass[t];
  };
  for (int i = 0; i < ni; i++) {
    put(i, &ion_x[3 * i], &ion_v[3 * i], d->ion.type[i], d->ion.charge[i]);
    bmh[i] = d->ion_bmh_type ? d->ion_bmh_type[i] : 0;
  }
  for (size_t k = 0; k < gin.size(); k++)
    for (int a = 0; a < ag; a++) {
      size_t src = 3 * ((size_t)gin[k] * ag + a);
      put(gas0 + (int)k * ag + a, &gx[src], &gvv[src], d->gas.type[a], d->gas.charge[a]);
    }
  for (size_t k = 0; k < vin.size(); k++)
    for (int a = 0; a < av; a++) {
      size_t src = 3 * ((size_t)vin[k] * av + a);
      const int at = vap0 + (int)k * av + a;
      put(at, &vx[src], &vvv[src], d->vapor.type[a], d->vapor.charge[a]);
      isvap[at] = 1;
    }
  /* ---- pairs ---- */
  const unsigned I = d->interactions;
  std::vector<int> pi, pj;
  std::vector<unsigned char> pk;
  auto addp = [&](int i, int j, int k) {
    pi.push_back(i);
    pj.push_back(j);
    pk.push_back((unsigned char)k);
  };
  if (I & MDN_I_GI) {
    int cnt = 0;
    if ((rc = mdn_pair_list(h, 0, 0, nullptr, 0, &cnt))) return rc;
    std::vector<int> pl(2 * (size_t)std::max(cnt, 1));
    if ((rc = mdn_pair_list(h, 0, 0, pl.data(), cnt, &cnt))) return rc;
    for (int e = 0; e < cnt; e++) {
      const int g = pl[2 * e], j = pl[2 * e + 1];
      if (gslot[g] < 0) return err(MDN_ERR_ARG, "mdn_adjoint: gas-ion list names molecule %d outside the domain", g);
      for (int a = 0; a < ag; a++) addp(gas0 + gslot[g] * ag + a, j, PK_GI);
    }
  }
  if (I & MDN_I_GV) {
    int cnt = 0;
    if ((rc = mdn_pair_list(h, 0, 1, nullptr, 0, &cnt))) return rc;
    std::vector<int> pl(2 * (size_t)std::max(cnt, 1));
    if ((rc = mdn_pair_list(h, 0, 1, pl.data(), cnt, &cnt))) return rc;
    const int nj = (quirks & MDN_Q_GV_GAS_COUNT) ? std::min(ag, av) : av;
    for (int e = 0; e < cnt; e++) {
      const int g = pl[2 * e], m = pl[2 * e + 1];
      if (gslot[g] < 0 || vslot[m] < 0) return err(MDN_ERR_ARG, "mdn_adjoint: gas-vapor list outside the domain");
      for (int a = 0; a < ag; a++)
        for (int b = 0; b < nj; b++) addp(gas0 + gslot[g] * ag + a, vap0 + vslot[m] * av + b, PK_GV);
    }
  }
  const int nvin = (int)vin.size();
  if (I & MDN_I_VI)
    for (int k = 0; k < nvin; k++)
      for (int a = 0; a < av; a++)
        for (int j = 0; j < ni; j++) addp(vap0 + k * av + a, j, PK_VI);
  if (I & MDN_I_VV)
    for (int k = 0; k < nvin; k++)
      for (int l = k + 1; l < nvin; l++)
        for (int a = 0; a < av; a++)
          for (int b = 0; b < av; b++) addp(vap0 + k * av + a, vap0 + l * av + b, PK_VV);
  if (I & MDN_I_AMBER) {
    std::vector<char> ex((size_t)ni * ni, 0);
    auto mark = [&](int a, int b) { ex[(size_t)a * ni + b] = ex[(size_t)b * ni + a] = 1; };
    for (int k = 0; k < d->ion.n_bonds; k++) mark(d->ion.bonds[3 * k], d->ion.bonds[3 * k + 1]);
    for (int k = 0; k < d->ion.n_rigid; k++) mark(d->ion.rigid[3 * k], d->ion.rigid[3 * k + 1]);
    for (int k = 0; k < d->ion.n_angles; k++) mark(d->ion.angles[4 * k], d->ion.angles[4 * k + 2]);
    for (int k = 0; k < d->ion.n_dihedrals; k++) mark(d->ion.dihedrals[5 * k], d->ion.dihedrals[5 * k + 3]);
    for (int i = 0; i < ni; i++)
      for (int j = i + 1; j < ni; j++)
        if (!ex[(size_t)i * ni + j]) addp(i, j, PK_ION_LJC);
  }
  if (I & MDN_I_BMH)
    for (int i = 0; i < ni; i++)
      for (int j = i + 1; j < ni; j++) addp(i, j, PK_ION_BMH);
  /* ---- bonded terms and constraints ---- */
  std::vector<int> bonds, angles, dih, cons;
  auto add_top = [&](const mdn_topology& t, int base, bool bonded) {
    if (bonded) {
      for (int k = 0; k < t.n_bonds; k++)
        bonds.insert(bonds.end(), {base + t.bonds[3 * k], base + t.bonds[3 * k + 1], t.bonds[3 * k + 2]});
      for (int k = 0; k < t.n_angles; k++)
        angles.insert(angles.end(), {base + t.angles[4 * k], base + t.angles[4 * k + 1], base + t.angles[4 * k + 2],
                                     t.angles[4 * k + 3]});
      for (int k = 0; k < t.n_dihedrals; k++)
        dih.insert(dih.end(), {base + t.dihedrals[5 * k], base + t.dihedrals[5 * k + 1], base + t.dihedrals[5 * k + 2],
                               base + t.dihedrals[5 * k + 3], t.dihedrals[5 * k + 4]});
    }
    if (I & MDN_I_SHAKE)
      for (int k = 0; k < t.n_rigid; k++)
        cons.insert(cons.end(), {base + t.rigid[3 * k], base + t.rigid[3 * k + 1], t.rigid[3 * k + 2]});
  };
  add_top(d->ion, 0, (I & MDN_I_AMBER) != 0);
  for (size_t k = 0; k < gin.size(); k++) add_top(d->gas, gas0 + (int)k * ag, (I & MDN_I_GAS_INTRA) != 0);
  for (size_t k = 0; k < vin.size(); k++) add_top(d->vapor, vap0 + (int)k * av, (I & MDN_I_VAPOR_INTRA) != 0);
  const int ncons = (int)cons.size() / 3;
  std::vector<int> color(ncons, 0);
  int ncolors = ncons ? 1 : 0;
  std::vector<std::vector<int>> by_atom(N);
  for (int k = 0; k < ncons; k++) {
    by_atom[cons[3 * k]].push_back(k);
    by_atom[cons[3 * k + 1]].push_back(k);
  }
  for (int k = 0; k < ncons; k++) {
    std::set<int> used;
    for (int a : {cons[3 * k], cons[3 * k + 1]})
      for (int l : by_atom[a])
        if (l < k) used.insert(color[l]);
    int c = 0;
    while (used.count(c)) c++;
    color[k] = c;
    ncolors = std::max(ncolors, c + 1);
  }
  std::vector<int> nboff(ncons + 1, 0), nb;
  for (int k = 0; k < ncons; k++) {
    std::set<int> s;
    for (int a : {cons[3 * k], cons[3 * k + 1]})
      for (int l : by_atom[a])
        if (l != k) s.insert(l);
    nb.insert(nb.end(), s.begin(), s.end());
    nboff[k + 1] = (int)nb.size();
  }
  /* ---- parameters ---- */
  const int nt = d->n_atom_types;
  std::vector<double> A((size_t)nt * nt), Bt((size_t)nt * nt), E((size_t)nt * nt), Sg((size_t)nt * nt);
  for (int i = 0; i < nt; i++)
    for (int j = 0; j < nt; j++) {
      const size_t t = (size_t)i * nt + j;
      E[t] = d->pair_eps ? d->pair_eps[t] : sqrt(d->atom_eps[i] * d->atom_eps[j]);
      Sg[t] = d->pair_sigma ? d->pair_sigma[t] : (d->atom_sigma[i] + d->atom_sigma[j]) * 0.5;
      A[t] = 48 * E[t] * pow(Sg[t], 12.0);
      Bt[t] = 24 * E[t] * pow(Sg[t], 6.0);
    }
  std::vector<ParamRow> rows = param_rows(d);
  const int n_params = 2 * (int)(rows.size() - 1) + 1;
  if (n_params > MAX_PARAMS) return err(MDN_ERR_CAPACITY, "mdn_adjoint: %d parameters, at most %d", n_params, MAX_PARAMS);
  std::vector<int> pidx((size_t)nt * nt, -1);
  for (size_t k = 0; k + 1 < rows.size(); k++) {
    const int a = rows[k].ta, b = rows[k].tb;
    if (pidx[(size_t)a * nt + b] >= 0) return err(MDN_ERR_ARG, "mdn_adjoint: type pair (%d, %d) is both gas-ion and vapor-ion", a, b);
    pidx[(size_t)a * nt + b] = pidx[(size_t)b * nt + a] = 2 * (int)k;
  }
  /* ---- device buffers ---- */
  const int K = spec->checkpoint_every;
  const long long nseg = (spec->n_steps + K - 1) / K;
  std::vector<void*> owned;
  auto cleanup = [&]() {
    for (void* p : owned) cudaFree(p);
  };
  Sys S;
  memset(&S, 0, sizeof S);
  S.N = N;
  S.n_ion = ni;
  S.nt = nt;
  S.type = dput(type, owned);
  S.q = dput(q, owned);
  S.mass = dput(mass, owned);
  S.c = dput(cc, owned);
  S.vapor = dput(isvap, owned);
  /* pairs grouped by kind and type pair: an atom's row takes them in this
   * order, so that the 32 pairs a warp has at a time are of few parameter rows
   * (vjp_rows adds a row's 32 terms up at once) */
  {
    std::vector<size_t> ord(pi.size());
    for (size_t k = 0; k < ord.size(); k++) ord[k] = k;
    auto key = [&](size_t k) { return ((long long)pk[k] * nt + type[pi[k]]) * nt + type[pj[k]]; };
    std::stable_sort(ord.begin(), ord.end(), [&](size_t a, size_t b) { return key(a) < key(b); });
    std::vector<int> pi2(pi.size()), pj2(pi.size());
    std::vector<unsigned char> pk2(pi.size());
    for (size_t k = 0; k < ord.size(); k++) {
      pi2[k] = pi[ord[k]];
      pj2[k] = pj[ord[k]];
      pk2[k] = pk[ord[k]];
    }
    pi.swap(pi2);
    pj.swap(pj2);
    pk.swap(pk2);
  }
  /* the pairs by atom, from both sides, in the sorted order (so that a
   * warp's lanes stay on few parameter rows).  One side is primary, the ion
   * atom's where there is one, the lower index in an ion-ion pair. */
  {
    std::vector<int> off(N + 1, 0), at, order(N);
    for (size_t k = 0; k < pi.size(); k++) {
      off[pi[k] + 1]++;
      off[pj[k] + 1]++;
    }
    for (int i = 0; i < N; i++) off[i + 1] += off[i];
    at.assign(off.begin(), off.end() - 1);
    std::vector<int2> row(2 * pi.size());
    for (size_t k = 0; k < pi.size(); k++) {
      const int a = pi[k], b = pj[k];
      row[at[a]++] = make_int2(b, pk[k] | (a < b ? kPrimary : 0));
      row[at[b]++] = make_int2(a, pk[k] | (b < a ? kPrimary : 0));
    }
    for (int i = 0; i < N; i++) order[i] = i;
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return off[a + 1] - off[a] > off[b + 1] - off[b]; });
    S.row_off = dput(off, owned);
    S.row = dput(row, owned);
    S.row_order = dput(order, owned);
  }
  /* the bonded terms' rows by atom (terms: bonds, angles, dihedrals) */
  {
    std::vector<std::vector<int>> by(N);
    int t = 0;
    auto add = [&](const std::vector<int>& v, int w) {
      for (size_t r = 0; r < v.size(); r += w, t++)
        for (int k = 0; k < w - 1; k++) by[v[r + k]].push_back(4 * t + k);
    };
    add(bonds, 3);
    add(angles, 4);
    add(dih, 5);
    std::vector<int> off(N + 1, 0), at(4 * (size_t)t, 0);
    for (int i = 0; i < N; i++) {
      off[i + 1] = off[i];
      for (int a : by[i]) at[a] = off[i + 1]++;
    }
    S.tb_off = dput(off, owned);
    S.tb_at = dput(at, owned);
  }
  /* the units */
  {
    std::vector<Unit> units;
    std::vector<char> seen_c(ncons, 0), seen_a(N, 0);
    bool big = false;
    for (int k = 0; k < ncons && !big; k++) {
      if (seen_c[k]) continue;
      std::vector<int> cs(1, k);
      seen_c[k] = 1;
      for (size_t q = 0; q < cs.size(); q++)
        for (int e = nboff[cs[q]]; e < nboff[cs[q] + 1]; e++)
          if (!seen_c[nb[e]]) {
            seen_c[nb[e]] = 1;
            cs.push_back(nb[e]);
          }
      if (cs.size() > 3) {
        big = true;
        break;
      }
      Unit U;
      memset(&U, 0, sizeof U);
      auto place = [&](int atom) {
        for (int a = 0; a < U.na; a++)
          if (U.atom[a] == atom) return a;
        U.atom[U.na] = atom;
        seen_a[atom] = 1;
        return U.na++;
      };
      for (int c : cs) {
        U.cons[U.nc] = c;
        U.ci[U.nc] = place(cons[3 * c]);
        U.cj[U.nc] = place(cons[3 * c + 1]);
        const double dk = d->bond_coeff[2 * cons[3 * c + 2] + 1];
        U.d2[U.nc] = dk * dk;
        U.nc++;
      }
      for (int k = 0; k < U.nc; k++)
        for (int l = 0; l < U.nc; l++) {
          const double mi = 1.0 / mass[U.atom[U.ci[l]]], mj = 1.0 / mass[U.atom[U.cj[l]]];
          U.cf[k][l] = (U.ci[l] == U.ci[k] ? mi : 0.0) - (U.cj[l] == U.ci[k] ? mj : 0.0) -
                       (U.ci[l] == U.cj[k] ? mi : 0.0) + (U.cj[l] == U.cj[k] ? mj : 0.0);
        }
      units.push_back(U);
    }
    Unit U;
    memset(&U, 0, sizeof U);
    for (int i = 0; i < N && !big; i++) {
      if (seen_a[i]) continue;
      U.atom[U.na++] = i;
      if (U.na == 8) {
        units.push_back(U);
        U.na = 0;
      }
    }
    if (U.na > 0) units.push_back(U);
    if (big) units.clear();
    S.n_units = (int)units.size();
    S.units = dput(units, owned);
  }
  S.A = dput(A, owned);
  S.B = dput(Bt, owned);
  for (double& v : E) v = 1.0 / v;
  for (double& v : Sg) v = 1.0 / v;
  S.ieps = dput(E, owned);
  S.isig = dput(Sg, owned);
  S.pidx = dput(pidx, owned);
  S.bmh = dput(bmh, owned);
  S.n_bonds = (int)bonds.size() / 3;
  S.n_angles = (int)angles.size() / 4;
  S.n_dih = (int)dih.size() / 5;
  S.bonds = dput(bonds, owned);
  S.angles = dput(angles, owned);
  S.dih = dput(dih, owned);
  S.bond_c = dput(std::vector<double>(d->bond_coeff, d->bond_coeff + 2 * d->n_bond_types), owned);
  S.angle_c = dput(std::vector<double>(d->angle_coeff, d->angle_coeff + 2 * d->n_angle_types), owned);
  S.dih_c = dput(std::vector<double>(d->dihedral_coeff, d->dihedral_coeff + 15 * d->n_dihedral_types), owned);
  S.dih_multi = dput(std::vector<int>(d->dihedral_multi, d->dihedral_multi + d->n_dihedral_types), owned);
  S.n_cons = ncons;
  S.n_colors = ncolors;
  S.cons = dput(cons, owned);
  S.cons_color = dput(color, owned);
  S.cons_nb_off = dput(nboff, owned);
  S.cons_nb = dput(nb, owned);
  S.n_cons_nb = (int)nb.size();
  S.ri2 = d->r_inter * d->r_inter;
  S.RI2 = (d->r_inter + d->overlap) * (d->r_inter + d->overlap);
  S.rcenter = d->r_inter - d->overlap * 0.5;
  S.overlap = d->overlap;
  double msum = 0;
  for (int i = 0; i < ni; i++) msum += mass[i];
  S.ion_msum = msum;
  S.qqrd2e = 1.602e-19 * 1.602e-19 / 4.0 / M_PI / 8.85e-12 * 6.02e23 * 1e10 / 4184.0; /* src/constants.hpp */
  S.dt = d->dt;
  for (int k = 0; k < 3; k++) S.efield[k] = d->efield[k];
  S.efield_on = (I & MDN_I_EFIELD) != 0;
  S.vcorr = !(quirks & MDN_Q_SHAKE_NO_VCORR);
  S.n_vmol = nvin;
  S.a_v = av;
  S.vmol_first = vap0;
  double vm = 0;
  for (int a = 0; a < av; a++) vm += d->atom_mass[d->vapor.type[a]];
  S.vmol_mass = vm;
  S.R0 = spec->count_radius;
  S.W = spec->count_width;
  S.w_energy = spec->w_energy;
  S.w_count = spec->w_count;
  S.inv_n = 1.0 / (double)spec->n_steps;
  S.n_params = n_params;
  const size_t n3 = 3 * (size_t)N;
  Buf Bf;
  memset(&Bf, 0, sizeof Bf);
  /* every segment's recomputed trajectory (the recomputes run at once) */
  const size_t n_terms = std::max(1, S.n_bonds + S.n_angles + S.n_dih);
  Bf.X = dzero<double>((size_t)nseg * (K + 1) * n3, owned);
  Bf.V = dzero<double>((size_t)nseg * n3, owned);
  Bf.F = dzero<double>((size_t)nseg * n3, owned);
  Bf.gam = dzero<double>((size_t)nseg * K * std::max(ncons, 1), owned);
  Bf.lx = dzero<double>(n3, owned);
  Bf.lv = dzero<double>(n3, owned);
  Bf.lf = dzero<double>(n3, owned);
  Bf.xb = dzero<double>(n3, owned);
  Bf.w = dzero<double>((size_t)nseg * (K + 1) * N, owned);
  Bf.dw = dzero<double>((size_t)nseg * (K + 1) * n3, owned);
  Bf.mg = dzero<double>((size_t)nseg * (K + 1) * 3 * (nvin + 1), owned);
  Bf.tb = dzero<double>((size_t)nseg * 12 * n_terms, owned);
  Bf.part = dzero<double>(3 * ADJ_CLUSTER, owned);
  Bf.mu = dzero<double>(std::max(ncons, 1), owned);
  Bf.grad = dzero<double>(n_params, owned);
  Bf.flag = dzero<int>(2 * (size_t)nseg, owned);
  double* d_jseg = dzero<double>((size_t)nseg * ADJ_CLUSTER, owned);
  /* the forces the state holds at the window start */
  std::vector<double> f0(3 * (size_t)N, 0.0);
  for (int i = 0; i < ni; i++)
    for (int k = 0; k < 3; k++) f0[3 * i + k] = ion_f[3 * i + k];
  for (size_t kq = 0; kq < gin.size(); kq++)
    for (int a = 0; a < ag; a++)
      for (int k = 0; k < 3; k++) f0[3 * (gas0 + kq * ag + a) + k] = gf[3 * ((size_t)gin[kq] * ag + a) + k];
  for (size_t kq = 0; kq < vin.size(); kq++)
    for (int a = 0; a < av; a++)
      for (int k = 0; k < 3; k++) f0[3 * (vap0 + kq * av + a) + k] = vf[3 * ((size_t)vin[kq] * av + a) + k];
  double* d_f0 = dput(f0, owned);
  const int f0_theta = info.step > 0 ? 1 : 0;
  /* checkpoints: x, v of every segment start, gathered on the device */
  double* cpx = dzero<double>((size_t)nseg * n3, owned);
  double* cpv = dzero<double>((size_t)nseg * n3, owned);
  long long* cpo = dzero<long long>(2, owned);
  int* cpt = dzero<int>(N, owned);
  for (void* p : owned)
    if (!p) {
      cleanup();
      return err(MDN_ERR_CUDA, "mdn_adjoint: device allocation failed");
    }
  /* the uploads and clears above were queued on the default stream, which the
   * handle's stream does not wait for */
  if (cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess) {
    cleanup();
    return err(MDN_ERR_CUDA, "mdn_adjoint: %s", cudaGetErrorString(cudaGetLastError()));
  }
  /* ---- forward window on the engine, checkpoint at each segment start ---- */
  cudaStream_t stream = (cudaStream_t)sa.stream;
  float fwd_ms = 0;
  {
    std::vector<double> chk(n3);
    for (long long s = 0; s < nseg; s++) {
      if (mdn_snapshot_device(sa.P, sa.D, sa.iblob, 1, sa.ion_x, sa.ion_v, sa.slab_x, sa.slab_v, sa.vslab_x,
                              sa.vslab_v, cpo, cpt, cpx + s * n3, cpv + s * n3, N, stream)) {
        cleanup();
        return err(MDN_ERR_CUDA, "mdn_adjoint: checkpoint gather failed");
      }
      if (s == 0) {
        /* the gather's row order must be the dense order */
        cudaStreamSynchronize(stream);
        cudaMemcpy(chk.data(), cpx, sizeof(double) * n3, cudaMemcpyDeviceToHost);
        if (memcmp(chk.data(), x0.data(), sizeof(double) * n3) != 0) {
          cleanup();
          return err(MDN_ERR_ARG, "mdn_adjoint: the engine's slab order differs from ascending molecule order");
        }
      }
      const long long n = std::min<long long>(K, spec->n_steps - s * K);
      rc = mdn_step(h, n, 0);
      if (rc) {
        cleanup();
        return rc;
      }
      double step_ms = 0;
      long long nl = 0;
      mdn_last_timing(h, &step_ms, &nl);
      fwd_ms += (float)step_ms;
    }
  }
  /* ---- backward, one segment per launch, last first ---- */
  const size_t cbytes = sizeof(double) * (2 * (size_t)ncons + (size_t)S.n_cons_nb);
  if (cbytes > 200 * 1024) {
    cleanup();
    return err(MDN_ERR_CAPACITY, "mdn_adjoint: %d constraints in the domain, too many for the reverse sweep", ncons);
  }
  /* x and the force adjoint of the reverse sweep in shared memory where they
   * fit beside the constraints' scratch; likewise the recompute's weights */
  const size_t fall = S.n_units == 0 ? cbytes : 0;
  const bool staged = 2 * n3 * sizeof(double) + fall <= 200 * 1024;
  const size_t seg_bytes = (staged ? 2 * n3 * sizeof(double) : 0) + fall;
  const bool sw_smem = N * sizeof(double) <= 200 * 1024;
  const size_t rec_bytes = sw_smem ? N * sizeof(double) : 0;
  auto* const segment = staged ? adjoint_segment<true> : adjoint_segment<false>;
  if (cudaFuncSetAttribute(segment, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess ||
      cudaFuncSetAttribute(adjoint_recompute, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) !=
          cudaSuccess ||
      cudaFuncSetAttribute(segment, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaFuncSetAttribute(adjoint_recompute, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cleanup();
    return err(MDN_ERR_CUDA, "mdn_adjoint: shared memory");
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof cfg);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(ADJ_THREADS);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, stream);
  /* the recompute on clusters as large as let every segment run at once; one
   * CTA each where the constraints go through block barriers or the weights
   * through global memory.  Fewer CTAs if the GPU cannot place that many. */
  int sms = 1, Cr = ADJ_CLUSTER;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, sa.dev);
  while (Cr > 1 && (nseg * Cr > sms || S.n_units == 0 || !sw_smem)) Cr /= 2;
  cudaError_t le = cudaErrorUnknown;
  for (; Cr >= 1; Cr /= 2) {
    cfg.gridDim = dim3((unsigned)(nseg * Cr));
    cfg.dynamicSmemBytes = rec_bytes;
    attr[0].val.clusterDim.x = Cr;
    le = cudaLaunchKernelEx(&cfg, adjoint_recompute, S, Bf, K, (long long)spec->n_steps, (const double*)cpx,
                            (const double*)cpv, (const double*)d_f0, d_jseg, sw_smem ? 1 : 0);
    if (le == cudaSuccess || Cr == 1) break;
    cudaGetLastError();
  }
  for (long long s = nseg - 1; s >= 0 && le == cudaSuccess; s--) {
    const int n = (int)std::min<long long>(K, spec->n_steps - s * K);
    Buf b = Bf;
    b.X += s * (K + 1) * n3;
    b.gam += (size_t)s * K * std::max(ncons, 1);
    b.w += (size_t)s * (K + 1) * N;
    b.dw += (size_t)s * (K + 1) * n3;
    b.mg += (size_t)s * (K + 1) * 3 * (nvin + 1);
    /* one cluster of ADJ_CLUSTER CTAs per segment (fewer if the GPU cannot
     * place that many) */
    for (int C = ADJ_CLUSTER; C >= 1; C /= 2) {
      cfg.gridDim = dim3(C);
      cfg.dynamicSmemBytes = seg_bytes;
      attr[0].val.clusterDim.x = C;
      le = cudaLaunchKernelEx(&cfg, segment, S, b, n, s == 0 ? 1 : 0, f0_theta);
      if (le == cudaSuccess) break;
      cudaGetLastError();
    }
  }
  if (le != cudaSuccess) {
    cudaStreamSynchronize(stream);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cleanup();
    return err(MDN_ERR_CUDA, "mdn_adjoint: launch: %s", cudaGetErrorString(le));
  }
  cudaEventRecord(e1, stream);
  cudaError_t ce = cudaStreamSynchronize(stream);
  float adj_ms = 0;
  cudaEventElapsedTime(&adj_ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (ce != cudaSuccess || (ce = cudaGetLastError()) != cudaSuccess) {
    cleanup();
    return err(MDN_ERR_CUDA, "mdn_adjoint: %s", cudaGetErrorString(ce));
  }
  std::vector<int> fl(2 * (size_t)nseg, 0);
  cudaMemcpy(fl.data(), Bf.flag, sizeof(int) * fl.size(), cudaMemcpyDeviceToHost);
  int flags[2] = {0, 0};
  for (long long s = 0; s < nseg; s++) flags[1] |= fl[2 * s + 1];
  /* J: the segments' objective sums, last first (the order the sequential
   * form added them in) */
  std::vector<double> js((size_t)nseg * Cr, 0.0);
  cudaMemcpy(js.data(), d_jseg, sizeof(double) * js.size(), cudaMemcpyDeviceToHost);
  double jsum = 0.0;
  for (long long s = (long long)js.size() - 1; s >= 0; s--) jsum += js[s] * S.inv_n;
  *J = jsum;
  cudaMemcpy(grad, Bf.grad, sizeof(double) * n_params, cudaMemcpyDeviceToHost);
  if (ms) {
    ms[0] = fwd_ms;
    ms[1] = adj_ms;
  }
  cleanup();
  if (flags[1] & MDN_ST_SHAKE_NOCONV) return err(MDN_ERR_REPLICA, "mdn_adjoint: SHAKE did not converge in the recomputation");
  return MDN_OK;
}
