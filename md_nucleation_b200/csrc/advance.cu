/*
 * advance.cu -- the persistent step kernel of the engine (sm_100a).
 *
 * One launch advances a batch of replicas by n steps.  Thread-block clusters
 * of C CTAs (C = the launch's cluster size, 1..8) pull replicas from a work
 * queue, largest first, and keep a replica on-chip for all n steps:
 *
 *   - the "core" -- the ion (seed) and the in-domain vapor molecules, at most
 *     a few hundred to ~1000 atoms -- lives in shared memory, replicated in
 *     every CTA of the cluster.  All CTAs integrate it identically; its forces
 *     are int64 fixed-point partial sums that the cluster adds over DSMEM, so
 *     every copy receives the same total and the copies never diverge;
 *   - the in-domain gas molecules (up to ~20,000 atoms) live in the gas slab in
 *     global memory (L2-resident while the replica is being stepped) and are
 *     split evenly over the cluster's CTAs;
 *   - gas-gas interactions are absent from the reference's configurations, so
 *     a gas molecule interacts only with the core: molecules whose gas-ion /
 *     gas-vapor lists are empty ("far") are advanced by one thread each, where
 *     they are many through all steps to the next rebuild at once; "near" ones are
 *     sorted by their number of partners and taken 32 to a warp (build_near,
 *     near_group), with shared-memory fixed-point atomics for the reaction on
 *     the core.
 *
 * Each step follows MD::verlet (src/verlet.cpp:20-39) exactly:
 *   kick (MD::velocity_calculation), [MD::velocity_scaling], drift with
 *   optional SHAKE (MD::update_position / updatePositionSHAKE), ion centre and
 *   taper weights, [MD::nosehoover_zeta], MD::check_pairlist -> make_pair on
 *   the device, forces of every enabled Potential, kick, [MD::nosehoover_ion].
 * The rebuild (MD::make_pair, src/pairList/pairlist.cpp:16-49) -- free flight,
 * updateInCenters, in/out classification with periodic wrap and
 * Maxwell-Boltzmann resampling, insertion with a random rotation, pair lists,
 * loop_update -- runs inside the same launch, decided per replica.
 *
 * Precision: FP64 for integration, SHAKE, centres, weights, the rebuild and
 * the bonded terms; FP32 for the pair terms (LJ, Coulomb, Born-Mayer-Huggins)
 * on coordinates taken relative to the ion centre; every sum with more than one
 * writer is an int64 fixed-point sum (units 2^-40 kcal/mol/A for forces,
 * 2^-36 kcal/mol for energies), so results do not depend on the launch shape.
 */
#include <cooperative_groups.h>

#include <type_traits>

#include "device_util.cuh"
#include "mdn_types.h"

namespace cg = cooperative_groups;
using namespace mdn;

namespace {

/* MDN_GG_TERMS selects the gas-gas term: compiled into its own kernels
 * (advance_gg.cu, advance_gg_fp64.cu), absent from the others */
#ifdef MDN_GG_TERMS
constexpr bool kGG = true;
#else
constexpr bool kGG = false;
#endif

/* taper weight, and the atom's kind in one word: type (bits 0-6), the
 * Born-Mayer-Huggins row of an ion atom (bit 7), vapor slot + 1 (bits 8-31, 0
 * for ion atoms), so that a pair reads both with one 8-byte access */
struct AtomTag {
  float w;
  unsigned k;
};
__device__ __forceinline__ int tag_type(unsigned k) { return (int)(k & 127u); }
__device__ __forceinline__ int tag_bmh(unsigned k) { return (int)((k >> 7) & 1u); }
__device__ __forceinline__ int tag_slot(unsigned k) { return (int)(k >> 8) - 1; }

/* pointers into the dynamic shared memory of a CTA */
struct Core {
  double* x;        /* [3*nc] positions                        */
  double* v;        /* [3*nc] velocities                       */
  double* f;        /* [3*nc] force of the last evaluation; from the drift to the
                     * next evaluation, the positions before the drift (the SHAKE
                     * reference vectors) */
  long long* acc;   /* [3*nc] this CTA's fixed-point force sums */
  unsigned* chunk;  /* [9*nc] the same sums in 32-bit chunks (acc_add) */
  float4* pos;      /* [nc] (x - ion centre, charge), FP32     */
  AtomTag* tag;     /* [nc] taper weight and kind              */
  unsigned* excl;   /* AMBER exclusions, n_ion rows            */
  float2* lj;       /* [nt*nt] 48 eps s^12, 24 eps s^6         */
  double* c2;       /* [nt] 0.5*dt*4.184e-4 / mass             */
  double* mass;     /* [nt]                                    */
};

struct Ctx {
  const KArgs* a;
  RepParams* P;
  RepDyn* D;
  Core c;
  int r;            /* replica                          */
  int rank, C;      /* cluster rank and size            */
  int n_core;       /* atoms in the core                */
  bool settled;     /* every CTA of the cluster has read this one's sums (settle) */
  int* iscr;        /* >= 64 ints of scratch            */
  int* cand;        /* [MDN_INSERT_MAX_VAPOR + 1] entering vapor molecules, count last */
  double* trial;    /* [3*MDN_MAX_VAP_ATOMS] trial atoms */
  double* dscr;     /* >= 64 doubles of scratch         */
  const int* ib;    /* int blob of the replica          */
  const double* db; /* double blob of the replica       */
};

__device__ __forceinline__ size_t gatom(const RepParams* P, int parity, int s, int a) {
  return (size_t)P->slab_off + ((size_t)parity * P->slab_cap + s) * P->a_g + a;
}
__device__ __forceinline__ size_t gmol(const RepParams* P, int parity, int s) {
  return (size_t)P->slab_moff + (size_t)parity * P->slab_cap + s;
}
__device__ __forceinline__ size_t vatom(const RepParams* P, int parity, int s, int a) {
  return (size_t)P->vslab_off + ((size_t)parity * P->vcap + s) * P->a_v + a;
}
__device__ __forceinline__ size_t vmol(const RepParams* P, int parity, int s) {
  return (size_t)P->vslab_moff + (size_t)parity * P->vcap + s;
}

/* per-phase SM cycles of the current job (thread 0 times phases that end in a
 * block barrier); flushed to KArgs::prof at the end of the job */
__shared__ long long s_prof[MDN_PROF_N];
__shared__ long long s_prof_t0;
__device__ __forceinline__ void prof_start(const Ctx& x) {
  if (x.a->prof && threadIdx.x == 0) s_prof_t0 = clock64();
}
__device__ __forceinline__ void prof_end(const Ctx& x, int phase) {
  if (x.a->prof && threadIdx.x == 0) s_prof[phase] += clock64() - s_prof_t0;
}

__device__ __forceinline__ void set_status(const Ctx& x, int bit) {
  atomicOr(&x.a->status[x.r], bit);
}

/* ------------------------------------------------------------------------- */
/* core load / store                                                          */
/* ------------------------------------------------------------------------- */
__device__ __forceinline__ void load_ion(Ctx& x) {
  const RepParams* P = x.P;
  const KArgs* a = x.a;
  const int ni = P->n_ion;
  for (int i = threadIdx.x; i < ni; i += blockDim.x) {
    size_t g = (size_t)P->ion_off + i;
    for (int k = 0; k < 3; k++) {
      x.c.x[3 * i + k] = a->ion_x[3 * g + k];
      x.c.v[3 * i + k] = a->ion_v[3 * g + k];
      x.c.f[3 * i + k] = a->ion_f[3 * g + k];
    }
    x.c.pos[i].w = (float)x.db[P->d_ion_q + i];
    x.c.tag[i].w = 1.0f;
    x.c.tag[i].k = (unsigned)x.ib[P->o_ion_type + i] | (x.ib[P->o_ion_bmh + i] ? 128u : 0u);
  }
}

/* the vapor part of the core, from the vapor slab of the current parity */
__device__ __forceinline__ void load_vapor(Ctx& x) {
  const RepParams* P = x.P;
  const KArgs* a = x.a;
  const int ni = P->n_ion, av = P->a_v, nv = x.D->n_vap_in, par = x.D->parity;
  x.n_core = ni + nv * av;
  for (int t = threadIdx.x; t < nv * av; t += blockDim.x) {
    int s = t / av, at = t - s * av;
    size_t g = vatom(P, par, s, at);
    int i = ni + t;
    for (int k = 0; k < 3; k++) {
      x.c.x[3 * i + k] = a->vslab_x[3 * g + k];
      x.c.v[3 * i + k] = a->vslab_v[3 * g + k];
      x.c.f[3 * i + k] = a->vslab_f[3 * g + k];
    }
    x.c.pos[i].w = (float)x.db[P->d_vap_q + at];
    x.c.tag[i].w = a->vslab_w[g];
    x.c.tag[i].k = (unsigned)x.ib[P->o_vap_type + at] | ((unsigned)(s + 1) << 8);
  }
  /* core_tile reads whole blocks of 32 and multiplies what it does not count
   * by 0: the places past the core hold finite positions, not what an earlier
   * replica of this CTA left there */
  for (int i = x.n_core + threadIdx.x; i < ((x.n_core + 31) & ~31); i += blockDim.x) {
    x.c.tag[i].k = 0;
    x.c.pos[i] = make_float4(0, 0, 0, 0);
  }
}

__device__ __forceinline__ void store_core(Ctx& x) {
  const RepParams* P = x.P;
  const KArgs* a = x.a;
  if (x.rank != 0) return;
  const int ni = P->n_ion, av = P->a_v, nv = x.D->n_vap_in, par = x.D->parity;
  for (int i = threadIdx.x; i < ni; i += blockDim.x) {
    size_t g = (size_t)P->ion_off + i;
    for (int k = 0; k < 3; k++) {
      a->ion_x[3 * g + k] = x.c.x[3 * i + k];
      a->ion_v[3 * g + k] = x.c.v[3 * i + k];
      a->ion_f[3 * g + k] = x.c.f[3 * i + k];
    }
  }
  for (int t = threadIdx.x; t < nv * av; t += blockDim.x) {
    int s = t / av, at = t - s * av;
    size_t g = vatom(P, par, s, at);
    int i = ni + t;
    for (int k = 0; k < 3; k++) {
      a->vslab_x[3 * g + k] = x.c.x[3 * i + k];
      a->vslab_v[3 * g + k] = x.c.v[3 * i + k];
      a->vslab_f[3 * g + k] = x.c.f[3 * i + k];
    }
    a->vslab_w[g] = x.c.tag[i].w;
  }
}

/* ------------------------------------------------------------------------- */
/* integration of the core                                                    */
/* ------------------------------------------------------------------------- */
/* First kick (unless it was made) and drift of the core, each thread its own
 * components (thread t: t, t + blockDim.x, ... of the 3 n_core), those whose
 * force it summed and whose second kick it made (core_reduce_kick): no
 * barrier in between.  The positions before the drift stay in c.f for the
 * constraints. */
__device__ __forceinline__ double core_c2(const Ctx& x, int q) { return x.c.c2[tag_type(x.c.tag[q / 3].k)]; }

__device__ __forceinline__ void core_drift(Ctx& x, bool kick) {
  const double dt = x.P->dt;
  const int n3 = 3 * x.n_core;
  for (int q = threadIdx.x; q < n3; q += blockDim.x) {
    double v = x.c.v[q];
    if (kick) {
      v += x.c.f[q] * core_c2(x, q);
      x.c.v[q] = v;
    }
    const double xo = x.c.x[q];
    x.c.f[q] = xo;
    x.c.x[q] = xo + v * dt;
  }
}

/* Observer::computeProps, ion part: Tion.  Warp 0, lane-strided sums then a
 * butterfly, so the result depends on the atom order only. */
__device__ __forceinline__ double ion_temperature(Ctx& x) {
  const RepParams* P = x.P;
  if (threadIdx.x < 32) {
    double K = 0;
    for (int i = threadIdx.x; i < P->n_ion; i += 32) {
      double m = x.c.mass[tag_type(x.c.tag[i].k)];
      K += x.c.v[3 * i] * x.c.v[3 * i] * m;
      K += x.c.v[3 * i + 1] * x.c.v[3 * i + 1] * m;
      K += x.c.v[3 * i + 2] * x.c.v[3 * i + 2] * m;
    }
    K = warp_sum_d(K);
    if (threadIdx.x == 0) {
      K *= 0.5 * P->real_to_kcalmol;
      x.dscr[40] = K / double(P->n_ion) * ((1.0 / P->kb_real) / 1.5);
    }
  }
  __syncthreads();
  double T = x.dscr[40];
  __syncthreads();
  return T;
}

/* one SHAKE correction with the constraint's table row c = (d^2, 1/m_i,
 * 1/m_j): the multiplier of shake_pair with one division */
__device__ __forceinline__ void shake_pair_c(double* Xi, double* Xj, const double* Ri, const double* Rj,
                                             const double* c) {
  double r0 = Ri[0] - Rj[0], r1 = Ri[1] - Rj[1], r2 = Ri[2] - Rj[2];
  double s0 = Xi[0] - Xj[0], s1 = Xi[1] - Xj[1], s2 = Xi[2] - Xj[2];
  double ss = s0 * s0 + s1 * s1 + s2 * s2;
  double dot = r0 * s0 + r1 * s1 + r2 * s2;
  if (dot < 1e-10) dot = 1e-10;
  double g = (c[0] - ss) / (2 * (c[1] + c[2]) * dot);
  double gi = g * c[1], gj = g * c[2];
  Xi[0] += r0 * gi; Xi[1] += r1 * gi; Xi[2] += r2 * gi;
  Xj[0] -= r0 * gj; Xj[1] -= r1 * gj; Xj[2] -= r2 * gj;
}

/* (|s|^2 - d^2)^2 of one constraint; the sweeps stop when every residual is
 * <= 1e-20 A^4 (src/shake.cpp:51-90), and a NaN residual counts as not
 * converged, so a sweep that diverged runs into the cap and is reported */
__device__ __forceinline__ double shake_res_c(const double* Xi, const double* Xj, const double* c) {
  double s0 = Xi[0] - Xj[0], s1 = Xi[1] - Xj[1], s2 = Xi[2] - Xj[2];
  double dr = s0 * s0 + s1 * s1 + s2 * s2 - c[0];
  return dr * dr;
}

/* Newton's method on one group of at most three constraints that share
 * atoms (M-SHAKE).  The positions move along the constraints' reference
 * bond vectors r_k exactly as in the sweeps (x_i += l_k r_k / m_i,
 * x_j -= l_k r_k / m_j), and the l_k solve |s_k|^2 = d_k^2 for the whole
 * group at once, so the result is the sweeps' fixed point; the equations
 * are quadratic in l, and a handful of steps reach it where the sweeps of a
 * rigid water take dozens.  For one constraint a step is the sweep's own
 * update.  ga, gc: the group's atoms (i, j) and coefficients (d^2, 1/m_i,
 * 1/m_j), constraint by constraint.  Returns true once every (|s_k|^2 -
 * d_k^2)^2 <= 1e-20 A^4, the sweeps' criterion; false after 50 steps or a
 * singular system, and the caller sweeps from there. */
template <int N>
__device__ __forceinline__ bool shake_group_n(double* X, const double* R, const int* ga, const double* gc) {
  int I[N], J[N];
  double r[N][3], d2[N], ci[N], cj[N], w[N][N];
#pragma unroll
  for (int k = 0; k < N; k++) {
    I[k] = ga[2 * k];
    J[k] = ga[2 * k + 1];
    d2[k] = gc[3 * k];
    ci[k] = gc[3 * k + 1];
    cj[k] = gc[3 * k + 2];
#pragma unroll
    for (int q = 0; q < 3; q++) r[k][q] = R[3 * I[k] + q] - R[3 * J[k] + q];
  }
  /* d s_k / d l_l = w_kl r_l */
#pragma unroll
  for (int k = 0; k < N; k++)
#pragma unroll
    for (int l = 0; l < N; l++) {
      const double ai = I[k] == I[l] ? ci[l] : (I[k] == J[l] ? -cj[l] : 0.0);
      const double aj = J[k] == I[l] ? ci[l] : (J[k] == J[l] ? -cj[l] : 0.0);
      w[k][l] = ai - aj;
    }
  for (int it = 0; it < 50; it++) {
    double s[N][3], f[N];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < N; k++) {
#pragma unroll
      for (int q = 0; q < 3; q++) s[k][q] = X[3 * I[k] + q] - X[3 * J[k] + q];
      f[k] = s[k][0] * s[k][0] + s[k][1] * s[k][1] + s[k][2] * s[k][2] - d2[k];
      if (!(f[k] * f[k] <= 1e-20)) ok = false;
    }
    if (ok) return true;
    double A[N][N];
#pragma unroll
    for (int k = 0; k < N; k++)
#pragma unroll
      for (int l = 0; l < N; l++)
        A[k][l] = 2.0 * (s[k][0] * r[l][0] + s[k][1] * r[l][1] + s[k][2] * r[l][2]) * w[k][l];
    /* A d = -f by Cramer's rule; for one and two constraints what the rule
     * for three gives with identity rows, without its products by 0 and 1 */
    double Dl[N];
    if constexpr (N == 1) {
      if (!(fabs(A[0][0]) > 1e-300)) return false;
      Dl[0] = -f[0] * (1.0 / A[0][0]);
    } else if constexpr (N == 2) {
      const double det = A[0][0] * A[1][1] - A[0][1] * A[1][0];
      if (!(fabs(det) > 1e-300)) return false;
      const double inv = 1.0 / det;
      const double b0 = -f[0], b1 = -f[1];
      Dl[0] = (b0 * A[1][1] - A[0][1] * b1) * inv;
      Dl[1] = (A[0][0] * b1 - b0 * A[1][0]) * inv;
    } else {
      const double c00 = A[1][1] * A[2][2] - A[1][2] * A[2][1];
      const double c01 = A[1][0] * A[2][2] - A[1][2] * A[2][0];
      const double c02 = A[1][0] * A[2][1] - A[1][1] * A[2][0];
      const double det = A[0][0] * c00 - A[0][1] * c01 + A[0][2] * c02;
      if (!(fabs(det) > 1e-300)) return false;
      const double inv = 1.0 / det;
      const double b0 = -f[0], b1 = -f[1], b2 = -f[2];
      Dl[0] = (b0 * c00 - A[0][1] * (b1 * A[2][2] - A[1][2] * b2) + A[0][2] * (b1 * A[2][1] - A[1][1] * b2)) * inv;
      Dl[1] = (A[0][0] * (b1 * A[2][2] - A[1][2] * b2) - b0 * c01 + A[0][2] * (A[1][0] * b2 - b1 * A[2][0])) * inv;
      Dl[2] = (A[0][0] * (A[1][1] * b2 - b1 * A[2][1]) - A[0][1] * (A[1][0] * b2 - b1 * A[2][0]) + b0 * c02) * inv;
    }
#pragma unroll
    for (int l = 0; l < N; l++)
#pragma unroll
      for (int q = 0; q < 3; q++) {
        X[3 * I[l] + q] += Dl[l] * ci[l] * r[l][q];
        X[3 * J[l] + q] -= Dl[l] * cj[l] * r[l][q];
      }
  }
  return false;
}

__device__ __forceinline__ bool shake_group(double* X, const double* R, const int* ga, const double* gc, int n) {
  if (n == 1) return shake_group_n<1>(X, R, ga, gc);
  if (n == 2) return shake_group_n<2>(X, R, ga, gc);
  return shake_group_n<3>(X, R, ga, gc);
}

__device__ __forceinline__ bool gas_rigid(const RepParams* P) {
  return (P->interactions & MDN_I_SHAKE) && P->n_gas_rigid > 0 && P->a_g == 2;
}

/* Which gas molecules a step integrates beside the core's constraints:
 * all of this CTA's, first kick and drift only, on the steps that rebuild the
 * domain (the lists follow the drift) or need the gas-gas forces (every
 * position first); on others the far ones, complete with their own bond and
 * second kick, unless gas_far_steps has already made their steps, and the
 * near ones, unless they are drifted where their forces are taken
 * (near_group).  That saves a pass over their slab rows, but it lengthens the
 * force items, while here the warps are idle: so it is done for more near
 * molecules than threads (dense domains: 4.96 -> 4.69 ms per 50 steps; the
 * 150-atom chain in thin gas would go from 1.89 to 1.93 ms per 100 steps),
 * and not for a rigid gas, whose constraint is longer still. */
struct GasWork {
  bool all, far, near;
};

__device__ __forceinline__ void gas_integrate(Ctx& x, GasWork w, bool eflag, int tid, int nthr);

/* which of the core's molecules have constraints */
struct CoreCons {
  bool ion;  /* the ion's constraints are on */
  int nv;    /* vapor molecules whose constraints are on */
};
__device__ __forceinline__ CoreCons core_cons(const Ctx& x) {
  const RepParams* P = x.P;
  const bool sh = (P->interactions & MDN_I_SHAKE) != 0;
  return CoreCons{sh && P->n_ion_rigid > 0, sh && P->n_vap_rigid > 0 ? x.D->n_vap_in : 0};
}

/* The sweeps in colour order (a colour's constraints share no atom, so the
 * lanes may take them in any order) until every constraint holds after a
 * sweep: for the ion by warp 0, for a vapor molecule by one thread.  Taken
 * when a molecule has no groups (more than three constraints share atoms)
 * or Newton's method gave one up; marked vapor molecules have a nonzero word
 * at their first chunk sum, which is cleared. */
__device__ __forceinline__ void core_sweeps(Ctx& x, const CoreCons& cc, bool ion, bool vapor) {
  const RepParams* P = x.P;
  const double* const xold = x.c.f;
  const int lane = threadIdx.x & 31;
  if (ion && threadIdx.x < 32) {
    const int* rig = x.ib + P->o_ion_rigid;
    const int* col = x.ib + P->o_ion_color;
    int sweeps = 0;
    for (;;) {
      for (int c = 0; c < P->n_ion_colors; c++) {
        for (int k = lane; k < P->n_ion_rigid; k += 32) {
          if (col[k] != c) continue;
          int i = rig[3 * k], j = rig[3 * k + 1];
          shake_pair_c(x.c.x + 3 * i, x.c.x + 3 * j, xold + 3 * i, xold + 3 * j, x.db + P->d_ion_cons + 3 * k);
        }
        __syncwarp();
      }
      bool ok = true;
      for (int k = lane; k < P->n_ion_rigid; k += 32)
        if (!(shake_res_c(x.c.x + 3 * rig[3 * k], x.c.x + 3 * rig[3 * k + 1], x.db + P->d_ion_cons + 3 * k) <= 1e-20))
          ok = false;
      if (__all_sync(0xffffffffu, ok)) break;
      if (++sweeps >= MDN_SHAKE_MAX_SWEEPS) {
        if (lane == 0 && x.rank == 0) set_status(x, MDN_ST_SHAKE_NOCONV);
        break;
      }
    }
  }
  if (vapor) {
    const int av = P->a_v, nr = P->n_vap_rigid, nco = P->n_vap_colors;
    const int* rig = x.ib + P->o_vap_rigid;
    const int* col = x.ib + P->o_vap_color;
    const double* ct = x.db + P->d_vap_cons;
    for (int s = threadIdx.x; s < cc.nv; s += blockDim.x) {
      const int base = P->n_ion + s * av;
      if (P->n_vap_groups > 0 && x.c.chunk[9 * base] == 0) continue;
      x.c.chunk[9 * base] = 0;
      double* X = x.c.x + 3 * base;
      const double* R = xold + 3 * base;
      bool conv = false;
      for (int sweep = 0; sweep < MDN_SHAKE_MAX_SWEEPS && !conv; sweep++) {
        for (int c = 0; c < nco; c++)
          for (int k = 0; k < nr; k++) {
            if (col[k] != c) continue;
            const int i = rig[3 * k], j = rig[3 * k + 1];
            shake_pair_c(X + 3 * i, X + 3 * j, R + 3 * i, R + 3 * j, ct + 3 * k);
          }
        conv = true;
        for (int k = 0; k < nr; k++)
          if (!(shake_res_c(X + 3 * rig[3 * k], X + 3 * rig[3 * k + 1], ct + 3 * k) <= 1e-20)) conv = false;
      }
      if (!conv && x.rank == 0) set_status(x, MDN_ST_SHAKE_NOCONV);
    }
  }
  __syncthreads();
}

/* The core's constraints, one group (constraints that share atoms) per
 * thread, in units of a warp whose groups have the same number of
 * constraints: the ion's groups of three, two and one (an atom and its
 * hydrogens), then the same group of every vapor molecule.  The step's gas
 * integration runs beside them (the gas pass touches only the gas slab), on
 * the warps that have no unit.  (One thread per vapor molecule, and the
 * ion's groups on one warp, made the serial solution of several groups the
 * longest chain of the step; groups of different sizes in one warp would be
 * solved one size after another.)  The velocities take the constraints'
 * displacement in core_place. */
__device__ __forceinline__ void core_shake(Ctx& x, const CoreCons& cc, GasWork gas, bool eflag) {
  const RepParams* P = x.P;
  const double* const xold = x.c.f;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int n3 = cc.ion ? P->ion_groups_n[2] : 0, n2 = cc.ion ? P->ion_groups_n[1] : 0,
            n1 = cc.ion ? P->ion_groups_n[0] : 0;
  const int u3 = (n3 + 31) >> 5, u2 = u3 + ((n2 + 31) >> 5), u1 = u2 + ((n1 + 31) >> 5);
  const int per = (cc.nv + 31) >> 5, units = u1 + P->n_vap_groups * per;
  const bool any_gas = gas.all || gas.far || gas.near;
  const int w_sh = min(units, any_gas ? max(1, (3 * nwarps) >> 2) : nwarps);
  if (warp < w_sh)
    for (int u = warp; u < units; u += w_sh) {
      if (u < u1) {
        /* the ion's groups are stored by size, largest first */
        const int in = u < u3 ? 32 * u + lane : u < u2 ? 32 * (u - u3) + lane : 32 * (u - u2) + lane;
        const int n = u < u3 ? 3 : u < u2 ? 2 : 1;
        const int g = in + (n < 3 ? n3 : 0) + (n < 2 ? n2 : 0);
        if (in < (n == 3 ? n3 : n == 2 ? n2 : n1) &&
            !shake_group(x.c.x, xold, x.ib + P->o_ion_gatoms + 6 * g, x.db + P->d_ion_gcons + 9 * g, n))
          atomicOr(&x.iscr[62], 1);
      } else {
        const int g = (u - u1) / per, m = 32 * (u - u1 - g * per) + lane, base = P->n_ion + m * P->a_v;
        if (m < cc.nv && !shake_group(x.c.x + 3 * base, xold + 3 * base, x.ib + P->o_vap_gatoms + 6 * g,
                                      x.db + P->d_vap_gcons + 9 * g, x.ib[P->o_vap_gsize + g])) {
          x.c.chunk[9 * base] = 1;
          atomicOr(&x.iscr[62], 2);
        }
      }
    }
  const int w_gas0 = min(w_sh, nwarps - 1);
  if (any_gas && warp >= w_gas0)
    gas_integrate(x, gas, eflag, threadIdx.x - 32 * w_gas0, blockDim.x - 32 * w_gas0);
  __syncthreads();
  const int fail = x.iscr[62];
  const bool ion = cc.ion && (u1 == 0 || (fail & 1)), vapor = cc.nv > 0 && (P->n_vap_groups == 0 || (fail & 2));
  if (ion || vapor) core_sweeps(x, cc, ion, vapor);
}

/* Centre of the ion atoms' `src` (positions or velocities): every warp for
 * itself, lane-strided partial sums then a butterfly, so the result depends
 * on the atom order only, and no warp waits for another's */
__device__ __forceinline__ void ion_centre(const Ctx& x, const double* src, double* com) {
  const RepParams* P = x.P;
  double s[3] = {0, 0, 0};
  for (int i = threadIdx.x & 31; i < P->n_ion; i += 32) {
    const double m = x.c.mass[tag_type(x.c.tag[i].k)];
#pragma unroll
    for (int k = 0; k < 3; k++) s[k] += src[3 * i + k] * m;
  }
  const double mInv = 1 / P->ion_msum;
#pragma unroll
  for (int k = 0; k < 3; k++) com[k] = warp_sum_d(s[k]) * mInv;
}

/* the ion centre in the reference's own order (sequential sum), used where a
 * threshold decision depends on it (the in/out classification) */
__device__ __forceinline__ void ion_centre_exact(Ctx& x) {
  const RepParams* P = x.P;
  if (threadIdx.x < 6) { /* one component each */
    const double* const src = threadIdx.x < 3 ? x.c.x + threadIdx.x : x.c.v + threadIdx.x - 3;
    double s = 0;
    for (int i = 0; i < P->n_ion; i++) s += src[3 * i] * x.c.mass[tag_type(x.c.tag[i].k)];
    const double mInv = 1 / P->ion_msum;
    x.D->ion_com[threadIdx.x] = s * mInv;
  }
  __syncthreads();
}

__device__ __forceinline__ double taper(const RepParams* P, const double* com, const double* xa) {
  double dx = xa[0] - com[0];
  double dy = xa[1] - com[1];
  double dz = xa[2] - com[2];
  double r2 = dx * dx + dy * dy + dz * dz;
  if (r2 < P->ri2) return 1;
  if (r2 > P->RI2) return 0;
  double dr = (sqrt(r2) - P->rcenter);
  double C = cos(3.141592653589793 / P->overlap * 0.5 * dr);
  return C * C;
}

/* The core's place relative to the ion centre `com`: the FP32 coordinates,
 * the vapor atoms' taper weights (when `weights`) and, with `cc`, what the
 * constraints' displacement adds to the velocities.  A molecule inserted by
 * the rebuild of this step carries w < 0 and gets 0 for this step:
 * MD::update_position ran before the rebuild, while the molecule was still
 * outside (src/verlet.cpp:109-134), so the reference leaves its weights
 * unset. */
__device__ __forceinline__ void core_place(Ctx& x, const double* com, bool weights, const CoreCons& cc) {
  const RepParams* P = x.P;
  const double dt = P->dt;
  if (threadIdx.x == 0) x.iscr[60] = blockDim.x >> 5; /* the force queue: every warp's first item is taken */
  for (int i = threadIdx.x; i < x.n_core; i += blockDim.x) {
    double* const X = x.c.x + 3 * i;
    if (i >= P->n_ion) {
      if (x.c.tag[i].w < 0.0f) x.c.tag[i].w = 0.0f;
      else if (weights) x.c.tag[i].w = (float)taper(P, com, X);
    }
    if (i < P->n_ion ? cc.ion : cc.nv > 0)
#pragma unroll
      for (int k = 0; k < 3; k++) {
        /* displacement by the constraints = x - (xold + v*dt) */
        const double v = x.c.v[3 * i + k], xd = x.c.f[3 * i + k] + v * dt;
        x.c.v[3 * i + k] = v + (X[k] - xd) / dt;
      }
    x.c.pos[i] = make_float4((float)(X[0] - com[0]), (float)(X[1] - com[1]), (float)(X[2] - com[2]), x.c.pos[i].w);
  }
  __syncthreads();
}

/* ------------------------------------------------------------------------- */
/* bonded terms (FP64, the reference's expressions)                           */
/* ------------------------------------------------------------------------- */
struct BondOut {
  double f[4][3];
  double e;
};

__device__ __forceinline__ void bond_fd(const double* X, const double* co, int i, int j, BondOut& o) {
  double dx = X[3 * i] - X[3 * j];
  double dy = X[3 * i + 1] - X[3 * j + 1];
  double dz = X[3 * i + 2] - X[3 * j + 2];
  double rsq = (dx * dx + dy * dy + dz * dz);
  double r = sqrt(rsq);
  double dr = (r - co[1]);
  double rk = co[0] * dr;
  double fb = -2.0 * rk / r;
  o.f[0][0] = fb * dx; o.f[0][1] = fb * dy; o.f[0][2] = fb * dz;
  o.f[1][0] = -(fb * dx); o.f[1][1] = -(fb * dy); o.f[1][2] = -(fb * dz);
  o.e = rk * dr;
}

__device__ __forceinline__ void angle_fd(const double* X, const double* co, int i, int j, int k, BondOut& o) {
  double dx1 = X[3 * i] - X[3 * j];
  double dy1 = X[3 * i + 1] - X[3 * j + 1];
  double dz1 = X[3 * i + 2] - X[3 * j + 2];
  double rsq1 = (dx1 * dx1 + dy1 * dy1 + dz1 * dz1);
  double r1 = sqrt(rsq1);
  double dx2 = X[3 * k] - X[3 * j];
  double dy2 = X[3 * k + 1] - X[3 * j + 1];
  double dz2 = X[3 * k + 2] - X[3 * j + 2];
  double rsq2 = (dx2 * dx2 + dy2 * dy2 + dz2 * dz2);
  double r2 = sqrt(rsq2);
  double C = dx1 * dx2 + dy1 * dy2 + dz1 * dz2;
  C /= r1 * r2;
  double Cs = 1 / (sqrt(1.0 - C * C));
  double dtheta = acos(C) - co[1];
  double tk = co[0] * dtheta;
  double a = -2.0 * tk * Cs;
  double a11 = a * C / rsq1;
  double a12 = -a / (r1 * r2);
  double a22 = a * C / rsq2;
  double f1[3] = {a11 * dx1 + a12 * dx2, a11 * dy1 + a12 * dy2, a11 * dz1 + a12 * dz2};
  double f3[3] = {a22 * dx2 + a12 * dx1, a22 * dy2 + a12 * dy1, a22 * dz2 + a12 * dz1};
  for (int q = 0; q < 3; q++) {
    o.f[0][q] = f1[q];
    o.f[1][q] = -(f1[q] + f3[q]);
    o.f[2][q] = f3[q];
  }
  o.e = tk * dtheta;
}

__device__ __forceinline__ void dihedral_fd(const double* X, const double* co, int multi, int i, int j, int k,
                                            int l, BondOut& o) {
  double vb1x = X[3 * i] - X[3 * j];
  double vb1y = X[3 * i + 1] - X[3 * j + 1];
  double vb1z = X[3 * i + 2] - X[3 * j + 2];
  double vb2x = X[3 * k] - X[3 * j];
  double vb2y = X[3 * k + 1] - X[3 * j + 1];
  double vb2z = X[3 * k + 2] - X[3 * j + 2];
  double vb2xm = -vb2x, vb2ym = -vb2y, vb2zm = -vb2z;
  double vb3x = X[3 * l] - X[3 * k];
  double vb3y = X[3 * l + 1] - X[3 * k + 1];
  double vb3z = X[3 * l + 2] - X[3 * k + 2];
  double ax = vb1y * vb2zm - vb1z * vb2ym;
  double ay = vb1z * vb2xm - vb1x * vb2zm;
  double az = vb1x * vb2ym - vb1y * vb2xm;
  double bx = vb3y * vb2zm - vb3z * vb2ym;
  double by = vb3z * vb2xm - vb3x * vb2zm;
  double bz = vb3x * vb2ym - vb3y * vb2xm;
  double rasq = ax * ax + ay * ay + az * az;
  double rbsq = bx * bx + by * by + bz * bz;
  double rgsq = vb2xm * vb2xm + vb2ym * vb2ym + vb2zm * vb2zm;
  double rg = sqrt(rgsq);
  double rginv = 0.0, ra2inv = 0.0, rb2inv = 0.0;
  if (rg > 0) rginv = 1.0 / rg;
  if (rasq > 0) ra2inv = 1.0 / rasq;
  if (rbsq > 0) rb2inv = 1.0 / rbsq;
  double rabinv = sqrt(ra2inv * rb2inv);
  double c = (ax * bx + ay * by + az * bz) * rabinv;
  double s = rg * rabinv * (ax * vb3x + ay * vb3y + az * vb3z);
  double df = 0.0, e = 0.0;
  for (int JJ = 0; JJ < multi; JJ++) {
    int J5 = JJ * 5;
    double p_ = 1.0, df1 = 0.0, ddf1 = 0.0;
    for (int loop = 0; loop < co[J5 + 1]; loop++) {
      ddf1 = p_ * c - df1 * s;
      df1 = p_ * s + df1 * c;
      p_ = ddf1;
    }
    p_ = p_ * co[J5 + 3] + df1 * co[J5 + 4];
    df1 = df1 * co[J5 + 3] - ddf1 * co[J5 + 4];
    df1 *= -co[J5 + 1];
    p_ += 1.0;
    if (co[1] == 0) { /* term 0's periodicity tested for every term (src/potential/compute_AMBER.cpp:199) */
      p_ = 1.0 + co[J5 + 3];
      df1 = 0.0;
    }
    df += (-co[J5] * df1);
    e += co[J5] * p_;
  }
  double fg = vb1x * vb2xm + vb1y * vb2ym + vb1z * vb2zm;
  double hg = vb3x * vb2xm + vb3y * vb2ym + vb3z * vb2zm;
  double fga = fg * ra2inv * rginv;
  double hgb = hg * rb2inv * rginv;
  double gaa = -ra2inv * rg;
  double gbb = rb2inv * rg;
  double dtf[3] = {gaa * ax, gaa * ay, gaa * az};
  double dtg[3] = {fga * ax - hgb * bx, fga * ay - hgb * by, fga * az - hgb * bz};
  double dth[3] = {gbb * bx, gbb * by, gbb * bz};
  for (int q = 0; q < 3; q++) {
    double s2 = df * dtg[q];
    double f1 = df * dtf[q];
    double f4 = df * dth[q];
    o.f[0][q] = f1;
    o.f[1][q] = s2 - f1;
    o.f[2][q] = -s2 - f4;
    o.f[3][q] = f4;
  }
  o.e = e;
}

/* ------------------------------------------------------------------------- */
/* FP32 pair terms                                                            */
/* ------------------------------------------------------------------------- */
/* LJ (+ Coulomb) force factor and energy, the reference's formulas:
 *   f = r^-6 (A r^-6 - B) r^-2 [+ qqrd2e qi qj r^-1 r^-2], times w
 *   U = r^-6 (A/12 r^-6 - B/6) [+ qqrd2e qi qj / r]  (unweighted)          */
/* rsqrtf without its scaling of subnormal arguments (three instructions per
 * pair): the same result for every r2 of two atoms that are not in one place */
__device__ __forceinline__ float rsqrt_ftz(float r2) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(r2));
  return r;
}

/* Two FP32 values in one register pair, and the packed operations on them:
 * one instruction for both, each rounded as the single operation is. */
struct Pair2 {
  unsigned long long b;
};
__device__ __forceinline__ Pair2 pack2(float lo, float hi) {
  Pair2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.b) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack2(Pair2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.b));
  return r;
}
__device__ __forceinline__ Pair2 mul2(Pair2 a, Pair2 b) {
  Pair2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
  return r;
}
__device__ __forceinline__ Pair2 fma2(Pair2 a, Pair2 b, Pair2 c) {
  Pair2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.b) : "l"(a.b), "l"(b.b), "l"(c.b));
  return r;
}
/* a + b in single additions: a packed one of a product was made one operation
 * with it, and rounded once, by the assembler */
__device__ __forceinline__ Pair2 add2(Pair2 a, Pair2 b) {
  const float2 u = unpack2(a), v = unpack2(b);
  return pack2(__fadd_rn(u.x, v.x), __fadd_rn(u.y, v.y));
}
__device__ __forceinline__ Pair2 rsqrt2(Pair2 a) {
  const float2 u = unpack2(a);
  return pack2(rsqrt_ftz(u.x), rsqrt_ftz(u.y));
}
__device__ __forceinline__ float lj_coul(float r2, float A, float B, float qq, bool coul, float* e) {
  float rinv = rsqrt_ftz(r2);
  float r2inv = rinv * rinv;
  float r6inv = r2inv * r2inv * r2inv;
  float flj = r6inv * fmaf(A, r6inv, -B);
  float fc = coul ? qq * rinv : 0.0f;
  *e = fmaf(r6inv, fmaf(A * (1.0f / 12.0f), r6inv, -B * (1.0f / 6.0f)), fc);
  return (flj + fc) * r2inv;
}

/* pair energies in FP64 from FP64 coordinates, evaluated only on the steps
 * that request energies: sums of Coulomb terms of both signs cancel by orders
 * of magnitude, which FP32 coordinates cannot resolve */
__device__ __forceinline__ double r2d(const double* a, const double* b) {
  double dx = a[0] - b[0], dy = a[1] - b[1], dz = a[2] - b[2];
  return dx * dx + dy * dy + dz * dz;
}
/* the pair's A / 12 and B / 6 come from tables (d_ljA12, d_ljB6): one
 * division per pair instead of three, and no square root without charges */
__device__ __forceinline__ double lj_energy(double r2, double A12, double B6) {
  double r2inv = 1 / r2;
  double r6inv = r2inv * r2inv * r2inv;
  return r6inv * (A12 * r6inv - B6);
}
__device__ __forceinline__ double lj_coul_energy(double r2, double A12, double B6, double qq) {
  double r2inv = 1 / r2;
  double r6inv = r2inv * r2inv * r2inv;
  return r6inv * (A12 * r6inv - B6) + qq * sqrt(r2inv);
}

/* Born-Mayer-Huggins (Tosi-Fumi NaCl, src/potential/BMHFT/potentialBMHFT.hpp:21-39) */
__constant__ float kBorn[2][2][5] = {
    {{25.4435f * 3.1546f / 4.184f, 6.f * 101.1719f / 4.184f, 8.f * 48.1771f / 4.184f, 2.340f, 3.1546f},
     {20.3548f * 3.1546f / 4.184f, 6.f * 674.4793f / 4.184f, 8.f * 837.077f / 4.184f, 2.755f, 3.1546f}},
    {{20.3548f * 3.1546f / 4.184f, 6.f * 674.4793f / 4.184f, 8.f * 837.077f / 4.184f, 2.755f, 3.1546f},
     {15.2661f * 3.1546f / 4.184f, 6.f * 6985.6786f / 4.184f, 8.f * 14031.5785f / 4.184f, 3.170f, 3.1546f}}};

__device__ __forceinline__ double born_energy(double r2, int ti, int tj, double qq) {
  const float* c = kBorn[ti][tj];
  double r2inv = 1 / r2;
  double r6inv = r2inv * r2inv * r2inv;
  double r = sqrt(r2);
  double rexp = exp((double)c[4] * ((double)c[3] - r));
  return qq * sqrt(r2inv) + rexp * c[0] - (double)c[1] / 6.0 * r6inv - (double)c[2] / 8.0 * r6inv * r2inv;
}

__device__ __forceinline__ float born(float r2, int ti, int tj, float qq, float* e) {
  const float* c = kBorn[ti][tj];
  float rinv = rsqrtf(r2);
  float r = r2 * rinv;
  float r2inv = rinv * rinv;
  float r6inv = r2inv * r2inv * r2inv;
  float rexp = expf(c[4] * (c[3] - r));
  float f1 = c[4] * c[0] * r * rexp;
  float f2 = -c[1] * r6inv;
  float f3 = -c[2] * r6inv * r2inv;
  float fc = qq * rinv;
  *e = fc + rexp * c[0] - c[1] * (1.0f / 6.0f) * r6inv - c[2] * (1.0f / 8.0f) * r6inv * r2inv;
  return (f1 + f2 + f3 + fc) * r2inv;
}

/* FP64 forms of the pair terms (mdn_options.force_mode = 1), with the
 * reference's FP64 constants (src/potential/BMHFT/potentialBMHFT.hpp:21-39) */
__constant__ double kBornD[2][2][5] = {
    {{25.4435 * 3.1546 / 4.184, 6. * 101.1719 / 4.184, 8. * 48.1771 / 4.184, 2.340, 3.1546},
     {20.3548 * 3.1546 / 4.184, 6. * 674.4793 / 4.184, 8. * 837.077 / 4.184, 2.755, 3.1546}},
    {{20.3548 * 3.1546 / 4.184, 6. * 674.4793 / 4.184, 8. * 837.077 / 4.184, 2.755, 3.1546},
     {15.2661 * 3.1546 / 4.184, 6. * 6985.6786 / 4.184, 8. * 14031.5785 / 4.184, 3.170, 3.1546}}};

__device__ __forceinline__ double lj_coul_d(double r2, double A, double B, double qq, bool coul) {
  double r2inv = 1 / r2;
  double r6inv = r2inv * r2inv * r2inv;
  double f = r6inv * (A * r6inv - B);
  if (coul) f += qq * sqrt(r2inv);
  return f * r2inv;
}

__device__ __forceinline__ double born_d(double r2, int ti, int tj, double qq) {
  const double* c = kBornD[ti][tj];
  double r2inv = 1 / r2;
  double r6inv = r2inv * r2inv * r2inv;
  double r = sqrt(r2);
  double rexp = exp(c[4] * (c[3] - r));
  return (c[4] * c[0] * r * rexp - c[1] * r6inv - c[2] * r6inv * r2inv + qq * sqrt(r2inv)) * r2inv;
}

/* taper weight of core atom i in FP64: the float copy is exact at 0 and 1 */
__device__ __forceinline__ double weight_d(const Ctx& x, int i) {
  const float w = x.c.tag[i].w;
  if (w == 0.0f || w == 1.0f) return (double)w;
  return taper(x.P, x.D->ion_com, x.c.x + 3 * i);
}

/* charge of core atom i */
__device__ __forceinline__ double charge_d(const Ctx& x, int i) {
  const RepParams* P = x.P;
  return i < P->n_ion ? x.db[P->d_ion_q + i] : x.db[P->d_vap_q + (i - P->n_ion) % P->a_v];
}

/* ------------------------------------------------------------------------- */
/* forces of the core (ion + vapor) among themselves, and the core kick        */
/* ------------------------------------------------------------------------- */
/* One term of the core force sums.  Each 64-bit fixed-point term
 * u = lo16 + 2^16 mid16 + 2^32 hi32 goes into three 32-bit sums (64-bit
 * shared-memory atomics measured far slower than 32-bit ones here).  The two 16-bit
 * sums are exact for up to 65,536 terms per atom and evaluation (one per
 * near gas molecule, whose list holds at most 64,511, plus at most one per
 * pair tile and per bonded term); the high sum only matters modulo 2^32.
 * core_reduce_kick folds the three into the 64-bit sum exactly, so the result
 * does not depend on the order of the adds. */
__device__ __forceinline__ void acc_add(Ctx& x, int i, const long long* f3) {
  unsigned* A = x.c.chunk + 9 * i;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const unsigned long long u = (unsigned long long)f3[k];
    atomicAdd(&A[3 * k], (unsigned)(u & 0xFFFFull));
    atomicAdd(&A[3 * k + 1], (unsigned)((u >> 16) & 0xFFFFull));
    atomicAdd(&A[3 * k + 2], (unsigned)(u >> 32));
  }
}

__device__ __forceinline__ void energy_add(Ctx& x, int bucket, long long e) {
  if (e != 0) atomicAdd((unsigned long long*)&x.a->energy[8 * x.r + bucket], (unsigned long long)e);
}

__device__ __forceinline__ bool term_on(const Ctx& x, unsigned bit) {
  return (x.P->interactions & bit) && (!x.a->term_mask || (x.a->term_mask & bit));
}

/* Core pairs as 32 x 32 tiles (i block ib <= j block jb), one warp each,
 * every unordered pair evaluated once.  Lane l owns atom i = 32 ib + l; at
 * step s it pairs with j = 32 jb + ((l + s) mod 32), so the lanes read 32
 * distinct j (no bank conflicts), and it keeps the reaction on that j in a
 * register that moves one lane down after every step: after 32 steps lane l
 * holds the whole reaction on j = 32 jb + l.  Diagonal tiles take steps
 * 1..15 and half of step 16, then the reactions move the rest of the way in
 * one shuffle.  Each side is summed over the tile's steps in the pair
 * precision, in that fixed order, and reaches the core sums once per tile as
 * a 64-bit integer, so the result does not depend on the launch shape.
 *
 * What bounds it: the dependent chain of one pair (a warp runs one tile, and
 * a small core has fewer tiles than the SM has warps).  So which pairs count
 * (the exclusions, the ion-vapor and vapor-vapor switches, the atoms of one
 * molecule, the diagonal's half) is worked out once per tile as one bit per
 * step, the LJ + Coulomb form is the same for all three kinds (an ion atom's
 * weight is 1), and the steps carry no branch, so that the compiler
 * interleaves several of them; only a tile with few steps or with
 * Born-Mayer-Huggins pairs (the ion's own, a small cluster) tests each step
 * (with the test in every tile the pairs of 786 atoms took 331 thousand
 * cycles on one CTA, without 244).  Against a branch on the kind per
 * pair: 36.0 -> 32.2 ms per 100 steps of 256 mixed replicas (tuned launch),
 * 2.23 -> 1.85 ms on one 13-atom core, bit-identical results. */
template <bool FP64, bool E>
__device__ __forceinline__ void core_tile(Ctx& x, int t, int nblk) {
  const RepParams* P = x.P;
  const int ni = P->n_ion, nc = x.n_core, nt = P->n_types, av = P->a_v;
  const bool amber = term_on(x, MDN_I_AMBER), bmh = term_on(x, MDN_I_BMH);
  const bool vi = term_on(x, MDN_I_VI), vv = term_on(x, MDN_I_VV);
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int ib = 0, rem = t;
  while (rem >= nblk - ib) {
    rem -= nblk - ib;
    ib++;
  }
  const int jb = ib + rem, j0 = jb * 32;
  const bool diag = ib == jb;
  const int i = ib * 32 + lane;
  const bool act = i < nc;
  const int ii = act ? i : 0;
  const AtomTag gi = x.c.tag[ii];
  const int rowi = tag_type(gi.k) * nt;
  /* the lowest n bits */
  auto low = [](int n) -> unsigned { return n >= 32 ? 0xffffffffu : n <= 0 ? 0u : (1u << n) - 1u; };
  /* bit jl of on: the pair (i, j0 + jl) has the LJ + Coulomb form; of born:
   * the Born-Mayer-Huggins form */
  unsigned on = 0, born_on = 0;
  if (act) {
    const unsigned live = low(nc - j0), ionj = low(ni - j0);
    if (ii < ni) {
      if (amber) on |= ionj & ~(j0 < ni ? x.c.excl[ii * P->excl_words + jb] : 0u);
      if (vi) on |= live & ~ionj;
      if (bmh) born_on = ionj;
    } else {
      if (vi) on |= ionj;
      if (vv) {
        const int m0 = ni + tag_slot(gi.k) * av - j0; /* the molecule's own atoms */
        on |= live & ~ionj & ~(low(m0 + av) & ~low(m0));
      }
    }
    /* rotated so that bit s is step s */
    on = __funnelshift_r(on, on, lane);
    born_on = __funnelshift_r(born_on, born_on, lane);
    if (diag) {
      const unsigned half = lane < 16 ? 0x1fffeu : 0xfffeu;
      on &= half;
      born_on &= half;
    }
  }
  const unsigned any_on = __reduce_or_sync(FULL, on | born_on);
  if (any_on == 0) return;
  long long e_ion = 0, e_vi = 0, e_vv = 0;
  using Acc = typename std::conditional<FP64, double, float>::type;
  Acc F0 = 0, F1 = 0, F2 = 0, R0 = 0, R1 = 0, R2 = 0;
  float4 pi = make_float4(0, 0, 0, 0);
  float qi = 0;
  double xd[3] = {0, 0, 0}, wid = 1.0, qid = 0.0;
  /* charge and taper weight of j0 + lane in FP64: once per tile, handed round
   * by shuffles (a division, loads and for a vapor atom in the shell a cosine
   * per pair otherwise) */
  double q_own = 0.0, w_own = 1.0;
  if constexpr (FP64 || E) {
    for (int k = 0; k < 3; k++) xd[k] = x.c.x[3 * ii + k];
    qid = P->qqrd2e * charge_d(x, ii);
    const int jo = min(j0 + lane, nc - 1);
    q_own = charge_d(x, jo);
    if (FP64) {
      wid = weight_d(x, ii);
      w_own = weight_d(x, jo);
    }
  }
  if constexpr (!FP64) {
    pi = x.c.pos[ii];
    qi = (float)P->qqrd2e * pi.w;
  }
  auto step = [&](int s, auto with_born) {
    constexpr bool kBorn = decltype(with_born)::value;
    const int j = min(j0 + ((lane + s) & 31), nc - 1);
    const AtomTag gj = x.c.tag[j];
    [[maybe_unused]] double qj = 0.0, wj = 1.0;
    if constexpr (FP64 || E) qj = __shfl_sync(FULL, q_own, (lane + s) & 31);
    if constexpr (FP64) wj = __shfl_sync(FULL, w_own, (lane + s) & 31);
    const int tt = rowi + tag_type(gj.k);
    if constexpr (FP64) {
      if (((on | born_on) >> s) & 1u) {
        const double ex = xd[0] - x.c.x[3 * j], ey = xd[1] - x.c.x[3 * j + 1], ez = xd[2] - x.c.x[3 * j + 2];
        const double R2d = ex * ex + ey * ey + ez * ez;
        const double qq = qid * qj;
        double fd = 0.0;
        if ((on >> s) & 1u)
          fd = lj_coul_d(R2d, x.db[P->d_ljA + tt], x.db[P->d_ljB + tt], qq, true) * (wid * wj);
        if (kBorn && ((born_on >> s) & 1u)) fd += born_d(R2d, tag_bmh(gi.k), tag_bmh(gj.k), qq);
        const double fx = fd * ex, fy = fd * ey, fz = fd * ez;
        F0 += fx; F1 += fy; F2 += fz;
        R0 -= fx; R1 -= fy; R2 -= fz;
      }
    } else {
      const float4 pj = x.c.pos[j];
      const float2 AB = x.c.lj[tt];
      const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
      const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
      const float qq = qi * pj.w;
      float ee;
      float fp = lj_coul(r2, AB.x, AB.y, qq, true, &ee) * (gi.w * gj.w);
      fp = ((on >> s) & 1u) ? fp : 0.0f;
      if (kBorn && ((born_on >> s) & 1u)) fp += born(r2, tag_bmh(gi.k), tag_bmh(gj.k), qq, &ee);
      if (((on | born_on) >> s) & 1u) {
        const float fx = fp * dx, fy = fp * dy, fz = fp * dz;
        F0 += fx; F1 += fy; F2 += fz;
        R0 -= fx; R1 -= fy; R2 -= fz;
      }
    }
    if constexpr (E) {
      if (((on | born_on) >> s) & 1u) {
        const double R2e = r2d(xd, x.c.x + 3 * j);
        const double qq = qid * qj;
        double ed = 0;
        if ((on >> s) & 1u) ed += lj_coul_energy(R2e, x.db[P->d_ljA12 + tt], x.db[P->d_ljB6 + tt], qq);
        if (kBorn && ((born_on >> s) & 1u)) ed += born_energy(R2e, tag_bmh(gi.k), tag_bmh(gj.k), qq);
        const bool iion = ii < ni, jion = j < ni;
        if (iion && jion) e_ion += efixd(ed);
        else if (iion != jion) e_vi += efixd(ed);
        else e_vv += efixd(ed);
      }
    }
  };
  const int s1 = diag ? 17 : 32;
  auto pass_on = [&]() {
    R0 = __shfl_sync(FULL, R0, (lane + 1) & 31);
    R1 = __shfl_sync(FULL, R1, (lane + 1) & 31);
    R2 = __shfl_sync(FULL, R2, (lane + 1) & 31);
  };
  if (__any_sync(FULL, born_on != 0) || __popc(any_on) < 12) {
    for (int s = 0; s < s1; s++) {
      if ((any_on >> s) & 1u) step(s, std::true_type());
      pass_on();
    }
  } else {
    /* several steps' forces (and energies) at once, a step that counts no pair
     * of the lane adding zeros, then their sums in order */
    constexpr int kSteps = FP64 || E ? 2 : 4;
    const float2* const row = x.c.lj + rowi;
    for (int s0 = 0; s0 < s1; s0 += kSteps) {
      Acc fx[kSteps], fy[kSteps], fz[kSteps];
      float A[kSteps], B[kSteps], qq[kSteps], w[kSteps];
      bool tk[kSteps];
#pragma unroll
      for (int u = 0; u < kSteps; u++) {
        const int jl = (lane + s0 + u) & 31, j = j0 + jl; /* past the core: type 0, not taken */
        const AtomTag gj = x.c.tag[j];
        const int tt = rowi + tag_type(gj.k);
        const bool take = (on >> u) & 1u; /* none past a diagonal tile's last step */
        double qj = 0.0, R2d = 1.0, ex = 0.0, ey = 0.0, ez = 0.0;
        if constexpr (FP64 || E) {
          qj = qid * __shfl_sync(FULL, q_own, jl);
          const double* const xj = x.c.x + 3 * min(j, nc - 1);
          ex = xd[0] - xj[0];
          ey = xd[1] - xj[1];
          ez = xd[2] - xj[2];
          R2d = ex * ex + ey * ey + ez * ez;
        }
        if constexpr (FP64) {
          const double wj = __shfl_sync(FULL, w_own, jl);
          const double f = lj_coul_d(R2d, x.db[P->d_ljA + tt], x.db[P->d_ljB + tt], qj, true) * (wid * wj);
          const double fd = take ? f : 0.0;
          fx[u] = fd * ex;
          fy[u] = fd * ey;
          fz[u] = fd * ez;
        } else {
          const float4 pj = x.c.pos[j];
          const float2 AB = row[tag_type(gj.k)];
          fx[u] = pi.x - pj.x;
          fy[u] = pi.y - pj.y;
          fz[u] = pi.z - pj.z;
          A[u] = AB.x;
          B[u] = AB.y;
          qq[u] = qi * pj.w;
          w[u] = gi.w * gj.w;
          tk[u] = take;
          if constexpr (kGG) {
            const float r2 = fmaf(fx[u], fx[u], fmaf(fy[u], fy[u], fz[u] * fz[u]));
            float ee;
            const float f = lj_coul(r2, A[u], B[u], qq[u], true, &ee) * w[u];
            const float fp = take ? f : 0.0f;
            fx[u] = fp * fx[u];
            fy[u] = fp * fy[u];
            fz[u] = fp * fz[u];
          }
        }
        if constexpr (E) {
          const double ed = lj_coul_energy(R2d, x.db[P->d_ljA12 + tt], x.db[P->d_ljB6 + tt], qj);
          const long long e = take ? efixd(ed) : 0;
          const bool iion = ii < ni, jion = j < ni;
          e_ion += iion && jion ? e : 0;
          e_vi += iion != jion ? e : 0;
          e_vv += !iion && !jion ? e : 0;
        }
      }
      /* lj_coul, two steps in a register pair: fewer instructions per
       * pair (100-atom chain 1418 -> 1371 us per 100 steps, 500-atom ion 2568
       * -> 2533); not beside the gas-gas term, whose kernel has no registers
       * left for it (1540 -> 1549 per 50 steps) */
      if constexpr (!FP64 && !kGG)
#pragma unroll
        for (int u = 0; u < kSteps; u += 2) {
          const Pair2 dx = pack2(fx[u], fx[u + 1]), dy = pack2(fy[u], fy[u + 1]), dz = pack2(fz[u], fz[u + 1]);
          const Pair2 rinv = rsqrt2(fma2(dx, dx, fma2(dy, dy, mul2(dz, dz))));
          const Pair2 r2inv = mul2(rinv, rinv), r6inv = mul2(mul2(r2inv, r2inv), r2inv);
          const float2 r6 = unpack2(r6inv);
          const Pair2 t = pack2(fmaf(A[u], r6.x, -B[u]), fmaf(A[u + 1], r6.y, -B[u + 1]));
          const Pair2 fc = mul2(pack2(qq[u], qq[u + 1]), rinv);
          const float2 f = unpack2(mul2(mul2(add2(mul2(r6inv, t), fc), r2inv), pack2(w[u], w[u + 1])));
          const Pair2 fp = pack2(tk[u] ? f.x : 0.0f, tk[u + 1] ? f.y : 0.0f);
          const float2 gx = unpack2(mul2(fp, dx)), gy = unpack2(mul2(fp, dy)), gz = unpack2(mul2(fp, dz));
          fx[u] = gx.x; fx[u + 1] = gx.y;
          fy[u] = gy.x; fy[u + 1] = gy.y;
          fz[u] = gz.x; fz[u + 1] = gz.y;
        }
      on >>= kSteps;
#pragma unroll
      for (int u = 0; u < kSteps; u++) {
        if (s0 + u == s1) break;
        F0 += fx[u]; F1 += fy[u]; F2 += fz[u];
        R0 -= fx[u]; R1 -= fy[u]; R2 -= fz[u];
        pass_on();
      }
    }
  }
  if (diag) {
    R0 = __shfl_sync(FULL, R0, (lane + 15) & 31);
    R1 = __shfl_sync(FULL, R1, (lane + 15) & 31);
    R2 = __shfl_sync(FULL, R2, (lane + 15) & 31);
  }
  auto fix = [](Acc v) -> long long {
    if constexpr (FP64) return fixd(v);
    else return fixf(v);
  };
  if (act && (F0 != 0 || F1 != 0 || F2 != 0)) {
    const long long F[3] = {fix(F0), fix(F1), fix(F2)};
    acc_add(x, i, F);
  }
  const int jj = j0 + lane;
  if (jj < nc && (R0 != 0 || R1 != 0 || R2 != 0)) {
    const long long Rv[3] = {fix(R0), fix(R1), fix(R2)};
    acc_add(x, jj, Rv);
  }
  if constexpr (E) {
    e_ion = warp_sum_ll(e_ion);
    e_vi = warp_sum_ll(e_vi);
    e_vv = warp_sum_ll(e_vv);
    if (lane == 0) {
      energy_add(x, MDN_U_ION, e_ion);
      energy_add(x, MDN_U_VI, e_vi);
      energy_add(x, MDN_U_VV, e_vv);
    }
  }
}

/* MDN_FP64_PAIRS selects the pair precision of this compilation: the FP64
 * form (mdn_options.force_mode = 1) is compiled into its own kernel,
 * mdn_advance_fp64 (advance_fp64.cu), so that the FP32 kernel's registers
 * and code are not shaped by it */
#ifdef MDN_FP64_PAIRS
constexpr bool kFP64Pairs = true;
#else
constexpr bool kFP64Pairs = false;
#endif


/* The bonded terms of the core: every dihedral (the ion's, then the vapor
 * molecules'), then every angle, then every bond, so that a warp's 32 terms
 * are of one kind but at the two seams. */
struct BondedCount {
  int nd, na, nb, vd, va, vb, nv; /* ion terms, terms per vapor molecule, vapor molecules */
  __device__ __forceinline__ int total() const { return nd + na + nb + (vd + va + vb) * nv; }
};
__device__ __forceinline__ BondedCount bonded_count(const Ctx& x) {
  const RepParams* P = x.P;
  const bool amber = term_on(x, MDN_I_AMBER), vin = term_on(x, MDN_I_VAPOR_INTRA);
  BondedCount c;
  c.nd = amber ? P->n_ion_dih : 0;
  c.na = amber ? P->n_ion_angles : 0;
  c.nb = amber ? P->n_ion_bonds : 0;
  c.vd = vin ? P->n_vap_dih : 0;
  c.va = vin ? P->n_vap_angles : 0;
  c.vb = vin ? P->n_vap_bonds : 0;
  c.nv = x.D->n_vap_in;
  return c;
}

/* terms 32 k .. 32 k + 31, one per lane */
template <bool E>
__device__ __forceinline__ void bonded_terms(Ctx& x, const BondedCount& bc, int k) {
  const RepParams* P = x.P;
  const bool qb = (P->quirks & MDN_Q_ENERGY_BUCKETS) != 0;
  const int lane = threadIdx.x & 31;
  int u = 32 * k + lane;
  const bool on = u < bc.total();
  long long e = 0;
  int bucket = MDN_U_ION;
  if (on) {
    /* kind: 2 dihedral, 1 angle, 0 bond; the row's place among the ion's
     * (base 0) or in vapor molecule s */
    int kind = 2, n_ion = bc.nd, per = bc.vd;
    if (u >= bc.nd + bc.vd * bc.nv) {
      u -= bc.nd + bc.vd * bc.nv;
      kind = 1, n_ion = bc.na, per = bc.va;
      if (u >= bc.na + bc.va * bc.nv) {
        u -= bc.na + bc.va * bc.nv;
        kind = 0, n_ion = bc.nb, per = bc.vb;
      }
    }
    const bool vap = u >= n_ion;
    int base = 0;
    if (vap) {
      const int s = (u - n_ion) / per;
      u = u - n_ion - s * per;
      base = P->n_ion + s * P->a_v;
      bucket = qb ? (kind == 2 ? MDN_U_ION : MDN_U_GAS) : MDN_U_VAP;
    }
    const double* X = x.c.x + 3 * base;
    BondOut o;
    int n;
    const int* row;
    if (kind == 2) {
      row = x.ib + (vap ? P->o_vap_dih : P->o_ion_dih) + 5 * u;
      dihedral_fd(X, x.db + P->d_dih + 15 * row[4], x.ib[P->o_dih_multi + row[4]], row[0], row[1], row[2], row[3], o);
      n = 4;
    } else if (kind == 1) {
      row = x.ib + (vap ? P->o_vap_angles : P->o_ion_angles) + 4 * u;
      angle_fd(X, x.db + P->d_angle + 2 * row[3], row[0], row[1], row[2], o);
      n = 3;
    } else {
      row = x.ib + (vap ? P->o_vap_bonds : P->o_ion_bonds) + 3 * u;
      bond_fd(X, x.db + P->d_bond + 2 * row[2], row[0], row[1], o);
      n = 2;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (q >= n) break;
      const long long F[3] = {fixd(o.f[q][0]), fixd(o.f[q][1]), fixd(o.f[q][2])};
      acc_add(x, base + row[q], F);
    }
    if (E) e = efixd(o.e);
  }
  if (E) {
    for (int b = MDN_U_ION; b <= MDN_U_VAP; b++) {
      const long long s = warp_sum_ll(bucket == b ? e : 0);
      if (lane == 0) energy_add(x, b, s);
    }
  }
}

/* the uniform field on the ion's charges, one warp */
__device__ __forceinline__ void field_terms(Ctx& x) {
  const RepParams* P = x.P;
  for (int i = threadIdx.x & 31; i < P->n_ion; i += 32) {
    const double coeff = 5.55e-5 * x.db[P->d_ion_q + i];
    const long long F[3] = {fixd(coeff * P->efield[0]), fixd(coeff * P->efield[1]), fixd(coeff * P->efield[2])};
    acc_add(x, i, F);
  }
}

/* ------------------------------------------------------------------------- */
/* gas molecules                                                              */
/* ------------------------------------------------------------------------- */
__device__ __forceinline__ void partition(const Ctx& x, int n, int* lo, int* hi) {
  *lo = (int)(((long long)n * x.rank) / x.C);
  *hi = (int)(((long long)n * (x.rank + 1)) / x.C);
}

/* This CTA's part of the slab.  Kept in shared memory (set_slab_part, where
 * n_gas_in is set): two 64-bit divisions would stand at the start of every
 * item that works on gas molecules. */
__device__ __forceinline__ void slab_part(const Ctx& x, int* lo, int* hi) {
  *lo = x.iscr[53];
  *hi = x.iscr[54];
}
__device__ __forceinline__ void set_slab_part(const Ctx& x) { /* one thread; a barrier follows */
  partition(x, x.D->n_gas_in, &x.iscr[53], &x.iscr[54]);
}

/* The near molecules' x, v and f between rebuilds: rows of 32 molecules by
 * component, in record order (heavy ones first, the light ones from the next
 * multiple of 32), so that a warp's group reads and writes whole lines.  In
 * the slab the records of a group, sorted by partners, lie apart: each of its
 * 18 loads and 18 stores touched 32 lines, 220 of the 494 thousand cycles
 * that the near pass of a 20,000-atom domain took on one CTA.  near_copy
 * brings them from the slab and back: at the start and the end of a launch
 * and around a rebuild. */
__device__ __forceinline__ int near_row(const Ctx& x, int k) { /* row of record k of this CTA */
  const int nh = x.iscr[56];
  return k < nh ? k : ((nh + 31) & ~31) + k - nh;
}
__device__ __forceinline__ double* near_base(const Ctx& x) {
  const RepParams* P = x.P;
  int lo, hi;
  slab_part(x, &lo, &hi);
  return x.a->near_s + P->ns_off + (size_t)9 * P->a_g * (((lo + 31) & ~31) + 64 * x.rank);
}
/* component q (x, then v, then f; 3 a_g of each) of a row */
template <int AG>
__device__ __forceinline__ double* near_at(double* base, int row) {
  return base + (size_t)(row >> 5) * (32 * 9 * AG) + (row & 31);
}

/* the row of record k, slab slot s; in the kernels with gas-gas terms the
 * slab's own, which those terms read on every step */
struct NearRow {
  double *px, *pv, *pf;
  __device__ __forceinline__ double& x(int q) const { return px[kGG ? q : 32 * q]; }
  __device__ __forceinline__ double& v(int q) const { return pv[kGG ? q : 32 * q]; }
  __device__ __forceinline__ double& f(int q) const { return pf[kGG ? q : 32 * q]; }
};
template <int AG>
__device__ __forceinline__ NearRow near_ref(const Ctx& x, int k, int s) {
  if constexpr (kGG) {
    const size_t g0 = 3 * gatom(x.P, x.D->parity, s, 0);
    return NearRow{x.a->slab_x + g0, x.a->slab_v + g0, x.a->slab_f + g0};
  } else {
    double* const S = near_at<AG>(near_base(x), near_row(x, k));
    return NearRow{S, S + 32 * 3 * AG, S + 32 * 6 * AG};
  }
}

/* intramolecular bond force of one gas molecule (PotentialGasIntra), FP64 */
/* Gas molecules have one or two atoms (AG); the bonded and SHAKE terms of a
 * two-atom molecule copy the pair into fixed slots (swapped when a row reads
 * (1, 0)) so that every array index is a compile-time constant and the
 * arrays stay in registers.  The arithmetic is that of bond_fd / shake_pair
 * on the row's own order. */
template <int AG>
__device__ __forceinline__ double gas_intra(const Ctx& x, const double* X, double* F) {
  if constexpr (AG == 1) {
    return 0.0;
  } else {
    const RepParams* P = x.P;
    double e = 0;
    for (int b = 0; b < P->n_gas_bonds; b++) {
      const int* row = x.ib + P->o_gas_bonds + 3 * b;
      const bool sw = row[0] != 0;
      double Y[6];
      for (int k = 0; k < 3; k++) {
        Y[k] = sw ? X[3 + k] : X[k];
        Y[3 + k] = sw ? X[k] : X[3 + k];
      }
      BondOut o;
      bond_fd(Y, x.db + P->d_bond + 2 * row[2], 0, 1, o);
      for (int k = 0; k < 3; k++) {
        F[k] += sw ? o.f[1][k] : o.f[0][k];
        F[3 + k] += sw ? o.f[0][k] : o.f[1][k];
      }
      e += o.e;
    }
    return e;
  }
}

/* SHAKE of a two-atom gas molecule: the sweeps of the vapor SHAKE with one colour */
__device__ __forceinline__ int shake_gas2(const Ctx& x, double* X, const double* R) {
  const RepParams* P = x.P;
  const int* rigid = x.ib + P->o_gas_rigid;
  const int n = P->n_gas_rigid;
  bool converge = false;
  for (int sweep = 0; sweep < MDN_SHAKE_MAX_SWEEPS && !converge; sweep++) {
    for (int k = 0; k < n; k++) {
      const bool sw = rigid[3 * k] != 0;
      double Y[6], RY[6];
      for (int q = 0; q < 3; q++) {
        Y[q] = sw ? X[3 + q] : X[q];
        Y[3 + q] = sw ? X[q] : X[3 + q];
        RY[q] = sw ? R[3 + q] : R[q];
        RY[3 + q] = sw ? R[q] : R[3 + q];
      }
      shake_pair_c(Y, Y + 3, RY, RY + 3, x.db + P->d_gas_cons + 3 * k);
      for (int q = 0; q < 3; q++) {
        X[q] = sw ? Y[3 + q] : Y[q];
        X[3 + q] = sw ? Y[q] : Y[3 + q];
      }
    }
    converge = true;
    for (int k = 0; k < n; k++)
      if (!(shake_res_c(X, X + 3, x.db + P->d_gas_cons + 3 * k) <= 1e-20)) converge = false;
  }
  return converge ? 0 : MDN_ST_SHAKE_NOCONV;
}

/* first kick, drift and constraint of one gas molecule in registers: X, V
 * and F of its atoms (F the force of the last evaluation) */
template <int AG>
__device__ __forceinline__ void gas_drift(Ctx& x, double* X, double* V, const double* F, const double* c2, bool sh,
                                          bool vcorr, double dt) {
  double R[3 * AG];
#pragma unroll
  for (int q = 0; q < 3 * AG; q++) {
    V[q] += F[q] * c2[q / 3];
    R[q] = X[q];
    X[q] = X[q] + V[q] * dt;
  }
  if constexpr (AG == 2) {
    if (sh) {
      double Xd[3 * AG];
#pragma unroll
      for (int q = 0; q < 3 * AG; q++) Xd[q] = X[q];
      const int st = shake_gas2(x, X, R);
      if (st) set_status(x, st);
      if (vcorr)
#pragma unroll
        for (int q = 0; q < 3 * AG; q++) V[q] += (X[q] - Xd[q]) / dt;
    }
  }
}

template <int AG>
__device__ __forceinline__ void gas_finite(const Ctx& x, const double* X, const double* V) {
  if (!isfinite(X[0] + X[1] + X[2] + V[0] + V[1] + V[2])) set_status(x, MDN_ST_NONFINITE);
}

/* thread tid of the nthr (whole warps) that take part */
template <int AG>
__device__ __forceinline__ void gas_integrate_t(Ctx& x, GasWork w, bool eflag, int tid, int nthr) {
  const RepParams* P = x.P;
  const KArgs* a = x.a;
  const int par = x.D->parity;
  const bool vcorr = !(P->quirks & MDN_Q_SHAKE_NO_VCORR);
  const bool intra = AG == 2 && term_on(x, MDN_I_GAS_INTRA) && P->n_gas_bonds > 0;
  int lo, hi;
  slab_part(x, &lo, &hi);
  double c2[AG];
#pragma unroll
  for (int at = 0; at < AG; at++) c2[at] = x.c.c2[x.iscr[58 + at]];
  const int nf = w.far ? x.iscr[61] : 0, n = w.all ? hi - lo : nf + (w.near ? x.iscr[57] : 0);
  long long eg = 0;
  for (int e = tid; e < n; e += nthr) {
    /* the slab's rows, or a near molecule's */
    const bool slab = w.all || e < nf;
    const size_t g0 = slab ? 3 * gatom(P, par, w.all ? lo + e : a->far_list[P->near_off + lo + e], 0) : 0;
    const NearRow S =
        near_ref<AG>(x, slab ? 0 : e - nf, kGG && !slab ? a->near_rec[P->near_off + lo + e - nf].x : 0);
    double* const rx = slab ? a->slab_x + g0 : S.px;
    double* const rv = slab ? a->slab_v + g0 : S.pv;
    double* const rf = slab ? a->slab_f + g0 : S.pf;
    const int st = slab || kGG ? 1 : 32;
    double X[3 * AG], V[3 * AG], F[3 * AG];
#pragma unroll
    for (int q = 0; q < 3 * AG; q++) {
      X[q] = rx[st * q];
      V[q] = rv[st * q];
      F[q] = rf[st * q];
    }
    gas_drift<AG>(x, X, V, F, c2, gas_rigid(P), vcorr, P->dt);
    gas_finite<AG>(x, X, V);
#pragma unroll
    for (int q = 0; q < 3 * AG; q++) F[q] = 0.0;
    if (!w.all && slab) {
      if (intra) {
        const double ei = gas_intra<AG>(x, X, F);
        if (eflag) eg += efixd(ei);
      }
#pragma unroll
      for (int q = 0; q < 3 * AG; q++) V[q] += F[q] * c2[q / 3];
    }
#pragma unroll
    for (int q = 0; q < 3 * AG; q++) {
      rx[st * q] = X[q];
      rv[st * q] = V[q];
      rf[st * q] = F[q];
    }
  }
  if (eflag && intra && w.far) {
    eg = warp_sum_ll(eg);
    if ((threadIdx.x & 31) == 0) energy_add(x, MDN_U_GAS, eg);
  }
}

__device__ __forceinline__ void gas_integrate(Ctx& x, GasWork w, bool eflag, int tid, int nthr) {
  if (x.P->a_g == 1) gas_integrate_t<1>(x, w, eflag, tid, nthr);
  else gas_integrate_t<2>(x, w, eflag, tid, nthr);
}

/* The far molecules (no list entry) over the next k steps at once, for a
 * CTA with more of them than threads.  Until the next rebuild nothing but
 * their own bond acts on them, so the k steps of a molecule run in one
 * thread's registers: the slab is read and written once per k steps (k: to
 * the rebuild or the end of the launch) instead of once per step, 144 B per
 * atom each time.  With fewer molecules the k dependent steps of a thread
 * would be waited for (134 rigid N2 over 8 CTAs: 2.06 ms per 100 steps
 * against 1.89 ms beside the core's constraints, GasWork).  The operations of each step are those of gas_drift
 * and the second kick, in their order.  energy_mode, last: as one_step's
 * eflag, energies of every step or of the last of these k. */
template <int AG>
__device__ __forceinline__ void gas_far_steps_t(Ctx& x, long long k, int energy_mode, bool last) {
  const RepParams* P = x.P;
  const KArgs* a = x.a;
  const int par = x.D->parity;
  const bool sh = gas_rigid(P);
  const bool vcorr = !(P->quirks & MDN_Q_SHAKE_NO_VCORR);
  const bool intra = AG == 2 && term_on(x, MDN_I_GAS_INTRA) && P->n_gas_bonds > 0;
  const double dt = P->dt;
  int lo, hi;
  slab_part(x, &lo, &hi);
  const int* far = a->far_list + P->near_off + lo;
  const int n_far = x.iscr[61];
  double c2[AG];
#pragma unroll
  for (int at = 0; at < AG; at++) c2[at] = x.c.c2[x.iscr[58 + at]];
  long long eg = 0;
  for (int e = threadIdx.x; e < n_far; e += blockDim.x) {
    const size_t g0 = 3 * gatom(P, par, far[e], 0);
    double X[3 * AG], V[3 * AG], F[3 * AG];
#pragma unroll
    for (int q = 0; q < 3 * AG; q++) {
      X[q] = a->slab_x[g0 + q];
      V[q] = a->slab_v[g0 + q];
      F[q] = a->slab_f[g0 + q];
    }
    for (long long t = 0; t < k; t++) {
      gas_drift<AG>(x, X, V, F, c2, sh, vcorr, dt);
#pragma unroll
      for (int q = 0; q < 3 * AG; q++) F[q] = 0.0;
      if (intra) {
        const double ei = gas_intra<AG>(x, X, F);
        if (energy_mode == 2 || (energy_mode == 1 && last && t == k - 1)) eg += efixd(ei);
      }
#pragma unroll
      for (int q = 0; q < 3 * AG; q++) V[q] += F[q] * c2[q / 3];
      if (AG == 1 && t == 0) {
        /* no force from here on: V stays as it is */
        for (t = 1; t < k; t++)
#pragma unroll
          for (int q = 0; q < 3 * AG; q++) X[q] = X[q] + V[q] * dt;
        break;
      }
    }
    gas_finite<AG>(x, X, V);
#pragma unroll
    for (int q = 0; q < 3 * AG; q++) {
      a->slab_x[g0 + q] = X[q];
      a->slab_v[g0 + q] = V[q];
      a->slab_f[g0 + q] = F[q];
    }
  }
  if (intra && (energy_mode == 2 || (energy_mode == 1 && last))) {
    eg = warp_sum_ll(eg);
    if ((threadIdx.x & 31) == 0) energy_add(x, MDN_U_GAS, eg);
  }
}

__device__ __forceinline__ void gas_far_steps(Ctx& x, long long k, int energy_mode, bool last) {
  if (x.P->a_g == 1) gas_far_steps_t<1>(x, k, energy_mode, last);
  else gas_far_steps_t<2>(x, k, energy_mode, last);
}

/* after a rebuild: intramolecular force and second kick of the far molecules */
template <int AG>
__device__ __forceinline__ void gas_far_pass_t(Ctx& x, bool eflag, bool kick) {
  const RepParams* P = x.P;
  const KArgs* a = x.a;
  constexpr int ag = AG;
  const int par = x.D->parity;
  const bool intra = term_on(x, MDN_I_GAS_INTRA) && P->n_gas_bonds > 0;
  const bool gg = kGG && term_on(x, MDN_I_GG) && P->ggl_cap > 0;
  int lo, hi;
  slab_part(x, &lo, &hi);
  double c2[AG];
#pragma unroll
  for (int at = 0; at < ag; at++) c2[at] = x.c.c2[x.ib[P->o_gas_type + at]];
  long long eg = 0;
  for (int s = lo + threadIdx.x; s < hi; s += blockDim.x) {
    if (a->near_gi[gmol(P, par, s)] >= 0) continue;
    double X[3 * AG], F[3 * AG];
    for (int at = 0; at < ag; at++) {
      size_t g = gatom(P, par, s, at);
      for (int k = 0; k < 3; k++) {
        X[3 * at + k] = a->slab_x[3 * g + k];
        F[3 * at + k] = 0.0;
      }
    }
    if (intra) {
      double e = gas_intra<AG>(x, X, F);
      if (eflag) eg += efixd(e);
    }
    if (gg)
      for (int at = 0; at < ag; at++)
        for (int k = 0; k < 3; k++) F[3 * at + k] += a->slab_fgg[3 * gatom(P, par, s, at) + k];
    for (int at = 0; at < ag; at++) {
      size_t g = gatom(P, par, s, at);
      for (int k = 0; k < 3; k++) {
        if (kick) a->slab_v[3 * g + k] += F[3 * at + k] * c2[at];
        a->slab_f[3 * g + k] = F[3 * at + k];
      }
    }
  }
  if (eflag && intra) {
    eg = warp_sum_ll(eg);
    if ((threadIdx.x & 31) == 0) energy_add(x, MDN_U_GAS, eg);
  }
}

__device__ __forceinline__ void gas_far_pass(Ctx& x, bool eflag, bool kick) {
  if (x.P->a_g == 1) gas_far_pass_t<1>(x, eflag, kick);
  else gas_far_pass_t<2>(x, eflag, kick);
}

/* gas-gas LJ, the corrected form of PotentialGasGas::compute
 * (src/potential/GasGas.cpp:4-38): every atom pair of two listed in-domain
 * gas molecules, force x w_i w_j with both atoms' taper weights, energy
 * unweighted into Ugg.  The reference's own routine pairs loop indices
 * instead of gas_in entries (:48-57), reads weight[0][jj] (:25), bounds the
 * partner loop by the first molecule's size (:13) and books the energy in
 * Uvg (:34); none of that is reproduced.  kGGLanes lanes per slab molecule
 * of this CTA walk its full (both-direction) partner list; their integer
 * sums are its force, so no reaction is scattered and the sum does not
 * depend on the launch shape.  A partner is a chain of loads (list entry,
 * position), so with one lane per molecule a CTA with 114 molecules waited
 * for some 20 of them one after another.  Weights come from the current positions and ion centre, as
 * MD::update_position sets them (src/verlet.cpp:109-134); molecules the
 * rebuild of this step inserted have weight 0 (`fresh`: this step rebuilt). */
constexpr int kGGLanes = 8;
template <int AG, bool FP64>
__device__ __forceinline__ void gas_gg_pass_t(Ctx& x, bool eflag, bool fresh) {
  const RepParams* P = x.P;
  const KArgs* a = x.a;
  const int par = x.D->parity, nt = P->n_types, nreb = x.D->n_rebuilds;
  int lo, hi;
  slab_part(x, &lo, &hi);
  int gtype[AG];
#pragma unroll
  for (int at = 0; at < AG; at++) gtype[at] = x.ib[P->o_gas_type + at];
  const double* com = x.D->ion_com;
  long long egg = 0;
  const int lane = threadIdx.x & (kGGLanes - 1);
  for (int s0 = lo; s0 < hi; s0 += blockDim.x / kGGLanes) {
    const int sm = s0 + (int)threadIdx.x / kGGLanes, s = min(sm, hi - 1); /* whole warps stay for the shuffles */
    const size_t ms = gmol(P, par, s);
    const bool s_new = fresh && __ldcg(a->slab_ins + ms) == nreb;
    double X[3 * AG], w[AG];
#pragma unroll
    for (int at = 0; at < AG; at++) {
      const size_t g = gatom(P, par, s, at);
      for (int k = 0; k < 3; k++) X[3 * at + k] = a->slab_x[3 * g + k];
      w[at] = s_new ? 0.0 : taper(P, com, X + 3 * at);
    }
    long long F[AG][3];
#pragma unroll
    for (int at = 0; at < AG; at++) F[at][0] = F[at][1] = F[at][2] = 0;
    const int start = a->ggl_start[ms], cnt = sm < hi ? a->ggl_n[ms] : 0;
    for (int q = lane; q < cnt; q += kGGLanes) {
      const int t = a->ggl[P->ggl_off + start + q];
      const bool t_new = fresh && __ldcg(a->slab_ins + gmol(P, par, t)) == nreb;
#pragma unroll
      for (int b = 0; b < AG; b++) {
        const size_t gt = gatom(P, par, t, b);
        /* another CTA's molecule, moved this step: from L2 */
        const double Y[3] = {__ldcg(a->slab_x + 3 * gt), __ldcg(a->slab_x + 3 * gt + 1),
                             __ldcg(a->slab_x + 3 * gt + 2)};
        const double wb = t_new ? 0.0 : taper(P, com, Y);
        const int tb = gtype[b];
#pragma unroll
        for (int at = 0; at < AG; at++) {
          const int ta = gtype[at];
          long long fx, fy, fz;
          if constexpr (FP64) {
            const double ex = X[3 * at] - Y[0], ey = X[3 * at + 1] - Y[1], ez = X[3 * at + 2] - Y[2];
            const double fd = lj_coul_d(ex * ex + ey * ey + ez * ez, x.db[P->d_ljA + ta * nt + tb],
                                        x.db[P->d_ljB + ta * nt + tb], 0.0, false) * (w[at] * wb);
            fx = fixd(fd * ex); fy = fixd(fd * ey); fz = fixd(fd * ez);
          } else {
            /* the displacement from the FP64 positions: both atoms may sit
             * 100 A from the ion centre, where FP32 coordinates would carry
             * 1e-5 A of rounding into a 3 A separation */
            const float dx = (float)(X[3 * at] - Y[0]), dy = (float)(X[3 * at + 1] - Y[1]),
                        dz = (float)(X[3 * at + 2] - Y[2]);
            const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            float ee;
            const float fp = lj_coul(r2, x.c.lj[ta * nt + tb].x, x.c.lj[ta * nt + tb].y, 0.0f, false, &ee) *
                             (float)(w[at] * wb);
            fx = fixf(fp * dx); fy = fixf(fp * dy); fz = fixf(fp * dz);
          }
          F[at][0] += fx; F[at][1] += fy; F[at][2] += fz;
          if (eflag && t > s)
            egg += efixd(lj_energy(r2d(X + 3 * at, Y), x.db[P->d_ljA12 + ta * nt + tb],
                                   x.db[P->d_ljB6 + ta * nt + tb]));
        }
      }
    }
#pragma unroll
    for (int at = 0; at < AG; at++) {
      const size_t g = gatom(P, par, s, at);
      for (int k = 0; k < 3; k++) {
        long long v = F[at][k];
#pragma unroll
        for (int m = kGGLanes / 2; m; m >>= 1) v += shfl_xor_ll(v, m);
        const double f = (double)v * MDN_FIX_INV;
        if (lane == 0 && sm < hi) {
          if (!(fabs(f) < MDN_FIX_LIMIT)) set_status(x, MDN_ST_FIXED_OVERFLOW);
          a->slab_fgg[3 * g + k] = f;
        }
      }
    }
  }
  if (eflag) {
    egg = warp_sum_ll(egg);
    if ((threadIdx.x & 31) == 0) energy_add(x, MDN_U_GG, egg);
  }
}

/* the gas-gas forces of this step, when gg LJ is on: every CTA of the
 * cluster must see the final gas positions first */
__device__ __forceinline__ void gas_gg_pass(Ctx& x, cg::cluster_group& cl, bool eflag, bool fresh) {
  if constexpr (kGG) {
    if (!(term_on(x, MDN_I_GG) && x.P->ggl_cap > 0)) return;
    __threadfence();
    cl.sync();
    if (x.P->a_g == 1) gas_gg_pass_t<1, kFP64Pairs>(x, eflag, fresh);
    else gas_gg_pass_t<2, kFP64Pairs>(x, eflag, fresh);
    __syncthreads();
  }
}

/* LJ force of one (gas atom, core atom j) pair as 64-bit fixed point, the
 * force on the gas atom (PotentialGasIon / PotentialVaporGas: no Coulomb,
 * no taper weight); the near pass adds it to the gas atom and its negative
 * to the core atom's sums. */
template <bool FP64>
__device__ __forceinline__ void gas_core_pair(const Ctx& x, const double* Xa, float3 ga, int ta, int j,
                                              long long* f) {
  const RepParams* P = x.P;
  const int nt = P->n_types, tj = tag_type(x.c.tag[j].k);
  if constexpr (FP64) {
    const double ex = Xa[0] - x.c.x[3 * j], ey = Xa[1] - x.c.x[3 * j + 1], ez = Xa[2] - x.c.x[3 * j + 2];
    const double fd = lj_coul_d(ex * ex + ey * ey + ez * ez, x.db[P->d_ljA + ta * nt + tj],
                                x.db[P->d_ljB + ta * nt + tj], 0.0, false);
    f[0] = fixd(fd * ex); f[1] = fixd(fd * ey); f[2] = fixd(fd * ez);
  } else {
    const float4 pj = x.c.pos[j];
    const float dx = ga.x - pj.x, dy = ga.y - pj.y, dz = ga.z - pj.z;
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    float ee;
    const float2 AB = x.c.lj[ta * nt + tj];
    const float fp = lj_coul(r2, AB.x, AB.y, 0.0f, false, &ee);
    f[0] = fixf(fp * dx); f[1] = fixf(fp * dy); f[2] = fixf(fp * dz);
  }
}

/* One core partner j of a near gas molecule: the LJ pairs of its AG atoms
 * with j, their forces added to F (64-bit fixed point), the reaction on j to
 * the core sums (shared 32-bit atomics on exact chunks, acc_add), and with
 * eflag the pair energy to e.  X holds the molecule's FP64 positions (used
 * by the FP64 pairs and the energies), gp its FP32 positions relative to the
 * ion centre. */
template <int AG, bool FP64>
__device__ __forceinline__ void near_partner(Ctx& x, const double* X, const float3* gp, const int* gtype, int j,
                                             bool eflag, long long (*F)[3], long long& e) {
  const RepParams* P = x.P;
  const int nt = P->n_types, tj = tag_type(x.c.tag[j].k);
  long long R[3] = {0, 0, 0};
#pragma unroll
  for (int at = 0; at < AG; at++) {
    long long f[3];
    gas_core_pair<FP64>(x, X + 3 * at, gp[at], gtype[at], j, f);
    F[at][0] += f[0]; F[at][1] += f[1]; F[at][2] += f[2];
    R[0] -= f[0]; R[1] -= f[1]; R[2] -= f[2];
    if (eflag)
      e += efixd(lj_energy(r2d(X + 3 * at, x.c.x + 3 * j), x.db[P->d_ljA12 + gtype[at] * nt + tj],
                           x.db[P->d_ljB6 + gtype[at] * nt + tj]));
  }
  acc_add(x, j, R);
}

/* exchange one int per CTA across the cluster: returns the prefix before this
 * rank and the total */
__device__ __forceinline__ void cluster_prefix(Ctx& x, cg::cluster_group& cl, int* slot_in_smem, int mine, int* before,
                               int* total) {
  if (threadIdx.x == 0) *slot_in_smem = mine;
  cl.sync();
  int b = 0, t = 0;
  for (int k = 0; k < x.C; k++) {
    int v = *cl.map_shared_rank(slot_in_smem, k);
    if (k < x.rank) b += v;
    t += v;
  }
  *before = b;
  *total = t;
  cl.sync();
}

/* A near molecule with more partners than this has them spread over several lanes. */
constexpr int kNearHeavy = 16;
/* bins of the near molecules by partners, most first: the heavy ones by
 * eights, then one bin per number */
constexpr int kHeavyBins = 32;
constexpr int kNearBins = kHeavyBins + kNearHeavy;
__device__ __forceinline__ int near_bin(int c) {
  return c > kNearHeavy ? max(0, kHeavyBins - 1 - (c - kNearHeavy - 1) / 8) : kHeavyBins + kNearHeavy - c;
}

/* core atoms a gas-vapor entry reaches in its vapor molecule */
__device__ __forceinline__ int gv_reach(const RepParams* P) {
  return (P->quirks & MDN_Q_GV_GAS_COUNT) ? min(P->a_g, P->a_v) : P->a_v;
}

/* The near molecules (those with a gas-ion or gas-vapor entry) of this CTA's
 * slab partition as records {slab slot, first item, items, 0}, most partners
 * first, and their partners as core atom indices: `near_item` holds a heavy
 * molecule's partners one after another, and those of a group of 32 light
 * records interleaved (entry e of the group's lane l at 32 e + l), so that a
 * warp reads one line per step and its lanes have (nearly) the same number
 * of steps.  The records of a CTA start at its partition's first slot, its
 * items where the lower ranks' end; they depend on the cluster size, which
 * RepDyn::near_C remembers, and are built again when a launch uses another.
 * The other molecules' slots follow in far_list, ascending.  Built at a
 * rebuild (every few hundred steps); all threads of the cluster. */
__device__ __forceinline__ void build_near(Ctx& x, cg::cluster_group& cl) {
  const RepParams* P = x.P;
  const KArgs* a = x.a;
  const int par = x.D->parity, ni = P->n_ion, av = P->a_v, nj = gv_reach(P);
  int lo, hi;
  slab_part(x, &lo, &hi);
  int* const hist = x.cand;        /* [kNearBins + 1] molecules per bin, then first record */
  int* const cur = x.cand + 64;    /* [kNearBins] next record                              */
  int* const heavy = x.cand + 128; /* partners of all heavy molecules, and the next one    */
  __syncthreads();
  if (threadIdx.x < kNearBins / 2) hist[threadIdx.x] = hist[kNearBins / 2 + threadIdx.x] = 0; /* a block may be one warp */
  if (threadIdx.x < 2) heavy[threadIdx.x] = 0;
  __syncthreads();
  auto items_of = [&](size_t ms) {
    return a->near_gi[ms] < 0 ? 0 : (int)a->gil_n[ms] + (int)a->gvl_n[ms] * nj;
  };
  for (int s = lo + (int)threadIdx.x; s < hi; s += blockDim.x) {
    const int c = items_of(gmol(P, par, s));
    if (c == 0) continue;
    atomicAdd(&hist[near_bin(c)], 1);
    if (c > kNearHeavy) atomicAdd(&heavy[0], c);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int run = 0, items = heavy[0], nh = 0;
    for (int b = 0; b < kNearBins; b++) {
      const int n = hist[b];
      hist[b] = cur[b] = run;
      if (b == kHeavyBins) nh = run;
      /* 32-record groups that start in this bin take its count of entries */
      if (b >= kHeavyBins)
        items += 32 * (kNearBins - b) * (((run + n - nh + 31) >> 5) - ((run - nh + 31) >> 5));
      run += n;
    }
    hist[kNearBins] = run;
    x.iscr[56] = nh;
    x.iscr[57] = run;
    heavy[2] = items;
    x.D->near_C = x.C;
  }
  __syncthreads();
  int base, tot;
  cluster_prefix(x, cl, &x.iscr[47], heavy[2], &base, &tot);
  const int nh = x.iscr[56], light0 = base + heavy[0];
  int4* const rec = a->near_rec + P->near_off + lo;
  unsigned short* const item = a->near_item + P->nit_off;
  int n_far = 0;
  for (int s0 = lo; s0 < hi; s0 += blockDim.x) {
    const int s = s0 + (int)threadIdx.x;
    const int f = s < hi && items_of(gmol(P, par, s)) == 0 ? 1 : 0;
    int t;
    const int o = block_exscan(f, x.iscr, &t);
    if (f) a->far_list[P->near_off + lo + n_far + o] = s;
    n_far += t;
  }
  if (threadIdx.x == 0) x.iscr[61] = n_far;
  for (int s = lo + (int)threadIdx.x; s < hi; s += blockDim.x) {
    const size_t ms = gmol(P, par, s);
    const int c = items_of(ms);
    if (c == 0) continue;
    int off, stride;
    if (c > kNearHeavy) {
      rec[atomicAdd(&cur[near_bin(c)], 1)] = make_int4(s, off = base + atomicAdd(&heavy[1], c), c, 0);
      stride = 1;
    } else {
      const int r = atomicAdd(&cur[near_bin(c)], 1), k = r - nh, g0 = k & ~31;
      off = light0 + (k & 31);
      for (int b = kHeavyBins; b < kNearBins; b++) { /* the groups before this one */
        const int s0 = min(hist[b] - nh, g0), s1 = min(hist[b + 1] - nh, g0);
        off += 32 * (kNearBins - b) * (((s1 + 31) >> 5) - ((s0 + 31) >> 5));
      }
      rec[r] = make_int4(s, off, c, 0);
      stride = 32;
    }
    const unsigned short* g = a->gil + P->gil_off + a->near_gi[ms];
    for (int q = 0; q < (int)a->gil_n[ms]; q++, off += stride) item[off] = g[q];
    const unsigned short* v = a->gvl + P->gvl_off + a->near_gv[ms];
    for (int q = 0; q < (int)a->gvl_n[ms]; q++)
      for (int b = 0; b < nj; b++, off += stride) item[off] = (unsigned short)(ni + (int)v[q] * av + b);
  }
  __syncthreads();
}

template <int AG, bool OUT>
__device__ __forceinline__ void near_copy_t(Ctx& x) {
  const RepParams* P = x.P;
  const KArgs* a = x.a;
  const int par = x.D->parity, nn = x.iscr[57];
  int lo, hi;
  slab_part(x, &lo, &hi);
  double* const base = near_base(x);
  for (int k = threadIdx.x; k < nn; k += blockDim.x) {
    const size_t g0 = 3 * gatom(P, par, a->near_rec[P->near_off + lo + k].x, 0);
    double* const S = near_at<AG>(base, near_row(x, k));
#pragma unroll
    for (int q = 0; q < 3 * AG; q++) {
      if (OUT) {
        a->slab_x[g0 + q] = S[32 * q];
        a->slab_v[g0 + q] = S[32 * (q + 3 * AG)];
        a->slab_f[g0 + q] = S[32 * (q + 6 * AG)];
      } else {
        S[32 * q] = a->slab_x[g0 + q];
        S[32 * (q + 3 * AG)] = a->slab_v[g0 + q];
        S[32 * (q + 6 * AG)] = a->slab_f[g0 + q];
      }
    }
  }
}
template <bool OUT>
__device__ __forceinline__ void near_copy(Ctx& x) {
  if constexpr (kGG) return;
  if (x.P->a_g == 1) near_copy_t<1, OUT>(x);
  else near_copy_t<2, OUT>(x);
}

/* One group of near molecules, one lane each: records first .. first + n.
 * Light molecules' lanes walk their own partners (lg = 0).  Heavy ones
 * (30-100 partners next to a large ion) are walked by 2^lg lanes each, the
 * lanes' sums added by shuffles and handed to the molecule's own lane, which
 * then finishes it like a light one: force, gas-gas and intramolecular terms,
 * second kick.  With `drift` the molecule's first kick and drift come first,
 * in the same registers: its slab rows are read and written once per step.  The reactions go to the core sums by
 * shared 32-bit integer atomics on exact chunks (acc_add); all sums are
 * integers, so neither the split nor the order changes the result. */
template <int AG, bool FP64, bool E>
__device__ __forceinline__ void near_group(Ctx& x, int first, int n, int lg, bool kick, bool drift) {
  const RepParams* P = x.P;
  const KArgs* a = x.a;
  const bool gi = term_on(x, MDN_I_GI), gv = term_on(x, MDN_I_GV);
  int gtype[AG];
#pragma unroll
  for (int at = 0; at < AG; at++) gtype[at] = x.iscr[58 + at];
  long long egi = 0, egv = 0, eintra = 0;
  const int par = x.D->parity, ni = P->n_ion;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const double* com = x.D->ion_com;
  const unsigned short* const item = a->near_item + P->nit_off;
  const bool own = lane < n;
  int lo, hi;
  slab_part(x, &lo, &hi);
  const int4 rc = own ? a->near_rec[P->near_off + lo + first + lane] : make_int4(0, 0, 0, 0);
  const NearRow S = near_ref<AG>(x, first + (own ? lane : 0), rc.x);
  double X[3 * AG], V[3 * AG];
  float3 gp[AG];
#pragma unroll
  for (int q = 0; q < 3 * AG; q++) {
    X[q] = S.x(q);
    V[q] = S.v(q);
  }
  if (drift) { /* a rigid gas was drifted before */
#pragma unroll
    for (int q = 0; q < 3 * AG; q++) {
      V[q] += S.f(q) * x.c.c2[gtype[q / 3]];
      X[q] = X[q] + V[q] * P->dt;
    }
    gas_finite<AG>(x, X, V);
  }
#pragma unroll
  for (int at = 0; at < AG; at++)
    gp[at] = make_float3((float)(X[3 * at] - com[0]), (float)(X[3 * at + 1] - com[1]),
                         (float)(X[3 * at + 2] - com[2]));
  long long F[AG][3];
#pragma unroll
  for (int at = 0; at < AG; at++) F[at][0] = F[at][1] = F[at][2] = 0;
  if (lg > 0) {
    const int per = 32 >> lg, sub = (1 << lg) - 1; /* molecules a round, lane's place in its molecule */
    for (int r = 0; r < n; r += per) {
      const int src = r + (lane >> lg);
      const int cnt = __shfl_sync(FULL, rc.z, src), off = __shfl_sync(FULL, rc.y, src);
      float3 gpo[AG];
      double Xo[3 * AG];
      long long Fo[AG][3];
#pragma unroll
      for (int at = 0; at < AG; at++) {
        gpo[at] = make_float3(__shfl_sync(FULL, gp[at].x, src), __shfl_sync(FULL, gp[at].y, src),
                              __shfl_sync(FULL, gp[at].z, src));
        Fo[at][0] = Fo[at][1] = Fo[at][2] = 0;
#pragma unroll
        for (int k = 0; k < 3; k++) Xo[3 * at + k] = FP64 || E ? __shfl_sync(FULL, X[3 * at + k], src) : 0.0;
      }
      for (int q = lane & sub; q < cnt; q += sub + 1) {
        const int j = item[off + q];
        const bool ion = j < ni;
        if (ion ? gi : gv) near_partner<AG, FP64>(x, Xo, gpo, gtype, j, E, Fo, ion ? egi : egv);
      }
#pragma unroll
      for (int at = 0; at < AG; at++)
#pragma unroll
        for (int k = 0; k < 3; k++) {
          long long v = Fo[at][k];
          for (int m = (sub + 1) >> 1; m; m >>= 1) v += shfl_xor_ll(v, m);
          v = __shfl_sync(FULL, v, (lane & (per - 1)) << lg);
          if (lane >= r && lane < r + per) F[at][k] = v;
        }
    }
  } else {
    for (int q = 0; q < rc.z; q++) {
      const int j = item[rc.y + 32 * q];
      const bool ion = j < ni;
      if (ion ? gi : gv) near_partner<AG, FP64>(x, X, gp, gtype, j, E, F, ion ? egi : egv);
    }
  }
  if (own) {
    double Fd[3 * AG];
#pragma unroll
    for (int q = 0; q < 3 * AG; q++) {
      Fd[q] = (double)F[q / 3][q % 3] * MDN_FIX_INV;
      if (!(fabs(Fd[q]) < MDN_FIX_LIMIT)) set_status(x, MDN_ST_FIXED_OVERFLOW);
    }
    if (kGG && term_on(x, MDN_I_GG) && P->ggl_cap > 0)
#pragma unroll
      for (int q = 0; q < 3 * AG; q++) Fd[q] += a->slab_fgg[3 * gatom(P, par, rc.x, 0) + q];
    if (term_on(x, MDN_I_GAS_INTRA) && P->n_gas_bonds > 0) {
      const double ei = gas_intra<AG>(x, X, Fd);
      if (E) eintra = efixd(ei);
    }
#pragma unroll
    for (int q = 0; q < 3 * AG; q++) {
      if (drift) S.x(q) = X[q];
      if (kick) S.v(q) = V[q] + Fd[q] * x.c.c2[gtype[q / 3]];
      S.f(q) = Fd[q];
    }
  }
  if (E) {
    egi = warp_sum_ll(egi);
    egv = warp_sum_ll(egv);
    eintra = warp_sum_ll(eintra);
    if (lane == 0) {
      energy_add(x, MDN_U_GI, egi);
      energy_add(x, MDN_U_VG, egv);
      energy_add(x, MDN_U_GAS, eintra);
    }
  }
}

/* How a CTA's nh heavy molecules are cut into groups: one at a time walked by
 * the whole warp while there are up to four per warp, then two, and at most
 * four, by 8 lanes each.  A group is one item of the queue, and the longest
 * lists have several hundred partners: with up to 16 molecules to a group,
 * in no order, the pass waited for the longest groups (641 heavy molecules
 * with 65 partners on average, one CTA: 269 of 396 thousand cycles). */
__device__ __forceinline__ void heavy_cut(int nh, int* size, int* lg) {
  const int nw = blockDim.x >> 5;
  const int h = min(4, max(1, (nh + 4 * nw - 1) / (4 * nw)));
  *size = h;
  *lg = h == 1 ? 5 : h == 2 ? 4 : 3;
}

/* Waits until every CTA of the cluster has read this one's sums, if that
 * has not been waited for: before they are written again, and before any
 * other barrier of the cluster. */
__device__ __forceinline__ void settle(Ctx& x) {
  if (!x.settled) {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    x.settled = true;
  }
}

/* The sums of the core over the cluster as forces, identical in every CTA,
 * and the second kick (with `cool`, the thermostat's factor on the ion
 * too).  Each thread keeps to its own components, so what follows up to the next
 * drift needs no barrier; and between two CTAs the wait for the other to have
 * read this one's sums is left to the next evaluation (settle), by when it
 * has. */
__device__ __forceinline__ void core_reduce_kick(Ctx& x, bool kick, bool cool) {
  const RepParams* P = x.P;
  long long* const mine = x.c.acc;
  const bool one = x.C == 1;
  settle(x);
  /* fold the chunk sums into 64-bit sums and clear them for the next
   * evaluation */
  const int n3 = 3 * x.n_core;
  for (int q = threadIdx.x; q < n3; q += blockDim.x) {
    unsigned* c = x.c.chunk + 3 * q;
    const unsigned long long s =
        (unsigned long long)c[0] + ((unsigned long long)c[1] << 16) + ((unsigned long long)c[2] << 32);
    c[0] = c[1] = c[2] = 0;
    mine[q] = (long long)s;
  }
  const unsigned at = (unsigned)__cvta_generic_to_shared(mine);
  auto peer = [&](int q, int r) { /* element q of CTA r */
    unsigned far;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(far) : "r"(at + 8 * q), "r"(r));
    return far;
  };
  auto meet = [&]() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  };
  /* Two CTAs read each other's sums.  More of them sum a slice each and write
   * it back to all, which costs a second meeting but moves 2 n3 elements per
   * CTA and not C n3: between 8 CTAs the plain form took 8.0 of 59 thousand
   * cycles a step for 500 atoms, 11.4 of 130 for 790. */
  const bool slices = x.C > 2;
  if (!one) meet();
  if (slices) {
    const int q0 = n3 * x.rank / x.C, q1 = n3 * (x.rank + 1) / x.C;
    for (int q = q0 + (int)threadIdx.x; q < q1; q += blockDim.x) {
      long long s = 0;
#pragma unroll 8
      for (int r = 0; r < x.C; r++) {
        long long v;
        asm volatile("ld.shared::cluster.s64 %0, [%1];" : "=l"(v) : "r"(peer(q, r)));
        s += v;
      }
#pragma unroll 8
      for (int r = 0; r < x.C; r++) asm volatile("st.shared::cluster.s64 [%0], %1;" ::"r"(peer(q, r)), "l"(s) : "memory");
    }
    meet();
  }
  if (threadIdx.x == 0) x.iscr[62] = 0; /* the constraints' failure marks */
  const double coeff = cool ? exp(-x.D->zeta * 0.5 * P->dt) : 1.0;
  for (int q = threadIdx.x; q < n3; q += blockDim.x) {
    long long s = mine[q];
    if (x.C == 2) {
      long long v;
      asm volatile("ld.shared::cluster.s64 %0, [%1];" : "=l"(v) : "r"(peer(q, x.rank ^ 1)));
      s += v;
    }
    const double f = (double)s * MDN_FIX_INV;
    double v = x.c.v[q];
    x.c.f[q] = f;
    /* flag saturated forces, and positions that are no longer finite */
    if (x.rank == 0) {
      if (!(fabs(f) < MDN_FIX_LIMIT)) set_status(x, MDN_ST_FIXED_OVERFLOW);
      if (!isfinite(x.c.x[q] + v)) set_status(x, MDN_ST_NONFINITE);
    }
    if (kick) {
      v += f * core_c2(x, q);
      if (cool && q < 3 * P->n_ion) v *= coeff;
      x.c.v[q] = v;
    }
  }
  if (x.C == 2) {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    x.settled = false;
  }
}

/* All forces of the step (after positions and lists are final) as one queue
 * of warp-sized items: 32 bonded terms, a core pair tile, a group of near
 * molecules.  They all add integers to the core sums, so they need no order
 * and no barrier among them; a warp takes its next item from a shared
 * counter, so that the CTA waits for its slowest warp once per step and not
 * once per kind.  The long items come first (the FP64 bonded terms, the
 * tiles, the heavy and then ever lighter near groups).  Bonded terms and
 * tiles are dealt to the cluster's CTAs in turn; near groups belong to the
 * CTA of their slab partition.  With the cycle accounting on, the kinds run
 * one after another, each with its own barrier. */
template <bool E>
__device__ __forceinline__ void force_items(Ctx& x, bool kick, bool drift) {
  const RepParams* P = x.P;
  const int nw = blockDim.x >> 5, lane = threadIdx.x & 31;
  const bool pairs = term_on(x, MDN_I_AMBER) || term_on(x, MDN_I_BMH) || term_on(x, MDN_I_VI) || term_on(x, MDN_I_VV);
  const BondedCount bc = bonded_count(x);
  const int nblk = pairs ? (x.n_core + 31) >> 5 : 0;
  const int field = term_on(x, MDN_I_EFIELD) ? 1 : 0;
  const int n_bond = field + ((bc.total() + 31) >> 5), n_tile = nblk * (nblk + 1) / 2;
  const int nh = x.iscr[56], nn = x.iscr[57];
  int hs, lg;
  heavy_cut(nh, &hs, &lg);
  const int gh = (nh + hs - 1) / hs;
  /* this CTA's items: bonded and tiles g = rank, rank + C, ..., then near */
  const int mb = (n_bond - x.rank + x.C - 1) / x.C, mc = (n_bond + n_tile - x.rank + x.C - 1) / x.C;
  const int total = mc + gh + ((nn - nh + 31) >> 5);
  const bool prof = x.a->prof != nullptr;
  for (int ph = 0; ph < (prof ? 3 : 1); ph++) {
    int first = 0, last = total;
    if (prof) {
      first = ph == 0 ? mc : ph == 1 ? 0 : mb;
      last = ph == 0 ? total : ph == 1 ? mb : mc;
      __syncthreads();
      prof_start(x);
      if (threadIdx.x == 0) x.iscr[60] = nw;
      __syncthreads();
    }
    for (int it = first + (int)(threadIdx.x >> 5); it < last;) {
      if (it < mb) {
        const int g = x.rank + it * x.C;
        if (g < field) field_terms(x);
        else bonded_terms<E>(x, bc, g - field);
      } else if (it < mc) {
        core_tile<kFP64Pairs, E>(x, x.rank + it * x.C - n_bond, nblk);
      } else {
        const int k = it - mc;
        const bool heavy = k < gh;
        const int f = heavy ? k * hs : nh + 32 * (k - gh), n = heavy ? min(hs, nh - f) : min(32, nn - f);
        if (P->a_g == 1) near_group<1, kFP64Pairs, E>(x, f, n, heavy ? lg : 0, kick, drift);
        else near_group<2, kFP64Pairs, E>(x, f, n, heavy ? lg : 0, kick, drift);
      }
      int next = 0;
      if (lane == 0) next = atomicAdd(&x.iscr[60], 1);
      it = first + __shfl_sync(0xffffffffu, next, 0);
    }
    if (prof) {
      __syncthreads();
      prof_end(x, ph == 0 ? MDN_PROF_NEAR : ph == 1 ? MDN_PROF_BONDED : MDN_PROF_PAIRS);
    }
  }
}

/* ------------------------------------------------------------------------- */
/* the effective-domain rebuild (MD::make_pair)                               */
/* ------------------------------------------------------------------------- */
/* Philox word of insertion draw `t` (word 1 is the N2 spin) */
__device__ __forceinline__ int insert_word(int t) { return t == 0 ? 0 : 1 + t; }

__device__ __forceinline__ void insert_vapor(const Ctx& x, int q, int n_rebuild, int t, double* X, double* V);

/* true when no atom of X[0..n) lies within MDN_INSERT_MIN_DIST of a core atom
 * (ion, vapor in the domain before this rebuild) or of a vapor molecule whose
 * entry this rebuild already accepted; with the gas-gas term on, nor of a gas
 * atom in the domain before this rebuild (gas molecules entering in the same
 * rebuild are not tested against each other).  One warp, X in every lane. */
__device__ __forceinline__ bool insert_clear(const Ctx& x, const double* X, int n, int n_rebuild) {
  const double d2min = MDN_INSERT_MIN_DIST * MDN_INSERT_MIN_DIST;
  const int lane = threadIdx.x & 31;
  bool clash = false;
  auto test = [&](double c0, double c1, double c2) {
    for (int a = 0; a < n; a++) {
      double dx = X[3 * a] - c0, dy = X[3 * a + 1] - c1, dz = X[3 * a + 2] - c2;
      if (dx * dx + dy * dy + dz * dz < d2min) clash = true;
    }
  };
  for (int i = lane; i < x.n_core; i += 32) test(x.c.x[3 * i], x.c.x[3 * i + 1], x.c.x[3 * i + 2]);
  const int nc = min(x.cand[MDN_INSERT_MAX_VAPOR], MDN_INSERT_MAX_VAPOR);
#pragma unroll 1
  for (int k = lane; k < nc; k += 32) {
    const int mi = x.cand[k];
    const int f = x.a->region[(size_t)x.P->mol_off + mi];
    if (!(f & 1)) continue;
    double Xv[3 * MDN_MAX_VAP_ATOMS], Vv[3 * MDN_MAX_VAP_ATOMS];
    insert_vapor(x, mi - 1 - x.P->n_gas, n_rebuild, f >> 2, Xv, Vv);
    for (int b = 0; b < x.P->a_v; b++) test(Xv[3 * b], Xv[3 * b + 1], Xv[3 * b + 2]);
  }
  if (kGG && (x.P->interactions & MDN_I_GG)) {
    const RepParams* P = x.P;
    const int G = x.D->n_gas_in, par = x.D->parity;
    for (int u = lane; u < G * P->a_g; u += 32) {
      const double* gpos = x.a->slab_x + 3 * ((size_t)P->slab_off + (size_t)par * P->slab_cap * P->a_g + u);
      test(__ldcg(gpos), __ldcg(gpos + 1), __ldcg(gpos + 2));
    }
  }
  return !__any_sync(0xffffffffu, clash);
}

__device__ __forceinline__ void insert_gas(const Ctx& x, int q, int n_rebuild, int t, double* X, double* V) {
  const RepParams* P = x.P;
  const int ag = P->a_g, mi = 1 + q;
  const double* cx = x.a->mol_x + 3 * ((size_t)P->mol_off + mi);
  const double* cv = x.a->mol_v + 3 * ((size_t)P->mol_off + mi);
  for (int at = 0; at < ag; at++)
    for (int k = 0; k < 3; k++) {
      X[3 * at + k] = x.db[P->d_gas_x + 3 * at + k];
      V[3 * at + k] = 0;
    }
  if (P->gas_kind == MDN_GAS_N2 && ag == 2) {
    U4 s = draw(*P, mi, n_rebuild, 1, 1);
    double vy, vz;
    box_muller(s.v[0], s.v[1], vy, vz);
    vy *= P->gas_sigma;
    vz *= P->gas_sigma;
    double vzu = (P->quirks & MDN_Q_N2_ROT_VYVZ) ? vy : vz;
    V[0] = 0; V[1] = vy; V[2] = vzu;
    V[3] = 0; V[4] = -vy; V[5] = -vzu;
  }
  U4 s = draw(*P, mi, n_rebuild, 1, insert_word(t));
  double A = u01(s.v[0]) * 2 * 3.141592653589793;
  double B = u01(s.v[1]) * 2 * 3.141592653589793;
  double Cc = u01(s.v[2]) * 2 * 3.141592653589793;
  const bool zy = (P->quirks & MDN_Q_GAS_ROT_ZY) != 0;
  for (int at = 0; at < ag; at++) {
    double* p = X + 3 * at;
    rotation(p[0], p[1], p[2], A, B, Cc, p[0], p[1], zy ? p[1] : p[2]);
    for (int k = 0; k < 3; k++) p[k] += cx[k];
  }
  for (int at = 0; at < ag; at++) {
    double* p = V + 3 * at;
    rotation(p[0], p[1], p[2], A, B, Cc, p[0], p[1], zy ? p[1] : p[2]);
    for (int k = 0; k < 3; k++) p[k] += cv[k];
  }
}

__device__ __forceinline__ void insert_vapor(const Ctx& x, int q, int n_rebuild, int t, double* X, double* V) {
  const RepParams* P = x.P;
  const int av = P->a_v, mi = 1 + P->n_gas + q;
  const double* cx = x.a->mol_x + 3 * ((size_t)P->mol_off + mi);
  const double* cv = x.a->mol_v + 3 * ((size_t)P->mol_off + mi);
  U4 s = draw(*P, mi, n_rebuild, 1, insert_word(t));
  double A = u01(s.v[0]) * 2 * 3.141592653589793;
  double B = u01(s.v[1]) * 2 * 3.141592653589793;
  double Cc = u01(s.v[2]) * 2 * 3.141592653589793;
  for (int at = 0; at < av; at++) {
    double* p = X + 3 * at;
    for (int k = 0; k < 3; k++) p[k] = x.db[P->d_vap_x + 3 * at + k];
    rotation(p[0], p[1], p[2], A, B, Cc, p[0], p[1], p[2]);
    for (int k = 0; k < 3; k++) p[k] += cx[k];
    double* u = V + 3 * at;
    u[0] = u[1] = u[2] = 0;
    rotation(u[0], u[1], u[2], A, B, Cc, u[0], u[1], u[2]);
    for (int k = 0; k < 3; k++) u[k] += cv[k];
  }
}

/* free flight, in/out test, wrap and resampling of one molecule; returns
 * (was_in << 1) | now_in.  Unless MDN_Q_BLIND_INSERT is set, entering
 * molecules become candidates: vapor ones that vapor_entries() decides,
 * provisionally in, and gas ones (into `entries`) that gas_entries() decides,
 * provisionally out.  A molecule inside the sphere whose draws all overlap
 * stays outside, unwrapped and not resampled, until the next rebuild. */
__device__ __forceinline__ int classify_one(const Ctx& x, int mi, double sigma, int n_rebuild, int loop_pair,
                                            const double* com, int kind /* 0 gas, 1 vapor */, int* entries) {
  const RepParams* P = x.P;
  const size_t g = (size_t)P->mol_off + mi;
  double* X = x.a->mol_x + 3 * g;
  double* V = x.a->mol_v + 3 * g;
  const int was = x.a->region[g] & 1;
  if (!was)
    for (int k = 0; k < 3; k++) X[k] += V[k] * P->dt * loop_pair;
  double dx = X[0] - com[0];
  double dy = X[1] - com[1];
  double dz = X[2] - com[2];
  double r2 = (dx * dx + dy * dy + dz * dz);
  int in = r2 < P->RI2 ? 1 : 0;
  if (in && !was && !(P->quirks & MDN_Q_BLIND_INSERT) && kind == 1) {
    /* decided by vapor_entries(): recorded as a candidate, provisionally in;
     * beyond MDN_INSERT_MAX_VAPOR candidates in one rebuild the entry waits
     * for the next */
    int c = atomicAdd(&x.cand[MDN_INSERT_MAX_VAPOR], 1);
    if (c >= MDN_INSERT_MAX_VAPOR) {
      x.a->region[g] = 0;
      return 0;
    }
    x.cand[c] = mi;
    x.a->region[g] = (unsigned char)1;
    return 1;
  }
  if (in && !was && !(P->quirks & MDN_Q_BLIND_INSERT)) {
    /* decided by gas_entries(), from this CTA's list */
    entries[atomicAdd(&x.iscr[50], 1)] = mi;
    x.a->region[g] = 0;
    return 0;
  }
  if (!in) {
    double HL = P->box * 0.5;
    if (dx < -HL) X[0] += P->box;
    if (dy < -HL) X[1] += P->box;
    if (dz < -HL) X[2] += P->box;
    if (dx > HL) X[0] -= P->box;
    if (dy > HL) X[1] -= P->box;
    if (dz > HL) X[2] -= P->box;
    U4 s = draw(*P, mi, n_rebuild, 0, 0);
    double z0, z1, z2, z3;
    box_muller(s.v[0], s.v[1], z0, z1);
    box_muller(s.v[2], s.v[3], z2, z3);
    V[0] = z0 * sigma;
    V[1] = z1 * sigma;
    V[2] = z2 * sigma;
  }
  x.a->region[g] = (unsigned char)((was << 1) | in);
  return (was << 1) | in;
}

/* gas-gas pair list of the slab (PotentialGasGas::makePair,
 * src/potential/GasGas.cpp:41-62, on the in-domain molecules it was meant
 * for): every other slab molecule whose centre lies within the list radius,
 * both directions, ascending slab slot, CSR by slab slot over the cluster */
__device__ __forceinline__ void relist_gg(Ctx& x, cg::cluster_group& cl) {
  const RepParams* P = x.P;
  const KArgs* a = x.a;
  const int par = x.D->parity, G = x.D->n_gas_in;
  int lo, hi;
  partition(x, G, &lo, &hi);
  const double* cen = a->mol_x + 3 * ((size_t)P->mol_off + 1);
  const int* smol = a->slab_mol + gmol(P, par, 0);
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  /* a warp per molecule: its lanes test 32 others at a time (centres and slab
   * entries of every CTA's molecules, from L2); returns the number of
   * partners, which go to out, ascending, when it is given */
  auto partners = [&](int s, int* out) {
    const double* c = cen + 3 * (size_t)__ldcg(smol + s);
    const double c0 = __ldcg(c), c1 = __ldcg(c + 1), c2 = __ldcg(c + 2);
    int n = 0;
#pragma unroll 4
    for (int t0 = 0; t0 < G; t0 += 32) {
      const int t = t0 + lane;
      bool in = false;
      if (t < G && t != s) {
        const double* d = cen + 3 * (size_t)__ldcg(smol + t);
        const double dx = c0 - __ldcg(d), dy = c1 - __ldcg(d + 1), dz = c2 - __ldcg(d + 2);
        in = (dx * dx + dy * dy + dz * dz) < P->ml2;
      }
      const unsigned m = __ballot_sync(0xffffffffu, in);
      if (in && out) out[n + __popc(m & ((1u << lane) - 1u))] = t;
      n += __popc(m);
    }
    return n;
  };
  /* counts, then starts (a prefix sum over the CTA's molecules), then lists */
  for (int s = lo + (int)(threadIdx.x >> 5); s < hi; s += nw) {
    const int c = partners(s, nullptr);
    if (lane == 0) a->ggl_n[gmol(P, par, s)] = c;
  }
  __syncthreads();
  int mine = 0;
  for (int s0 = lo; s0 < hi; s0 += blockDim.x) {
    const int s = s0 + (int)threadIdx.x;
    const int c = s < hi ? a->ggl_n[gmol(P, par, s)] : 0;
    int t;
    const int o = block_exscan(c, x.iscr, &t);
    if (s < hi) a->ggl_start[gmol(P, par, s)] = mine + o;
    mine += t;
  }
  int base, tot;
  cluster_prefix(x, cl, &x.iscr[46], mine, &base, &tot);
  const bool over = tot > P->ggl_cap;
  if (over && threadIdx.x == 0 && x.rank == 0) set_status(x, MDN_ST_LIST_OVERFLOW);
  for (int s = lo + (int)(threadIdx.x >> 5); s < hi; s += nw) {
    const size_t ms = gmol(P, par, s);
    const int start = over ? 0 : base + a->ggl_start[ms];
    if (!over) partners(s, a->ggl + P->ggl_off + start);
    __syncwarp();
    if (lane == 0) {
      a->ggl_start[ms] = start;
      if (over) a->ggl_n[ms] = 0;
    }
  }
  if (threadIdx.x == 0) x.D->gg_count = over ? 0 : tot / 2;
  __threadfence();
  cl.sync();
}

/* pair lists of the gas slab (current parity) from the centres: gas-ion
 * (PotentialGasIon::makePair) and gas-vapor (PotentialVaporGas::makePair) */
__device__ __forceinline__ void relist(Ctx& x, cg::cluster_group& cl) {
  const RepParams* P = x.P;
  const KArgs* a = x.a;
  const int par = x.D->parity, ni = P->n_ion, nv = x.D->n_vap_in;
  const bool gi = (P->interactions & MDN_I_GI) != 0, gv = (P->interactions & MDN_I_GV) != 0;
  int lo, hi;
  slab_part(x, &lo, &hi);
  int* sc = x.iscr;
  /* the vapor centres, from L2 (rank 0 set them), into the core's sum buffer,
   * which no CTA reads now: from global memory each test of a gas molecule
   * against them was two dependent loads */
  double* const sv = (double*)x.c.acc;
  if (gv)
    for (int q = threadIdx.x; q < 3 * nv; q += blockDim.x) {
      const int vm = __ldcg(a->vslab_mol + vmol(P, par, q / 3));
      sv[q] = __ldcg(a->mol_x + 3 * ((size_t)P->mol_off + 1 + P->n_gas + vm) + q % 3);
    }
  __syncthreads();
  int gi_tot = 0, gv_tot = 0, nn_tot = 0;
  int gi_base = 0, gv_base = 0, nn_before = 0;
  /* pass 1: counts */
  int my_gi = 0, my_gv = 0, my_nn = 0;
  for (int s0 = lo; s0 < hi; s0 += blockDim.x) {
    int s = s0 + threadIdx.x;
    int cgi = 0, cgv = 0;
    if (s < hi) {
      int m = __ldcg(a->slab_mol + gmol(P, par, s));
      const double* cm = a->mol_x + 3 * ((size_t)P->mol_off + 1 + m);
      /* centres set by whichever CTA classified the molecule: from L2 */
      const double cx0 = __ldcg(cm), cx1 = __ldcg(cm + 1), cx2 = __ldcg(cm + 2);
      if (gi)
        for (int j = 0; j < ni; j++) {
          double dx = cx0 - x.c.x[3 * j], dy = cx1 - x.c.x[3 * j + 1], dz = cx2 - x.c.x[3 * j + 2];
          if ((dx * dx + dy * dy + dz * dz) < P->ml2) cgi++;
        }
      if (gv)
        for (int q = 0; q < nv; q++) {
          double dx = cx0 - sv[3 * q], dy = cx1 - sv[3 * q + 1], dz = cx2 - sv[3 * q + 2];
          if ((dx * dx + dy * dy + dz * dz) < P->ml2) cgv++;
        }
    }
    my_gi += cgi;
    my_gv += cgv;
    my_nn += (cgi + cgv) > 0 ? 1 : 0;
  }
  my_gi = block_sum_i(my_gi, sc);
  my_gv = block_sum_i(my_gv, sc);
  my_nn = block_sum_i(my_nn, sc);
  cluster_prefix(x, cl, &sc[40], my_gi, &gi_base, &gi_tot);
  cluster_prefix(x, cl, &sc[41], my_gv, &gv_base, &gv_tot);
  cluster_prefix(x, cl, &sc[42], my_nn, &nn_before, &nn_tot);
  bool over = gi_tot > P->gil_cap || gv_tot > P->gvl_cap || nn_tot > P->near_cap;
  if (over && threadIdx.x == 0 && x.rank == 0) set_status(x, MDN_ST_LIST_OVERFLOW);
  /* pass 2: fill, ascending slab slot */
  int run_gi = gi_base, run_gv = gv_base;
  for (int s0 = lo; s0 < hi; s0 += blockDim.x) {
    int s = s0 + threadIdx.x;
    int cgi = 0, cgv = 0;
    const double* cm = nullptr;
    double cx0 = 0, cx1 = 0, cx2 = 0;
    if (s < hi) {
      int m = __ldcg(a->slab_mol + gmol(P, par, s));
      cm = a->mol_x + 3 * ((size_t)P->mol_off + 1 + m);
      cx0 = __ldcg(cm);
      cx1 = __ldcg(cm + 1);
      cx2 = __ldcg(cm + 2);
      if (gi)
        for (int j = 0; j < ni; j++) {
          double dx = cx0 - x.c.x[3 * j], dy = cx1 - x.c.x[3 * j + 1], dz = cx2 - x.c.x[3 * j + 2];
          if ((dx * dx + dy * dy + dz * dz) < P->ml2) cgi++;
        }
      if (gv)
        for (int q = 0; q < nv; q++) {
          double dx = cx0 - sv[3 * q], dy = cx1 - sv[3 * q + 1], dz = cx2 - sv[3 * q + 2];
          if ((dx * dx + dy * dy + dz * dz) < P->ml2) cgv++;
        }
    }
    int t_gi, t_gv;
    int o_gi = block_exscan(cgi, sc, &t_gi);
    int o_gv = block_exscan(cgv, sc, &t_gv);
    const bool isn = (cgi + cgv) > 0;
    if (s < hi) {
      size_t ms = gmol(P, par, s);
      if (isn && !over) {
        int bgi = run_gi + o_gi, bgv = run_gv + o_gv;
        a->near_gi[ms] = bgi;
        a->near_gv[ms] = bgv;
        a->gil_n[ms] = (unsigned short)cgi;
        a->gvl_n[ms] = (unsigned short)cgv;
        int w = 0;
        if (gi)
          for (int j = 0; j < ni; j++) {
            double dx = cx0 - x.c.x[3 * j], dy = cx1 - x.c.x[3 * j + 1], dz = cx2 - x.c.x[3 * j + 2];
            if ((dx * dx + dy * dy + dz * dz) < P->ml2) a->gil[P->gil_off + bgi + w++] = (unsigned short)j;
          }
        w = 0;
        if (gv)
          for (int q = 0; q < nv; q++) {
            double dx = cx0 - sv[3 * q], dy = cx1 - sv[3 * q + 1], dz = cx2 - sv[3 * q + 2];
            if ((dx * dx + dy * dy + dz * dz) < P->ml2) a->gvl[P->gvl_off + bgv + w++] = (unsigned short)q;
          }
      } else {
        a->near_gi[ms] = -1;
        a->near_gv[ms] = -1;
        a->gil_n[ms] = 0;
        a->gvl_n[ms] = 0;
      }
    }
    run_gi += t_gi;
    run_gv += t_gv;
  }
  if (threadIdx.x == 0) {
    x.D->gi_count = over ? 0 : gi_tot;
    x.D->gv_count = over ? 0 : gv_tot;
    x.D->n_near = over ? 0 : nn_tot;
  }
  __threadfence();
  cl.sync();
  build_near(x, cl);
  if (kGG && P->ggl_cap > 0 && (P->interactions & MDN_I_GG)) relist_gg(x, cl);
}

/* The overlap test of the gas molecules that enter at this rebuild, the CTA's
 * list of n: a warp each, the draws in the first lanes, each tested by the
 * whole warp against the core (a thread that tested its own molecule against
 * 800 core atoms held up the 31 others of its warp, one to three million
 * cycles per rebuild).  The region flag of an accepted one is (draw << 2) | 1;
 * returns how many this warp accepted, in its first lane. */
__device__ __forceinline__ int gas_entries(const Ctx& x, const int* entries, int n, int nreb) {
  const RepParams* P = x.P;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, ag = P->a_g;
  int taken = 0;
  for (int k = threadIdx.x >> 5; k < n; k += blockDim.x >> 5) {
    const int mi = entries[k];
    double Xt[3 * MDN_MAX_GAS_ATOMS], Vt[3 * MDN_MAX_GAS_ATOMS];
    for (int q = 0; q < 3 * MDN_MAX_GAS_ATOMS; q++) Xt[q] = 0.0;
    if (lane < MDN_INSERT_TRIES) insert_gas(x, mi - 1, nreb, lane, Xt, Vt);
    int ok = -1;
#pragma unroll 1
    for (int t = 0; t < MDN_INSERT_TRIES && ok < 0; t++) {
      double X[3 * MDN_MAX_GAS_ATOMS];
      for (int q = 0; q < 3 * MDN_MAX_GAS_ATOMS; q++) X[q] = __shfl_sync(FULL, Xt[q], t);
      if (insert_clear(x, X, ag, nreb)) ok = t;
    }
    if (lane == 0 && ok >= 0) {
      x.a->region[(size_t)P->mol_off + mi] = (unsigned char)((ok << 2) | 1);
      taken++;
    }
  }
  return taken;
}

/* The overlap test of entering vapor molecules: against the ion, the vapor
 * already in the domain and every in-domain gas atom (up to ~20,000), so the
 * whole block tests each candidate's draws.  Rank 0 only; returns the number
 * of entries that must wait. */
__device__ __forceinline__ int vapor_entries(Ctx& x, int nreb) {
  const RepParams* P = x.P;
  const KArgs* a = x.a;
  const int av = P->a_v, ag = P->a_g, par = x.D->parity, G = x.D->n_gas_in;
  const double d2min = MDN_INSERT_MIN_DIST * MDN_INSERT_MIN_DIST;
  const int nc = min(x.cand[MDN_INSERT_MAX_VAPOR], MDN_INSERT_MAX_VAPOR);
  int deferred = 0;
  for (int c = 0; c < nc; c++) {
    const int mi = x.cand[c];
    const int q = mi - 1 - P->n_gas;
    int t = 0;
    for (; t < MDN_INSERT_TRIES; t++) {
      if (threadIdx.x == 0) {
        double V[3 * MDN_MAX_VAP_ATOMS];
        insert_vapor(x, q, nreb, t, x.trial, V);
        x.iscr[51] = 1;
      }
      __syncthreads();
      bool clash = false;
      for (int i = threadIdx.x; i < x.n_core && !clash; i += blockDim.x) {
        const double* cpos = x.c.x + 3 * i;
        for (int k = 0; k < av; k++) {
          double dx = x.trial[3 * k] - cpos[0], dy = x.trial[3 * k + 1] - cpos[1], dz = x.trial[3 * k + 2] - cpos[2];
          if (dx * dx + dy * dy + dz * dz < d2min) clash = true;
        }
      }
      for (int u = threadIdx.x; u < G * ag && !clash; u += blockDim.x) {
        const double* gp = a->slab_x + 3 * ((size_t)P->slab_off + (size_t)par * P->slab_cap * ag + u);
        const double g0 = __ldcg(gp), g1 = __ldcg(gp + 1), g2 = __ldcg(gp + 2);  /* moved this step by any CTA */
        for (int k = 0; k < av; k++) {
          double dx = x.trial[3 * k] - g0, dy = x.trial[3 * k + 1] - g1, dz = x.trial[3 * k + 2] - g2;
          if (dx * dx + dy * dy + dz * dz < d2min) clash = true;
        }
      }
      if (clash) x.iscr[51] = 0;
      __syncthreads();
      int ok = x.iscr[51];
      __syncthreads();
      if (ok) break;
    }
    if (threadIdx.x == 0) {
      size_t g = (size_t)P->mol_off + mi;
      if (t == MDN_INSERT_TRIES) {
        a->region[g] = 0; /* the entry waits for the next rebuild */
        deferred++;
      } else {
        a->region[g] = (unsigned char)((t << 2) | 1);
      }
    }
  }
  if (threadIdx.x == 0) x.iscr[52] = deferred;
  __syncthreads();
  int d = x.iscr[52];
  __syncthreads();
  return d;
}

__device__ __forceinline__ void make_pair(Ctx& x, cg::cluster_group& cl) {
  const RepParams* P = x.P;
  const KArgs* a = x.a;
  const int ag = P->a_g, av = P->a_v, par = x.D->parity, npar = par ^ 1;
  const int loop_pair = x.D->loop_pair, nreb = x.D->n_rebuilds;
  int* sc = x.iscr;
  /* updateInCenters: gas slab partition of this CTA, vapor core by rank 0 */
  {
    int lo, hi;
    slab_part(x, &lo, &hi);
    for (int s = lo + threadIdx.x; s < hi; s += blockDim.x) {
      int m = a->slab_mol[gmol(P, par, s)];
      double sx[3] = {0, 0, 0}, sv[3] = {0, 0, 0};
      for (int at = 0; at < ag; at++) {
        size_t g = gatom(P, par, s, at);
        double mm = x.db[P->d_mass + x.ib[P->o_gas_type + at]];
        for (int k = 0; k < 3; k++) {
          sx[k] += a->slab_x[3 * g + k] * mm;
          sv[k] += a->slab_v[3 * g + k] * mm;
        }
      }
      double massInv = 1 / P->gas_com_mass;
      size_t g = (size_t)P->mol_off + 1 + m;
      for (int k = 0; k < 3; k++) {
        a->mol_x[3 * g + k] = sx[k] * massInv;
        a->mol_v[3 * g + k] = sv[k] * massInv;
      }
    }
    if (x.rank == 0)
      for (int s = threadIdx.x; s < x.D->n_vap_in; s += blockDim.x) {
        int m = a->vslab_mol[vmol(P, par, s)];
        double sx[3] = {0, 0, 0}, sv[3] = {0, 0, 0};
        for (int at = 0; at < av; at++) {
          int i = P->n_ion + s * av + at;
          double mm = x.c.mass[tag_type(x.c.tag[i].k)];
          for (int k = 0; k < 3; k++) {
            sx[k] += x.c.x[3 * i + k] * mm;
            sv[k] += x.c.v[3 * i + k] * mm;
          }
        }
        double massInv = 1 / P->vap_com_mass;
        size_t g = (size_t)P->mol_off + 1 + P->n_gas + m;
        for (int k = 0; k < 3; k++) {
          a->mol_x[3 * g + k] = sx[k] * massInv;
          a->mol_v[3 * g + k] = sv[k] * massInv;
        }
      }
  }
  /* the ion centre in the reference's summation order (MD::update_position
   * computed it just before check_pairlist); MD::MD's first make_pair and the
   * re-centring in MD::run use the stored entry instead */
  if (!a->keep_com) ion_centre_exact(x);
  if (x.rank == 0 && threadIdx.x == 0) {
    size_t g = (size_t)P->mol_off;
    for (int k = 0; k < 3; k++) {
      a->mol_x[3 * g + k] = x.D->ion_com[k];
      a->mol_v[3 * g + k] = x.D->ion_com[3 + k];
    }
  }
  __threadfence();
  cl.sync();
  double com[3] = {x.D->ion_com[0], x.D->ion_com[1], x.D->ion_com[2]};
  int mlo, mhi;
  partition(x, P->n_gas, &mlo, &mhi);
  int my_in = 0;
  double vmax2 = 0;
  /* vapor molecules (rank 0; events) */
  int my_vin = 0;
  if (threadIdx.x == 0) {
    x.cand[MDN_INSERT_MAX_VAPOR] = 0;
    x.iscr[50] = 0;
  }
  __syncthreads();
  if (x.rank == 0)
    for (int q = threadIdx.x; q < P->n_vap; q += blockDim.x) {
      int mi = 1 + P->n_gas + q;
      size_t g = (size_t)P->mol_off + mi;
      int was = a->region[g] & 1;
      if (was) {
        /* MD::Ovin / MD::Ovout log the centre before any change */
        double dx[3], dv[3];
        for (int k = 0; k < 3; k++) {
          dx[k] = a->mol_x[3 * g + k] - com[k];
          dv[k] = a->mol_v[3 * g + k] - x.D->ion_com[3 + k];
        }
        double r2 = dx[0] * dx[0] + dx[1] * dx[1] + dx[2] * dx[2];
        int e = atomicAdd(a->n_events, 1);
        if (e < a->ev_cap) {
          DevEvent& ev = a->events[e];
          ev.replica = x.r;
          ev.molecule = q;
          ev.kind = r2 < P->RI2 ? 1 : 2;
          ev.step = x.D->step;
          for (int k = 0; k < 3; k++) { ev.dx[k] = dx[k]; ev.dv[k] = dv[k]; }
        } else {
          set_status(x, MDN_ST_EVENT_OVERFLOW);
        }
      }
      int f = classify_one(x, mi, P->vap_sigma, nreb, loop_pair, com, 1, nullptr);
      my_vin += f & 1;
      const double* V = a->mol_v + 3 * g;
      double v2 = V[0] * V[0] + V[1] * V[1] + V[2] * V[2];
      vmax2 = fmax(vmax2, v2);
    }
  /* the vapor decisions (and their accepted draws) before any gas entry is
   * tested against them: every CTA takes rank 0's candidate list */
  my_vin = block_sum_i(my_vin, sc);
  if (x.rank == 0 && !(P->quirks & MDN_Q_BLIND_INSERT)) my_vin -= vapor_entries(x, nreb);
  __threadfence();
  cl.sync();
  if (x.rank != 0) {
    for (int k = threadIdx.x; k <= MDN_INSERT_MAX_VAPOR; k += blockDim.x) x.cand[k] = *cl.map_shared_rank(&x.cand[k], 0);
  }
  __syncthreads();
  /* free flight + classification of the gas molecules of this CTA's range */
  int* const entries = a->entries + P->mol_off + 1 + mlo;
  for (int q = mlo + threadIdx.x; q < mhi; q += blockDim.x) {
    int f = classify_one(x, 1 + q, P->gas_sigma, nreb, loop_pair, com, 0, entries);
    my_in += f & 1;
    const double* V = a->mol_v + 3 * ((size_t)P->mol_off + 1 + q);
    double v2 = V[0] * V[0] + V[1] * V[1] + V[2] * V[2];
    vmax2 = fmax(vmax2, v2);
  }
  __syncthreads();
  my_in += gas_entries(x, entries, x.iscr[50], nreb);
  {
    const double* V = x.D->ion_com + 3;
    vmax2 = fmax(vmax2, V[0] * V[0] + V[1] * V[1] + V[2] * V[2]);
  }
  my_in = block_sum_i(my_in, sc);
  vmax2 = block_max_d(vmax2, x.dscr);
  __threadfence();
  int gin_base, gin_tot, vin_base, vin_tot;
  cluster_prefix(x, cl, &sc[43], my_in, &gin_base, &gin_tot);
  cluster_prefix(x, cl, &sc[44], my_vin, &vin_base, &vin_tot);
  /* vmax over the cluster */
  if (threadIdx.x == 0) x.dscr[45] = vmax2;
  cl.sync();
  double vm2 = 0;
  for (int k = 0; k < x.C; k++) vm2 = fmax(vm2, *cl.map_shared_rank(&x.dscr[45], k));
  cl.sync();
  const bool slab_over = gin_tot > P->slab_cap;
  const bool core_over = vin_tot > P->vcap || P->n_ion + vin_tot * av > a->nc_cap;
  /* new gas slab, ascending molecule index */
  int run = gin_base;
  for (int q0 = mlo; q0 < mhi; q0 += blockDim.x) {
    int q = q0 + threadIdx.x;
    int f = 0;
    if (q < mhi) f = a->region[(size_t)P->mol_off + 1 + q];
    int in = f & 1, tot;
    int off = block_exscan(in, sc, &tot);
    if (q < mhi) {
      size_t g = (size_t)P->mol_off + 1 + q;
      if (in && !slab_over) {
        int ns = run + off;
        double X[3 * MDN_MAX_GAS_ATOMS], V[3 * MDN_MAX_GAS_ATOMS];
        if (f & 2) {
          int os = a->slot[g];
          for (int at = 0; at < ag; at++) {
            size_t go = gatom(P, par, os, at);
            for (int k = 0; k < 3; k++) {
              /* the old slab slot may belong to another CTA, which moved
               * it this step: from L2 */
              X[3 * at + k] = __ldcg(a->slab_x + 3 * go + k);
              V[3 * at + k] = __ldcg(a->slab_v + 3 * go + k);
            }
          }
        } else {
          insert_gas(x, q, nreb, f >> 2, X, V);
        }
        for (int at = 0; at < ag; at++) {
          size_t gn = gatom(P, npar, ns, at);
          for (int k = 0; k < 3; k++) {
            a->slab_x[3 * gn + k] = X[3 * at + k];
            a->slab_v[3 * gn + k] = V[3 * at + k];
            a->slab_f[3 * gn + k] = 0.0;
          }
        }
        a->slab_mol[gmol(P, npar, ns)] = q;
        if (a->slab_ins) a->slab_ins[gmol(P, npar, ns)] = (f & 2) ? -1 : nreb + 1;
        a->slot[g] = ns;
      } else {
        a->slot[g] = -1;
      }
      a->region[g] = (unsigned char)in;
    }
    run += tot;
  }
  /* new vapor slab (rank 0), from the core copy (current positions); each
   * molecule reads its own old slot before overwriting it */
  if (x.rank == 0) {
    int runv = 0;
    for (int q0 = 0; q0 < P->n_vap; q0 += blockDim.x) {
      int q = q0 + threadIdx.x;
      int f = 0;
      if (q < P->n_vap) f = a->region[(size_t)P->mol_off + 1 + P->n_gas + q];
      int in = f & 1, tot;
      int off = block_exscan(in, sc, &tot);
      if (q < P->n_vap) {
        size_t g = (size_t)P->mol_off + 1 + P->n_gas + q;
        if (in && !core_over) {
          int ns = runv + off;
          double X[3 * MDN_MAX_VAP_ATOMS], V[3 * MDN_MAX_VAP_ATOMS];
          if (f & 2) {
            int os = a->slot[g];
            for (int at = 0; at < av; at++) {
              int i = P->n_ion + os * av + at;
              for (int k = 0; k < 3; k++) {
                X[3 * at + k] = x.c.x[3 * i + k];
                V[3 * at + k] = x.c.v[3 * i + k];
              }
            }
          } else {
            insert_vapor(x, q, nreb, f >> 2, X, V);
          }
          for (int at = 0; at < av; at++) {
            size_t gn = vatom(P, npar, ns, at);
            for (int k = 0; k < 3; k++) {
              a->vslab_x[3 * gn + k] = X[3 * at + k];
              a->vslab_v[3 * gn + k] = V[3 * at + k];
              a->vslab_f[3 * gn + k] = 0.0;
            }
            a->vslab_w[gn] = (f & 2) ? 0.0f : -1.0f;
          }
          a->vslab_mol[vmol(P, npar, ns)] = q;
          a->slot[g] = ns;
        } else {
          a->slot[g] = -1;
        }
        a->region[g] = (unsigned char)in;
      }
      runv += tot;
    }
  }
  __threadfence();
  cl.sync();
  /* new counters, identical in every CTA */
  if (threadIdx.x == 0) {
    if (slab_over && x.rank == 0) set_status(x, MDN_ST_SLAB_OVERFLOW);
    if (core_over && x.rank == 0) set_status(x, MDN_ST_CORE_OVERFLOW);
    x.D->parity = npar;
    x.D->n_gas_in = slab_over ? 0 : gin_tot;
    set_slab_part(x);
    x.D->n_vap_in = core_over ? 0 : vin_tot;
    double vmax = sqrt(vm2);
    double lu = x.D->margin_length / (vmax * P->dt);
    x.D->loop_update = lu >= 2147483647.0 ? 2147483647 : (int)lu;
    x.D->loop_pair = 0;
    x.D->n_rebuilds = nreb + 1;
  }
  __syncthreads();
  /* reload the vapor part of the core from the new vapor slab */
  load_vapor(x);
  __syncthreads();
  core_place(x, x.D->ion_com, true, CoreCons{false, 0});
}

/* ------------------------------------------------------------------------- */
/* what the launch is asked to do with a replica */
struct Turn {
  bool step, forces;  /* an MD step / the forces alone (else the rebuild or the lists alone) */
  bool rebuild, eflag, gg, last;
  bool far_done;      /* the far molecules have made this step (gas_far_steps) */
};

/* One step, or the part of it that the launch's mode asks for.  Between the
 * second kick of a step and the drift of the next each thread keeps to its
 * own components of the core, so a step has four block barriers: after the drift, the
 * constraints, the coordinates and the force items.  loop_pair is the
 * caller's copy of MD::loopPair. */
__device__ __forceinline__ void one_turn(Ctx& x, cg::cluster_group& cl, const Turn& t, int& loop_pair) {
  const RepParams* P = x.P;
  const int nvt = x.D->nvt_mode;
  prof_start(x);
  /* with gas-gas forces, and before a rebuild, every gas molecule is drifted
   * first; otherwise GasWork says where */
  const bool apart = t.rebuild || t.gg, fused = !apart && !gas_rigid(P) && x.iscr[57] > (int)blockDim.x;
  CoreCons cc = {false, 0};
  if (t.step) {
    if (t.rebuild) near_copy<true>(x); /* the rebuild reads the slab */
    loop_pair++;
    if (nvt == MDN_NVT_SCALE) {
      for (int q = threadIdx.x; q < 3 * x.n_core; q += blockDim.x) x.c.v[q] += x.c.f[q] * core_c2(x, q);
      __syncthreads();
      const double ratio = sqrt(300.0 / ion_temperature(x));
      for (int q = threadIdx.x; q < 3 * P->n_ion; q += blockDim.x) x.c.v[q] *= ratio;
    }
    core_drift(x, nvt != MDN_NVT_SCALE);
    __syncthreads();
    cc = core_cons(x);
    core_shake(x, cc, GasWork{apart, !apart && !t.far_done, !apart && !fused}, t.eflag);
  }
  if (t.step || t.forces) {
    double com[3];
    ion_centre(x, x.c.x, com);
    if (threadIdx.x == 0)
      for (int k = 0; k < 3; k++) x.D->ion_com[k] = com[k];
    if (P->quirks & MDN_Q_SHAKE_NO_VCORR) cc = CoreCons{false, 0};
    core_place(x, com, t.step, cc);
  }
  if (t.step && nvt == MDN_NVT_NH) {
    const double T = ion_temperature(x);
    if (threadIdx.x == 0) {
      int g = P->n_ion * 3;
      x.D->zeta += (T - x.D->nvt_T) * g * P->kb_real * 0.0001 * P->dt;
    }
    __syncthreads();
  }
  if (t.step && t.last && threadIdx.x < 32) {
    /* the ion centre's velocity, as MD::update_position leaves it */
    double vel[3];
    ion_centre(x, x.c.v, vel);
    if (threadIdx.x == 0)
      for (int k = 0; k < 3; k++) x.D->ion_com[3 + k] = vel[k];
  }
  prof_end(x, MDN_PROF_CORE_INT);
  if (t.rebuild) {
    prof_start(x);
    settle(x);
    if (threadIdx.x == 0 && t.step) x.D->loop_pair = loop_pair;
    __syncthreads();
    make_pair(x, cl);
    loop_pair = 0;
    prof_end(x, MDN_PROF_REBUILD);
  }
  if (t.rebuild || !(t.step || t.forces)) {
    settle(x);
    relist(x, cl);
  }
  if (!(t.step || t.forces)) return;
  if (t.gg) {
    settle(x);
    gas_gg_pass(x, cl, t.eflag, t.rebuild);
  }
  if (apart || t.forces) {
    prof_start(x);
    gas_far_pass(x, t.eflag, t.step);
    near_copy<false>(x);
    __syncthreads();
    prof_end(x, MDN_PROF_REBUILD);
  }
  if (t.eflag) force_items<true>(x, t.step, fused && t.step);
  else force_items<false>(x, t.step, fused && t.step);
  __syncthreads();
  if (t.forces) near_copy<true>(x);
  prof_start(x);
  core_reduce_kick(x, t.step, t.step && nvt == MDN_NVT_NH);
  prof_end(x, MDN_PROF_REDUCE);
  if (t.step && threadIdx.x == 0) x.D->step += 1;
}

}  // namespace

#if defined(MDN_GG_TERMS) && defined(MDN_FP64_PAIRS)
#define MDN_ADVANCE_KERNEL mdn_advance_gg_fp64
#elif defined(MDN_GG_TERMS)
#define MDN_ADVANCE_KERNEL mdn_advance_gg
#elif defined(MDN_FP64_PAIRS)
#define MDN_ADVANCE_KERNEL mdn_advance_fp64
#else
#define MDN_ADVANCE_KERNEL mdn_advance
#endif
extern "C" __global__ void __launch_bounds__(512, 1) MDN_ADVANCE_KERNEL(KArgs a) {
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ RepParams sP;
  __shared__ RepDyn sD;
  __shared__ int s_job;
  __shared__ int iscr[64];
  __shared__ double dscr[64];
  __shared__ int cand[MDN_INSERT_MAX_VAPOR + 1];
  __shared__ double trial[3 * MDN_MAX_VAP_ATOMS];

  Ctx x;
  x.a = &a;
  x.P = &sP;
  x.D = &sD;
  x.rank = (int)cl.block_rank();
  x.C = (int)cl.num_blocks();
  x.iscr = iscr;
  x.dscr = dscr;
  x.cand = cand;
  x.trial = trial;
  x.settled = true;
  /* carve the dynamic shared memory */
  {
    unsigned char* p = dsm;
    const int nc = a.nc_cap, nc32 = (nc + 31) & ~31;
    auto take = [&](size_t bytes) { unsigned char* q = p; p += (bytes + 15) & ~(size_t)15; return q; };
    x.c.acc = (long long*)take(sizeof(long long) * 3 * nc);
    x.c.chunk = (unsigned*)take(sizeof(unsigned) * 9 * nc);
    x.c.x = (double*)take(sizeof(double) * 3 * nc);
    x.c.v = (double*)take(sizeof(double) * 3 * nc);
    x.c.f = (double*)take(sizeof(double) * 3 * nc);
    x.c.pos = (float4*)take(sizeof(float4) * nc32);
    x.c.tag = (AtomTag*)take(sizeof(AtomTag) * nc32);
    x.c.excl = (unsigned*)take(sizeof(unsigned) * a.excl_cap);
    x.c.lj = (float2*)take(sizeof(float2) * a.nt_cap * a.nt_cap);
    x.c.c2 = (double*)take(sizeof(double) * a.nt_cap);
    x.c.mass = (double*)take(sizeof(double) * a.nt_cap);
  }
  /* the chunk sums start at zero and every core_reduce_kick leaves them so */
  for (int q = threadIdx.x; q < 9 * a.nc_cap; q += blockDim.x) x.c.chunk[q] = 0;
  if (threadIdx.x == 0) iscr[62] = 0;
  __syncthreads();
  for (;;) {
    if (x.rank == 0 && threadIdx.x == 0) s_job = (int)(atomicAdd(a.job_counter, 1u) - a.job_base);
    cl.sync();
    const int job = *cl.map_shared_rank(&s_job, 0);
    cl.sync();
    if (job >= a.n_jobs) break;
    const int r = a.job_order[job];
    x.r = r;
    if (threadIdx.x == 0) {
      sP = a.P[r];
      sD = a.D[r];
      sD.nvt_mode = a.ctl_mode[r];
      sD.nvt_T = a.ctl_T[r];
      set_slab_part(x);
    }
    __syncthreads();
    x.ib = a.iblob + sP.iblob_off;
    x.db = a.dblob + sP.dblob_off;
    const bool fatal = (a.status[r] & MDN_ST_FATAL) != 0;
    /* the CTAs of the cluster have to agree on it, or some would wait for ones
     * that skipped the replica: no CTA goes on to where it could set the status
     * before all have read it (the wait stands behind the loads) */
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    const bool fits = sP.n_types <= a.nt_cap && sP.n_ion * sP.excl_words <= a.excl_cap &&
                      sP.n_ion + sD.n_vap_in * sP.a_v <= a.nc_cap;
    /* the lists of an uploaded state are made even before its status is
     * cleared: the near records and their counts have to be of that state */
    if ((fatal && a.mode != MDN_MODE_RELIST) || !fits) {
      if (!fits && x.rank == 0 && threadIdx.x == 0) atomicOr(&a.status[r], MDN_ST_CORE_OVERFLOW);
      __syncthreads();
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      continue;
    }
    /* tables */
    const int nt = sP.n_types;
    for (int q = threadIdx.x; q < nt * nt; q += blockDim.x)
      x.c.lj[q] = make_float2((float)x.db[sP.d_ljA + q], (float)x.db[sP.d_ljB + q]);
    for (int q = threadIdx.x; q < nt; q += blockDim.x) {
      x.c.c2[q] = x.db[sP.d_c2 + q];
      x.c.mass[q] = x.db[sP.d_mass + q];
    }
    for (int q = threadIdx.x; q < sP.n_ion * sP.excl_words; q += blockDim.x) x.c.excl[q] = (unsigned)x.ib[sP.o_excl + q];
    load_ion(x);
    load_vapor(x);
    if (threadIdx.x < sP.a_g) iscr[58 + threadIdx.x] = x.ib[sP.o_gas_type + threadIdx.x];
    if (threadIdx.x < 3) /* build_near's counts; it makes them anew for another cluster size */
      iscr[threadIdx.x < 2 ? 56 + threadIdx.x : 61] = a.near_cnt[3 * ((size_t)r * 8 + x.rank) + threadIdx.x];
    if (threadIdx.x < MDN_PROF_N) s_prof[threadIdx.x] = 0;
    __syncthreads();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const long long job_t0 = clock64();
    if ((a.mode == MDN_MODE_STEP || a.mode == MDN_MODE_FORCES) && sD.near_C != x.C) build_near(x, cl);
    {
      Turn t;
      t.step = a.mode == MDN_MODE_STEP;
      t.forces = a.mode == MDN_MODE_FORCES;
      t.gg = kGG && (sP.interactions & MDN_I_GG) && sP.ggl_cap > 0;
      t.rebuild = a.mode == MDN_MODE_MAKE_PAIR;
      t.eflag = t.forces;
      t.far_done = t.last = false;
      int loop_pair = sD.loop_pair, loop_update = sD.loop_update;
      long long ahead = 0; /* steps the far molecules have already made */
      /* FORCES: the ion centre serves only as the origin of the FP32
       * coordinates, and the stored one is kept */
      double keep[3];
      for (int k = 0; k < 3; k++) keep[k] = sD.ion_com[k];
      __syncthreads();
      const long long n = t.step ? a.n_steps : 1;
      if (t.step) {
        near_copy<false>(x);
        __syncthreads();
      }
      for (long long s = 0; s < n; s++) {
        if (t.step) {
          t.last = s == n - 1;
          t.eflag = a.energy_mode == 2 || (a.energy_mode == 1 && t.last);
          t.rebuild = loop_pair + 1 > loop_update;
          if (t.rebuild || t.gg) {
            t.far_done = false;
          } else {
            if (ahead == 0 && (t.far_done = iscr[61] > (int)blockDim.x)) {
              ahead = min(n - s, (long long)loop_update - loop_pair);
              prof_start(x);
              gas_far_steps(x, ahead, a.energy_mode, s + ahead == n);
              prof_end(x, MDN_PROF_GAS_INT);
            }
            if (t.far_done) ahead--;
          }
        }
        one_turn(x, cl, t, loop_pair);
        if (t.rebuild) loop_update = sD.loop_update;
      }
      settle(x);
      if (t.step) near_copy<true>(x);
      __syncthreads();
      if (threadIdx.x == 0) {
        if (t.step) sD.loop_pair = loop_pair;
        if (t.forces)
          for (int k = 0; k < 3; k++) sD.ion_com[k] = keep[k];
      }
    }
    __syncthreads();
    if (a.prof && threadIdx.x == 0) {
      s_prof[MDN_PROF_TOTAL] = clock64() - job_t0;
      for (int k = 0; k < MDN_PROF_N; k++)
        atomicAdd((unsigned long long*)&a.prof[(size_t)r * MDN_PROF_N + k], (unsigned long long)s_prof[k]);
    }
    store_core(x);
    if (threadIdx.x < 3)
      a.near_cnt[3 * ((size_t)r * 8 + x.rank) + threadIdx.x] = iscr[threadIdx.x < 2 ? 56 + threadIdx.x : 61];
    __syncthreads();
    if (x.rank == 0 && threadIdx.x == 0) {
      a.D[r] = sD;
      if (a.mode == MDN_MODE_STEP) {
        size_t g = (size_t)sP.mol_off;
        for (int k = 0; k < 3; k++) {
          a.mol_x[3 * g + k] = sD.ion_com[k];
          a.mol_v[3 * g + k] = sD.ion_com[3 + k];
        }
      }
    }
    __threadfence();
    __syncthreads();
  }
}
