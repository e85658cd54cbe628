/*
 * gp_iface.cuh -- interface tiles of the time step, one TX x TY tile per CTA of
 * NTI threads.
 *
 * A tile's fields arrive as one TMA box (every phi and mu plane with a two-cell
 * halo) while the CTA works on the tile before it; tiles whose halo leaves the
 * domain are staged by plain loads through the boundary copy tables instead.
 * One pass over the ring cells (the tile plus a one-cell ring) finds the cells
 * whose 5-point phi stencil is not constant; only these can have an active phase,
 * and only faces next to them a current.  They go on lists, so that the long
 * arithmetic runs on dense warps wherever the interface crosses the tile:
 *   TEST   the cells to be tested for active phases
 *   TASK   (cell, active phase): lambda of one phase of one cell per thread
 *   LIST   cells with an active phase: the mean of lambda and the projection
 *   FLIST  the faces of those cells (anisotropy terms)
 *   JLIST  faces of the tile that may carry an anti-trapping current
 * The code of each pass is written for one phase (or pair) chosen at run time,
 * not unrolled over phases: an interface tile runs several thousand instructions
 * once per warp, and fetching them is part of its cost.
 *
 * What bounds it: the chains of dependent FP64 operations of one tile, and the
 * instructions fetched for them; DRAM moves 0.5 TB/s and the FP64 pipe is a
 * quarter busy.  Hence lists and short passes rather than long ones over every
 * cell, two CTAs of eight warps (four half tiles per SM stalled twice as long on
 * instruction fetches as the two whole ones), and in a batch of one the constants
 * in the kernel's parameters, where they are operands and not shared-memory loads.
 * Measured, all interface tiles of a step before and after (B200, FP64): 5034
 * tiles of a 4096^2 ternary three-phase grid 394 to 226 us; 1260 anisotropic ones
 * of a 2048^2 grid 155 to 100 us; 440 with a rotated pair and 1.5-spaced cells 150
 * to 77 us; 268 four-phase ones 58 to 41 us.
 * The arithmetic of each cell is the reference's, in its order (FP64; the FP32
 * form's tiles are in gp_iface32.cuh).  Terms of a
 * phase that is exactly zero over a stencil, and off-diagonal terms whose constants
 * are zero, are left out: each is +-0 added to a sum that starts at +0, as long as
 * its other factors are finite.  That is checked for a whole tile (tame): every phi
 * of its frame below PHI_TAME and every mu of its ring below MU_TAME, between
 * spacings of 2^-60 to 2^60, which keeps the eighth powers of the anisotropy and the
 * products of the free energies finite; a tile that fails takes every term.
 */
#pragma once
#include "gp_tiles.cuh"

namespace gpd {

constexpr double PHI_TAME = 16.0, MU_TAME = 1e18;
constexpr int NTI = NT;                                      /* threads of the step kernels' CTAs */
constexpr int FR = TX + 4, FC = TY + 4;                      /* staged frame: two-cell halo */
constexpr int RR = TX + 2, RC = TY + 2, RS = RR * RC;        /* ring region: one-cell halo */
constexpr int IXF = (TX + 3) * RC, IYF = RR * (TY + 3), IFT = IXF + IYF;   /* faces around the ring cells */
constexpr int JXF = (TX + 1) * TY, JYF = TX * (TY + 1), JFT = JXF + JYF;   /* faces of the tile's cells */

/* A frame row in shared memory: the box starts CO columns left of the frame so
 * that its first column is 16-byte aligned; BW columns are a multiple of 16 bytes. */
template <typename R>
struct ItemGeom {
  static constexpr int CO = sizeof(R) == 8 ? 0 : 2;
  static constexpr int BW = sizeof(R) == 8 ? FC : FC + 4;
};

/* shared memory of both precisions' interface tiles */
template <typename R, int N, int K>
struct alignas(128) ItemCommon {
  R F[2][N + K][FR][ItemGeom<R>::BW];   /* phi then mu; the tile in work and the next one */
  double ext[NTI / 32][2 * (N + K)];    /* per warp: running extremes of the simulation as the warp last saw them */
  unsigned long long bar[2];
  int4 ent[2];
  unsigned fm[2][TX];                   /* per tile row: flag bits of the new phi (row_flag_bits) */
  int row[2][FR], col[2][FC];           /* of phi and mu: the rows and columns that a frame's are copies of, or -1 */
};

template <typename R, int N, int K, bool ANISO>
struct ItemSmem : ItemCommon<R, N, K> {
  static constexpr int NPAIR = ANISO ? NP<N>::v : 1, NT_ = ANISO ? IFT : 1;
  R DP[N][RS];                          /* lambda of the active phases, then delta-phi */
  R SP[N - 1][RS];                      /* s_phi of the obstacle anti-trapping where 0 < phi < 1 (solid phases) */
  R DD[K][K][RS];                       /* D_kl */
  union {
    R T[NPAIR][2][NT_];                 /* anisotropy terms of the ring's faces: a_c^2 P and a_c |q|^2 dA/dq */
    R J[K][JFT];                        /* anti-trapping current of the listed faces */
  } w;
  unsigned long long JW[TX + 1 + TX];   /* per row of x- and y-faces: faces on JLIST */
  unsigned NU[RR], NUX;                 /* listed ring cells: columns 0..31 of each row, and columns 32 and 33 (two
                                           bits per row) */
  int n_test, n_act, n_task, n_extra, n_j;
  short TEST[RS], LIST[RS], TASK[N * RS], FLIST[IFT], JLIST[JFT];
  unsigned char ACT[RS];                /* active phases */
};

#define RI(i, j) ((i) * RC + (j))

template <typename R, int N, int K>
using ItemFrame = const R (&)[N + K][FR][ItemGeom<R>::BW];

/* c_a,i(mu), Mu_a,i(c) and f_a(c); dg: every off-diagonal constant is zero and
 * the operands are of ordinary size, so the off-diagonal terms are +-0 */
template <typename R, int K, typename CT>
__device__ __forceinline__ R c_mu_d(const CT &D, const R *m, int a, int i, bool dg) {
  R s = R(0.0);
#pragma unroll
  for (int k = 0; k < K; k++)
    if (k == i || !dg) s += D.cmu[a][i][k] * (m[k] - D.E[a][k]);
  return s;
}
template <typename R, int K, typename CT>
__device__ __forceinline__ R mu_d(const CT &D, const R *c, int a, int i, bool dg) {
  R s = D.twoA[a][i] * c[i] + D.E[a][i];
#pragma unroll
  for (int j = 0; j < K; j++)
    if (i != j && !dg) s += D.A[a][i][j] * c[j];
  return s;
}
template <typename R, int K, typename CT>
__device__ __forceinline__ R fe_d(const CT &D, const R *c, int a, bool dg) {
  R s = R(0.0);
#pragma unroll
  for (int i = 0; i < K; i++) {
#pragma unroll
    for (int j = 0; j < K; j++)
      if (i == j || (i < j && !dg)) s += D.A[a][i][j] * c[i] * c[j];
    s += D.B[a][i] * c[i];
  }
  s += D.C[a];
  return s;
}

/* d h_b / d phi_a for a phase a chosen at run time (functionH.h:1-23) */
template <typename R, int N>
__device__ __forceinline__ R dh_rt(const R (&ph)[N], R pa, int b, int a) {
  R s = R(0.0);
  if (a == b) {
    s = R(6.0) * pa * (R(1.0) - pa);
#pragma unroll
    for (int e = 0; e < N; e++)
#pragma unroll
      for (int f = e + 1; f < N; f++)
        if (e != b && f != b) s += R(2.0) * ph[e] * ph[f];
  } else {
#pragma unroll
    for (int e = 0; e < N; e++)
      if (e != b && e != a) s += R(2.0) * ph[e];
    s *= ph[b];
  }
  return s;
}

/* dw/dphi_a for a phase a chosen at run time (functionW_01.h:6-39, functionW_02.h:4-33) */
template <typename R, int N, typename CT>
__device__ __forceinline__ R dwdphi_rt(const CT &D, const R (&ph)[N], R pa, unsigned act, int a) {
  R s = R(0.0);
#pragma unroll
  for (int b = 0; b < N; b++) {
    if (b == a || !((act >> b) & 1u)) continue;
    const R gm = D.gamma[a][b];
    if (D.well) s += R(2.0) * gm * (ph[b] * ph[b] * pa);
    else if ((pa * ph[b]) >= R(0.00000)) s += gm * (ph[b]);
    else s += -gm * (ph[b]);
  }
  if (D.well) s *= R(9.0);
  else s *= D.c16pi2;
#pragma unroll
  for (int b = 0; b < N; b++)
#pragma unroll
    for (int c = b + 1; c < N; c++)
      if (N > 2 && b != a && c != a && ((act >> b) & (act >> c) & 1u)) {
        const R bc = ph[b] * ph[c];
        if (pa * bc >= R(0.00000)) s += D.gamma_abc[a][b][c] * bc;
        else s += -D.gamma_abc[a][b][c] * bc;
      }
  return s;
}

/* anisotropy terms of face fidx of the ring for the pairs present on its
 * stencil (function_A_01.h:163-215 through functionQ.h and anisotropy_01.h):
 * T[p][0] = a_c^2 P_ab and T[p][1] = a_c |q|^2 (dA/dq), whose products with the
 * face means -phi_b and (negated) -phi_a are the divergence terms of (a,b) and
 * (b,a).  x-faces lie between frame rows i and i+1 at column j, y-faces between
 * columns j and j+1 of row i. */
template <typename R, int N, int K, bool ANISO, typename CT>
__device__ __forceinline__ void item_face(const CT &D, ItemFrame<R, N, K> F, ItemSmem<R, N, K, ANISO> &sm, int fidx,
                                          bool tame) {
  constexpr int CO = ItemGeom<R>::CO, BW = ItemGeom<R>::BW;
  const bool xface = fidx < IXF;
  const int f = fidx - IXF;
  const int i = xface ? fidx / RC : f / (TY + 3) + 1, j = xface ? fidx - i * RC + 1 : f - (i - 1) * (TY + 3);
  const int o = i * BW + j + CO, along = xface ? BW : 1, cross = xface ? 1 : BW;
  R s[2], gr[2], cc[2];
  int p = 0;
#pragma unroll 1
  for (int a = 0; a < N - 1; a++)
#pragma unroll 1
    for (int b = a + 1; b < N; b++, p++) {
      R U = R(0.0), W = R(0.0);
      /* both phases on the face's stencil (its two cells, where no pair is rotated) */
      bool have = true;
      if (N > 2) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const R *S = &F[q ? b : a][0][0] + o;
          bool any = (S[0] != R(0.0)) | (S[along] != R(0.0));
          if (!D.rot_identity)
            any = any | (S[cross] != R(0.0)) | (S[-cross] != R(0.0)) | (S[along + cross] != R(0.0)) |
                  (S[along - cross] != R(0.0));
          have = have & any;
        }
        have = have | !tame;
      }
      if (have) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
          const R *S = &F[q ? b : a][0][0] + o;
          const R p0 = S[0], p1 = S[along];
          const R p0p = S[cross], p0m = S[-cross], p1p = S[along + cross], p1m = S[along - cross];
          s[q] = R(0.5) * (p1 + p0);
          if (xface) {
            gr[q] = divx(p1 - p0, D);
            cc[q] = div2y(p0p - p0m, D) + div2y(p1p - p1m, D);
          } else {
            gr[q] = divy(p1 - p0, D);
            cc[q] = R(0.5) * (divx(p0p - p0, D) + divx(p0 - p0m, D)) + R(0.5) * (divx(p1p - p1, D) + divx(p1 - p1m, D));
          }
        }
        const R Pab = s[0] * gr[1] - s[1] * gr[0];
        const R tq = R(0.5) * (s[0] * cc[1] - s[1] * cc[0]);
        R q0, q1;
        rot2(D, D.rot[a][b], xface ? Pab : tq, xface ? tq : Pab, q0, q1);
        const R acv = ac(q0, q1, D.dab[a][b]);
        const QPow<R> qp = qpow(q0, q1);
        R rd;
        if (D.rot_identity) {
          rd = dadq_c(xface ? q0 : q1, qp, D.dab16[a][b]) + R(0.0);
        } else {
          const R d0 = dadq_c(q0, qp, D.dab16[a][b]), d1 = dadq_c(q1, qp, D.dab16[a][b]);
          R r0, r1;
          rot2(D, D.rinv[a][b], d0, d1, r0, r1);
          rd = xface ? r0 : r1;
        }
        const R ac2 = acv * acv;
        U = ac2 * Pab;
        W = acv * qp.q2 * rd;
      }
      sm.w.T[p][0][fidx] = U;
      sm.w.T[p][1][fidx] = W;
    }
}

/* lambda of phase a of ring cell e (calculate_divergence_phasefield_2D,
 * calculate_divergence_phasefield.h:4-62) into DP[a][e] */
template <typename R, int N, int K, bool ANISO, bool TG, typename CT>
__device__ __forceinline__ void item_lambda(const CT &D, ItemFrame<R, N, K> F, ItemSmem<R, N, K, ANISO> &sm, int e,
                                            int a, bool tame, bool dg, double Tpf) {
  constexpr int CO = ItemGeom<R>::CO, BW = ItemGeom<R>::BW;
  const int ri = e / RC, rj = e - ri * RC, i = ri + 1, j = rj + 1, o = i * BW + j + CO;
  const unsigned act = sm.ACT[e];
  R ph[N], m[K];
#pragma unroll
  for (int b = 0; b < N; b++) ph[b] = F[b][i][j + CO];
#pragma unroll
  for (int k = 0; k < K; k++) m[k] = F[N + k][i][j + CO];
  const R *A = &F[a][0][0] + o;
  const R pa = A[0], axp = A[BW], axm = A[-BW], ayp = A[1], aym = A[-1];
  const R gxa = R(0.5) * (divx(axp - pa, D) + divx(pa - axm, D)), gya = div2y(ayp - aym, D);
  R s1 = R(0.0), s2 = R(0.0), t1 = R(0.0), t2 = R(0.0);
#pragma unroll 1
  for (int b = 0; b < N; b++) {
    if (b == a) continue;
    const R *B = &F[b][0][0] + o;
    const R pb = B[0], bxp = B[BW], bxm = B[-BW], byp = B[1], bym = B[-1];
    /* a phase that is zero on the 5-point stencil has no term here */
    if (N > 2 && tame && ((pb == R(0.0)) & (bxp == R(0.0)) & (bxm == R(0.0)) & (byp == R(0.0)) & (bym == R(0.0)))) continue;
    const R gxb = R(0.5) * (divx(bxp - pb, D) + divx(pb - bxm, D)), gyb = div2y(byp - bym, D);
    const R gam = D.gamma[a][b];
    /* face means of the other phase: forward and backward x, right and left y */
    const R fb0 = R(0.5) * (bxp + pb), fb1 = R(0.5) * (pb + bxm), fb2 = R(0.5) * (byp + pb), fb3 = R(0.5) * (pb + bym);
    if (ANISO) {
      const int lo = min(a, b), hi = max(a, b);
      const R sg = a < b ? R(1.0) : R(-1.0);   /* the terms of (b,a) are those of (a,b) negated */
      const R pl = a < b ? pa : pb, ph_ = a < b ? pb : pa, gxl = a < b ? gxa : gxb, gxh = a < b ? gxb : gxa;
      const R gyl = a < b ? gya : gyb, gyh = a < b ? gyb : gya;
      R q0, q1, w0, w1;
      rot2(D, D.rot[lo][hi], pl * gxh - ph_ * gxl, pl * gyh - ph_ * gyl, q0, q1);
      rot2(D, D.rot[a][b], gxb, gyb, w0, w1);
      const QPow<R> qp = qpow(q0, q1);
      R d0 = dadq_c(q0, qp, D.dab16[lo][hi]), d1 = dadq_c(q1, qp, D.dab16[lo][hi]);
      const R cq2 = (q0 * q0 + q1 * q1 + R(0.0) * R(0.0));
      const R cac = ac(q0, q1, D.dab[lo][hi]);
      q0 *= sg;
      q1 *= sg;
      d0 *= sg;
      d1 *= sg;
      R sp1 = R(0.0), sp2 = R(0.0);
      sp1 += q0 * w0;
      sp1 += q1 * w1;
      sp2 += d0 * w0;
      sp2 += d1 * w1;
      sp1 *= gam * (cac * cac);
      sp2 *= gam * cac * cq2;
      s1 += sp1;
      s2 += sp2;
      const int p = lo * N - lo * (lo + 1) / 2 + (hi - lo - 1);
      const int xf = i * RC + rj, xb = (i - 1) * RC + rj;
      const int yr = IXF + ri * (TY + 3) + j, yl = IXF + ri * (TY + 3) + rj;
      const R *U = sm.w.T[p][0], *W = sm.w.T[p][1];
      R d1v = divx((sg * U[xf]) * (-fb0) - (sg * U[xb]) * (-fb1), D);
      d1v += divy((sg * U[yr]) * (-fb2) - (sg * U[yl]) * (-fb3), D);
      d1v *= gam;
      t1 += d1v;
      R d2v = divx((sg * W[xf]) * (-fb0) - (sg * W[xb]) * (-fb1), D);
      d2v += divy((sg * W[yr]) * (-fb2) - (sg * W[yl]) * (-fb3), D);
      d2v *= gam;
      t2 += d2v;
    } else {
      R sp = R(0.0);
      sp += (pa * gxb - pb * gxa) * gxb;
      sp += (pa * gyb - pb * gya) * gyb;
      sp *= gam;
      s1 += sp;
      const R u0 = (R(0.5) * (axp + pa)) * divx(bxp - pb, D) - fb0 * divx(axp - pa, D);
      const R u1 = (R(0.5) * (pa + axm)) * divx(pb - bxm, D) - fb1 * divx(pa - axm, D);
      const R u2 = (R(0.5) * (ayp + pa)) * divy(byp - pb, D) - fb2 * divy(ayp - pa, D);
      const R u3 = (R(0.5) * (pa + aym)) * divy(pb - bym, D) - fb3 * divy(pa - aym, D);
      R dv = divx(u0 * (-fb0) - u1 * (-fb1), D);
      dv += divy(u2 * (-fb2) - u3 * (-fb3), D);
      dv *= gam;
      t1 += dv;
    }
  }
  R dA, div;
  if (ANISO) {
    dA = R(2.0) * (s1 + s2);
    div = (R(2.0) * (t1 + t2) + R(0.0));
  } else {
    dA = R(2.0) * s1;
    div = R(2.0) * t1;
  }
  /* driving force sum_b psi_b dh_b/dphi_a; the terms of an absent phase are +-0 */
  R dpsi = R(0.0);
  R E[TG ? N : 1][K], Bt[TG ? N : 1][K], Ct[TG ? N : 1];
  if constexpr (TG) {
    /* init_propertymatrices(T) at the cell's temperature before dpsi
     * (calculate_divergence_phasefield.h:21-29) */
    if (D.tgrad) {
      e_at<R, N, K>(D, Tpf, E);
      bc_at<R, N, K>(D, Tpf, Bt, Ct);
    }
  }
#pragma unroll
  for (int b = 0; b < N; b++) {
    if (N > 2 && tame && ph[b] == R(0.0) && b != a) continue;
    R c[K], ps = R(0.0);
    bool at_T = false;
    if constexpr (TG) at_T = D.tgrad;
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (TG && at_T) c[k] = c_muE<R, K>(D, E[TG ? b : 0], m, b, k);
      else c[k] = c_mu_d<R, K>(D, m, b, k, dg);
      ps -= m[k] * c[k];
    }
    if (TG && at_T) ps += feBC<R, K>(D, Bt[TG ? b : 0], Ct[TG ? b : 0], c, b);
    else ps += fe_d<R, K>(D, c, b, dg);
    dpsi += ps * dh_rt<R, N>(ph, pa, b, a);
  }
  sm.DP[a][e] = D.eps * (-dA + div) - D.inv_eps * dwdphi_rt<R, N>(D, ph, pa, act, a) - dpsi;
}

/* delta-phi of an active ring cell from its lambdas: their mean, the time step
 * and the simplex projection (calculate_divergence_phasefield.h:45-62) */
template <typename R, int N, int K, bool ANISO, typename CT>
__device__ __forceinline__ void item_dphi(const CT &D, ItemFrame<R, N, K> F, ItemSmem<R, N, K, ANISO> &sm, int e) {
  constexpr int CO = ItemGeom<R>::CO;
  const int ri = e / RC, rj = e - ri * RC;
  const unsigned mask = sm.ACT[e];
  R ph[N], lam[N], d[N], sl = R(0.0);
  bool act[N];
#pragma unroll
  for (int a = 0; a < N; a++) {
    ph[a] = F[a][ri + 1][rj + 1 + CO];
    act[a] = (mask >> a) & 1u;
    if (act[a]) {
      lam[a] = sm.DP[a][e];
      sl += lam[a];
    }
  }
  const int nact = __popc(mask);
  if (nact == 2) sl *= R(0.5);
  else if (nact > 2) sl /= (R)nact;
  const R tau = tau_of<R, N>(D, ph);
#pragma unroll
  for (int a = 0; a < N; a++) d[a] = act[a] ? D.dt * (lam[a] - sl) / (tau * D.eps) : R(0.0);
  project<R, N>(ph, act, d);
#pragma unroll
  for (int a = 0; a < N; a++) sm.DP[a][e] = d[a];
}

/* s_phi of the obstacle anti-trapping of phase a where 0 < phi_a < 1 */
template <typename R, int N, int K>
__device__ __forceinline__ R item_sphi(ItemFrame<R, N, K> F, int i, int j, int a) {
  constexpr int CO = ItemGeom<R>::CO;
  R ph[N];
#pragma unroll
  for (int b = 0; b < N; b++) ph[b] = F[b][i][j + CO];
  const R pa = F[a][i][j + CO];
  /* h_a (functionH.h:24-36) of a phase chosen at run time */
  R t = R(0.0);
  const R s = R(3.0) * pa * pa - R(2.0) * pa * pa * pa;
#pragma unroll
  for (int b = 0; b < N; b++)
#pragma unroll
    for (int c = b + 1; c < N; c++)
      if (b != a && c != a) t += ph[b] * ph[c];
  t *= R(2.0) * pa;
  const R hv = s + t;
  return pa * (R(1.0) - hv) / (sqrt(pa * (R(1.0) - pa)));
}

/* Anti-trapping current through face f of the tile (calculate_fluxes_concentration.h:4-145) */
template <typename R, int N, int K, bool ANISO, bool TG, typename CT>
__device__ __forceinline__ void item_current(const CT &D, ItemFrame<R, N, K> F, ItemSmem<R, N, K, ANISO> &sm, int f,
                                             int y0, int my, bool dg, const double *tcc) {
  constexpr int L = N - 1, CO = ItemGeom<R>::CO, BW = ItemGeom<R>::BW;
  const bool xface = f < JXF;
  const int f0 = f - JXF;
  /* ring row and column of the face's lower cell */
  const int fi = xface ? f / TY : f0 / (TY + 1) + 1, fj = xface ? f - fi * TY + 1 : f0 - (fi - 1) * (TY + 1);
  const int o = (fi + 1) * BW + fj + 1 + CO, along = xface ? BW : 1, cross = xface ? 1 : BW;
  const int c0 = RI(fi, fj), c1 = xface ? c0 + RC : c0 + 1;
  R jat[K], m0[K], m1[K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    jat[k] = R(0.0);
    m0[k] = (&F[N + k][0][0])[o];
    m1[k] = (&F[N + k][0][0])[o + along];
  }
  R E0[TG ? N : 1][K], E1[TG ? N : 1][K];
  bool at_T = false;
  if constexpr (TG) {
    at_T = D.tgrad;
    if (at_T) {
      /* the ghosted columns of the two cells (cells past my+1 are not needed: clamped) */
      e_at<R, N, K>(D, ld_step(tcc + min(y0 - 1 + fj + 3, my + 5)), E0);
      e_at<R, N, K>(D, ld_step(tcc + min(y0 - 1 + (xface ? fj : fj + 1) + 3, my + 5)), E1);
    }
  }
  /* the gradient across the face and the mean tangential one */
  auto grads = [&](int a, R &gr, R &cn) {
    const R *S = &F[a][0][0] + o;
    const R p0 = S[0], p1 = S[along];
    const R p0p = S[cross], p0m = S[-cross], p1p = S[along + cross], p1m = S[along - cross];
    if (xface) {
      gr = divx(p1 - p0, D);
      cn = R(0.5) * (div2y(p0p - p0m, D) + div2y(p1p - p1m, D));
    } else {
      gr = divy(p1 - p0, D);
      const R gc0 = R(0.5) * (divx(p0p - p0, D) + divx(p0 - p0m, D));
      const R gc1 = R(0.5) * (divx(p1p - p1, D) + divx(p1 - p1m, D));
      cn = R(0.5) * (gc0 + gc1);
    }
  };
  /* calculate_fluxes_concentration.h:65: no y-current where gidy is 0 or MESH_Y-2 */
  const bool yskip = !xface && (y0 - 1 + fj) + 3 == my - 2;
  R grL, cnL;
  grads(L, grL, cnL);
  const R nl = sqrt(cnL * cnL + grL * grL);
#pragma unroll 1
  for (int a = 0; a < L; a++) {
    R gr, cn;
    grads(a, gr, cn);
    /* sqrt(s2) != 0 exactly when s2 != 0 (s2 >= 0, or NaN on both sides) */
    const R s2 = cn * cn + gr * gr;
    if (s2 != R(0.0) && !yskip) {
      const R ng = sqrt(s2);
      R sp = gr * grL;
      sp += cn * cnL;
      if (nl > R(0.0)) sp /= (nl * ng);
      R w0 = R(1.0), w1 = R(1.0);
      if (D.obstacle) {
        const R p0 = (&F[a][0][0])[o], p1 = (&F[a][0][0])[o + along];
        w0 = p0 * (R(1.0) - p0) > R(0.0) ? sm.SP[a][c0] : R(0.0);
        w1 = p1 * (R(1.0) - p1) > R(0.0) ? sm.SP[a][c1] : R(0.0);
      }
      const R d0 = sm.DP[a][c0], d1 = sm.DP[a][c1];
#pragma unroll
      for (int k = 0; k < K; k++) {
        R cl1, cl0, cs1, cs0;
        if (TG && at_T) {
          cl1 = c_muE<R, K>(D, E1[TG ? L : 0], m1, L, k);
          cl0 = c_muE<R, K>(D, E0[TG ? L : 0], m0, L, k);
          cs1 = cs0 = R(0.0);
#pragma unroll
          for (int b = 0; b < L; b++)
            if (b == a) {
              cs1 = c_muE<R, K>(D, E1[TG ? b : 0], m1, b, k);
              cs0 = c_muE<R, K>(D, E0[TG ? b : 0], m0, b, k);
            }
        } else {
          cl1 = c_mu_d<R, K>(D, m1, L, k, dg);
          cl0 = c_mu_d<R, K>(D, m0, L, k, dg);
          cs1 = c_mu_d<R, K>(D, m1, a, k, dg);
          cs0 = c_mu_d<R, K>(D, m0, a, k, dg);
        }
        R bracket;
        if (D.obstacle) bracket = w1 * (cl1 - cs1) * d1 + w0 * (cl0 - cs0) * d0;
        else bracket = (cl1 - cs1) * d1 + (cl0 - cs0) * d0;
        jat[k] += D.atf[a][k] * fabs(sp) * (D.obstacle ? R(0.5) : D.well_half) * bracket * gr / ng;
      }
    }
  }
#pragma unroll
  for (int k = 0; k < K; k++) sm.w.J[k][f] = jat[k];
}

/* mu update and phi commit of the tile's cell (tx, ty)
 * (calculate_divergence_concentration.h:24-140): divergences of the diffusion
 * flux and the current, then the bulk branch (mu = Mu_a(c_a(mu) + dc)) or the
 * interface branch (dmu = (dc/dmu)^-1 dc, inverted in FP64), then phi +=
 * delta-phi.  x, y: the cell's interior coordinates; currents: some face of the tile
 * may carry one. */
template <typename R, int N, int K, bool ANISO, bool TG, typename CT>
__device__ __forceinline__ void item_commit(const CT &D, ItemFrame<R, N, K> F, const ItemSmem<R, N, K, ANISO> &sm,
                                            int tx, int ty, int x, int y, bool tame, bool dg, bool currents,
                                            const R *ph, const R *dp, const R *m, R *nph, R *nm, double *dmu, double Tc) {
  constexpr int CO = ItemGeom<R>::CO;
  const R cst = D.obstacle ? D.jat_obst : D.jat_well;
  const int c = RI(tx + 1, ty + 1);
  const bool hxf = currents && ((sm.JW[tx + 1] >> ty) & 1u), hxb = currents && ((sm.JW[tx] >> ty) & 1u);
  const bool hyr = currents && ((sm.JW[TX + 1 + tx] >> (ty + 1)) & 1u), hyl = currents && ((sm.JW[TX + 1 + tx] >> ty) & 1u);
  const int xf = (tx + 1) * TY + ty, xb = tx * TY + ty, yr = JXF + tx * (TY + 1) + ty + 1, yl = yr - 1;
  R divflux[K], divjat[K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    divflux[k] = R(0.0);
#pragma unroll
    for (int l = 0; l < K; l++) {
      if (k != l && dg) continue;
      const R *DD = sm.DD[k][l];
      const R dc = DD[c];
#define M_(u, v) F[N + l][tx + 2 + (u)][ty + 2 + (v) + CO]
      const R mc = M_(0, 0);
      const R fxf = ((DD[c + RC] + dc) * R(0.5)) * divx(M_(1, 0) - mc, D);
      const R fxb = ((dc + DD[c - RC]) * R(0.5)) * divx(mc - M_(-1, 0), D);
      const R fyr = ((DD[c + 1] + dc) * R(0.5)) * divy(M_(0, 1) - mc, D);
      const R fyl = ((dc + DD[c - 1]) * R(0.5)) * divy(mc - M_(0, -1), D);
#undef M_
      divflux[k] += divx(fxf - fxb, D);
      divflux[k] += divy(fyr - fyl, D);
    }
    const R *J = sm.w.J[k];
    const R jxf = hxf ? J[xf] : R(0.0), jxb = hxb ? J[xb] : R(0.0);
    const R jyr = hyr ? J[yr] : R(0.0), jyl = hyl ? J[yl] : R(0.0);
    divjat[k] = divx((jxf - jxb) * cst, D);
    divjat[k] += divy((jyr - jyl) * cst, D);
  }
  R E[TG ? N : 1][K];
  bool at_T = false;
  if constexpr (TG) {
    at_T = D.tgrad;
    if (at_T) e_at<R, N, K>(D, Tc, E);
  }
  int bulk = -1;
#pragma unroll
  for (int a = 0; a < N; a++)
    if (bulk < 0 && ph[a] == R(1.0)) bulk = a;
  if (bulk >= 0) {
    {
      R cn[K];
      bool ordinary = true;   /* (a current may not be, where a lambda was not) */
#pragma unroll
      for (int k = 0; k < K; k++) {
        R cm = R(0.0);
        if (TG && at_T) {
#pragma unroll
          for (int a = 0; a < N; a++)
            if (a == bulk) cm = c_muE<R, K>(D, E[TG ? a : 0], m, a, k);
        } else {
          cm = c_mu_d<R, K>(D, m, bulk, k, dg);
        }
        cn[k] = cm + D.dt * (divflux[k]) - divjat[k];
        if (K > 1) ordinary = ordinary & (fabs(cn[k]) < R(MU_TAME));
      }
#pragma unroll
      for (int k = 0; k < K; k++) {
        if (TG && at_T) {
#pragma unroll
          for (int a = 0; a < N; a++)
            if (a == bulk) nm[k] = MuE<R, K>(D, E[TG ? a : 0], cn, a, k);
        } else {
          nm[k] = mu_d<R, K>(D, cn, bulk, k, dg && ordinary);
        }
        dmu[k] = (double)nm[k] - (double)m[k];
      }
#pragma unroll
      for (int a = 0; a < N; a++) nph[a] = ph[a] + dp[a];
    }
  } else {
    /* sum_a c_a(mu) sum_b dh_a/dphi_b dphi_b (calculate_divergence_concentration.h:23-31) */
    R sum[K];
    double dc[K], dcdmu[K][K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      sum[k] = R(0.0);
#pragma unroll
      for (int l = 0; l < K; l++) dcdmu[k][l] = 0.0;
    }
    /* non-isothermal (calculate_divergence_concentration.h:85): minus
     * sum_a dcbdT_phase h_a * dt * (-GRADIENT * velocity); dcbdT_phase is
     * allocated but never filled by the reference (taken as 0) and the struct
     * member GRADIENT is never set, so the term is a signed zero */
    R sdc = R(0.0);
    bool ordinary = tame;
#pragma unroll
    for (int a = 0; a < N; a++)
      if (N > 2) ordinary = ordinary & (fabs(dp[a]) < R(MU_TAME));
#pragma unroll
    for (int a = 0; a < N; a++) {
      /* a phase the cell neither holds nor gains: h and its terms are +-0 */
      if (N > 2 && ordinary && ph[a] == R(0.0) && dp[a] == R(0.0)) continue;
      R sdh = R(0.0);
#pragma unroll
      for (int b = 0; b < N; b++) sdh += dh<R, N>(ph, a, b) * dp[b];
      const R hv = h<R, N>(ph, a);
      if (TG && at_T) sdc += R(0.0) * hv;
#pragma unroll
      for (int k = 0; k < K; k++) {
        R cm;
        if (TG && at_T) cm = c_muE<R, K>(D, E[TG ? a : 0], m, a, k);
        else cm = c_mu_d<R, K>(D, m, a, k, dg);
        sum[k] += cm * sdh;
#pragma unroll
        for (int l = 0; l < K; l++)
          if (k == l || !dg) dcdmu[k][l] += D.cmu64[a][k][l] * (double)hv;
      }
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (TG && at_T) dc[k] = (double)(D.dt * (divflux[k]) - divjat[k] - sum[k] - sdc * D.dt * (R(-0.0) * (R)D.tg_vel));
      else dc[k] = (double)(D.dt * (divflux[k]) - divjat[k] - sum[k]);
    }
    double m64[K];
#pragma unroll
    for (int k = 0; k < K; k++) m64[k] = (double)m[k];
    solve_dmu<R, K>(D, dcdmu, dc, m64, dmu);
#pragma unroll
    for (int k = 0; k < K; k++) nm[k] = (R)m64[k];
#pragma unroll
    for (int a = 0; a < N; a++) nph[a] = ph[a] + dp[a];
  }
}

/* FP64 sums of the progress record over the tile's cells into its slot (the
 * host folds the slots in a fixed order); call with all threads. */
template <typename R, int N, int K, bool TG, typename CT>
__device__ __forceinline__ void item_sums(const CT &D, bool valid, const R *nph, const R *nm, const R *dp,
                                          const double *dmu, const StatBufs &st, long long slot, double Tc) {
  constexpr int NS = 2 * N + 2 * K + 1, NW = NTI / 32;
  __shared__ double red[NW][NS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int f = 0; f < NS; f++) {   /* unrolled: the cell's values stay in registers */
    double v = 0.0;
    if (valid) {
      if (f < N) v = (double)dp[f] * (double)dp[f];
      else if (f < N + K) v = dmu[f - N] * dmu[f - N];
      else if (f < 2 * N + K) v = (double)nph[f - N - K];
      else if (f < 2 * N + 2 * K) {
        const int k = f - 2 * N - K;
        R comp = R(0.0);
        if (TG && D.tgrad) {
          R E[N][K];
          e_at<R, N, K>(D, Tc, E);
#pragma unroll
          for (int b = 0; b < N; b++) comp += c_muE<R, K>(D, E[b], nm, b, k) * h<R, N>(nph, b);
        } else {
#pragma unroll
          for (int b = 0; b < N; b++) comp += c_mu<R, K>(D, nm, b, k) * h<R, N>(nph, b);
        }
        v = (double)comp;
      } else {
        bool bad = false;
#pragma unroll
        for (int a = 0; a < N; a++) bad |= !isfinite(nph[a]);
#pragma unroll
        for (int k = 0; k < K; k++) bad |= !isfinite(nm[k]);
        v = bad ? 1.0 : 0.0;
      }
    }
    v = warp_sum(v);
    if (lane == 0) red[wid][f] = v;
  }
  __syncthreads();
  if (threadIdx.x < NS) {
    double r = 0.0;
    for (int w = 0; w < NW; w++) r += red[w][threadIdx.x];
    st.partials[slot * NS + threadIdx.x] = r;
  }
  __syncthreads();
}

/* The simulation's running extremes take the new values of a warp's cells (in: the
 * lane's cell counts): compared with the extremes as the warp last saw them (older
 * ones at worst), reduced over the warp only where a lane beats one, and sent to the
 * slot by one lane when they beat that too.  On the first step of a context every mu
 * does: with an atomic per cell on these few addresses that step took 2.0 ms at
 * 4096^2 and 0.55 ms at 2048^2; it takes 0.34 and 0.13 ms, as the next one does.
 * Exact and order-free; NaN is ignored.  Call with the whole warp. */
template <typename R, int N, int K>
__device__ __forceinline__ void item_extremes(double *ext, bool in, const R *nph, const R *nm, const StatBufs &st, int s) {
  /* slot layout: max phi[N], min phi[N], max mu[K], min mu[K] */
  bool beats = false;
#pragma unroll
  for (int f = 0; f < N + K; f++) {
    const double v = f < N ? (double)nph[f < N ? f : 0] : (double)nm[f < N ? 0 : f - N];
    const int hi = f < N ? f : 2 * N + (f - N), lo = f < N ? N + f : 2 * N + K + (f - N);
    beats = beats | (v > ext[hi]) | (v < ext[lo]);
  }
  if (!__any_sync(0xffffffffu, in & beats)) return;
  long long *slot = st.ext + (long long)s * (2 * (N + K));
  auto from_ord = [](long long o) { return __longlong_as_double(o < 0 ? o ^ 0x7fffffffffffffffLL : o); };
#pragma unroll
  for (int f = 0; f < N + K; f++) {
    const double v = f < N ? (double)nph[f < N ? f : 0] : (double)nm[f < N ? 0 : f - N];
    const int hi = f < N ? f : 2 * N + (f - N), lo = f < N ? N + f : 2 * N + K + (f - N);
    const bool up = in & (v > ext[hi]), down = in & (v < ext[lo]);
    if (__any_sync(0xffffffffu, up)) {
      const double m = warp_max(up ? v : -INFINITY);
      if ((threadIdx.x & 31) == 0) {
        const double now = from_ord(*(volatile long long *)(slot + hi));
        if (m > now) atomicMax(slot + hi, ord(m));
        ext[hi] = m > now ? m : now;
      }
    }
    if (__any_sync(0xffffffffu, down)) {
      const double m = warp_min(down ? v : INFINITY);
      if ((threadIdx.x & 31) == 0) {
        const double now = from_ord(*(volatile long long *)(slot + lo));
        if (m < now) atomicMin(slot + lo, ord(m));
        ext[lo] = m < now ? m : now;
      }
    }
  }
  __syncwarp();
}

}  // namespace gpd
