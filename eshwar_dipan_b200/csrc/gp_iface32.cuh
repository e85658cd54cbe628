/*
 * gp_iface32.cuh -- the arithmetic of an interface tile of the FP32 storage form,
 * on the frame staged by general_tiles (gp_fused.cuh).
 *
 * The FP32 unit is compiled with fused multiply-adds, and a triple junction
 * magnifies a last-bit difference a thousandfold within a thousand steps, so the
 * expressions here (unlike the FP64 ones of gp_iface.cuh, which are exact
 * whatever the order of evaluation around them) stay in the shape whose
 * contraction the form's results were measured with.
 */
#pragma once
#include "gp_iface.cuh"

namespace gpd {

template <typename R, int N, int K>
struct ItemSmem32 {
  R DP[N][SS];             /* delta-phi of the ring region */
  unsigned char ACT[SS];   /* active phases of each ring cell (bit a) */
  short LIST[SS];          /* ring cells with an active phase, in no particular order */
  short FLIST[IFT];        /* anisotropy faces those cells read */
  int nlist, nflist;
  union {
    R T[NP<N>::v][4][IFT]; /* anisotropy face terms of the ring region */
    struct {
      R CM[N][K][SS];      /* c_a,k(mu) per cell */
      R H[N][SS];          /* h_a(phi) per cell */
      R SP[N][SS];         /* s_phi of the obstacle anti-trapping (solid phases) */
      R DD[K][K][SS];      /* D_kl per cell */
      R JX[K][NXF], JY[K][NYF];
      R FX[K][K][NXF], FY[K][K][NYF];
    } u;
  } w;
};

#define FS_(i, j) F[a][i][(j) + CO]
#define FA(i, j) F[a][i][(j) + CO]
#define FB(i, j) F[b][i][(j) + CO]

/* Anisotropy terms of one face of the ring region for all pairs: the same
 * order of operations as the reference (function_A_01.h:163-215 through functionQ.h and
 * anisotropy_01.h) on the two-cell-halo layout.  xface: face between P rows
 * i and i+1 at column j; else between columns j and j+1 of row i. */
template <typename R, int N, int K, typename CT>
__device__ __forceinline__ void ring_face_terms(const CT &D, ItemFrame<R, N, K> F, R (*T)[4][IFT],
                                                bool xface, int i, int j, int fidx) {
  constexpr int CO = ItemGeom<R>::CO;
  R s[N], gr[N], c0[N], c1[N];
#pragma unroll
  for (int a = 0; a < N; a++) {
    if (xface) {
      R p0 = FS_(i, j), p1 = FS_(i + 1, j);
      s[a] = R(0.5) * (p1 + p0);
      gr[a] = divx(p1 - p0, D);
      c0[a] = div2y(FS_(i, j + 1) - FS_(i, j - 1), D);
      c1[a] = div2y(FS_(i + 1, j + 1) - FS_(i + 1, j - 1), D);
    } else {
      R p0 = FS_(i, j), p1 = FS_(i, j + 1);
      s[a] = R(0.5) * (p1 + p0);
      gr[a] = divy(p1 - p0, D);
      c0[a] = R(0.5) * (divx(FS_(i + 1, j) - FS_(i, j), D) + divx(FS_(i, j) - FS_(i - 1, j), D));
      c1[a] = R(0.5) * (divx(FS_(i + 1, j + 1) - FS_(i, j + 1), D) +
                        divx(FS_(i, j + 1) - FS_(i - 1, j + 1), D));
    }
  }
#pragma unroll
  for (int a = 0; a < N; a++)
#pragma unroll
    for (int b = a + 1; b < N; b++) {
      const int p = pidx<N>(a, b);
      R Pab = s[a] * gr[b] - s[b] * gr[a];
      R Pba = s[b] * gr[a] - s[a] * gr[b];
      R tq = R(0.5) * (s[a] * (c0[b] + c1[b]) - s[b] * (c0[a] + c1[a]));
      R q0, q1;
      if (xface) rot2(D, D.rot[a][b], Pab, tq, q0, q1);
      else rot2(D, D.rot[a][b], tq, Pab, q0, q1);
      R acv = ac(q0, q1, D.dab[a][b]);
      QPow<R> qp = qpow(q0, q1);
      R rd;
      if (D.rot_identity) {
        rd = (xface ? dadq_c(q0, qp, D.dab16[a][b]) : dadq_c(q1, qp, D.dab16[a][b])) + R(0.0);
      } else {
        R d0 = dadq_c(q0, qp, D.dab16[a][b]), d1 = dadq_c(q1, qp, D.dab16[a][b]);
        R r0, r1;
        rot2(D, D.rinv[a][b], d0, d1, r0, r1);
        rd = xface ? r0 : r1;
      }
      R ac2 = acv * acv, acq = acv * qp.q2;
      T[p][0][fidx] = ac2 * Pab * (-s[b]);
      T[p][1][fidx] = ac2 * Pba * (-s[a]);
      T[p][2][fidx] = acq * rd * (-s[b]);
      T[p][3][fidx] = acq * (R(0.0) - rd) * (-s[a]);
    }
}

/* delta-phi of one ring cell (ring coordinates ri, rj; its phi at P row ri+1,
 * column rj+1) from the staged tile: calculate_divergence_phasefield_2D
 * (calculate_divergence_phasefield.h:4-62).
 * Not inlined: as a call of its own it gets its own register allocation. Under
 * the 128-register cap of two CTAs per SM it spills nothing and the tile's code
 * around it at most 120 bytes. */
template <typename R, int N, int K, bool ANISO, typename CT>
__device__ __noinline__ void ring_dphi(const CT &D, ItemFrame<R, N, K> F, const ItemSmem32<R, N, K> &sm, int ri, int rj,
                                          unsigned mask, R *d, double Tpf) {
  constexpr int CO = ItemGeom<R>::CO;
  const int i = ri + 1, j = rj + 1;
  R ph[N];
  bool act[N];
#pragma unroll
  for (int a = 0; a < N; a++) {
    ph[a] = F[a][i][j + CO];
    act[a] = (mask >> a) & 1u;
  }
  if (!mask) {
#pragma unroll
    for (int a = 0; a < N; a++) {
      d[a] = R(0.0);
      if ((ph[a] + d[a]) < R(0.0)) d[a] += fabs(d[a] + ph[a]);
    }
    return;
  }
  R m[K];
#pragma unroll
  for (int k = 0; k < K; k++) m[k] = F[N + k][i][j + CO];
  R gcx[N], gcy[N];
#pragma unroll
  for (int a = 0; a < N; a++) {
    gcx[a] = R(0.5) * (divx(FS_(i + 1, j) - FS_(i, j), D) + divx(FS_(i, j) - FS_(i - 1, j), D));
    gcy[a] = div2y(FS_(i, j + 1) - FS_(i, j - 1), D);
  }
  R psi[N];
  if (D.tgrad) {
    /* init_propertymatrices(T) at the cell's temperature before dpsi
     * (calculate_divergence_phasefield.h:21-29) */
    R E[N][K], Bt[N][K], Ct[N];
    e_at<R, N, K>(D, Tpf, E);
    bc_at<R, N, K>(D, Tpf, Bt, Ct);
#pragma unroll
    for (int b = 0; b < N; b++) {
      R c[K], ps = R(0.0);
#pragma unroll
      for (int k = 0; k < K; k++) {
        c[k] = c_muE<R, K>(D, E[b], m, b, k);
        ps -= m[k] * c[k];
      }
      ps += feBC<R, K>(D, Bt[b], Ct[b], c, b);
      psi[b] = ps;
    }
  } else {
#pragma unroll
    for (int b = 0; b < N; b++) {
      R c[K], ps = R(0.0);
#pragma unroll
      for (int k = 0; k < K; k++) {
        c[k] = c_mu<R, K>(D, m, b, k);
        ps -= m[k] * c[k];
      }
      ps += fe<R, K>(D, c, b);
      psi[b] = ps;
    }
  }
  R cq0[NP<N>::v], cq1[NP<N>::v], cd0[NP<N>::v], cd1[NP<N>::v], cac[NP<N>::v], cq2[NP<N>::v];
  if (ANISO) {
#pragma unroll
    for (int a = 0; a < N; a++)
#pragma unroll
      for (int b = a + 1; b < N; b++) {
        const int p = pidx<N>(a, b);
        R q0, q1;
        rot2(D, D.rot[a][b], (ph[a] * gcx[b] - ph[b] * gcx[a]), (ph[a] * gcy[b] - ph[b] * gcy[a]), q0, q1);
        QPow<R> qp = qpow(q0, q1);
        cq0[p] = q0;
        cq1[p] = q1;
        cd0[p] = dadq_c(q0, qp, D.dab16[a][b]);
        cd1[p] = dadq_c(q1, qp, D.dab16[a][b]);
        cq2[p] = (q0 * q0 + q1 * q1 + R(0.0) * R(0.0));
        cac[p] = ac(q0, q1, D.dab[a][b]);
      }
  }
  const R tau = tau_of<R, N>(D, ph);
  R lam[N], sl = R(0.0);
  long nact = 0;
  /* face indices of this cell in the ring face cache */
  const int xf = i * (TY + 2) + (j - 1), xb = (i - 1) * (TY + 2) + (j - 1);
  const int yr = IXF + (i - 1) * (TY + 3) + j, yl = IXF + (i - 1) * (TY + 3) + (j - 1);
#pragma unroll
  for (int a = 0; a < N; a++) {
    if (!act[a]) continue;
    R dA, div;
    if (ANISO) {
      R s1 = R(0.0), s2 = R(0.0), t1 = R(0.0), t2 = R(0.0);
#pragma unroll
      for (int b = 0; b < N; b++) {
        if (b == a) continue;
        const int p = a < b ? pidx<N>(a, b) : pidx<N>(b, a);
        const R sg = R(0.0);
        R q0 = a < b ? cq0[p] : sg - cq0[p], q1 = a < b ? cq1[p] : sg - cq1[p];
        R d0 = a < b ? cd0[p] : sg - cd0[p], d1 = a < b ? cd1[p] : sg - cd1[p];
        R w0, w1;
        rot2(D, D.rot[a][b], gcx[b], gcy[b], w0, w1);
        R sp1 = R(0.0), sp2 = R(0.0);
        sp1 += q0 * w0;
        sp1 += q1 * w1;
        sp2 += (d0) * w0;
        sp2 += (d1) * w1;
        sp1 *= D.gamma[a][b] * (cac[p] * cac[p]);
        sp2 *= D.gamma[a][b] * cac[p] * cq2[p];
        s1 += sp1;
        s2 += sp2;
        const int o = a < b ? 0 : 1;
        const R(*T)[IFT] = sm.w.T[p];
        R d1v = divx((T[o][xf]) - (T[o][xb]), D);
        d1v += divy((T[o][yr]) - (T[o][yl]), D);
        d1v *= D.gamma[a][b];
        t1 += d1v;
        R d2v = divx(T[2 + o][xf] - T[2 + o][xb], D);
        d2v += divy(T[2 + o][yr] - T[2 + o][yl], D);
        d2v *= D.gamma[a][b];
        t2 += d2v;
      }
      dA = R(2.0) * (s1 + s2);
      div = (R(2.0) * (t1 + t2) + R(0.0));
    } else {
      R s = R(0.0), t = R(0.0);
#pragma unroll
      for (int b = 0; b < N; b++) {
        if (b == a) continue;
        R sp = R(0.0);
        sp += (ph[a] * gcx[b] - ph[b] * gcx[a]) * gcx[b];
        sp += (ph[a] * gcy[b] - ph[b] * gcy[a]) * gcy[b];
        sp *= D.gamma[a][b];
        s += sp;
        R pa = FA(i, j), pb = FB(i, j);
        R sxa = R(0.5) * (FA(i + 1, j) + pa), sxb = R(0.5) * (FB(i + 1, j) + pb);
        R gxa = divx(FA(i + 1, j) - pa, D), gxb = divx(FB(i + 1, j) - pb, D);
        R bxa = R(0.5) * (pa + FA(i - 1, j)), bxb = R(0.5) * (pb + FB(i - 1, j));
        R hxa = divx(pa - FA(i - 1, j), D), hxb = divx(pb - FB(i - 1, j), D);
        R sya = R(0.5) * (FA(i, j + 1) + pa), syb = R(0.5) * (FB(i, j + 1) + pb);
        R gya = divy(FA(i, j + 1) - pa, D), gyb = divy(FB(i, j + 1) - pb, D);
        R lya = R(0.5) * (pa + FA(i, j - 1)), lyb = R(0.5) * (pb + FB(i, j - 1));
        R hya = divy(pa - FA(i, j - 1), D), hyb = divy(pb - FB(i, j - 1), D);
        R dvg = divx((sxa * gxb - sxb * gxa) * (-sxb) - ((bxa * hxb - bxb * hxa) * (-bxb)), D);
        dvg += divy((sya * gyb - syb * gya) * (-syb) - ((lya * hyb - lyb * hya) * (-lyb)), D);
        dvg *= D.gamma[a][b];
        t += dvg;
      }
      dA = R(2.0) * s;
      div = R(2.0) * t;
    }
    R dpsi = R(0.0);
#pragma unroll
    for (int b = 0; b < N; b++) dpsi += psi[b] * dh<R, N>(ph, b, a);
    lam[a] = D.eps * (-dA + div) - D.inv_eps * dwdphi<R, N>(D, ph, act, a, false) - dpsi;
    sl += lam[a];
    nact++;
  }
  if (nact) sl /= (R)nact;
#pragma unroll
  for (int a = 0; a < N; a++) d[a] = act[a] ? D.dt * (lam[a] - sl) / (tau * D.eps) : R(0.0);
  project<R, N>(ph, act, d);
}

/* FP32 commit of a pure-phase cell: mu += muc_a * dc in FP64, phi += dphi,
 * both rounded stochastically. */
template <typename R, int N, int K>
__device__ __forceinline__ void bulk_commit_f32(const Consts<R> &D, int a, const R *dc, const R *ph, const R *dp,
                                                const R *m, R *nph, R *nm, double *dmu, unsigned key) {
#pragma unroll
  for (int k = 0; k < K; k++) {
    double s = 0.0;
#pragma unroll
    for (int l = 0; l < K; l++) s += D.muc64[a][k][l] * (double)dc[l];
    dmu[k] = s;
    nm[k] = (R)round_stochastic((double)m[k] + s, key, N + k);
  }
#pragma unroll
  for (int a2 = 0; a2 < N; a2++) nph[a2] = (R)round_stochastic((double)ph[a2] + (double)dp[a2], key, a2);
}

/* mu update and phi commit of one tile cell from the tile's face fluxes
 * (calculate_divergence_concentration.h:24-140): divergences, then the bulk
 * branch (mu += dmu/dc dc, bulk_commit_f32) or the interface branch (dmu = (dc/dmu)^-1 dc,
 * inverted in FP64), then phi += delta-phi, all rounded stochastically.  i, j: the
 * cell's position in the one-cell-halo tile layout; x, y: its interior coordinates. */
template <typename R, int N, int K, typename CT>
__device__ __forceinline__ void commit_cell(const CT &D, const R (&FX)[K][K][NXF], const R (&FY)[K][K][NYF],
                                            const R (&JX)[K][NXF], const R (&JY)[K][NYF], const R (&CM)[N][K][SS],
                                            const R (&H)[N][SS], int i, int j, int x, int y, const R *ph,
                                            const R *dp, const R *m, R *nph, R *nm, double *dmu,
                                            const StatBufs &st) {
  const R cst = D.obstacle ? D.jat_obst : D.jat_well;
  const int c = LI(i, j);
  R divflux[K], divjat[K];
  const int xf = i * TY + (j - 1), xb = (i - 1) * TY + (j - 1);
  const int yr = (i - 1) * (TY + 1) + j, yl = (i - 1) * (TY + 1) + (j - 1);
#pragma unroll
  for (int k = 0; k < K; k++) {
    divflux[k] = R(0.0);
#pragma unroll
    for (int l = 0; l < K; l++) {
      divflux[k] += divx(FX[k][l][xf] - FX[k][l][xb], D);
      divflux[k] += divy(FY[k][l][yr] - FY[k][l][yl], D);
    }
    divjat[k] = divx((JX[k][xf] - JX[k][xb]) * cst, D);
    divjat[k] += divy((JY[k][yr] - JY[k][yl]) * cst, D);
  }
  int bulk = -1;
#pragma unroll
  for (int a = 0; a < N; a++)
    if (bulk < 0 && ph[a] == R(1.0)) bulk = a;
  if (bulk >= 0) {
    R cn[K];
#pragma unroll
    for (int k = 0; k < K; k++) cn[k] = D.dt * (divflux[k]) - divjat[k];
    bulk_commit_f32<R, N, K>(D, bulk, cn, ph, dp, m, nph, nm, dmu, round_key(ld_step(st.round_step), x, y));
  } else {
    /* sum_a c_a(mu) sum_b dh_a/dphi_b dphi_b (calculate_divergence_concentration.h:23-31) */
    R sum[K];
    double dc[K], dcdmu[K][K];
#pragma unroll
    for (int k = 0; k < K; k++) sum[k] = R(0.0);
#pragma unroll
    for (int a = 0; a < N; a++) {
      R sdh = R(0.0);
#pragma unroll
      for (int b = 0; b < N; b++) sdh += dh<R, N>(ph, a, b) * dp[b];
#pragma unroll
      for (int k = 0; k < K; k++) sum[k] += CM[a][k][c] * sdh;
    }
    /* non-isothermal (calculate_divergence_concentration.h:85): minus
     * sum_a dcbdT_phase h_a * dt * (-GRADIENT * velocity); dcbdT_phase is
     * allocated but never filled by the reference (taken as 0) and the struct
     * member GRADIENT is never set, so the term is a signed zero */
    R sdc = R(0.0);
    if (D.tgrad) {
#pragma unroll
      for (int a = 0; a < N; a++) sdc += R(0.0) * H[a][c];
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (D.tgrad) dc[k] = (double)(D.dt * (divflux[k]) - divjat[k] - sum[k] - sdc * D.dt * (R(-0.0) * (R)D.tg_vel));
      else dc[k] = (double)(D.dt * (divflux[k]) - divjat[k] - sum[k]);
#pragma unroll
      for (int l = 0; l < K; l++) {
        dcdmu[k][l] = 0.0;
#pragma unroll
        for (int a = 0; a < N; a++) dcdmu[k][l] += D.cmu64[a][k][l] * (double)H[a][c];
      }
    }
    double m64[K];
#pragma unroll
    for (int k = 0; k < K; k++) m64[k] = (double)m[k];
    solve_dmu<R, K>(D, dcdmu, dc, m64, dmu);
    const unsigned key = round_key(ld_step(st.round_step), x, y);
#pragma unroll
    for (int k = 0; k < K; k++) nm[k] = round_stochastic(m64[k], key, N + k);
#pragma unroll
    for (int a = 0; a < N; a++) nph[a] = round_stochastic((double)ph[a] + (double)dp[a], key, a);
  }
}

/* One staged interface tile (cells (x0+tx, y0+ty)): delta-phi on the tile and its
 * ring, then the concentration pass (calculate_fluxes_concentration_2D +
 * calculate_divergence_concentration_2D, calculate_fluxes_concentration.h:4-145,
 * calculate_divergence_concentration.h:4-153); the thread's cell into dp, nph, nm,
 * dmu.  hook: called once by every thread after the first pass. */
template <typename R, int N, int K, bool ANISO, typename CT, typename HOOK>
__device__ __forceinline__ void tile32(const CT &D, const Grid &g, ItemFrame<R, N, K> F, int x0, int y0,
                                       const StatBufs &st, ItemSmem32<R, N, K> &sm, const double *tpf,
                                       const double *tcc, R (&dp)[N], R (&nph)[N], R (&nm)[K],
                                       double (&dmu)[K], HOOK &&hook) {
  constexpr int L = N - 1, CO = ItemGeom<R>::CO;

  /* ---- active phases of the ring cells (interior plus ring: x <= mx, y <= my).
   * A cell with no active phase gets its delta-phi here (no phase active:
   * 0, then the projection's clamp of a negative phi; outside the needed
   * region: 0); the others go on a list, so that the expensive delta-phi
   * work is spread over every thread of the CTA wherever the active cells
   * lie in the tile. */
  for (int e = threadIdx.x; e < SS; e += NT) {
    const int ri = e / SW, rj = e - ri * SW, i = ri + 1, j = rj + 1;
    const bool vd = (x0 - 1 + ri <= g.mx) && (y0 - 1 + rj <= g.my);
    unsigned mask = 0;
#pragma unroll
    for (int a = 0; a < N; a++) {
      R gxf = divx(FS_(i + 1, j) - FS_(i, j), D), gxb = divx(FS_(i, j) - FS_(i - 1, j), D);
      R gyr = divy(FS_(i, j + 1) - FS_(i, j), D), gyl = divy(FS_(i, j) - FS_(i, j - 1), D);
      R dv = divx(gxf - gxb, D);
      dv += divy(gyr - gyl, D);
      if (fabs(dv) > R(0.0)) mask |= 1u << a;
    }
    if (!vd) mask = 0;
    sm.ACT[e] = (unsigned char)mask;
    if (mask) {
      sm.LIST[atomicAdd(&sm.nlist, 1)] = (short)e;
    } else {
#pragma unroll
      for (int a = 0; a < N; a++) {
        R d = R(0.0);
        if (vd) {
          const R ph = F[a][i][j + CO];
          if ((ph + d) < R(0.0)) d += fabs(d + ph);
        }
        sm.DP[a][e] = d;
      }
    }
  }
  __syncthreads();
  const int nact = sm.nlist;
  hook();
  if (ANISO && nact > 0) {
    /* only the faces of active ring cells are read by ring_dphi: list them,
     * then compute them spread over the CTA */
    for (int e = threadIdx.x; e < IFT; e += NT) {
      bool need;
      if (e < IXF) {
        const int fi = e / (TY + 2), fj = e - fi * (TY + 2) + 1;
        /* ring cells (fi-1, fj-1) and (fi, fj-1) */
        need = (fi >= 1 && sm.ACT[LI(fi - 1, fj - 1)]) || (fi < SH && sm.ACT[LI(fi, fj - 1)]);
      } else {
        const int f = e - IXF, fi = f / (TY + 3) + 1, fj = f - (fi - 1) * (TY + 3);
        /* ring cells (fi-1, fj-1) and (fi-1, fj) */
        need = (fj >= 1 && sm.ACT[LI(fi - 1, fj - 1)]) || (fj < SW && sm.ACT[LI(fi - 1, fj)]);
      }
      if (need) sm.FLIST[atomicAdd(&sm.nflist, 1)] = (short)e;
    }
    __syncthreads();
    const int nf = sm.nflist;
    for (int q = threadIdx.x; q < nf; q += NT) {
      const int e = sm.FLIST[q];
      if (e < IXF) {
        const int fi = e / (TY + 2), fj = e - fi * (TY + 2) + 1;
        ring_face_terms<R, N, K>(D, F, sm.w.T, true, fi, fj, e);
      } else {
        const int f = e - IXF, fi = f / (TY + 3) + 1, fj = f - (fi - 1) * (TY + 3);
        ring_face_terms<R, N, K>(D, F, sm.w.T, false, fi, fj, e);
      }
    }
    __syncthreads();
  }
  for (int q = threadIdx.x; q < nact; q += NT) {
    const int e = sm.LIST[q];
    const int ri = e / SW, rj = e - ri * SW;
    R d[N];
    ring_dphi<R, N, K, ANISO>(D, F, sm, ri, rj, sm.ACT[e], d, D.tgrad ? ld_step(tpf + y0 - 1 + rj + 3) : 0.0);
#pragma unroll
    for (int a = 0; a < N; a++) sm.DP[a][e] = d[a];
  }
  __syncthreads();   /* the face-term cache is dead from here: its space holds the update's arrays */
  if (threadIdx.x == 0) {
    sm.nlist = 0;    /* for the next tile */
    sm.nflist = 0;
  }

#define PR(a, e) F[a][(e) / SW + 1][(e) % SW + 1 + CO]
#define MR(k, e) F[N + (k)][(e) / SW + 1][(e) % SW + 1 + CO]
  /* ---- per-cell quantities of the ring region */
  for (int e = threadIdx.x; e < SS; e += NT) {
    R p[N], mm[K];
#pragma unroll
    for (int a = 0; a < N; a++) p[a] = PR(a, e);
#pragma unroll
    for (int k = 0; k < K; k++) mm[k] = MR(k, e);
    R Ec[N][K];
    /* the ghosted column of ring cell e (cells past my+1 are not needed: clamped) */
    if (D.tgrad) e_at<R, N, K>(D, ld_step(tcc + min(y0 - 1 + e % SW + 3, g.my + 5)), Ec);
#pragma unroll
    for (int a = 0; a < N; a++) {
      R hv = h<R, N>(p, a);
      sm.w.u.H[a][e] = hv;
#pragma unroll
      for (int k = 0; k < K; k++)
        sm.w.u.CM[a][k][e] = D.tgrad ? c_muE<R, K>(D, Ec[a], mm, a, k) : c_mu<R, K>(D, mm, a, k);
      if (a < L)
        sm.w.u.SP[a][e] =
            (p[a] * (R(1.0) - p[a]) > R(0.0)) ? p[a] * (R(1.0) - hv) / (sqrt(p[a] * (R(1.0) - p[a]))) : R(0.0);
    }
#pragma unroll
    for (int k = 0; k < K; k++)
#pragma unroll
      for (int l = 0; l < K; l++) sm.w.u.DD[k][l][e] = Dcell<R, N, K>(D, p, k, l);
  }
  __syncthreads();

#define PRIJ(a, i, j) F[a][(i) + 1][(j) + 1 + CO]
  /* ---- faces of the tile: anti-trapping current and diffusion flux products */
  for (int e = threadIdx.x; e < NXF + NYF; e += NT) {
    const bool xface = e < NXF;
    int fi, fj, i1, j1, fidx;
    if (xface) { fi = e / TY; fj = e - fi * TY + 1; i1 = fi + 1; j1 = fj; fidx = e; }
    else { int f = e - NXF; fi = f / (TY + 1) + 1; fj = f - (fi - 1) * (TY + 1); i1 = fi; j1 = fj + 1; fidx = f; }
    const int c0 = LI(fi, fj), c1 = LI(i1, j1);
    R gr[N], cn[N];
#pragma unroll
    for (int a = 0; a < N; a++) {
      if (xface) {
        gr[a] = divx(PRIJ(a, i1, j1) - PRIJ(a, fi, fj), D);
        cn[a] = R(0.5) * (div2y(PRIJ(a, fi, fj + 1) - PRIJ(a, fi, fj - 1), D) +
                          div2y(PRIJ(a, i1, fj + 1) - PRIJ(a, i1, fj - 1), D));
      } else {
        gr[a] = divy(PRIJ(a, i1, j1) - PRIJ(a, fi, fj), D);
        R gc0 = R(0.5) * (divx(PRIJ(a, fi + 1, fj) - PRIJ(a, fi, fj), D) + divx(PRIJ(a, fi, fj) - PRIJ(a, fi - 1, fj), D));
        R gc1 = R(0.5) * (divx(PRIJ(a, fi + 1, j1) - PRIJ(a, i1, j1), D) + divx(PRIJ(a, i1, j1) - PRIJ(a, fi - 1, j1), D));
        cn[a] = R(0.5) * (gc0 + gc1);
      }
    }
    R jat[K];
#pragma unroll
    for (int k = 0; k < K; k++) jat[k] = R(0.0);
    /* calculate_fluxes_concentration.h:65: no y-current where gidy is 0 or MESH_Y-2 */
    const bool yskip = !xface && ((y0 - 1 + fj) + 3 == g.my - 2);
    R nl = R(-1.0);
#pragma unroll
    for (int a = 0; a < L; a++) {
      const R s2 = cn[a] * cn[a] + gr[a] * gr[a];
      if (s2 != R(0.0) && !yskip) {
        const R ng = sqrt(s2);
        if (nl < R(0.0)) nl = sqrt(cn[L] * cn[L] + gr[L] * gr[L]);
        R sp = gr[a] * gr[L];
        sp += cn[a] * cn[L];
        if (nl > R(0.0)) sp /= (nl * ng);
#pragma unroll
        for (int k = 0; k < K; k++) {
          R cl1 = sm.w.u.CM[L][k][c1], cl0 = sm.w.u.CM[L][k][c0];
          R cs1 = sm.w.u.CM[a][k][c1], cs0 = sm.w.u.CM[a][k][c0];
          R bracket;
          if (D.obstacle)
            bracket = sm.w.u.SP[a][c1] * (cl1 - cs1) * sm.DP[a][c1] + sm.w.u.SP[a][c0] * (cl0 - cs0) * sm.DP[a][c0];
          else
            bracket = (cl1 - cs1) * sm.DP[a][c1] + (cl0 - cs0) * sm.DP[a][c0];
          jat[k] += D.atf[a][k] * fabs(sp) * (D.obstacle ? R(0.5) : D.well_half) * bracket * gr[a] / ng;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (xface) sm.w.u.JX[k][fidx] = jat[k];
      else sm.w.u.JY[k][fidx] = jat[k];
#pragma unroll
      for (int l = 0; l < K; l++) {
        R dm = (sm.w.u.DD[k][l][c1] + sm.w.u.DD[k][l][c0]) * R(0.5);
        R gm = xface ? divx(MR(l, c1) - MR(l, c0), D) : divy(MR(l, c1) - MR(l, c0), D);
        if (xface) sm.w.u.FX[k][l][fidx] = dm * gm;
        else sm.w.u.FY[k][l][fidx] = dm * gm;
      }
    }
  }
  __syncthreads();

  /* ---- per cell: mu update, phi commit */
  const int tx = threadIdx.x / TY, ty = threadIdx.x - (threadIdx.x / TY) * TY;
  const int x = x0 + tx, y = y0 + ty, i = tx + 1, j = ty + 1, c = LI(i, j);
  if (x < g.mx && y < g.my) {
    R ph[N], m[K];
#pragma unroll
    for (int a = 0; a < N; a++) { ph[a] = PRIJ(a, i, j); dp[a] = sm.DP[a][c]; }
#pragma unroll
    for (int k = 0; k < K; k++) m[k] = MR(k, c);
    commit_cell<R, N, K>(D, sm.w.u.FX, sm.w.u.FY, sm.w.u.JX, sm.w.u.JY, sm.w.u.CM, sm.w.u.H, i, j, x, y, ph, dp, m,
                         nph, nm, dmu, st);
  }
#undef PRIJ
#undef PR
#undef MR
}
#undef FS_
#undef FA
#undef FB

}  // namespace gpd
