// The reverse sweep of one point's algebra: the cotangents of the right-hand side's nonlinear inputs.
//
// With lambda the cotangent of du at the point, the scalar
//   Phi = W (sum_v lambda_h,v d_t h_v + lin + sum_v lambda_Pi,v msrc_v) - rho sum_v lambda_h,v (h_v - target_v)
// is a function of h, d_i h and Pi through the metric, the coefficient divergences, the gauge source and the
// reduced source (metric_quantities, metric_divergences, ks_gauge_source, gh_source), whose stencil sums
// against lambda_Pi (lin's) are given. adjoint_phi_reverse evaluates it forwards once and then runs
// backwards through the same steps, each step's transpose in closed form: about 7,000 FP64 operations
// where 53 forward-mode passes (one per input and parameter) took about 400,000.
//
// A symmetric matrix's cotangent is kept as the symmetric matrix Y with d Phi = sum_ab Y_ab dA_ab over all
// (a, b): the derivative with respect to a packed component is Y on the diagonal and 2 Y off it (pmul).
#pragma once
#include "algebra.cuh"

namespace tgh {

TGH_HD constexpr double pmul(int n) { return prow(n) == pcol(n) ? 1.0 : 2.0; }

struct PhiInputs {
  const double *h, *d1, *dth, *Pi;        // h, d_i h (3 x 10), d_t h, Pi
  double eh, ih, ih2;
  const double *lh, *lP;                  // lambda of d_t h and of d_t Pi
  const double *P1, *P2;                  // sum_v lP_v of the first differences of Pi, the second ones of h
  double P0, PKO;                         // ... of Pi, of Pi's dissipation
  double W, rho;                          // the layer's weight and relaxation (1 and 0 outside)
  double g0;                              // the damping rate
  const double *Hl, *dHs;                 // the sampled gauge source: H_a, d_a H_b + d_b H_a packed
};
struct PhiCotangents {
  double h[NC], d1[3 * NC], dth[NC];      // of h, d_i h and (as passed on to Pi and the dissipation) d_t h
  double g0;                              // of the damping rate
  double phiP;                            // lin + sum_v lP_v msrc_v
};

// U Y U for symmetric U, Y
TGH_HD void sandwich(const double* U, const double* Y, double* out) {
  for (int m = 0; m < 4; ++m) {
    double e[4];
    for (int c = 0; c < 4; ++c) {
      double s = 0.0;
      for (int x = 0; x < 4; ++x) s = fma(U[pidx(m, x)], Y[pidx(x, c)], s);
      e[c] = s;
    }
    for (int n = m; n < 4; ++n) {
      double s = 0.0;
      for (int y = 0; y < 4; ++y) s = fma(e[y], U[pidx(y, n)], s);
      out[pidx(m, n)] = s;
    }
  }
}
// sum over all (a, b) of A_ab B_ab
TGH_HD double pdot(const double* A, const double* B) {
  double s = 0.0;
#pragma unroll
  for (int n = 0; n < NC; ++n) s = fma(pmul(n) * A[n], B[n], s);
  return s;
}

static __host__ __device__ TGH_NOINLINE void adjoint_phi_reverse(const Case& cs, const PhiInputs& in,
                                                                 PhiCotangents& out) {
  // ---- forwards ----
  Coef<double> C;
  metric_quantities(in.h, C);
  const double* U = C.gu;
  const double it = 1.0 / U[0], al = C.alpha, rg = C.sqrtg, as = al * rg;
  const double* D[4] = {in.dth, in.d1, in.d1 + NC, in.d1 + 2 * NC};
  double Cu[4][NC], V[4], Gup[4];
  for (int a = 0; a < 4; ++a) sandwich(U, D[a], Cu[a]);
  for (int x = 0; x < 4; ++x) {
    double s = -0.5 * pdot(U, D[x]);
    for (int a = 0; a < 4; ++a)
      for (int b = 0; b < 4; ++b) s = fma(U[pidx(a, b)], D[a][pidx(x, b)], s);
    V[x] = s;
  }
  for (int c = 0; c < 4; ++c) {
    double s = 0.0;
    for (int x = 0; x < 4; ++x) s = fma(U[pidx(c, x)], V[x], s);
    Gup[c] = s;
  }
  // the gauge source
  const bool has_h = cs.gauge != TGH_GAUGE_NONE, ks = has_h && cs.gauge != TGH_GAUGE_SAMPLED;
  double H[4] = {0, 0, 0, 0}, wv[4], K = 0, sw = 0, root = 0, iD = 0, iroot = 0;
  if (ks) {
    for (int a = 0; a < 4; ++a) {
      wv[a] = 0.0;
      for (int b = 0; b < 4; ++b) wv[a] = fma(in.h[pidx(a, b)], cs.ksU[b], wv[a]);
    }
    for (int a = 0; a < 4; ++a) {
      K = fma(cs.ksU[a], wv[a], K);
      sw = fma(cs.ksS[a], wv[a], sw);
    }
    const double rad = cs.ksM * cs.ksM - sw * sw;
    root = rad > 0.0 ? dsqrt(rad) : 0.0;
    iroot = root > 0.0 ? 1.0 / root : 0.0;
    iD = 1.0 / (cs.ksM + root);
    for (int a = 0; a < 4; ++a) H[a] = -K * iD * wv[a];
  } else if (has_h) {
    for (int a = 0; a < 4; ++a) H[a] = in.Hl[a];
  }

  // ---- backwards, W applied at the end: msrc = -as S, S = sum of the terms below; X_ab the cotangent of S_ab ----
  double Db[4][NC], Ub[NC], X[NC], Hb[4], Vb[4], Gb[4], SX = 0.0;  // SX = sum_ab X_ab S_ab
  double alb = 0.0, rgb = 0.0, asb = 0.0;
  for (int n = 0; n < NC; ++n) {
    X[n] = -as * in.lP[n] / pmul(n);
    Ub[n] = 0.0;
    for (int a = 0; a < 4; ++a) Db[a][n] = 0.0;
  }
  for (int a = 0; a < 4; ++a) Hb[a] = Vb[a] = Gb[a] = 0.0;
  double hd[NC];  // packed derivatives with respect to h that do not pass through g^-1
  for (int n = 0; n < NC; ++n) hd[n] = 0.0;

  // - (d_a H_b + d_b H_a)
  double Kb = 0.0, swb = 0.0, iDb = 0.0, irb = 0.0, wb[4] = {0, 0, 0, 0};  // completed with H_a's cotangent below
  if (ks) {
    for (int k = 0; k < 4; ++k) {
      double dw[4], dK = 0.0, Sd = 0.0, s1 = 0.0, s2 = 0.0, q[4], dwb[4];
      for (int a = 0; a < 4; ++a) {
        dw[a] = 0.0;
        for (int b = 0; b < 4; ++b) dw[a] = fma(D[k][pidx(a, b)], cs.ksU[b], dw[a]);
        q[a] = -2.0 * X[pidx(k, a)];  // the cotangent of d_k H_a
        s1 = fma(q[a], wv[a], s1);
        s2 = fma(q[a], dw[a], s2);
      }
      for (int a = 0; a < 4; ++a) {
        dK = fma(cs.ksU[a], dw[a], dK);
        Sd = fma(cs.ksS[a], dw[a], Sd);
      }
      const double dD = -sw * Sd * iroot;
      SX += -iD * (dK * s1 + K * s2) + K * s1 * dD * iD * iD;
      const double dDb = K * s1 * iD * iD, dKb = -iD * s1, Sdb = -dDb * sw * iroot;
      Kb += -iD * s2 + s1 * dD * iD * iD;
      iDb += -(dK * s1 + K * s2) + 2.0 * K * s1 * dD * iD;
      swb -= dDb * Sd * iroot;
      irb -= dDb * sw * Sd;
      for (int a = 0; a < 4; ++a) {
        wb[a] += (K * dD * iD - dK) * iD * q[a];
        dwb[a] = -K * iD * q[a] + dKb * cs.ksU[a] + Sdb * cs.ksS[a];
      }
      for (int n = 0; n < NC; ++n)
        Db[k][n] += 0.5 * (dwb[prow(n)] * cs.ksU[pcol(n)] + dwb[pcol(n)] * cs.ksU[prow(n)]);
    }
  } else if (has_h) {
    SX -= pdot(X, in.dHs);
  }
  // - Gamma^c d_c g_ab
  for (int c = 0; c < 4; ++c) {
    const double xd = pdot(X, D[c]);
    SX -= Gup[c] * xd;
    Gb[c] -= xd;
    for (int n = 0; n < NC; ++n) Db[c][n] = fma(-Gup[c], X[n], Db[c][n]);
  }
  // C2 + C2^T, C2_ab = (C_a)^mn d_m g_nb; and C_a's cotangents, completed by the divergences below
  double Cb[4][NC];
  for (int a = 0; a < 4; ++a)
    for (int m = 0; m < 4; ++m)
      for (int n = m; n < 4; ++n) {
        double s = 0.0;
        for (int b = 0; b < 4; ++b) s = fma(X[pidx(a, b)], D[m][pidx(n, b)] + D[n][pidx(m, b)], s);
        Cb[a][pidx(m, n)] = s;  // 2 X_ab (D_m,nb + D_n,mb) / 2
      }
  for (int a = 0; a < 4; ++a) SX += pdot(Cb[a], Cu[a]);
  for (int m = 0; m < 4; ++m)
    for (int n = 0; n < 4; ++n)
      for (int b = n; b < 4; ++b) {
        double s = 0.0;
        for (int a = 0; a < 4; ++a)
          s += Cu[a][pidx(m, n)] * X[pidx(a, b)] + Cu[a][pidx(m, b)] * X[pidx(a, n)];
        Db[m][pidx(n, b)] += s;  // 2 (R_nb + R_bn) / 2
      }
  // -2 Gamma^x_ya Gamma^y_xb + 2 Gamma^c_ab H_c, Gamma^a_bc = g^ax L_x,bc
  {
    double G[4][NC];
    for (int n = 0; n < NC; ++n) {
      const int i = prow(n), j = pcol(n);
      double low[4];
      for (int x = 0; x < 4; ++x) low[x] = 0.5 * (D[i][pidx(x, j)] + D[j][pidx(x, i)] - D[x][n]);
      for (int a = 0; a < 4; ++a) {
        double s = 0.0;
        for (int x = 0; x < 4; ++x) s = fma(U[pidx(a, x)], low[x], s);
        G[a][n] = s;
      }
    }
    double GB[4][NC];  // cotangent of Gamma^x_ya, symmetric in (y, a)
    for (int x = 0; x < 4; ++x)
      for (int y = 0; y < 4; ++y)
        for (int a = y; a < 4; ++a) {
          double s = 0.0;
          for (int b = 0; b < 4; ++b) s += X[pidx(a, b)] * G[y][pidx(x, b)] + X[pidx(y, b)] * G[a][pidx(x, b)];
          GB[x][pidx(y, a)] = -2.0 * s;
        }
    for (int x = 0; x < 4; ++x) SX += 0.5 * pdot(GB[x], G[x]);  // quadratic: half of G . dPhi/dG
    if (has_h)
      for (int c = 0; c < 4; ++c) {
        const double xg = 2.0 * pdot(X, G[c]);
        SX += xg * H[c];
        Hb[c] += xg;
        for (int n = 0; n < NC; ++n) GB[c][n] = fma(2.0 * H[c], X[n], GB[c][n]);
      }
    // through Gamma = g^-1 L
    double LB[4][NC], L[4][NC];
    for (int n = 0; n < NC; ++n) {
      const int i = prow(n), j = pcol(n);
      for (int x = 0; x < 4; ++x) {
        L[x][n] = 0.5 * (D[i][pidx(x, j)] + D[j][pidx(x, i)] - D[x][n]);
        double s = 0.0;
        for (int c = 0; c < 4; ++c) s = fma(U[pidx(c, x)], GB[c][n], s);
        LB[x][n] = s;
      }
    }
    for (int c = 0; c < 4; ++c)
      for (int x = c; x < 4; ++x) Ub[pidx(c, x)] += 0.5 * (pdot(GB[c], L[x]) + pdot(GB[x], L[c]));
    for (int a = 0; a < 4; ++a)
      for (int n = 0; n < NC; ++n)
        Db[a][n] += 0.5 * (LB[prow(n)][pidx(a, pcol(n))] + LB[pcol(n)][pidx(a, prow(n))]) - 0.5 * LB[a][n];
  }
  // the damping: Z = t_a C_b + t_b C_a - (1 + gamma2) (t.C) g_ab, C = V + H
  double gb[NC];
  {
    double Cl[4], xc = 0.0, uc = 0.0;
    for (int a = 0; a < 4; ++a) {
      Cl[a] = V[a] + H[a];
      xc = fma(X[pidx(0, a)], Cl[a], xc);
      uc = fma(U[pidx(0, a)], Cl[a], uc);
    }
    const double tl = -al, tC = tl * uc, k2 = 1.0 + cs.g2, xg = pdot(X, C.g);
    out.g0 = 2.0 * tl * xc - k2 * tC * xg;
    SX += in.g0 * out.g0;
    const double tCb = -in.g0 * k2 * xg;
    alb -= in.g0 * 2.0 * xc + tCb * uc;
    for (int a = 0; a < 4; ++a) {
      const double cb = in.g0 * 2.0 * tl * X[pidx(0, a)] + tCb * tl * U[pidx(0, a)];
      Vb[a] += cb;
      if (has_h) Hb[a] += cb;
      Ub[pidx(0, a)] += (a == 0 ? 1.0 : 0.5) * tCb * tl * Cl[a];
    }
    for (int n = 0; n < NC; ++n) gb[n] = -in.g0 * k2 * tC * X[n];
  }
  // H_a of the closed-form source
  if (ks) {
    double t = 0.0;
    for (int a = 0; a < 4; ++a) {
      t = fma(Hb[a], wv[a], t);
      wb[a] -= K * iD * Hb[a];
    }
    Kb -= iD * t;
    iDb -= K * t;
    const double rootb = -iDb * iD * iD - irb * iroot * iroot;
    swb -= rootb * iroot * sw;  // root = sqrt(M^2 - sw^2)
    for (int a = 0; a < 4; ++a) wb[a] += Kb * cs.ksU[a] + swb * cs.ksS[a];
    for (int n = 0; n < NC; ++n)
      hd[n] = pmul(n) * 0.5 * (wb[prow(n)] * cs.ksU[pcol(n)] + wb[pcol(n)] * cs.ksU[prow(n)]);
  }
  // Gup = g^-1 V, V_x = g^ab d_a g_xb - g^ab d_x g_ab / 2
  for (int x = 0; x < 4; ++x)
    for (int c = 0; c < 4; ++c) Vb[x] = fma(U[pidx(c, x)], Gb[c], Vb[x]);
  for (int c = 0; c < 4; ++c)
    for (int x = c; x < 4; ++x) Ub[pidx(c, x)] += 0.5 * (Gb[c] * V[x] + Gb[x] * V[c]);
  for (int a = 0; a < 4; ++a)
    for (int n = 0; n < NC; ++n) {
      const int x = prow(n), b = pcol(n);
      Db[a][n] += 0.5 * (Vb[x] * U[pidx(a, b)] + Vb[b] * U[pidx(a, x)]) - 0.5 * Vb[a] * U[n];
    }
  for (int n = 0; n < NC; ++n) {
    const int a = prow(n), b = pcol(n);
    double s = 0.0;
    for (int x = 0; x < 4; ++x) s += Vb[x] * (0.5 * (D[a][pidx(x, b)] + D[b][pidx(x, a)]) - 0.5 * D[x][n]);
    Ub[n] += s;
  }
  // msrc = -as S
  asb += SX / as;

  // ---- lin: beta.P1 + divb P0 + divA.sd + A:P2 + KO ----
  double bb[3], gmb[6], itb = 0.0;  // cotangents of beta, gamma^ij (symmetric matrix) and 1 / g^tt
  double sd[3], lin = 0.0;
  const double db = in.P0;
  for (int i = 0; i < 3; ++i) {
    sd[i] = 0.0;
    for (int v = 0; v < NC; ++v) sd[i] = fma(in.lP[v], D[i + 1][v], sd[i]);
    bb[i] = in.ih * in.P1[i];
    lin = fma(C.beta[i], in.ih * in.P1[i], lin);
  }
  {
    const double* P2 = in.P2;
    const double q[6] = {P2[0], P2[3], P2[4], P2[1], P2[5], P2[2]};  // packed (xx, xy, xz, yy, yz, zz)
    double a2 = 0.0;
    for (int n = 0; n < 6; ++n) {
      a2 += (n == 0 || n == 3 || n == 5 ? 1.0 : 2.0) * C.gamu[n] * q[n];
      gmb[n] = in.ih2 * as * q[n];
    }
    asb += in.ih2 * a2;
    lin += in.ih2 * as * a2 + in.eh * in.PKO;
  }
  for (int i = 0; i < 3; ++i) {
    const double* c = Cu[i + 1];
    double* cb = Cb[i + 1];
    const double bi = C.beta[i], c0 = c[0], ci = c[pidx(0, i + 1)];
    // d_i beta^i
    const double dv = ci + bi * c0;
    lin = fma(dv * it, in.P0, lin);
    itb += dv * db;
    bb[i] += c0 * it * db;
    cb[pidx(0, i + 1)] += 0.5 * it * db;
    cb[0] += bi * it * db;
    // d_i (alpha sqrt(gamma)) gamma^ik + alpha sqrt(gamma) d_i gamma^ik, contracted with sd_k
    double tr = 0.0, e = 0.0, mb = 0.0, mc = 0.0;
    for (int j = 0; j < 3; ++j)
      for (int k = 0; k < 3; ++k) tr = fma(C.gamu[sidx3(j, k)], D[i + 1][pidx(j + 1, k + 1)], tr);
    const double fac = 0.5 * as * tr - 0.5 * al * al * al * c0 * rg;
    for (int k = 0; k < 3; ++k) {
      const double dA = sd[k], m = as * dA;
      const double ck = c[pidx(0, k + 1)], bk = C.beta[k];
      const double dg = -(c[pidx(i + 1, k + 1)] + bk * ci + bi * ck + bi * bk * c0);
      lin = fma(fac * C.gamu[sidx3(i, k)] + as * dg, sd[k], lin);
      e = fma(dA, C.gamu[sidx3(i, k)], e);
      gmb[sidx3(i, k)] += (i == k ? 1.0 : 0.5) * fac * dA;
      asb += dA * dg;
      cb[pidx(i + 1, k + 1)] -= (i == k ? 1.0 : 0.5) * m;
      cb[pidx(0, k + 1)] -= 0.5 * m * bi;
      bb[k] -= m * (ci + bi * c0);
      mb = fma(m, bk, mb);
      mc = fma(m, ck, mc);
    }
    cb[pidx(0, i + 1)] -= 0.5 * mb;
    cb[0] -= bi * mb;
    bb[i] -= mc + mb * c0;
    // fac = as tr / 2 - alpha^3 sqrt(gamma) c0 / 2
    alb += e * (0.5 * rg * tr - 1.5 * al * al * c0 * rg);
    rgb += e * (0.5 * al * tr - 0.5 * al * al * al * c0);
    cb[0] -= 0.5 * al * al * al * rg * e;
    const double trb = 0.5 * as * e;
    for (int j = 0; j < 3; ++j)
      for (int k = j; k < 3; ++k) {
        gmb[sidx3(j, k)] += trb * D[i + 1][pidx(j + 1, k + 1)];
        Db[i + 1][pidx(j + 1, k + 1)] += trb * C.gamu[sidx3(j, k)];
      }
  }
  out.phiP = lin + SX;
  out.g0 *= in.W;
  // C_a = g^-1 (d_a g) g^-1
  for (int a = 0; a < 4; ++a) {
    double s[NC], N[4][4];
    sandwich(U, Cb[a], s);
    for (int n = 0; n < NC; ++n) Db[a][n] += s[n];
    for (int x = 0; x < 4; ++x) {
      double e[4];
      for (int y = 0; y < 4; ++y) {
        e[y] = 0.0;
        for (int z = 0; z < 4; ++z) e[y] = fma(D[a][pidx(x, z)], U[pidx(z, y)], e[y]);
      }
      for (int y = 0; y < 4; ++y) {
        N[x][y] = 0.0;
        for (int z = 0; z < 4; ++z) N[x][y] = fma(e[z], Cb[a][pidx(z, y)], N[x][y]);
      }
    }
    for (int n = 0; n < NC; ++n) Ub[n] += N[prow(n)][pcol(n)] + N[pcol(n)][prow(n)];
  }
  // the packed derivatives of d_i h and d_t h; divA_k = d_i A^ik multiplies sd_k
  for (int k = 0; k < 3; ++k) {
    double dA = 0.0;
    for (int i = 0; i < 3; ++i) {
      const double* c = Cu[i + 1];
      const double bi = C.beta[i], bk = C.beta[k];
      double tr = 0.0;
      for (int j = 0; j < 3; ++j)
        for (int l = 0; l < 3; ++l) tr = fma(C.gamu[sidx3(j, l)], D[i + 1][pidx(j + 1, l + 1)], tr);
      const double fac = 0.5 * as * tr - 0.5 * al * al * al * c[0] * rg;
      dA += fac * C.gamu[sidx3(i, k)] -
            as * (c[pidx(i + 1, k + 1)] + bk * c[pidx(0, i + 1)] + bi * c[pidx(0, k + 1)] + bi * bk * c[0]);
    }
    for (int v = 0; v < NC; ++v) out.d1[k * NC + v] = fma(dA, in.lP[v], pmul(v) * Db[k + 1][v]);
  }
  // d_t h = beta.d h + (alpha / sqrt(gamma)) Pi + dissipation
  double adb = 0.0;
  for (int v = 0; v < NC; ++v) {
    const double gd = in.lh[v] + pmul(v) * Db[0][v];
    out.dth[v] = in.W * gd;
    for (int i = 0; i < 3; ++i) {
      bb[i] = fma(gd, D[i + 1][v], bb[i]);
      out.d1[i * NC + v] = in.W * fma(C.beta[i], gd, out.d1[i * NC + v]);
    }
    adb = fma(gd, in.Pi[v], adb);
  }
  alb += adb / rg + asb * rg;
  rgb += asb * al - adb * al / (rg * rg);

  // ---- the metric: alpha = (-g^tt)^(-1/2), beta^i = -g^ti / g^tt, gamma^ij = g^ij - g^ti g^tj / g^tt ----
  for (int i = 0; i < 3; ++i) {
    const double ui = U[pidx(0, i + 1)];
    itb -= ui * bb[i];
    double s = 0.0;
    for (int j = 0; j < 3; ++j) s = fma(gmb[sidx3(i, j)], U[pidx(0, j + 1)], s);
    itb -= ui * s;
    Ub[pidx(0, i + 1)] += 0.5 * (-it * bb[i] - 2.0 * it * s);
    for (int j = i; j < 3; ++j) Ub[pidx(i + 1, j + 1)] += gmb[sidx3(i, j)];
  }
  Ub[0] += 0.5 * al * al * al * alb - it * it * itb;
  double ug[NC];
  sandwich(U, Ub, ug);
  for (int n = 0; n < NC; ++n) {
    const int a = prow(n), b = pcol(n);
    double y = gb[n] - ug[n];
    if (a > 0 && b > 0) y += 0.5 * rg * rgb * C.gamu[sidx3(a - 1, b - 1)];
    out.h[n] = in.W * (pmul(n) * y + hd[n]) - in.rho * in.lh[n];
  }
}

}  // namespace tgh
