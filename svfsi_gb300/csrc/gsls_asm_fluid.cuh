// FLUID3D_M + FLUID3D_C (Code/Source/svFSI/FLUID.f:192-560, 813-1084) for
// P1-P1 tet4 with VMS stabilisation, one element per thread, with the
// constant, Carreau-Yasuda or Casson viscosity of GETVISCOSITY
// (FLUID.f:1690-1739).  Included by gsls_assemble.cu (needs AsmArgs,
// c_rule, adj_det3, kAsmThreads).
//
// Same quantities as the reference, arranged for GB300:
//  * the momentum and continuity passes of CONSTRUCT_FLUID run over the same
//    four Gauss points with the same basis (GETTHOODFS, FS.f:270-286) and
//    write disjoint entries, so they are fused into one point loop;
//  * tet4 gradients are constant and the second derivatives vanish, so
//    uxx, d2u2, es_x, mu_x and rS are zero; the shear rate, mu and mu_g are
//    element constants, and the viscosity model adds
//    4 wl mu_g esNx_i(a) esNx_j(b) to Kuu (zero for constant viscosity);
//  * the residual (u, ud, p, tauM, tauC, tauB, up, lR) is FP64 at every Gauss
//    point; the tangent runs in TT and is rebuilt per block (a,b) from factors
//    accumulated over the points:
//      Kuu(i,j) = wl [4 mu Nx_i(b)Nx_j(a) + (sum tauC) Nx_i(a)Nx_j(b) + d_ij S_ab]
//      S_ab     = 4 mu Nx_a.Nx_b + rho amd M_ab
//                 + sum_g [rho^2 tauM uaNx_a (uNx_b + amd N_b)
//                          + rho N_a (uNx_b + upNx_b) + tauB upNx_a upNx_b]
//      Kup(i)   = -wl [Nx_i(a) Ns_b - rho Nx_i(b) sum_g tauM uaNx_a]
//      Kpu(j)   =  wl [Ns_a Nx_j(b) + rho Nx_j(a) sum_g tauM (uNx_b + amd N_b)]
//      Kpp      =  wl (sum tauM) Nx_a.Nx_b
//    which is the reference's per-point sum with updu = -rho uNx d_ij.
//
// The element is bound by the FP64 pipe (0.51 T FMA/s), so its FP64 work is
// cut by identities of the tet4 rule, which change only the rounding:
//  * N_a(g) = t + (s - t) d_ag: point values are t sum_a y_a + (s - t) y_g, and
//    sums over the points of N_a(g) f_g are t sum_g f_g + (s - t) f_a;
//  * sum_a Nx_a = 0: every quantity f.Nx_a, and every sum of them, is formed
//    for three nodes and is minus their sum at the fourth (not in an FP32
//    tangent, see below);
//  * x.K.x = sum_{a<3} (x.Nx_a)^2 for the metric tensor K = sum_{a<3} Nx_a Nx_a^T;
//  * div-free scalars: 1/rho, amd, 4 (ctM/dt)^2 come from the host, tauM,
//    tauC and tauB from one rsqrt each instead of roots and divisions.
// An FP32 tangent forms u.Nx and up.Nx of all four nodes in FP64 and carries
// all 4 x 4 sums: minus the sum of three rounded values has the error of the
// largest of them, on a flat element many times the fourth.
// FP64 assembly of the h = 0.04 cylinder (371,520 tets): 2.87 ms before, 1.38
// ms with these and the element buffer (3.3 ms with these and the colour
// scatter).
#pragma once

namespace gsls {

// GETVISCOSITY (FLUID.f:1690-1739) for the Carreau-Yasuda and Casson models:
// mu and mu_x = d mu / d gamma at shear rate gam (Casson raises gam to its
// threshold lam first)
__device__ __forceinline__ void visc_model(const AsmArgs &A, double &gam, double &mu,
                                           double &mu_x) {
  if (A.viscType == GSLS_VISC_CY) {
    const double mi = A.mu_f, mo = A.mu_o, lam = A.vlam, a = A.va, n = A.vn;
    double T1 = 1.0 + pow(lam * gam, a);
    double T2 = pow(T1, (n - 1.0) / a);
    mu = mi + (mo - mi) * T2;
    T1 = T2 / T1;
    T2 = pow(lam, a) * pow(gam, a - 1.0) * T1;
    mu_x = (mo - mi) * (n - 1.0) * T2;
  } else {
    const double mi = A.mu_f, lam = A.vlam;
    double mo;
    if (gam < lam) {
      mo = A.mu_o / sqrt(lam);
      gam = lam;
    } else {
      mo = A.mu_o / sqrt(gam);
    }
    mu = (mi + mo) * (mi + mo);
    mu_x = 2.0 * mo * (mo + mi) / gam;
  }
}

// NN: a shear-rate dependent viscosity (Carreau-Yasuda or Casson); the
// constant-viscosity kernel carries none of its terms
template <class TT, bool NN>
__global__ void __launch_bounds__(kAsmThreads) k_asm_fluid(AsmArgs A) {
  extern __shared__ __align__(16) unsigned char asm_smem[];
  const EmitAt E = emit_at(A, asm_smem, emit_bytes<TT, 4>(), sizeof(TT) * 256, 4);
  const int e = A.el0 + min((int)(blockIdx.x * blockDim.x + threadIdx.x), A.nColorEl - 1);
  const int4 nd = A.ien[e];
  const int n4[4] = {nd.x, nd.y, nd.z, nd.w};
  const int tD = A.tDof, s0 = A.s;

  // ---- geometry (GNN with ks, FP64, precomputed per mesh): xiX(a,i) = Nx(i,a)
  double Nx[3][4], kk, trk;
  const double w = c_rule.w * load_geo(A, e, Nx);
  load_metric(A, e, kk, trk);

  // ---- nodal values and element-constant gradients (FP64)
  double yl[4][4], al[4][3];
#pragma unroll
  for (int a = 0; a < 4; a++) {
    const size_t k = (size_t)n4[a] * tD + s0;
#pragma unroll
    for (int c = 0; c < 4; c++) yl[a][c] = __ldg(A.Yg + k + c);
#pragma unroll
    for (int c = 0; c < 3; c++) al[a][c] = __ldg(A.Ag + k + c);
  }
  double ux[3][3], px[3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
#pragma unroll
    for (int j = 0; j < 3; j++)
      ux[i][j] = Nx[i][0] * yl[0][j] + Nx[i][1] * yl[1][j] + Nx[i][2] * yl[2][j] + Nx[i][3] * yl[3][j];
    px[i] = Nx[i][0] * yl[0][3] + Nx[i][1] * yl[1][3] + Nx[i][2] * yl[2][3] + Nx[i][3] * yl[3][3];
  }
  const double divU = ux[0][0] + ux[1][1] + ux[2][2];
  double es[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) es[i][j] = ux[i][j] + ux[j][i];

  // shear rate (2 e_ij e_ij)^(1/2), FLUID.f:358-373, and the viscosity
  double mu = A.mu_f, mu_g = 0.0;
  if (NN) {
    double gam = 0.0;
#pragma unroll
    for (int j = 0; j < 3; j++)
#pragma unroll
      for (int i = 0; i < 3; i++) gam += es[i][j] * es[i][j];
    gam = sqrt(0.5 * gam);
    double mu_x;
    visc_model(A, gam, mu, mu_x);
    // ISZERO (MATFUN.f:763-780): |x| < eps^2
    mu_g = (fabs(gam) < 4.930380657631324e-32) ? 0.0 : mu_x / gam;
  }
  const double rho = A.rho, irho = A.fl_irho;
  const double wl = w * A.fl_T1, wr = w * rho;
  const double nu = mu * irho;
  const double kTS = A.fl_kT + A.ctC * kk * (nu * nu);
  const double rtrK = rho / trk;

  // point values: rt sum_a + rd (value at node g)
  const double rt = c_rule.N[0][1], rd = c_rule.N[0][0] - c_rule.N[0][1];
  double uS[3], aS[3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    uS[i] = rt * ((yl[0][i] + yl[1][i]) + (yl[2][i] + yl[3][i]));
    aS[i] = rt * ((al[0][i] + al[1][i]) + (al[2][i] + al[3][i])) - A.fb[i];
  }
  const double pS = rt * ((yl[0][3] + yl[1][3]) + (yl[2][3] + yl[3][3]));

  // sums over the points: of rV2, pa and, for the first three nodes, of the
  // gradient part of lR (gR) and of up.Nx_a (sU); lN: rd rV2 at node g
  double vS[3] = {0, 0, 0}, paS = 0.0, gR[3][3], sU[3] = {0, 0, 0}, lN[4][3];
  // tangent factors (of the first NA nodes): Q = sum tauM uaNx, QU = sum tauM
  // uNx, UA = sum uaNx, H = the two quadratic sums of S_ab; q2[a][g] = (tauM
  // uaNx_a) and u2[g][b] = uaNx_b at point g, tMg = tauM at point g
  constexpr int NA = sizeof(TT) == 4 ? 4 : 3;
  const TT rh = TT(rho), rh2 = rh * rh, md = TT(A.fl_amd);
  TT SC = TT(0), ST = TT(0), Q[NA], QU[NA], UA[NA], H[NA][NA], q2[NA][4], u2[4][NA], tMg[4];
#pragma unroll
  for (int a = 0; a < NA; a++) {
    Q[a] = QU[a] = UA[a] = TT(0);
#pragma unroll
    for (int b = 0; b < NA; b++) H[a][b] = TT(0);
  }
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) gR[a][b] = 0.0;
#pragma unroll
  for (int g = 0; g < 4; g++) {
    double u[3], uN[3], rV[3], up[3], upN[3];
#pragma unroll
    for (int i = 0; i < 3; i++) u[i] = uS[i] + rd * yl[g][i];
    const double pr = pS + rd * yl[g][3];
#pragma unroll
    for (int a = 0; a < 3; a++) uN[a] = u[0] * Nx[0][a] + u[1] * Nx[1][a] + u[2] * Nx[2][a];
    const double X = kTS + uN[0] * uN[0] + uN[1] * uN[1] + uN[2] * uN[2];
    const double rX = rsqrt(X);
    const double tauM = rX * irho, tauC = X * rX * rtrK;
#pragma unroll
    for (int j = 0; j < 3; j++) {
      rV[j] = (aS[j] + rd * al[g][j]) + u[0] * ux[0][j] + u[1] * ux[1][j] + u[2] * ux[2][j];
      up[j] = -tauM * (rho * rV[j] + px[j]);
    }
#pragma unroll
    for (int a = 0; a < 3; a++) upN[a] = up[0] * Nx[0][a] + up[1] * Nx[1][a] + up[2] * Nx[2][a];
    double tB2 = upN[0] * upN[0] + upN[1] * upN[1] + upN[2] * upN[2];
    // ISZERO (MATFUN.f:763-780): |x| < eps^2
    if (fabs(tB2) < 4.930380657631324e-32) tB2 = 2.220446049250313e-16;
    const double tauB = rho * rsqrt(tB2);
    paS += pr - tauC * divU;
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const double q = up[0] * ux[0][j] + up[1] * ux[1][j] + up[2] * ux[2][j];
      const double rV2 = rV[j] + q, rB = tauB * q;
      vS[j] += rV2;
      lN[g][j] = rV2;
      // sum_i Nx_i(a) (rB_j up_i - rho up_j ua_i), a < 3
      const double rup = rho * up[j];
#pragma unroll
      for (int a = 0; a < 3; a++) gR[a][j] += rB * upN[a] - rup * (uN[a] + upN[a]);
    }
    const TT tM = TT(tauM), tB = TT(tauB);
    SC += TT(tauC);
    ST += tM;
    tMg[g] = tM;
    TT un[NA], pn[NA];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      sU[a] += upN[a];
      un[a] = TT(uN[a]);
      pn[a] = TT(upN[a]);
    }
    if constexpr (NA == 4) {
      un[3] = TT(u[0] * Nx[0][3] + u[1] * Nx[1][3] + u[2] * Nx[2][3]);
      pn[3] = TT(up[0] * Nx[0][3] + up[1] * Nx[1][3] + up[2] * Nx[2][3]);
    }
#pragma unroll
    for (int a = 0; a < NA; a++) {
      const TT ua = un[a] + pn[a], ta = tM * ua;
      Q[a] += ta;
      QU[a] += tM * un[a];
      UA[a] += ua;
      q2[a][g] = ta;
      u2[g][a] = ua;
      const TT c1 = rh2 * ta, c3 = tB * pn[a];
#pragma unroll
      for (int b = 0; b < NA; b++) H[a][b] += c1 * un[b] + c3 * pn[b];
    }
  }
  // lR(a,j) = wr (rt sum_g rV2_j + rd rV2_j(a)) + w [4 mu es.Nx_a + gR - paS Nx_a]_j,
  // lR(a,4) = w (Ns_a divU - sum_g up.Nx_a); the bracket sums to zero over a
  __align__(16) double lR[4][4];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    double s4 = 0.0;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const double v =
          gR[a][j] - paS * Nx[j][a] +
          4.0 * mu * (Nx[0][a] * es[0][j] + Nx[1][a] * es[1][j] + Nx[2][a] * es[2][j]);
      s4 -= v;
      lR[a][j] = w * v;
    }
    lR[3][j] = w * s4;
#pragma unroll
    for (int a = 0; a < 4; a++) lR[a][j] += wr * (rt * vS[j] + rd * lN[a][j]);
  }
  const double wdN = w * c_rule.Ns[0] * divU;
#pragma unroll
  for (int a = 0; a < 3; a++) lR[a][3] = wdN - w * sU[a];
  lR[3][3] = wdN + w * (sU[0] + sU[1] + sU[2]);

  emit_res<4>(E, &lR[0][0]);

  // ---- tangent (TT), everything scaled by wl
  const TT wlt = TT(wl), trt = TT(rt), trd = TT(rd), ns = TT(c_rule.Ns[0]);
  const TT wmu4 = wlt * TT(4.0 * mu), wSC = wlt * SC, wST = wlt * ST, wNs = wlt * ns,
           wrh = wlt * rh;
  TT Nxa[3][4];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int a = 0; a < 4; a++) Nxa[i][a] = TT(Nx[i][a]);
  // wl (G2 + G3 + H)_ab of S_ab: G2 = rho^2 amd sum_g tauM uaNx_a N_b, G3 = rho
  // sum_g N_a uaNx_b
  const TT w2 = wlt * rh2 * md;
  TT S[4][4];
#pragma unroll
  for (int a = 0; a < NA; a++)
#pragma unroll
    for (int b = 0; b < 4; b++) S[a][b] = w2 * (trt * Q[a] + trd * q2[a][b]);
  if constexpr (NA == 3) {
#pragma unroll
    for (int b = 0; b < 4; b++) S[3][b] = -(S[0][b] + S[1][b] + S[2][b]);
  }
#pragma unroll
  for (int a = 0; a < 4; a++) {
    TT s4 = TT(0);
#pragma unroll
    for (int b = 0; b < NA; b++) {
      const TT v = wrh * (trt * UA[b] + trd * u2[a][b]);
      S[a][b] += v;
      s4 -= v;
    }
    if constexpr (NA == 3) S[a][3] += s4;
  }
  if constexpr (NA == 4) {
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = 0; b < 4; b++) S[a][b] += wlt * H[a][b];
  } else {
    TT h3[4] = {TT(0), TT(0), TT(0), TT(0)};
#pragma unroll
    for (int a = 0; a < 3; a++) {
      TT s4 = TT(0);
#pragma unroll
      for (int b = 0; b < 3; b++) {
        const TT v = wlt * H[a][b];
        S[a][b] += v;
        s4 -= v;
        h3[b] -= v;
      }
      S[a][3] += s4;
      h3[3] -= s4;
    }
#pragma unroll
    for (int b = 0; b < 4; b++) S[3][b] += h3[b];
  }
  // Q and Vc = sum_g tauM (uNx + amd N) of all four nodes, times wl rho
  TT Qw[4], Vw[4];
#pragma unroll
  for (int a = 0; a < 4; a++) {
    const TT qa = a < NA ? Q[a < NA ? a : 0] : -(Q[0] + Q[1] + Q[2]);
    const TT qu = a < NA ? QU[a < NA ? a : 0] : -(QU[0] + QU[1] + QU[2]);
    Qw[a] = wrh * qa;
    Vw[a] = wrh * (qu + md * (trt * ST + trd * tMg[a]));
  }
  // esNx_i(a) = sum_k es(k,i) Nx_k(a) for the term 4 mu_g esNx_i(a) esNx_j(b)
  const TT g4 = wlt * TT(4.0 * mu_g);
  TT eN[3][4];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int a = 0; a < 4; a++)
      eN[i][a] = NN ? TT(es[0][i] * Nx[0][a] + es[1][i] * Nx[1][a] + es[2][i] * Nx[2][a]) : TT(0);
  const TT wrM0 = wrh * md;
#pragma unroll
  for (int a = 0; a < 4; a++) {
    __align__(16) TT row[64];
    TT mN[3], cN[3], nN[3];  // 4 mu wl Nx(a), wl sum tauC Nx(a), -wl Ns Nx(a)
#pragma unroll
    for (int i = 0; i < 3; i++) {
      mN[i] = wmu4 * Nxa[i][a];
      cN[i] = wSC * Nxa[i][a];
      nN[i] = -wNs * Nxa[i][a];
    }
#pragma unroll
    for (int b = 0; b < 4; b++) {
      const TT NxNx = Nxa[0][a] * Nxa[0][b] + Nxa[1][a] * Nxa[1][b] + Nxa[2][a] * Nxa[2][b];
      const TT Sab = wmu4 * NxNx + (wrM0 * TT(c_rule.M[a][b]) + S[a][b]);
      TT *v = row + b * 16;
#pragma unroll
      for (int i = 0; i < 3; i++) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
          v[i * 4 + j] = mN[j] * Nxa[i][b] + (cN[i] * Nxa[j][b] + (i == j ? Sab : TT(0)));
          if (NN) v[i * 4 + j] += (g4 * eN[i][a]) * eN[j][b];
        }
        v[i * 4 + 3] = Qw[a] * Nxa[i][b] + nN[i];
        v[12 + i] = Vw[b] * Nxa[i][a] + wNs * Nxa[i][b];
      }
      v[15] = wST * NxNx;
    }
    emit_row<TT, 4>(E, a, row);
  }
}

}  // namespace gsls
