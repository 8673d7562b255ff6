// Hand-written adjoint of the broken-line fit: d(chi2_line + chi2_circle)/d(hits).
//
// Both broken-line systems are the stationarity conditions of a quadratic form
// in the corrections u: C = (1/2) Hessian(Q) and the right-hand side is w*Z, where
//   Q_line(u)   = sum_i w_i (Z_i - u_i)^2 + sum_kinks beta_i^2 / VB_i,
//   Q_circle(u) = same with the curvature correction u_N added to each kink,
// and the fit's chi2 is Q at the solution u*. By the envelope theorem
// d chi2 / d theta = dQ/d theta at fixed u*, so the backward pass needs no
// adjoint solve: it recomputes the forward fit (nothing is stored between the
// passes), takes the partial derivatives of Q with respect to the weights w,
// residuals Z, abscissae s or S and scattering variances VB, and propagates them
// by hand, in reverse order, through the line weights, the multiple-scattering
// model, the (s, z) rotation, the arc lengths and the fast-fit circle down to the
// hit coordinates. The chi2 is invariant under a common translation of the hits,
// so the hit-0 frame of the forward fit is kept and hit 0 receives minus the sum
// of the others' gradients.
//
// The backward pass divides almost nowhere: it reuses the forward pass's inverse segment lengths,
// scattering variances and radii, and its angles (the arc lengths and the slope give them back).
//
// Arithmetic is FP64 throughout (the gradient is checked against central finite
// differences and forward-mode derivatives at 1e-6 relative).
#pragma once
#include "bl_fit.cuh"

namespace pxl {
namespace bl {

// chi2 of the fit and its gradient with respect to the hit coordinates (grad[3][N])
template <int N>
BL_HD double chi2_adjoint(const double hits[3][N], const float ge[6][N], double B, double grad[3][N]) {
  using T = double;
  Geo<N, T> G;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    G.h0[a] = hits[a][0];
#pragma unroll
    for (int i = 0; i < N; ++i) G.p[a][i] = hits[a][i] - hits[a][0];
  }
  // ---------------------------------------------------------------- forward (recomputed)
  // The line system's partials are taken before the circle system is built, so that the two
  // systems' arrays are not live together.
  Prep<N, T> P;
  fast_fit<N, T>(G, P);
  prepare<N, T>(G, B, P);
  T wl[N], iv[N], hl[N - 1];
  Band<N, false> fl;
  double ul[N];
  inverse_variances<N, T>(P, iv);
  line_system<N, T>(ge, P, iv, wl, hl, fl, ul);
  const T m = P.slope, a = P.Rl[0][0], b = P.Rl[0][1];
  const T sig = 1.0 + m * m;
  const T* s = P.s;
  const T* S = P.S;
  const double iR = 1.0 / P.R;
  double chi2 = 0.0;

  // adjoint accumulators
  double gS[N] = {}, gs[N] = {}, gZl[N] = {}, gwl[N] = {}, gVB[N] = {}, gwc[N] = {}, gZc[N] = {};
  double grx[N] = {}, gry[N] = {}, gp[3][N] = {};
  double gm = 0.0, gR = 0.0, ga = 0.0, gb = 0.0;

  // ---------------------------------------------------------------- line chi2 partials
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const double r = P.Z[i] - ul[i];
    chi2 += wl[i] * r * r;
    gwl[i] += r * r;
    gZl[i] += 2.0 * wl[i] * r;
    if (i > 0 && i < N - 1) {
      const double e1 = (ul[i] - ul[i - 1]) * hl[i - 1], e2 = (ul[i] - ul[i + 1]) * hl[i];
      const double beta = -(e1 + e2), bv = beta * iv[i];
      chi2 += beta * bv;
      gVB[i] -= bv * bv;
      const double dd1 = e1 * hl[i - 1], dd2 = e2 * hl[i], gbeta = 2.0 * bv;
      gS[i] += gbeta * (dd1 - dd2);
      gS[i - 1] -= gbeta * dd1;
      gS[i + 1] += gbeta * dd2;
    }
  }
  // ---------------------------------------------------------------- line weights
  {
    const double tol = 1e-12;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      auto z = [&](float v) { return fabs(double(v)) < tol ? 0.0 : double(v); };
      const double V[3][3] = {{double(ge[0][i]), z(ge[1][i]), z(ge[3][i])}, {z(ge[1][i]), double(ge[2][i]), z(ge[4][i])},
                              {z(ge[3][i]), z(ge[4][i]), double(ge[5][i])}};
      const double in = P.irn[i], hx = P.rx[i] * in, hy = P.ry[i] * in;
      const double rj[3] = {-b * hy, b * hx, a};
      // w = 1 / (rj^T V rj): g_rj = -w^2 * 2 V rj * g_w
      const double gm22 = -gwl[i] * wl[i] * wl[i];
      double grj[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) grj[k] = 2.0 * gm22 * (V[k][0] * rj[0] + V[k][1] * rj[1] + V[k][2] * rj[2]);
      gb += grj[1] * hx - grj[0] * hy;
      ga += grj[2];
      const double bi = b * in;
      const double gn = bi * (grj[0] * hy - grj[1] * hx);
      grx[i] += grj[1] * bi + gn * hx;
      gry[i] += gn * hy - grj[0] * bi;
    }
  }
  // ---------------------------------------------------------------- circle system
  T VBc[N], ivc[N], Zc[N], rn[N], wc[N], hc[N - 1];
  Band<N, true> fc;
  double uc[N + 1];
  circle_system<N, T>(ge, G, P, iv, VBc, ivc, Zc, rn, wc, hc, fc, uc);
  // ---------------------------------------------------------------- circle chi2 partials
  double gsig = 0.0;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const double r = Zc[i] - uc[i];
    chi2 += wc[i] * r * r;
    gwc[i] += r * r;
    gZc[i] += 2.0 * wc[i] * r;
    if (i > 0 && i < N - 1) {
      const double e1 = (uc[i] - uc[i - 1]) * hc[i - 1], e2 = (uc[i] - uc[i + 1]) * hc[i];
      const double t = 0.5 * ((s[i + 1] - s[i - 1]) * uc[N]) - (e1 + e2), tv = t * ivc[i];
      chi2 += t * tv;
      const double gvbc = -tv * tv;
      gVB[i] += gvbc * sig;
      gsig += gvbc * P.VB[i];
      const double dd1 = e1 * hc[i - 1] + 0.5 * uc[N], dd2 = e2 * hc[i] + 0.5 * uc[N], gt = 2.0 * tv;
      gs[i] += gt * (dd1 - dd2);
      gs[i - 1] -= gt * dd1;
      gs[i + 1] += gt * dd2;
    }
  }
  gm += gsig * 2.0 * m;
  // circle weights w = |r|^2 / (r^T V r) (so 1 / (r^T V r) = w / |r|^2) and residuals Z = |r| - R
  {
    const double tol = 1e-12;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      auto z = [&](float v) { return fabs(double(v)) < tol ? 0.0 : double(v); };
      const double vxx = z(ge[0][i]), vxy = z(ge[1][i]), vyy = z(ge[2][i]);
      const double rx = P.rx[i], ry = P.ry[i];
      const double g = 2.0 * gwc[i] * wc[i] * (P.irn[i] * P.irn[i]);
      const double gz = gZc[i] * P.irn[i];
      grx[i] += g * (rx - wc[i] * (rx * vxx + ry * vxy)) + gz * rx;
      gry[i] += g * (ry - wc[i] * (ry * vyy + rx * vxy)) + gz * ry;
      gR -= gZc[i];
    }
  }
  // ---------------------------------------------------------------- multiple scattering VB(S), by segment
  {
    const double XXI_0 = 0.06 / 16.0, c = 0.038;
    double gms = 0.0;  // sum of the segments' variances times their gradients
#pragma unroll
    for (int i = 0; i + 1 < N; ++i) {
      const double g = (i > 0 ? gVB[i] : 0.0) + (i + 1 < N - 1 ? gVB[i + 1] : 0.0);
      const double L = S[i + 1] - S[i], l = P.lt[i];
      const double k = g * P.scale * XXI_0;
      const double dL = k * (L < 0 ? -1.0 : 1.0) * (l * l + 2.0 * c * l);
      gms += k * fabs(L) * (l * l);
      gS[i + 1] += dL;
      gS[i] -= dL;
    }
    if (B * P.R < 20.0) gR -= 2.0 * gms * iR;
    gm -= 2.0 * gms * m * (a * a);
  }
  // ---------------------------------------------------------------- rotation (S, Z) = R(m) (s, z)
#pragma unroll
  for (int i = 0; i < N; ++i) {
    gs[i] += a * gS[i] - b * gZl[i];
    gp[2][i] += b * gS[i] + a * gZl[i];
    ga += s[i] * gS[i] + G.p[2][i] * gZl[i];
    gb += G.p[2][i] * gS[i] - s[i] * gZl[i];
  }
  gm += (gb - ga * m) * (a * a * a);
  // ---------------------------------------------------------------- arc lengths s_i = -q R alpha_i, slope m = -q dz / (R alpha_n)
  // with alpha_i = atan2(u x p_i, |u|^2 + u.p_i), whose arguments' squares add up to R^2 |r_i|^2
  constexpr int n1 = N - 1;
  const double q = P.q;
  const double ux = -P.cx, uy = -P.cy, uu = ux * ux + uy * uy;
  double gux = 0.0, guy = 0.0, guu = 0.0;
  const double idz = 1.0 / G.p[2][n1];
  gR -= gm * m * iR;
  gp[2][n1] += gm * m * idz;
#pragma unroll
  for (int i = 1; i < N; ++i) {
    const double px = G.p[0][i], py = G.p[1][i];
    const double cr = ux * py - uy * px, dt = uu + ux * px + uy * py;
    double galpha = -q * P.R * gs[i];
    if (i == n1) galpha += gm * q * (m * m) * P.R * idz;
    gR += s[i] * gs[i] * iR;
    const double f = galpha * (iR * iR) * (P.irn[i] * P.irn[i]);
    const double gcr = f * dt, gdt = -f * cr;
    gux += gcr * py + gdt * px;
    guy += -gcr * px + gdt * py;
    gp[1][i] += gcr * ux + gdt * uy;
    gp[0][i] += -gcr * uy + gdt * ux;
    guu += gdt;
  }
  gux += 2.0 * ux * guu;
  guy += 2.0 * uy * guu;
  double gcx = -gux, gcy = -guy;
  // radii r_i = p_i - c
#pragma unroll
  for (int i = 0; i < N; ++i) {
    gp[0][i] += grx[i];
    gp[1][i] += gry[i];
    gcx -= grx[i];
    gcy -= gry[i];
  }
  // ---------------------------------------------------------------- R = |c|
  gcx += gR * P.cx * iR;
  gcy += gR * P.cy * iR;
  // ---------------------------------------------------------------- fast-fit centre (circumcentre of hits 0, mid, N-1)
  {
    constexpr int mid = N >> 1;
    const double a1 = G.p[0][mid], a2 = G.p[1][mid];
    const double c1 = -G.p[0][n1], c2 = -G.p[1][n1];
    const double ca = c1 * a2 - c2 * a1;
    const double nc = c1 * c1 + c2 * c2, na = a1 * a1 + a2 * a2;
    const double tmp = 0.5 / ca;  // d tmp / d ca = -2 tmp^2
    const double Nx = a2 * nc + c2 * na, Ny = a1 * nc + c1 * na;
    const double gNx = -gcx * tmp, gNy = gcy * tmp;
    const double gtmp = -gcx * Nx + gcy * Ny;
    const double gca = -2.0 * gtmp * tmp * tmp;
    double ga1 = gNy * nc - gca * c2, ga2 = gNx * nc + gca * c1;
    double gc1 = gNy * na + gca * a2, gc2 = gNx * na - gca * a1;
    const double gnc = gNx * a2 + gNy * a1, gna = gNx * c2 + gNy * c1;
    gc1 += 2.0 * c1 * gnc;
    gc2 += 2.0 * c2 * gnc;
    ga1 += 2.0 * a1 * gna;
    ga2 += 2.0 * a2 * gna;
    gp[0][mid] += ga1;
    gp[1][mid] += ga2;
    gp[0][n1] -= gc1;
    gp[1][n1] -= gc2;
  }
  // ---------------------------------------------------------------- p_i = h_i - h_0
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    double sum = 0.0;
#pragma unroll
    for (int i = 1; i < N; ++i) {
      grad[k][i] = gp[k][i];
      sum += gp[k][i];
    }
    grad[k][0] = -sum;
  }
  return chi2;
}

}  // namespace bl
}  // namespace pxl
