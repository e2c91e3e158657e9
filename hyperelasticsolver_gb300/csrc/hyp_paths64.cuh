// hyp_paths64.cuh -- the two-phase model's non-conservative products on the compact FP64
// cell forms: B(Q) of HyperelasticityMPh.jl:178-250 at a node and its path integrals
// (NumFluxes.jl:36-47, 97-107), for the two-phase step and the face evaluators.
#pragma once
#include "hyp_cell64.cuh"
#include "hyp_physics_mph.cuh"

namespace hyp {

// The two phases' EOS with the constants of the compact forms.
struct Eos2x {
  EosC e[2];
  Eos64 k[2];
};

// Rows of a phase's 15 whose physical flux is identically zero: alpha and the first row
// of alpha rho A.
HYP_HD constexpr bool zero_flux_row(int r) { return r == 0 || (r >= 6 && (r - 6) % 3 == 0); }
inline Eos2x make_eos2x(const EosC* e) {
  Eos2x E;
  for (int p = 0; p < 2; ++p) {
    E.e[p] = e[p];
    E.k[p] = make_eos64(e[p]);
  }
  return E;
}

// What the other phase needs of one phase at a node (HyperelasticityMPh.jl:186-217):
// velocity, stress row 1 (sigma symmetric), temperature dE/dS (:212).
struct Half64 {
  double u[3], K[3], T;
};
template <int kDef>
HYP_HD int half64(const EosC& e, const Eos64& k, double ia, const double* m, double rE,
                                      const double* R, Half64& h) {
  const Cell64 c = cell64<kDef, false>(e, k, ia, m, rE, R);
  const double m2 = -add64(k, c.td, c.td);
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    h.u[v] = c.u[v];
    h.K[v] = mul64(k, m2, c.w[v]);
  }
  h.T = e.t0 * add64(k, c.Pg, c.px);
  return c.st;
}

// Interface velocity, stress and its power (HyperelasticityMPh.jl:218-232, omega = 0,
// k = 1/2): the same for both phases.
struct Face64 {
  double u[3], s[3], p;
};
HYP_HD Face64 interface64(const Eos64& k, const Half64& a, const Half64& b) {
  Face64 I;
  const double inv = rcp64(k, add64(k, a.T, b.T)), ha = mul64(k, b.T, inv), hb = mul64(k, a.T, inv);
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    I.u[v] = mul64(k, k.half, add64(k, a.u[v], b.u[v]));
    I.s[v] = fma(hb, b.K[v], mul64(k, ha, a.K[v]));
  }
  I.p = fma(I.s[2], I.u[2], fma(I.s[1], I.u[1], mul64(k, I.s[0], I.u[0])));
  return I;
}

// acc += wd B(q) e_alpha for one phase's rows (row 1 of B is zero), B's rho A part with
// alpha rho A / alpha in place of rho A.
HYP_HD void add_b64(const Eos64& k, double wd, double ia, const double* R, const double* u, const Face64& I,
                    double* acc) {
  acc[0] = fma(wd, I.u[0], acc[0]);
  acc[2] = fma(wd, I.s[0], acc[2]);
  acc[3] = fma(wd, I.s[1], acc[3]);
  acc[4] = fma(wd, I.s[2], acc[4]);
  acc[5] = fma(wd, I.p, acc[5]);
  const double wi = mul64(k, wd, ia), d1 = sub64(k, I.u[1], u[1]), d2 = sub64(k, I.u[2], u[2]);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double* r = R + 3 * c;
    const double w0 = mul64(k, wi, r[0]);
    acc[6 + 3 * c] = fma(wi, fma(r[2], d2, fma(r[1], d1, mul64(k, r[0], I.u[0]))), acc[6 + 3 * c]);
    acc[7 + 3 * c] = fma(w0, u[1], acc[7 + 3 * c]);
    acc[8 + 3 * c] = fma(w0, u[2], acc[8 + 3 * c]);
  }
}

// Nodes a path integral from a to b (30 values) needs to be its 6-point value to FP64
// rounding: 2, 3 or 6 points of Gauss-Legendre.
//
// Along the path B is analytic in s: its singularities are alpha = 0, det R = 0 and a
// vanishing temperature (the entropy clamp aside). If every one of these quantities
// changes by at most w (relatively) from a to b, then for |s - s'| <= 1 / (4 w) they stay
// within a quarter of their values, B within a small factor M of its own, and Cauchy's
// estimate of its derivatives in the error term of the m-point rule gives
//   (m!)^4 / ((2m + 1) ((2m)!)^2) (4 w)^(2m) M d(alpha):
// 5.6e-3 (4w)^4 for m = 2, 3.6e-4 (4w)^6 for m = 3. The rule is taken when this is below
// 2^-57 alpha M, a sixteenth of the rounding of the flux difference the integral is
// added to. All estimates in FP32 on generous sides; NaN gives 6.
HYP_HD int path_nodes(const EosC* e, const double* a, const double* b) {
  float w = 0.0f, jump = 0.0f;
  for (int p = 0; p < 2; ++p) {
    const double *qa = a + 15 * p, *qb = b + 15 * p;
    const float al = to_f32(qa[0]), be = to_f32(qb[0]), lo = fminf(al, be);
    if (!(lo > 0.0f)) return 6;
    // the jump itself, subtracted in FP64 (of FP32 fractions it would be 0 below 1e-7 of them,
    // and the bound with it) and rounded up
    const float da = 1.0001f * fabsf(to_f32(qb[0] - qa[0]));
    const float ra = da / lo, ia = 1.0f / al, ib = 1.0f / be;
    // B depends on the path through q / alpha alone, and q / alpha runs on a straight line
    float F[9], dF2 = 0.0f, F2 = 0.0f, v2 = 0.0f, dv2 = 0.0f;
    for (int k = 0; k < 9; ++k) {
      F[k] = to_f32(qa[6 + k]) * ia;
      const float d = to_f32(qb[6 + k]) * ib - F[k];
      dF2 += d * d;
      F2 += F[k] * F[k];
    }
    for (int k = 0; k < 3; ++k) {
      const float v = to_f32(qa[2 + k]) * ia, d = to_f32(qb[2 + k]) * ib - v;
      v2 += v * v;
      dv2 += d * d;
    }
    const float rE = to_f32(qa[5]) * ia, drE = fabsf(to_f32(qb[5]) * ib - rE);
    const float c00 = F[4] * F[8] - F[5] * F[7], c01 = F[7] * F[2] - F[1] * F[8], c02 = F[1] * F[5] - F[4] * F[2];
    const float c10 = F[5] * F[6] - F[3] * F[8], c11 = F[0] * F[8] - F[2] * F[6], c12 = F[2] * F[3] - F[0] * F[5];
    const float c20 = F[3] * F[7] - F[4] * F[6], c21 = F[1] * F[6] - F[0] * F[7], c22 = F[0] * F[4] - F[1] * F[3];
    const float det = F[0] * c00 + F[3] * c01 + F[6] * c02;
    const float cc = c00 * c00 + c01 * c01 + c02 * c02 + c10 * c10 + c11 * c11 + c12 * c12 + c20 * c20 + c21 * c21 +
                     c22 * c22;
    if (!(det > 0.0f)) return 6;
    // ||dF|| ||F^-1||, with the FP32 rounding of dF
    const float dF = (sqrtf(dF2) + 2e-7f * sqrtf(F2)) * sqrtf(cc) / det;
    const float rho = sqrtf(det * (float)e[p].inv_rho0), s = rho * (float)e[p].inv_rho0;
    if (!(s > 0.25f && s < 4.0f)) return 6;
    // specific energy minus the elastic part: (x - 1) cv t0 Pg, x the temperature over t0 Pg
    const float u = sqrtf(v2) / rho, du = (sqrtf(dv2) + 1.5f * sqrtf(v2) * dF) / rho, E = rE / rho;
    // |G| and its deviator from F: G = rho^2 (F F^T)^-1, tr G = rho^2 cc / det^2
    const float i1 = rho * rho * cc / (det * det), i2 = s * s * F2 / (rho * rho);  // det G = s^2, tr G^-1 = |F|^2 / rho^2
    const float psi = fmaxf(i1 * i1 * (1.0f / 3.0f) - i2, 0.0f);
    const float ga = (float)e[p].gamma, be_ = (float)e[p].beta, aa = (float)e[p].alpha;
    const float Pa = powf(s, aa), Pb = powf(s, be_), Pg = powf(s, ga);
    const float cvt0 = (float)e[p].cvt0, kU = (float)e[p].kU, b0sq = (float)e[p].b0sq;
    const float therm = E - 0.5f * u * u - 0.5f * b0sq * Pb * psi - kU * (Pa - 1.0f) * (Pa - 1.0f);
    const float x = therm / (cvt0 * Pg) + 1.0f;
    const float grow = powf(1.25f * fmaxf(s, 1.0f / s), fmaxf(2.0f * fabsf(aa), fmaxf(fabsf(be_), fabsf(ga))));
    const float dE = drE / rho + 1.5f * fabsf(E) * dF + u * du + du * du +
                     4.0f * (2.0f * fabsf(kU) * aa * aa + 2.0f * b0sq) * grow * dF;
    if (!(x > 1e-3f)) return 6;
    const float wF = 3.0f * dF, wx = dE / (cvt0 * Pg * x) + 2.0f * fabsf(ga) * dF;
    if (!(ra < 0.125f && wF < 0.125f && wx < 0.125f)) return 6;  // (NaN too)
    w = fmaxf(w, fmaxf(ra, fmaxf(wF, wx)));
    jump = fmaxf(jump, ra);
  }
  const float d = 4.0f * w, d2 = d * d;
  if (5.6e-3f * d2 * d2 * jump <= 7e-18f) return 2;
  if (3.6e-4f * d2 * d2 * d2 * jump <= 7e-18f) return 3;
  return 6;
}

// One thread per face: acc += the path integral from a to b (30 values each): the nodes
// path_nodes asks for, of both phases, 360 slots a node. Rolled: six copies of the node
// overflow the instruction cache. qd: the 6-point rule; kSix: always that, for who gets the
// integral by itself (path_nodes keeps its error small beside a flux difference, not beside
// the integral, which is as small as the volume fractions' jump).
template <int kDef, bool kSix = false>
HYP_HD int path_thread(const Eos2x& E, const Quad6D& qd, const double* a, const double* b, double* acc) {
  int st = 0;
  const double da0 = b[0] - a[0], da1 = b[15] - a[15];
  const int nodes = kSix ? 6 : path_nodes(E.e, a, b);
#pragma unroll 1
  for (int i = 0; i < nodes; ++i) {
    double s, w;
    if (nodes == 6) {
      s = qd.x[i];
      w = qd.w[i];
    } else if (nodes == 2) {  // 1/2 -+ 1/(2 sqrt 3)
      s = i ? 0.78867513459481288 : 0.21132486540518712;
      w = 0.5;
    } else {  // 1/2, 1/2 -+ sqrt(3/5)/2
      s = i == 0 ? 0.11270166537925831 : (i == 1 ? 0.5 : 0.88729833462074169);
      w = i == 1 ? 4.0 / 9.0 : 5.0 / 18.0;
    }
    double R[2][9], ia[2];
    Half64 h[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      double m[3];
      const Eos64& kp = E.k[p];
      auto at = [&](int r) { return fma(s, sub64(kp, b[15 * p + r], a[15 * p + r]), a[15 * p + r]); };
#pragma unroll
      for (int v = 0; v < 3; ++v) m[v] = at(2 + v);
#pragma unroll
      for (int v = 0; v < 9; ++v) R[p][v] = at(6 + v);
      ia[p] = rcp64(kp, at(0));
      st |= half64<kDef>(E.e[p], kp, ia[p], m, at(5), R[p], h[p]);
    }
    const Face64 I = interface64(E.k[0], h[0], h[1]);
    add_b64(E.k[0], w * da0, ia[0], R[0], h[0].u, I, acc);
    add_b64(E.k[1], w * da1, ia[1], R[1], h[1].u, I, acc + 15);
  }
  return st;
}

}  // namespace hyp
