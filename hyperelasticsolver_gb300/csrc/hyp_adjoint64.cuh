// hyp_adjoint64.cuh -- the cell's vector-Jacobian product on the compact forms of
// hyp_cell64.cuh: qb += (df/dq)^T fb + (dlambda/dq) lb, eb likewise, as cell_vjp
// (hyp_adjoint.cuh) gives them, in half its FP64 instructions, which are what the
// adjoint step is bound by.
//
// The forward forms are reversed statement by statement. What the compact ones save
// beside their own counts: the acoustic tensor's derivatives are those of its six
// closed entries instead of three directional derivatives each; every power of det G
// contributes to one logarithmic derivative, and the scalings by rho to another (p, G
// and the unscaled primitives are powers of rho times something else); below the
// entropy clamp the thermal term does not depend on det G at all.
#pragma once
#include "hyp_adjoint.cuh"
#include "hyp_cell64.cuh"

namespace hyp {

// Out of line: cells whose top eigenvalue does not stand clear.
#ifdef __CUDACC__
static __host__ __device__ __noinline__
#else
inline
#endif
int cell_vjp_general(const EosC& e, const double* q, const double* fb, double lb, double* qb, EosBar& eb) {
  return cell_vjp(e, q, fb, lb, qb, eb);
}

template <int kDef>
HYP_HD int cell_vjp64(const EosC& e, const Eos64& k, const double* q, const double* fb, double lb, double* qb,
                      EosBar& eb) {
  const double *m = q + 1, *R = q + 5;
  const Cell64 c = cell64<kDef, true>(e, k, 1.0, m, q[4], R);
  const double r = c.inv_den, ms = k.inv_rho0sq;
  const double th = (c.G00 + c.G11 + c.G22) * (1.0 / 3.0);
  const double d0 = c.G00 - th, d1 = c.G11 - th, d2 = c.G22 - th;
  const double n00 = R[0] * R[0] + R[3] * R[3] + R[6] * R[6], n11 = R[1] * R[1] + R[4] * R[4] + R[7] * R[7];
  const double n22 = R[2] * R[2] + R[5] * R[5] + R[8] * R[8], n01 = R[0] * R[1] + R[3] * R[4] + R[6] * R[7];
  const double n02 = R[0] * R[2] + R[3] * R[5] + R[6] * R[8], n12 = R[1] * R[2] + R[4] * R[5] + R[7] * R[8];
  // adjoints
  double u0b = 0.0, w0b = 0.0, w1b = 0.0, w2b = 0.0;
  double g00 = 0.0, g01 = 0.0, g02 = 0.0, g11 = 0.0, g12 = 0.0, g22 = 0.0;  // of G
  double ab = 0.0, bMb = 0.0, bhb = 0.0, T2b = 0.0, T3b = 0.0, E3b = 0.0, Pab = 0.0, bb = 0.0;
  // ---- wave speed lambda = |u1| + sqrt(2 nu), nu the top eigenvalue of O ----
  if (bits_of(lb) << 1) {
    const double f = (4.0 / 3.0) * c.b;
    const double rest = c.w[0] + k.beta22 * c.wE + e.gamma * c.T2 + e.beta * c.T3 +
                        e.alpha * (k.kE3a * c.Pa * (2.0 * c.Pa - 1.0));
    const double f0 = f * c.G00, f1 = f * c.G01, f2 = f * c.G02;
    const double o00 = f0 * c.G00 + rest, o01 = f0 * c.G01 + k.beta2 * c.w[1], o02 = f0 * c.G02 + k.beta2 * c.w[2];
    const double o11 = f1 * c.G01 + (c.a * c.G11 - c.bM), o22 = f2 * c.G02 + (c.a * c.G22 - c.bM);
    const double o12 = f1 * c.G02 + c.a * c.G12;
    double nu;
    if (!top_root64(k, o00, o11, o22, o01, o02, o12, nu)) return cell_vjp_general(e, q, fb, lb, qb, eb);
    u0b = c.u[0] > 0.0 ? lb : (c.u[0] < 0.0 ? -lb : 0.0);
    // d nu / d O = Cof(nu I - O) / its trace; an off-diagonal entry stands for two
    const double b00 = nu - o00, b11 = nu - o11, b22 = nu - o22;
    const double C00 = b11 * b22 - o12 * o12, C11 = b00 * b22 - o02 * o02, C22 = b00 * b11 - o01 * o01;
    const double C01 = o02 * o12 + o01 * b22, C02 = o01 * o12 + o02 * b11, C12 = o01 * o02 + b00 * o12;
    const double g = lb * rsqrt64(k, nu + nu) * rcp64(k, C00 + C11 + C22), g2 = g + g;
    const double p00 = g * C00, p11 = g * C11, p22 = g * C22, p01 = g2 * C01, p02 = g2 * C02, p12 = g2 * C12;
    // O_ij = f G0i G0j + ...
    const double t0 = 2.0 * p00 * c.G00 + p01 * c.G01 + p02 * c.G02;
    const double t1 = p01 * c.G00 + 2.0 * p11 * c.G01 + p12 * c.G02;
    const double t2 = p02 * c.G00 + p12 * c.G01 + 2.0 * p22 * c.G02;
    g00 = f * t0;
    g01 = f * t1;
    g02 = f * t2;
    bb = (2.0 / 3.0) * (t0 * c.G00 + t1 * c.G01 + t2 * c.G02);  // f = 4/3 b, each product counted twice
    ab = p11 * c.G11 + p22 * c.G22 + p12 * c.G12;
    g11 = c.a * p11;
    g22 = c.a * p22;
    g12 = c.a * p12;
    bMb = -(p11 + p22);
    w1b = k.beta2 * p01;
    w2b = k.beta2 * p02;
    w0b = p00;  // rest = w0 + (2 beta + 2) b h + gamma T2 + beta T3 + alpha kE3a Pa (2 Pa - 1)
    bhb = k.beta22 * p00;
    T2b = e.gamma * p00;
    T3b = e.beta * p00;
    Pab = e.alpha * k.kE3a * ((4.0 * c.Pa - 1.0) * p00);
    eb.k0 += 0.5 * p00 * (c.Pa * (2.0 * c.Pa - 1.0));
  }
  // ---- flux ----
  const double tr = 2.0 * c.td;  // S = 2 rho w
  const double s0 = fb[1] + fb[4] * c.u[0], s1 = fb[2] + fb[4] * c.u[1], s2 = fb[3] + fb[4] * c.u[2];
  const double e4 = fb[4] * tr;
  const double m0b = fb[0] + (fb[1] * c.u[0] + fb[2] * c.u[1] + fb[3] * c.u[2] + fb[4] * c.E);
  u0b += fb[1] * m[0] + e4 * c.w[0];
  double u1b = fb[2] * m[0] + e4 * c.w[1], u2b = fb[3] * m[0] + e4 * c.w[2];
  double Eb = fb[4] * m[0];
  double Rb[9];
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    const double h1 = fb[6 + 3 * b], h2 = fb[7 + 3 * b];
    u0b += h1 * R[1 + 3 * b] + h2 * R[2 + 3 * b];
    u1b -= h1 * R[3 * b];
    u2b -= h2 * R[3 * b];
    Rb[3 * b] = -(h1 * c.u[1] + h2 * c.u[2]);
    Rb[1 + 3 * b] = h1 * c.u[0];
    Rb[2 + 3 * b] = h2 * c.u[0];
  }
  w0b += tr * s0;
  w1b += tr * s1;
  w2b += tr * s2;
  const double rhob_w = 2.0 * (s0 * c.w[0] + s1 * c.w[1] + s2 * c.w[2]);
  // ---- w0 = b h + E3 p, h = G00 d0 + G01^2 + G02^2; w_j = a G0j + b ms n0j; bM = b ms n00 ----
  bhb += w0b;
  E3b += w0b;
  const double hb = bhb * c.b;
  ab += w1b * c.G01 + w2b * c.G02;
  g01 += c.a * w1b;
  g02 += c.a * w2b;
  bb += bhb * (c.G00 * d0 + (c.G01 * c.G01 + c.G02 * c.G02)) + ms * (w1b * n01 + w2b * n02 + bMb * n00);
  const double bms = c.b * ms;
  // ---- E3 p = T1 + T2 + T3 ----
  T2b += E3b;
  T3b += E3b;
  double bpb = k.hbeta * T3b;
  // T2 = kE3g px, px = Pg (x - 1) = y / (cv t0) unless clamped, y = e_int - b psi - kU am1^2
  const double pxb = k.kE3g * T2b;
  const double am1 = c.Pa - 1.0, z = k.kU * am1;
  double yb = 0.0, Lp = 0.0;  // Lp: derivative to log p
  if (c.clamped)
    Lp = (0.5 * e.gamma) * (pxb * c.px);
  else
    yb = pxb * e.inv_cvt0;
  // T1 = alpha z Pa, z = kU am1
  const double T1a = e.alpha * E3b;
  const double zb = T1a * c.Pa - yb * am1;
  Pab += z * (T1a - yb) + k.kU * zb;
  eb.k0 += zb * am1 * k.h_alphasq;
  bpb -= yb;
  // ---- b psi, a = 2 b th, psi = |d|^2/2 + G01^2 + G02^2 + G12^2 ----
  const double psi = 0.5 * (d0 * d0 + d1 * d1 + d2 * d2) + (c.G12 * c.G12 + (c.G01 * c.G01 + c.G02 * c.G02));
  bb += bpb * psi + 2.0 * (ab * th);
  const double psib = bpb * c.b, ob = 2.0 * (hb + psib);
  g01 += ob * c.G01;
  g02 += ob * c.G02;
  g12 += (psib + psib) * c.G12;
  const double d0b = hb * c.G00 + psib * d0, d1b = psib * d1, d2b = psib * d2;
  const double i1b = (1.0 / 3.0) * (2.0 * (ab * c.b) - (d0b + d1b + d2b));  // of th, a third to each diagonal
  g00 += hb * d0 + d0b + i1b;
  g11 += d1b + i1b;
  g22 += d2b + i1b;
  // ---- powers: Pa, b = b0sq/2 Pb ----
  eb.b0sq += 0.5 * (bb * c.Pb);
  Lp += (0.5 * e.alpha) * (Pab * c.Pa) + k.hbeta * (bb * c.b);
  // ---- rho: p ~ rho^2, G ~ rho^-2 C, u, E ~ 1/rho, S ~ rho ----
  const double eib = yb;  // e_int = E - |u|^2/2
  Eb += eib;
  u0b -= eib * c.u[0];
  u1b -= eib * c.u[1];
  u2b -= eib * c.u[2];
  const double GG = (g00 * c.G00 + g11 * c.G11 + g22 * c.G22) + (g01 * c.G01 + g02 * c.G02 + g12 * c.G12);
  const double rhob = rhob_w + r * (2.0 * (Lp - GG) - (Eb * c.E + (u0b * c.u[0] + u1b * c.u[1] + u2b * c.u[2])));
  qb[1] += m0b + u0b * r;
  qb[2] += u1b * r;
  qb[3] += u2b * r;
  qb[4] += Eb * r;
  // ---- G = C gs, C the cofactors of N; N = R R^T ----
  const double t = r * k.inv_rho0, gs = t * t;
  const double h00 = g00 * gs, h11 = g11 * gs, h22 = g22 * gs, h01 = g01 * gs, h02 = g02 * gs, h12 = g12 * gs;
  const double N00 = 2.0 * (h11 * n22 + h22 * n11 - h12 * n12 + bMb * bms);  // doubled: R's rows meet it twice
  const double N11 = 2.0 * (h00 * n22 + h22 * n00 - h02 * n02);
  const double N22 = 2.0 * (h00 * n11 + h11 * n00 - h01 * n01);
  const double N01 = -2.0 * (h22 * n01) - h01 * n22 + h02 * n12 + h12 * n02 + w1b * bms;
  const double N02 = -2.0 * (h11 * n02) + h01 * n12 - h02 * n11 + h12 * n01 + w2b * bms;
  const double N12 = -2.0 * (h00 * n12) + h01 * n02 + h02 * n01 - h12 * n00;
  // ---- rho = sqrt(det R / rho0) ----
  const double db = rhob * (0.5 * k.inv_rho0) * r;
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    const double *x = R + 3 * ((b + 1) % 3), *y = R + 3 * ((b + 2) % 3);  // cofactors of column b: x cross y
    const double r0 = R[3 * b], r1 = R[3 * b + 1], r2 = R[3 * b + 2];
    qb[5 + 3 * b] += Rb[3 * b] + (N00 * r0 + N01 * r1 + N02 * r2) + db * (x[1] * y[2] - x[2] * y[1]);
    qb[6 + 3 * b] += Rb[3 * b + 1] + (N01 * r0 + N11 * r1 + N12 * r2) + db * (x[2] * y[0] - x[0] * y[2]);
    qb[7 + 3 * b] += Rb[3 * b + 2] + (N02 * r0 + N12 * r1 + N22 * r2) + db * (x[0] * y[1] - x[1] * y[0]);
  }
  return c.st;
}

}  // namespace hyp
