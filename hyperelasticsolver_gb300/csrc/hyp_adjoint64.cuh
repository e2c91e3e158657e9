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
// entropy clamp the thermal term does not depend on det G at all. Sums, products and
// constants as in hyp_cell64.cuh.
#pragma once
#include "hyp_adjoint.cuh"
#include "hyp_cell64.cuh"

namespace hyp {

// How an evaluation ended: on the compact forms; not at all, with qb and eb that mean nothing
// and the same to be done with the hardware's products (cell_try64); by the general form, for a
// top eigenvalue that does not stand clear.
enum { kVjpDone = 0, kVjpPlain = 1, kVjpGeneral = 2 };

// The general form, out of line.
#ifdef __CUDACC__
static __host__ __device__ __noinline__
#else
inline
#endif
int cell_vjp_general(const EosC& e, const double* q, const double* fb, double lb, double* qb, EosBar* eb) {
  return cell_vjp(e, q, fb, lb, qb, *eb);
}

template <int kDef, class K>
HYP_HD int cell_vjp_of64(const EosC& e, const K& k, const double* q, const double* fb, double lb, double* qb,
                         EosBar& eb, int& st) {
  auto M = [&k](double x, double y) { return mul64(k, x, y); };
  auto A = [&k](double x, double y) { return add64(k, x, y); };
  auto S = [&k](double x, double y) { return sub64(k, x, y); };
  auto D = [&k](double x) { return add64(k, x, x); };
  auto dot = [&k](double a, double b, double c, double d, double f, double g) {  // a b + c d + f g
    return fma(f, g, fma(c, d, mul64(k, a, b)));
  };
  const double *m = q + 1, *R = q + 5;
  const Cell64 c = cell64<kDef, true>(e, k, 1.0, m, q[4], R);
  st = c.st;
  const double r = c.inv_den, ms = k.inv_rho0sq;
  const double i1 = A(A(c.G00, c.G11), c.G22), th = M(k.third, i1);
  const double d0 = S(c.G00, th), d1 = S(c.G11, th), d2 = S(c.G22, th);
  const double n00 = dot(R[0], R[0], R[3], R[3], R[6], R[6]), n11 = dot(R[1], R[1], R[4], R[4], R[7], R[7]);
  const double n22 = dot(R[2], R[2], R[5], R[5], R[8], R[8]), n01 = dot(R[0], R[1], R[3], R[4], R[6], R[7]);
  const double n02 = dot(R[0], R[2], R[3], R[5], R[6], R[8]), n12 = dot(R[1], R[2], R[4], R[5], R[7], R[8]);
  // adjoints
  double u0b = 0.0, w0b = 0.0, w1b = 0.0, w2b = 0.0;
  double g00 = 0.0, g01 = 0.0, g02 = 0.0, g11 = 0.0, g12 = 0.0, g22 = 0.0;  // of G
  double ab = 0.0, bMb = 0.0, bhb = 0.0, T2b = 0.0, T3b = 0.0, E3b = 0.0, Pab = 0.0, bb = 0.0;
  // ---- wave speed lambda = |u1| + sqrt(2 nu), nu the top eigenvalue of O ----
  if (bits_of(lb) << 1) {
    const double f = M(k.four3, c.b);
    const double P2 = fma(c.Pa, D(c.Pa), -c.Pa);  // Pa (2 Pa - 1)
    const double rest = fma(M(e.alpha, k.kE3a), P2, fma(e.beta, c.T3, fma(e.gamma, c.T2, fma(k.beta22, c.wE, c.w[0]))));
    const double f0 = M(f, c.G00), f1 = M(f, c.G01), f2 = M(f, c.G02);
    const double o00 = fma(f0, c.G00, rest);
    const double o01 = fma(f0, c.G01, M(k.beta2, c.w[1])), o02 = fma(f0, c.G02, M(k.beta2, c.w[2]));
    const double o11 = fma(f1, c.G01, fma(c.a, c.G11, -c.bM)), o22 = fma(f2, c.G02, fma(c.a, c.G22, -c.bM));
    const double o12 = fma(f1, c.G02, M(c.a, c.G12));
    double nu;
    if (!top_root64(k, o00, o11, o22, o01, o02, o12, nu)) {
      if (out_of_range(k)) return kVjpPlain;
      // on copies: the arrays themselves, had they an address, would lie in local memory in
      // every cell
      double qs[14], fs[14], bs[14];
      EosBar es = eb;
#pragma unroll
      for (int v = 0; v < 14; ++v) {
        qs[v] = q[v];
        fs[v] = fb[v];
        bs[v] = qb[v];
      }
      st = cell_vjp_general(e, qs, fs, lb, bs, &es);
#pragma unroll
      for (int v = 0; v < 14; ++v) qb[v] = bs[v];
      eb = es;
      return kVjpGeneral;
    }
    u0b = c.u[0] > 0.0 ? lb : (c.u[0] < 0.0 ? -lb : 0.0);
    // d nu / d O = Cof(nu I - O) / its trace; an off-diagonal entry stands for two
    const double b00 = S(nu, o00), b11 = S(nu, o11), b22 = S(nu, o22);
    const double C00 = fma(b11, b22, -M(o12, o12)), C11 = fma(b00, b22, -M(o02, o02)), C22 = fma(b00, b11, -M(o01, o01));
    const double C01 = fma(o02, o12, M(o01, b22)), C02 = fma(o01, o12, M(o02, b11)), C12 = fma(o01, o02, M(b00, o12));
    const double g = M(lb, M(rsqrt64(k, D(nu)), rcp64(k, A(A(C00, C11), C22)))), g2 = D(g);
    const double p00 = M(g, C00), p11 = M(g, C11), p22 = M(g, C22);
    const double p01 = M(g2, C01), p02 = M(g2, C02), p12 = M(g2, C12);
    // O_ij = f G0i G0j + ...
    const double t0 = dot(D(p00), c.G00, p01, c.G01, p02, c.G02);
    const double t1 = dot(p01, c.G00, D(p11), c.G01, p12, c.G02);
    const double t2 = dot(p02, c.G00, p12, c.G01, D(p22), c.G02);
    g00 = M(f, t0);
    g01 = M(f, t1);
    g02 = M(f, t2);
    bb = M(k.two3, dot(t0, c.G00, t1, c.G01, t2, c.G02));  // f = 4/3 b, each product counted twice
    ab = dot(p11, c.G11, p22, c.G22, p12, c.G12);
    g11 = M(c.a, p11);
    g22 = M(c.a, p22);
    g12 = M(c.a, p12);
    bMb = -A(p11, p22);
    w1b = M(k.beta2, p01);
    w2b = M(k.beta2, p02);
    w0b = p00;  // rest = w0 + (2 beta + 2) b h + gamma T2 + beta T3 + alpha kE3a Pa (2 Pa - 1)
    bhb = M(k.beta22, p00);
    T2b = e.gamma * p00;
    T3b = e.beta * p00;
    Pab = M(M(e.alpha, k.kE3a), M(S(D(D(c.Pa)), k.one), p00));
    eb.k0 = fma(M(k.half, p00), P2, eb.k0);
  }
  // ---- flux ----
  const double tr = D(c.td);  // S = 2 rho w
  const double s0 = fma(fb[4], c.u[0], fb[1]), s1 = fma(fb[4], c.u[1], fb[2]), s2 = fma(fb[4], c.u[2], fb[3]);
  const double e4 = M(fb[4], tr);
  const double m0b = fma(fb[4], c.E, fma(fb[3], c.u[2], fma(fb[2], c.u[1], fma(fb[1], c.u[0], fb[0]))));
  u0b = fma(e4, c.w[0], fma(fb[1], m[0], u0b));
  double u1b = fma(e4, c.w[1], M(fb[2], m[0])), u2b = fma(e4, c.w[2], M(fb[3], m[0]));
  double Eb = M(fb[4], m[0]);
  double Rb[9];
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    const double h1 = fb[6 + 3 * b], h2 = fb[7 + 3 * b];
    u0b = fma(h2, R[2 + 3 * b], fma(h1, R[1 + 3 * b], u0b));
    u1b = fma(-h1, R[3 * b], u1b);
    u2b = fma(-h2, R[3 * b], u2b);
    Rb[3 * b] = -fma(h2, c.u[2], M(h1, c.u[1]));
    Rb[1 + 3 * b] = M(h1, c.u[0]);
    Rb[2 + 3 * b] = M(h2, c.u[0]);
  }
  w0b = fma(tr, s0, w0b);
  w1b = fma(tr, s1, w1b);
  w2b = fma(tr, s2, w2b);
  const double rhob_w = D(dot(s0, c.w[0], s1, c.w[1], s2, c.w[2]));
  // ---- w0 = b h + E3 p, h = G00 d0 + G01^2 + G02^2; w_j = a G0j + b ms n0j; bM = b ms n00 ----
  bhb = A(bhb, w0b);
  E3b = w0b;
  const double hb = M(bhb, c.b);
  ab = fma(w2b, c.G02, fma(w1b, c.G01, ab));
  g01 = fma(c.a, w1b, g01);
  g02 = fma(c.a, w2b, g02);
  const double off = fma(c.G02, c.G02, M(c.G01, c.G01));
  bb = fma(ms, dot(w1b, n01, w2b, n02, bMb, n00), fma(bhb, fma(c.G00, d0, off), bb));
  const double bms = M(c.b, ms);
  // ---- E3 p = T1 + T2 + T3 ----
  T2b = A(T2b, E3b);
  T3b = A(T3b, E3b);
  double bpb = M(k.hbeta, T3b);
  // T2 = kE3g px, px = Pg (x - 1) = y / (cv t0) unless clamped, y = e_int - b psi - kU am1^2
  const double pxb = M(k.kE3g, T2b);
  const double am1 = S(c.Pa, k.one), z = M(k.kU, am1);
  double yb = 0.0, Lp = 0.0;  // Lp: derivative to log p
  if (c.clamped)
    Lp = (0.5 * e.gamma) * M(pxb, c.px);
  else
    yb = M(pxb, k.inv_cvt0);
  // T1 = alpha z Pa, z = kU am1
  const double T1a = e.alpha * E3b;
  const double zb = fma(T1a, c.Pa, -M(yb, am1));
  Pab = fma(z, S(T1a, yb), fma(k.kU, zb, Pab));
  eb.k0 = fma(M(zb, am1), k.h_alphasq, eb.k0);
  bpb = S(bpb, yb);
  // ---- b psi, a = 2 b th, psi = |d|^2/2 + G01^2 + G02^2 + G12^2 ----
  const double psi = fma(k.half, dot(d0, d0, d1, d1, d2, d2), fma(c.G12, c.G12, off));
  bb = fma(bpb, psi, fma(D(ab), th, bb));
  const double psib = M(bpb, c.b), ob = D(A(hb, psib));
  g01 = fma(ob, c.G01, g01);
  g02 = fma(ob, c.G02, g02);
  g12 = fma(D(psib), c.G12, g12);
  const double d0b = fma(hb, c.G00, M(psib, d0)), d1b = M(psib, d1), d2b = M(psib, d2);
  const double i1b = M(k.third, fma(D(ab), c.b, -A(A(d0b, d1b), d2b)));  // of th, a third to each diagonal
  g00 = A(fma(hb, d0, g00), A(d0b, i1b));
  g11 = A(g11, A(d1b, i1b));
  g22 = A(g22, A(d2b, i1b));
  // ---- powers: Pa, b = b0sq/2 Pb ----
  eb.b0sq = fma(M(k.half, bb), c.Pb, eb.b0sq);
  Lp = fma(k.hbeta, M(bb, c.b), fma(0.5 * e.alpha, M(Pab, c.Pa), Lp));
  // ---- rho: p ~ rho^2, G ~ rho^-2 C, u, E ~ 1/rho, S ~ rho ----
  const double eib = yb;  // e_int = E - |u|^2/2
  Eb = A(Eb, eib);
  u0b = fma(-eib, c.u[0], u0b);
  u1b = fma(-eib, c.u[1], u1b);
  u2b = fma(-eib, c.u[2], u2b);
  const double GG = fma(g12, c.G12, fma(g02, c.G02, fma(g01, c.G01, dot(g00, c.G00, g11, c.G11, g22, c.G22))));
  const double uE = fma(Eb, c.E, dot(u0b, c.u[0], u1b, c.u[1], u2b, c.u[2]));
  const double rhob = fma(r, S(D(S(Lp, GG)), uE), rhob_w);
  qb[1] = A(qb[1], fma(u0b, r, m0b));
  qb[2] = fma(u1b, r, qb[2]);
  qb[3] = fma(u2b, r, qb[3]);
  qb[4] = fma(Eb, r, qb[4]);
  // ---- G = C gs, C the cofactors of N; N = R R^T ----
  const double t = M(r, k.inv_rho0), gs = M(t, t);
  const double h00 = M(g00, gs), h11 = M(g11, gs), h22 = M(g22, gs), h01 = M(g01, gs), h02 = M(g02, gs), h12 = M(g12, gs);
  const double N00 = D(fma(bMb, bms, dot(h11, n22, h22, n11, -h12, n12)));  // doubled: R's rows meet it twice
  const double N11 = D(dot(h00, n22, h22, n00, -h02, n02));
  const double N22 = D(dot(h00, n11, h11, n00, -h01, n01));
  const double N01 = fma(w1b, bms, fma(h12, n02, dot(h02, n12, -h01, n22, -D(h22), n01)));
  const double N02 = fma(w2b, bms, fma(h12, n01, dot(h01, n12, -h02, n11, -D(h11), n02)));
  const double N12 = fma(-h12, n00, dot(h01, n02, h02, n01, -D(h00), n12));
  // ---- rho = sqrt(det R / rho0) ----
  const double db = M(rhob, M(M(k.half, k.inv_rho0), r));
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    const double *x = R + 3 * ((b + 1) % 3), *y = R + 3 * ((b + 2) % 3);  // cofactors of column b: x cross y
    const double r0 = R[3 * b], r1 = R[3 * b + 1], r2 = R[3 * b + 2];
    qb[5 + 3 * b] = A(qb[5 + 3 * b], fma(db, fma(x[1], y[2], -M(x[2], y[1])), fma(N02, r2, fma(N01, r1, fma(N00, r0, Rb[3 * b])))));
    qb[6 + 3 * b] = A(qb[6 + 3 * b], fma(db, fma(x[2], y[0], -M(x[0], y[2])), fma(N12, r2, fma(N11, r1, fma(N01, r0, Rb[3 * b + 1])))));
    qb[7 + 3 * b] = A(qb[7 + 3 * b], fma(db, fma(x[0], y[1], -M(x[1], y[0])), fma(N22, r2, fma(N12, r1, fma(N02, r0, Rb[3 * b + 2])))));
  }
  return out_of_range(k) || (std::is_same<K, Soft64>::value && st) ? kVjpPlain : kVjpDone;
}

// kSoft: lone products on the integer pipe (hyp_cell64.cuh), the same values bit for bit.
template <int kDef, bool kSoft>
HYP_HD int cell_vjp_try64(const EosC& e, const Eos64& k, const double* q, const double* fb, double lb, double* qb,
                          EosBar& eb, int& st) {
  // (the adjoints, which have tails of their own, enter linearly)
  if (kSoft && !warp_holds(soft_inputs64(q + 1, 13) & soft_inputs64(fb, 14, 500u) & soft_inputs64(&lb, 1, 500u)))
    return kVjpPlain;
  return cell_vjp_of64<kDef>(e, typename std::conditional<kSoft, Soft64, Plain64>::type(k), q, fb, lb, qb, eb, st);
}

// All of it; returns the status.
template <int kDef, bool kSoft>
HYP_HD int cell_vjp64(const EosC& e, const Eos64& k, const double* q, const double* fb, double lb, double* qb,
                      EosBar& eb) {
  double qs[14];
  for (int v = 0; v < 14; ++v) qs[v] = qb[v];
  const EosBar es = eb;
  int st;
  if (cell_vjp_try64<kDef, kSoft>(e, k, q, fb, lb, qb, eb, st) == kVjpPlain) {
    for (int v = 0; v < 14; ++v) qb[v] = qs[v];
    eb = es;
    cell_vjp_try64<kDef, false>(e, k, q, fb, lb, qb, eb, st);
  }
  return st;
}

}  // namespace hyp
