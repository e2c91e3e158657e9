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
__device__ __forceinline__ constexpr bool zero_flux_row(int r) { return r == 0 || (r >= 6 && (r - 6) % 3 == 0); }
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
__device__ __forceinline__ int half64(const EosC& e, const Eos64& k, double ia, const double* m, double rE,
                                      const double* R, Half64& h) {
  const Cell64 c = cell64<kDef>(e, k, ia, m, rE, R);
  const double m2 = -2.0 * c.td;
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    h.u[v] = c.u[v];
    h.K[v] = m2 * c.w[v];
  }
  h.T = e.t0 * (c.Pg + c.px);
  return c.st;
}

// Interface velocity, stress and its power (HyperelasticityMPh.jl:218-232, omega = 0,
// k = 1/2): the same for both phases.
struct Face64 {
  double u[3], s[3], p;
};
__device__ __forceinline__ Face64 interface64(const Half64& a, const Half64& b) {
  Face64 I;
  const double inv = rcp64(a.T + b.T), ha = b.T * inv, hb = a.T * inv;
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    I.u[v] = 0.5 * (a.u[v] + b.u[v]);
    I.s[v] = ha * a.K[v] + hb * b.K[v];
  }
  I.p = I.s[0] * I.u[0] + I.s[1] * I.u[1] + I.s[2] * I.u[2];
  return I;
}

// acc += wd B(q) e_alpha for one phase's rows (row 1 of B is zero), B's rho A part with
// alpha rho A / alpha in place of rho A.
__device__ __forceinline__ void add_b64(double wd, double ia, const double* R, const double* u, const Face64& I,
                                        double* acc) {
  acc[0] = fma(wd, I.u[0], acc[0]);
  acc[2] = fma(wd, I.s[0], acc[2]);
  acc[3] = fma(wd, I.s[1], acc[3]);
  acc[4] = fma(wd, I.s[2], acc[4]);
  acc[5] = fma(wd, I.p, acc[5]);
  const double wi = wd * ia, d1 = I.u[1] - u[1], d2 = I.u[2] - u[2];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double* r = R + 3 * c;
    const double w0 = wi * r[0];
    acc[6 + 3 * c] = fma(wi, r[0] * I.u[0] + r[1] * d1 + r[2] * d2, acc[6 + 3 * c]);
    acc[7 + 3 * c] = fma(w0, u[1], acc[7 + 3 * c]);
    acc[8 + 3 * c] = fma(w0, u[2], acc[8 + 3 * c]);
  }
}

// One thread per face: acc += the path integral from a to b (30 values each), 6 nodes of
// both phases, 360 slots a node. Rolled: six copies of the node overflow the
// instruction cache.
template <int kDef>
__device__ __forceinline__ int path_thread(const Eos2x& E, const Quad6D& qd, const double* a, const double* b,
                                           double* acc) {
  int st = 0;
  const double da0 = b[0] - a[0], da1 = b[15] - a[15];
#pragma unroll 1
  for (int i = 0; i < 6; ++i) {
    const double s = qd.x[i];
    double R[2][9], ia[2];
    Half64 h[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      double m[3];
      auto at = [&](int k) { return fma(s, b[15 * p + k] - a[15 * p + k], a[15 * p + k]); };
#pragma unroll
      for (int v = 0; v < 3; ++v) m[v] = at(2 + v);
#pragma unroll
      for (int v = 0; v < 9; ++v) R[p][v] = at(6 + v);
      ia[p] = rcp64(at(0));
      st |= half64<kDef>(E.e[p], E.k[p], ia[p], m, at(5), R[p], h[p]);
    }
    const Face64 I = interface64(h[0], h[1]);
    add_b64(qd.w[i] * da0, ia[0], R[0], h[0].u, I, acc);
    add_b64(qd.w[i] * da1, ia[1], R[1], h[1].u, I, acc + 15);
  }
  return st;
}

}  // namespace hyp
