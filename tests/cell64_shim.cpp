// Host build of the FP64 step's compact cell forms (hyp_cell64.cuh) beside the general
// ones (hyp_physics.cuh), for tests/test_cell64_host.py.
#include "../hyperelasticsolver_gb300/csrc/hyp_adjoint64.cuh"

using namespace hyp;

template <int kDef>
static int compact(const EosC& e, const double* q, double* out) {
  const Eos64 k = make_eos64(e);
  return cell_speed64<kDef, false, true, true>(e, k, q[0], q + 2, q[5], q + 6, out, out[14], out[15]);
}

extern "C" {
// q: one phase (15 values); out: flux (14 after alpha), u1, c_max; returns the status bits
int c64_compact(const double* p, const double* q, double* out) {
  const EosC e = make_eos(p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7]);
  return e.default_exp ? compact<1>(e, q, out) : compact<0>(e, q, out);
}
int c64_general(const double* p, const double* q, double* out) {
  const EosC e = make_eos(p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7]);
  Prim P;
  const int st = cons_to_prim(e, q[0], q + 2, q[5], q + 6, P);
  const StressC c = stress_coeffs(e, P.k, P.w, P.xm1);
  double s0[3];
  phase_flux(e, q[0], P, c, out, s0);
  out[14] = P.u[0];
  out[15] = phase_cmax(e, P, c);
  return st;
}
// out: qb (14), d/db0sq, d/dk0 of one single-phase cell
int c64_vjp_compact(const double* p, const double* q, const double* fb, double lb, double* out) {
  const EosC e = make_eos(p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7]);
  const Eos64 k = make_eos64(e);
  EosBar b{0.0, 0.0};
  const int st = e.default_exp ? cell_vjp64<1, true>(e, k, q, fb, lb, out, b) : cell_vjp64<0, true>(e, k, q, fb, lb, out, b);
  out[14] = b.b0sq;
  out[15] = b.k0;
  return st;
}
int c64_vjp_plain(const double* p, const double* q, const double* fb, double lb, double* out) {
  const EosC e = make_eos(p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7]);
  const Eos64 k = make_eos64(e);
  EosBar b{0.0, 0.0};
  const int st = e.default_exp ? cell_vjp64<1, false>(e, k, q, fb, lb, out, b) : cell_vjp64<0, false>(e, k, q, fb, lb, out, b);
  out[14] = b.b0sq;
  out[15] = b.k0;
  return st;
}
int c64_vjp_general(const double* p, const double* q, const double* fb, double lb, double* out) {
  const EosC e = make_eos(p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7]);
  EosBar b{0.0, 0.0};
  const int st = cell_vjp(e, q, fb, lb, out, b);
  out[14] = b.b0sq;
  out[15] = b.k0;
  return st;
}
// the forms with the hardware's products (cell_plain64)
int c64_plain(const double* p, const double* q, double* out) {
  const EosC e = make_eos(p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7]);
  const Eos64 k = make_eos64(e);
  return e.default_exp ? cell_plain64<1, false>(e, k, q[0], q + 2, out) : cell_plain64<0, false>(e, k, q[0], q + 2, out);
}
double c64_soft_mul(double x, double y, int* in_range) {
  unsigned worst = 0u;
  const double r = soft_mul64(x, y, worst);
  *in_range = worst <= kSoftWide;
  return r;
}
float c64_to_f32(double x) { return to_f32(x); }
double c64_to_f64(float x) { return to_f64(x); }
}
