// Host build of the compact forms' integer-product route (hyp_cell64.cuh, hyp_adjoint64.cuh),
// for tests/test_tails64_host.py.
#include "../hyperelasticsolver_gb300/csrc/hyp_adjoint64.cuh"

using namespace hyp;

static EosC eos(const double* p) { return make_eos(p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7]); }

static const double EP0[8] = {8.93, 4.6, 3.9e-4, 300.0, 2.1, 1.0, 3.0, 2.0};

extern "C" {
// q: one phase (15 values); out, plain: flux (14), u1, c_max by integer and by the hardware's
// products, st their statuses; returns whether the integer products are held for
int t64_cell(const double* p, const double* q, double* out, double* plain, int* st) {
  const EosC e = eos(p);
  const Eos64 k = make_eos64(e);
  st[0] = cell_speed64<1, false, true, true>(e, k, q[0], q + 2, q[5], q + 6, out, out[14], out[15]);
  st[1] = cell_plain64<1, false>(e, k, q[0], q + 2, plain);
  double f[14], u1, cm;
  int s;
  return cell_try64<1, false, true, true>(e, k, q[0], q + 2, q[5], q + 6, f, u1, cm, s);
}
// q: one single-phase cell (14 values); out, plain: qb (14), d/db0sq, d/dk0. left: what the
// integer products leave to do, and the hardware's after them
void t64_vjp(const double* p, const double* q, const double* fb, double lb, double* out, double* plain, int* left) {
  const EosC e = eos(p);
  const Eos64 k = make_eos64(e);
  EosBar a{0.0, 0.0}, b{0.0, 0.0}, c{0.0, 0.0}, d{0.0, 0.0};
  cell_vjp64<1, true>(e, k, q, fb, lb, out, a);
  cell_vjp64<1, false>(e, k, q, fb, lb, plain, b);
  out[14] = a.b0sq, out[15] = a.k0, plain[14] = b.b0sq, plain[15] = b.k0;
  double qb[14] = {};
  int st;
  left[0] = cell_vjp_try64<1, true>(e, k, q, fb, lb, qb, c, st);
  left[1] = cell_vjp_try64<1, false>(e, k, q, fb, lb, qb, d, st);
}
// dt, the LxF lambda and dt/dx of a step
void t64_scalars(double cfl, double dx, double lmax, int lxf, double* out) {
  const StepScalars s = step_scalars64(make_eos64(eos(EP0)), cfl, dx, lmax, lxf != 0);
  out[0] = s.dt, out[1] = s.lam_lxf, out[2] = s.dtdx;
}
}
