// Host build of the path integrals on the compact forms (hyp_paths64.cuh) for
// tests/test_paths64_host.py.
#include "../hyperelasticsolver_gb300/csrc/hyp_paths64.cuh"

using namespace hyp;

extern "C" {
// e: two phases' 8 parameters each; rule: 6 nodes then 6 weights; a, b: 30 values. acc
// (30) = the integral as the step takes it; ref (30) = with all 6 nodes of the general
// forms (path_integral_add). Returns the nodes taken.
int p64_path(const double* e, const double* rule, const double* a, const double* b, double* acc, double* ref) {
  EosC eos[2];
  Eos2x E;
  for (int p = 0; p < 2; ++p) {
    const double* q = e + 8 * p;
    eos[p] = make_eos(q[0], q[1], q[2], q[3], q[4], q[5], q[6], q[7]);
  }
  E = make_eos2x(eos);
  Quad6D qd;
  for (int i = 0; i < 6; ++i) {
    qd.x[i] = rule[i];
    qd.w[i] = rule[6 + i];
  }
  if (eos[0].default_exp && eos[1].default_exp)
    path_thread<1>(E, qd, a, b, acc);
  else
    path_thread<0>(E, qd, a, b, acc);
  path_integral_add(eos, qd, a, b, ref);
  return path_nodes(eos, a, b);
}
}
