// hyp_cell64.cuh -- one phase of one cell for the FP64 step, in the fewest FP64
// instructions.
//
// What bounds the FP64 kernels on GB300 is one number. Each of an SM's four
// schedulers issues an FP64 instruction (add, multiply, fused multiply-add, compare,
// FP32 <-> FP64 conversion) over 64 cycles, whether 1 or 32 lanes are active and
// whether or not it depends on the one before: measured 64.2 cycles per warp
// instruction for one dependent chain per scheduler and for eight independent ones, a
// divide about 9 such slots, a square root about 10. In those 64 cycles the scheduler
// issues 64 FP32, integer or special-function instructions. So the time of a pass is
// (FP64 instructions per cell) x 64 cycles, no occupancy or overlap changes it, and
// everything below trades FP64 instructions for other ones:
//
//  - The closed forms use H = G^2 = i1 G - i2 I + p M with M = A A^T = G^-1
//    (Cayley-Hamilton, p = det G), so G^2 is never formed. With b = b0sq/2 p^(beta/2)
//    and a = 2/3 b i1, row 1 of the stress is s0 = -2 rho w,
//      w_j = a G0j + b p M0j + (E3 p - b i2) [j = 0] = b (H_0j - i1/3 G0j) + E3 p [j = 0]
//    (the first form for j = 1, 2, the second, without cancellation, for j = 0),
//    and along dA = e_j A[0,:] the derivatives of M's row 1 are dM_0i = [j=0] M_0i +
//    M_00 [i=j]: the acoustic tensor (n = e1) collapses to Omega = 2 O with
//      O_ij = f G0i G0j + a G_ij - b p M00 [i=j]   (i, j >= 1),  f = 4/3 b,
//      O_0j = f G00 G0j + (beta + 2) w_j           (j >= 1),
//      O_00 = f G00^2 + w_0 + (2 beta + 2)(w_0 - E3 p) + gamma T2 + beta T3
//             + alpha kE3a Pa (2 Pa - 1),
//    E3 p = T1 + T2 + T3 its bulk, thermal and shear terms. O is symmetric, so six
//    entries and the characteristic polynomial of a symmetric matrix do.
//  - Nothing is scaled that need not be: with R = alpha rho A as stored, N = R R^T and
//    its cofactors C, one factor each takes them to G and p M, and the flux of rho A
//    and its non-conservative products need R alone.
//  - Reciprocals and square roots start from rcp.approx.ftz.f64 / rsqrt.approx.ftz.f64
//    (special-function instructions, measured error 1e-6) and take one third-order step:
//    3 slots for a reciprocal, 5 for a (reciprocal) square root, to about an ulp.
//  - The spectral radius starts from FP32 roots (conversions done on the integer pipe)
//    and takes two steps with the FP32 slope, enough when the top root stands well
//    clear; the general eigen-solve is kept for the rest.
//  - Range and NaN checks compare bit patterns.
//  - Every sum and product is a fused multiply-add on registers: x + y as x 1 + y, x y as
//    x y + (-0), with 1, -0 and all other constants in registers. Measured per scheduler
//    and warp instruction: 64.1 cycles for an FMA of three registers, 76.1 for an add, a
//    multiply or an FMA with an immediate or constant-bank operand. The results are the
//    same bit for bit. Whole runs, plain operators before and FMAs now: 1,000,003 cells x
//    10 steps 6.03 -> 5.53 ms, 1000 cells x 100 steps 1.26 -> 1.19 ms, 96 problems of 256 to
//    65536 cells x 10 steps 7.10 -> 6.51 ms, two phases of 1000 cells x 50 steps 2.25 -> 2.17
//    ms, 65536 cells x 50 steps forward and back 9.55 -> 8.69 ms.
//
// Per cell 183 FP64 instructions as executed (106 to 110 with the lone products on the
// integer pipe, soft_mul64), where the forms of hyp_physics.cuh (which the function-level
// evaluators use, and these forms where wave speeds are close) execute 379; the two agree to
// a few ulps (tests/test_cell64_host.py).
#pragma once
#include <type_traits>
#include <string.h>
#include "hyp_physics.cuh"

namespace hyp {

HYP_HD long long bits_of(double x) {
#ifdef __CUDA_ARCH__
  return __double_as_longlong(x);
#else
  long long b;
  memcpy(&b, &x, sizeof b);
  return b;
#endif
}
HYP_HD double of_bits(long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(b);
#else
  double x;
  memcpy(&x, &b, sizeof x);
  return x;
#endif
}
HYP_HD unsigned bits_of_f(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  unsigned b;
  memcpy(&b, &x, sizeof b);
  return b;
#endif
}
HYP_HD float of_bits_f(unsigned b) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float x;
  memcpy(&x, &b, sizeof x);
  return x;
#endif
}

constexpr long long kInfBits = 0x7ff0000000000000ll;
HYP_HD bool is_nan64(double x) { return (bits_of(x) & 0x7fffffffffffffffll) > kInfBits; }
HYP_HD bool is_finite64(double x) { return (bits_of(x) & 0x7fffffffffffffffll) < kInfBits; }
HYP_HD bool is_positive64(double x) { return bits_of(x) > 0 && bits_of(x) <= kInfBits; }  // x > 0, NaN: no
// x < t for t < 0, NaN: no: a negative double's bit pattern, unsigned, grows with its size
HYP_HD bool below_negative64(double x, double t) {
  return (unsigned long long)bits_of(x) > (unsigned long long)bits_of(t) && !is_nan64(x);
}

// FP64 -> FP32 of x 2^-s (truncated; under- and overflow to 0 and infinity) and FP32 ->
// FP64 of x 2^s (exact for normal values and results, 0 for subnormal x) on the integer pipe:
// a conversion instruction would take a slot of the FP64 pipe.
HYP_HD float to_f32(double x, int s = 0) {
  const long long b = bits_of(x);
  const unsigned sg = (unsigned)((unsigned long long)b >> 32) & 0x80000000u;
  const int ex = (int)((b >> 52) & 0x7ff) - 896 - s;
  const unsigned m = (unsigned)(b >> 29) & 0x7fffffu;
  if (ex <= 0) return of_bits_f(sg);
  if (ex >= 255) return of_bits_f(sg | (is_nan64(x) ? 0x7fc00000u : 0x7f800000u));
  return of_bits_f(sg | ((unsigned)ex << 23) | m);
}
HYP_HD double to_f64(float x, int s = 0) {
  const unsigned b = bits_of_f(x), ex = (b >> 23) & 0xffu;
  const unsigned long long sg = (unsigned long long)(b & 0x80000000u) << 32;
  if (ex == 0u) return of_bits((long long)sg);
  if (ex == 255u) return of_bits((long long)(sg | (unsigned long long)kInfBits | ((unsigned long long)(b & 0x7fffffu) << 29)));
  return of_bits((long long)(sg | ((unsigned long long)(ex + 896u + (unsigned)s) << 52) | ((unsigned long long)(b & 0x7fffffu) << 29)));
}

// 1/x and 1/sqrt(x), sqrt(x): a special-function seed (relative error e0 < 2^-19) and
// one step of the third-order iterations r (1 + e + e^2), e = 1 - x r (Householder
// 1970, order 2) and y (1 + e/2 + 3/8 e^2), e = 1 - x y^2: remainders e0^3 and
// 5/16 (2 e0)^3, below 2^-56. 0, infinities and negative arguments come out as NaN or
// infinity, never as a finite value.
HYP_HD double seed_rcp(double x) {
#ifdef __CUDA_ARCH__
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
#else
  return of_bits(bits_of(1.0 / x) & ~0xffffffffll);
#endif
}
HYP_HD double seed_rsqrt(double x) {
#ifdef __CUDA_ARCH__
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
#else
  return of_bits(bits_of(1.0 / sqrt(x)) & ~0xffffffffll);
#endif
}
// Constants of one phase's EOS and of the forms below. A kernel takes them through
// in_registers64, so that the compiler knows them as register values only.
struct Eos64 {
  double one, nz;                            // 1, -0
  double half, c375, third, two3, four3;     // 1/2, 3/8, 1/3, 2/3, 4/3
  double c5, c6, c7, c9;                     // 5, 6, 7, 9
  double clamp;                              // 1e-6 - 1
  double inv_rho0, inv_rho0sq, inv_cvt0;     // 1/rho0, its square, 1 / (cv t0)
  double hb0sq;                              // b0sq / 2
  double kU, kE3a, kE3g;                     // as EosT
  double hbeta, beta2, beta22;               // beta/2, beta + 2, 2 beta + 2
  double h_alphasq;                          // 1 / (2 alpha^2)
};
HYP_HD Eos64 make_eos64(const EosC& e) {
  Eos64 c;
  c.one = 1.0;
  c.nz = -0.0;
  c.half = 0.5;
  c.c375 = 0.375;
  c.third = 1.0 / 3.0;
  c.two3 = 2.0 / 3.0;
  c.four3 = 4.0 / 3.0;
  c.c5 = 5.0;
  c.c6 = 6.0;
  c.c7 = 7.0;
  c.c9 = 9.0;
  c.clamp = 1e-6 - 1.0;
  c.inv_rho0 = e.inv_rho0;
  c.inv_rho0sq = e.inv_rho0 * e.inv_rho0;
  c.inv_cvt0 = e.inv_cvt0;
  c.hb0sq = 0.5 * e.b0sq;
  c.kU = e.kU;
  c.kE3a = e.kE3a;
  c.kE3g = e.kE3g;
  c.hbeta = 0.5 * e.beta;
  c.beta2 = e.beta + 2.0;
  c.beta22 = 2.0 * e.beta + 2.0;
  c.h_alphasq = 0.5 / (e.alpha * e.alpha);
  return c;
}

// x y on the integer pipe, rounded to nearest even as the FP64 pipe does: the product of
// the 53-bit significands from four 32 x 32-bit products, one shift to 53 bits, and the
// rounding carried into the exponent. worst collects the largest distance of a product's
// exponent sum from the low end of what this holds for; beyond kSoftWide some product
// overflowed or underflowed. Factors of a zero exponent count as zeros, of the largest one
// as numbers: subnormal, infinite and NaN ones are what soft_inputs64 and the callers' check
// of status and result are for (cell_try64).
// About 50 instructions and 62 cycles of a scheduler's issue, but none of its FP64 pipe:
// 16 register FMAs take a warp 1029 cycles, 8 and 8 of these together 545 (4 warps a
// scheduler) or 732 (a single warp).
constexpr unsigned kSoftLow = 0x40300000u, kSoftWide = 0x60000000u;
HYP_HD double soft_mul64(double x, double y, unsigned& worst) {
  typedef unsigned long long u64;
  const u64 bx = (u64)bits_of(x), by = (u64)bits_of(y);
  const unsigned xh = (unsigned)(bx >> 32), xl = (unsigned)bx, yh = (unsigned)(by >> 32), yl = (unsigned)by;
  const unsigned ex = xh & 0x7ff00000u, ey = yh & 0x7ff00000u, sum = ex + ey;
  // significands: x's shifted to bit 63, y's as it is; their product's high 64 bits have
  // 52 or 53 bits
  const unsigned ah = (xh << 11 | xl >> 21) | 0x80000000u, al = xl << 11, bh = (yh & 0xfffffu) | 0x100000u;
  const u64 ll = (u64)al * yl, t = (u64)ah * yl + (ll >> 32), u = (u64)al * bh + (unsigned)t;
  const u64 P = (u64)ah * bh + (t >> 32) + (u >> 32);
  const unsigned ph = (unsigned)(P >> 32), pl = (unsigned)P, lh = (unsigned)u, l0 = (unsigned)ll;
  const unsigned full = ph >> 20, up = 1u - full;  // 53 bits already, or one to shift
  unsigned mh = up ? ph << 1 | pl >> 31 : ph, ml = up ? pl << 1 | lh >> 31 : pl;
  const unsigned rest = lh << up, base = sum - 0x40000000u + (full << 20);
#ifdef __CUDA_ARCH__
  mh = __funnelshift_l(pl, ph, up);
  ml = __funnelshift_l(lh, pl, up);
  unsigned none;  // a carry out of rest.l0 + (one half less a bit) + (ml odd) rounds up
  asm("add.cc.u32 %2, %3, 0xffffffff;\n\t"
      "addc.cc.u32 %2, %4, 0xffffffff;\n\t"
      "addc.cc.u32 %2, %5, 0x7fffffff;\n\t"
      "addc.cc.u32 %0, %0, 0;\n\t"
      "addc.u32 %1, %1, %6;"
      : "+r"(ml), "+r"(mh), "=&r"(none)
      : "r"(ml & 1u), "r"(l0), "r"(rest), "r"(base));
  (void)none;
#else
  const u64 r = (u64)rest << 32 | l0, half = 1ull << 63;
  const u64 m = ((u64)(mh + base) << 32 | ml) + (r > half || (r == half && (ml & 1u)) ? 1u : 0u);
  mh = (unsigned)(m >> 32);
  ml = (unsigned)m;
#endif
  const bool zero = (ex < ey ? ex : ey) == 0u;
  const unsigned off = (zero ? 0x7fe00000u : sum) - kSoftLow;
  worst = off > worst ? off : worst;
  const unsigned sign = (xh ^ yh) & 0x80000000u;
  return of_bits((long long)((u64)((zero ? 0u : mh) | sign) << 32 | (zero ? 0u : ml)));
}

// The constants for forms whose lone products run on the FP64 pipe, and on the integer pipe.
struct Plain64 : Eos64 {
  HYP_HD explicit Plain64(const Eos64& k) : Eos64(k) {}
};
struct Soft64 : Eos64 {
  mutable unsigned worst;
  HYP_HD explicit Soft64(const Eos64& k) : Eos64(k), worst(0u) {}
};
HYP_HD bool out_of_range(const Eos64&) { return false; }
HYP_HD bool out_of_range(const Soft64& k) { return k.worst > kSoftWide; }

// Whether n values are what the forms may take on the integer pipe: zeros, or 2^-lo (250 for a
// state, of which they form fourth powers) to 2^251 in size. The tail of a wave has others: its
// components shrink by a factor a cell, down to zero, and squares of them leave the range of a
// double. A tail's cells are told here, by their state, before anything is evaluated: after 200
// to 1000 steps of a run they had taken the integer products, a general form on their results
// and then the hardware's products (two phases, 40,000 cells, 500 steps 89 -> 70 us a step; an
// adjoint step of 65,536 cells after 1000 steps 154 -> 78 with a dense seed, 140 -> 55 with a
// density misfit's). Each product that fails by itself on the FP64 pipe, where it is met, was no
// way: its 79 branches keep the compiler from mixing the two pipes' instructions (1,000,003
// cells 332 -> 437 us a step).
HYP_HD bool soft_inputs64(const double* x, int n, unsigned lo = 250u) {
  const unsigned least = (1023u - lo) << 21, wide = (lo + 251u) << 21;
  bool in = true;
  for (int v = 0; v < n; ++v) {
    const unsigned long long b = (unsigned long long)bits_of(x[v]) << 1;
    in &= (unsigned)(b >> 32) - least < wide || b == 0ull;
  }
  return in;
}

// Whether all of the warp's cells at hand are held for: one that is not has the whole warp
// take the hardware's products, which costs what they cost for that one alone, instead of one
// pass after the other (the runs above: 74 -> 70 us and, with the misfit's seed, 73 -> 55).
HYP_HD bool warp_holds(bool in) {
#ifdef __CUDA_ARCH__
  return !__any_sync(__activemask(), !in);
#else
  return in;
#endif
}

// x y, x + y, x - y: on the FP64 pipe, products by a Soft64 on the integer pipe.
HYP_HD double mul64(const Soft64& k, double x, double y) { return soft_mul64(x, y, k.worst); }
HYP_HD double mul64(const Eos64& k, double x, double y) {
#ifdef __CUDA_ARCH__
  return __fma_rn(x, y, k.nz);
#else
  return x * y;
#endif
}
HYP_HD double add64(const Eos64& k, double x, double y) {
#ifdef __CUDA_ARCH__
  return __fma_rn(x, k.one, y);
#else
  return x + y;
#endif
}
HYP_HD double sub64(const Eos64& k, double x, double y) { return add64(k, x, -y); }

HYP_HD double rcp64(const Eos64& k, double x) {
  const double r = seed_rcp(x);
  const double e = fma(-x, r, k.one);
  return fma(r, fma(e, e, e), r);
}
HYP_HD double rsqrt64(const Eos64& k, double x) {
  const double y = seed_rsqrt(x);
  const double e = fma(-mul64(k, x, y), y, k.one);
  return fma(mul64(k, y, e), fma(k.c375, e, k.half), y);
}
HYP_HD double sqrt64(const Eos64& k, double x) {
  const double y = seed_rsqrt(x), t = mul64(k, x, y);
  const double e = fma(-t, y, k.one);
  return fma(mul64(k, t, e), fma(k.c375, e, k.half), t);
}

// a / b from rb, about 1 / b: a product and one residual correction (Markstein 1990),
// 3 slots; correctly rounded up to rare last-bit cases.
HYP_HD double quot64(const Eos64& k, double a, double b, double rb) {
  const double q = mul64(k, a, rb);
  return fma(fma(-b, q, a), rb, q);
}

// A step's dt = cfl dx / max lambda, the LxF lambda = dx / dt and dt/dx (main.jl:223-225;
// for LxF the update's dt/dx is 1 / lambda, main.jl:40) without FP64 divisions (about 9 slots
// each): 13 slots for the Rusanov step, 22 for LxF. Where an argument or a quotient may be too
// large or small for the special-function seeds and the correction, or is not finite, the
// divisions. The quotients' exponents follow from the arguments', so that the check runs beside
// the products (on the quotients themselves it cost small problems 90 ns a step).
struct StepScalars {
  double dt, lam_lxf, dtdx;
};
HYP_HD StepScalars step_scalars64(const Eos64& k, double cfl, double dx, double lmax, bool lxf) {
  const double cdx = cfl * dx;
  // sign and biased exponent of the arguments, of dt (or one less) and of dt/dx (or up to two
  // less), whose reciprocal the LxF lambda is: positive, 2^-813 to 2^813
  const int el = (int)(bits_of(lmax) >> 52), ex = (int)(bits_of(dx) >> 52), ec = (int)(bits_of(cdx) >> 52);
  const int et = ec - el + 1023, er = et - ex + 1023;
  auto plain = [](int e) { return (unsigned)(e - 210) < 1626u; };
  if (!(plain(el) & plain(ex) & plain(ec) & plain(et) & plain(er))) {
    const double dt = cdx / lmax, lam = dx / dt;
    return StepScalars{dt, lam, lxf ? 1.0 / lam : dt / dx};
  }
  StepScalars s{0.0, 0.0, 0.0};
  s.dt = quot64(k, cdx, lmax, rcp64(k, lmax));
  if (lxf) {
    s.lam_lxf = quot64(k, dx, s.dt, rcp64(k, s.dt));
    s.dtdx = quot64(k, k.one, s.lam_lxf, rcp64(k, s.lam_lxf));
  } else {
    s.dtdx = quot64(k, s.dt, dx, rcp64(k, dx));
  }
  return s;
}

// One phase of a cell: primitives, stress row 1 = -2 td w, and what the acoustic
// tensor takes (unused members cost nothing once inlined).
struct Cell64 {
  double td, inv_den;  // rho_true, 1/(alpha rho_true)
  double u[3], E;
  double w[3];
  double G00, G01, G02, G11, G12, G22;
  double a, b, bM;            // a, b, b p M00
  double wE;                  // w_0 - E3 p (finite where E3 p is not)
  double T1, T2, T3, E3p;     // bulk, thermal and shear terms of E3 p, their sum
  double Pa, Pb, Pg, px;      // p^(alpha/2), p^(beta/2), p^(gamma/2), Pg (x - 1)
  bool clamped;               // the entropy argument is at its clamp
  int st;
};

// HyperelasticityMPh.jl:106-133 and EquationsOfState.jl:118-190 for one phase: ia =
// 1/alpha (kUnit: alpha is 1, ia not read), m = alpha rho u, rE = alpha rho E, R = alpha
// rho A (column-major). In three parts, the first two independent of each other: density,
// velocity and energies; N = R R^T and its cofactors; the rest. kDef = 1: the default
// exponents alpha 1, beta 3, gamma 2 at compile time; 0: any.
template <bool kUnit, class K>
HYP_HD double cell_density64(const K& k, double ia, const double* m, double rE, const double* R, Cell64& o) {
  auto M = [&k](double x, double y) { return mul64(k, x, y); };
  const double c0 = fma(R[4], R[8], -M(R[5], R[7])), c1 = fma(R[1], R[8], -M(R[7], R[2]));
  const double c2 = fma(R[1], R[5], -M(R[4], R[2]));
  const double d = fma(R[6], c2, fma(-R[3], c1, M(R[0], c0)));
  o.st = is_positive64(d) ? HYP_CELL_OK : HYP_CELL_NEG_DET;
  // rho_true = sqrt(det(R / alpha) / rho0) and its reciprocal from one root
  const double t = kUnit ? k.inv_rho0 : M(ia, k.inv_rho0);
  const double x = M(d, kUnit ? t : M(t, M(ia, ia)));
  const double r = rsqrt64(k, x);
  o.td = M(x, r);
  o.inv_den = kUnit ? r : M(r, ia);
  for (int c = 0; c < 3; ++c) o.u[c] = M(m[c], o.inv_den);
  o.E = M(rE, o.inv_den);
  return fma(-k.half, fma(o.u[2], o.u[2], fma(o.u[1], o.u[1], M(o.u[0], o.u[0]))), o.E);  // e_int
}

struct Gram64 {
  double n00, n01, n02;                 // of N
  double k00, k01, k02, k11, k12, k22;  // its cofactors
};
template <class K>
HYP_HD Gram64 gram64(const K& k, const double* R) {
  auto M = [&k](double x, double y) { return mul64(k, x, y); };
  Gram64 g;
  g.n00 = fma(R[6], R[6], fma(R[3], R[3], M(R[0], R[0])));
  g.n01 = fma(R[6], R[7], fma(R[3], R[4], M(R[0], R[1])));
  g.n02 = fma(R[6], R[8], fma(R[3], R[5], M(R[0], R[2])));
  const double n11 = fma(R[7], R[7], fma(R[4], R[4], M(R[1], R[1])));
  const double n22 = fma(R[8], R[8], fma(R[5], R[5], M(R[2], R[2])));
  const double n12 = fma(R[7], R[8], fma(R[4], R[5], M(R[1], R[2])));
  g.k00 = fma(n11, n22, -M(n12, n12));
  g.k11 = fma(g.n00, n22, -M(g.n02, g.n02));
  g.k22 = fma(g.n00, n11, -M(g.n01, g.n01));
  g.k01 = fma(g.n02, n12, -M(g.n01, n22));
  g.k02 = fma(g.n01, n12, -M(g.n02, n11));
  g.k12 = fma(g.n01, g.n02, -M(g.n00, n12));
  return g;
}

template <int kDef, bool kUnit, class K>
HYP_HD void cell_stress64(const EosC& e, const K& k, double ia, double e_int, const Gram64& g, Cell64& o) {
  auto M = [&k](double x, double y) { return mul64(k, x, y); };
  auto A = [&k](double x, double y) { return add64(k, x, y); };
  const double t = kUnit ? k.inv_rho0 : M(ia, k.inv_rho0);
  // M = N inv_den^2, p = (rho_true / rho0)^2, G = adj(M) p: p M = N (ia/rho0)^2 and
  // G = C (ia inv_den / rho0)^2
  const double g1 = M(t, o.inv_den), gs = M(g1, g1), ms = kUnit ? k.inv_rho0sq : M(t, t);
  o.G00 = M(g.k00, gs);
  o.G01 = M(g.k01, gs);
  o.G02 = M(g.k02, gs);
  o.G11 = M(g.k11, gs);
  o.G12 = M(g.k12, gs);
  o.G22 = M(g.k22, gs);
  const double i1 = M(A(A(g.k00, g.k11), g.k22), gs);
  const double s = M(o.td, k.inv_rho0);  // 1/det A = sqrt(p)
  const double p = M(s, s);
  // psi = i1^2/3 - i2 = |dev G|^2 / 2, and row 1 of the stress below, from the deviator's
  // diagonal: small numbers squared instead of large ones subtracted
  const double d0 = fma(-k.third, i1, o.G00), d1 = fma(-k.third, i1, o.G11), d2 = fma(-k.third, i1, o.G22);
  const double off = fma(o.G02, o.G02, M(o.G01, o.G01));
  const double psi = fma(k.half, fma(d2, d2, fma(d1, d1, M(d0, d0))), fma(o.G12, o.G12, off));
  if (kDef == 1) {
    o.Pa = s;
    o.Pb = M(s, p);
    o.Pg = p;
  } else {
    const double lp = log(p);
    o.Pa = exp(0.5 * e.alpha * lp);
    o.Pb = exp(0.5 * e.beta * lp);
    o.Pg = exp(0.5 * e.gamma * lp);
  }
  o.b = M(k.hb0sq, o.Pb);
  const double bp = M(o.b, psi);  // shear energy
  const double am1 = A(o.Pa, -k.one), z = M(k.kU, am1);
  // Pg (x - 1), x the entropy argument (EquationsOfState.jl:150), and its clamp (:152-154)
  o.px = M(fma(-z, am1, A(e_int, -bp)), k.inv_cvt0);
  if (is_nan64(e_int) || is_nan64(o.px) || !is_finite64(p)) o.st |= HYP_CELL_NONFINITE;
  const double least = M(k.clamp, o.Pg);
  o.clamped = below_negative64(o.px, least);
  if (o.clamped) o.px = least;
  o.T1 = kDef == 1 ? M(z, s) : e.alpha * (z * o.Pa);
  o.T2 = M(k.kE3g, o.px);
  o.T3 = M(k.hbeta, bp);
  o.E3p = A(A(o.T1, o.T2), o.T3);
  o.a = M(k.two3, M(o.b, i1));
  o.bM = M(o.b, M(g.n00, ms));
  const double h = fma(o.G00, d0, off);
  o.wE = M(o.b, h);
  o.w[0] = fma(o.b, h, o.E3p);
  o.w[1] = fma(o.a, o.G01, M(o.b, M(g.n01, ms)));
  o.w[2] = fma(o.a, o.G02, M(o.b, M(g.n02, ms)));
}

template <int kDef, bool kUnit, class K>
HYP_HD Cell64 cell64(const EosC& e, const K& k, double ia, const double* m, double rE, const double* R) {
  Cell64 o;
  const double e_int = cell_density64<kUnit>(k, ia, m, rE, R, o);
  cell_stress64<kDef, kUnit>(e, k, ia, e_int, gram64(k, R), o);
  return o;
}

// Spectral radius of 2 O by the general route, for an acoustic tensor whose top root
// does not stand clear: kept out of line, off the path of every ordinary cell.
#ifdef __CUDACC__
static __host__ __device__ __noinline__
#else
inline
#endif
double radius_general(double o00, double o11, double o22, double o01, double o02, double o12) {
  const double a[9] = {2.0 * o00, 2.0 * o01, 2.0 * o02, 2.0 * o01, 2.0 * o11, 2.0 * o12, 2.0 * o02, 2.0 * o12, 2.0 * o22};
  return spectral_radius(a);
}

// The largest eigenvalue of a symmetric O, false where it does not stand clear of the
// others' moduli: an FP32 root of the characteristic polynomial, then two steps with the
// FP32 slope. FP32 has the polynomial with the power of two of the trace taken out: its last
// coefficient is the sixth power of a speed, which in centimetres per picosecond or
// millimetres per second is not an FP32 number.
template <class K>
HYP_HD bool top_root64(const K& k, double o00, double o11, double o22, double o01, double o02, double o12,
                       double& root) {
  auto M = [&k](double x, double y) { return mul64(k, x, y); };
  auto A = [&k](double x, double y) { return add64(k, x, y); };
  // mu^3 - c2 mu^2 + c1 mu - c0
  const double tr = A(o11, o22), q = fma(o11, o22, -M(o12, o12));
  const double c2 = A(o00, tr);
  const double c1 = fma(-o02, o02, fma(-o01, o01, fma(o00, tr, q)));
  const double e1 = fma(o01, o22, -M(o12, o02)), e2 = fma(o01, o12, -M(o11, o02));
  const double c0 = fma(o02, e2, fma(-o01, e1, M(o00, q)));
  const int sh = (int)(bits_of(c2) >> 52) - 1023;  // of c2 > 0
  if (!(sh > -300 && sh < 300)) return false;
  const float C2 = to_f32(c2, sh), C1 = to_f32(c1, 2 * sh), C0 = to_f32(c0, 3 * sh);
  const float P = C1 - C2 * C2 * (1.0f / 3.0f);
  const float Q = -2.0f / 27.0f * C2 * C2 * C2 + C2 * C1 * (1.0f / 3.0f) - C0;
  // A symmetric matrix has three real roots; two equal ones (a material at rest or under
  // isotropic strain has two equal shear speeds) put the cosine at 1 up to rounding,
  // where the clamp below costs the largest root an error of second order only.
  if (!(P < 0.0f)) return false;
  const float am = 2.0f * sqrtf(-P * (1.0f / 3.0f));
  const float cc = fminf(1.0f, fmaxf(-1.0f, 3.0f * Q / (P * am)));
  const float y = am * cosf(acosf(cc) * (1.0f / 3.0f)) + C2 * (1.0f / 3.0f);
  const float sm = C2 - y, pr = C0 / y;  // sum and product of the other two
  const float other = 0.5f * fabsf(sm) + sqrtf(fmaxf(0.25f * sm * sm - pr, 0.0f));
  const float slope = (3.0f * y - 2.0f * C2) * y + C1;
  // With the others below 0.35 of it, the seed is within ~1e-6 and the slope within
  // ~1e-6 of theirs at the root: a step leaves 5e-12, the next 5e-17.
  if (!(other < 0.35f * y && slope > 1e-30f)) return false;
  const double inv = to_f64(1.0f / slope, -2 * sh);
  double rt = to_f64(y, sh);
  for (int it = 0; it < 2; ++it) rt = fma(-inv, fma(fma(A(rt, -c2), rt, c1), rt, -c0), rt);
  root = rt;
  return true;
}

// Largest acoustic wave speed sqrt(max |eig Omega|) of one phase (HyperelasticityMPh.jl:258-266).
template <int kDef, class K>
HYP_HD double cmax64(const EosC& e, const K& k, const Cell64& c) {
  auto M = [&k](double x, double y) { return mul64(k, x, y); };
  const double f = M(k.four3, c.b);
  const double f0 = M(f, c.G00), f1 = M(f, c.G01), f2 = M(f, c.G02);
  double rest;
  if (kDef == 1)  // -8 E3p + 2 T2 + 3 T3 + kE3a s (2 s - 1), T1 = kE3a s (s - 1)
    rest = fma(k.c9, c.w[0], fma(-k.c7, c.T1, fma(-k.c6, c.T2, fma(-k.c5, c.T3, M(k.kE3a, c.Pg)))));
  else
    rest = c.w[0] + k.beta22 * c.wE + e.gamma * c.T2 + e.beta * c.T3 +
           e.alpha * (k.kE3a * c.Pa * (2.0 * c.Pa - 1.0));
  const double o00 = fma(f0, c.G00, rest);
  const double o01 = fma(f0, c.G01, M(k.beta2, c.w[1])), o02 = fma(f0, c.G02, M(k.beta2, c.w[2]));
  const double o11 = fma(f1, c.G01, fma(c.a, c.G11, -c.bM)), o22 = fma(f2, c.G02, fma(c.a, c.G22, -c.bM));
  const double o12 = fma(f1, c.G02, M(c.a, c.G12));
  double rt;
  if (top_root64(k, o00, o11, o22, o01, o02, o12, rt)) return sqrt64(k, add64(k, rt, rt));
  if (out_of_range(k)) return 0.0;  // O means nothing; the cell is evaluated again
  return sqrt(radius_general(o00, o11, o22, o01, o02, o12));
}

// Physical x-flux of one phase (HyperelasticityMPh.jl:146-175), the 14 entries after
// alpha: alpha rho u1 is m1 itself, and the rho A part is u1 R - u (row 1 of R), whose
// first row is zero.
template <bool kUnit, class K>
HYP_HD void flux64(const K& k, double alpha, const Cell64& c, const double* m, const double* R, double* f) {
  auto M = [&k](double x, double y) { return mul64(k, x, y); };
  const double den = kUnit ? c.td : M(alpha, c.td), d2 = add64(k, den, den);  // -alpha s0 = 2 alpha rho w
  const double S0 = M(d2, c.w[0]), S1 = M(d2, c.w[1]), S2 = M(d2, c.w[2]);
  f[0] = m[0];
  f[1] = fma(m[0], c.u[0], S0);
  f[2] = fma(m[0], c.u[1], S1);
  f[3] = fma(m[0], c.u[2], S2);
  f[4] = fma(m[0], c.E, fma(c.u[2], S2, fma(c.u[1], S1, M(c.u[0], S0))));
  for (int b = 0; b < 3; ++b) {
    f[5 + 3 * b] = 0.0;
    f[6 + 3 * b] = fma(c.u[0], R[1 + 3 * b], -M(c.u[1], R[3 * b]));
    f[7 + 3 * b] = fma(c.u[0], R[2 + 3 * b], -M(c.u[2], R[3 * b]));
  }
}

// One phase of a cell: status, u1, c_max and with kFlux the flux; kSoft: lone products on
// the integer pipe, the same values bit for bit. False where those are not held for: a state
// or product out of their range, or a bad cell; the results then mean nothing, and the caller
// evaluates the cell with the hardware's products. A kernel does so out of line with the
// state loaded again, so that nothing of the ordinary path is kept for it.
template <int kDef, bool kUnit, bool kFlux, bool kSoft>
HYP_HD bool cell_try64(const EosC& e, const Eos64& k, double alpha, const double* m, double rE, const double* R,
                       double* f, double& u1, double& cm, int& st) {
  if (kSoft && !warp_holds(soft_inputs64(m, 3) & soft_inputs64(&rE, 1) & soft_inputs64(R, 9) &
                           (kUnit || soft_inputs64(&alpha, 1))))
    return false;
  const typename std::conditional<kSoft, Soft64, Plain64>::type s(k);
  const Cell64 c = cell64<kDef, kUnit>(e, s, kUnit ? 1.0 : rcp64(k, alpha), m, rE, R);
  if (kFlux) flux64<kUnit>(s, alpha, c, m, R, f);
  u1 = c.u[0];
  cm = cmax64<kDef>(e, s, c);
  st = c.st;
  return !kSoft || (!out_of_range(s) && !st && is_finite64(cm));
}

// The same with the second evaluation in it. cell_plain64: with the hardware's products, q
// m, rE, R and out flux (14), u1, c_max.
template <int kDef, bool kUnit, bool kFlux, bool kSoft>
HYP_HD int cell_speed64(const EosC& e, const Eos64& k, double alpha, const double* m, double rE, const double* R,
                        double* f, double& u1, double& cm) {
  int st;
  if (!cell_try64<kDef, kUnit, kFlux, kSoft>(e, k, alpha, m, rE, R, f, u1, cm, st))
    cell_try64<kDef, kUnit, kFlux, false>(e, k, alpha, m, rE, R, f, u1, cm, st);
  return st;
}
template <int kDef, bool kUnit>
HYP_HD int cell_plain64(const EosC& e, const Eos64& k, double alpha, const double* q, double* out) {
  return cell_speed64<kDef, kUnit, true, false>(e, k, alpha, q, q[3], q + 4, out, out[14], out[15]);
}

}  // namespace hyp
