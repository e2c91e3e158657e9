// hyp_step64.cuh -- device helpers shared by the FP64 step kernels (hyp_step1.cu,
// hyp_batch.cu, hyp_step2.cu).
#pragma once
#include "hyp_internal.cuh"
#include "hyp_cell64.cuh"

namespace hyp {

// Threads of an FP64 cell block. One block's four warps sit on an SM's four
// schedulers, so 152 blocks (19,456 cells) already take one pass of the GPU; with 256
// threads a small problem runs two warps on each scheduler of half as many SMs, twice the
// time of one.
constexpr int kBlock64 = 128;

// Grids of more blocks than this, one a multiprocessor, take the lone products of a cell
// pass on the integer pipe (hyp_cell64.cuh): the two pipes overlap where a scheduler has
// warps to choose from, so those kernels keep to 128 registers and four blocks resident
// (1,000,003 cells x 10 steps: 4.53 ms, 4.49 now; with two, three, five 5.19, 4.71, 4.68, and 5.48
// with all products on the FP64 pipe). 50 steps of 20,000 cells (158 blocks) 1.05 -> 1.01 ms, of
// 38,000 1.18 -> 1.13, of 70,000 1.99 -> 1.64; two phases (64 cells a block), 20 HLL steps of
// 9,700 cells (152 blocks) 1.02 -> 1.10 ms, of 14,000 1.15 on either pipe, of 38,000 1.57 ->
// 1.51, and 20 LxF steps 0.78 -> 0.83, 0.92 -> 0.88, 1.42 -> 1.26.
constexpr unsigned kSoftBlocks = 152;
constexpr int kSoftResident = 4;

// The constants as register values (hyp_cell64.cuh: an operand from the constant bank or
// a uniform register slows an FMA by a fifth). Their high words pass through an exclusive
// or with a zero that only the launch knows (all grids here have gridDim.y = 1) and that a
// thread's index makes a per-thread value: two integer instructions each, which may be
// done again where a register is short. Through shared memory instead they took a barrier
// and 0.9 us more of each kernel.
__device__ __forceinline__ Eos64 in_registers64(const Eos64& k) {
  const int zero = (int)(threadIdx.x & (gridDim.y - 1));
  Eos64 r;
  const double* from = &k.one;
  double* to = &r.one;
#pragma unroll
  for (int i = 0; i < (int)(sizeof(Eos64) / sizeof(double)); ++i)
    to[i] = __hiloint2double(__double2hiint(from[i]) ^ zero, __double2loint(from[i]));
  return r;
}

// The caller's phase of two: those of the phase by selection, which leaves registers too.
__device__ __forceinline__ Eos64 in_registers64(const Eos64* k, int ph) {
  Eos64 r = in_registers64(k[0]);
  const double *k0 = &k[0].inv_rho0, *k1 = &k[1].inv_rho0;
  double* to = &r.inv_rho0;
#pragma unroll
  for (int i = 0; i < (int)(&r.h_alphasq - &r.inv_rho0) + 1; ++i) to[i] = ph ? k1[i] : k0[i];
  return r;
}

__device__ __forceinline__ void record_err64(DevState* S, int code, long long cell) {
  if (atomicCAS(&S->err_code, 0, code) == 0) S->err_cell = cell;
}

// Maximum over the block of a wave speed l >= 0 (a NaN counts as 0, as fmax treats it),
// valid in thread 0: non-negative doubles order as their bit patterns, high word
// first, so the integer pipe's warp reductions do it (a shuffle tree of FP64 maxima is
// 15 slots of the FP64 pipe).
template <int BLOCK>
__device__ __forceinline__ unsigned long long block_max_bits(double l) {
  __shared__ unsigned long long red[BLOCK / 32];
  const unsigned long long b = is_nan64(l) ? 0ull : (unsigned long long)bits_of(l);
  const unsigned hi = (unsigned)(b >> 32), lo = (unsigned)b;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ((unsigned long long)mh << 32) | ml;
  __syncthreads();
  unsigned long long m = red[0];
  if (threadIdx.x == 0)
    for (int w = 1; w < BLOCK / 32; ++w) m = red[w] > m ? red[w] : m;
  return m;
}

// The single-phase cell pass of cell i in state q, which is at Q too: its flux (kNFlux1 rows
// of F) and wave speed, stored and returned; a bad cell is recorded. e and kc are the
// kernel's own parameters (__grid_constant__: they have an address), k is kc in registers.
template <int kDef>
static __device__ __noinline__ double cell1_again(const double* Q, int64_t n, int64_t i, const EosC& e, const Eos64& kc,
                                                  double* F, double* lam, DevState* S);
template <int kDef, bool kSoft>
__device__ __forceinline__ double cell1_pass(const double* q, const double* Q, int64_t n, int64_t i, const EosC& e,
                                             const Eos64& kc, const Eos64& k, double* __restrict__ F,
                                             double* __restrict__ lam, DevState* S) {
  double f[14];
  double u1, cm;
  int st;
  if (!cell_try64<kDef, true, true, kSoft>(e, k, 1.0, q + 1, q[4], q + 5, f, u1, cm, st) && kSoft)
    return cell1_again<kDef>(Q, n, i, e, kc, F, lam, S);
  const double l = add64(k, fabs(u1), cm);
#pragma unroll
  for (int v = 0; v < 14; ++v) {
    const int sl = flux_slot1(v);
    if (sl >= 0) F[sl * n + i] = f[v];
  }
  lam[i] = l;
  st |= is_finite64(l) ? HYP_CELL_OK : HYP_CELL_NONFINITE;
  if (st) record_err64(S, st, i);
  return l;
}
template <int kDef, bool kSoft>
__device__ __forceinline__ double cell1_load_pass(const double* Q, int64_t n, int64_t i, const EosC& e,
                                                  const Eos64& kc, const Eos64& k, double* __restrict__ F,
                                                  double* __restrict__ lam, DevState* S) {
  double q[14];
#pragma unroll
  for (int v = 0; v < 14; ++v) q[v] = Q[v * n + i];
  return cell1_pass<kDef, kSoft>(q, Q, n, i, e, kc, k, F, lam, S);
}
template <int kDef>
static __device__ __noinline__ double cell1_again(const double* Q, int64_t n, int64_t i, const EosC& e, const Eos64& kc,
                                                  double* F, double* lam, DevState* S) {
  return cell1_load_pass<kDef, false>(Q, n, i, e, kc, in_registers64(kc), F, lam, S);
}

// Cells a block of the update kernels owns: thread j evaluates the face left of cell
// first + j, so the last thread's face closes the last owned cell and no thread
// evaluates two (a second face on one thread is a second pass of its whole warp).
constexpr int kCells64 = kBlock64 - 1;

// Twice the Rusanov flux of the face between cells f - 1 and f of the problem [lo, hi)
// (a zero-gradient ghost past either end): (f_a + f_b) - lambda (q_b - q_a), lambda =
// max(lambda_a, lambda_b) (NumFluxes.jl:25-33, main.jl:45-48) or the LxF one. Doubling is
// exact, so this is the flux's own rounding with a multiplication less per variable;
// the rounding sequence is fixed (explicit intrinsics), so the step commutes with x -> -x.
__device__ __forceinline__ void face_twice(const Eos64& k, const double* __restrict__ Q, const double* __restrict__ F,
                                           const double* __restrict__ lam, int64_t n, int64_t lo, int64_t hi,
                                           int64_t f, bool lxf, double lam_lxf, double* f2) {
  const int64_t a = f > lo ? f - 1 : lo, b = f < hi ? f : hi - 1;
  double lf = lam_lxf;
  if (!lxf) {
    const double la = lam[a], lb = lam[b];  // la > lb ? la : lb of non-negative values
    lf = bits_of(la) > bits_of(lb) && !is_nan64(la) ? la : lb;
  }
#pragma unroll
  for (int v = 0; v < 14; ++v) {
    const int sl = flux_slot1(v);
    const double dq = sub64(k, Q[v * n + b], Q[v * n + a]);
    f2[v] = sl >= 0 ? __fma_rn(-lf, dq, add64(k, F[sl * n + a], F[sl * n + b])) : mul64(k, -lf, dq);
  }
}

}  // namespace hyp
