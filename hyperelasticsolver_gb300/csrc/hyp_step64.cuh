// hyp_step64.cuh -- device helpers shared by the FP64 step kernels (hyp_step1.cu,
// hyp_batch.cu, hyp_step2.cu).
#pragma once
#include "hyp_internal.cuh"
#include "hyp_cell64.cuh"

namespace hyp {

// Threads of an FP64 cell block. One block's four warps sit on an SM's four
// schedulers, so 152 blocks (19,456 cells) already take one pass of the GPU; with 256
// threads a small problem ran two warps on each scheduler of half as many SMs (1000
// cells: 33 us per cell pass against 16 with the same code at 128).
constexpr int kBlock64 = 128;

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

// The single-phase cell pass of cell i: its flux (kNFlux1 rows of F) and wave speed,
// stored and returned; a bad cell is recorded.
template <int kDef>
__device__ __forceinline__ double cell1_pass(const double* __restrict__ Q, int64_t n, int64_t i, const EosC& e,
                                             const Eos64& k, double* __restrict__ F, double* __restrict__ lam,
                                             DevState* S) {
  double q[14], f[14];
#pragma unroll
  for (int v = 0; v < 14; ++v) q[v] = Q[v * n + i];
  const Cell64 c = cell64<kDef>(e, k, 1.0, q + 1, q[4], q + 5);
  flux64(1.0, c, q + 1, q + 5, f);
  const double l = fabs(c.u[0]) + cmax64<kDef>(e, k, c);
#pragma unroll
  for (int v = 0; v < 14; ++v) {
    const int sl = flux_slot1(v);
    if (sl >= 0) F[sl * n + i] = f[v];
  }
  lam[i] = l;
  const int st = c.st | (is_finite64(l) ? HYP_CELL_OK : HYP_CELL_NONFINITE);
  if (st) record_err64(S, st, i);
  return l;
}

}  // namespace hyp
