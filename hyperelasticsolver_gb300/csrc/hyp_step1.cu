// hyp_step1.cu -- single-phase FP64 step: Rusanov / LxF first-order update of
// main.jl:202-227 with the per-phase model of HyperelasticityMPh.jl at alpha == 1.
//
// One step = two kernels on the context stream:
//   cell   : per cell cons2prim -> stress -> flux (11 non-zero components) and
//            lambda_i = |u1| + sqrt(max|eig(acoustic)|); block max of lambda by
//            warp shuffles and one shared-memory pass, one atomicMax per block.
//            (main.jl:204-211; HyperelasticityMPh.jl:106-175, 252-266)
//   update : dt = cfl*dx / max lambda, t += dt, and per interior cell
//            Q - dt/dx (F_{i+1/2} - F_{i-1/2}) with the Rusanov face flux
//            0.5 (f_L + f_R) - 0.5 max(lambda_L, lambda_R) (Q_R - Q_L)
//            (NumFluxes.jl:25-33; main.jl:45-48, 43-60); end cells frozen
//            (main.jl:219-220) or transmissive.
// The flux/wave-speed work is done once per cell; the update kernel streams
// state, fluxes and speeds (SoA, coalesced 8-byte loads along the cell index).
#include "hyp_internal.cuh"
#include "hyp_step64.cuh"

namespace hyp {

// What bounds it: FP64 issue (hyp_cell64.cuh). 1,000,003 cells, whole 10-step run with its copies:
// 10.48 ms with the general forms, 7.26 ms with these; 1000 cells, 100 steps: 4.14 ms at 256
// threads a block with the general forms, 2.38 ms.
template <int kDef>
__global__ void __launch_bounds__(kBlock64) cell1_f64_kernel(const double* __restrict__ Q, int64_t n, EosC e, Eos64 k,
                                                             double* __restrict__ F, double* __restrict__ lam,
                                                             unsigned long long* lam_slot, const double* t_now,
                                                             double t_end, DevState* S) {
  if (!(*t_now < t_end)) return;  // uniform across the grid
  const int64_t i = (int64_t)blockIdx.x * kBlock64 + threadIdx.x;
  const double l = i < n ? cell1_pass<kDef>(Q, n, i, e, k, F, lam, S) : 0.0;
  const unsigned long long m = block_max_bits<kBlock64>(l);
  if (threadIdx.x == 0) atomicMax(lam_slot, m);
}

// Each face is evaluated once per block, by the thread of the cell on its right, into
// shared memory; both cells of a face read the same value, so the update conserves
// exactly. What bounds it: FP64 issue again, 67 slots a cell plus the step's scalars
// (84 and three divisions per warp with halved faces and a block of 256 whose last
// thread took two); warp 0 evaluates the scalars while the others wait at the barrier.
// Whole runs as above: 1000 cells 2.38 -> 1.97 ms, 1,000,003 cells 7.26 -> 6.07 ms.
__global__ void __launch_bounds__(kBlock64) update1_f64_kernel(const double* __restrict__ Q, double* __restrict__ Qn,
                                                               int64_t n, const double* __restrict__ F,
                                                               const double* __restrict__ lam,
                                                               const unsigned long long* lam_in,
                                                               unsigned long long* lam_next, const double* t_in,
                                                               double* t_out, long long* steps, double t_end,
                                                               double cfl, double dx, int flux, int bc) {
  __shared__ double sF[14][kBlock64];  // twice the left face of cell i0 + k
  __shared__ double s_hdt;             // half dt/dx
  const int j = threadIdx.x;
  const double tn = *t_in;
  const bool active = tn < t_end;
  const double lmax = __longlong_as_double((long long)*lam_in);
  const bool lxf = flux == HYP_FLUX_LXF;
  // Rusanov: dt/dx (main.jl:225); LxF: 1/lambda with lambda = dx/dt (main.jl:223, :40)
  StepScalars sc{0.0, 0.0, 0.0};
  if (j < 32 || lxf) sc = step_scalars64(cfl, dx, lmax, lxf);
  if (j == 0) s_hdt = 0.5 * sc.dtdx;
  if (blockIdx.x == 0 && j == 0) {
    *t_out = active ? tn + sc.dt : tn;
    *lam_next = 0ull;
    if (active) *steps += 1;
  }
  if (!active) return;  // the same for every block
  const int64_t i = (int64_t)blockIdx.x * kCells64 + j;  // this thread's cell, and the face on its left
  double f2[14];
  if (i <= n) {
    face_twice(Q, F, lam, n, 0, n, i, lxf, sc.lam_lxf, f2);
#pragma unroll
    for (int v = 0; v < 14; ++v) sF[v][j] = f2[v];
  }
  __syncthreads();
  if (j == kCells64 || i >= n) return;
  const bool frozen = bc_holds(bc, i == 0, i == n - 1);
  const double hdt = s_hdt;
#pragma unroll
  for (int v = 0; v < 14; ++v) {
    const double qc = Q[v * n + i];
    Qn[v * n + i] = frozen ? qc : __fma_rn(-hdt, __dsub_rn(sF[v][j + 1], f2[v]), qc);
  }
}

cudaError_t launch_cell1(cudaStream_t s, const double* Q, int64_t n, const EosC& e, double* F, double* lam,
                         unsigned long long* lam_slot, const double* t_now, double t_end, DevState* S) {
  const unsigned grid = (unsigned)((n + kBlock64 - 1) / kBlock64);
  const Eos64 k = make_eos64(e);
  if (e.default_exp)
    cell1_f64_kernel<1><<<grid, kBlock64, 0, s>>>(Q, n, e, k, F, lam, lam_slot, t_now, t_end, S);
  else
    cell1_f64_kernel<0><<<grid, kBlock64, 0, s>>>(Q, n, e, k, F, lam, lam_slot, t_now, t_end, S);
  return cudaGetLastError();
}

cudaError_t launch_update1(cudaStream_t s, const double* Q, double* Qn, int64_t n, const double* F, const double* lam,
                           const unsigned long long* lam_in, unsigned long long* lam_next, const double* t_in,
                           double* t_out, long long* steps, double t_end, double cfl, double dx, int flux, int bc) {
  const unsigned grid = (unsigned)((n + kCells64 - 1) / kCells64);
  update1_f64_kernel<<<grid, kBlock64, 0, s>>>(Q, Qn, n, F, lam, lam_in, lam_next, t_in, t_out, steps, t_end, cfl, dx,
                                               flux, bc);
  return cudaGetLastError();
}

cudaError_t launch_cell1_f64(hyp_ctx* c, int p, unsigned long long* lam_slot, const double* t_now, double t_end) {
  return launch_cell1(c->stream, c->Q[p], c->n, c->eos[0], c->F, c->lam, lam_slot, t_now, t_end, c->st);
}

cudaError_t launch_update1_f64(hyp_ctx* c, int p, double t_end) {
  return launch_update1(c->stream, c->Q[p], c->Q[1 - p], c->n, c->F, c->lam, &c->st->lam_bits[p],
                        &c->st->lam_bits[1 - p], &c->st->t[p], &c->st->t[1 - p], &c->st->steps, t_end, c->cfg.cfl,
                        ctx_dx(c), c->cfg.flux, ctx_bc(c));
}

}  // namespace hyp
