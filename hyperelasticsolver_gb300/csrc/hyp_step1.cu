// hyp_step1.cu -- single-phase FP64 step: Rusanov / LxF first-order update of
// main.jl:202-227 with the per-phase model of HyperelasticityMPh.jl at alpha == 1.
//
// A run of steps is a cell pass of the first state and one kernel per step after it:
//   cell : per cell cons2prim -> stress -> flux (11 non-zero components) and
//          lambda_i = |u1| + sqrt(max|eig(acoustic)|); block max of lambda, one
//          atomicMax per block (main.jl:204-211; HyperelasticityMPh.jl:106-175, 252-266)
//   step : dt = cfl*dx / max lambda, t += dt, and per interior cell
//          Q - dt/dx (F_{i+1/2} - F_{i-1/2}) with the Rusanov face flux
//          0.5 (f_L + f_R) - 0.5 max(lambda_L, lambda_R) (Q_R - Q_L)
//          (NumFluxes.jl:25-33; main.jl:45-48, 43-60); end cells frozen
//          (main.jl:219-220) or transmissive; then, unless it is the run's last step,
//          the cell pass of the new state from registers.
// The last step of a run leaves the cell pass out: a state the caller takes home is
// evaluated (and a bad cell in it reported) only when it is stepped from.
#include "hyp_internal.cuh"
#include "hyp_step64.cuh"

namespace hyp {

// What bounds it: FP64 issue (hyp_cell64.cuh). 1,000,003 cells, whole 10-step run with its copies:
// 10.48 ms with the general forms, 7.26 ms with these; 1000 cells, 100 steps: 4.14 ms at 256
// threads a block with the general forms, 2.38 ms.
template <int kDef, bool kSoft>
__global__ void __launch_bounds__(kBlock64, kSoft ? kSoftResident : 0) cell1_f64_kernel(const double* __restrict__ Q, int64_t n,
                                                             const __grid_constant__ EosC e,
                                                             const __grid_constant__ Eos64 kc,
                                                             double* __restrict__ F, double* __restrict__ lam,
                                                             unsigned long long* lam_slot, const double* t_now,
                                                             double t_end, DevState* S) {
  if (!(*t_now < t_end)) return;  // uniform across the grid
  const Eos64 k = in_registers64(kc);
  const int64_t i = (int64_t)blockIdx.x * kBlock64 + threadIdx.x;
  const double l = i < n ? cell1_load_pass<kDef, kSoft>(Q, n, i, e, kc, k, F, lam, S) : 0.0;
  const unsigned long long m = block_max_bits<kBlock64>(l);
  if (threadIdx.x == 0) atomicMax(lam_slot, m);
}

// Each face is evaluated once per block, by the thread of the cell on its right, into
// shared memory; both cells of a face read the same value, so the update conserves
// exactly. What bounds it: FP64 issue again, 67 slots a cell plus the step's scalars
// (84 and three divisions per warp with halved faces and a block of 256 whose last
// thread took two); warp 0 evaluates the scalars while the others wait at the barrier.
// With kCell the new state's cell pass follows in the same kernel: its FP64 work is the
// same, but a small problem saves a launch, the second kernel's ramp and its reload of
// the state, and the fluxes alternate between two buffers: 1000 cells x 100 steps 1.59 -> 1.40
// ms, 8192 cells x 4 steps on device buffers 129 -> 110 us, 1,000,003 cells unchanged (6.03 ms).
template <int kDef, bool kCell, bool kSoft>
__global__ void __launch_bounds__(kBlock64, kSoft ? kSoftResident : 0) step1_f64_kernel(Step1Args a, const __grid_constant__ EosC e,
                                                                                    const __grid_constant__ Eos64 kc) {
  __shared__ double sF[14][kBlock64];  // twice the left face of cell i0 + k
  __shared__ double s_hdt;             // half dt/dx
  __shared__ int s_more;               // the state this step makes is stepped from
  const Eos64 k = in_registers64(kc);
  const int j = threadIdx.x;
  const int64_t n = a.n;
  const double tn = *a.t_in;
  const bool active = tn < a.t_end;
  const double lmax = __longlong_as_double((long long)*a.rd);
  const bool lxf = a.flux == HYP_FLUX_LXF;
  // Rusanov: dt/dx (main.jl:225); LxF: 1/lambda with lambda = dx/dt (main.jl:223, :40)
  StepScalars sc{0.0, 0.0, 0.0};
  if (j < 32 || lxf) sc = step_scalars64(k, a.cfl, a.dx, lmax, lxf);
  if (j == 0) {
    s_hdt = 0.5 * sc.dtdx;
    s_more = kCell && tn + sc.dt < a.t_end;
    if (blockIdx.x == 0) {
      *a.t_out = active ? tn + sc.dt : tn;
      if (active) {  // an inactive step leaves the slots of the state it does not step from
        for (int c = 0; c < 2; ++c)
          if (a.clr[c]) *a.clr[c] = 0ull;
        *a.steps += 1;
      }
    }
  }
  if (!active) return;  // the same for every block
  const int64_t i = (int64_t)blockIdx.x * kCells64 + j;  // this thread's cell, and the face on its left
  double f2[14];
  if (i <= n) {
    face_twice(k, a.Q, a.F, a.lam, n, 0, n, i, lxf, sc.lam_lxf, f2);
#pragma unroll
    for (int v = 0; v < 14; ++v) sF[v][j] = f2[v];
  }
  __syncthreads();
  const bool own = j < kCells64 && i < n;
  double q[14];
  if (own) {
    const bool frozen = bc_holds(a.bc, i == 0, i == n - 1);
    const double hdt = s_hdt;
    // every load before the first store: the compiler has to keep their order
#pragma unroll
    for (int v = 0; v < 14; ++v) q[v] = a.Q[v * n + i];
#pragma unroll
    for (int v = 0; v < 14; ++v) {
      q[v] = frozen ? q[v] : __fma_rn(-hdt, sub64(k, sF[v][j + 1], f2[v]), q[v]);
      a.Qn[v * n + i] = q[v];
    }
  }
  if (!kCell || !s_more) return;
  const double l = own ? cell1_pass<kDef, kSoft>(q, a.Qn, n, i, e, kc, k, a.Fn, a.lamn, a.S) : 0.0;
  const unsigned long long m = block_max_bits<kBlock64>(l);
  if (j == 0) atomicMax(a.wr, m);
}

// ---- a whole run in one launch --------------------------------------------------

// Values of a cell its neighbour needs for their face: Q (14), fluxes (11), wave speed.
constexpr int kEdge = 14 + kNFlux1 + 1;

// Bounded wait of the run's blocks for one another (one arrival per block and step):
// what the threads of every block wrote before is visible to all after it. False if
// the wait ran out; the caller leaves the kernel. 8 blocks spend 1.5 us a step here and
// in the maximum's atomics, 150 blocks 4.2 us; a word per block that every block, or one
// block for all, reads instead measured no better (1.4 and 5.2 us; 8 blocks 1.2 us more).
__device__ __forceinline__ bool run_barrier(unsigned* count, unsigned target, int tries) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    int left = tries;
    unsigned c;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(count) : "memory");
    } while (c < target && --left > 0);
    s_ok = left > 0;
  }
  __syncthreads();
  return s_ok != 0;
}

// The end of a run at time t after s steps: the device struct, with its slots and counters
// at zero again.
__device__ __forceinline__ void run1_finish(const Run1Args& a, double t, int s) {
  if (threadIdx.x == 0) {
    if (blockIdx.x == 0) {
      a.t_out[0] = a.t_out[1] = t;
      a.S->steps += s;
    }
    __threadfence();
    if (atomicAdd(&a.S->run_done, 1u) == gridDim.x - 1) {  // the last block: all others are past the loop
      a.S->run_count = a.S->run_done = 0u;
      for (int c = 0; c < 3; ++c) a.S->lam_slots[c] = 0ull;
    }
  }
}

// Steps of a problem of at most one block per multiprocessor (127 cells each, 19,304 on
// 152 of them), all in one cooperative launch. A step of such a problem is one pass of
// FP64 issue, 240 slots (7.4 us), whatever it does about memory; as kernels of their own,
// steps spent as long again on the launch, on reloading the state and on the tail. Here
// a thread keeps its cell's state in registers, a block its cells' fluxes in shared
// memory, and the blocks meet once a step: before it they publish their edge cells and
// their part of the maximum wave speed, after it they read their neighbours' edges and
// the maximum. The arithmetic is that of cell1_pass and step1_f64_kernel, in the same
// order. 1000 cells x 100
// steps 1.39 -> 1.26 ms (1.19 since all operators are FMAs; now run1_split_f64_kernel's size), 8192 cells x 4 steps on device buffers 111 -> 80 us.
// One block a multiprocessor may have all its registers (201; held to 168 it spills: 15,000
// cells x 50 steps 608 -> 596 us).
template <int kDef>
__global__ void __launch_bounds__(kBlock64, 1) run1_f64_kernel(Run1Args a, EosC e, Eos64 kc) {
  __shared__ double sh[kEdge][kBlock64 + 1];  // slot j + 1: cell i0 + j; slot 0 and the last: the halo
  __shared__ double sF[14][kBlock64];         // twice the left face of cell i0 + j
  __shared__ double s_hdt, s_t;
  const Eos64 k = in_registers64(kc);
  const int j = threadIdx.x;
  const int64_t n = a.n, i0 = (int64_t)blockIdx.x * kCells64, i = i0 + j;
  const int cells = (int)(n - i0 < kCells64 ? n - i0 : kCells64);
  const bool own = j < cells, lxf = a.flux == HYP_FLUX_LXF;
  const bool frozen = own && bc_holds(a.bc, i == 0, i == n - 1);
  double q[14];
  if (own)
#pragma unroll
    for (int v = 0; v < 14; ++v) q[v] = a.Q[v * n + i];
  double t = *a.t_in;
  int s = 0;
  for (; s < a.max_steps && t < a.t_end; ++s) {
    double* const mine = a.edge + (size_t)((s & 1) * gridDim.x + blockIdx.x) * 2 * kEdge;
    double l = 0.0, f[14];
    if (own) {
      double u1, cm;
      int st = cell_speed64<kDef, true, true, false>(e, k, 1.0, q + 1, q[4], q + 5, f, u1, cm);
      l = add64(k, fabs(u1), cm);
      st |= is_finite64(l) ? HYP_CELL_OK : HYP_CELL_NONFINITE;
      if (st) record_err64(a.S, st, i);
#pragma unroll
      for (int v = 0; v < 14; ++v) {
        sh[v][j + 1] = q[v];
        if (flux_slot1(v) >= 0) sh[14 + flux_slot1(v)][j + 1] = f[v];
      }
      sh[kEdge - 1][j + 1] = l;
    }
    const unsigned long long top = block_max_bits<kBlock64>(l);  // (its barrier publishes sh)
    if (j < 2 * kEdge) {  // the first and the last cell, for the neighbours
      const int side = j >= kEdge, r = j - side * kEdge;
      mine[j] = sh[r][side ? cells : 1];
    }
    if (j == 0) atomicMax(&a.S->lam_slots[(a.slot0 + s) % 3], top);
    if (!run_barrier(&a.S->run_count, (unsigned)(s + 1) * gridDim.x, a.tries)) {
      if (j == 0) record_err64(a.S, HYP_CELL_TIMEOUT, i0);
      break;
    }
    const double lmax = __longlong_as_double((long long)__ldcg(&a.S->lam_slots[(a.slot0 + s) % 3]));
    if (blockIdx.x == 0 && j == 0) a.S->lam_slots[(a.slot0 + s + 2) % 3] = 0ull;  // all have read it
    if (j < 2 * kEdge) {  // the neighbours' cells beside this block's; past an end a zero-gradient ghost
      const int side = j >= kEdge, r = j - side * kEdge;
      const int nb = (int)blockIdx.x + (side ? 1 : -1);
      const double* const theirs = a.edge + (size_t)((s & 1) * gridDim.x + nb) * 2 * kEdge;
      const bool end = nb < 0 || nb >= (int)gridDim.x;
      sh[r][side ? cells + 1 : 0] = end ? sh[r][side ? cells : 1] : __ldcg(&theirs[side ? r : kEdge + r]);
    }
    StepScalars sc{0.0, 0.0, 0.0};
    if (j < 32 || lxf) sc = step_scalars64(k, a.cfl, a.dx, lmax, lxf);
    if (j == 0) {
      s_hdt = 0.5 * sc.dtdx;
      s_t = t + sc.dt;
    }
    __syncthreads();
    double f2[14];
    if (j <= cells) {  // the face between slots j and j + 1, as face_twice
      double lf = sc.lam_lxf;
      if (!lxf) {
        const double la = sh[kEdge - 1][j], lb = sh[kEdge - 1][j + 1];
        lf = bits_of(la) > bits_of(lb) && !is_nan64(la) ? la : lb;
      }
      if (!own) {  // the right cell of the block's last face
#pragma unroll
        for (int v = 0; v < 14; ++v) {
          q[v] = sh[v][j + 1];
          if (flux_slot1(v) >= 0) f[v] = sh[14 + flux_slot1(v)][j + 1];
        }
      }
#pragma unroll
      for (int v = 0; v < 14; ++v) {
        const int sl = flux_slot1(v);
        const double dq = sub64(k, q[v], sh[v][j]);
        f2[v] = sl >= 0 ? __fma_rn(-lf, dq, add64(k, sh[14 + sl][j], f[v])) : mul64(k, -lf, dq);
        sF[v][j] = f2[v];
      }
    }
    t = s_t;
    const double hdt = s_hdt;
    __syncthreads();
    if (own && !frozen)
#pragma unroll
      for (int v = 0; v < 14; ++v) q[v] = __fma_rn(-hdt, sub64(k, sF[v][j + 1], f2[v]), q[v]);
  }
  if (own && s > 0) {
    double* const Qn = a.out[s & 1];
#pragma unroll
    for (int v = 0; v < 14; ++v) Qn[v * n + i] = q[v];
  }
  run1_finish(a, t, s);
}

// The same for problems of at most 63 cells per multiprocessor (9576 on 152), two threads a
// cell, on different schedulers: FP64 issue is what a step of run1_f64_kernel waits for, and
// most schedulers have no warp of it. The second thread (half 1) forms N and its cofactors
// beside the first one's density and energies, the flux beside its wave speed, and half of
// the variables' faces and updates: about 160 FP64 instructions in sequence instead of 255.
// The state lives in shared memory. The arithmetic is the same, instruction by instruction.
// Whole runs, one thread a cell and two: 1000 cells x 100 steps 1.22 -> 0.99 ms, 8192 cells x 4
// steps on device buffers 81 -> 73 us, 50 steps of 64 to 9576 cells 0.61 to 0.77 -> 0.51 to
// 0.65 ms. With 211 registers instead of 168 (one block a multiprocessor) 1000 cells x 100 steps
// 941 -> 920 us.
constexpr int kSplitSlots = 64, kSplitCells = kSplitSlots - 1;
constexpr int kGram = sizeof(Gram64) / sizeof(double), kCellShared = 8;

template <int kDef>
__global__ void __launch_bounds__(2 * kSplitSlots, 1) run1_split_f64_kernel(Run1Args a, EosC e, Eos64 kc) {
  __shared__ double sh[kEdge][kSplitSlots + 2];  // slot j + 1: cell i0 + j; slot 0 and the last: the halo
  __shared__ double sF[14][kSplitSlots];         // twice the left face of cell i0 + j
  __shared__ double sG[kGram][kSplitSlots], sC[kCellShared][kSplitSlots];
  __shared__ double s_hdt, s_t;
  const Eos64 k = in_registers64(kc);
  const int half = threadIdx.x / kSplitSlots, j = threadIdx.x % kSplitSlots;
  const int64_t n = a.n, i0 = (int64_t)blockIdx.x * kSplitCells, i = i0 + j;
  const int cells = (int)(n - i0 < kSplitCells ? n - i0 : kSplitCells);
  const bool own = j < cells, lxf = a.flux == HYP_FLUX_LXF;
  const bool frozen = own && bc_holds(a.bc, i == 0, i == n - 1);
  if (own)
#pragma unroll
    for (int u = 0; u < 7; ++u) sh[u + 7 * half][j + 1] = a.Q[(u + 7 * half) * n + i];
  double t = *a.t_in;
  int s = 0;
  for (; s < a.max_steps && t < a.t_end; ++s) {
    double* const mine = a.edge + (size_t)((s & 1) * gridDim.x + blockIdx.x) * 2 * kEdge;
    __syncthreads();  // the state, by both halves
    double q[14], l = 0.0, e_int = 0.0;
    Cell64 c;
    if (own) {
#pragma unroll
      for (int v = 0; v < 14; ++v) q[v] = sh[v][j + 1];
      if (half) {
        const Gram64 g = gram64(k, q + 5);
        const double* p = &g.n00;
#pragma unroll
        for (int v = 0; v < kGram; ++v) sG[v][j] = p[v];
      } else {
        e_int = cell_density64<true>(k, 1.0, q + 1, q[4], q + 5, c);
      }
    }
    __syncthreads();
    if (own && !half) {
      Gram64 g;
      double* p = &g.n00;
#pragma unroll
      for (int v = 0; v < kGram; ++v) p[v] = sG[v][j];
      cell_stress64<kDef, true>(e, k, 1.0, e_int, g, c);
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        sC[v][j] = c.u[v];
        sC[3 + v][j] = c.w[v];
      }
      sC[6][j] = c.E;
      sC[7][j] = c.td;
    }
    __syncthreads();
    if (own) {
      if (half) {
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          c.u[v] = sC[v][j];
          c.w[v] = sC[3 + v][j];
        }
        c.E = sC[6][j];
        c.td = sC[7][j];
        double f[14];
        flux64<true>(k, 1.0, c, q + 1, q + 5, f);
#pragma unroll
        for (int v = 0; v < 14; ++v)
          if (flux_slot1(v) >= 0) sh[14 + flux_slot1(v)][j + 1] = f[v];
      } else {
        l = add64(k, fabs(c.u[0]), cmax64<kDef>(e, k, c));
        const int st = c.st | (is_finite64(l) ? HYP_CELL_OK : HYP_CELL_NONFINITE);
        if (st) record_err64(a.S, st, i);
        sh[kEdge - 1][j + 1] = l;
      }
    }
    const unsigned long long top = block_max_bits<2 * kSplitSlots>(l);  // (its barrier publishes sh)
    if ((int)threadIdx.x < 2 * kEdge) {  // the first and the last cell, for the neighbours
      const int side = threadIdx.x >= kEdge, r = threadIdx.x - side * kEdge;
      mine[threadIdx.x] = sh[r][side ? cells : 1];
    }
    if (threadIdx.x == 0) atomicMax(&a.S->lam_slots[(a.slot0 + s) % 3], top);
    if (!run_barrier(&a.S->run_count, (unsigned)(s + 1) * gridDim.x, a.tries)) {
      if (threadIdx.x == 0) record_err64(a.S, HYP_CELL_TIMEOUT, i0);
      break;
    }
    const double lmax = __longlong_as_double((long long)__ldcg(&a.S->lam_slots[(a.slot0 + s) % 3]));
    if (blockIdx.x == 0 && threadIdx.x == 0) a.S->lam_slots[(a.slot0 + s + 2) % 3] = 0ull;  // all have read it
    if ((int)threadIdx.x < 2 * kEdge) {  // the neighbours' cells beside this block's, as run1_f64_kernel
      const int side = threadIdx.x >= kEdge, r = threadIdx.x - side * kEdge;
      const int nb = (int)blockIdx.x + (side ? 1 : -1);
      const double* const theirs = a.edge + (size_t)((s & 1) * gridDim.x + nb) * 2 * kEdge;
      const bool end = nb < 0 || nb >= (int)gridDim.x;
      sh[r][side ? cells + 1 : 0] = end ? sh[r][side ? cells : 1] : __ldcg(&theirs[side ? r : kEdge + r]);
    }
    StepScalars sc{0.0, 0.0, 0.0};
    if (threadIdx.x >= 96 || lxf) sc = step_scalars64(k, a.cfl, a.dx, lmax, lxf);  // (a warp that loads no halo)
    if (threadIdx.x == 96) {
      s_hdt = 0.5 * sc.dtdx;
      s_t = t + sc.dt;
    }
    __syncthreads();
    double f2[7];
    auto faces = [&](auto first) {  // the face between slots j and j + 1, as face_twice
      double lf = sc.lam_lxf;
      if (!lxf) {
        const double la = sh[kEdge - 1][j], lb = sh[kEdge - 1][j + 1];
        lf = bits_of(la) > bits_of(lb) && !is_nan64(la) ? la : lb;
      }
#pragma unroll
      for (int u = 0; u < 7; ++u) {
        const int v = decltype(first)::value + u, sl = flux_slot1(v);
        const double dq = sub64(k, sh[v][j + 1], sh[v][j]);
        f2[u] = sl >= 0 ? __fma_rn(-lf, dq, add64(k, sh[14 + sl][j], sh[14 + sl][j + 1])) : mul64(k, -lf, dq);
        sF[v][j] = f2[u];
      }
    };
    if (j <= cells) {
      if (half)
        faces(std::integral_constant<int, 7>{});
      else
        faces(std::integral_constant<int, 0>{});
    }
    t = s_t;
    const double hdt = s_hdt;
    __syncthreads();
    if (own && !frozen)
#pragma unroll
      for (int u = 0; u < 7; ++u) {
        const int v = u + 7 * half;
        sh[v][j + 1] = __fma_rn(-hdt, sub64(k, sF[v][j + 1], f2[u]), sh[v][j + 1]);
      }
  }
  if (own && s > 0) {  // (each thread its own variables)
    double* const Qn = a.out[s & 1];
#pragma unroll
    for (int u = 0; u < 7; ++u) Qn[(u + 7 * half) * n + i] = sh[u + 7 * half][j + 1];
  }
  run1_finish(a, t, s);
}

// (the split kernel's blocks are the smaller ones)
size_t run1_edge_doubles(int64_t n) { return (size_t)((n + kSplitCells - 1) / kSplitCells) * 4 * kEdge; }
bool run1_fits(int64_t n, int sms) { return (n + kCells64 - 1) / kCells64 <= sms; }

cudaError_t launch_run1(cudaStream_t s, Run1Args a, EosC e) {
  Eos64 k = make_eos64(e);
  void* args[] = {&a, &e, &k};
  const unsigned split = (unsigned)((a.n + kSplitCells - 1) / kSplitCells);
  if (split <= (unsigned)a.sms) {
    const void* kern = e.default_exp ? (const void*)run1_split_f64_kernel<1> : (const void*)run1_split_f64_kernel<0>;
    return cudaLaunchCooperativeKernel(kern, dim3(split), dim3(2 * kSplitSlots), args, 0, s);
  }
  const void* kern = e.default_exp ? (const void*)run1_f64_kernel<1> : (const void*)run1_f64_kernel<0>;
  return cudaLaunchCooperativeKernel(kern, dim3((unsigned)((a.n + kCells64 - 1) / kCells64)), dim3(kBlock64), args, 0,
                                     s);
}

cudaError_t launch_cell1(cudaStream_t s, const double* Q, int64_t n, const EosC& e, double* F, double* lam,
                         unsigned long long* lam_slot, const double* t_now, double t_end, DevState* S) {
  const unsigned grid = (unsigned)((n + kBlock64 - 1) / kBlock64);
  const Eos64 k = make_eos64(e);
  auto kern = grid > kSoftBlocks ? (e.default_exp ? cell1_f64_kernel<1, true> : cell1_f64_kernel<0, true>)
                                 : (e.default_exp ? cell1_f64_kernel<1, false> : cell1_f64_kernel<0, false>);
  kern<<<grid, kBlock64, 0, s>>>(Q, n, e, k, F, lam, lam_slot, t_now, t_end, S);
  return cudaGetLastError();
}

cudaError_t launch_step1(cudaStream_t s, const Step1Args& a, const EosC& e) {
  const unsigned grid = (unsigned)((a.n + kCells64 - 1) / kCells64);
  const Eos64 k = make_eos64(e);
  auto kern = !a.Fn ? step1_f64_kernel<1, false, false>
              : grid > kSoftBlocks
                  ? (e.default_exp ? step1_f64_kernel<1, true, true> : step1_f64_kernel<0, true, true>)
                  : (e.default_exp ? step1_f64_kernel<1, true, false> : step1_f64_kernel<0, true, false>);
  kern<<<grid, kBlock64, 0, s>>>(a, e, k);
  return cudaGetLastError();
}

cudaError_t launch_cell1_f64(hyp_ctx* c, int p, unsigned long long* lam_slot, const double* t_now, double t_end) {
  return launch_cell1(c->stream, c->Q[p], c->n, c->eos[0], c->flux1[p], c->lam1[p], lam_slot, t_now, t_end, c->st);
}

static Step1Args step1_args(hyp_ctx* c, int p, unsigned long long* rd, unsigned long long* wr, unsigned long long* clr0,
                     unsigned long long* clr1, double t_end) {
  Step1Args a;
  a.Q = c->Q[p];
  a.Qn = c->Q[1 - p];
  a.F = c->flux1[p];
  a.lam = c->lam1[p];
  a.Fn = wr ? c->flux1[1 - p] : nullptr;
  a.lamn = wr ? c->lam1[1 - p] : nullptr;
  a.rd = rd;
  a.wr = wr;
  a.clr[0] = clr0;
  a.clr[1] = clr1;
  a.t_in = &c->st->t[p];
  a.t_out = &c->st->t[1 - p];
  a.steps = &c->st->steps;
  a.t_end = t_end;
  a.cfl = c->cfg.cfl;
  a.dx = ctx_dx(c);
  a.n = c->n;
  a.flux = c->cfg.flux;
  a.bc = ctx_bc(c);
  a.S = c->st;
  return a;
}

// The update of the step of parity p, with the max wave speed in `rd`, clearing the
// `clr` slots.
cudaError_t launch_update1_f64(hyp_ctx* c, int p, unsigned long long* rd, unsigned long long* clr0,
                               unsigned long long* clr1, double t_end) {
  return launch_step1(c->stream, step1_args(c, p, rd, nullptr, clr0, clr1, t_end), c->eos[0]);
}

// At most max_steps steps from step k on, of a problem that fits run1_fits.
cudaError_t launch_run1_f64(hyp_ctx* c, long long k, int max_steps, double t_end) {
  const int p = (int)(k & 1);
  Run1Args a;
  a.slot0 = (int)(k % 3);
  a.Q = c->Q[p];
  a.out[0] = c->Q[p];
  a.out[1] = c->Q[1 - p];
  a.edge = c->flux1[0];
  a.t_in = &c->st->t[p];
  a.t_out = c->st->t;
  a.max_steps = max_steps;
  a.t_end = t_end;
  a.cfl = c->cfg.cfl;
  a.dx = ctx_dx(c);
  a.n = c->n;
  a.flux = c->cfg.flux;
  a.bc = ctx_bc(c);
  a.tries = c->run_tries;
  a.sms = c->sms;
  a.S = c->st;
  return launch_run1(c->stream, a, c->eos[0]);
}

// Step k of a run (first / last of it): the max wave speed of the state before step k
// is in lam_slots[k % 3]. The slots rotate: step k reads k % 3, its cell pass writes
// (k + 1) % 3 and it clears (k + 2) % 3; a run's last step clears both others, and a step
// past t_end none, so a run always starts on a cleared slot with the next one cleared.
// A context without room for the second flux buffer runs the two kernels apart.
cudaError_t launch_run_step1_f64(hyp_ctx* c, long long k, double t_end, bool first, bool last) {
  const int p = (int)(k & 1);
  unsigned long long* s = c->st->lam_slots;
  unsigned long long *rd = s + k % 3, *nx = s + (k + 1) % 3, *cl = s + (k + 2) % 3;
  const bool apart = c->flux1[1] == c->flux1[0];
  if (first || apart) {
    const cudaError_t e = launch_cell1_f64(c, p, rd, &c->st->t[p], t_end);
    if (e != cudaSuccess) return e;
  }
  if (last || apart) return launch_update1_f64(c, p, rd, nx, cl, t_end);
  return launch_step1(c->stream, step1_args(c, p, rd, nx, cl, nullptr, t_end), c->eos[0]);
}

}  // namespace hyp
