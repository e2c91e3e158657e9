// hyp_step2.cu -- two-phase FP64 step with the path-conservative HLL flux
// (main.jl:202-241 with update_cell :43-60 and NumFluxes.hll :70-132) or the
// path-conservative Lax-Friedrichs flux (update_cell :30-41, NumFluxes.lxf :25-60).
//
// A run of steps is a cell pass of the first state and three kernels per step:
//   cell   : per cell and phase, the flux (HyperelasticityMPh.jl:140-175) and
//            wave-speed bounds (:252-266); lambda_i = max |speed|, block max ->
//            one atomicMax (main.jl:204-212);
//   face   : per face and phase, the midpoint's wave speeds and s_l, s_r (HLL), and the
//            whole face wherever its path integrals vanish; the other faces go to a list;
//   paths  : the listed faces' path integrals of B (HLL: three Gauss-Legendre ones, up to
//            18 evaluations of B instead of the 30 the reference makes, since the
//            integrals repeated in D- and D+ are the same; LxF: one Gauss-Lobatto);
//   step   : dt = cfl dx / max lambda, t += dt, Q_i - dt/dx ((F_r - F_l) + (D-_{i+1/2} + D+_{i-1/2}))
//            with frozen or transmissive ends (F = 0 for HLL, which folds the conservative
//            part into D+-; the LxF face flux otherwise), then, unless it is the run's
//            last step, the cell pass of the new state.
//
// What bounds them is FP64 issue (hyp_cell64.cuh), so the counts per face matter and
// nothing else does. B dQ is a column times d(alpha) (HyperelasticityMPh.jl:178-250):
// where both cells of a face have the same volume fractions every path integral is
// exactly zero and so is Q_hll's jump in alpha, and the face is the plain HLL (or LxF)
// formula: about 370 FP64 instructions instead of 10,400 (6,600 with the integrals). That holds on most faces of a run
// that starts from states of piecewise-constant volume fraction (main.jl:99-106, the
// smoothed interface away from its 8 cells); where the fractions vary in every cell
// (main.jl:110-123) all faces are listed.
#include <algorithm>
#include "hyp_internal.cuh"
#include "hyp_paths64.cuh"
#include "hyp_step64.cuh"

namespace hyp {

constexpr int kPairCells = 64;             // cells (faces) of a block: one thread per phase of each
constexpr int kPair64 = 2 * kPairCells;    // its threads; the phase is uniform over a warp

struct CellOut2 {
  double *F, *smin, *smax;  // fluxes [30][n], wave-speed bounds
  int64_t n;
  DevState* S;
};

// A phase's rows of F, u1 and c_max (returned) of cell i in state q (at Q too), with a bad
// cell recorded; E: the kernel's parameter, k: its constants of the phase in registers.
template <int kDef>
static __device__ __noinline__ double2 cell2_again(const double* Q, int64_t i, int ph, const Eos2x& E, const CellOut2& o);
template <int kDef, bool kSoft>
__device__ __forceinline__ double2 cell2_phase(const double* q, const double* Q, int64_t i, int ph, const Eos2x& E,
                                               const Eos64& k, const CellOut2& o) {
  double f[14], u1, cm;
  int st;
  if (!cell_try64<kDef, false, true, kSoft>(E.e[ph], k, q[0], q + 2, q[5], q + 6, f, u1, cm, st) && kSoft)
    return cell2_again<kDef>(Q, i, ph, E, o);
  double* f0 = o.F + 15 * ph * o.n + i;
#pragma unroll
  for (int r = 1; r < 15; ++r)
    if (!zero_flux_row(r)) f0[r * o.n] = f[r - 1];
  if (st) record_err64(o.S, st, i);
  return make_double2(u1, cm);
}
__device__ __forceinline__ void load_phase(const double* Q, int64_t n, int64_t i, int ph, double* q) {
  const double* q0 = Q + 15 * ph * n + i;
#pragma unroll
  for (int r = 0; r < 15; ++r) q[r] = q0[r * n];
}
template <int kDef>
static __device__ __noinline__ double2 cell2_again(const double* Q, int64_t i, int ph, const Eos2x& E, const CellOut2& o) {
  double q[15];
  load_phase(Q, o.n, i, ph, q);
  return cell2_phase<kDef, false>(q, Q, i, ph, E, in_registers64(E.k, ph), o);
}

// The cell pass of a block's 64 cells, a thread per phase in state q (15 values, at Q too;
// `in`: there is a cell): fluxes, speed bounds, and the block's max |speed| into slot. All
// threads of the block call it.
template <int kDef, bool kSoft>
__device__ __forceinline__ void cell2_pass(const double* q, const double* Q, bool in, int64_t i, const Eos2x& E,
                                           const Eos64& k, const CellOut2& o, unsigned long long* slot) {
  __shared__ double s_lo[kPairCells], s_hi[kPairCells];
  const int ph = threadIdx.x / kPairCells, j = threadIdx.x % kPairCells;
  double lo = 0.0, hi = 0.0;
  if (in) {
    const double2 s = cell2_phase<kDef, kSoft>(q, Q, i, ph, E, k, o);
    lo = sub64(k, s.x, s.y);
    hi = add64(k, s.x, s.y);
    if (ph == 1) {
      s_lo[j] = lo;
      s_hi[j] = hi;
    }
  }
  __syncthreads();
  double l = 0.0;
  if (ph == 0 && in) {
    if (s_lo[j] < lo) lo = s_lo[j];
    if (s_hi[j] > hi) hi = s_hi[j];
    o.smin[i] = lo;
    o.smax[i] = hi;
    l = fmax(fabs(lo), fabs(hi));
    if (!is_finite64(l)) record_err64(o.S, HYP_CELL_NONFINITE, i);
  }
  const unsigned long long m = block_max_bits<kPair64>(l);
  if (threadIdx.x == 0) atomicMax(slot, m);
}

template <int kDef, bool kSoft>
__global__ void __launch_bounds__(kPair64, kSoft ? kSoftResident : 0) cell2_f64_kernel(const double* __restrict__ Q, const __grid_constant__ Eos2x E,
                                                            const __grid_constant__ CellOut2 o,
                                                            unsigned long long* lam_slot, const double* t_now,
                                                            double t_end) {
  if (!(*t_now < t_end)) return;
  const int ph = threadIdx.x / kPairCells;
  const Eos64 k = in_registers64(E.k, ph);
  const int64_t i = (int64_t)blockIdx.x * kPairCells + threadIdx.x % kPairCells;
  double q[15];
  if (i < o.n) load_phase(Q, o.n, i, ph, q);
  cell2_pass<kDef, kSoft>(q, Q, i < o.n, i, E, k, o, lam_slot);
}

// ---- faces ---------------------------------------------------------------------

// Faces whose path integrals are still to be done, and their s_l, s_r (by list
// position); the count lives in DevState.
struct FaceList {
  int* face;
  int* mark;  // LxF: per face block, whether it has such a face (null: not kept)
  double *sl, *sr;
};

// u1 and c_max of a phase at the midpoint of q_l = a and q_r = b (the forms are homogeneous, so
// q_l + q_r serves), a bad state recorded with the right cell.
template <int kDef>
static __device__ __noinline__ double2 mid2_again(const double* Q, int64_t n, int64_t L, int64_t R, int ph, const Eos2x& E,
                                                  DevState* S);
template <int kDef, bool kSoft>
__device__ __forceinline__ double2 mid2(const double* a, const double* b, const double* Q, int64_t n, int64_t L, int64_t R,
                                        int ph, const Eos2x& E, const Eos64& k, DevState* S) {
  double m[3], Rm[9];
#pragma unroll
  for (int v = 0; v < 3; ++v) m[v] = add64(k, a[2 + v], b[2 + v]);
#pragma unroll
  for (int v = 0; v < 9; ++v) Rm[v] = add64(k, a[6 + v], b[6 + v]);
  double u1, cm;
  int st;
  if (!cell_try64<kDef, false, false, kSoft>(E.e[ph], k, add64(k, a[0], b[0]), m, add64(k, a[5], b[5]), Rm, nullptr, u1,
                                             cm, st) && kSoft)
    return mid2_again<kDef>(Q, n, L, R, ph, E, S);
  if (st) record_err64(S, st, R);
  return make_double2(u1, cm);
}
template <int kDef>
static __device__ __noinline__ double2 mid2_again(const double* Q, int64_t n, int64_t L, int64_t R, int ph, const Eos2x& E,
                                                  DevState* S) {
  double a[15], b[15];
  load_phase(Q, n, L, ph, a);
  load_phase(Q, n, R, ph, b);
  return mid2<kDef, false>(a, b, Q, n, L, R, ph, E, in_registers64(E.k, ph), S);
}

// HLL faces: s_l, s_r and, where the volume fractions do not jump and no state on the
// way between the cells (through Q_hll) can be singular, D- and D+ (doubles of the
// formula of NumFluxes.jl:85-132 with its integrals zero). 186 slots a phase; the others are
// listed.
template <int kDef, bool kSoft>
__global__ void __launch_bounds__(kPair64, kSoft ? kSoftResident : 0) face2_f64_kernel(const double* __restrict__ Q, int64_t n,
                                                            const __grid_constant__ Eos2x E,
                                                            const double* __restrict__ F,
                                                            const double* __restrict__ smin,
                                                            const double* __restrict__ smax, double* __restrict__ DM,
                                                            double* __restrict__ DP, FaceList list,
                                                            const double* t_now, double t_end, DevState* S) {
  __shared__ double s_lo[2][kPairCells], s_hi[2][kPairCells];
  __shared__ int s_flag[2][kPairCells];  // bit 0: both cells equal; bit 1: alpha does not jump
  __shared__ int s_hard[2][kPairCells];
  if (!(*t_now < t_end)) return;
  const int ph = threadIdx.x / kPairCells, j = threadIdx.x % kPairCells;
  const Eos64 k = in_registers64(E.k, ph);
  const int64_t f = (int64_t)blockIdx.x * kPairCells + j;  // face between cells f-1 and f
  const int64_t nf = n + 1;
  const bool in = f <= n;
  const int64_t L = f > 0 ? f - 1 : 0, R = f < n ? f : n - 1;
  const double* ql = Q + 15 * ph * n + (in ? L : 0);
  const double* qr = Q + 15 * ph * n + (in ? R : 0);
  double a[15], b[15];
  bool same = true;
#pragma unroll
  for (int r = 0; r < 15; ++r) {
    a[r] = ql[r * n];
    b[r] = qr[r * n];
    same &= bits_of(a[r]) == bits_of(b[r]);
  }
  s_flag[ph][j] = (same ? 1 : 0) | (bits_of(a[0]) == bits_of(b[0]) ? 2 : 0);
  __syncthreads();
  const int flag = s_flag[0][j] & s_flag[1][j];
  const bool equal = flag & 1;  // (also the boundary face with its zero-gradient ghost)
  double* dm = DM + 15 * ph * nf + f;
  double* dp = DP + 15 * ph * nf + f;
  // equal cells: no jump, no fluctuation; the midpoint is the cell itself
  if (in && equal) {
#pragma unroll
    for (int r = 0; r < 15; ++r) dm[r * nf] = dp[r * nf] = 0.0;
  }
  const bool work = in && !equal;
  if (work) {
    const double2 s = mid2<kDef, kSoft>(a, b, Q, n, L, R, ph, E, k, S);
    s_lo[ph][j] = sub64(k, s.x, s.y);
    s_hi[ph][j] = add64(k, s.x, s.y);
  }
  __syncthreads();
  double sl = 0.0, sr = 0.0;
  bool hard = false;
  if (work) {
    const double l0 = s_lo[0][j], l1 = s_lo[1][j], h0 = s_hi[0][j], h1 = s_hi[1][j];
    const double mmin = l1 < l0 ? l1 : l0, mmax = h1 > h0 ? h1 : h0;
    if (mmin < sl) sl = mmin;
    if (smin[L] < sl) sl = smin[L];
    if (mmax > sr) sr = mmax;
    if (smax[R] > sr) sr = smax[R];
    hard = !(flag & 2);
    if (!hard) {
      const double idsr = rcp64(k, sub64(k, sr, sl));
      const double cm = mul64(k, -sl, idsr), cp = mul64(k, sr, idsr), cq = mul64(k, mul64(k, sl, sr), idsr);
      const double* fl = F + 15 * ph * n + L;
      const double* fr = F + 15 * ph * n + R;
      const float g = to_f32(cp), h = to_f32(idsr);
      float far = 0.0f, farh = 0.0f;  // squared distances of q_r and Q_hll from q_l in R
      bool finite = true;
      dm[0] = dp[0] = 0.0;
#pragma unroll
      for (int r = 1; r < 15; ++r) {
        const double jump = sub64(k, b[r], a[r]), qj = mul64(k, cq, jump);
        const double df = zero_flux_row(r) ? 0.0 : sub64(k, fr[r * n], fl[r * n]);
        if (r > 1) finite &= is_finite64(jump) && is_finite64(df);  // (alpha rho is unused by the forms)
        if (r >= 6) {  // Q_hll - q_l = (jump s_r - df) / (s_r - s_l)
          const float jf = to_f32(jump), hf = jf * g - to_f32(df) * h;
          far += jf * jf;
          farh += hf * hf;
        }
        dm[r * nf] = zero_flux_row(r) ? qj : fma(cm, df, qj);
        dp[r * nf] = zero_flux_row(r) ? -qj : fma(cp, df, -qj);
      }
      float Rf[9];
#pragma unroll
      for (int v = 0; v < 9; ++v) Rf[v] = to_f32(a[6 + v]);
      hard = !finite || !det_keeps_sign(Rf, fmaxf(far, farh));
    }
  }
  s_hard[ph][j] = hard;
  __syncthreads();
  if (ph == 0 && (s_hard[0][j] | s_hard[1][j])) {  // one atomic per warp
    const unsigned mask = __activemask();
    const int lead = __ffs(mask) - 1;
    int at = 0;
    if ((int)(threadIdx.x & 31) == lead) at = atomicAdd(&S->n_listed, __popc(mask));
    at = __shfl_sync(mask, at, lead) + __popc(mask & ((1u << (threadIdx.x & 31)) - 1u));
    list.face[at] = (int)f;
    list.sl[at] = sl;
    list.sr[at] = sr;
  }
}

// LxF faces: twice the conservative flux, (f_l + f_r) - lambda (q_r - q_l). Faces where the
// volume fractions jump are listed; blocks with such a face are marked and write the
// fluctuations' zeros of their other faces, which in unmarked blocks nobody reads (30 rows
// less to write and read a face, and 15 sums less a cell and phase: 131,072 cells, 4 steps
// 1.03 -> 0.95 ms). Grids up to kSoftBlocks write all zeros and keep no marks: the update
// would wait for its block's mark before the loads that follow from it (1000 cells with
// every face listed, 20 steps: 0.884 -> 0.898 ms).
__global__ void __launch_bounds__(kPair64) face2_lxf_f64_kernel(const double* __restrict__ Q, int64_t n, Eos64 kc,
                                                                const double* __restrict__ F,
                                                                const unsigned long long* lam_now, double cfl,
                                                                double dx, double* __restrict__ FF,
                                                                double* __restrict__ DM, FaceList list,
                                                                const double* t_now, double t_end, DevState* S) {
  __shared__ int s_hard[2][kPairCells];
  __shared__ double s_lam;
  if (!(*t_now < t_end)) return;
  const Eos64 k = in_registers64(kc);
  const int ph = threadIdx.x / kPairCells, j = threadIdx.x % kPairCells;
  const int64_t f = (int64_t)blockIdx.x * kPairCells + j;  // face between cells f-1 and f
  const int64_t nf = n + 1;
  const bool in = f <= n;
  const int64_t L = f > 0 ? f - 1 : 0, R = f < n ? f : n - 1;
  if (threadIdx.x < 32) {  // lambda = dx/dt (main.jl:223)
    const double lam = step_scalars64(k, cfl, dx, __longlong_as_double((long long)*lam_now), true).lam_lxf;
    if (threadIdx.x == 0) s_lam = lam;
  }
  __syncthreads();
  bool hard = false;
  if (in) {
    const double nlam = -s_lam;
    const double* ql = Q + 15 * ph * n;
    const double* fc = F + 15 * ph * n;
    float far = 0.0f, Rf[9];
    bool finite = true, jumps = false;
#pragma unroll
    for (int r = 0; r < 15; ++r) {
      const double a = ql[r * n + L], b = ql[r * n + R], jump = sub64(k, b, a);
      const int64_t o = (15 * ph + r) * nf + f;
      if (zero_flux_row(r)) {
        FF[o] = mul64(k, nlam, jump);
      } else {
        const double fs = add64(k, fc[r * n + L], fc[r * n + R]);
        finite &= is_finite64(fs);
        FF[o] = fma(nlam, jump, fs);
      }
      if (!list.mark) DM[o] = 0.0;
      finite &= is_finite64(jump);
      if (r == 0) jumps = bits_of(a) != bits_of(b);
      if (r >= 6) {
        const float jf = to_f32(jump);
        far += jf * jf;
        Rf[r - 6] = to_f32(a);
      }
    }
    hard = L != R && (jumps || !finite || !det_keeps_sign(Rf, far));
  }
  s_hard[ph][j] = hard;
  const int marked = __syncthreads_or(hard);
  if (list.mark && threadIdx.x == 0) list.mark[blockIdx.x] = marked;
  if (!marked) return;
  hard = s_hard[0][j] | s_hard[1][j];
  if (list.mark && in && !hard)
#pragma unroll
    for (int r = 0; r < 15; ++r) DM[(15 * ph + r) * nf + f] = 0.0;
  if (ph == 0 && hard) {
    const unsigned mask = __activemask();
    const int lead = __ffs(mask) - 1;
    int at = 0;
    if ((int)(threadIdx.x & 31) == lead) at = atomicAdd(&S->n_listed, __popc(mask));
    at = __shfl_sync(mask, at, lead) + __popc(mask & ((1u << (threadIdx.x & 31)) - 1u));
    list.face[at] = (int)f;
  }
}

// ---- path integrals of the listed faces -------------------------------------------

constexpr int kPathBlock = 128;
constexpr int kGroups = kPathBlock / 16;  // faces a block works on at a time, 16 lanes each

// Per group of 16 lanes: what the nodes add to each row, and the states of the face.
struct GroupMem {
  double part[12][15];  // by lane: B's rows times weight and d(alpha)
  double q[3][30];      // q_l, q_r, Q_hll
};

// 16 lanes per face, lane r < 12 on node r % 6 of phase r / 6: one integral is one pass
// of a phase's forms (about 190 slots) and an exchange with the lane of the other phase,
// against 12 passes on one thread; adds the integral from q[from] to q[to] to the
// partials.
template <int kDef>
__device__ __forceinline__ int path_group(const Eos2x& E, const Eos64& k, const Quad6D& qd, int lane16, GroupMem& g,
                                          int from, int to, double* acc) {
  const int ph = lane16 < 6 ? 0 : 1, node = lane16 < 12 ? lane16 - 6 * ph : 0;
  const double s = qd.x[node];
  const double* a = g.q[from] + 15 * ph;
  const double* b = g.q[to] + 15 * ph;
  auto at = [&](int r) { return fma(s, sub64(k, b[r], a[r]), a[r]); };
  double m[3], R[9];
#pragma unroll
  for (int v = 0; v < 3; ++v) m[v] = at(2 + v);
#pragma unroll
  for (int v = 0; v < 9; ++v) R[v] = at(6 + v);
  const double ia = rcp64(k, at(0));
  Half64 h, o;
  int st = half64<kDef>(E.e[ph], k, ia, m, at(5), R, h);
  const int other = (threadIdx.x & 16) + (ph ? node : node + 6);  // its node's lane of the other phase
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    o.u[v] = __shfl_sync(0xffffffffu, h.u[v], other);
    o.K[v] = __shfl_sync(0xffffffffu, h.K[v], other);
  }
  o.T = __shfl_sync(0xffffffffu, h.T, other);
  const Face64 I = interface64(k, h, o);
  add_b64(k, mul64(k, qd.w[node], sub64(k, b[0], a[0])), ia, R, h.u, I, acc);
  return lane16 < 12 ? st : 0;
}

// The sum over a face's six nodes of row k (30 rows).
__device__ __forceinline__ double node_sum(const Eos64& k, const GroupMem& g, int row) {
  const int ph = row < 15 ? 0 : 1, r = row - 15 * ph;
  double v = g.part[6 * ph][r];
#pragma unroll
  for (int i = 1; i < 6; ++i) v = add64(k, v, g.part[6 * ph + i][r]);
  return v;
}

// Lists of up to kGroupFaces faces per multiprocessor run in groups: a warp spends 620
// slots on the two faces of its groups, and on 32 faces with a thread each 6,600 (2,300
// where the states are smooth enough for two nodes, path_nodes): groups win up to 10.6 x
// 2 (3.7 x 2) faces on each of an SM's four schedulers, 85 (30) a multiprocessor. 1000
// cells, 50 HLL steps of a Riemann problem (whole run): 22.3 ms before this file's split
// of the faces, 2.95 ms now; 100,003 cells with all faces listed, 4 steps: 10.3 ms, 6.8 with
// six nodes a path, 3.3 with the nodes path_nodes asks for.
constexpr int kGroupFaces = 48;

// kLxf: one Gauss-Lobatto integral, D- = D+ = half of it (NumFluxes.jl:36-47), stored
// doubled as the LxF faces are. Otherwise Q_hll and the fluctuations of
// NumFluxes.jl:85-132.
template <int kDef, bool kLxf>
__global__ void __launch_bounds__(kPathBlock, 2)
    paths2_f64_kernel(const double* __restrict__ Q, int64_t n, Eos2x E, Quad6D qd, const double* __restrict__ F,
                      double* __restrict__ DM, double* __restrict__ DP, FaceList list, const double* t_now,
                      double t_end, int sms, DevState* S) {
  __shared__ GroupMem sg[kGroups];
  if (!(*t_now < t_end)) return;
  const int count = S->n_listed;
  const int64_t nf = n + 1;
  if (count <= kGroupFaces * sms) {
    const int blocks = min((int)gridDim.x, 2 * sms);  // a scheduler's second warp covers what is not FP64
    if ((int)blockIdx.x >= blocks) return;
    const int lane16 = threadIdx.x & 15;
    const Eos64 k = in_registers64(E.k, lane16 < 6 ? 0 : 1);
    GroupMem& g = sg[threadIdx.x >> 4];
    // A list of no more faces than schedulers gives each a warp: both its groups do the
    // first integral, then each one of the two through Q_hll.
    const bool wide = !kLxf && count <= 4 * sms;
    const int grp = (threadIdx.x >> 4) & 1, base = (threadIdx.x >> 4) & ~1;
    // both groups of a warp go round together (the exchanges are warp-wide): an idle one
    // repeats the list's last face and stores nothing
    const int group = blockIdx.x * kGroups + (threadIdx.x >> 4);
    const int first = wide ? group >> 1 : group, pair = wide ? first : first & ~1;
    const int stride = blocks * (wide ? kGroups / 2 : kGroups);
    for (int t = first, tp = pair; tp < count; t += stride, tp += stride) {
      const bool live = t < count;
      const int at = live ? t : count - 1;
      const int64_t f = list.face[at], L = f - 1, R = f;
      for (int r = lane16; r < 30; r += 16) {
        g.q[0][r] = Q[r * n + L];
        g.q[1][r] = Q[r * n + R];
      }
      __syncwarp();
      double acc[15];
#pragma unroll
      for (int r = 0; r < 15; ++r) acc[r] = 0.0;
      int st = path_group<kDef>(E, k, qd, lane16, g, 0, 1, acc);
      if (lane16 < 12)
#pragma unroll
        for (int r = 0; r < 15; ++r) g.part[lane16][r] = acc[r];
      __syncwarp();
      if (kLxf) {
        if (live)
          for (int r = lane16; r < 30; r += 16) DM[r * nf + f] = node_sum(k, g, r);
      } else {
        const double sl = list.sl[at], sr = list.sr[at], idsr = rcp64(k, sub64(k, sr, sl));
        for (int r = lane16; r < 30; r += 16) {
          const double df = zero_flux_row(r % 15) ? 0.0 : sub64(k, F[r * n + R], F[r * n + L]);
          const double qs = fma(g.q[1][r], sr, -mul64(k, g.q[0][r], sl));
          g.q[2][r] = mul64(k, sub64(k, qs, add64(k, node_sum(k, g, r), df)), idsr);
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < 15; ++r) acc[r] = 0.0;
#pragma unroll 1
        for (int h = wide ? grp : 0; h < (wide ? grp + 1 : 2); ++h)
          st |= path_group<kDef>(E, k, qd, lane16, g, h ? 2 : 0, h ? 1 : 2, acc);
        if (lane16 < 12)
#pragma unroll
          for (int r = 0; r < 15; ++r) g.part[lane16][r] = acc[r];
        __syncwarp();
        const double cm = mul64(k, -sl, idsr), cp = mul64(k, sr, idsr), cq = mul64(k, mul64(k, sl, sr), idsr);
        if (live)
          for (int r = wide ? threadIdx.x & 31 : lane16; r < 30; r += wide ? 32 : 16) {
            const double df = zero_flux_row(r % 15) ? 0.0 : sub64(k, F[r * n + R], F[r * n + L]);
            const double sum = wide ? add64(k, node_sum(k, sg[base], r), node_sum(k, sg[base + 1], r)) : node_sum(k, g, r);
            const double inner = add64(k, df, sum), qj = mul64(k, cq, sub64(k, g.q[1][r], g.q[0][r]));
            DM[r * nf + f] = fma(cm, inner, qj);
            DP[r * nf + f] = fma(cp, inner, -qj);
          }
      }
      if (st && live) record_err64(S, st, R);
      __syncwarp();
    }
    return;
  }
  Eos2x X;
  X.e[0] = E.e[0];
  X.e[1] = E.e[1];
  X.k[0] = in_registers64(E.k[0]);
  X.k[1] = in_registers64(E.k[1]);
  const Eos64& k = X.k[0];
  const int t = blockIdx.x * kPathBlock + threadIdx.x;
  if (t < count) {
    const int64_t f = list.face[t], L = f - 1, R = f;
    double a[30], b[30], acc[30];
    for (int r = 0; r < 30; ++r) {
      a[r] = Q[r * n + L];
      b[r] = Q[r * n + R];
      acc[r] = 0.0;
    }
    int st = path_thread<kDef>(X, qd, a, b, acc);
    if (kLxf) {
      for (int r = 0; r < 30; ++r) DM[r * nf + f] = acc[r];
    } else {
      const double sl = list.sl[t], sr = list.sr[t], idsr = rcp64(k, sub64(k, sr, sl));
      double h[30];
      for (int r = 0; r < 30; ++r) {
        const double df = zero_flux_row(r % 15) ? 0.0 : sub64(k, F[r * n + R], F[r * n + L]);
        const double qs = fma(b[r], sr, -mul64(k, a[r], sl));
        h[r] = mul64(k, sub64(k, qs, add64(k, acc[r], df)), idsr);
        acc[r] = df;
      }
#pragma unroll 1
      for (int half = 0; half < 2; ++half) st |= path_thread<kDef>(X, qd, half ? h : a, half ? b : h, acc);
      const double cm = mul64(k, -sl, idsr), cp = mul64(k, sr, idsr), cq = mul64(k, mul64(k, sl, sr), idsr);
      for (int r = 0; r < 30; ++r) {
        const double qj = mul64(k, cq, sub64(k, b[r], a[r]));
        DM[r * nf + f] = fma(cm, acc[r], qj);
        DP[r * nf + f] = fma(cp, acc[r], -qj);
      }
    }
    if (st) record_err64(S, st, R);
  }
}

// The update of a step: FF twice the LxF face flux (with D- = D+ doubled as well), or null
// for HLL. rd: the max wave speed; an active step zeroes the clr slots.
struct Step2Args {
  const double* Q;
  double* Qn;
  const double *FF, *DM, *DP;
  const int* mark;  // LxF: face blocks with fluctuations (null: all)
  const unsigned long long* rd;
  unsigned long long* wr;
  unsigned long long* clr[2];
  const double* t_in;
  double* t_out;
  double t_end, cfl, dx;
  int bc;
  CellOut2 o;
};

// A thread per cell and phase; with kCell the new state's cell pass follows in the same
// kernel (a launch and a reload of the state less per step, which a small problem feels).
template <int kDef, bool kCell, bool kSoft, bool kLxf>
__global__ void __launch_bounds__(kPair64, kSoft ? kSoftResident : 0) step2_f64_kernel(const __grid_constant__ Step2Args a,
                                                                                    const __grid_constant__ Eos2x E) {
  __shared__ double s_r;
  __shared__ int s_more;
  const int ph = threadIdx.x / kPairCells;
  const Eos64 k = in_registers64(E.k, ph);
  const int64_t n = a.o.n, nf = n + 1;
  const double tn = *a.t_in;
  const bool active = tn < a.t_end;
  const int64_t i = (int64_t)blockIdx.x * kPairCells + threadIdx.x % kPairCells;
  int markl = 0, markr = 0;  // the faces on both sides have fluctuations
  if (kLxf && i < n) {
    markl = a.mark ? a.mark[i / kPairCells] : 1;
    markr = a.mark ? a.mark[(i + 1) / kPairCells] : 1;
  }
  if (threadIdx.x < 32) {
    const StepScalars sc = step_scalars64(k, a.cfl, a.dx, __longlong_as_double((long long)*a.rd), false);
    if (threadIdx.x == 0) {
      s_r = kLxf ? 0.5 * sc.dtdx : sc.dtdx;
      s_more = kCell && tn + sc.dt < a.t_end;
      if (blockIdx.x == 0) {
        *a.t_out = active ? tn + sc.dt : tn;
        a.o.S->n_listed = 0;
        if (active) {
          for (int c = 0; c < 2; ++c)
            if (a.clr[c]) *a.clr[c] = 0ull;
          a.o.S->steps += 1;
        }
      }
    }
  }
  if (!active) return;
  __syncthreads();
  double q[15];
  if (i < n) {
    const bool frozen = a.bc == HYP_BC_FROZEN && (i == 0 || i == n - 1);
    const double r = s_r;
    // every load before the first store: the compiler has to keep their order
    double d[15];
    if (kLxf) {
#pragma unroll
      for (int v = 0; v < 15; ++v) {
        const int64_t row = 15 * ph + v;
        q[v] = a.Q[row * n + i];
        d[v] = sub64(k, a.FF[row * nf + i + 1], a.FF[row * nf + i]);
      }
      if (markl | markr) {
#pragma unroll
        for (int v = 0; v < 15; ++v) {
          const int64_t row = 15 * ph + v;
          d[v] = add64(k, add64(k, markr ? a.DM[row * nf + i + 1] : 0.0, markl ? a.DM[row * nf + i] : 0.0), d[v]);
        }
      }
    } else {
      // F_r = F_l = zeros(30) for hll (NumFluxes.jl:82), NF_r = D- of face i+1/2, NF_l = D+ of face i-1/2
#pragma unroll
      for (int v = 0; v < 15; ++v) {
        const int64_t row = 15 * ph + v;
        q[v] = a.Q[row * n + i];
        d[v] = add64(k, a.DM[row * nf + i + 1], a.DP[row * nf + i]);
      }
    }
#pragma unroll
    for (int v = 0; v < 15; ++v) {
      q[v] = frozen ? q[v] : fma(-r, d[v], q[v]);
      a.Qn[(15 * ph + v) * n + i] = q[v];
    }
  }
  if (!kCell || !s_more) return;
  cell2_pass<kDef, kSoft>(q, a.Qn, i < n, i, E, k, a.o, a.wr);
}

static inline unsigned grid_n(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }

static Eos2x eos2x(const hyp_ctx* c) { return make_eos2x(c->eos2.e); }
static bool default_exp2(const hyp_ctx* c) { return c->eos2.e[0].default_exp && c->eos2.e[1].default_exp; }

static CellOut2 cell_out(hyp_ctx* c) { return CellOut2{c->F, c->smin, c->smax, c->n, c->st}; }

// The LxF faces' marks, of grids that keep them (both kernels of a step have to agree).
static int* face_marks(const hyp_ctx* c) {
  return grid_n(c->n + 1, kPairCells) > kSoftBlocks ? c->face_list + c->n + 1 : nullptr;
}
int64_t face_list_ints(int64_t n) { return n + 1 + grid_n(n + 1, kPairCells); }

cudaError_t launch_cell2_f64(hyp_ctx* c, int p, unsigned long long* lam_slot, const double* t_now, double t_end) {
  const unsigned grid = grid_n(c->n, kPairCells);
  const bool def = default_exp2(c);
  auto kern = grid > kSoftBlocks ? (def ? cell2_f64_kernel<1, true> : cell2_f64_kernel<0, true>)
                                 : (def ? cell2_f64_kernel<1, false> : cell2_f64_kernel<0, false>);
  kern<<<grid, kPair64, 0, c->stream>>>(c->Q[p], eos2x(c), cell_out(c), lam_slot, t_now, t_end);
  return cudaGetLastError();
}
cudaError_t launch_face2_f64(hyp_ctx* c, int p, const unsigned long long* rd, double t_end) {
  const bool lxf = c->cfg.flux == HYP_FLUX_LXF, def = default_exp2(c);
  const FaceList list{c->face_list, face_marks(c), c->face_s, c->face_s ? c->face_s + c->n + 1 : nullptr};
  const unsigned grid = grid_n(c->n + 1, kPairCells);
  const Eos2x E = eos2x(c);
  if (lxf) {
    const double dx = c->cfg.x_length / (double)c->n;
    face2_lxf_f64_kernel<<<grid, kPair64, 0, c->stream>>>(c->Q[p], c->n, E.k[0], c->F, rd, c->cfg.cfl, dx,
                                                          c->FF, c->DM, list, &c->st->t[p], t_end, c->st);
  } else {
    auto kern = grid > kSoftBlocks ? (def ? face2_f64_kernel<1, true> : face2_f64_kernel<0, true>)
                                   : (def ? face2_f64_kernel<1, false> : face2_f64_kernel<0, false>);
    kern<<<grid, kPair64, 0, c->stream>>>(c->Q[p], c->n, E, c->F, c->smin, c->smax, c->DM, c->DP, list, &c->st->t[p],
                                          t_end, c->st);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  auto paths = lxf ? (def ? paths2_f64_kernel<1, true> : paths2_f64_kernel<0, true>)
                   : (def ? paths2_f64_kernel<1, false> : paths2_f64_kernel<0, false>);
  // a block per 128 faces, were all of them listed; those past the list's end return at once
  const unsigned pgrid = std::max(grid_n(c->n + 1, kPathBlock), (unsigned)(2 * c->sms));
  paths<<<pgrid, kPathBlock, 0, c->stream>>>(c->Q[p], c->n, E, lxf ? c->lobatto : c->quad, c->F, c->DM, c->DP, list,
                                             &c->st->t[p], t_end, c->sms, c->st);
  return cudaGetLastError();
}
template <bool kLxf>
static void launch_step2_of(const Step2Args& a, const Eos2x& E, bool cell, bool def, unsigned grid, cudaStream_t s) {
  auto kern = !cell ? step2_f64_kernel<1, false, false, kLxf>
              : grid > kSoftBlocks
                  ? (def ? step2_f64_kernel<1, true, true, kLxf> : step2_f64_kernel<0, true, true, kLxf>)
                  : (def ? step2_f64_kernel<1, true, false, kLxf> : step2_f64_kernel<0, true, false, kLxf>);
  kern<<<grid, kPair64, 0, s>>>(a, E);
}
// The update of step k, and with `cell` the cell pass of the new state.
static cudaError_t launch_step2(hyp_ctx* c, long long k, double t_end, bool cell) {
  const int p = (int)(k & 1);
  const bool lxf = c->cfg.flux == HYP_FLUX_LXF;
  unsigned long long* s = c->st->lam_slots;
  Step2Args a;
  a.Q = c->Q[p];
  a.Qn = c->Q[1 - p];
  a.FF = lxf ? c->FF : nullptr;
  a.mark = face_marks(c);
  a.DM = c->DM;
  a.DP = lxf ? c->DM : c->DP;
  a.rd = s + k % 3;
  a.wr = s + (k + 1) % 3;
  a.clr[0] = s + (k + 2) % 3;
  a.clr[1] = cell ? nullptr : a.wr;
  a.t_in = &c->st->t[p];
  a.t_out = &c->st->t[1 - p];
  a.t_end = t_end;
  a.cfl = c->cfg.cfl;
  a.dx = c->cfg.x_length / (double)c->n;
  a.bc = c->cfg.bc;
  a.o = cell_out(c);
  const unsigned grid = grid_n(c->n, kPairCells);
  const bool def = default_exp2(c);
  const Eos2x E = eos2x(c);
  lxf ? launch_step2_of<true>(a, E, cell, def, grid, c->stream) : launch_step2_of<false>(a, E, cell, def, grid, c->stream);
  return cudaGetLastError();
}
cudaError_t launch_update2_f64(hyp_ctx* c, long long k, double t_end) { return launch_step2(c, k, t_end, false); }

// Step k of a run (first / last of it), the slots as in launch_run_step1_f64. Relaxation
// changes the new state after the update, so its cell pass waits for the next step.
cudaError_t launch_run_step2_f64(hyp_ctx* c, long long k, double t_end, bool first, bool last) {
  const int p = (int)(k & 1);
  unsigned long long* rd = c->st->lam_slots + k % 3;
  cudaError_t e = cudaSuccess;
  if (first || c->relax) e = launch_cell2_f64(c, p, rd, &c->st->t[p], t_end);
  if (e == cudaSuccess) e = launch_face2_f64(c, p, rd, t_end);
  if (e == cudaSuccess) e = launch_step2(c, k, t_end, !last && !c->relax);
  return e;
}

// Gauss-Legendre 6 on [0,1]: Newton on P6 from Chebyshev-like guesses in long
// double, mapped (x + 1)/2, w/2, ascending (FastGaussQuadrature.gausslegendre(6)).
Quad6D gauss_legendre6() {
  long double xs[6], ws[6];
  for (int i = 0; i < 6; ++i) {
    long double x = cosl(3.14159265358979323846264338327950288L * (i + 0.75L) / 6.5L);
    long double dp = 1.0L;
    for (int it = 0; it < 100; ++it) {
      long double p0 = 1.0L, p1 = x;
      for (int k = 2; k <= 6; ++k) {
        long double p2 = ((2 * k - 1) * x * p1 - (k - 1) * p0) / k;
        p0 = p1;
        p1 = p2;
      }
      dp = 6.0L * (x * p1 - p0) / (x * x - 1.0L);
      long double dx = p1 / dp;
      x -= dx;
      if (fabsl(dx) < 1e-30L) break;
    }
    {
      long double p0 = 1.0L, p1 = x;
      for (int k = 2; k <= 6; ++k) {
        long double p2 = ((2 * k - 1) * x * p1 - (k - 1) * p0) / k;
        p0 = p1;
        p1 = p2;
      }
      dp = 6.0L * (x * p1 - p0) / (x * x - 1.0L);
    }
    xs[i] = x;
    ws[i] = 2.0L / ((1.0L - x * x) * dp * dp);
  }
  Quad6D q;
  for (int i = 0; i < 6; ++i) {
    const double nx = (double)xs[5 - i], nw = (double)ws[5 - i];
    q.x[i] = (nx + 1.0) / 2.0;
    q.w[i] = nw / 2.0;
  }
  return q;
}

// Gauss-Lobatto 6 on [0,1] (FastGaussQuadrature.gausslobatto(6), NumFluxes.jl:36):
// nodes -1, -a, -b, b, a, 1 with a, b = sqrt(1/3 +- 2 sqrt(7)/21), weights 1/15 at the
// ends and (14 -+ sqrt 7)/30 inside, mapped (x + 1)/2, w/2; evaluated in long double.
Quad6D gauss_lobatto6() {
  const long double s7 = sqrtl(7.0L);
  const long double a = sqrtl(1.0L / 3.0L + 2.0L * s7 / 21.0L), b = sqrtl(1.0L / 3.0L - 2.0L * s7 / 21.0L);
  const long double xs[6] = {-1.0L, -a, -b, b, a, 1.0L};
  const long double ws[6] = {1.0L / 15.0L, (14.0L - s7) / 30.0L, (14.0L + s7) / 30.0L,
                             (14.0L + s7) / 30.0L, (14.0L - s7) / 30.0L, 1.0L / 15.0L};
  Quad6D q;
  for (int i = 0; i < 6; ++i) {
    q.x[i] = ((double)xs[i] + 1.0) / 2.0;
    q.w[i] = (double)ws[i] / 2.0;
  }
  return q;
}

}  // namespace hyp
