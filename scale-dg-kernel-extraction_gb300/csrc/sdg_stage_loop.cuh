// Whole sdg_solver_step calls of a small box in one launch (FP64 form).
//
// A stage of a small box is the latency of one block: a launch, instruction
// fetches that miss, two rounds of loads, three lines one after the other.  Here
// every block stays resident for all stages of the call, with a barrier over
// the grid between them (a cooperative launch), and the three directions of an
// element run side by side, one line a thread.  A stage is then: q and u of the
// thread's line, the two face fluxes (their velocity factors stay in
// registers), the line sums in fixed point as in stage_fix_kernel, and after a
// block barrier the nodes' sums and RK update.  Same bits as stage_fix_kernel:
// the same values reach the same integer sums.
//
// Measured on GB300, us a stage (100 steps), against one stage_fix_kernel launch
// a stage: see fix_loop_most.
//
// The wait at the grid barrier is bounded: a block that gives up sets a flag and
// leaves.  Launches that find the flag set leave at once (the arrivals of the
// one that gave up would let their stages run unordered); the solver's next
// call that waits for its stream reports it and clears both words.
#pragma once

#include "sdg_stage_fix.cuh"

namespace sdg {

template <int P>
struct LoopShape {
  static constexpr int N = P + 1, N2 = N * N;
  static constexpr int EPB = N2 < 32 ? 32 / N2 : 1;           // elements a block
  static constexpr int G = (EPB * N2 + 31) / 32 * 32;         // threads a direction
  static constexpr int THREADS = 3 * G;
  static constexpr int BLOCKS = THREADS > 512 ? 1 : 1024 / THREADS;   // resident, an SM
  static constexpr int IT = (EPB * N2 * N + THREADS - 1) / THREADS;  // nodes a thread
  static constexpr size_t SMEM =
      sizeof(int64_t) * 3 * EPB * FixShape<P>::EW + sizeof(short) * 3 * EPB * N2;
};

template <int P, bool EO>
struct FixLoopArgs {
  FixStageArgs<P, EO> f;  // f.s: velocity, box, tables
  double* q[3];           // rotating state buffers, the current one first
  double dt;
  int nstep;
  unsigned* bar;          // [0] arrivals (zero between launches), [1] a wait ran out
  int polls;              // reads of the arrivals before a wait gives up
};

// Waits until every block has arrived `round` times; false when the wait ran
// out (here or in another block).
__device__ __forceinline__ bool fix_grid_barrier(unsigned* bar, unsigned round, int polls) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&bar[0], 1u);
    const unsigned want = round * gridDim.x;
    int good = 0;
    for (int t = 0; t < polls; t++) {
      unsigned v;
      asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if ((int)(v - want) >= 0) {  // both may pass 2^32
        good = 1;
        break;
      }
    }
    if (!good) atomicExch(&bar[1], 1u);
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

// Line r of direction AX of one element for a stage: q the state, g the
// element's first node, fc the velocity factors of the line's - and + face, nbr
// the nodes beyond them; results to s (the element's padded array), returns the
// line's exponent.
template <int P, bool EO, int AX>
__device__ __forceinline__ int fix_loop_line(const FixStageArgs<P, EO>& a, const double* q,
                                             long long g, int r, const double2 fc[2],
                                             const long long nbr[2], int64_t* s) {
  constexpr int N = P + 1, N2 = N * N, NS = FixShape<P>::NS;
  constexpr int S = AX == 0 ? 1 : AX == 1 ? N : N2;
  constexpr int SO = AX == 0 ? 1 : AX == 1 ? NS : NS * N;
  const int i = r % N, j = r / N;
  const long long at = g + (AX == 0 ? N * r : AX == 1 ? i + j * N2 : r);
  int64_t* out = s + (AX == 0 ? NS * r : AX == 1 ? i + NS * N * j : i + NS * j);
  const double* __restrict__ u =
      static_cast<const double*>(AX == 0 ? a.s.u : AX == 1 ? a.s.v : a.s.w);
  // the state was written by other blocks during this launch: not through L1
  const double qPm = __ldcg(q + nbr[0]), qPp = __ldcg(q + nbr[1]);
  double F[N], qm = 0.0, qp = 0.0;
  FixScan<P, EO> scan;
#pragma unroll
  for (int l = 0; l < N; l++) {
    const double v = __ldcg(q + at + l * S);
    if (l == 0) qm = v;
    if (l == N - 1) qp = v;
    F[l] = fix_product(v, u[at + l * S]);
    scan.add(l, fix_value_exp(F[l]));
  }
  auto flux = [](double qP, double qM, double2 c) {
    return EO ? fma(qP, c.x, -(qM * c.y)) : fma(qP, c.x, (qP - qM) * c.y);
  };
  const double gm = flux(qPm, qm, fc[0]), gp = flux(qPp, qp, fc[1]);
  const int32_t E = fix_line_scale<N>(
      F, scan.scale(max(fix_face_exp(gm), fix_face_exp(gp)), !EO && a.thin), gm, gp);
  if (a.ok && fix_in_range(E)) {
    fix_line<P, EO>(a.tab + AX * a.TAB, a.lift(AX, r), F, E, fix_align_face(gm, E),
                    fix_align_face(gp, E), [&](int m, int64_t v) { out[m * SO] = v; });
    return fix_line_exp(E);
  }
  double in[N], d[N];  // in: F itself stays in registers
#pragma unroll
  for (int l = 0; l < N; l++) in[l] = F[l];
  fix_line_fp64<P, EO>(&a.s, AX, r, in, 1, gm, gp, d);
  for (int m = 0; m < N; m++) out[m * SO] = __double_as_longlong(d[m]);
  return kFixDouble;
}

template <int P, bool EO>
__global__ void __launch_bounds__(LoopShape<P>::THREADS,
                                  LoopShape<P>::BLOCKS)
    stage_fix_loop_kernel(const __grid_constant__ FixLoopArgs<P, EO> a) {
  using Ls = LoopShape<P>;
  using Args = FixStageArgs<P, EO>;
  constexpr int N = Ls::N, N2 = Ls::N2, NP = N * N2, NS = FixShape<P>::NS, EW = FixShape<P>::EW,
                EPB = Ls::EPB, G = Ls::G, IT = Ls::IT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  int64_t* s0 = reinterpret_cast<int64_t*>(smem_raw);           // [3][EPB][EW]
  short* sE = reinterpret_cast<short*>(s0 + 3 * EPB * EW);      // [3][EPB][N2]
  // one thread's answer for the block: another block may give up meanwhile
  if (__syncthreads_or(threadIdx.x == 0 && __ldcg(a.bar + 1) != 0)) return;
  const long long eb = (long long)blockIdx.x * EPB;
  const int nloc = (int)min((long long)EPB, a.f.s.elem_count - eb);
  // one direction a group of whole warps
  const int d = threadIdx.x / G, t = threadIdx.x - d * G;
  const int le = t / N2, r = t - le * N2;
  const bool on = le < nloc;
  const long long g = (eb + le) * NP;
  double2 fc[2];
  long long nbr[2] = {0, 0};
  if (on) {
    unsigned nb[6];
    fix_neighbors(a.f.s.box, (unsigned)(eb + le), nb);
    const int i = r % N, j = r / N;
    const int first = d == 0 ? N * r : d == 1 ? i + j * N2 : r;
    const int last = first + (N - 1) * (d == 0 ? 1 : d == 1 ? N : N2);
    nbr[0] = (long long)(d == 0 ? nb[3] : d == 1 ? nb[0] : nb[4]) * NP + last;
    nbr[1] = (long long)(d == 0 ? nb[1] : d == 1 ? nb[2] : nb[5]) * NP + first;
    const double* vel = static_cast<const double*>(d == 0 ? a.f.s.u : d == 1 ? a.f.s.v : a.f.s.w);
#pragma unroll
    for (int side = 0; side < 2; side++) {
      const double uM = vel[g + (side ? last : first)], uP = vel[nbr[side]];
      const double a2 = abs_ct(uP + uM), tw = side ? 2.0 : -2.0;
      fc[side] = make_double2(EO ? fma(tw, uP, -a2) : tw * (uP - uM), fma(tw, uM, -a2));
    }
  }
  unsigned round = 0;
  int c0 = 0;
  for (int step = 0; step < a.nstep; step++) {
    const double* qs = c0 == 0 ? a.q[0] : c0 == 1 ? a.q[1] : a.q[2];
    double* q1 = c0 == 0 ? a.q[1] : c0 == 1 ? a.q[2] : a.q[0];
    double* q2 = c0 == 0 ? a.q[2] : c0 == 1 ? a.q[0] : a.q[1];
    for (int stage = 0; stage < 3; stage++) {
      const double* in = stage == 0 ? qs : stage == 1 ? q1 : q2;
      double* out = stage == 1 ? q2 : q1;
      // the states of the thread's nodes, in flight during the lines
      double qv[IT], q0[IT];
#pragma unroll
      for (int it = 0; it < IT; it++) {
        const int w = threadIdx.x + it * Ls::THREADS;
        qv[it] = q0[it] = 0.0;
        if (w < nloc * NP) {
          qv[it] = __ldcg(in + eb * NP + w);
          if (stage != 0) q0[it] = __ldcg(qs + eb * NP + w);
        }
      }
      if (on) {
        int64_t* s = s0 + (d * EPB + le) * EW;
        const int e = d == 0   ? fix_loop_line<P, EO, 0>(a.f, in, g, r, fc, nbr, s)
                      : d == 1 ? fix_loop_line<P, EO, 1>(a.f, in, g, r, fc, nbr, s)
                               : fix_loop_line<P, EO, 2>(a.f, in, g, r, fc, nbr, s);
        sE[(d * EPB + le) * N2 + r] = (short)e;
      }
      __syncthreads();
      const double ra = stage == 1 ? 0.75 : 1.0 / 3.0, rb = stage == 1 ? 0.25 : 2.0 / 3.0;
      const double c = EO ? (stage == 0 ? 1.0 : rb) * a.dt : a.dt;
#pragma unroll
      for (int it = 0; it < IT; it++) {
        const int w = threadIdx.x + it * Ls::THREADS;
        if (w >= nloc * NP) break;
        const int l = w / NP, n = w - l * NP;
        const int k = n / N2, m = n - k * N2, j = m / N, i = m - j * N;
        const int at = l * EW + i + NS * (j + N * k);
        const short* x = sE + l * N2;
        const double v = fix_node(
            s0[at], x[j + N * k] + a.f.row[Args::row_of(i)], s0[EPB * EW + at],
            x[EPB * N2 + i + N * k] + a.f.row[Args::ROWS + Args::row_of(j)], s0[2 * EPB * EW + at],
            x[2 * EPB * N2 + i + N * j] + a.f.row[2 * Args::ROWS + Args::row_of(k)]);
        const long long gn = eb * NP + w;
        if (stage == 0)
          out[gn] = fma(c, v, qv[it]);
        else
          out[gn] = EO ? fma(ra, q0[it], fma(rb, qv[it], c * v))
                       : fma(ra, q0[it], rb * fma(c, v, qv[it]));
      }
      if (step + 1 < a.nstep || stage < 2)
        if (!fix_grid_barrier(a.bar, ++round, a.polls)) return;
    }
    c0 = c0 == 2 ? 0 : c0 + 1;
  }
  // the last block to leave clears the arrivals for the next launch
  if (threadIdx.x == 0 && atomicAdd(&a.bar[0], 1u) == (round + 1) * gridDim.x - 1)
    atomicExch(&a.bar[0], 0u);
}

template <int P, bool EO>
int launch_stage_fix_loop(const StageArgs& s, double* const* q, double dt, int nstep, unsigned* bar,
                          int polls, cudaStream_t st) {
  using Ls = LoopShape<P>;
  FixLoopArgs<P, EO> a;
  fix_fill<P, EO>(a.f, s);
  for (int i = 0; i < 3; i++) a.q[i] = q[i];
  a.dt = dt;
  a.nstep = nstep;
  a.bar = bar;
  a.polls = polls;
  const void* kernel = (const void*)stage_fix_loop_kernel<P, EO>;
  SDG_TRY(set_kernel_smem(kernel, (int)Ls::SMEM, carve_for(Ls::SMEM, Ls::BLOCKS)));
  const unsigned nblk = (unsigned)((s.elem_count + Ls::EPB - 1) / Ls::EPB);
  void* args[1] = {&a};
  const cudaError_t e =
      cudaLaunchCooperativeKernel(kernel, dim3(nblk), dim3(Ls::THREADS), args, Ls::SMEM, st);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();
    return kLoopTooLarge;
  }
  SDG_CUDA_TRY(e);
  return SDG_OK;
}

// The most elements one launch takes on the current device: what a resident grid
// holds (152 SMs: 3040 elements at p = 3, 760 at p = 7, 152 at p = 15), but for the
// even-odd type at p = 1 past 6600 elements (6.4 us a stage in one launch, 6.2 in a
// launch a stage at 21^3) and from p = 14 (23.1 / 21.2 us at p = 15: 768 threads a
// block leave it 80 registers).  One launch / a launch a stage elsewhere, us a
// stage, OPT1 and EVENODD: p = 3 8^3 3.6 / 8.2 and 3.1 / 6.4, 13^3 8.8 / 10.3 and
// 7.7 / 8.2; p = 7 4^3 5.8 / 14.3 and 4.7 / 9.6, 9^3 13.1 / 19.8 and 10.5 / 13.7;
// p = 11 5^3 14.4 / 23.9 and 11.6 / 15.2; p = 15 5^3 29.6 / 34.7 (OPT1).
template <int P, bool EO>
int fix_loop_most(long long* elems) {
  using Ls = LoopShape<P>;
  const void* kernel = (const void*)stage_fix_loop_kernel<P, EO>;
  SDG_TRY(set_kernel_smem(kernel, (int)Ls::SMEM, carve_for(Ls::SMEM, Ls::BLOCKS)));
  int dev = 0, sms = 0, per = 0;
  SDG_CUDA_TRY(cudaGetDevice(&dev));
  SDG_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  SDG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, Ls::THREADS, Ls::SMEM));
  *elems = (long long)sms * per * Ls::EPB;
  if (EO && P == 1) *elems = std::min(*elems, 6600LL);
  if (EO && P >= 14) *elems = 0;
  return SDG_OK;
}

}  // namespace sdg
