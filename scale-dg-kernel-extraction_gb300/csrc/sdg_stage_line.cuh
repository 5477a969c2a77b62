// Fused RK-stage kernel of the FP32-compute form with the even-odd pair sums:
// FP64 state, FP32 velocity, products and sums, FP64 RK update.
//
// Thread r of an element's N^2 owns line r of each direction and node r of
// each face (the layout of stage_fix_kernel): its face fluxes and the z line's
// pair values never leave its registers, shared memory holds the x and y
// fluxes and then their line results.  The coefficients, scaled for the stage,
// are kernel parameters, which a multiply-add takes from the constant bank; in
// the batch, whose instances each have their own, they are in shared memory.
// Products are rounded before the pair sums, line results add up as x + y + z
// in FP32 and the increment is widened: the same bits in both kernels.
//
// Bound: 28 bytes a node in the first stage and 36 in the others, read and
// written once, at 0.7-0.85 of the copy bandwidth; 32 warps an SM wait on the
// loads at the two ends of a block.  On GB300, 16.8M DOF, against the kernels
// this replaced (GDOF-updates/s): p = 2 140 from 110, p = 3 147 from 106, p = 5
// 145 from 82, p = 7 171 from 108, p = 9 148 from 87, p = 11 146 from 93, p = 15
// 148 from 87 (p = 1 level at 130).  Half of it comes from L1: with the largest
// shared-memory carveout 84 at p = 5.  The state is read by __ldg: plain reads of
// q and q0 wait for the store of the node before (p = 7 151, and 89 against 131 in
// the batch).  64 registers (1024 threads an SM): 1280 threads 0.85-1.0x, 768
// 0.9-1.03x.  Velocity factors of the faces stored by the call's first stage, as
// the FP64 form does: 0.88-1.03x.
#pragma once

#include "sdg_stage_fix.cuh"

namespace sdg {

template <int P>
__host__ __device__ constexpr int line_min_blocks() {
  return 1024 / FixShape<P>::THREADS;
}

template <int P>
struct LineStageArgs {
  StageArgs s;
  float tab[3 * EoShape<P>::TE];  // a direction's EoShape table, scaled for the stage
};

template <int P>
__host__ __device__ constexpr size_t line_smem(int epb) {
  return sizeof(float) * 2 * epb * FixShape<P>::EW;
}

// A direction's coefficients as EoShape lays them out (kernel parameters).
template <int P>
struct LineTable {
  using Sh = EoShape<P>;
  const float* T;
  // c: E(i, .), D(i, mid) (odd N), B(i), O(i, .), A(i)
  __device__ __forceinline__ void row(int i, float* c) const {
    constexpr int H = Sh::H;
#pragma unroll
    for (int l = 0; l < H; l++) {
      c[l] = T[Sh::OFF_E + i * H + l];
      c[H + Sh::ODD + 1 + l] = T[Sh::OFF_O + i * H + l];
    }
    if constexpr (Sh::ODD != 0) c[H] = T[Sh::OFF_DM + i];
    c[H + Sh::ODD] = T[Sh::OFF_B + i];
    c[2 * H + Sh::ODD + 1] = T[Sh::OFF_A + i];
  }
  // c: O(H, .), A(H): the middle row of an odd N
  __device__ __forceinline__ void mid(float* c) const {
#pragma unroll
    for (int l = 0; l < Sh::H; l++) c[l] = T[Sh::OFF_O + Sh::H * Sh::H + l];
    c[Sh::H] = T[Sh::OFF_A + Sh::H];
  }
};

// The same row by row in shared memory, each row padded to whole 16-byte loads
// (a quarter of the loads).
template <int P>
struct LineRows {
  using Sh = EoShape<P>;
  static constexpr int ROW = (2 * Sh::H + 2 + Sh::ODD + 3) / 4 * 4;
  static constexpr int MID = Sh::ODD ? (Sh::H + 1 + 3) / 4 * 4 : 0;
  static constexpr int DIR = Sh::H * ROW + MID;  // words of a direction
  const float* T;                                // 16-byte aligned
  // where EoShape's entry t of a direction goes
  static __device__ __forceinline__ int at(int t) {
    constexpr int H = Sh::H;
    if (t < Sh::OFF_O) return t / H * ROW + t % H;
    if (t < Sh::OFF_DM) {
      const int i = (t - Sh::OFF_O) / H, l = (t - Sh::OFF_O) % H;
      return i < H ? i * ROW + H + Sh::ODD + 1 + l : H * ROW + l;
    }
    if (t < Sh::OFF_A) return (t - Sh::OFF_DM) * ROW + H;
    if (t < Sh::OFF_B) {
      const int i = t - Sh::OFF_A;
      return i < H ? i * ROW + 2 * H + Sh::ODD + 1 : H * ROW + H;
    }
    return (t - Sh::OFF_B) * ROW + H + Sh::ODD;
  }
  __device__ __forceinline__ void row(int i, float* c) const { load<ROW>(T + i * ROW, c); }
  __device__ __forceinline__ void mid(float* c) const { load<MID>(T + Sh::H * ROW, c); }
  template <int W>
  static __device__ __forceinline__ void load(const float* p, float* c) {
#pragma unroll
    for (int k = 0; k < W; k += 4) {
      const float4 x = *reinterpret_cast<const float4*>(p + k);
      c[k] = x.x;
      c[k + 1] = x.y;
      c[k + 2] = x.z;
      c[k + 3] = x.w;
    }
  }
};

// One line from its pair values s, d and face fluxes: the N results to
// emit(m, value).
template <int P, typename Table, typename Emit>
__device__ __forceinline__ void line_pairs(const float* s, const float* d, float fm,
                                           const Table& T, float gm, float gp, Emit&& emit) {
  using Sh = EoShape<P>;
  constexpr int N = Sh::N, H = Sh::H;
  const float gs = gm + gp, gd = gm - gp;
#pragma unroll
  for (int i = 0; i < H; i++) {
    float c[LineRows<P>::ROW];
    T.row(i, c);
    const float* co = c + H + Sh::ODD + 1;
    float e = c[0] * s[0], o = co[0] * d[0];
#pragma unroll
    for (int l = 1; l < H; l++) {
      e = fmaf(c[l], s[l], e);
      o = fmaf(co[l], d[l], o);
    }
    if constexpr (Sh::ODD != 0) e = fmaf(c[H], fm, e);
    e = fmaf(c[H + Sh::ODD], gd, e);
    o = fmaf(co[H], gs, o);
    emit(i, e + o);
    emit(N - 1 - i, o - e);
  }
  if constexpr (Sh::ODD != 0) {
    float c[LineRows<P>::MID];
    T.mid(c);
    float o = c[0] * d[0];
#pragma unroll
    for (int l = 1; l < H; l++) o = fmaf(c[l], d[l], o);
    o = fmaf(c[H], gs, o);
    emit(H, o);
  }
}

// Line at `line` (stride S) in shared memory, results over it.
template <int P, int S, typename Table>
__device__ __forceinline__ void line_shared(float* line, const Table& T, float gm, float gp) {
  using Sh = EoShape<P>;
  constexpr int N = Sh::N, H = Sh::H;
  float s[H], d[H], fm = 0.0f;
#pragma unroll
  for (int l = 0; l < H; l++) {
    const float lo = line[l * S], hi = line[(N - 1 - l) * S];
    s[l] = lo + hi;
    d[l] = lo - hi;
  }
  if constexpr (Sh::ODD != 0) fm = line[H * S];
  line_pairs<P>(s, d, fm, T, gm, gp, [&](int m, float v) { line[m * S] = v; });
}

// A read of what this launch does not write (RO: as a read-only load).
template <bool RO, typename T>
__device__ __forceinline__ T line_read(const T* p) {
  if constexpr (RO)
    return __ldg(p);
  else
    return *p;
}

// Elements [eb, eb + nloc) through one stage by a block of at least nloc N^2
// threads; smem: line_smem of epb elements; tab(d): the table of direction d;
// pre(): runs after the loads and before the block's first barrier.
template <int P, int RK, bool RO, typename Tab, typename Pre>
__device__ __forceinline__ void line_elements(const double* __restrict__ q,
                                              const double* __restrict__ q0,
                                              double* __restrict__ qout,
                                              const float* __restrict__ u,
                                              const float* __restrict__ v,
                                              const float* __restrict__ w, const Box& box,
                                              double ra, double rb, long long eb, int nloc, int epb,
                                              float* smem, Tab&& tab, Pre&& pre) {
  using Sh = FixShape<P>;
  using Eo = EoShape<P>;
  constexpr int N = Sh::N, N2 = Sh::N2, NP = N * N2, NS = Sh::NS, EW = Sh::EW, H = Eo::H;
  const int le = threadIdx.x / N2, r = threadIdx.x - le * N2;
  const bool on = le < nloc;
  const int i = r % N, j = r / N;
  float* sX = smem + le * EW;
  float* sY = sX + epb * EW;
  const long long ge = (eb + le) * NP;  // the element's first node
  const int zat = i + NS * j;  // the z line's first node in the padded arrays

  // the z line's fluxes, of which it keeps the pair values; the six face fluxes
  float g[6], s[H], d[H], fm = 0.0f;
  if (on) {
    if constexpr (RK == kRkGeneral)
      for (int t = 16 * r; t < NP; t += 16 * N2) prefetch_l2(q0 + ge + t);
    float F[N];
#pragma unroll
    for (int m = 0; m < N; m++) {
      const long long n = ge + r + m * N2;
      const float qv = to_ct<float>(line_read<RO>(q + n));
      sX[zat + m * NS * N] = qv * line_read<RO>(u + n);
      sY[zat + m * NS * N] = qv * line_read<RO>(v + n);
      F[m] = __fmul_rn(qv, line_read<RO>(w + n));
    }
#pragma unroll
    for (int l = 0; l < H; l++) {
      s[l] = F[l] + F[N - 1 - l];
      d[l] = F[l] - F[N - 1 - l];
    }
    if constexpr (Eo::ODD != 0) fm = F[H];
    unsigned nb[6];
    fix_neighbors(box, (unsigned)(eb + le), nb);
    const int x0 = i * N + j * N2, y0 = i + j * N2;
    const int nM[6] = {y0, x0 + (N - 1), y0 + (N - 1) * N, x0, r, r + (N - 1) * N2};
    const int nP[6] = {y0 + (N - 1) * N, x0, y0, x0 + (N - 1), r + (N - 1) * N2, r};
#pragma unroll
    for (int f = 0; f < 6; f++) {
      const long long gP = (long long)nb[f] * NP + nP[f];
      const float qP = to_ct<float>(line_read<RO>(q + gP)), qM = to_ct<float>(line_read<RO>(q + ge + nM[f]));
      const float* vel = (f == 1 || f == 3) ? u : (f == 0 || f == 2) ? v : w;
      const float uM = line_read<RO>(vel + ge + nM[f]), uP = line_read<RO>(vel + gP);
      const float a2 = fabsf(uP + uM);
      const float tw = (f == 1 || f == 2 || f == 5) ? 2.0f : -2.0f;
      g[f] = fmaf(qP, fmaf(tw, uP, -a2), -(qM * fmaf(tw, uM, -a2)));
    }
  }
  pre();
  __syncthreads();
  if (on) {
    // lines along i (r = j + N k) and along j (r = i + N k)
    line_shared<P, 1>(sX + NS * r, tab(0), g[3], g[1]);
    line_shared<P, NS>(sY + i + NS * N * j, tab(1), g[0], g[2]);
  }
  __syncthreads();
  if (on) {
    line_pairs<P>(s, d, fm, tab(2), g[4], g[5], [&](int m, float z) {
      const int at = zat + m * NS * N;
      const double inc = f32_to_f64_bits((sX[at] + sY[at]) + z);
      const long long n = ge + r + m * N2;
      if constexpr (RK == kRkTend)
        qout[n] = inc;
      else
        qout[n] = rk_combine<RK>(inc, line_read<RO>(q + n), RK == kRkGeneral ? line_read<RO>(q0 + n) : 0.0, ra, rb);
    });
  }
}

template <int P, int RK>
__global__ void __launch_bounds__(FixShape<P>::THREADS, line_min_blocks<P>())
    stage_line_kernel(const __grid_constant__ LineStageArgs<P> a) {
  const int epb = blockDim.x / FixShape<P>::N2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const long long eb = a.s.elem_begin + (long long)blockIdx.x * epb;
  const long long left = a.s.elem_begin + a.s.elem_count - eb;
  // p = 1: its two nodes a line wait little; plain reads 130 against 126
  line_elements<P, RK, (P > 1)>(a.s.q_in, a.s.q0, a.s.q_out, static_cast<const float*>(a.s.u),
                       static_cast<const float*>(a.s.v), static_cast<const float*>(a.s.w), a.s.box,
                       a.s.a, a.s.b, eb, (int)(left < epb ? left : epb), epb,
                       reinterpret_cast<float*>(smem_raw),
                       [&](int d) { return LineTable<P>{a.tab + d * EoShape<P>::TE}; }, [] {});
}

template <int P, int RK>
int launch_stage_line_kind(const LineStageArgs<P>& a, cudaStream_t st) {
  // small boxes take smaller blocks, as in launch_stage_fix_kind
  constexpr int N2 = FixShape<P>::N2;
  const long long want = std::max(a.s.elem_count / (2 * 152), 1LL);
  const int threads = (int)std::min<long long>((want * N2 + 31) / 32 * 32, FixShape<P>::THREADS);
  const int epb = threads / N2;
  const long long nblk = (a.s.elem_count + epb - 1) / epb;
  if (nblk <= 0) return SDG_OK;
  if (nblk > 0x7fffffffLL) return fail(SDG_ERR_INVALID_ARG, "too many elements");
  constexpr size_t smem = line_smem<P>(FixShape<P>::EPB);
  SDG_TRY(set_kernel_smem((const void*)stage_line_kernel<P, RK>, (int)smem,
                          carve_for(smem, line_min_blocks<P>())));
  stage_line_kernel<P, RK><<<(unsigned)nblk, threads, line_smem<P>(epb), st>>>(a);
  SDG_CUDA_TRY(cudaGetLastError());
  return SDG_OK;
}

template <int P>
int launch_stage_line_impl(const StageArgs& s, cudaStream_t st) {
  LineStageArgs<P> a;
  a.s = s;
  constexpr int TE = EoShape<P>::TE;
  for (int d = 0; d < 3; d++)
    for (int t = 0; t < TE; t++)
      a.tab[d * TE + t] =
          s.eo_host[d * TE + t] * (t < EoShape<P>::OFF_A ? s.eo_sDf[d] : s.eo_sLf[d]);
  switch (rk_kind(s)) {
    case kRkTend: return launch_stage_line_kind<P, kRkTend>(a, st);
    case kRkFirst: return launch_stage_line_kind<P, kRkFirst>(a, st);
    default: return launch_stage_line_kind<P, kRkGeneral>(a, st);
  }
}

}  // namespace sdg
