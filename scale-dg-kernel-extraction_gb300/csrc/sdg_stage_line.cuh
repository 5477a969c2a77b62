// Fused RK-stage kernel of the FP32-compute form with the even-odd pair sums:
// FP64 state, FP32 velocity, products and sums, FP64 RK update.
//
// Thread r of an element's N^2 owns line r of each direction and node r of
// each face (the layout of stage_fix_kernel): its face fluxes and the z line's
// pair values never leave its registers, shared memory holds the x and y
// fluxes and then their line results, and the coefficients, scaled for the
// stage on the host, are kernel parameters, which a multiply-add takes from
// the constant bank.  Every value is formed in the order of operations of
// stage_eo_block (products rounded before the pair sums, x + y + z, widened
// increment), so both give the same bits.
//
// Bound: 28 bytes a node in the first stage and 36 in the others, read and
// written once, at two thirds of the copy bandwidth; 32 warps an SM wait on
// the loads at the two ends of a block.  On GB300, 16.8M DOF, against the
// kernels this replaced (GDOF-updates/s): p = 2 136 from 110, p = 3 140 from
// 106, p = 4 143 from 82, p = 5 137 from 82, p = 7 151 from 108, p = 9 131 from
// 87, p = 11 134 from 93, p = 15 130 from 87 (p = 1 level at 130).  Most of it
// comes from L1: with the largest shared-memory carveout 84 at p = 5.  64
// registers (1024 threads an SM): 1280 threads 0.85-1.0x, 768 0.9-1.03x.
// Velocity factors of the faces stored by the call's first stage, as the FP64
// form does: 0.88-1.03x.
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

// One line from its pair values s, d and face fluxes: the N results to
// emit(m, value), in the order of operations of eo_line_f.
template <int P, typename Emit>
__device__ __forceinline__ void line_pairs(const float* s, const float* d, float fm, const float* T,
                                           float gm, float gp, Emit&& emit) {
  using Sh = EoShape<P>;
  constexpr int N = Sh::N, H = Sh::H;
  const float gs = gm + gp, gd = gm - gp;
#pragma unroll
  for (int i = 0; i < H; i++) {
    float e = T[Sh::OFF_E + i * H] * s[0], o = T[Sh::OFF_O + i * H] * d[0];
#pragma unroll
    for (int l = 1; l < H; l++) {
      e = fmaf(T[Sh::OFF_E + i * H + l], s[l], e);
      o = fmaf(T[Sh::OFF_O + i * H + l], d[l], o);
    }
    if constexpr (Sh::ODD != 0) e = fmaf(T[Sh::OFF_DM + i], fm, e);
    e = fmaf(T[Sh::OFF_B + i], gd, e);
    o = fmaf(T[Sh::OFF_A + i], gs, o);
    emit(i, e + o);
    emit(N - 1 - i, o - e);
  }
  if constexpr (Sh::ODD != 0) {
    float o = T[Sh::OFF_O + H * H] * d[0];
#pragma unroll
    for (int l = 1; l < H; l++) o = fmaf(T[Sh::OFF_O + H * H + l], d[l], o);
    o = fmaf(T[Sh::OFF_A + H], gs, o);
    emit(H, o);
  }
}

// Line at `line` (stride S) in shared memory, results over it.
template <int P, int S>
__device__ __forceinline__ void line_shared(float* line, const float* T, float gm, float gp) {
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

template <int P, int RK>
__global__ void __launch_bounds__(FixShape<P>::THREADS, line_min_blocks<P>())
    stage_line_kernel(const __grid_constant__ LineStageArgs<P> a) {
  using Sh = FixShape<P>;
  using Eo = EoShape<P>;
  constexpr int N = Sh::N, N2 = Sh::N2, NP = N * N2, NS = Sh::NS, EW = Sh::EW,
                H = Eo::H;
  const int epb = blockDim.x / N2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const long long eb = a.s.elem_begin + (long long)blockIdx.x * epb;
  const long long left = a.s.elem_begin + a.s.elem_count - eb;
  const int nloc = (int)(left < epb ? left : epb);
  const int le = threadIdx.x / N2, r = threadIdx.x - le * N2;
  const bool on = le < nloc;
  const int i = r % N, j = r / N;
  float* sX = reinterpret_cast<float*>(smem_raw) + le * EW;
  float* sY = sX + epb * EW;
  const long long ge = (eb + le) * NP;  // the element's first node
  const double* __restrict__ q = a.s.q_in;
  const int zat = i + NS * j;  // the z line's first node in the padded arrays

  // the z line's fluxes, of which it keeps the pair values; the six face fluxes
  float g[6], s[H], d[H], fm = 0.0f;
  if (on) {
    if constexpr (RK == kRkGeneral)
      for (int t = 16 * r; t < NP; t += 16 * N2) prefetch_l2(a.s.q0 + ge + t);
    const float* __restrict__ u = static_cast<const float*>(a.s.u);
    const float* __restrict__ v = static_cast<const float*>(a.s.v);
    const float* __restrict__ w = static_cast<const float*>(a.s.w);
    float F[N];
#pragma unroll
    for (int m = 0; m < N; m++) {
      const long long n = ge + r + m * N2;
      const float qv = to_ct<float>(q[n]);
      sX[zat + m * NS * N] = qv * u[n];
      sY[zat + m * NS * N] = qv * v[n];
      F[m] = __fmul_rn(qv, w[n]);
    }
#pragma unroll
    for (int l = 0; l < H; l++) {
      s[l] = F[l] + F[N - 1 - l];
      d[l] = F[l] - F[N - 1 - l];
    }
    if constexpr (Eo::ODD != 0) fm = F[H];
    unsigned nb[6];
    fix_neighbors(a.s.box, (unsigned)(eb + le), nb);
    const int x0 = i * N + j * N2, y0 = i + j * N2;
    const int nM[6] = {y0, x0 + (N - 1), y0 + (N - 1) * N, x0, r, r + (N - 1) * N2};
    const int nP[6] = {y0 + (N - 1) * N, x0, y0, x0 + (N - 1), r + (N - 1) * N2, r};
#pragma unroll
    for (int f = 0; f < 6; f++) {
      const long long gP = (long long)nb[f] * NP + nP[f];
      const float qP = to_ct<float>(q[gP]), qM = to_ct<float>(q[ge + nM[f]]);
      const float* vel = (f == 1 || f == 3) ? u : (f == 0 || f == 2) ? v : w;
      const float uM = vel[ge + nM[f]], uP = vel[gP];
      const float a2 = fabsf(uP + uM);
      const float tw = (f == 1 || f == 2 || f == 5) ? 2.0f : -2.0f;
      g[f] = fmaf(qP, fmaf(tw, uP, -a2), -(qM * fmaf(tw, uM, -a2)));
    }
  }
  __syncthreads();
  if (on) {
    // lines along i (r = j + N k) and along j (r = i + N k)
    line_shared<P, 1>(sX + NS * r, a.tab, g[3], g[1]);
    line_shared<P, NS>(sY + i + NS * N * j, a.tab + Eo::TE, g[0], g[2]);
  }
  __syncthreads();
  if (on) {
    const double* __restrict__ q0 = a.s.q0;
    double* __restrict__ qout = a.s.q_out;
    const double ra = a.s.a, rb = a.s.b;
    line_pairs<P>(s, d, fm, a.tab + 2 * Eo::TE, g[4], g[5], [&](int m, float z) {
      const int at = zat + m * NS * N;
      const double inc = f32_to_f64_bits((sX[at] + sY[at]) + z);
      const long long n = ge + r + m * N2;
      if constexpr (RK == kRkTend)
        qout[n] = inc;
      else
        qout[n] = rk_combine<RK>(inc, q[n], RK == kRkGeneral ? q0[n] : 0.0, ra, rb);
    });
  }
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
