// The element contractions with their sums in fixed point (sdg_fix.cuh):
// tensorprod_divlike_dirXYZ (mod_dg_optr_kernel.f90:62-136), gradlike and the
// single-direction matvecs (opt1 erb:51-129, :166-219).
//
// In FP64 these kernels kept the FP64 pipe 93-96 % busy (24 FP64 instructions a
// node at p = 7 for 48 bytes).  As integer sums they have none; a sum is then
// the exact one to about 2^-59 of the product of its row's magnitudes and its
// line's largest value, rounded once, whatever the order GENERAL or OPT1 asks for.
//
// That is no less than FP64 gives where the largest value meets an entry of some
// size in every row.  So
//   * a matrix with an entry off its diagonal below 2^-10 of its row's magnitudes (a
//     filter, an identity, a triangular matrix: the derivative's smallest is 2^-9 at
//     p = 15) keeps FP64 sums, in the order asked for;
//   * where the diagonal has such entries (a derivative's interior rows), the row of
//     a line's largest value is summed in FP64 when no other value is within 2^6
//     of it (kFixAlone);
//   * lines with infinities, NaN or magnitudes near the ends of the exponent range
//     are summed in FP64.
//
// Measured on 10M nodes on GB300, us, against the FP64 kernels: divlike p = 3
// 126 / 212, p = 7 160 / 406 (3.0 TB/s, 44 % of the measured HBM rate), p = 15
// 272 / 980; gradlike p = 7 154 / 402; one direction p = 7 60 / 140.  The Lift
// operator, six products a node with a scale of their own, measured level as
// integer sums (98-109 / 105-107, and slower below 1M nodes) and stays in FP64.
#pragma once

#include "sdg_stage_fix.cuh"

namespace sdg {

struct DivArgs {
  double* ox;
  double* oy;
  double* oz;
  const double* D;
  const double* Dt;
  const double* ix;
  const double* iy;
  const double* iz;
  int nelem;
  bool staged = false;  // divlike: an output is another direction's input
  bool split = false;   // FP64 sums in OPT1's three parts (p > 7)
};

// The exponent of a row whose magnitudes add up to sum (with room for the
// rounding of the sum and of a coefficient's high limb), kBadRow outside +-200.
constexpr int kBadRow = 1 << 20;
__device__ __forceinline__ int fix_row_exp(double sum) {
  const int e = (int)((unsigned)__double2hiint(sum * (1.0 + 1e-8)) >> 20 & 0x7FFu);
  if (sum == 0.0) return 0;
  return e < 1022 - 200 || e > 1022 + 200 ? kBadRow : e - 1022;
}

// A line's sums in FP64, M(i,l) at M[i * si + l * sl].
template <int P>
__device__ __noinline__ void ops_line_fp64(const double* __restrict__ M, int si, int sl,
                                           const double* F, int fs, double* out, int os) {
  constexpr int N = P + 1;
  double r[N];
#pragma unroll 1
  for (int i = 0; i < N; i++) {
    double s = M[i * si] * F[0];
#pragma unroll 1
    for (int l = 1; l < N; l++) s = fma(M[i * si + l * sl], F[l * fs], s);
    r[i] = s;
  }
  for (int i = 0; i < N; i++) out[i * os] = r[i];  // out may be F
}

// How a matrix's rows are summed: kOpsFixed in fixed point, kOpsDiag the same with
// small entries on the diagonal, kOpsDouble in FP64.
constexpr int kOpsFixed = 0, kOpsDiag = 1, kOpsDouble = 2;

// The kind row i of a matrix allows: v(l) its entries, sum their magnitudes.
template <int N, typename V>
__device__ __forceinline__ int ops_row_kind(int i, double sum, V&& v) {
  if (fix_row_exp(sum) == kBadRow) return kOpsDouble;
  const double least = sum * (1.0 / 1024.0);
  int kind = kOpsFixed;
  for (int l = 0; l < N; l++)
    if (fabs(v(l)) < least) kind = max(kind, l == i ? kOpsDiag : kOpsDouble);
  return kind;
}

// One line: out(i) = sum_l M(i,l) F(l), F at in with
// stride S, out with SO (one array, for lines in shared memory); T and row are the
// matrix's limbs (kOpsDouble: its entries) and row exponents, M, si, sl the matrix
// itself.
template <int P, int S, int SO>
__device__ __forceinline__ void ops_line(const fixlimb* T, const int* row, int kind, bool split,
                                         const double* __restrict__ M, int si, int sl,
                                         const double* in, double* out) {
  constexpr int N = P + 1;
  double F[N];
#pragma unroll
  for (int l = 0; l < N; l++) F[l] = in[l * S];
  if (kind == kOpsDouble) {
    const double* A = reinterpret_cast<const double*>(T);
#pragma unroll 2
    for (int i = 0; i < N; i++) {
      if constexpr (P > 7) {
        if (split) {
          out[i * SO] = line_sum<N, true, 1>(A + i * N, F, 1);
          continue;
        }
      }
      out[i * SO] = line_sum<N, false, 1>(A + i * N, F, 1);
    }
    return;
  }
  int32_t E = 0, E2 = 0;  // the largest exponent, the next
#pragma unroll
  for (int l = 0; l < N; l++) {
    const int32_t x = fix_value_exp(F[l]);
    E2 = max(E2, min(E, x));
    E = max(E, x);
  }
  const bool spike = kind == kOpsDiag && E - E2 > kFixAlone;
  E = fix_line_scale<N>(F, E, 0.0, 0.0);
  if (!fix_in_range(E)) {
    ops_line_fp64<P>(M, si, sl, in, S, out, SO);
    return;
  }
  int at = 0;
  double sum = 0.0;
  if (spike) {
#pragma unroll
    for (int l = 0; l < N; l++)
      if (fix_value_exp(F[l]) == E) at = l;
#pragma unroll
    for (int l = 0; l < N; l++) sum = fma(M[at * si + l * sl], F[l], sum);
  }
  fixlimb f[N];
#pragma unroll
  for (int l = 0; l < N; l++) f[l] = fix_split(fix_align(F[l], E));
  const int B = fix_line_exp(E) - 61;
#pragma unroll 2
  for (int i = 0; i < N; i++) {
    fixacc o;
    fix_mul(o, T[i * N], f[0]);
#pragma unroll
    for (int l = 1; l < N; l++) fix_fma(o, T[i * N + l], f[l]);
    out[i * SO] = fix_to_double(fix_sum(o), B + row[i]);
  }
  if (spike) out[at * SO] = sum;
}

template <int P>
__host__ __device__ constexpr size_t ops_smem() {
  using Sh = FixShape<P>;
  return sizeof(double) * Sh::EPB * Sh::EW + sizeof(fixlimb) * 2 * Sh::N2 + sizeof(int) * 2 * Sh::N;
}

// GRAD: the three derivatives of one field (a.ix; a null output is skipped),
// else one of each of three.  Blocks walk the elements with a grid stride, so
// the matrices become limbs once a block; thread r of an element owns line r of
// each direction.  y and z lines are read and written in place, coalesced along
// i; x lines go through shared memory.  An output may be its own direction's
// input, and any of gradlike's, which stages its field, may be the field.
template <int P, bool GRAD>
__global__ void __launch_bounds__(FixShape<P>::THREADS, 1024 / FixShape<P>::THREADS)
    ops_kernel(const DivArgs a) {
  using Sh = FixShape<P>;
  constexpr int N = Sh::N, N2 = Sh::N2, NP = N * N2, NS = Sh::NS, EW = Sh::EW, EPB = Sh::EPB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sF = reinterpret_cast<double*>(smem_raw);
  fixlimb* sT = reinterpret_cast<fixlimb*>(sF + EPB * EW);  // D1D, then D1D_tr: (i, l)
  int* sRow = reinterpret_cast<int*>(sT + 2 * N2);
  const int le = threadIdx.x / N2, r = threadIdx.x - le * N2;
  const int i = r % N, j = r / N;
  auto M = [&](int k) {  // entry k of the two matrices, (i, l) at i N + l
    const int w = k % N2;
    return k < N2 ? a.D[w / N + (w % N) * N] : a.Dt[w % N + (w / N) * N];
  };
  __shared__ int sKind[2];
  if (threadIdx.x < 2) sKind[threadIdx.x] = kOpsFixed;
  __syncthreads();
  for (int t = threadIdx.x; t < 2 * N; t += blockDim.x) {
    double s = 0.0;
    for (int l = 0; l < N; l++) s += fabs(M(t * N + l));
    sRow[t] = fix_row_exp(s);
    atomicMax(&sKind[t / N], ops_row_kind<N>(t % N, s, [&](int l) { return M(t * N + l); }));
  }
  __syncthreads();
  const int kx = sKind[0], kyz = sKind[1];  // D1D, D1D_tr
  for (int t = threadIdx.x; t < 2 * N2; t += blockDim.x) {
    const int k = sRow[t / N];
    if (sKind[t / N2] == kOpsDouble)
      reinterpret_cast<double*>(sT)[t] = M(t);
    else
      sT[t] = fix_coef(fix_unit(M(t) * __hiloint2double((1023 - k) << 20, 0)));
  }
  __syncthreads();
  double* sE = sF + le * EW;
  for (long long eb = (long long)blockIdx.x * EPB; eb < a.nelem;
       eb += (long long)gridDim.x * EPB) {
    const bool on = le < EPB && eb + le < a.nelem;
    const long long g = (eb + le) * NP;
    const int zat = i + NS * j;
    if (on && (GRAD || a.ox)) {
#pragma unroll
      for (int m = 0; m < N; m++) sE[zat + m * NS * N] = a.ix[g + r + m * N2];
    }
    if (!GRAD && on) {
      ops_line<P, N, N>(sT + N2, sRow + N, kyz, a.split, a.Dt, N, 1, a.iy + g + i + j * N2,
                     a.oy + g + i + j * N2);
      ops_line<P, N2, N2>(sT + N2, sRow + N, kyz, a.split, a.Dt, N, 1, a.iz + g + r, a.oz + g + r);
    }
    __syncthreads();
    if (GRAD && on) {
      // from shared memory, the results straight out
      if (a.oy) ops_line<P, NS, N>(sT + N2, sRow + N, kyz, a.split, a.Dt, N, 1, sE + i + NS * N * j,
                                      a.oy + g + i + j * N2);
      if (a.oz) ops_line<P, NS * N, N2>(sT + N2, sRow + N, kyz, a.split, a.Dt, N, 1, sE + zat,
                                           a.oz + g + r);
    }
    if (!GRAD || a.ox) {
      if (GRAD) __syncthreads();
      if (on) ops_line<P, 1, 1>(sT, sRow, kx, a.split, a.D, 1, N, sE + NS * r, sE + NS * r);
      __syncthreads();
      if (on) {
#pragma unroll
        for (int m = 0; m < N; m++) a.ox[g + r + m * N2] = sE[zat + m * NS * N];
      }
    }
    __syncthreads();
  }
}

template <int P, bool GRAD>
int launch_ops(const DivArgs& a, cudaStream_t st) {
  using Sh = FixShape<P>;
  if (a.nelem <= 0) return SDG_OK;
  constexpr size_t smem = ops_smem<P>();
  SDG_TRY(set_kernel_smem((const void*)ops_kernel<P, GRAD>, (int)smem, kCarveMax));
  // as many blocks as the registers let reside
  const long long nblk = ((long long)a.nelem + Sh::EPB - 1) / Sh::EPB;
  const long long most = 152LL * (1024 / Sh::THREADS);
  ops_kernel<P, GRAD><<<(unsigned)std::min(nblk, most), Sh::THREADS, smem, st>>>(a);
  SDG_CUDA_TRY(cudaGetLastError());
  return SDG_OK;
}

}  // namespace sdg
