// Fused RK-stage kernel of the FP64 form with the line sums in 60-bit fixed
// point (sdg_fix.cuh).
//
// An FP64 even-odd stage spends 28.8 FP64 instructions a DOF at p = 7 and kept
// the FP64 pipe 90 % busy at 19.8 GDOF-updates/s.  Here the even-odd pair
// sums, the derivative and the lift are integer multiply-adds, and FP64 keeps
// the products q u_d, the face flux and the RK update (6.8 instructions a
// DOF): 68 GDOF-updates/s at p = 7 on 32^3 elements (246 us a stage, from
// 848), 46-68 across p = 1..15 (from 13-22), with 32 warps an SM waiting on
// the loads of its two ends.  Error of a tendency against a long-double one: 0.5-1.1 times the
// FP64 body's at every order, on smooth, narrow and random fields (the
// coefficients' symmetrisation, common to both, dominates from p = 5).
//
// The pairs: S(l) = F(l) + F(N-1-l), d(l) = F(l) -
// F(N-1-l), e_i = sum E(i,l) S(l) [+ D(i,mid) F(mid)] + B(i) (g- - g+),
// o_i = sum O(i,l) d(l) + A(i) (g- + g+), out(i) = o_i + e_i, out(N-1-i) =
// o_i - e_i.  The coefficients (Escale, Fscale and the minus sign of dqdt
// folded in) are kernel parameters, so a multiply-add takes them from the
// constant bank.  The x, y and z results of a node add up as integers; the
// increment is their sum times one factor of the element and the stage.
//
// Face flux: qP tP - qM tM with tP = 2VelP - 2a, tM = 2VelM - 2a, 2a = |uP + uM|
// (a quarter of Fscale is in the lift coefficients).  With operators as given
// it is formed as qP (tP - tM) + (qP - qM) tM: a rounding of tM or of its product
// then weighs with the jump, not with q, which keeps the tendency's error on
// smooth fields at 0.6-0.95 of the FP64 node body's (p = 11: 7e-16 against
// 8.8e-16; 1.7e-15 with the first form).  The factors, (tP, tM) or
// (tP - tM, tM), come from the first stage of a call, which stores them.
//
// Scale: a line's values share the power of two that bounds its fluxes q u_d
// and its two face fluxes, and a row of coefficients has a power of two of its
// own, so every line result keeps about 2^-61 of its own bound.  The three
// results of a node are added as integers on the largest of their scales and
// become one double.  A line with infinities, NaN, magnitudes near the ends of
// the exponent range or a value alone in it (FixScan) is formed in FP64 by its
// thread, and its nodes add up in FP64.
//
// Thread layout: thread r of an element's N^2 owns line r of each direction
// and node r of each face, so a line's face fluxes never leave their thread.
//   0  the z line's x and y fluxes to shared memory, the six face fluxes
//   1  x line and y line r, results over the fluxes
//   2  z line r, and the RK update of its nodes
#pragma once

#include <algorithm>

#include "sdg_fix.cuh"
#include "sdg_stage_eo.cuh"

namespace sdg {

template <int P>
struct FixShape {
  static constexpr int N = P + 1, N2 = N * N;
  static constexpr int NS = (N & 1) ? N : N + 1;  // padded x row: odd, so that
                                                  // rows start on distinct banks
  static constexpr int EW = NS * N2;              // words of an element's array
  // threads: whole elements of N^2 lines in 128 or 256 threads, whichever
  // leaves fewer idle; one element in whole warps from p = 10
  static constexpr int THREADS = (N2 > 100) ? ((N2 + 31) / 32) * 32
                                 : (N2 == 49 || N2 == 81) ? 256 : 128;
  static constexpr int EPB = THREADS / N2;
};

// EO: coefficients of the even-odd pairs; else those of D1D as given, with the
// lift entries of every node (operators without the symmetries, and the
// GENERAL and OPT1 types, whose sums differ only in an order that integer sums
// do not have).
template <int P, bool EO>
struct FixStageArgs {
  static constexpr int TAB = EO ? EoShape<P>::TE : (P + 1) * (P + 1);
  static constexpr int ROWS = EO ? EoShape<P>::HR : P + 1;
  StageArgs s;
  double c;              // EO: b dt, else dt
  fixlimb tab[3 * TAB];  // per direction: EoShape's table, or D(i,l) at i N + l
  int row[3 * ROWS];     // exponent of a row's scale, less 61
  int ok;                // 0: coefficients out of range, every line in FP64
  int thin;              // the lift has zeros
  static __host__ __device__ constexpr int row_of(int m) {
    return EO ? (m < P - m ? m : P - m) : m;
  }
  __device__ const int4* lift(int ax, int r) const {
    return static_cast<const int4*>(s.fix_lift) + ax * (P + 1) * (P + 1) * (P + 1) + r;
  }
};

template <int P>
__host__ __device__ constexpr size_t fix_smem(int epb) {
  return sizeof(double) * 2 * epb * FixShape<P>::EW + sizeof(short) * 2 * epb * FixShape<P>::N2;
}

// A line in FP64, for values the fixed-point path does not take: F holds the
// line's fluxes with stride fs, results to out[0..N).  A call of its own, so that
// its registers do not count against the kernel's.
template <int P, bool EO>
__device__ __noinline__ void fix_line_fp64(const StageArgs* a, int ax, int r, const double* F,
                                           int fs, double gm, double gp, double* out) {
  using Sh = EoShape<P>;
  constexpr int N = Sh::N, H = Sh::H, N2 = N * N, NP = N * N2;
  const double sD = -a->box.Es[ax], sL = -(0.25 * a->box.Fs[ax]);
  const double* __restrict__ T = static_cast<const double*>(a->D);
  if constexpr (!EO) {
    const int fm = ax == 0 ? 3 : ax == 1 ? 0 : 4, fp = ax == 0 ? 1 : ax == 1 ? 2 : 5;
    const double* __restrict__ L = static_cast<const double*>(a->Lift);
#pragma unroll 1
    for (int i = 0; i < N; i++) {
      double d = 0.0;
#pragma unroll 1
      for (int l = 0; l < N; l++) d = fma(T[i + l * N], F[l * fs], d);
      const int n = ax == 0 ? i + N * r : ax == 1 ? r % N + N * i + N2 * (r / N) : r + N2 * i;
      out[i] = fma(sD, d, sL * fma(L[n + fm * NP], gm, L[n + fp * NP] * gp));
    }
    return;
  }
  T += ax * Sh::TE;
  const double gs = gm + gp, gd = gm - gp;
#pragma unroll 1
  for (int i = 0; i < Sh::HR; i++) {
    double e = 0.0, o = 0.0;
#pragma unroll 1
    for (int l = 0; l < H; l++) {
      const double f1 = F[l * fs], f2 = F[(N - 1 - l) * fs];
      if (i < H) e = fma(T[Sh::OFF_E + i * H + l], f1 + f2, e);
      o = fma(T[Sh::OFF_O + i * H + l], f1 - f2, o);
    }
    if (Sh::ODD != 0 && i < H) e = fma(T[Sh::OFF_DM + i], F[H * fs], e);
    o = fma(sD, o, sL * (T[Sh::OFF_A + i] * gs));
    if (i < H) {
      e = fma(sD, e, sL * (T[Sh::OFF_B + i] * gd));
      out[i] = o + e;
      out[N - 1 - i] = o - e;
    } else {
      out[i] = o;
    }
  }
}

// One line: F its fluxes q u_d on the scale E, im / ip its - and + face's
// fluxes as integers, T its direction's coefficients and (operators as given)
// lift its nodes' lift limbs, N^2 apart; emit(m, I): the result is I times two
// to the line's exponent (fix_line_exp) plus its row's.
template <int P, bool EO, typename Emit>
__device__ __forceinline__ void fix_line(const fixlimb* T, const int4* __restrict__ lift,
                                         const double* F, int32_t E, int64_t im, int64_t ip,
                                         Emit&& emit) {
  using Sh = EoShape<P>;
  constexpr int N = Sh::N, H = Sh::H;
  if constexpr (!EO) {
    const fixlimb lm = fix_split(im), lp = fix_split(ip);
    fixlimb f[N];
#pragma unroll
    for (int l = 0; l < N; l++) f[l] = fix_split(fix_align(F[l], E));
    // four rows at a time up to p = 7 (1.00-1.05x), two above (four 0.99x)
    constexpr int kRows = N <= 8 ? 4 : 2;
#pragma unroll kRows
    for (int i = 0; i < N; i++) {
      const int4 c = lift[i * N * N];
      fixacc o;
      fix_mul(o, fixlimb{c.x, c.y}, lm);
      fix_fma(o, fixlimb{c.z, c.w}, lp);
#pragma unroll
      for (int l = 0; l < N; l++) fix_fma(o, T[i * N + l], f[l]);
      emit(i, fix_sum(o));
    }
    return;
  }
  fixlimb s[H], d[H], fm{0, 0};
#pragma unroll
  for (int l = 0; l < H; l++) {
    const int64_t f1 = fix_align(F[l], E), f2 = fix_align(F[N - 1 - l], E);
    s[l] = fix_split(f1 + f2);
    d[l] = fix_split(f1 - f2);
  }
  if constexpr (Sh::ODD != 0) fm = fix_split(fix_align(F[H], E));
  const fixlimb gs = fix_split(im + ip), gd = fix_split(im - ip);
#pragma unroll
  for (int i = 0; i < H; i++) {
    fixacc e, o;
    fix_mul(e, T[Sh::OFF_B + i], gd);
    fix_mul(o, T[Sh::OFF_A + i], gs);
#pragma unroll
    for (int l = 0; l < H; l++) {
      fix_fma(e, T[Sh::OFF_E + i * H + l], s[l]);
      fix_fma(o, T[Sh::OFF_O + i * H + l], d[l]);
    }
    if constexpr (Sh::ODD != 0) fix_fma(e, T[Sh::OFF_DM + i], fm);
    const int64_t es = fix_sum(e), os = fix_sum(o);
    emit(i, os + es);
    emit(N - 1 - i, os - es);
  }
  if constexpr (Sh::ODD != 0) {
    fixacc o;
    fix_mul(o, T[Sh::OFF_A + H], gs);
#pragma unroll
    for (int l = 0; l < H; l++) fix_fma(o, T[Sh::OFF_O + H * H + l], d[l]);
    emit(H, fix_sum(o));
  }
}

// The largest exponent field of a line's values, and whether a node of the line
// would lose what FP64 has: one whose own value is alone (kFixAlone), where
// the derivative has a zero on its diagonal (every row between the ends, of
// operators as given; the middle one of the even-odd pairs, whose other rows form
// sums and differences of the two values in either arithmetic), or, where the lift
// has zeros (thin), one that does not see a face flux that is.  Such a line's scale
// lies out of range: it is formed in FP64.  (A face flux counted so for every lift
// takes a tracer's fronts to FP64: OPT1, p = 7 147 us a stage against 95; a value
// eight times all others for alone 110.)
template <int P, bool EO>
struct FixScan {
  static constexpr int N = P + 1, MID = EO && (N & 1) ? N / 2 : -1;
  static constexpr bool SECOND = !EO && P > 1;
  int32_t e = 0, next = 0;  // next: the second largest (SECOND), all but MID's
  __device__ __forceinline__ void add(int l, int32_t x) {
    if constexpr (SECOND) next = max(next, min(e, x));
    if constexpr (MID >= 0) {
      if (l != MID) next = max(next, x);
    }
    e = max(e, x);
  }
  // face: the larger exponent field of the line's faces (negative: none)
  __device__ __forceinline__ int32_t scale(int32_t face, bool thin) const {
    const int32_t E = max(e, face);
    const int32_t rest = thin ? next : max(next, face);
    return (SECOND || MID >= 0) && E - rest > kFixAlone ? kFixRefused : E;
  }
};

// The scale of a line whose largest exponent field is E: a line of zeros (a
// tracer that fills part of the box, a velocity without a component) stays in
// fixed point; in FP64 its nodes' sums cost more than all others (p = 7 113 us a
// stage against 72).
template <int N>
__device__ __forceinline__ int32_t fix_line_scale(const double* F, int32_t E, double gm,
                                                  double gp) {
  if (E > 0) return E;
  auto bits = [](double x) { return __double2hiint(x) << 1 | __double2loint(x); };
  int any = bits(gm) | bits(gp);
#pragma unroll
  for (int l = 0; l < N; l++) any |= bits(F[l]);
  return any == 0 ? kFixZeros : 0;
}

// Exponent of a line formed in FP64: its results are doubles.
constexpr int kFixDouble = 1 << 14;

// The line of direction AX held in shared memory with stride S, its results
// over it as integers (or doubles); returns the line's exponent.
template <int P, bool EO, int AX, int S>
__device__ __forceinline__ int fix_line_shared(const FixStageArgs<P, EO>& a, int r, double* line,
                                               double gm, double gp) {
  constexpr int N = P + 1;
  double F[N];
  FixScan<P, EO> scan;
#pragma unroll
  for (int l = 0; l < N; l++) {
    F[l] = line[l * S];
    scan.add(l, fix_value_exp(F[l]));
  }
  const int32_t E = scan.scale(max(fix_face_exp(gm), fix_face_exp(gp)), !EO && a.thin);
  if (a.ok && fix_in_range(E)) {
    int64_t* out = reinterpret_cast<int64_t*>(line);
    fix_line<P, EO>(a.tab + AX * a.TAB, a.lift(AX, r), F, E, fix_align_face(gm, E),
                    fix_align_face(gp, E), [&](int m, int64_t v) { out[m * S] = v; });
    return fix_line_exp(E);
  }
  // zeros (fix_product's are +0) are their own results
  if (a.ok && fix_line_scale<N>(F, E, gm, gp) == kFixZeros) return fix_line_exp(kFixZeros);
  double out[N];
  fix_line_fp64<P, EO>(&a.s, AX, r, line, S, gm, gp, out);
  for (int m = 0; m < N; m++) line[m * S] = out[m];
  return kFixDouble;
}

// A node's tendency from its three line results v with exponents e (at least
// one a double): the sum in FP64.
static __device__ __noinline__ double fix_node_fp64(int64_t x, int ex, int64_t y, int ey, int64_t z,
                                             int ez) {
  auto value = [](int64_t v, int e) {
    return e >= kFixDouble / 2 ? __longlong_as_double(v) : v == 0 ? 0.0 : fix_to_double(v, e);
  };
  return (value(x, ex) + value(y, ey)) + value(z, ez);
}

// A node's tendency from its three line results v with exponents e, as
// integers (each below 2^61) on the largest of their scales.
__device__ __forceinline__ double fix_node(int64_t x, int ex, int64_t y, int ey, int64_t z,
                                           int ez) {
  const int e = max(ex, max(ey, ez));
  if (e >= kFixDouble / 2) return fix_node_fp64(x, ex, y, ey, z, ez);
  return fix_to_double(fix_sar(x, e - ex) + fix_sar(y, e - ey) + fix_sar(z, e - ez), e);
}

// Neighbour elements of e across the faces -y, +x, +y, -x, -z, +z with
// periodic wrap.
__device__ __forceinline__ void fix_neighbors(const Box& b, unsigned e, unsigned nb[6]) {
  const unsigned NX = b.NeX, NY = b.NeY, NZ = b.NeZ, sy = NX, sz = NX * NY;
  const unsigned rxy = e / NX, ex = e - rxy * NX, ez = rxy / NY, ey = rxy - ez * NY;
  nb[0] = (ey == 0) ? e + (NY - 1) * sy : e - sy;
  nb[2] = (ey == NY - 1) ? e - (NY - 1) * sy : e + sy;
  nb[3] = (ex == 0) ? e + (NX - 1) : e - 1;
  nb[1] = (ex == NX - 1) ? e - (NX - 1) : e + 1;
  nb[4] = (ez == 0) ? e + (NZ - 1) * sz : e - sz;
  nb[5] = (ez == NZ - 1) ? e - (NZ - 1) * sz : e + sz;
}

template <int P>
__host__ __device__ constexpr int fix_min_blocks() {
  return P >= 14 ? 3 : 1024 / FixShape<P>::THREADS;
}

// RK: the stage's update kind; FCIN: the velocity factors of the face flux
// come from an earlier stage of the call.
template <int P, bool EO, int RK, bool FCIN>
__global__ void __launch_bounds__(FixShape<P>::THREADS, fix_min_blocks<P>())
    stage_fix_kernel(const __grid_constant__ FixStageArgs<P, EO> a) {
  using Args = FixStageArgs<P, EO>;
  using Sh = FixShape<P>;
  constexpr int N = Sh::N, N2 = Sh::N2, NP = N * N2, NFT = 6 * N2, NS = Sh::NS, EW = Sh::EW;
  const int epb = blockDim.x / N2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const long long eb = a.s.elem_begin + (long long)blockIdx.x * epb;
  const long long left = a.s.elem_begin + a.s.elem_count - eb;
  const int nloc = (int)(left < epb ? left : epb);
  const int le = threadIdx.x / N2, r = threadIdx.x - le * N2;
  const bool on = le < nloc;
  const int i = r % N, j = r / N;
  double* sX = reinterpret_cast<double*>(smem_raw) + le * EW;
  double* sY = sX + epb * EW;
  // exponents of the element's x and y lines
  short* sEx =
      reinterpret_cast<short*>(reinterpret_cast<double*>(smem_raw) + 2 * epb * EW) + le * N2;
  short* sEy = sEx + epb * N2;
  const long long ge = (eb + le) * NP;  // the element's first node
  const double* __restrict__ q = a.s.q_in;
  const int zat = i + NS * j;  // the z line's first node in the padded arrays

  // 0: the z line's x and y fluxes, the six face fluxes; what phase 2 reads
  // starts towards L2
  double g[6];
  if (on) {
    for (int t = 16 * r; t < NP; t += 16 * N2) {
      prefetch_l2(static_cast<const double*>(a.s.w) + ge + t);
      if constexpr (RK == kRkGeneral) prefetch_l2(a.s.q0 + ge + t);
    }
    const double* __restrict__ u = static_cast<const double*>(a.s.u);
    const double* __restrict__ v = static_cast<const double*>(a.s.v);
#pragma unroll
    for (int m = 0; m < N; m++) {
      const double qv = q[ge + r + m * N2];
      sX[zat + m * NS * N] = fix_product(qv, u[ge + r + m * N2]);
      sY[zat + m * NS * N] = fix_product(qv, v[ge + r + m * N2]);
    }
    unsigned nb[6];
    fix_neighbors(a.s.box, (unsigned)(eb + le), nb);
    // node of face f on this side and on the neighbour's
    const int x0 = i * N + j * N2, y0 = i + j * N2;
    const int nM[6] = {y0, x0 + (N - 1), y0 + (N - 1) * N, x0, r, r + (N - 1) * N2};
    const int nP[6] = {y0 + (N - 1) * N, x0, y0, x0 + (N - 1), r + (N - 1) * N2, r};
#pragma unroll
    for (int f = 0; f < 6; f++) {
      const long long gP = (long long)nb[f] * NP + nP[f];
      const double qP = q[gP], qM = q[ge + nM[f]];
      const long long fi = (eb + le) * NFT + f * N2 + r;
      double2 fc;
      if constexpr (FCIN) {
        fc = reinterpret_cast<const double2*>(a.s.fc_in)[fi];
      } else {
        const double* vel = static_cast<const double*>((f == 1 || f == 3)   ? a.s.u
                                                       : (f == 0 || f == 2) ? a.s.v
                                                                            : a.s.w);
        const double uM = vel[ge + nM[f]], uP = vel[gP];
        const double a2 = abs_ct(uP + uM);
        const double tw = (f == 1 || f == 2 || f == 5) ? 2.0 : -2.0;
        fc = make_double2(EO ? fma(tw, uP, -a2) : tw * (uP - uM), fma(tw, uM, -a2));
        if (a.s.fc_out) reinterpret_cast<double2*>(a.s.fc_out)[fi] = fc;
      }
      g[f] = EO ? fma(qP, fc.x, -(qM * fc.y)) : fma(qP, fc.x, (qP - qM) * fc.y);
    }
  }
  __syncthreads();
  if (on) {
    // lines along i (r = j + N k), faces -x (3) and +x (1)
    sEx[r] = fix_line_shared<P, EO, 0, 1>(a, r, sX + NS * r, g[3], g[1]);
    // lines along j (r = i + N k), faces -y (0) and +y (2)
    sEy[r] = fix_line_shared<P, EO, 1, NS>(a, r, sY + i + NS * N * j, g[0], g[2]);
  }
  // lines along k (r = i + N j), faces -z (4) and +z (5); the RK update
  double F[N];
  int32_t E = 0;
  if (on) {
    const double* __restrict__ w = static_cast<const double*>(a.s.w);
    FixScan<P, EO> scan;
#pragma unroll
    for (int m = 0; m < N; m++) {
      F[m] = fix_product(q[ge + r + m * N2], w[ge + r + m * N2]);
      scan.add(m, fix_value_exp(F[m]));
    }
    E = scan.scale(max(fix_face_exp(g[4]), fix_face_exp(g[5])), !EO && a.thin);
    E = fix_line_scale<N>(F, E, g[4], g[5]);
  }
  __syncthreads();
  if (on) {
    const double* __restrict__ q0 = a.s.q0;
    double* __restrict__ qout = a.s.q_out;
    const double c = a.c, ra = a.s.a, rb = a.s.b;
    const int Bz = a.ok && fix_in_range(E) ? fix_line_exp(E) : kFixDouble;
    const int rx = a.row[Args::row_of(i)], ry = a.row[Args::ROWS + Args::row_of(j)];
    const int64_t* iX = reinterpret_cast<const int64_t*>(sX) + zat;
    const int64_t* iY = reinterpret_cast<const int64_t*>(sY) + zat;
    auto emit = [&](int m, int64_t z) {
      const int64_t x = iX[m * NS * N], y = iY[m * NS * N];
      const int ex = sEx[j + N * m] + rx, ey = sEy[i + N * m] + ry;
      const int ez = Bz + a.row[2 * Args::ROWS + Args::row_of(m)];
      const double t = fix_node(x, ex, y, ey, z, ez);
      const long long n = ge + r + m * N2;
      if constexpr (RK == kRkTend)
        qout[n] = t;
      else if constexpr (RK == kRkFirst)
        qout[n] = fma(c, t, q[n]);
      else
        // the even-odd type adds b dt t to b q; the others keep the reference's
        // a q0 + b (q + dt t) (main.f90:69-73)
        qout[n] = EO ? rk_combine<RK>(c * t, q[n], q0[n], ra, rb)
                     : fma(ra, q0[n], rb * fma(c, t, q[n]));
    };
    if (Bz != kFixDouble) {
      fix_line<P, EO>(a.tab + 2 * a.TAB, a.lift(2, r), F, E, fix_align_face(g[4], E),
                      fix_align_face(g[5], E), emit);
    } else {
      double in[N], out[N];  // in: F itself stays in registers
#pragma unroll
      for (int m = 0; m < N; m++) in[m] = F[m];
      fix_line_fp64<P, EO>(&a.s, 2, r, in, 1, g[4], g[5], out);
#pragma unroll 1
      for (int m = 0; m < N; m++) emit(m, __double_as_longlong(out[m]));
    }
  }
}

template <int P, bool EO, int RK, bool FCIN>
int launch_stage_fix_kind(const FixStageArgs<P, EO>& a, cudaStream_t st) {
  // a small box takes blocks of a warp's elements, so that its blocks cover
  // the chip: 8^3 elements at p = 3 as 256 blocks of 32 threads, not 64 of 128
  constexpr int N2 = FixShape<P>::N2;
  const long long want = std::max(a.s.elem_count / (2 * 152), 1LL);
  const int threads = (int)std::min<long long>((want * N2 + 31) / 32 * 32, FixShape<P>::THREADS);
  const int epb = threads / N2;
  const long long nblk = (a.s.elem_count + epb - 1) / epb;
  if (nblk <= 0) return SDG_OK;
  if (nblk > 0x7fffffffLL) return fail(SDG_ERR_INVALID_ARG, "too many elements");
  // no more shared memory than the resident blocks take: the rest of the SM's
  // 256 KB is L1, from which a node's value is read again by the RK update and a
  // face value by the threads that share its sector (all of it as shared memory:
  // 55.0 against 58.4 GDOF-updates/s at p = 3, 64.0 against 68.2 at p = 7, 46.0
  // against 53.3 at p = 11)
  constexpr size_t smem = fix_smem<P>(FixShape<P>::EPB);
  SDG_TRY(set_kernel_smem((const void*)stage_fix_kernel<P, EO, RK, FCIN>, (int)smem,
                          carve_for(smem, fix_min_blocks<P>())));
  stage_fix_kernel<P, EO, RK, FCIN><<<(unsigned)nblk, threads, fix_smem<P>(epb), st>>>(a);
  SDG_CUDA_TRY(cudaGetLastError());
  return SDG_OK;
}

template <int P, bool EO>
void fix_fill(FixStageArgs<P, EO>& a, const StageArgs& s) {
  a.s = s;
  a.c = EO ? s.b * s.dt : s.dt;
  for (int t = 0; t < 3 * a.TAB; t++)
    a.tab[t] = fixlimb{s.fix->coef[2 * t], s.fix->coef[2 * t + 1]};
  for (int t = 0; t < 3 * a.ROWS; t++) a.row[t] = s.fix->row[t];
  a.ok = s.fix->ok;
  a.thin = s.fix->thin;
}

template <int P, bool EO>
int launch_stage_fix_impl(const StageArgs& s, cudaStream_t st) {
  FixStageArgs<P, EO> a;
  fix_fill<P, EO>(a, s);
  const bool in = s.fc_in != nullptr;
  switch (rk_kind(s)) {
    case kRkTend: return launch_stage_fix_kind<P, EO, kRkTend, false>(a, st);
    case kRkFirst:
      return in ? launch_stage_fix_kind<P, EO, kRkFirst, true>(a, st)
                : launch_stage_fix_kind<P, EO, kRkFirst, false>(a, st);
    default:
      return in ? launch_stage_fix_kind<P, EO, kRkGeneral, true>(a, st)
                : launch_stage_fix_kind<P, EO, kRkGeneral, false>(a, st);
  }
}

}  // namespace sdg
