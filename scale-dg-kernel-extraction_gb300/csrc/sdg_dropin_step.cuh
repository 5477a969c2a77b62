// The tendency and the SSP-RK3 stages for meshes given as the reference's
// arrays, with the line sums in fixed point (sdg_fix.cuh, sdg_stage_fix.cuh).
//
// One kernel serves advect3d_eq_cal_tend (mod_advect3d_eq.f90:41-85; MODE
// kRkTend) and the time loop of main.f90:51-80 (per stage update_halo,
// cal_tend and the RK update in one launch; the other MODEs).  What the
// caller's arrays decide, and how they are honoured:
//   * VMapM / VMapP (1-based flat DOF ids, halo slots for periodic
//     neighbours), normal_fn and Fscale: a tendency gathers q, u, v, w through
//     them, range-checked, and forms the flux as cal_elembnd_flux does
//     (mod_advect3d_eq.f90:116-140).  In the time loop step_face_kernel
//     resolves them once per call to the owned node each entry reads (the
//     value update_halo would have copied into the slot) and to the velocity
//     factors of the flux, which every stage of the loop shares (main.f90:58-67
//     passes the same u, v, w each time);
//   * Escale (per node, per direction): where an element's is one value per
//     direction over all its nodes (mesh_setup's affine elements,
//     mod_mesh.f90:147-149), its significand is folded into the element's copy
//     of the derivative coefficients and its exponent into the line's (the
//     faces aligned against it); in other elements a line's derivative and lift
//     sums become doubles and Escale is applied per node in between
//     (mod_advect3d_eq.f90:185-198).
//
// EO: coefficients of the even-odd pairs, for operators with the symmetries
// (type EVENODD); else rows of D1D (x) and D1D_tr (y, z) as given and every
// node's lift entries (GENERAL, OPT1).
//
// Measured on GB300 at about 7M DOF against the FP64 kernels this replaced
// (GDOF-updates/s): the time loop at p = 7 46.9 from 18.2 (EVENODD) and 39.7
// from 10.7 (OPT1), p = 3 43.8 / 38.8 from 19.1 / 10.7, p = 15 34.4 / 22.3 from
// 13.1 / 6.8; the per-stage calls 24.5 from 10.6 at p = 7.  A stage is bound by
// the latency of its gathers and loads (long-scoreboard stalls 6.5 of 17 cycles
// an instruction, 32 warps an SM); a tendency, which gathers 14 values a face
// node, by them alone.
#pragma once

#include "sdg_dropin_ops.cuh"
#include "sdg_stage_fix.cuh"

namespace sdg {

struct RefArgs {
  const double* q_in;   // state (the tendency's with halos)
  const double* q0;     // step-start state (stages 2 and 3)
  double* out;          // dqdt, or the stage result (may be q0 in the third)
  const double* u;      // caller's velocity
  const double* v;
  const double* w;
  const double* D;      // operators as given
  const double* Dt;
  const double* Lift;
  // tables (ref_tables_kernel): rows of coefficients times 2^-row, the rows'
  // exponents (kBadRow: out of range) and, behind them, which rows' lift has zeros
  // and the nodes' lift limbs (both not EO)
  const double* tab;
  const int* row;
  const int4* lift;
  // faces of a tendency
  const int* VMapM;
  const int* VMapP;
  const double* normal_fn;
  const double* Fscale;
  int* err;             // set to 1 on an out-of-range VMap entry
  long long NpNeA;      // valid 1-based indices are 1..NpNeA
  // faces of the time loop: the 0-based nodes qM and qP come from (-1: a map
  // entry was out of range), and the velocity factors.  Operators as given may
  // name halo slots beyond halo_src_map's, whose values q_halo (the caller's q)
  // holds through the call; *slots: some entry does (a select a face for all
  // meshes: p = 3 66.6 against 63.4 us a stage)
  const int2* res;
  const double* q_halo;
  const int* slots;
  const double2* fc;
  const double* Escale;
  // coefficients for the Escale of the mesh's first node (null: not built), and
  // in the time loop per element (Es_x, Es_y, Es_z, 1) when its Escale is one
  // value per direction, (.., 0) otherwise (null: read Escale)
  const fixlimb* shared;
  const double4* esu;
  int Ne;
  double a, b, dt;      // q_out = a q0 + b (q + dt dqdt)
};

template <int P, bool EO>
struct RefShape {
  static constexpr int N = P + 1;
  static constexpr int TAB = EO ? EoShape<P>::TE : N * N;
  static constexpr int ROWS = EO ? EoShape<P>::HR : N;
  // bytes of the tables: lift limbs, coefficients, rows (16-byte aligned base)
  static constexpr size_t LIFT = EO ? 0 : sizeof(int4) * 3 * N * N * N;
  static constexpr size_t LEAST =
      LIFT + sizeof(double) * 3 * TAB + sizeof(int) * (EO ? 3 : 6) * ROWS;
  // with the coefficients for the first node's Escale
  static constexpr size_t SHARED = (LEAST + 7) / 8 * 8;
  static constexpr size_t BYTES = SHARED + sizeof(fixlimb) * 3 * TAB;
  // a table entry's row, and whether Escale applies to it
  static __host__ __device__ constexpr int row_of_entry(int w) {
    using Sh = EoShape<P>;
    constexpr int H1 = Sh::H;
    return !EO                 ? w / N
           : w < Sh::OFF_O     ? w / H1
           : w < Sh::OFF_DM    ? (w - Sh::OFF_O) / H1
           : w < Sh::OFF_A     ? w - Sh::OFF_DM
           : w < Sh::OFF_B     ? w - Sh::OFF_A
                               : w - Sh::OFF_B;
  }
  static __host__ __device__ constexpr bool derivative(int w) { return !EO || w < EoShape<P>::OFF_A; }
  static __host__ __device__ constexpr int row_of(int m) {
    return EO ? (m < P - m ? m : P - m) : m;
  }
};

__device__ __forceinline__ double ref_pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }

// Escale of a direction: its exponent x (Es = sig 2^x, sig in [0.5, 1)), and
// sig 2^60.
__device__ __forceinline__ int ref_escale_exp(double es) {
  return (int)((unsigned)__double2hiint(es) >> 20 & 0x7FFu) - 1022;
}
__device__ __forceinline__ int64_t ref_escale_sig(double es) {
  return fix_unit(
      __hiloint2double(__double2hiint(es) - (ref_escale_exp(es) << 20), __double2loint(es)));
}
// The exponent field of a line's two faces, less that of its Escale; past the
// fields of a double (an Escale below a half, faces infinite, NaN or huge) the
// largest, which no line takes in fixed point.
__device__ __forceinline__ int32_t ref_face_exp(double gm, double gp, int xe) {
  return min((max(fix_value_exp(gm), fix_value_exp(gp)) >> 20) - xe, 2047) << 20;
}
// The limbs of a table entry (its minus sign is dqdt's), a derivative entry
// with the significand of Escale.
__device__ __forceinline__ fixlimb ref_coef(double entry, bool derivative, int64_t sig) {
  const int64_t c = fix_unit(entry);
  return fix_coef(derivative ? -fix_times(c, sig) : -c);
}

// The three directions' unscaled even-odd tables from D1D and Lift_mat (the
// lift column of a face from its tangential node (0, 0)) with their row scales,
// and (shared not null) the coefficients for the Escale of the mesh's first
// node, one block; it checks the symmetries the factorisation needs -- D1D
// centro-antisymmetric, D1D_tr its transpose, each face's lift constant over
// the tangential nodes, the + face's column the mirror of the - face's, all to
// 1e-13 of the largest entry -- and sets *err = 2 when one fails.
template <int P>
__global__ void __launch_bounds__(256) ref_tables_eo_kernel(const double* __restrict__ D,
                                                            const double* __restrict__ Dt,
                                                            const double* __restrict__ L,
                                                            const double* __restrict__ Es,
                                                            long long NpNe, double* tab, int* row,
                                                            fixlimb* shared, int* err) {
  using O = Ord<P>;
  using Sh = EoShape<P>;
  using Rs = RefShape<P, true>;
  constexpr int NQ = O::NQ, NQ2 = O::NQ2, NP = O::NP, TE = Sh::TE, N = Sh::N, H = Sh::H;
  __shared__ unsigned long long smax[2];
  __shared__ double sT[3 * TE];
  __shared__ int sRow[3 * Sh::HR];
  auto Dv = [&](int i, int l) { return D[i + l * N]; };  // D1D(i,l), column-major
  auto Ds = [&](int i, int l) { return 0.5 * (Dv(i, l) - Dv(N - 1 - i, N - 1 - l)); };
  auto node = [](int ax, int m, int t1, int t2) {
    return (ax == 0) ? m + NQ * t1 + NQ2 * t2 : (ax == 1) ? t1 + NQ * m + NQ2 * t2
                                                           : t1 + NQ * t2 + NQ2 * m;
  };
  auto col = [&](int ax, int side, int m) {
    const int f = (ax == 0) ? (side ? 1 : 3) : (ax == 1) ? (side ? 2 : 0) : (side ? 5 : 4);
    return L[node(ax, m, 0, 0) + (long long)f * NP];
  };
  auto lam = [&](int ax, int m) { return 0.5 * (col(ax, 0, m) + col(ax, 1, N - 1 - m)); };
  for (int t = threadIdx.x; t < 3 * TE; t += blockDim.x) {
    const int ax = t / TE, w = t - ax * TE;
    const int i = Rs::row_of_entry(w);
    double v;
    if (w < Sh::OFF_O) {
      const int l = w - i * H;
      v = 0.5 * (Ds(i, l) + Ds(i, N - 1 - l));
    } else if (w < Sh::OFF_DM) {
      const int l = (w - Sh::OFF_O) - i * H;
      v = 0.5 * (Ds(i, l) - Ds(i, N - 1 - l));
    } else if (w < Sh::OFF_A) {
      v = Ds(i, H);
    } else if (w < Sh::OFF_B) {
      v = 0.5 * (lam(ax, i) + lam(ax, N - 1 - i));
    } else {
      v = 0.5 * (lam(ax, i) - lam(ax, N - 1 - i));
    }
    sT[t] = v;
  }
  if (threadIdx.x == 0) smax[0] = smax[1] = 0ull;
  __syncthreads();
  for (int t = threadIdx.x; t < 3 * Sh::HR; t += blockDim.x) {
    const double* T = sT + (t / Sh::HR) * TE;
    const int i = t % Sh::HR;
    // what the row's two outputs can reach on values and faces below one
    auto pair = [&](int e, int o) {
      // (0 * x keeps a NaN that fmax would drop)
      return 2.0 * fmax(i < H ? fabs(T[e]) : 0.0, fabs(T[o])) + 0.0 * (T[e] + T[o]);
    };
    double most = pair(i < H ? Sh::OFF_B + i : Sh::OFF_A + i, Sh::OFF_A + i);
    for (int l = 0; l < H; l++) most += pair(Sh::OFF_E + i * H + l, Sh::OFF_O + i * H + l);
    if (i < H && Sh::ODD) most += fabs(T[Sh::OFF_DM + i]);
    row[t] = sRow[t] = fix_row_exp(most);
  }
  unsigned long long mD = 0, mL = 0;
  for (int t = threadIdx.x; t < NQ2; t += blockDim.x)
    mD = max(mD, (unsigned long long)__double_as_longlong(fabs(D[t])));
  for (int t = threadIdx.x; t < 6 * NP; t += blockDim.x)
    mL = max(mL, (unsigned long long)__double_as_longlong(fabs(L[t])));
  atomicMax(&smax[0], mD);
  atomicMax(&smax[1], mL);
  __syncthreads();
  for (int t = threadIdx.x; t < 3 * TE; t += blockDim.x) {
    const int w = t % TE, k = sRow[t / TE * Sh::HR + Rs::row_of_entry(w)];
    const double c = k == kBadRow ? sT[t] : sT[t] * ref_pow2(-k);
    tab[t] = c;
    if (shared)
      shared[t] = ref_coef(c, Rs::derivative(w), ref_escale_sig(Es[(t / TE) * NpNe]));
  }
  const double tD = 1e-13 * __longlong_as_double((long long)smax[0]);
  const double tL = 1e-13 * __longlong_as_double((long long)smax[1]);
  bool bad = false;
  for (int t = threadIdx.x; t < NQ2; t += blockDim.x) {
    const int i = t % N, l = t / N;
    bad |= fabs(Dv(i, l) + Dv(N - 1 - i, N - 1 - l)) > tD;
    bad |= fabs(Dt[l + i * N] - Dv(i, l)) > tD;
  }
  for (int t = threadIdx.x; t < 6 * NP; t += blockDim.x) {
    const int f = t / NP, n = t - f * NP;
    const int ax = (f == 1 || f == 3) ? 0 : (f == 0 || f == 2) ? 1 : 2;
    const int side = (f == 1 || f == 2 || f == 5) ? 1 : 0;
    const int c[3] = {n % NQ, (n / NQ) % NQ, n / NQ2};
    bad |= fabs(L[t] - col(ax, side, c[ax])) > tL;
    if (n < N && ax == 0 && side == 0)
      for (int x = 0; x < 3; x++) bad |= fabs(col(x, 0, n) - col(x, 1, N - 1 - n)) > tL;
  }
  if (bad) atomicExch(err, 2);
}

// Operators as given: block (d, i) forms row i of direction d -- its scale over
// the derivative entries and all its nodes' lift entries (kBadRow where an entry is
// below 2^-10 of those: the reference's smallest is 2^-9.6 at p = 15), the scaled
// derivative entries (D1D for x, D1D_tr for y and z), the nodes' lift limbs
// (-, + face) and the coefficients for the Escale of the mesh's first node.
template <int P>
__global__ void __launch_bounds__(256) ref_tables_kernel(const double* __restrict__ D,
                                                         const double* __restrict__ Dt,
                                                         const double* __restrict__ L,
                                                         const double* __restrict__ Es,
                                                         long long NpNe, double* tab, int* row,
                                                         int4* lift, fixlimb* shared) {
  constexpr int N = P + 1, N2 = N * N, NP = N * N2;
  const int d = blockIdx.x / N, i = blockIdx.x - d * N, r = threadIdx.x;
  const int fm = d == 0 ? 3 : d == 1 ? 0 : 4, fp = d == 0 ? 1 : d == 1 ? 2 : 5;
  __shared__ unsigned long long smax;
  if (r == 0) smax = 0ull;
  __syncthreads();
  const int n = d == 0 ? i + N * r : d == 1 ? r % N + N * i + N2 * (r / N) : r + N2 * i;
  double m = 0.0, p = 0.0;
  if (r < N2) {
    m = L[n + fm * NP];
    p = L[n + fp * NP];
    atomicMax(&smax, (unsigned long long)__double_as_longlong(fabs(m) + fabs(p)));
  }
  __syncthreads();
  auto Dv = [&](int l) { return d == 0 ? D[i + l * N] : Dt[l + i * N]; };
  double sum = __longlong_as_double((long long)smax);
  for (int l = 0; l < N; l++) sum += fabs(Dv(l));
  // entries too small for the row's scale: in FP64 (lift entries may be zero)
  const double least = sum * (1.0 / 1024.0);
  bool small = r < N && r != i && fabs(Dv(r)) < least;
  small |= r < N2 && ((m != 0.0 && fabs(m) < least) || (p != 0.0 && fabs(p) < least));
  const int k = __syncthreads_or(small) ? kBadRow : fix_row_exp(sum);
  const int thin = __syncthreads_or(r < N2 && (m == 0.0 || p == 0.0));
  if (r == 0) {
    row[blockIdx.x] = k;
    row[3 * N + blockIdx.x] = thin;
  }
  const double scale = k == kBadRow ? 1.0 : ref_pow2(-k);
  if (r < N) {
    const double c = Dv(r) * scale;
    tab[blockIdx.x * N + r] = c;
    if (shared) shared[blockIdx.x * N + r] = ref_coef(c, true, ref_escale_sig(Es[d * NpNe]));
  }
  if (r < N2) {
    const fixlimb a = fix_coef(-fix_unit(m * scale)), b = fix_coef(-fix_unit(p * scale));
    lift[(long long)blockIdx.x * N2 + r] = make_int4(a.hi, a.lo, b.hi, b.lo);
  }
}

// A line in FP64 with the caller's Escale per node (Es, stride es): F its
// fluxes (stride fs), out[m] = -(Es(m) (D F)(m) + lift(m)).
template <int P, bool EO>
__device__ __noinline__ void ref_line_fp64(const RefArgs* a, int ax, int r, const double* F, int fs,
                                           double gm, double gp, const double* __restrict__ Es,
                                           int es, double* out) {
  using Sh = EoShape<P>;
  constexpr int N = Sh::N, H = Sh::H, N2 = N * N, NP = N * N2;
  if constexpr (!EO) {
    const int fm = ax == 0 ? 3 : ax == 1 ? 0 : 4, fp = ax == 0 ? 1 : ax == 1 ? 2 : 5;
    double f[N];
#pragma unroll
    for (int l = 0; l < N; l++) f[l] = F[l * fs];
    const double* __restrict__ D = ax == 0 ? a->D : a->Dt;
#pragma unroll 1
    for (int i = 0; i < N; i++) {
      double s = 0.0;
#pragma unroll
      for (int l = 0; l < N; l++) s = fma(ax == 0 ? D[i + l * N] : D[l + i * N], f[l], s);
      const int n = ax == 0 ? i + N * r : ax == 1 ? r % N + N * i + N2 * (r / N) : r + N2 * i;
      out[i] = -fma(Es[i * es], s, fma(a->Lift[n + fm * NP], gm, a->Lift[n + fp * NP] * gp));
    }
    return;
  }
  double s[H], d[H];
#pragma unroll
  for (int l = 0; l < H; l++) {
    const double f1 = F[l * fs], f2 = F[(N - 1 - l) * fs];
    s[l] = f1 + f2;
    d[l] = f1 - f2;
  }
  const double fmid = Sh::ODD ? F[H * fs] : 0.0;
  const double gs = gm + gp, gd = gm - gp;
  const double* __restrict__ T = a->tab + ax * Sh::TE;
#pragma unroll 1
  for (int i = 0; i < Sh::HR; i++) {
    const int k = a->row[ax * Sh::HR + i];
    const double c = k == kBadRow ? -1.0 : -ref_pow2(k);
    double o = T[Sh::OFF_O + i * H] * d[0];
#pragma unroll
    for (int l = 1; l < H; l++) o = fma(T[Sh::OFF_O + i * H + l], d[l], o);
    const double ag = c * (T[Sh::OFF_A + i] * gs);
    if (i == H) {
      out[H] = fma(c * Es[H * es], o, ag);
      continue;
    }
    double e = T[Sh::OFF_E + i * H] * s[0];
#pragma unroll
    for (int l = 1; l < H; l++) e = fma(T[Sh::OFF_E + i * H + l], s[l], e);
    if (Sh::ODD != 0) e = fma(T[Sh::OFF_DM + i], fmid, e);
    const double bg = c * (T[Sh::OFF_B + i] * gd);
    out[i] = fma(c * Es[i * es], o + e, ag + bg);
    out[N - 1 - i] = fma(c * Es[(N - 1 - i) * es], o - e, ag - bg);
  }
}

// A line's derivative and lift sums apart, each in fixed point on a scale of its
// own: im / ip the faces' fluxes as integers, the rest as fix_line; emit(m, d, l).
template <int P, bool EO, typename Emit>
__device__ __forceinline__ void ref_line_parts(const fixlimb* T, const int4* __restrict__ lift,
                                               const double* F, int32_t E, int64_t im, int64_t ip,
                                               Emit&& emit) {
  using Sh = EoShape<P>;
  constexpr int N = Sh::N, H = Sh::H;
  fixacc l;
  if constexpr (!EO) {
    const fixlimb lm = fix_split(im), lp = fix_split(ip);
    fixlimb f[N];
#pragma unroll
    for (int k = 0; k < N; k++) f[k] = fix_split(fix_align(F[k], E));
#pragma unroll 1
    for (int i = 0; i < N; i++) {
      const int4 c = lift[i * N * N];
      fix_mul(l, fixlimb{c.x, c.y}, lm);
      fix_fma(l, fixlimb{c.z, c.w}, lp);
      fixacc d;
      fix_mul(d, T[i * N], f[0]);
#pragma unroll
      for (int k = 1; k < N; k++) fix_fma(d, T[i * N + k], f[k]);
      emit(i, fix_sum(d), fix_sum(l));
    }
    return;
  }
  fixlimb s[H], d[H], fm{0, 0};
#pragma unroll
  for (int k = 0; k < H; k++) {
    const int64_t f1 = fix_align(F[k], E), f2 = fix_align(F[N - 1 - k], E);
    s[k] = fix_split(f1 + f2);
    d[k] = fix_split(f1 - f2);
  }
  if constexpr (Sh::ODD != 0) fm = fix_split(fix_align(F[H], E));
  const fixlimb gs = fix_split(im + ip), gd = fix_split(im - ip);
#pragma unroll 1
  for (int i = 0; i < Sh::HR; i++) {
    fix_mul(l, T[Sh::OFF_A + i], gs);
    const int64_t ol = fix_sum(l);
    fixacc o, e;
    fix_mul(o, T[Sh::OFF_O + i * H], d[0]);
#pragma unroll
    for (int k = 1; k < H; k++) fix_fma(o, T[Sh::OFF_O + i * H + k], d[k]);
    const int64_t od = fix_sum(o);
    if (i == H) {
      emit(i, od, ol);
      continue;
    }
    fix_mul(e, T[Sh::OFF_E + i * H], s[0]);
#pragma unroll
    for (int k = 1; k < H; k++) fix_fma(e, T[Sh::OFF_E + i * H + k], s[k]);
    if constexpr (Sh::ODD != 0) fix_fma(e, T[Sh::OFF_DM + i], fm);
    const int64_t ed = fix_sum(e);
    fix_mul(l, T[Sh::OFF_B + i], gd);
    const int64_t el = fix_sum(l);
    emit(i, od + ed, ol + el);
    emit(N - 1 - i, od - ed, ol - el);
  }
}

// A line the folded coefficients do not take: F its fluxes (stride fs), Es its
// nodes' Escale (stride es), out[m] = -(Es(m) (D F)(m) + lift(m)).  With T (an
// element whose Escale varies: its coefficients without Escale) the sums are
// formed in fixed point where F and the faces allow.
template <int P, bool EO>
__device__ __noinline__ void ref_line_nodes(const RefArgs* a, const fixlimb* T, int ax, int r,
                                            const double* F, int fs, double gm, double gp,
                                            const double* __restrict__ Es, int es, double* out) {
  constexpr int N = P + 1;
  using Rs = RefShape<P, EO>;
  double f[N];
  FixScan<P, EO> scan;
#pragma unroll
  for (int l = 0; l < N; l++) {
    f[l] = F[l * fs];
    scan.add(l, fix_value_exp(f[l]));
  }
  // (the faces have a scale of their own)
  const int32_t E = fix_line_scale<N>(f, scan.scale(0, false), 0.0, 0.0);
  int32_t Eg = max(fix_value_exp(gm), fix_value_exp(gp));
  if (gm == 0.0 && gp == 0.0) Eg = kFixZeros;
  if (T == nullptr || !fix_in_range(E) || !fix_in_range(Eg)) {
    ref_line_fp64<P, EO>(a, ax, r, F, fs, gm, gp, Es, es, out);
    return;
  }
  const int B = fix_line_exp(E) - 61, Bg = fix_line_exp(Eg) - 61;
  ref_line_parts<P, EO>(T, EO ? nullptr : a->lift + ax * N * N * N + r, f, E,
                        fix_align_signed(gm, Eg), fix_align_signed(gp, Eg),
                        [&](int m, int64_t d, int64_t l) {
                          const int k = a->row[ax * Rs::ROWS + Rs::row_of(m)];
                          out[m] = fma(Es[m * es], fix_to_double(d, B + k), fix_to_double(l, Bg + k));
                        });
}

// u . n with the components whose normal entry is a zero left out: the same
// value, as long as those components are finite, for two of three FP64
// operations a side on the axis-aligned normals of mesh_setup.
__device__ __forceinline__ double ref_normal_velocity(double u, double v, double w, double n1,
                                                      double n2, double n3, int axis) {
  if (axis == 0) return u * n1;
  if (axis == 1) return v * n2;
  if (axis == 2) return w * n3;
  return u * n1 + v * n2 + w * n3;
}

// Face flux of a tendency at face node m with map entries at
// (cal_elembnd_flux, mod_advect3d_eq.f90:116-140).
__device__ __forceinline__ double ref_flux(const RefArgs& a, long long m, long long NT, int2 at) {
  // 1..NpNeA, which a map entry's 31 bits bound as well
  const unsigned iM = (unsigned)at.x - 1u, iP = (unsigned)at.y - 1u;
  const unsigned lim = a.NpNeA < 0x7fffffffLL ? (unsigned)a.NpNeA : 0x7fffffffu;
  if (iM >= lim || iP >= lim) {
    atomicExch(a.err, 1);
    return 0.0;
  }
  const double n1 = a.normal_fn[m], n2 = a.normal_fn[m + NT], n3 = a.normal_fn[m + 2 * NT];
  const double qM = a.q_in[iM], qP = a.q_in[iP];
  const double uM = a.u[iM], vM = a.v[iM], wM = a.w[iM], uP = a.u[iP], vP = a.v[iP],
               wP = a.w[iP];
  auto zero = [](double x) { return (__double2hiint(x) << 1 | __double2loint(x)) == 0; };
  auto exp = [](double x) { return (unsigned)__double2hiint(x) & 0x7FF00000u; };
  const bool z1 = zero(n1), z2 = zero(n2), z3 = zero(n3);
  const unsigned top = max(max(max(exp(uM), exp(vM)), max(exp(wM), exp(uP))),
                           max(exp(vP), exp(wP)));
  const int axis = top == 0x7FF00000u ? 3 : z2 && z3 ? 0 : z1 && z3 ? 1 : z1 && z2 ? 2 : 3;
  const double VelM = ref_normal_velocity(uM, vM, wM, n1, n2, n3, axis);
  const double VelP = ref_normal_velocity(uP, vP, wP, n1, n2, n3, axis);
  const double alpha = 0.5 * fabs(VelP + VelM);
  return (0.5 * a.Fscale[m]) * ((qP * VelP - qM * VelM) - alpha * (qP - qM));
}

template <int P, bool EO>
__host__ __device__ constexpr size_t ref_smem(int epb) {
  return sizeof(double) * 2 * epb * FixShape<P>::EW +
         sizeof(fixlimb) * 3 * epb * RefShape<P, EO>::TAB +
         sizeof(short) * 2 * epb * FixShape<P>::N2;
}

// The line of direction AX held in shared memory with stride S, its results
// over it; returns its exponent.  T: the element's coefficients of the
// direction, with Escale folded in but for its exponent xe (ok), without it
// (curved) or not usable (neither).
template <int P, bool EO, int AX, int S, int ES>
__device__ __forceinline__ int ref_line_shared(const RefArgs& a, const fixlimb* T, int xe, bool ok,
                                               bool curved, bool thin, int r, double* line, double gm, double gp,
                                               const double* Es) {
  constexpr int N = P + 1;
  double F[N];
  FixScan<P, EO> scan;
#pragma unroll
  for (int l = 0; l < N; l++) {
    F[l] = line[l * S];
    scan.add(l, fix_value_exp(F[l]));
  }
  const int32_t E = scan.scale(ref_face_exp(gm, gp, xe), thin);
  if (ok && fix_in_range(E)) {
    int64_t* out = reinterpret_cast<int64_t*>(line);
    const int32_t Ef = E + (xe << 20);
    fix_line<P, EO>(T, EO ? nullptr : a.lift + AX * N * N * N + r, F, E, fix_align_signed(gm, Ef),
                    fix_align_signed(gp, Ef), [&](int m, int64_t v) { out[m * S] = v; });
    return fix_line_exp(E) + xe;
  }
  // zeros (fix_product's are +0, as doubles too) are their own results
  if ((ok || curved) && fix_line_scale<N>(F, E, gm, gp) == kFixZeros)
    return fix_line_exp(kFixZeros);
  double out[N];
  ref_line_nodes<P, EO>(&a, curved ? T : nullptr, AX, r, line, S, gm, gp, Es, ES, out);
  for (int m = 0; m < N; m++) line[m * S] = out[m];
  return kFixDouble;
}

template <int P, bool EO>
__host__ __device__ constexpr int ref_min_blocks() {
  return P >= 12 ? 3 : 1024 / FixShape<P>::THREADS;
}

// MODE kRkTend: dqdt of elements [blockIdx.x*epb, ...); kRkFirst, kRkGeneral:
// one stage of the time loop.  Thread layout as stage_fix_kernel.
template <int P, bool EO, int MODE>
__global__ void __launch_bounds__(FixShape<P>::THREADS, ref_min_blocks<P, EO>())
    step_ref_kernel(const __grid_constant__ RefArgs a) {
  using Sh = FixShape<P>;
  using Rs = RefShape<P, EO>;
  constexpr int N = Sh::N, N2 = Sh::N2, NP = N * N2, NFT = 6 * N2, NS = Sh::NS, EW = Sh::EW,
                TAB = Rs::TAB, ROWS = Rs::ROWS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // elements whose Escale the coefficients do not take (1), rows out of range (2),
  // a lift with zeros (4)
  __shared__ int sMix[FixShape<P>::EPB];
  const int epb = blockDim.x / N2;
  const long long eb = (long long)blockIdx.x * epb;
  const long long left = (long long)a.Ne - eb;
  const int nloc = (int)(left < epb ? left : epb);
  const int le = threadIdx.x / N2, r = threadIdx.x - le * N2;
  const bool on = le < nloc;
  const int i = r % N, j = r / N;
  double* sX = reinterpret_cast<double*>(smem_raw) + le * EW;
  double* sY = sX + epb * EW;
  fixlimb* sT0 = reinterpret_cast<fixlimb*>(reinterpret_cast<double*>(smem_raw) + 2 * epb * EW);
  fixlimb* sT = sT0 + le * 3 * TAB;
  short* sEx = reinterpret_cast<short*>(sT0 + 3 * epb * TAB) + le * N2;
  short* sEy = sEx + epb * N2;
  const long long e = eb + le, ge = e * NP, NpNe = (long long)NP * a.Ne;
  const double* __restrict__ q = a.q_in;
  const double* __restrict__ Es = a.Escale;
  const int zat = i + NS * j;

  if (threadIdx.x < nloc) sMix[threadIdx.x] = 0;
  __syncthreads();
  // 0: the z line's x and y fluxes, the element's coefficients, the face fluxes
  double g[6];
  int xe[3] = {0, 0, 0};
  bool mix = false;
  if (on) {
    // the gathers wait for these: first
    const bool slots = !EO && MODE != kRkTend && *a.slots != 0;
    int2 at[6];
    const long long NT = (long long)NFT * a.Ne;
#pragma unroll
    for (int f = 0; f < 6; f++) {
      const long long m = e * NFT + f * N2 + r;
      at[f] = MODE == kRkTend ? make_int2(a.VMapM[m], a.VMapP[m]) : a.res[m];
    }
    for (int t = 16 * r; t < NP; t += 16 * N2) {
      prefetch_l2(a.w + ge + t);
      if constexpr (MODE == kRkGeneral) prefetch_l2(a.q0 + ge + t);
    }
    double es[3];
    if (MODE == kRkTend || a.esu == nullptr) {
#pragma unroll
      for (int d = 0; d < 3; d++) {
        es[d] = Es[ge + d * NpNe];
#pragma unroll
        for (int m = 0; m < N; m++)
          mix |= __double_as_longlong(Es[ge + r + m * N2 + d * NpNe]) != __double_as_longlong(es[d]);
      }
    } else {
      const double4 x = a.esu[e];
      es[0] = x.x;
      es[1] = x.y;
      es[2] = x.z;
      mix = __double2hiint(x.w) == 0;
    }
    bool same = a.shared != nullptr;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      xe[d] = ref_escale_exp(es[d]);
      mix |= xe[d] < -150 || xe[d] > 150;
      same = same && __double_as_longlong(es[d]) == __double_as_longlong(Es[d * NpNe]);
    }
    // a row's exponent with Escale's: with a line's, whose results have to lie in
    // the normal range, at most the 900 of the box solver
    bool bad = false;
    for (int t = r; t < 3 * ROWS; t += N2) {
      const int k = a.row[t], x = k + (t < ROWS ? xe[0] : t < 2 * ROWS ? xe[1] : xe[2]);
      mix |= x < -200 || x > 200;
      bad |= k == kBadRow;
      if (!EO && a.row[3 * ROWS + t] != 0) atomicOr(&sMix[le], 4);
    }
    if (mix) atomicOr(&sMix[le], bad ? 3 : 1);
#pragma unroll
    for (int m = 0; m < N; m++) {
      const double qv = q[ge + r + m * N2];
      sX[zat + m * NS * N] = fix_product(qv, a.u[ge + r + m * N2]);
      sY[zat + m * NS * N] = fix_product(qv, a.v[ge + r + m * N2]);
    }
    if (same) {
      for (int t = r; t < 3 * TAB; t += N2) sT[t] = a.shared[t];
    } else {
      for (int t = r; t < 3 * TAB; t += N2) {
        const int d = t / TAB, w = t - d * TAB;
        sT[t] = ref_coef(a.tab[t], Rs::derivative(w),
                         ref_escale_sig(d == 0 ? es[0] : d == 1 ? es[1] : es[2]));
      }
    }
    if constexpr (MODE == kRkTend) {
#pragma unroll
      for (int f = 0; f < 6; f++) g[f] = ref_flux(a, e * NFT + f * N2 + r, NT, at[f]);
    } else if (EO || !slots) {
#pragma unroll
      for (int f = 0; f < 6; f++) {
        const double2 fc = a.fc[e * NFT + f * N2 + r];
        g[f] = 0.0;
        if (at[f].x >= 0) {
          const double qP = q[at[f].y], qM = q[at[f].x];
          g[f] = EO ? fma(qP, fc.x, -(qM * fc.y)) : fma(qP, fc.x, (qP - qM) * fc.y);
        }
      }
    } else {
#pragma unroll
      for (int f = 0; f < 6; f++) {
        const double2 fc = a.fc[e * NFT + f * N2 + r];
        auto value = [&](int n) { return (n < (int)NpNe ? q : a.q_halo)[n]; };
        g[f] = 0.0;
        if (at[f].x >= 0) {
          const double qP = value(at[f].y), qM = value(at[f].x);
          g[f] = fma(qP, fc.x, (qP - qM) * fc.y);
        }
      }
    }
  }
  if (__syncthreads_or(mix)) {
    if (on && (sMix[le] & 3) == 1)
      for (int t = r; t < 3 * TAB; t += N2) sT[t] = fix_coef(-fix_unit(a.tab[t]));
    __syncthreads();
  }
  const int cls = on ? sMix[le] : 0;
  const bool ok = (cls & 3) == 0, curved = (cls & 3) == 1, thin = !EO && cls >= 4;
  if (on) {
    // lines along i (r = j + N k), faces -x (3) and +x (1); along j (r = i + N k),
    // faces -y (0) and +y (2)
    sEx[r] = ref_line_shared<P, EO, 0, 1, 1>(a, sT, xe[0], ok, curved, thin, r, sX + NS * r, g[3], g[1],
                                             Es + ge + N * r);
    sEy[r] = ref_line_shared<P, EO, 1, NS, N>(a, sT + TAB, xe[1], ok, curved, thin, r, sY + i + NS * N * j,
                                              g[0], g[2], Es + NpNe + ge + i + j * N2);
  }
  // lines along k (r = i + N j), faces -z (4) and +z (5); the node's result
  double F[N];
  int32_t E = 0;
  if (on) {
    FixScan<P, EO> scan;
#pragma unroll
    for (int m = 0; m < N; m++) {
      F[m] = fix_product(q[ge + r + m * N2], a.w[ge + r + m * N2]);
      scan.add(m, fix_value_exp(F[m]));
    }
    E = fix_line_scale<N>(F, scan.scale(ref_face_exp(g[4], g[5], xe[2]), thin), g[4], g[5]);
  }
  __syncthreads();
  if (on) {
    const double dt = a.dt, ra = a.a, rb = a.b;
    const bool zok = ok && fix_in_range(E);
    const int Bz = zok ? fix_line_exp(E) + xe[2] : kFixDouble;
    const int rx = a.row[Rs::row_of(i)] - 61, ry = a.row[ROWS + Rs::row_of(j)] - 61;
    const int64_t* iX = reinterpret_cast<const int64_t*>(sX) + zat;
    const int64_t* iY = reinterpret_cast<const int64_t*>(sY) + zat;
    // a line in FP64 has doubles whatever its row (a bad row's exponent is large)
    auto add = [](int line, int row) { return line == kFixDouble ? kFixDouble : line + row; };
    auto finish = [&](int m, double t) {
      const long long n = ge + r + m * N2;
      if constexpr (MODE == kRkTend)
        a.out[n] = t;
      else if constexpr (MODE == kRkFirst)
        a.out[n] = fma(dt, t, q[n]);
      else
        // q0 is read before out is written at the same node, by this thread
        // only, so the third stage may write the result over q0.  The even-odd
        // type adds b dt t to b q, the others keep the reference's order
        // (main.f90:69-73)
        a.out[n] = EO ? fma(ra, a.q0[n], fma(rb, q[n], (rb * dt) * t))
                      : fma(ra, a.q0[n], rb * fma(dt, t, q[n]));
    };
    auto emit = [&](int m, int64_t z) {
      finish(m, fix_node(iX[m * NS * N], add(sEx[j + N * m], rx), iY[m * NS * N],
                         add(sEy[i + N * m], ry), z,
                         add(Bz, a.row[2 * ROWS + Rs::row_of(m)] - 61)));
    };
    if (zok) {
      const int32_t Ef = E + (xe[2] << 20);
      fix_line<P, EO>(sT + 2 * TAB, EO ? nullptr : a.lift + 2 * NP + r, F, E,
                      fix_align_signed(g[4], Ef), fix_align_signed(g[5], Ef), emit);
    } else {
      double in[N], out[N];  // in: F itself stays in registers
#pragma unroll
      for (int m = 0; m < N; m++) in[m] = F[m];
      ref_line_nodes<P, EO>(&a, curved ? sT + 2 * TAB : nullptr, 2, r, in, 1, g[4], g[5],
                            Es + 2 * NpNe + ge + r, N2, out);
      if (curved) {  // all lines are doubles
#pragma unroll 1
        for (int m = 0; m < N; m++)
          finish(m, (sX[zat + m * NS * N] + sY[zat + m * NS * N]) + out[m]);
      } else {
#pragma unroll 1
        for (int m = 0; m < N; m++) emit(m, __double_as_longlong(out[m]));
      }
    }
  }
}

template <int P, bool EO, int MODE>
int launch_ref_mode(const RefArgs& a, cudaStream_t st) {
  // blocks of fewer elements on small meshes, as launch_stage_fix_kind
  constexpr int N2 = FixShape<P>::N2;
  const long long want = std::max(a.Ne / (2 * 152), 1);
  const int threads = (int)std::min<long long>((want * N2 + 31) / 32 * 32, FixShape<P>::THREADS);
  const int epb = threads / N2;
  const long long nblk = ((long long)a.Ne + epb - 1) / epb;
  if (nblk == 0) return SDG_OK;
  // carveout: the gathers of the faces live on L1 hits, as in launch_stage_fix_kind
  // (loop, even-odd, 24^3: p = 2 34.5 from 26.3, p = 4 42.1 from 33.2, p = 7 46.9
  // from 42.0 GDOF-updates/s; level at p = 15, whose blocks need all of it)
  constexpr size_t smem = ref_smem<P, EO>(FixShape<P>::EPB);
  SDG_TRY(set_kernel_smem((const void*)step_ref_kernel<P, EO, MODE>, (int)smem,
                          carve_for(smem, ref_min_blocks<P, EO>())));
  step_ref_kernel<P, EO, MODE><<<(unsigned)nblk, threads, ref_smem<P, EO>(epb), st>>>(a);
  SDG_CUDA_TRY(cudaGetLastError());
  return SDG_OK;
}

// Points a's tables into `base` (16-byte aligned, `bytes` of at least
// RefShape::LEAST) and builds them there.
template <int P, bool EO>
int launch_ref_tables(RefArgs& a, void* base, size_t bytes, cudaStream_t st) {
  using Rs = RefShape<P, EO>;
  char* p = static_cast<char*>(base);
  int4* lift = reinterpret_cast<int4*>(p);
  double* tab = reinterpret_cast<double*>(p + Rs::LIFT);
  int* row = reinterpret_cast<int*>(tab + 3 * Rs::TAB);
  a.tab = tab;
  a.row = row;
  a.lift = EO ? nullptr : lift;
  fixlimb* shared = bytes >= Rs::BYTES ? reinterpret_cast<fixlimb*>(p + Rs::SHARED) : nullptr;
  const long long npne = (long long)(P + 1) * (P + 1) * (P + 1) * a.Ne;
  if constexpr (EO)
    ref_tables_eo_kernel<P><<<1, 256, 0, st>>>(a.D, a.Dt, a.Lift, a.Escale, npne, tab, row, shared,
                                               a.err);
  else
    ref_tables_kernel<P><<<3 * (P + 1), 256, 0, st>>>(a.D, a.Dt, a.Lift, a.Escale, npne, tab, row,
                                                      lift, shared);
  SDG_CUDA_TRY(cudaGetLastError());
  a.shared = shared;
  return SDG_OK;
}

}  // namespace sdg
