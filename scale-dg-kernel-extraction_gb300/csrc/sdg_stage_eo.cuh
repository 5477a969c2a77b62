// The even-odd factorisation of the 1D operators (opt type SDG_OPT_EVENODD): the
// tables' layout, shared by the FP64 stage (sdg_stage_fix.cuh) and the FP32
// stage (sdg_stage_line.cuh).
//
// The pair sums cost about half the operations of the plain line sums, and
// one thread a line replaces the node body's per-node shared-memory reads of a
// whole line by one read per line value:
//
//  * Centro-antisymmetry of the GLL differentiation matrix,
//    D(N-1-i, N-1-l) = -D(i, l), splits a line's N-term sums into pairs:
//    with S(l) = F(l) + F(N-1-l) and Δ(l) = F(l) - F(N-1-l), l < N/2,
//        e_i = Σ_l E(i,l) S(l) [+ D(i,mid) F(mid)],  o_i = Σ_l O(i,l) Δ(l),
//        out(i) = e_i + o_i,   out(N-1-i) = o_i - e_i,
//    where E / O are the half-sums / half-differences of D's columns l and
//    N-1-l.  A line of N outputs costs N²/2 + 2N operations instead of N².
//  * The lift of a face is a 1D column along the face normal, constant over
//    the tangential nodes, and the + face's column is the mirror of the -
//    face's (Lift_mat of operator_data/p*.dat has both properties to
//    rounding).  With gs = g- + g+ and gd = g- - g+ the two faces of a line
//    join the same pairs: e_i += B(i) gd, o_i += A(i) gs.
//  * Escale, the stage's b*dt and the minus sign of dqdt are folded into the
//    coefficients, and 0.5*Fscale into the lift columns,
//    so a node's increment is the plain sum of its three line results and
//    the RK update is q_out = b*q + inc (+ a*q0).
//  * The face flux 0.5 Fs (qP VelP - qM VelM - α (qP - qM)) is formed as
//    qP (2VelP - 2α) - qM (2VelM - 2α) with 2α = |uP + uM| (the normal sign
//    applied through the constant ±2): five operations per face node.
//
// The summation order is neither GENERAL's nor OPT1's; the result agrees
// with both to rounding (the parity tests hold it to the same tolerance).
// The host builds the E / O / lift tables only after checking the operator
// symmetries; operators without them are refused for this opt type.
#pragma once

#include "sdg_stage.cuh"

namespace sdg {

template <int P>
struct EoShape {
  static constexpr int N = P + 1;
  static constexpr int H = N / 2;          // pairs (l, N-1-l)
  static constexpr int HR = (N + 1) / 2;   // output rows incl. the middle row
  static constexpr int ODD = N & 1;
  static constexpr int OFF_E = 0;                      // E(i,l), i < H, l < H
  static constexpr int OFF_O = H * H;                  // O(i,l), i < HR, l < H
  static constexpr int OFF_DM = OFF_O + HR * H;        // D(i,mid), i < H (odd N)
  static constexpr int OFF_A = OFF_DM + ODD * H;       // lift sym part, i < HR
  static constexpr int OFF_B = OFF_A + HR;             // lift antisym part, i < H
  static constexpr int TE = OFF_B + H;                 // entries per direction
};

// Starts moving the 128-byte line holding p into L2 (no register, no wait).
__device__ __forceinline__ void prefetch_l2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

__device__ __forceinline__ double abs_ct(double x) {
  return __longlong_as_double(__double_as_longlong(x) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ float abs_ct(float x) { return fabsf(x); }

}  // namespace sdg
