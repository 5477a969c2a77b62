// Kernels behind the reference-shaped entry points, for meshes given as the
// reference's arrays (VMapM/VMapP with a halo buffer, normal_fn, Escale,
// Fscale), so any connectivity the caller builds is honoured.
//
//   step_ref_kernel  the whole tendency, and the stages of the time loop
//                    (sdg_dropin_step.cuh); EVENODD always, GENERAL and OPT1
//                    tendencies from 160,000 DOF or p = 12;
//   flux_kernel      cal_elembnd_flux (mod_advect3d_eq.f90:89-142), one
//                    thread per face node, VMap indices range-checked, and
//   dqdt_kernel      cal_dqdt (mod_advect3d_eq.f90:146-201), EPB elements
//                    per block staged in shared memory: the GENERAL and OPT1
//                    tendencies of smaller meshes (tend_dev has the
//                    measurements) and of so few elements (about Nq) that the
//                    flux scratch does not hold step_ref_kernel's tables, and
//                    a tendency written over one of its fields;
//   ops_kernel       tensorprod_divlike_dirXYZ (mod_dg_optr_kernel.f90:62-136),
//                    gradlike and matvec over a batch of elements
//                    (sdg_dropin_ops.cuh), and
//   divlike_kernel, gradlike_kernel  the same in FP64 over few elements, and
//                    divlike with outputs over other directions' inputs;
//   lift_kernel      tensorprod_Lift_hexahedral (mod_dg_optr_kernel.f90:139-190).
#pragma once

#include "sdg_dropin_ops.cuh"
#include "sdg_stage.cuh"
#include "sdg_stage_eo.cuh"

namespace sdg {

struct TendArgs {
  double* dqdt;
  const double* q;
  const double* u;
  const double* v;
  const double* w;
  const double* D;      // D1D(Nq,Nq)
  const double* Dt;     // D1D_tr(Nq,Nq)
  const double* Lift;   // Lift_mat(Nq,Nq,Nq,6)
  const int* VMapM;
  const int* VMapP;
  const double* normal_fn;
  const double* Escale;
  const double* Fscale;
  double* flux;         // ebnd_flux(NfpTot,Ne)
  int* err;             // set to 1 on an out-of-range VMap entry
  int Ne;
  long long NpNeA;      // Np*NeA: valid 1-based indices are 1..NpNeA
};

// Elements per block: as many whole elements as the block has threads for
// (32 at p = 1, 9 at p = 2, 4 at p = 3, 2 at p = 4, one from p = 5), so that
// every thread owns a node at low orders; R nodes a thread in all.
template <int P>
struct DropCfg {
  static constexpr int THREADS = (P >= 10) ? 512 : 256;
  static constexpr int EPB = (THREADS / Ord<P>::NP) > 0 ? THREADS / Ord<P>::NP : 1;
  static constexpr int R = (EPB * Ord<P>::NP + THREADS - 1) / THREADS;
};

template <int P>
constexpr size_t dqdt_smem_bytes() {
  using O = Ord<P>;
  return sizeof(double) * (size_t)(2 * O::NQ2 + DropCfg<P>::EPB * 3 * O::NP);
}

// cal_dqdt for elements [blockIdx.x*EPB, ...): F_d = q*u_d, divergence with
// D1D (x) and D1D_tr (y, z) exactly as tensorprod_divlike_dirXYZ reads them,
// lift of flux(:,ke), combine with Escale(:,ke,d).
template <int P, bool SPLIT3>
__global__ void __launch_bounds__(DropCfg<P>::THREADS) dqdt_kernel(const TendArgs a) {
  using O = Ord<P>;
  constexpr int NQ = O::NQ, NQ2 = O::NQ2, NP = O::NP, NFT = O::NFT,
                EPB = DropCfg<P>::EPB, T = DropCfg<P>::THREADS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sD = reinterpret_cast<double*>(smem_raw);
  double* sDt = sD + NQ2;
  double* fx = sDt + NQ2;
  double* fy = fx + EPB * NP;
  double* fz = fy + EPB * NP;
  const long long eb = (long long)blockIdx.x * EPB;
  const int nloc = (int)min((long long)EPB, (long long)a.Ne - eb);
  if (nloc <= 0) return;
  for (int t = threadIdx.x; t < NQ2; t += T) {
    sD[t] = a.D[t];
    sDt[t] = a.Dt[t];
  }
  const long long g0 = eb * NP;
  for (int t = threadIdx.x; t < nloc * NP; t += T) {
    const double qq = a.q[g0 + t];
    fx[t] = qq * a.u[g0 + t];
    fy[t] = qq * a.v[g0 + t];
    fz[t] = qq * a.w[g0 + t];
  }
  __syncthreads();
  const long long NpNe = (long long)NP * a.Ne;
  // one direction at a time, each node's running sum
  // Escale_x D F_x + Escale_y D F_y + Escale_z D F_z kept in acc: a thread
  // keeps one line sum live, not three (94 registers and two blocks an SM at
  // p = 3 with the three interleaved)
  constexpr int R = DropCfg<P>::R;
  double acc[R];
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int t = threadIdx.x + r * T;
    if (t < nloc * NP) {
      const int le = t / NP, n = t - le * NP;
      const int j = (n / NQ) % NQ, k = n / NQ2;
      const double dx =
          line_sum<NQ, SPLIT3, NQ>(sD + n % NQ, fx + le * NP + j * NQ + k * NQ2, 1);
      acc[r] = a.Escale[g0 + t] * dx;
    }
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int t = threadIdx.x + r * T;
    if (t < nloc * NP) {
      const int le = t / NP, n = t - le * NP;
      const int i = n % NQ, j = (n / NQ) % NQ, k = n / NQ2;
      const double dy = line_sum<NQ, SPLIT3, 1>(sDt + j * NQ, fy + le * NP + i + k * NQ2, NQ);
      acc[r] = fma(a.Escale[g0 + t + NpNe], dy, acc[r]);
    }
  }
#pragma unroll
  for (int r = 0; r < R; r++) {
    const int t = threadIdx.x + r * T;
    if (t < nloc * NP) {
      const int le = t / NP, n = t - le * NP;
      const int i = n % NQ, j = (n / NQ) % NQ, k = n / NQ2;
      const double dz = line_sum<NQ, SPLIT3, 1>(sDt + k * NQ, fz + le * NP + i + j * NQ, NQ2);
      const double lf = lift_node<P>(a.Lift + n, a.flux + (eb + le) * NFT, i, j, k);
      a.dqdt[g0 + t] = -(fma(a.Escale[g0 + t + 2 * NpNe], dz, acc[r]) + lf);
    }
  }
}

template <int P>
constexpr size_t divlike_smem_bytes() {
  using O = Ord<P>;
  return sizeof(double) * (size_t)(2 * O::NQ2 + DropCfg<P>::EPB * 3 * O::NP);
}

template <int P, bool SPLIT3>
__global__ void __launch_bounds__(DropCfg<P>::THREADS) divlike_kernel(const DivArgs a) {
  using O = Ord<P>;
  constexpr int NQ = O::NQ, NQ2 = O::NQ2, NP = O::NP, EPB = DropCfg<P>::EPB,
                T = DropCfg<P>::THREADS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sD = reinterpret_cast<double*>(smem_raw);
  double* sDt = sD + NQ2;
  double* fx = sDt + NQ2;
  double* fy = fx + EPB * NP;
  double* fz = fy + EPB * NP;
  const long long eb = (long long)blockIdx.x * EPB;
  const int nloc = (int)min((long long)EPB, (long long)a.nelem - eb);
  if (nloc <= 0) return;
  for (int t = threadIdx.x; t < NQ2; t += T) {
    sD[t] = a.D[t];
    sDt[t] = a.Dt[t];
  }
  const long long g0 = eb * NP;
  for (int t = threadIdx.x; t < nloc * NP; t += T) {
    fx[t] = a.ix[g0 + t];
    fy[t] = a.iy[g0 + t];
    fz[t] = a.iz[g0 + t];
  }
  __syncthreads();
  // one direction at a time (a thread keeps one line sum live; 74 registers
  // at p = 3 with the three interleaved)
  for (int t = threadIdx.x; t < nloc * NP; t += T) {
    const int le = t / NP, n = t - le * NP;
    const int j = (n / NQ) % NQ, k = n / NQ2;
    a.ox[g0 + t] = line_sum<NQ, SPLIT3, NQ>(sD + n % NQ, fx + le * NP + j * NQ + k * NQ2, 1);
  }
  for (int t = threadIdx.x; t < nloc * NP; t += T) {
    const int le = t / NP, n = t - le * NP;
    const int i = n % NQ, j = (n / NQ) % NQ, k = n / NQ2;
    a.oy[g0 + t] = line_sum<NQ, SPLIT3, 1>(sDt + j * NQ, fy + le * NP + i + k * NQ2, NQ);
  }
  for (int t = threadIdx.x; t < nloc * NP; t += T) {
    const int le = t / NP, n = t - le * NP;
    const int i = n % NQ, j = (n / NQ) % NQ;
    a.oz[g0 + t] = line_sum<NQ, SPLIT3, 1>(sDt + (n / NQ2) * NQ, fz + le * NP + i + j * NQ, NQ2);
  }
}

template <int P>
__global__ void lift_kernel(double* out, const double* Lift, const double* in,
                            int nelem) {
  using O = Ord<P>;
  const long long total = (long long)O::NP * nelem;
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const long long e = g / O::NP;
    const int n = (int)(g - e * O::NP);
    const int i = n % O::NQ, j = (n / O::NQ) % O::NQ, k = n / O::NQ2;
    out[g] = lift_node<P>(Lift + n, in + e * O::NFT, i, j, k);
  }
}

template <int P, bool SPLIT3>
int launch_dqdt_impl(const TendArgs& a, cudaStream_t st) {
  constexpr size_t smem = dqdt_smem_bytes<P>();
  SDG_CUDA_TRY(cudaFuncSetAttribute(dqdt_kernel<P, SPLIT3>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)smem));
  const long long nblk = ((long long)a.Ne + DropCfg<P>::EPB - 1) / DropCfg<P>::EPB;
  if (nblk == 0) return SDG_OK;
  dqdt_kernel<P, SPLIT3><<<(unsigned)nblk, DropCfg<P>::THREADS, smem, st>>>(a);
  SDG_CUDA_TRY(cudaGetLastError());
  return SDG_OK;
}

// element_operation_kernel_matvec_gradlike_dirXYZ_P* (erb:166-219): the
// three directional contractions of ONE field (a.ix; a.iy and a.iz unused),
// always as a running sum over l (the template has no three-way split).  The
// z direction contracts along k, Σ_l vec_in(i,j,l) Mat_tr(l,k); the
// template's first z term, vec_in(i,1,k)*Mat_tr(1,j), is a typo and is not
// reproduced.  The field is staged once per element, so a DOF costs one read
// and three writes.  A NULL output is skipped: with one output this is the
// single-direction matvec_dirX / dirY / dirZ (erb:51-129).
template <int P>
constexpr size_t gradlike_smem_bytes() {
  using O = Ord<P>;
  return sizeof(double) * (size_t)(2 * O::NQ2 + DropCfg<P>::EPB * O::NP);
}

template <int P>
__global__ void __launch_bounds__(DropCfg<P>::THREADS) gradlike_kernel(const DivArgs a) {
  using O = Ord<P>;
  constexpr int NQ = O::NQ, NQ2 = O::NQ2, NP = O::NP, EPB = DropCfg<P>::EPB,
                T = DropCfg<P>::THREADS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* sD = reinterpret_cast<double*>(smem_raw);
  double* sDt = sD + NQ2;
  double* f = sDt + NQ2;
  const long long eb = (long long)blockIdx.x * EPB;
  const int nloc = (int)min((long long)EPB, (long long)a.nelem - eb);
  if (nloc <= 0) return;
  for (int t = threadIdx.x; t < NQ2; t += T) {
    sD[t] = a.D[t];
    sDt[t] = a.Dt[t];
  }
  const long long g0 = eb * NP;
  for (int t = threadIdx.x; t < nloc * NP; t += T) f[t] = a.ix[g0 + t];
  __syncthreads();
  // one direction at a time: a thread keeps one running sum live, not three
  // (82 registers and three blocks an SM at p = 7 when the three were
  // interleaved)
  if (a.ox)
    for (int t = threadIdx.x; t < nloc * NP; t += T) {
      const int le = t / NP, n = t - le * NP;
      const int i = n % NQ, j = (n / NQ) % NQ, k = n / NQ2;
      a.ox[g0 + t] = line_sum<NQ, false, NQ>(sD + i, f + le * NP + j * NQ + k * NQ2, 1);
    }
  if (a.oy)
    for (int t = threadIdx.x; t < nloc * NP; t += T) {
      const int le = t / NP, n = t - le * NP;
      const int i = n % NQ, j = (n / NQ) % NQ, k = n / NQ2;
      a.oy[g0 + t] = line_sum<NQ, false, 1>(sDt + j * NQ, f + le * NP + i + k * NQ2, NQ);
    }
  if (a.oz)
    for (int t = threadIdx.x; t < nloc * NP; t += T) {
      const int le = t / NP, n = t - le * NP;
      const int i = n % NQ, j = (n / NQ) % NQ, k = n / NQ2;
      a.oz[g0 + t] = line_sum<NQ, false, 1>(sDt + k * NQ, f + le * NP + i + j * NQ, NQ2);
    }
}

template <int P>
int launch_gradlike_impl(const DivArgs& a, cudaStream_t st) {
  constexpr size_t smem = gradlike_smem_bytes<P>();
  SDG_CUDA_TRY(cudaFuncSetAttribute(gradlike_kernel<P>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const long long nblk = ((long long)a.nelem + DropCfg<P>::EPB - 1) / DropCfg<P>::EPB;
  if (nblk == 0) return SDG_OK;
  gradlike_kernel<P><<<(unsigned)nblk, DropCfg<P>::THREADS, smem, st>>>(a);
  SDG_CUDA_TRY(cudaGetLastError());
  return SDG_OK;
}

template <int P, bool SPLIT3>
int launch_divlike_impl(const DivArgs& a, cudaStream_t st) {
  constexpr size_t smem = divlike_smem_bytes<P>();
  SDG_CUDA_TRY(cudaFuncSetAttribute(divlike_kernel<P, SPLIT3>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)smem));
  const long long nblk = ((long long)a.nelem + DropCfg<P>::EPB - 1) / DropCfg<P>::EPB;
  if (nblk == 0) return SDG_OK;
  divlike_kernel<P, SPLIT3><<<(unsigned)nblk, DropCfg<P>::THREADS, smem, st>>>(a);
  SDG_CUDA_TRY(cudaGetLastError());
  return SDG_OK;
}

template <int P>
int launch_lift_impl(double* out, const double* Lift, const double* in, int nelem,
                     cudaStream_t st) {
  const long long total = (long long)Ord<P>::NP * nelem;
  if (total == 0) return SDG_OK;
  const long long nb = (total + 255) / 256;
  lift_kernel<P><<<(unsigned)(nb < 65535LL * 32 ? nb : 65535LL * 32), 256, 0, st>>>(
      out, Lift, in, nelem);
  SDG_CUDA_TRY(cudaGetLastError());
  return SDG_OK;
}

}  // namespace sdg

#include "sdg_dropin_step.cuh"

namespace sdg {

// A call of step_ref_kernel: its arguments, its mode (kRkTend, kRkFirst,
// kRkGeneral) and where its tables go.
struct RefCall {
  RefArgs* a;
  int mode;
  void* tables;
  size_t bytes;
};

// Whether a contraction over nelem elements runs in fixed point: from 150k nodes
// (about one wave of blocks; below it the FP64 kernels' blocks of one node a
// thread wait less: p = 3 6.6 / 4.6 us at 20k nodes, level at 100k, 16.8 / 25.2 at
// 1M; p = 7 8.8 / 10.7 at 100k) and always from p = 11 (15 / 23 us at 100k nodes,
// p = 15 23 / 62).  divlike at p = 1, 48 bytes a node for 6 FP64 instructions,
// stays in FP64 (115 / 118 us at 10M nodes).
template <int P>
constexpr bool ops_always() { return P >= 11; }
template <int P>
bool ops_fixed(int nelem) {
  return ops_always<P>() || (long long)nelem * Ord<P>::NP >= 150000;
}

// Per-order entry used by the dispatch in sdg_dropin.cu.  what: 0 cal_dqdt,
// 1 divlike, 2 lift, 3 gradlike, 4 step_ref_kernel, 5 its tables, 6 the bytes
// of these (into the two size_t args points at: at least, and the whole).
template <int P>
int dropin_order(int what, int opt, const void* args, cudaStream_t st) {
  constexpr bool kCanSplit = (P > 7);
  const bool split = kCanSplit && opt == SDG_OPT_OPT1;
  switch (what) {
    case 0: {
      const TendArgs& a = *static_cast<const TendArgs*>(args);
      return split ? launch_dqdt_impl<P, kCanSplit>(a, st) : launch_dqdt_impl<P, false>(a, st);
    }
    case 1: {
      // ops_kernel writes y and z lines while other lines of the element's inputs
      // are still read; divlike_kernel reads all three inputs of an element first
      const DivArgs& a = *static_cast<const DivArgs*>(args);
      if (P > 1 && ops_fixed<P>(a.nelem) && !a.staged) return launch_ops<P, false>(a, st);
      return split ? launch_divlike_impl<P, kCanSplit>(a, st)
                   : launch_divlike_impl<P, false>(a, st);
    }
    case 3:
      if constexpr (ops_always<P>()) {
        return launch_ops<P, true>(*static_cast<const DivArgs*>(args), st);
      } else {
        return ops_fixed<P>(static_cast<const DivArgs*>(args)->nelem)
                   ? launch_ops<P, true>(*static_cast<const DivArgs*>(args), st)
                   : launch_gradlike_impl<P>(*static_cast<const DivArgs*>(args), st);
      }
    case 4: {
      const RefCall& c = *static_cast<const RefCall*>(args);
      const bool eo = opt == SDG_OPT_EVENODD;
      switch (c.mode) {
        case kRkTend:
          return eo ? launch_ref_mode<P, true, kRkTend>(*c.a, st)
                    : launch_ref_mode<P, false, kRkTend>(*c.a, st);
        case kRkFirst:
          return eo ? launch_ref_mode<P, true, kRkFirst>(*c.a, st)
                    : launch_ref_mode<P, false, kRkFirst>(*c.a, st);
        default:
          return eo ? launch_ref_mode<P, true, kRkGeneral>(*c.a, st)
                    : launch_ref_mode<P, false, kRkGeneral>(*c.a, st);
      }
    }
    case 5: {
      const RefCall& c = *static_cast<const RefCall*>(args);
      return opt == SDG_OPT_EVENODD ? launch_ref_tables<P, true>(*c.a, c.tables, c.bytes, st)
                                    : launch_ref_tables<P, false>(*c.a, c.tables, c.bytes, st);
    }
    case 6: {
      size_t* out = static_cast<size_t*>(const_cast<void*>(args));
      const bool eo = opt == SDG_OPT_EVENODD;
      out[0] = eo ? RefShape<P, true>::LEAST : RefShape<P, false>::LEAST;
      out[1] = eo ? RefShape<P, true>::BYTES : RefShape<P, false>::BYTES;
      return SDG_OK;
    }
    default: {
      const DivArgs& a = *static_cast<const DivArgs*>(args);
      // lift: ox = out, D = Lift, ix = in
      return launch_lift_impl<P>(a.ox, a.D, a.ix, a.nelem, st);
    }
  }
}

}  // namespace sdg
