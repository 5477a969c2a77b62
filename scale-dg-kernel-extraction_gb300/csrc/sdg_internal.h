// Internal declarations shared by the translation units of libsdg_gb300.
#pragma once

#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <vector>

#include "sdg_advect.h"

namespace sdg {

constexpr int kMaxOrder = 15;

// Records a message for sdg_last_error() (thread-local) and returns status.
int fail(int status, const char* fmt, ...);
// Maps a CUDA error to SDG_ERR_CUDA / SDG_ERR_OUT_OF_MEMORY with a message.
int cuda_fail(cudaError_t e, const char* what, const char* file, int line);

#define SDG_CUDA_TRY(call)                                              \
  do {                                                                  \
    cudaError_t sdg_e_ = (call);                                        \
    if (sdg_e_ != cudaSuccess)                                          \
      return ::sdg::cuda_fail(sdg_e_, #call, __FILE__, __LINE__);       \
  } while (0)

#define SDG_TRY(expr)                 \
  do {                                \
    int sdg_s_ = (expr);              \
    if (sdg_s_ != SDG_OK) return sdg_s_; \
  } while (0)

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Raises a kernel's dynamic shared-memory limit to smem bytes and sets its
// preferred shared-memory carveout in percent (kCarveDefault: the driver's
// choice) on the current device.
// Kernel attributes are per device, so this records them per kernel and device
// and sets them when they change; it is safe to call from several host threads
// at once.
int set_kernel_smem(const void* func, int smem, int carve);
constexpr int kCarveDefault = -1, kCarveMax = 100;
// The carveout that holds `blocks` blocks of smem bytes on an SM (228 KB, 1 KB
// of each block's taken by the system): what is left of the 256 KB is L1.
constexpr int carve_for(size_t smem, int blocks) {
  const size_t pct = (blocks * (smem + 1024) * 100 + 228 * 1024 - 1) / (228 * 1024);
  return pct < 100 ? (int)pct : 100;
}

// Maps the pages of a pageable host buffer that a device copy is about to fill
// (map_pages: no store to them).  On GB300 a copy's writes to pages that the
// process has not touched yet (fresh from the allocator) fault one by one
// through the address translation, about 45 us a 64 KB page.  A download of 101
// MB into a fresh array takes 3.5 ms mapped first (33 ms with a store of the CPU
// a page, 0.54 into pages that are there).  Pinned, managed and device memory is
// left alone.
void touch_pages(void* p, size_t bytes);

// Checks the first CUDA device is usable; returns SDG_OK or an error status.
int require_device();

// Structured periodic box: what the fused stage kernel needs to know about the
// mesh of mod_mesh.f90:74-193 (element order, per-axis scale factors).
struct Box {
  int NeX, NeY, NeZ;
  long long Ne;
  double Es[3];  // Escale(:,:,d) = 2/dx_d  (mod_mesh.f90:147-149)
  double Fs[3];  // Fscale of the faces normal to axis d (mod_mesh.f90:366-394)
  // FP32 copies made on the host (Es, and 0.5*Fs as the flux uses it): a
  // conversion in the kernel would run on GB300's 1/64-rate FP64 pipe
  float Esf[3];
  float hFsf[3];
};
Box make_box(int NeX, int NeY, int NeZ, double Lx, double Ly, double Lz);

// Coefficients of the fixed-point stage (sdg_stage_fix.cuh) on the host: per
// direction the even-odd table of EoShape as limb pairs (hi, lo) of
// c 2^(60 - k), c = -(derivative entry) Es_d or -(lift entry) Fs_d, k the
// row's exponent: what its outputs can reach on values below one is below 2^k.
// row: k - 61.  ok = 0
// when an exponent lies outside +-200: every line is then formed in FP64.
struct FixTables {
  std::vector<int32_t> coef;
  std::vector<int> row;
  int ok = 0;
  int thin = 0;  // operators as given: the lift has zeros
};
// Fills t from the unscaled tables of eo_tables.
void fix_tables(int Nq, const Box& box, const std::vector<double>& eo, FixTables& t);
// The same for operators as given (coef: per direction D(i,l) at i Nq + l; one
// scale a row, over all its nodes' lift entries).  lift receives, per direction
// d, row i and line r of the direction, the limb pairs of the - and the + face's
// lift entry at that node: 4 * 3 * Nq^3 values.
void fix_tables_general(int Nq, const Box& box, const double* D1D, const double* Lift_mat,
                        FixTables& t, std::vector<int32_t>& lift);

// Arguments of one fused stage launch.
struct StageArgs {
  const double* q_in;   // state read by the stage (Np*Ne)
  const double* q0;     // step-start state (stages 2 and 3), may be null if a==0
  double* q_out;        // RK result (Np*Ne), or the tendency when tend_only
  const void* u;        // velocity components (double or float, Np*Ne)
  const void* v;
  const void* w;
  const void* D;        // D1D(Nq,Nq), column-major, compute type
  const void* Lift;     // Lift_mat(Nq,Nq,Nq,6), compute type
  Box box;
  long long elem_begin;  // first element of this launch
  long long elem_count;  // elements of this launch
  double a, b, dt;      // q_out = a*q0 + b*(q_in + dt*dqdt)
  float cdt_hi;         // b*dt in FP32
  int b_is_one;         // b == 1 (stage 1): the kernels branch on integers,
  int a_nonzero;        // since an FP64 comparison also uses the FP64 pipe
  int tend_only;        // write dqdt instead of the RK update
  // even-odd stages: D points at the 3-direction table built by the solver; the
  // FP32 form's per-direction factors of its D part (-c*Es_d) and of its lift
  // part (-c*Fs_d/4), c = b*dt (1 for tend_only)
  float eo_sDf[3], eo_sLf[3];
  const float* eo_host;  // FP32: the table on the host
  // FP64 stage: the velocity factors of the face flux, two per face node of
  // each element (2*Nfp*6 doubles an element).  A stage with
  // fc_out forms them from u, v, w and stores them; a stage with fc_in reads
  // them instead (same bits), so the stages of one solver call, which share
  // the velocity (main.f90:58-67 passes the same u, v, w to every
  // advect3d_eq_cal_tend call), form them once.  Both null: formed inline.
  double* fc_out;
  const double* fc_in;
  // FP64 stage: its fixed-point coefficients (host memory, copied into the
  // launch), and for operators as given the nodes' lift limbs (device memory,
  // one int4 a node and direction)
  const FixTables* fix;
  const void* fix_lift;
};

// Even-odd tables (3 directions, unscaled) from D1D and Lift_mat after the
// symmetry checks; SDG_ERR_INVALID_ARG when the operators lack them.
int eo_tables(int Nq, const double* D1D, const double* Lift_mat, std::vector<double>& tab);

// Fused stage launchers (sdg_stage_*.cu).  prec = SDG_PREC_*.
int launch_stage(int p, int prec, int opt, const StageArgs& a, cudaStream_t st);
// nstep whole steps of a small box in one launch (FP64 form): q the rotating
// state buffers, the current one first; bar two device words, zero (the second
// set by a wait between the stages that gave up after `polls` reads);
// the result is in q[nstep % 3].  With q null: *most = the most elements.
// kLoopTooLarge, with nothing launched, where the stream has fewer SMs than the
// device (a green context's) and they do not hold the grid.
constexpr int kLoopTooLarge = 1;
int launch_loop(int p, int opt, const StageArgs& a, double* const* q, double dt, int nstep,
                unsigned* bar, int polls, long long* most, cudaStream_t st);

// min / max of q[0..n) as order keys (see sdg_minmax.cu); resets both keys first.
int minmax_launch(const double* q, long long n, unsigned long long* kmin, unsigned long long* kmax,
                  cudaStream_t st);
double minmax_key_to_double(unsigned long long k);
// Dynamic shared memory the launcher uses for order p, to size opt-in limits.
int stage_setup_attributes(int p, int prec, int opt);

}  // namespace sdg
