// The batched stage kernels and their helpers (see sdg_batch.cuh).
#include "sdg_batch.cuh"
#include "sdg_stage_line.cuh"

namespace sdg {

namespace {

// SSP-RK3 coefficients, mod_common.f90:28-30
__constant__ double c_rk_a[3] = {0.0, 0.75, 1.0 / 3.0};
__constant__ double c_rk_b[3] = {1.0, 0.25, 2.0 / 3.0};

// 32-bit words of an instance header, copied into shared memory by as many
// threads.
constexpr int kInstWords = (int)(sizeof(BatchInst) / 4);
static_assert(sizeof(BatchInst) % 4 == 0, "instance header is copied as 32-bit words");
static_assert(kInstWords < 128, "the smallest block must copy the header in one pass");

// Bytes of shared memory of a block of `threads` threads of the even-odd body:
// the instance's scaled coefficients, then the line arrays of the elements a
// block holds at once.
template <int P>
__host__ __device__ constexpr size_t batch_line_smem(int threads) {
  return sizeof(float) * 3 * LineRows<P>::DIR + line_smem<P>(threads / FixShape<P>::N2);
}
// The block size an item is run with: at least one element's lines.
template <int P>
__host__ __device__ constexpr int batch_line_threads(int threads) {
  constexpr int least = (FixShape<P>::N2 + 31) / 32 * 32;
  return threads < least ? least : threads;
}

// One work item through one stage: the instance's buffers for the stage from
// its current index, then the order's stage body.
template <int P, int EO, int RK>
__device__ __forceinline__ void batch_item_body(const BatchInst& I, const BatchItem& w,
                                                int stage, unsigned char* smem) {
  if constexpr (EO != 0) {
    // the even-odd line stage (sdg_stage_line.cuh), the coefficients scaled for
    // this instance in shared memory; blockDim.x / N^2 elements at a time
    using Rows = LineRows<P>;
    constexpr int TE = EoShape<P>::TE, OFF_A = EoShape<P>::OFF_A, NP = FixShape<P>::N * FixShape<P>::N2;
    float* T = reinterpret_cast<float*>(smem);
    // read now, stored once the state's loads are on their way; where a
    // coefficient goes and its factor also now, but for the orders with the
    // fewest instructions between (p = 3 111.6 from 106.6, p = 7 133.0 from 132.0,
    // p = 10 123.9 from 116.6 GDOF-updates/s; p = 2 99.3 against 102.3, p = 4 117.0
    // against 126.8)
    constexpr int LEAST = (FixShape<P>::N2 + 31) / 32 * 32;  // threads, at least
    constexpr int PER = (3 * TE + LEAST - 1) / LEAST;
    constexpr bool EARLY = P == 3 || P >= 5;
    float c[PER], by[PER];
    int to[PER];
    auto place = [&](int k) {
      const int t = threadIdx.x + k * blockDim.x;
      const int d = t / TE, n = t - d * TE;
      to[k] = t < 3 * TE ? d * Rows::DIR + Rows::at(n) : -1;
      by[k] = t < 3 * TE ? (n < OFF_A ? I.eo_sD[stage][d] : I.eo_sL[stage][d]) : 0.0f;
    };
#pragma unroll
    for (int k = 0; k < PER; k++) {
      const int t = threadIdx.x + k * blockDim.x;
      c[k] = t < 3 * TE ? I.eo_tab[t] : 0.0f;
      if constexpr (EARLY) place(k);
    }
    auto store = [&] {
#pragma unroll
      for (int k = 0; k < PER; k++) {
        if constexpr (!EARLY) place(k);
        if (to[k] >= 0) T[to[k]] = c[k] * by[k];
      }
    };
    const int s0 = I.cur, s1 = s0 == 2 ? 0 : s0 + 1, s2 = s1 == 2 ? 0 : s1 + 1;
    const double* q = I.q[stage == 0 ? s0 : stage == 1 ? s1 : s2];
    const int epb = blockDim.x / FixShape<P>::N2;
    // No barrier between two rounds: a thread reads last, and writes first, its
    // own z line of the arrays; the first barrier inside orders the coefficients
    // before their first use.
    for (int e = 0; e < w.e_count; e += epb)
      line_elements<P, RK, true>(
          q, I.q[s0], I.q[stage == 1 ? s2 : s1], I.u, I.v, I.w, I.box, c_rk_a[stage],
          c_rk_b[stage], w.e_begin + e, min(epb, w.e_count - e), epb, T + 3 * Rows::DIR,
          [&](int d) { return Rows{T + d * Rows::DIR}; },
          [&] {
            if (e == 0) store();
          });
    return;
  }
  const int s0 = I.cur, s1 = (s0 + 1) % 3, s2 = (s0 + 2) % 3;
  StageArgs a;
  a.q_in = (stage == 0) ? I.q[s0] : (stage == 1) ? I.q[s1] : I.q[s2];
  a.q0 = (stage == 0) ? nullptr : I.q[s0];
  a.q_out = (stage == 1) ? I.q[s2] : I.q[s1];
  a.u = I.u;
  a.v = I.v;
  a.w = I.w;
  a.D = I.D;
  a.Lift = I.Lift;
  a.box = I.box;
  a.fc_out = nullptr;
  a.fc_in = nullptr;
  a.elem_begin = 0;
  a.elem_count = I.box.Ne;
  a.a = c_rk_a[stage];
  a.b = c_rk_b[stage];
  a.dt = I.dt;
  a.cdt_hi = I.cdt[stage];  // FP32 increment factor of the FP32 form
  a.b_is_one = (stage == 0);
  a.a_nonzero = (stage != 0);
  a.tend_only = 0;
  stage_block<P, float, float, false, RK>(a, w.e_begin, w.e_count, smem);
}

// Even-odd body: one block per work item; no work-item state stays live across
// the stage.  64 registers a thread, as in the single-box kernel (40: 0.95x at
// p = 3, 0.8x at p = 7).  Against a block body with every flux and face staged in
// shared memory, four boxes of 3.5M DOF, GDOF-updates/s: p = 1 89 from 63, p = 2
// 104 from 82, p = 3 114 from 96, p = 4 127 from 92, p = 5 122 from 86, p = 7 132
// from 103, p = 9 116 from 86, p = 11 110 from 89.  A block starts with two
// dependent reads (item, instance) that the single-box kernel does without:
// it waits on loads (long-scoreboard stalls 9 of 15 cycles an instruction).
template <int P, int RK>
__global__ void __launch_bounds__(kBatchThreadsMax, 2)
    batch_item_kernel(const BatchInst* __restrict__ insts, const BatchItem* __restrict__ items,
                      int n_items, int stage) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(16) BatchInst s_inst;
  if ((int)blockIdx.x >= n_items) return;  // uniform across the block
  const BatchItem item = items[blockIdx.x];
  for (int t = threadIdx.x; t < kInstWords; t += blockDim.x)
    reinterpret_cast<uint32_t*>(&s_inst)[t] =
        reinterpret_cast<const uint32_t*>(insts + item.inst)[t];
  __syncthreads();
  if (s_inst.active) batch_item_body<P, 1, RK>(s_inst, item, stage, smem);
}

// Node body: one persistent launch runs the items of one order group.
// Compiling one order per kernel keeps each at its own register count; four
// blocks of 512 threads an SM (32 registers) measured 4-16 % above three.
//
// Items are assigned round-robin (block b runs items b, b + G, b + 2G, ...).
// The next item's instance header is fetched into shared memory while the
// current item computes, and the item after that into a register, so that a
// block never waits on the item -> instance -> data chain of dependent loads.
template <int P, int RK>
__global__ void __launch_bounds__(kBatchThreadsMax, 4)
    batch_order_kernel(const BatchInst* __restrict__ insts, const BatchItem* __restrict__ items,
                       int n_items, int stage) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(16) BatchInst s_inst[2];
  __shared__ BatchItem s_items[2];
  const int G = gridDim.x, tid = threadIdx.x;
  int it = blockIdx.x;
  if (it >= n_items) return;  // uniform across the block
  // prologue: the first item, its header, and the second item
  if (tid == 0) {
    s_items[0] = items[it];
    if (it + G < n_items) s_items[1] = items[it + G];
  }
  __syncthreads();
  if (tid < kInstWords)
    reinterpret_cast<uint32_t*>(&s_inst[0])[tid] =
        reinterpret_cast<const uint32_t*>(insts + s_items[0].inst)[tid];
  __syncthreads();

  for (int k = 0; it < n_items; k++, it += G) {
    const int slot = k & 1;
    const bool has_next = it + G < n_items, has_next2 = it + 2 * G < n_items;
    // prefetch, consumed after this item: the next item's header words and
    // the item after it
    uint32_t hw = 0;
    BatchItem nn{};
    if (has_next && tid < kInstWords)
      hw = reinterpret_cast<const uint32_t*>(insts + s_items[slot ^ 1].inst)[tid];
    if (has_next2 && tid == blockDim.x - 1) nn = items[it + 2 * G];

    const BatchItem w = s_items[slot];
    const BatchInst& I = s_inst[slot];
    if (I.active) batch_item_body<P, 0, RK>(I, w, stage, smem);
    // every read of this item's slots happened before the body's barriers
    __syncthreads();
    if (has_next && tid < kInstWords) reinterpret_cast<uint32_t*>(&s_inst[slot ^ 1])[tid] = hw;
    if (has_next2 && tid == blockDim.x - 1) s_items[slot] = nn;
    __syncthreads();  // the next item's header and the dynamic shared memory are ready
  }
}

// ONE persistent launch per RK stage over the work items of every order:
// blocks take items round-robin, read the item's instance header and run the
// stage body compiled for that instance's order and body (a switch over the
// 22 (order, body) pairs).  Block size and dynamic shared memory are the
// largest the present orders need; each body takes the block size at run
// time, so an item's bits are the per-order kernels'.  The kernel carries the
// register needs of every body at once (capped at 64 for two blocks of 512
// threads an SM), which is why the per-order launches are the default.
template <int RK>
__global__ void __launch_bounds__(kBatchThreadsMax, 2)
    batch_stage_kernel(const BatchInst* __restrict__ insts, const BatchItem* __restrict__ items,
                       int n_items, int stage) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(16) BatchInst s_inst;
  __shared__ BatchItem s_item;
  const int tid = threadIdx.x;
  for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
    __syncthreads();  // the previous item's readers of s_inst / smem are done
    if (tid == 0) s_item = items[it];
    __syncthreads();
    if (tid < kInstWords)
      reinterpret_cast<uint32_t*>(&s_inst)[tid] =
          reinterpret_cast<const uint32_t*>(insts + s_item.inst)[tid];
    __syncthreads();
    if (!s_inst.active) continue;  // uniform across the block
    // the body recorded in the item, which the groups' shared-memory sizes
    // were computed for (the device instance table's copy of the body flag
    // is not refreshed when the body changes)
    switch (s_item.body) {
#define SDG_FUSED_CASE(P)                                                    \
  case 2 * P: batch_item_body<P, 0, RK>(s_inst, s_item, stage, smem); break; \
  case 2 * P + 1: batch_item_body<P, 1, RK>(s_inst, s_item, stage, smem); break;
      SDG_FUSED_CASE(1) SDG_FUSED_CASE(2) SDG_FUSED_CASE(3) SDG_FUSED_CASE(4)
      SDG_FUSED_CASE(5) SDG_FUSED_CASE(6) SDG_FUSED_CASE(7) SDG_FUSED_CASE(8)
      SDG_FUSED_CASE(9) SDG_FUSED_CASE(10) SDG_FUSED_CASE(11)
#undef SDG_FUSED_CASE
      default: break;
    }
  }
}

__global__ void batch_advance_kernel(BatchInst* insts, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && insts[i].active) insts[i].cur = (insts[i].cur + 1) % 3;
}

__global__ void init_blob_kernel(double* q, float* u, float* v, float* w, const double* x1D,
                                 Box box, int nq, double cx, double cy, double cz,
                                 double inv2s2, float ux, float uy, float uz) {
  const long long np = (long long)nq * nq * nq;
  const long long total = np * box.Ne;
  const double dx = 2.0 / box.Es[0], dy = 2.0 / box.Es[1], dz = 2.0 / box.Es[2];
  for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < total;
       g += (long long)gridDim.x * blockDim.x) {
    const long long e = g / np;
    const int n = (int)(g - e * np);
    const int i = n % nq, j = (n / nq) % nq, k = n / (nq * nq);
    const int ex = (int)(e % box.NeX);
    const int ey = (int)((e / box.NeX) % box.NeY);
    const int ez = (int)(e / ((long long)box.NeX * box.NeY));
    // node position as mesh_setup places it (mod_mesh.f90:141-145, :344-347)
    const double x = (ex + 0.5) * dx + 0.5 * dx * x1D[i];
    const double y = (ey + 0.5) * dy + 0.5 * dy * x1D[j];
    const double z = (ez + 0.5) * dz + 0.5 * dz * x1D[k];
    double ddx = x - cx, ddy = y - cy, ddz = z - cz;
    ddx -= rint(ddx);
    ddy -= rint(ddy);
    ddz -= rint(ddz);
    q[g] = exp(-(ddx * ddx + ddy * ddy + ddz * ddz) * inv2s2);
    u[g] = ux;
    v[g] = uy;
    w[g] = uz;
  }
}

// What bounds an item's elements: the node body stages them all at once; the
// even-odd body, which takes them a block of lines at a time, keeps the bound of
// a body that would (q, the fluxes, the sums and the face fluxes of each).
template <int P>
size_t smem_for(int epb, int eo) {
  if (!eo) return stage_block_smem<P, float>(epb);
  using O = Ord<P>;
  constexpr int arrays = P <= 4 ? 4 : (P == 6 || P == 8) ? 3 : 5;
  return sizeof(float) * (size_t)(3 * EoShape<P>::TE + epb * (arrays * O::NP + O::NFT)) +
         sizeof(int) * 6 * (size_t)epb;
}

}  // namespace

size_t batch_smem_bytes(int p, int epb, int eo) {
  switch (p) {
    case 1: return smem_for<1>(epb, eo);
    case 2: return smem_for<2>(epb, eo);
    case 3: return smem_for<3>(epb, eo);
    case 4: return smem_for<4>(epb, eo);
    case 5: return smem_for<5>(epb, eo);
    case 6: return smem_for<6>(epb, eo);
    case 7: return smem_for<7>(epb, eo);
    case 8: return smem_for<8>(epb, eo);
    case 9: return smem_for<9>(epb, eo);
    case 10: return smem_for<10>(epb, eo);
    case 11: return smem_for<11>(epb, eo);
    default: return 0;
  }
}

namespace {
// What an order group needs, for one (P, EO) pair: the launch's block size and
// shared memory for a group's, the blocks an SM holds, the launch.
template <int P, int EO>
struct GroupOps {
  static int threads(const BatchGroup& g) {
    return EO ? batch_line_threads<P>(g.threads) : g.threads;
  }
  static size_t smem(const BatchGroup& g, int threads) {
    return EO ? batch_line_smem<P>(threads) : g.smem;
  }
  static int setup(const BatchGroup& g, int* per_sm) {
    if constexpr (EO != 0) {
      int dev = 0, most = 0;
      SDG_CUDA_TRY(cudaGetDevice(&dev));
      SDG_CUDA_TRY(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
      if (g.smem + 2 * (sizeof(BatchInst) + sizeof(BatchItem)) > (size_t)most)
        return cuda_fail(cudaErrorInvalidValue, "batch item size", __FILE__, __LINE__);
      // at most 46 KB at any block size; the carveout holds 1024 threads' worth
      static_assert(batch_line_smem<P>(kBatchThreadsMax) + sizeof(BatchInst) + sizeof(BatchItem) <=
                    48 * 1024);
      constexpr int carve = carve_for(batch_line_smem<P>(128 < FixShape<P>::N2 ? 256 : 128),
                                      128 < FixShape<P>::N2 ? 4 : 8);
      constexpr int limit = (int)batch_line_smem<P>(kBatchThreadsMax);
      SDG_TRY(set_kernel_smem((const void*)batch_item_kernel<P, kRkFirst>, limit, carve));
      SDG_TRY(set_kernel_smem((const void*)batch_item_kernel<P, kRkGeneral>, limit, carve));
      *per_sm = 1;
      return SDG_OK;
    } else {
      SDG_CUDA_TRY(cudaFuncSetAttribute(batch_order_kernel<P, kRkFirst>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)g.smem));
      SDG_CUDA_TRY(cudaFuncSetAttribute(batch_order_kernel<P, kRkGeneral>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)g.smem));
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, batch_order_kernel<P, kRkGeneral>,
                                                        g.threads, g.smem) != cudaSuccess) {
        cudaGetLastError();
        *per_sm = 0;
      }
      return SDG_OK;
    }
  }
  static int launch(const BatchInst* d_inst, const BatchItem* d_items, const BatchGroup& g,
                    int stage, cudaStream_t st) {
    const int t = threads(g);
    const size_t sm = smem(g, t);
    if constexpr (EO != 0) {
      if (stage == 0)
        batch_item_kernel<P, kRkFirst><<<g.grid, t, sm, st>>>(d_inst, d_items, g.count, stage);
      else
        batch_item_kernel<P, kRkGeneral><<<g.grid, t, sm, st>>>(d_inst, d_items, g.count, stage);
    } else {
      if (stage == 0)
        batch_order_kernel<P, kRkFirst><<<g.grid, t, sm, st>>>(d_inst, d_items, g.count, stage);
      else
        batch_order_kernel<P, kRkGeneral><<<g.grid, t, sm, st>>>(d_inst, d_items, g.count, stage);
    }
    SDG_CUDA_TRY(cudaGetLastError());
    return SDG_OK;
  }
};

template <template <int, int> class OPS, typename F>
int with_group(int p, int eo, F&& f) {
  switch (p * 2 + (eo ? 1 : 0)) {
#define SDG_GROUP_CASE(P) \
  case 2 * P: return f(OPS<P, 0>{}); \
  case 2 * P + 1: return f(OPS<P, 1>{});
    SDG_GROUP_CASE(1) SDG_GROUP_CASE(2) SDG_GROUP_CASE(3) SDG_GROUP_CASE(4)
    SDG_GROUP_CASE(5) SDG_GROUP_CASE(6) SDG_GROUP_CASE(7) SDG_GROUP_CASE(8)
    SDG_GROUP_CASE(9) SDG_GROUP_CASE(10) SDG_GROUP_CASE(11)
#undef SDG_GROUP_CASE
    default: return fail(SDG_ERR_UNSUPPORTED_ORDER, "batched order %d outside 1..11", p);
  }
}
}  // namespace

void batch_default_shape(int p, int* threads, int* epb) {
  // index = order; block sizes 128/256/512 and one to four rounds of a block's
  // lines an item, four boxes of 3.5M DOF (p = 3: 111.6 at 128/16, 110.4 at 128/8,
  // 105.0 at 256/32; p = 6: 117.3 at 256/5, 109.0 at 128/4).  From p = 10 a block
  // of one element's lines.
  static const int kThreads[kBatchMaxOrder + 1] = {256, 128, 128, 128, 128, 256,
                                                   256, 128, 256, 128, 128, 128};
  static const int kEpb[kBatchMaxOrder + 1] = {1, 128, 56, 16, 10, 14, 5, 2, 3, 3, 2, 2};
  const int i = (p >= 1 && p <= kBatchMaxOrder) ? p : 0;
  *threads = kThreads[i];
  *epb = kEpb[i];
}

int batch_default_eo(int p) { return p >= 1 ? 1 : 0; }

int batch_group_setup(BatchGroup& g) {
  int dev = 0, nsm = 0;
  SDG_CUDA_TRY(cudaGetDevice(&dev));
  SDG_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  int per_sm = 0;
  const int st = with_group<GroupOps>(
      g.p, g.eo, [&](auto ops) { return decltype(ops)::setup(g, &per_sm); });
  if (st != SDG_OK) return st;
  if (per_sm <= 0)
    return fail(SDG_ERR_INVALID_ARG, "batch kernel of order %d does not fit: %d threads, %zu B",
                g.p, g.threads, g.smem);
  const long long cap = (long long)nsm * per_sm;
  g.grid = g.eo ? g.count : (int)(g.count < cap ? g.count : cap);
  return SDG_OK;
}

int batch_group_launch(const BatchInst* d_inst, const BatchItem* d_items, const BatchGroup& g,
                       int stage, cudaStream_t st) {
  if (g.count <= 0) return SDG_OK;
  return with_group<GroupOps>(g.p, g.eo, [&](auto ops) {
    return decltype(ops)::launch(d_inst, d_items + g.begin, g, stage, st);
  });
}

BatchForkJoin::~BatchForkJoin() {
  for (cudaStream_t s : streams) cudaStreamDestroy(s);
  for (cudaEvent_t e : done) cudaEventDestroy(e);
  if (fork) cudaEventDestroy(fork);
}

// The three stages as one persistent launch each over every group's items
// (they are contiguous, sorted by order and body), then the index advance.
static int batch_fused_enqueue(BatchInst* d_inst, int n_inst, const BatchItem* d_items,
                               const std::vector<BatchGroup>& groups, cudaStream_t st) {
  int n_items = 0, threads = 32;
  size_t smem = 0;
  for (const BatchGroup& g : groups) {
    n_items = g.begin + g.count > n_items ? g.begin + g.count : n_items;
    SDG_TRY(with_group<GroupOps>(g.p, g.eo, [&](auto ops) {
      threads = std::max(threads, decltype(ops)::threads(g));
      return SDG_OK;
    }));
  }
  for (const BatchGroup& g : groups)
    SDG_TRY(with_group<GroupOps>(g.p, g.eo, [&](auto ops) {
      smem = std::max(smem, decltype(ops)::smem(g, threads));
      return SDG_OK;
    }));
  if (n_items > 0) {
    SDG_TRY(set_kernel_smem((const void*)batch_stage_kernel<kRkFirst>, (int)smem, kCarveDefault));
    SDG_TRY(set_kernel_smem((const void*)batch_stage_kernel<kRkGeneral>, (int)smem, kCarveDefault));
    int dev = 0, nsm = 0, per_sm = 0;
    SDG_CUDA_TRY(cudaGetDevice(&dev));
    SDG_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    SDG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &per_sm, batch_stage_kernel<kRkGeneral>, threads, smem));
    if (per_sm < 1)
      return fail(SDG_ERR_INVALID_ARG, "the single-launch stage kernel does not fit an SM "
                  "(%d threads, %zu bytes of shared memory)", threads, smem);
    const long long cap = (long long)nsm * per_sm;
    const int grid = (int)(n_items < cap ? n_items : cap);
    for (int s = 0; s < 3; s++) {
      if (s == 0)
        batch_stage_kernel<kRkFirst><<<grid, threads, smem, st>>>(d_inst, d_items, n_items, s);
      else
        batch_stage_kernel<kRkGeneral><<<grid, threads, smem, st>>>(d_inst, d_items, n_items, s);
      SDG_CUDA_TRY(cudaGetLastError());
    }
  }
  return batch_advance_launch(d_inst, n_inst, st);
}

int batch_step_enqueue(BatchForkJoin& fj, BatchInst* d_inst, int n_inst,
                       const BatchItem* d_items, const std::vector<BatchGroup>& groups,
                       cudaStream_t st) {
  if (fj.fused) return batch_fused_enqueue(d_inst, n_inst, d_items, groups, st);
  const size_t ng = groups.size();
  if (ng <= 1 || !fj.parallel) {
    for (int s = 0; s < 3; s++)
      for (const BatchGroup& g : groups) SDG_TRY(batch_group_launch(d_inst, d_items, g, s, st));
    return batch_advance_launch(d_inst, n_inst, st);
  }
  if (!fj.fork) SDG_CUDA_TRY(cudaEventCreateWithFlags(&fj.fork, cudaEventDisableTiming));
  while (fj.streams.size() < ng) {
    cudaStream_t s;
    cudaEvent_t e;
    SDG_CUDA_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    fj.streams.push_back(s);
    SDG_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    fj.done.push_back(e);
  }
  SDG_CUDA_TRY(cudaEventRecord(fj.fork, st));
  for (size_t i = 0; i < ng; i++) {
    SDG_CUDA_TRY(cudaStreamWaitEvent(fj.streams[i], fj.fork, 0));
    for (int s = 0; s < 3; s++)
      SDG_TRY(batch_group_launch(d_inst, d_items, groups[i], s, fj.streams[i]));
    SDG_CUDA_TRY(cudaEventRecord(fj.done[i], fj.streams[i]));
    SDG_CUDA_TRY(cudaStreamWaitEvent(st, fj.done[i], 0));
  }
  return batch_advance_launch(d_inst, n_inst, st);
}

int batch_groups(const std::vector<BatchItem>& items, const std::vector<BatchInst>& inst,
                 const int* epb, const int* threads, std::vector<BatchGroup>& groups) {
  groups.clear();
  for (size_t i = 0; i < items.size();) {
    const BatchInst& I = inst[items[i].inst];
    BatchGroup g;
    g.p = I.p;
    g.eo = I.eo;
    g.begin = (int)i;
    size_t j = i;
    while (j < items.size() && inst[items[j].inst].p == g.p && inst[items[j].inst].eo == g.eo)
      j++;
    g.count = (int)(j - i);
    g.threads = threads[g.p];
    g.smem = batch_smem_bytes(g.p, epb[g.p], g.eo);
    g.grid = 0;
    SDG_TRY(batch_group_setup(g));
    groups.push_back(g);
    i = j;
  }
  return SDG_OK;
}

int batch_advance_launch(BatchInst* d_inst, int n_inst, cudaStream_t st) {
  if (n_inst <= 0) return SDG_OK;
  batch_advance_kernel<<<(n_inst + 255) / 256, 256, 0, st>>>(d_inst, n_inst);
  SDG_CUDA_TRY(cudaGetLastError());
  return SDG_OK;
}

int batch_init_blob(const BatchInst& inst, const double* d_x1D, const double centre[3],
                    double sigma, const double vel[3], cudaStream_t st) {
  const int nq = inst.p + 1;
  const long long total = (long long)nq * nq * nq * inst.box.Ne;
  long long nb = (total + 255) / 256;
  if (nb > 152LL * 32) nb = 152LL * 32;
  init_blob_kernel<<<(unsigned)(nb > 0 ? nb : 1), 256, 0, st>>>(
      inst.q[inst.cur], const_cast<float*>(inst.u), const_cast<float*>(inst.v),
      const_cast<float*>(inst.w), d_x1D, inst.box, nq, centre[0], centre[1], centre[2],
      1.0 / (2.0 * sigma * sigma), (float)vel[0], (float)vel[1], (float)vel[2]);
  SDG_CUDA_TRY(cudaGetLastError());
  return SDG_OK;
}

}  // namespace sdg
