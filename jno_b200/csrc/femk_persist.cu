// Jacobi-PCG and BiCGStab as one persistent launch, for systems whose operator stays on the chip
// (femk_persist.cuh).
//
// The chunked solver (femk_cg.cu) runs three kernels an iteration, each with its launch gap, its ramp and a
// last-block reduction: at P1 32^3 (35,937 rows, 5.3 MB of operator) that takes 17.8 us an iteration, 13.3 us of it
// in the kernels.
// Here an iteration is two phases of one kernel, the same floating-point operations as k_update_r /
// k_pupdate_x / the product, in the same order within a row:
//   A  p_i = z_i + beta p_i;  q_i = sum_j a_ij (z_j + beta p_j);  <p, q>                     -> alpha
//   B  x += alpha p;  r -= alpha q;  z = D^-1 r;  <r, z>, <r, r>                                  -> beta, stop test
// The product forms the new direction at every gather from the pair {z_j, p_j} (one 16-byte load), so the
// direction needs no phase, and no barrier, of its own. What is left is bound by the two barriers an iteration
// (4.3 of the 7.3 us at 32^3) and, from 64^3 on, by the gathers and the operator's share that L2 holds. 512
// threads: 768 and 1024 spill at 80 and 64 registers (64^3: 12.0 us an iteration, against 12.9 and 14.3).
// The recurrence q = A z + beta q would gather z alone and gained 5-15 %, but its true residual at tolerances of
// 1e-13 and below was up to 2.5 times larger, so the product keeps the textbook form.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <string>

#include "femk_persist.cuh"

namespace femk {
namespace {

constexpr int kPT = 512;                    // threads of a block, one block per SM
constexpr int kPersistSmem = 220 * 1024;    // dynamic shared memory of a block (227 KB less the static part)
// ... with a 32-bit column an entry (no regular order): the gathers of the pairs then need L1, which is what shared
// memory leaves (us an iteration with 220 / 100 KB: shuffled P1 40^3 14.0 / 9.6; with column tables P1 64^3 11.9 /
// 12.3, P2 18^3 9.6 / 11.8, 34^3 21.3 / 27.1)
constexpr int kPersistSmemWide = 100 * 1024;

struct PersistOut {
  double rr, gamma, atol2, ww, bb;
  int32_t iter, status;
  // a profiled solve, block 0: clock cycles of the products, the updates and the directions; of the whole loop,
  // in cycles and in nanoseconds
  long long cycles[3], loop_cycles, loop_ns;
};

struct PcgArgs {
  const int64_t* sptr;
  const void* cols;  // columns, or the column tables that start at tptr
  const double* svals;
  const int64_t* tptr;
  const int32_t* runs;
  int64_t n, nslices;
  const double* b;
  double* x;
  const double* dinv;
  double2* zp;      // {z, p} of every row: what other blocks gather
  double* work;     // r, p, q (vstride apart) of blocks whose rows do not fit in shared memory
  int64_t vstride;
  GridWords* words;
  int32_t turn, skip;
  long long limit;
  int32_t smem;     // dynamic shared memory of a block
  double tol2, atol2;
  int32_t maxiter, relres, timed;
  PersistOut* out;  // pinned host memory
  int* err;
};

__device__ __forceinline__ long long global_ns() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

template <int SET, typename IDX, bool TAB>
__global__ void __launch_bounds__(kPT, 1) k_pcg_persist(PcgArgs a) {
  extern __shared__ __align__(16) unsigned char ps_smem[];
  constexpr int W = kPT / 32;
  constexpr bool ONE = SET == kOneBlock;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t nsl = (int32_t)a.nslices;
  const int G = (int)gridDim.x, bid = (int)blockIdx.x;
  BlockMatrix<IDX, TAB> m;
  m.s0 = block_slice(a.sptr, nsl, bid, G);
  m.ns = block_slice(a.sptr, nsl, bid + 1, G) - m.s0;
  const int32_t r0 = m.s0 * 32, nr = m.ns * 32;
  // shared memory: slice offsets, the block's x, r, p, q, D^-1 (and the pairs, when one block owns all), slices
  int32_t* off = reinterpret_cast<int32_t*>(ps_smem);
  const int32_t head = offset_bytes<TAB>(m.ns);
  const bool vin = ONE || head + 40 * nr <= a.smem;
  double* vec = reinterpret_cast<double*>(ps_smem + head);
  double* xs = vin ? vec : a.x + r0;
  double* rs = vin ? vec + nr : a.work + r0;
  double* ps = vin ? vec + 2 * nr : a.work + a.vstride + r0;
  double* qs = vin ? vec + 3 * nr : a.work + 2 * a.vstride + r0;
  const double* ds = vin ? vec + 4 * nr : a.dinv + r0;  // not read without a preconditioner
  double2* zps = reinterpret_cast<double2*>(vec + 5 * nr);
  unsigned char* mat = ONE ? reinterpret_cast<unsigned char*>(zps + nr)
                           : reinterpret_cast<unsigned char*>(vec + (vin ? 5 * nr : 0));
  if (SET == kGrid && bid == 0 && threadIdx.x == 0) a.words->counter[a.turn ^ 1][0] = 0u;
  hold_slices<kPT>(m, a.sptr, a.cols, a.svals, a.tptr, a.runs, off, mat, a.smem - (int32_t)(mat - ps_smem));
  BlockSum<SET, kPT> grid(a.words, a.turn, a.limit, a.skip, bid, G);
  // r = b - A x0, z = D^-1 r
  // gathers of x and of the pairs, range-checked in the bounds-checked build
  auto xat = [&](int32_t j) { return FEMK_IN_BOUNDS(j, a.n, a.err) ? __ldcg(a.x + j) : 0.0; };
  double acc[3] = {0.0, 0.0, 0.0};
  for (int32_t s = warp; s < m.ns; s += W) {
    const int32_t i = s * 32 + lane, row = r0 + i;
    if (row >= a.n) continue;
    const double ax = block_row(m, s, lane, row, xat);
    const double bi = __ldg(a.b + row);
    const double ri = bi - ax;
    const double di = a.dinv ? __ldg(a.dinv + row) : 1.0;
    const double zi = a.dinv ? di * ri : ri;
    rs[i] = ri;
    if (vin) vec[4 * nr + i] = di;
    ps[i] = 0.0;
    if (ONE)
      zps[i] = make_double2(zi, 0.0);
    else
      a.zp[row] = make_double2(zi, 0.0);
    acc[0] += ri * zi;
    acc[1] += ri * ri;
    acc[2] += bi * bi;
  }
  if (vin)
    for (int32_t i = threadIdx.x; i < nr; i += kPT)
      if (r0 + i < a.n) xs[i] = a.x[r0 + i];
  bool live = grid.template sum<3>(acc);
  double gamma = acc[0], rr = acc[1], beta = 0.0;
  const double bb = acc[2], atol2 = fmax(a.tol2 * bb, a.atol2);
  int32_t status = isfinite(gamma) && isfinite(rr) ? FEMK_OK : FEMK_NONFINITE;
  int32_t iter = 0;
  bool done = !((a.dinv ? rr : gamma) > atol2) || a.maxiter <= 0 || status != FEMK_OK;
  long long t0 = 0, ns0 = 0, spent[3] = {0, 0, 0}, first = 0;
  if (a.timed) {
    first = t0 = clock64();
    ns0 = global_ns();
  }
  auto lap = [&](int k) {
    const long long t = clock64();
    spent[k] += t - t0;
    t0 = t;
  };
  auto direction = [&](int32_t i) { return fma(beta, ps[i], a.dinv ? ds[i] * rs[i] : rs[i]); };
  while (live && !done) {
    double pq[1] = {0.0};
    if (a.timed) {  // a profiled solve forms the directions in a pass of their own (the same bits)
      for (int32_t i = warp * 32 + lane; i < nr; i += kPT)
        if (r0 + i < a.n) ps[i] = direction(i);
      lap(2);
    }
    for (int32_t s = warp; s < m.ns; s += W) {
      const int32_t i = s * 32 + lane, row = r0 + i;
      if (row >= a.n) continue;
      const double qi = block_row(m, s, lane, row, [&](int32_t j) {
        if (!FEMK_IN_BOUNDS(j, a.n, a.err)) return 0.0;
        const double2 v = ONE ? zps[j] : a.zp[j];
        return fma(beta, v.y, v.x);
      });
      const double pi = a.timed ? ps[i] : direction(i);
      ps[i] = pi;
      qs[i] = qi;
      pq[0] += pi * qi;
    }
    live = grid.template sum<1>(pq);
    if (a.timed) lap(0);
    if (!live) break;
    if (!(pq[0] > 0.0) || !isfinite(pq[0])) {
      status = isfinite(pq[0]) ? FEMK_BREAKDOWN : FEMK_NONFINITE;
      break;
    }
    const double alpha = gamma / pq[0];
    double rz[2] = {0.0, 0.0};
    for (int32_t s = warp; s < m.ns; s += W) {
      const int32_t i = s * 32 + lane, row = r0 + i;
      if (row >= a.n) continue;
      const double pi = ps[i];
      xs[i] = fma(alpha, pi, xs[i]);
      const double ri = fma(-alpha, qs[i], rs[i]);
      const double zi = a.dinv ? ds[i] * ri : ri;
      rs[i] = ri;
      if (ONE)
        zps[i] = make_double2(zi, pi);
      else
        a.zp[row] = make_double2(zi, pi);
      rz[0] += ri * zi;
      rz[1] += ri * ri;
    }
    live = grid.template sum<2>(rz);
    if (a.timed) lap(1);
    beta = rz[0] / gamma;
    gamma = rz[0];
    rr = rz[1];
    ++iter;
    if (!isfinite(gamma) || !isfinite(rr)) {
      status = FEMK_NONFINITE;
      done = true;
    } else {
      done = !((a.dinv ? rr : gamma) > atol2) || iter >= a.maxiter;
    }
  }
  const long long last = t0, ns1 = a.timed ? global_ns() : 0;
  if (vin) {
    __syncthreads();
    for (int32_t i = threadIdx.x; i < nr; i += kPT)
      if (r0 + i < a.n) a.x[r0 + i] = xs[i];
  }
  double w2[1] = {0.0};
  if (live && a.relres) {  // <b - A x, b - A x> of the returned x
    double none[1] = {0.0};
    live = grid.template sum<1>(none);
    for (int32_t s = warp; s < m.ns; s += W) {
      const int32_t row = r0 + s * 32 + lane;
      if (row >= a.n) continue;
      const double wi = __ldg(a.b + row) - block_row(m, s, lane, row, xat);
      w2[0] += wi * wi;
    }
    if (live) live = grid.template sum<1>(w2);
  }
  grid.leave();
  if (bid == 0 && threadIdx.x == 0) {
    a.out->rr = rr;
    a.out->gamma = gamma;
    a.out->atol2 = atol2;
    a.out->ww = w2[0];
    a.out->bb = bb;
    a.out->iter = iter;
    a.out->status = live ? status : FEMK_TIMEOUT;
    for (int k = 0; k < 3; ++k) a.out->cycles[k] = spent[k];
    a.out->loop_cycles = last - first;
    a.out->loop_ns = ns1 - ns0;
  }
}

struct BicgArgs {
  const int64_t* sptr;
  const void* cols;  // columns, or the column tables that start at tptr
  const double* svals;
  const int64_t* tptr;
  const int32_t* runs;
  int64_t n, nslices;
  const double* b;
  double* x;
  const double* dinv;
  double *phat, *shat;  // what other blocks gather
  double* work;         // r, rhat, p, q, s, t (vstride apart) of blocks whose rows do not fit in shared memory
  int64_t vstride;
  GridWords* words;
  int32_t turn, skip;
  long long limit;
  int32_t smem;
  double tol2, atol2;
  int32_t maxiter;
  BicgResult* out;  // pinned host memory
  int* err;
};

// BiCGStab with the steps, operands and stop rule of femk_bicgstab.cu: per iteration the direction (a barrier, the
// others gather phat), q = A phat with <rhat, q>, s and shat with <s, s>, t = A shat with <t, s> and <t, t>, and
// the x and r updates with <r, r> and <rhat, r>: four sums and one barrier. The chunked solver's five kernels took
// 36.5 us an iteration at 2-D P2 131x118 (62,331 rows, vertices in no order), 19.4 us here, 10.5 of them in the five
// waits; at P1 44x40x47 a Crank-Nicolson march of 12 steps went from 14.6 to 6.9 ms.
template <int SET, typename IDX, bool TAB>
__global__ void __launch_bounds__(kPT, 1) k_bicg_persist(BicgArgs a) {
  extern __shared__ __align__(16) unsigned char ps_smem[];
  constexpr int W = kPT / 32;
  constexpr bool ONE = SET == kOneBlock;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int32_t nsl = (int32_t)a.nslices;
  const int G = (int)gridDim.x, bid = (int)blockIdx.x;
  BlockMatrix<IDX, TAB> m;
  m.s0 = block_slice(a.sptr, nsl, bid, G);
  m.ns = block_slice(a.sptr, nsl, bid + 1, G) - m.s0;
  const int32_t r0 = m.s0 * 32, nr = m.ns * 32;
  // shared memory: slice offsets, the block's x, r, rhat, p, q, s, t, D^-1 (and phat, shat of one block), slices
  int32_t* off = reinterpret_cast<int32_t*>(ps_smem);
  const int32_t head = offset_bytes<TAB>(m.ns);
  const bool vin = ONE || head + 64 * nr <= a.smem;
  double* vec = reinterpret_cast<double*>(ps_smem + head);
  auto slot = [&](int k) { return vin ? vec + (k + 1) * nr : a.work + k * a.vstride + r0; };
  double* xs = vin ? vec : a.x + r0;
  double *rs = slot(0), *hs = slot(1), *ps = slot(2), *qs = slot(3), *ss = slot(4), *ts = slot(5);
  const double* ds = vin ? vec + 7 * nr : a.dinv + r0;  // not read without a preconditioner
  double* phat = ONE ? vec + 8 * nr : a.phat;
  double* shat = ONE ? vec + 9 * nr : a.shat;
  unsigned char* mat = reinterpret_cast<unsigned char*>(vec + (ONE ? 10 * nr : (vin ? 8 * nr : 0)));
  if (SET == kGrid && bid == 0 && threadIdx.x == 0) a.words->counter[a.turn ^ 1][0] = 0u;
  hold_slices<kPT>(m, a.sptr, a.cols, a.svals, a.tptr, a.runs, off, mat, a.smem - (int32_t)(mat - ps_smem));
  BlockSum<SET, kPT> grid(a.words, a.turn, a.limit, a.skip, bid, G);
  auto xat = [&](int32_t j) { return FEMK_IN_BOUNDS(j, a.n, a.err) ? __ldcg(a.x + j) : 0.0; };
  // body(local row, row) for every row of the block that this thread owns
  auto rows = [&](auto&& body) {
    for (int32_t s = warp; s < m.ns; s += W) {
      const int32_t i = s * 32 + lane, row = r0 + i;
      if (row < a.n) body(s, i, row);
    }
  };
  double acc[2] = {0.0, 0.0};
  rows([&](int32_t s, int32_t i, int32_t row) {
    const double bi = __ldg(a.b + row);
    const double ri = bi - block_row(m, s, lane, row, xat);
    rs[i] = ri;
    hs[i] = ri;
    ps[i] = ri;
    qs[i] = ri;
    if (vin) {
      xs[i] = a.x[row];
      vec[7 * nr + i] = a.dinv ? __ldg(a.dinv + row) : 1.0;
    }
    acc[0] += ri * ri;
    acc[1] += bi * bi;
  });
  bool live = grid.template sum<2>(acc);
  double rr = acc[0], rho_n = acc[0], bb = acc[1];
  const double atol2 = fmax(a.tol2 * bb, a.atol2);
  double rho = 1.0, alpha = 1.0, omega = 1.0;
  int32_t k = 0, iters = 0, status = isfinite(rr) && isfinite(bb) ? FEMK_OK : FEMK_NONFINITE;
  bool done = status != FEMK_OK || !(rr > atol2) || a.maxiter <= 0;
  while (live && !done) {
    const double beta = rho_n / rho * alpha / omega;
    rows([&](int32_t, int32_t i, int32_t row) {
      const double pi = rs[i] + beta * (ps[i] - omega * qs[i]);
      ps[i] = pi;
      phat[row] = a.dinv ? ds[i] * pi : pi;
    });
    if (!(live = grid.barrier())) break;
    double v1[1] = {0.0};
    rows([&](int32_t s, int32_t i, int32_t row) {
      const double qi = block_row(m, s, lane, row, [&](int32_t j) {
        return FEMK_IN_BOUNDS(j, a.n, a.err) ? phat[j] : 0.0;
      });
      qs[i] = qi;
      v1[0] += hs[i] * qi;
    });
    if (!(live = grid.template sum<1>(v1))) break;
    alpha = rho_n / v1[0];
    v1[0] = 0.0;
    rows([&](int32_t, int32_t i, int32_t row) {
      const double si = rs[i] - alpha * qs[i];
      ss[i] = si;
      shat[row] = a.dinv ? ds[i] * si : si;
      v1[0] += si * si;
    });
    if (!(live = grid.template sum<1>(v1))) break;
    const bool early = v1[0] < atol2;
    double v2[2] = {0.0, 0.0};
    rows([&](int32_t s, int32_t i, int32_t row) {
      const double ti = block_row(m, s, lane, row, [&](int32_t j) {
        return FEMK_IN_BOUNDS(j, a.n, a.err) ? shat[j] : 0.0;
      });
      ts[i] = ti;
      v2[0] += ti * ss[i];
      v2[1] += ti * ti;
    });
    if (!(live = grid.template sum<2>(v2))) break;
    omega = v2[0] / v2[1];
    v2[0] = v2[1] = 0.0;
    rows([&](int32_t, int32_t i, int32_t) {
      const double si = ss[i];
      const double ph = a.dinv ? ds[i] * ps[i] : ps[i];
      double ri;
      if (early) {
        xs[i] = xs[i] + alpha * ph;
        ri = si;
      } else {
        const double sh = a.dinv ? ds[i] * si : si;
        xs[i] = xs[i] + (alpha * ph + omega * sh);
        ri = si - omega * ts[i];
      }
      rs[i] = ri;
      v2[0] += ri * ri;
      v2[1] += hs[i] * ri;
    });
    if (!(live = grid.template sum<2>(v2))) break;
    ++iters;
    k = rho_n == 0.0 ? -10 : (omega == 0.0 || alpha == 0.0 ? -11 : k + 1);
    rho = rho_n;
    rho_n = v2[1];
    rr = v2[0];
    if (!isfinite(rr) || !isfinite(rho_n)) {
      status = FEMK_NONFINITE;
      done = true;
    } else {
      done = !(rr > atol2) || k >= a.maxiter || k < 0;
    }
  }
  if (vin) rows([&](int32_t, int32_t i, int32_t row) { a.x[row] = xs[i]; });
  double w2[1] = {0.0};  // the true residual of the returned x
  if (live) live = grid.barrier();
  if (live) {
    rows([&](int32_t s, int32_t, int32_t row) {
      const double wi = __ldg(a.b + row) - block_row(m, s, lane, row, xat);
      w2[0] += wi * wi;
    });
    live = grid.template sum<1>(w2);
  }
  grid.leave();
  if (bid == 0 && threadIdx.x == 0) {
    a.out->rr = rr;
    a.out->ss = w2[0];
    a.out->atol2 = atol2;
    a.out->bb = bb;
    a.out->k = k;
    a.out->iters = iters;
    a.out->status = live ? status : FEMK_TIMEOUT;
  }
}

constexpr int kNoCluster = -1;  // launch_columns: the device holds no such cluster, nothing was launched

// The launch of co-resident blocks (a cluster, or a cooperative grid).
void launch_config(int set, int grid, int smem, cudaStream_t s, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
  cfg->gridDim = dim3(grid);
  cfg->blockDim = dim3(kPT);
  cfg->dynamicSmemBytes = (size_t)smem;
  cfg->stream = s;
  cfg->attrs = at;
  cfg->numAttrs = set == kOneBlock ? 0 : 1;
  if (set == kOneCluster) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = grid;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  } else if (set == kGrid) {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
}

// One launch of a persistent kernel.
template <typename Args>
int launch_set(void (*kern)(Args), int set, int grid, const Args& a, cudaStream_t s) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[1];
  launch_config(set, grid, a.smem, s, &cfg, at);
  counted_launch();
  FEMK_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, a));
  return FEMK_OK;
}

// shared-memory limit and cluster size of a kernel, set once per device
template <typename Args>
int prepare_kernel(void (*kern)(Args), int set, int device, std::atomic<uint64_t>& ready) {
  const uint64_t bit = 1ull << (device & 63);
  if (ready.load(std::memory_order_acquire) & bit) return FEMK_OK;
  FEMK_CUDA_TRY(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPersistSmem));
  if (set == kOneCluster)
    FEMK_CUDA_TRY(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  ready.fetch_or(bit, std::memory_order_release);
  return FEMK_OK;
}

template <int SET, typename IDX, bool TAB>
struct PcgKernel {
  static constexpr auto fn = k_pcg_persist<SET, IDX, TAB>;
};
template <int SET, typename IDX, bool TAB>
struct BicgKernel {
  static constexpr auto fn = k_bicg_persist<SET, IDX, TAB>;
};

template <template <int, typename, bool> class K, int SET, typename IDX, bool TAB, typename Args>
int launch_kernel(const femk_plan* p, const Args& a, int grid, cudaStream_t s) {
  static std::atomic<uint64_t> ready{0};
  FEMK_TRY(prepare_kernel(K<SET, IDX, TAB>::fn, SET, p->device, ready));
  // Whether the device holds a cluster of so many blocks (more than 8, or any with this much shared memory, are not
  // promised: a part of a GPU may not). Asked once per device and size, a bit for "asked", one for the answer.
  if constexpr (SET == kOneCluster) {
    static std::atomic<uint32_t> known[64];
    std::atomic<uint32_t>& k = known[p->device & 63];
    const uint32_t bit = (uint32_t)grid;  // 2, 4, 8 or 16
    if (!(k.load(std::memory_order_acquire) & bit)) {
      int fit = 0;
      cudaLaunchConfig_t cfg{};
      cudaLaunchAttribute at[1];
      launch_config(SET, grid, a.smem, s, &cfg, at);
      if (cudaOccupancyMaxActiveClusters(&fit, K<SET, IDX, TAB>::fn, &cfg) != cudaSuccess) {
        cudaGetLastError();
        fit = 0;
      }
      k.fetch_or(bit | (fit > 0 ? bit << 16 : 0u), std::memory_order_release);
    }
    if (!(k.load(std::memory_order_acquire) & (bit << 16))) return kNoCluster;
  }
  return launch_set(K<SET, IDX, TAB>::fn, SET, grid, a, s);
}

template <template <int, typename, bool> class K, int SET, typename Args>
int launch_columns(const femk_plan* p, const Args& a, int grid, cudaStream_t s) {
  if (p->sell_cu) return launch_kernel<K, SET, int16_t, true>(p, a, grid, s);
  if (p->sell_ct) return launch_kernel<K, SET, int32_t, true>(p, a, grid, s);
  if (p->sell_c16) return launch_kernel<K, SET, int16_t, false>(p, a, grid, s);
  return launch_kernel<K, SET, int32_t, false>(p, a, grid, s);
}

// The launch of kernel K for the plan. One block, with no wait for others, when all of it fits one SM
// (one_row: bytes of vectors a row takes there). Then one cluster of up to 16 blocks: its barrier is twice as fast
// as the grid's, until 16 SMs take longer over the rows than that gains (CG, us an iteration, cluster against
// grid: 2-D P1 100^2, 319 slices, 4.1 / 5.7; P1 20x22x24, 378 slices, 5.8 / 7.0; 2-D P2 60^2, 458 slices, 6.3 /
// 6.9; 2-D P2 70^2, 622 slices, 7.0 / 6.7; P1 28^3, 763 slices, 8.4 / 7.2). Then a grid of 16 slices a block, a
// slice a warp, at most a block an SM (P1 32^3, 1,124 slices: 71 blocks; the wait takes the same for 148), which also
// serves devices that hold no such cluster.
template <template <int, typename, bool> class K, typename Args>
int launch_persist(femk_plan* p, Args& a, int one_row, cudaStream_t s) {
  a.sptr = p->sell_ptr;
  a.cols = p->sell_cu   ? (const void*)p->sell_cu
           : p->sell_ct ? (const void*)p->sell_ct
                        : (p->sell_c16 ? (const void*)p->sell_c16 : (const void*)p->sell_cols);
  a.tptr = p->sell_cu ? p->sell_cuptr : p->sell_ctptr;
  a.runs = p->sell_runs;
  a.svals = p->sell_vals;
  a.n = p->n;
  a.nslices = p->n_slices;
  a.vstride = p->vstride;
  a.words = (GridWords*)p->persist_words;
  a.turn = p->persist_turn;
  a.skip = p->skip_arrival;
  a.limit = p->barrier_spin;
  a.smem = p->sell_c16 || p->sell_ct ? kPersistSmem : kPersistSmemWide;
  a.err = p->dev_err;
  const int64_t one = 4 * (3 * p->n_slices + 2) + 16 + p->n_slices * 32 * one_row + operator_bytes(p);
  if (one <= a.smem) return launch_columns<K, kOneBlock>(p, a, 1, s);
  if (p->n_slices <= 32 * kMaxCluster) {
    int grid = 2;
    while (grid < kMaxCluster && grid * 16 < p->n_slices) grid *= 2;
    const int rc = launch_columns<K, kOneCluster>(p, a, grid, s);
    if (rc != kNoCluster) return rc;
  }
  const int grid = (int)std::min<int64_t>(std::min(p->n_sm, kMaxBlocks), (p->n_slices + 15) / 16);
  FEMK_TRY((launch_columns<K, kGrid>(p, a, grid, s)));
  p->persist_turn ^= 1;
  return FEMK_OK;
}

// One allocation for all of the solver's global memory: the pairs, the vectors of blocks whose rows do not fit
// in shared memory, and the grid's words (zeroed on the stream that the launch goes to: another one's clearing could
// come during the solve).
int ensure_persist(femk_plan* p, cudaStream_t s) {
  if (!p->persist_ws) {
    const size_t vec = sizeof(double) * 5 * (size_t)p->vstride;
    char* ws = nullptr;
    FEMK_CUDA_TRY(cudaMalloc(&ws, vec + sizeof(GridWords)));
    const cudaError_t e = cudaMemsetAsync(ws + vec, 0, sizeof(GridWords), s);
    if (e != cudaSuccess) cudaFree(ws);
    FEMK_CUDA_TRY(e);
    p->persist_ws = ws;
    p->persist_words = ws + vec;
  }
  if (!p->persist_out) FEMK_CUDA_TRY(cudaMallocHost(&p->persist_out, sizeof(PersistOut)));
  return FEMK_OK;
}

}  // namespace

// Bytes of the sliced-ELL operator: what every iteration reads.
int64_t operator_bytes(const femk_plan* p) {
  if (p->sell_cu) return 8 * p->sell_nnz + 2 * p->sell_cu_len;
  if (p->sell_ct) return 8 * p->sell_nnz + 4 * p->sell_ct_len;
  return p->sell_nnz * (p->sell_c16 ? 10 : 12);
}

// Whether the slices' columns mostly are those of runs of rows (femk_order.cu), not one an entry.
bool columns_shared(const femk_plan* p) {
  return (p->sell_cu && 4 * p->sell_cu_len < p->sell_nnz) || (p->sell_ct && 4 * p->sell_ct_len < p->sell_nnz);
}

// The single launch wins while what an iteration touches stays on the chip: the operator, and 134 B a row of vectors
// and gathered pairs (fitted: the sizes at which both forms take the same agree on it from 7 to 65 entries a row).
// Past that its 16 warps an SM wait for HBM where the chunked solver's 64 stream. Columns of their own an entry (no
// runs) lower the limit: the gathers spread, and more of them miss L1. B200, FP64, us an iteration, chunked -> single
// launch (MB touched), CG | BiCGStab:
//   shared columns    P1 32^3 17.4 -> 7.3 (9), 64^3 21.4 -> 12.0, 84^3 30.1 -> 20.1 (156), 86^3 31.8 -> 22.9 (167),
//                     88^3 32.8 -> 36.3 (179); P2 35^3 32.8 -> 22.6 (132); 2-D P1 900^2 26.0 -> 23.2 (155), 930^2
//                     27.1 -> 26.4 (165), 960^2 28.0 -> 30.1 (176), 1100^2 34.1 -> 51.6 (231); 2-D P2 415^2
//                     30.2 -> 23.2 (158), 430^2 31.3 -> 31.4 (170), 460^2 33.8 -> 48.0 (194)
//                   | P1 80^3 60 -> 45 (135), 84^3 64 -> 62 (156), 88^3 70 -> 88 (179); P2 35^3 64 -> 43 (132);
//                     2-D P1 850^2 55 -> 47 (138), 900^2 58 -> 59 (155), 960^2 64 -> 75 (176); 2-D P2 400^2
//                     61.6 -> 58.6 (147), 415^2 62 -> 65 (158)
//   own columns, P1   shuffled 40^3 26.5 -> 9.5 (21), 76^3 66 -> 44 (143), 2-D 800^2 51 -> 33 (140); shuffled within
//                     512 vertices 74^3 31.0 -> 29.0 (119), 80^3 36.6 -> 35.8 (150), 2-D 850^2 30.4 -> 28.6 (148),
//                     900^2 32.5 -> 41.1 (166)
//                   | shuffled 73^3 86 -> 78 (127), 76^3 90 -> 97 (143), 2-D 700^2 63 -> 54 (107), 800^2 74 -> 78
//                     (140); within 512 vertices 74^3 65 -> 42 (119), 78^3 72 -> 77 (140)
//   own columns, P2   shuffled 29^3 39.5 -> 31.5 (106), 2-D 320^2 34.9 -> 31.5 (112), 340^2 36.5 -> 37.5 (126),
//                     385^2 42.7 -> 55.4 (162)
//                   | shuffled 29^3 101 -> 64 (106), 2-D 320^2 73 -> 68 (112), 340^2 74 -> 88 (126)
// The operator alone is held to kPersistBytes as well: no system above it was measured to gain.
bool persist_fits(const femk_plan* p, bool bicg) {
  if (!p->persist_ok || !p->coop || !p->use_sell || !p->sell_cols || operator_bytes(p) > kPersistBytes) return false;
  const double touched = (double)operator_bytes(p) + 134.0 * (double)p->n;
  const double limit = columns_shared(p) ? (bicg ? 150e6 : 173e6)
                       : p->order == 1   ? (bicg ? 130e6 : 147e6)
                                         : (bicg ? 115e6 : 118e6);
  return touched <= limit;
}

bool pcg_persist_fits(const femk_plan* p) { return persist_fits(p, false); }

int pcg_persist(const femk_plan* pc, const double* vals, const double* b, double* x, const double* dinv, double tol,
                double atol, int32_t maxiter, int32_t* iters_out, double* relres_out, cudaStream_t s) {
  femk_plan* p = const_cast<femk_plan*>(pc);
  FEMK_TRY(ensure_persist(p, s));
  FEMK_TRY(ensure_sell_values(p, false));
  FEMK_TRY(launch_sell_values(p, vals, false, s));
  PersistOut* out = (PersistOut*)p->persist_out;
  out->status = FEMK_TIMEOUT;
  PcgArgs a{};
  a.b = b;
  a.x = x;
  a.dinv = dinv;
  a.zp = (double2*)p->persist_ws;
  a.work = (double*)p->persist_ws + 2 * p->vstride;
  a.tol2 = tol * tol;
  a.atol2 = atol * atol;
  a.maxiter = maxiter;
  a.relres = relres_out != nullptr;
  ProfData* pd = (ProfData*)p->prof;
  a.timed = pd != nullptr;
  a.out = out;
  FEMK_TRY(launch_persist<PcgKernel>(p, a, 56, s));
  FEMK_CUDA_TRY(cudaStreamSynchronize(s));
  if (iters_out) *iters_out = out->iter;
  if (relres_out) *relres_out = std::sqrt(out->ww) / (std::sqrt(out->bb) + 1e-30);
  if (pd && out->loop_cycles > 0) {
    const double ms = 1e-6 * (double)out->loop_ns / (double)out->loop_cycles;  // per cycle
    for (int k = 0; k < 3; ++k) pd->ms[k] += ms * (double)out->cycles[k];
    pd->iters += out->iter;
  }
  switch (out->status) {
    case FEMK_BREAKDOWN:
      set_error("femk_pcg: <p, A p> <= 0 (operator not symmetric positive definite)");
      return FEMK_BREAKDOWN;
    case FEMK_NONFINITE:
      set_error("femk_pcg: non-finite value in a CG reduction");
      return FEMK_NONFINITE;
    case FEMK_TIMEOUT:
      set_error("femk_pcg: a grid-wide wait of the persistent solver gave up");
      return FEMK_TIMEOUT;
    default:
      break;
  }
  FEMK_TRY(check_bounds(p, s, "femk_pcg"));
  if ((dinv ? out->rr : out->gamma) > out->atol2) {
    set_error("femk_pcg: iteration cap reached above tolerance");
    return FEMK_NOT_CONVERGED;
  }
  return FEMK_OK;
}

bool bicg_persist_fits(const femk_plan* p) { return persist_fits(p, true); }

int bicg_persist(femk_plan* p, const double* b, double* x, const double* dinv, double* ws, double tol, double atol,
                 int32_t maxiter, cudaStream_t s, BicgResult* out) {
  FEMK_TRY(ensure_persist(p, s));
  out->status = FEMK_TIMEOUT;
  BicgArgs a{};
  a.b = b;
  a.x = x;
  a.dinv = dinv;
  a.phat = ws;
  a.shat = ws + p->vstride;
  a.work = ws + 2 * p->vstride;
  a.tol2 = tol * tol;
  a.atol2 = atol * atol;
  a.maxiter = maxiter;
  a.out = out;
  FEMK_TRY(launch_persist<BicgKernel>(p, a, 80, s));
  FEMK_CUDA_TRY(cudaStreamSynchronize(s));
  return check_bounds(p, s, "femk_bicgstab");
}

}  // namespace femk
