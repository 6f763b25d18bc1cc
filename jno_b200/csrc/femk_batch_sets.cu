// Batched Jacobi-PCG, a problem to a set of blocks of its own (femk_persist.cuh): the problems do not wait for one
// another.
//
// The grid form (femk_batch.cu) advances all problems together: every iteration streams the operators of all that are
// still running from HBM, and its four grid barriers and two owner passes take 11 us. Here a set of blocks (a block,
// a cluster, or a group of a cooperative grid) takes the next problem of a queue, largest first, solves it alone and
// takes another. What is in flight is a problem a set, whose operators stay in shared memory and L2 from one iteration
// to the next, and an iteration's two barriers are the set's own (0.7-1.0 us in a cluster). 96 P1 cubes of sides 8 to
// 48 (2.2M rows, 306M row-iterations), the solve alone: 18.2 -> 10.1 ms; bound by the latency of a row's loads at 16
// warps an SM.
// The steps are those of the grid form (q = A p by the recurrence w + beta q, z the only vector that other blocks
// gather), its sums in another order:
//   A  w = A z, p = z + beta p, q = w + beta q, <p, q>      -> alpha
//   B  x += alpha p, r -= alpha q, z = D^-1 r, <r, z>, <r, r>   -> beta, stop test
// Of the block's parts of p, q, r, x and D^-1 as many as fit stay in shared memory, in that order (accesses an
// iteration: 3, 3, 3, 2, 1 of 8 bytes; an entry of the operator is read once, so the vectors come before it).
#include <algorithm>
#include <cmath>
#include <numeric>
#include <vector>

#include "femk_persist.cuh"

namespace femk {
namespace {

constexpr int kCT = 512;  // threads of a block, one block per SM
// rows in flight a thread in the updates (ms with 1 / 2 / 4: 96 cubes of sides 8 to 48 10.28 / 10.07 / 10.31, 9 x 48^3
// 6.16 / 6.11 / 6.21, 12 x 64^3 24.5 / 24.2 / 24.9)
constexpr int kUnroll = 2;
constexpr int kSetSmem = 220 * 1024;

struct BatchOut {
  double relres;
  int32_t iter, status;
};

struct SetArgs {
  const int64_t* sptr;
  const void* cols;  // columns, or the column tables that start at tptr
  const double* svals;
  const int64_t* tptr;
  const int32_t* runs;
  unsigned int* queue;   // problems taken
  const int32_t* order;  // [nprob] problems of this launch by falling size
  const int32_t* off;    // first row of every problem of the batch, and the end
  int32_t nprob;
  int32_t group;         // kGrid: blocks of a group
  GridWords* words;      // kGrid: a group's words each, zeroed
  long long limit;
  int32_t skip;          // kGrid, testing: the block of a group that never arrives (-1: none)
  const double* b;
  double* x;
  const double* dinv;
  double* z;     // what other blocks gather
  double* work;  // p, q, r (vstride apart) of blocks whose rows do not fit in shared memory
  int64_t vstride;
  int32_t smem;  // dynamic shared memory of a block
  double tol2, atol2;
  int32_t maxiter;
  BatchOut* out;
};

template <int SET, typename IDX, bool TAB>
__global__ void __launch_bounds__(kCT, 1) k_batch_sets(SetArgs a) {
  extern __shared__ __align__(16) unsigned char bc_smem[];
  constexpr int W = kCT / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int C = SET == kOneBlock ? 1 : (SET == kOneCluster ? (int)cluster_size() : a.group);
  const int me = SET == kOneBlock ? 0 : (SET == kOneCluster ? (int)cluster_rank() : (int)blockIdx.x % a.group);
  BlockSum<SET, kCT> all(SET == kGrid ? a.words + blockIdx.x / a.group : nullptr, 0, a.limit, a.skip, me, C);
  for (;;) {
    // the next problem; the sum tells every block (whole numbers below 2^53 are exact)
    double next[1] = {me == 0 && threadIdx.x == 0 ? (double)atomicAdd(a.queue, 1u) : 0.0};
    if (!all.template sum<1>(next)) return;
    if (next[0] >= (double)a.nprob) break;
    const int32_t k = __ldg(a.order + (int32_t)next[0]);
    const int32_t lo = __ldg(a.off + k), hi = __ldg(a.off + k + 1);
    // its slices: the first and the last may hold rows of its neighbours too
    const int32_t first = lo >> 5, slices = ((hi - 1) >> 5) - first + 1;
    BlockMatrix<IDX, TAB> m;
    const int32_t b0 = block_slice(a.sptr + first, slices, me, C);
    m.s0 = first + b0;
    m.ns = block_slice(a.sptr + first, slices, me + 1, C) - b0;
    const int32_t r0 = m.s0 * 32, nr = m.ns * 32;
    // shared memory: slice offsets, the vectors that fit, slices
    int32_t* offs = reinterpret_cast<int32_t*>(bc_smem);
    const int32_t head = offset_bytes<TAB>(m.ns);
    const int32_t held = nr ? min(5, (a.smem - head) / (8 * nr)) : 0;
    double* vec = reinterpret_cast<double*>(bc_smem + head);
    double* ps = held > 0 ? vec : a.work + r0;
    double* qs = held > 1 ? vec + nr : a.work + a.vstride + r0;
    double* rs = held > 2 ? vec + 2 * nr : a.work + 2 * a.vstride + r0;
    double* xs = held > 3 ? vec + 3 * nr : a.x + r0;
    const double* ds = held > 4 ? vec + 4 * nr : a.dinv + r0;  // not read without a preconditioner
    unsigned char* mat = reinterpret_cast<unsigned char*>(vec + held * nr);
    hold_slices<kCT>(m, a.sptr, a.cols, a.svals, a.tptr, a.runs, offs, mat, a.smem - (int32_t)(mat - bc_smem));
    // body(slice, local row, row) for every row of the problem that this thread owns
    auto rows = [&](auto&& body) {
      for (int32_t s = warp; s < m.ns; s += W) {
        const int32_t i = s * 32 + lane, row = r0 + i;
        if (row >= lo && row < hi) body(s, i, row);
      }
    };
    // A padding entry (value 0) of a table may name a row of another problem, whose vectors hold anything: row lo is
    // read instead (a select; as a load under a condition the 96 cubes took 18.7 ms in place of 9.9).
    auto own = [&](int32_t j) { return (uint32_t)(j - lo) < (uint32_t)(hi - lo) ? j : lo; };
    auto xat = [&](int32_t j) { return __ldcg(a.x + own(j)); };
    auto zat = [&](int32_t j) { return a.z[own(j)]; };
    // r = b - A x0, z = D^-1 r
    double acc[3] = {0.0, 0.0, 0.0};
    rows([&](int32_t s, int32_t i, int32_t row) {
      const double ax = block_row(m, s, lane, row, xat);
      const double bi = __ldg(a.b + row), di = a.dinv ? __ldg(a.dinv + row) : 1.0;
      const double ri = bi - ax, zi = a.dinv ? di * ri : ri;
      rs[i] = ri;
      a.z[row] = zi;
      if (held > 3) xs[i] = a.x[row];
      if (held > 4) vec[4 * nr + i] = di;
      acc[0] += ri * zi;
      acc[1] += ri * ri;
      acc[2] += bi * bi;
    });
    if (!all.template sum<3>(acc)) return;  // out of time: the problem keeps the status FEMK_TIMEOUT
    double gamma = acc[0], rr = acc[1], beta = 0.0;  // the first direction is z itself
    const double atol2 = fmax(a.tol2 * acc[2], a.atol2);
    int32_t status = isfinite(gamma) && isfinite(rr) ? FEMK_OK : FEMK_NONFINITE;
    int32_t iter = 0;
    bool done = status != FEMK_OK || !((a.dinv ? rr : gamma) > atol2) || a.maxiter <= 0;
    while (!done) {
      double pq[1] = {0.0};
      const bool step = beta != 0.0;
      rows([&](int32_t s, int32_t i, int32_t row) {
        const double w = block_row(m, s, lane, row, zat);
        const double zi = a.z[row];
        const double pi = step ? fma(beta, ps[i], zi) : zi;
        const double qi = step ? fma(beta, qs[i], w) : w;
        ps[i] = pi;
        qs[i] = qi;
        pq[0] += pi * qi;
      });
      if (!all.template sum<1>(pq)) return;
      if (!(pq[0] > 0.0) || !isfinite(pq[0])) {
        status = isfinite(pq[0]) ? FEMK_BREAKDOWN : FEMK_NONFINITE;
        break;
      }
      const double alpha = gamma / pq[0];
      double rz[2] = {0.0, 0.0};
      for (int32_t i0 = threadIdx.x; i0 < nr; i0 += kUnroll * kCT) {
        double xv[kUnroll], pv[kUnroll], rv[kUnroll], qv[kUnroll], dv[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
          const int32_t i = i0 + u * kCT, row = r0 + i;
          if (i < nr && row >= lo && row < hi) {
            xv[u] = xs[i];
            pv[u] = ps[i];
            rv[u] = rs[i];
            qv[u] = qs[i];
            dv[u] = a.dinv ? ds[i] : 1.0;
          }
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
          const int32_t i = i0 + u * kCT, row = r0 + i;
          if (i < nr && row >= lo && row < hi) {
            xs[i] = xv[u] + alpha * pv[u];
            const double ri = rv[u] - alpha * qv[u];
            const double zi = a.dinv ? dv[u] * ri : ri;
            rs[i] = ri;
            a.z[row] = zi;
            rz[0] += ri * zi;
            rz[1] += ri * ri;
          }
        }
      }
      if (!all.template sum<2>(rz)) return;
      beta = rz[0] / gamma;
      gamma = rz[0];
      rr = rz[1];
      ++iter;
      const bool finite = isfinite(gamma) && isfinite(rr);
      if (!finite) status = FEMK_NONFINITE;
      done = !finite || !((a.dinv ? rr : gamma) > atol2) || iter >= a.maxiter;
    }
    // ||b - A x|| / ||b|| of the returned x
    if (held > 3) rows([&](int32_t, int32_t i, int32_t row) { a.x[row] = xs[i]; });
    if (!all.barrier()) return;
    double ww[2] = {0.0, 0.0};
    rows([&](int32_t s, int32_t, int32_t row) {
      const double bi = __ldg(a.b + row), wi = bi - block_row(m, s, lane, row, xat);
      ww[0] += wi * wi;
      ww[1] += bi * bi;
    });
    if (!all.template sum<2>(ww)) return;
    if (me == 0 && threadIdx.x == 0) {
      a.out[k].relres = sqrt(ww[0]) / (sqrt(ww[1]) + 1e-30);
      a.out[k].iter = iter;
      a.out[k].status = status;
    }
  }
  all.leave();
}

template <int SET, typename IDX, bool TAB>
int launch_set(const SetArgs& a, int size, int sets, cudaStream_t s) {
  const void* kern = (const void*)k_batch_sets<SET, IDX, TAB>;
  FEMK_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSetSmem));
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[1];
  cfg.gridDim = dim3(size * sets);
  cfg.blockDim = dim3(kCT);
  cfg.dynamicSmemBytes = (size_t)a.smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = SET == kOneBlock ? 0 : 1;
  if (SET == kOneCluster) {
    FEMK_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = size;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  counted_launch();
  FEMK_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_batch_sets<SET, IDX, TAB>, a));
  return FEMK_OK;
}

template <int SET>
int launch_columns(const femk_plan* p, const SetArgs& a, int size, int sets, cudaStream_t s) {
  if (p->sell_cu) return launch_set<SET, int16_t, true>(a, size, sets, s);
  if (p->sell_ct) return launch_set<SET, int32_t, true>(a, size, sets, s);
  if (p->sell_c16) return launch_set<SET, int16_t, false>(a, size, sets, s);
  return launch_set<SET, int32_t, false>(a, size, sets, s);
}

// clusters of 2^i blocks that the device holds at once (a part of a GPU may hold none of the larger ones)
int clusters_fit(femk_plan* p, int i) {
  if (i == 0) return p->n_sm;
  if (p->batch_fit[i]) return p->batch_fit[i] - 1;
  const auto kern = k_batch_sets<kOneCluster, int16_t, true>;  // the others take the same shared memory and threads
  int fit = 0;
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute at[1];
  cfg.gridDim = dim3(1 << i);
  cfg.blockDim = dim3(kCT);
  cfg.dynamicSmemBytes = kSetSmem;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1 << i;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  if (cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSetSmem) != cudaSuccess ||
      cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) != cudaSuccess) {
    cudaGetLastError();
    fit = 0;
  }
  p->batch_fit[i] = fit + 1;
  return fit;
}

// The set of blocks for a problem: class 0-4 a cluster of 2^i blocks, class 13 - g one of g groups (8 .. 1) of the
// grid, in rising size. The smallest set of which as many as run at once keep their operators on the chip (in L2 and
// shared memory, kPersistBytes), so that the problems share the chip with the fewest waits: 64 slices for a block
// alone, 150 a block of a cluster (148 x 0.57 MB of P1 operator), a cluster of 16 as long as the ones that the device
// holds (7) stay within that, a group of the grid above. A larger set where the problem is so much of the batch that
// blocks would be left idle. B200, FP64 to 1e-8, ms of a batch, grid form -> clusters of 1 / 2 / 4 / 8 / 16, groups
// of 24 / 37 / 49 / 74 / 148 blocks (P1 cubes; the choice in brackets; all columns without own(), which costs 4 %, and
// with four rows in flight in the updates, which cost 1-3. As it is now: 148 x 10^3 0.26, 148 x 16^3 1.38, 112 x 24^3
// 5.4, 56 x 32^3 8.0, 28 x 40^3 9.7, 12 x 64^3 24.2):
//   148 x 10^3   1.24 -> [0.28] / 0.48 / 0.83        28 x 40^3  16.6 -> 17.7 (8) [9.5] (16) / 10.4 / 11.5 / 13.4 / 17.1
//   148 x 16^3   3.38 -> 2.02 / [1.34] / 1.95        28 x 48^3  32.8 -> 31.3 (16) / [18.7] / 18.6 / 21.8 / 25.5 / 39.5
//   112 x 24^3   9.52 -> 19.7 / 8.1 / [5.3] / 6.1    24 x 56^3  49.8 -> 60.3 (16) / 43.6 / 30.4 / [28.2] / 31.1 / 44.9
//   56 x 32^3   14.3 -> 58 / 17 / 15 / [8.0] / 9.6   12 x 64^3  42.1 -> 56.2 (16) / 37.4 / 35.6 / 33.9 / [23.4] / 30.2
//                                                    12 x 80^3  95.8 -> 138 (16) / 102 / 95 / 90 / 90 / [56.5]
constexpr int kClusterClasses = 5, kClasses = 13;
constexpr int kMaxGroups = 8;
int class_sets(femk_plan* p, int c) { return c < kClusterClasses ? clusters_fit(p, c) : kClasses - c; }
int class_size(const femk_plan* p, int c) {
  return c < kClusterClasses ? 1 << c : std::min(p->n_sm, kMaxBlocks) / (kClasses - c);
}
// share: the problem's part of the batch's work
constexpr int kBlockSlices = 150;  // slices a block of a cluster; 64 of a block alone
int problem_class(femk_plan* p, int32_t nprob, int64_t rows, double bytes, double share) {
  const int64_t slices = rows / 32 + 2;
  const double want = share * p->n_sm;
  for (int c = 0; c < kClusterClasses; ++c) {
    const bool last = c + 1 == kClusterClasses;
    if (clusters_fit(p, c) < 1) continue;
    if (last ? std::min<int>(nprob, clusters_fit(p, c)) * bytes > (double)kPersistBytes
             : slices > (c ? kBlockSlices << c : 64))
      continue;
    if (16 << c >= slices) return c;  // a slice a warp: more blocks have nothing to do
    // up to 16,384 rows a cluster's faster wait gains more than blocks beyond 16 (femk_persist.cu)
    if (last ? slices <= 32 * kMaxCluster || want < 24.0 : 2 << c > want) return c;
  }
  return kClusterClasses;
}

// Time of problems [i, j) (rows, falling) on g groups, in units common to all g: a group takes the next problem when
// it is done. An iteration is 6 us of waits and 1.7 us for each round of a slice a warp, and what does not stay on the
// chip slows the rounds (fitted to the table above, within 25 %); steps go with the side of a cube.
double groups_time(const femk_plan* p, const std::vector<double>& rows, int i, int j, int g, double row_bytes) {
  const int size = class_size(p, kClasses - g);
  double busy[kMaxGroups] = {};
  for (int k = i; k < j; ++k) {
    const double over = std::max(0.0, std::min(g, j - i) * rows[k] * row_bytes / (double)kPersistBytes - 1.0);
    const double rounds = rows[k] / (512.0 * size);
    *std::min_element(busy, busy + g) += std::cbrt(rows[k]) * (6.0 + 1.7 * rounds * (1.0 + 3.0 * over));
  }
  return *std::max_element(busy, busy + g);
}

// Groups for the problems that want more than a cluster (rows, falling): the first `split` on g1 groups, the rest on
// g2, in two launches at most.
void choose_groups(const femk_plan* p, const std::vector<double>& rows, double row_bytes, int* split, int* g1,
                   int* g2) {
  const int m = (int)rows.size();
  double best = HUGE_VAL;
  for (int cut = 0; cut < std::min(m, 2 * kMaxGroups); ++cut) {
    double t[2] = {cut ? HUGE_VAL : 0.0, HUGE_VAL};
    int g[2] = {1, 1};
    for (int h = 0; h < 2; ++h)
      for (int n = 1; n <= kMaxGroups; ++n) {
        const double v = groups_time(p, rows, h ? cut : 0, h ? m : cut, n, row_bytes);
        if (v < t[h]) {
          t[h] = v;
          g[h] = n;
        }
      }
    if (t[0] + t[1] < best) {
      best = t[0] + t[1];
      *split = cut;
      *g1 = std::min(g[0], g[1]);
      *g2 = g[1];
    }
  }
}

}  // namespace

// Whether a batch runs here or in the grid form. Three things let that one win, beside a problem that does not stay on
// the chip (B200, FP64 to 1e-8, ms a batch, grid form / here):
//  * Thousands of problems of a few rows: a problem costs a block 13 us to take, which the grid form does not have.
//    20000 x 1^3 (8 rows) 0.84 / 1.77, 3000 x 1^3 0.36 / 0.32; 20000 x 2^3 (27 rows) 1.16 / 2.32, 3000 x 2^3 0.39 /
//    0.38; 20000 x 3^3 (64 rows) 3.09 / 3.92, 6000 x 3^3 1.21 / 1.18; 20000 x 4^3 (125 rows) 6.93 / 5.73.
//  * Gathers spread over many lines of z: L1 looks up a line a cycle on an SM, and a set is a part of the SMs. Lines a
//    row, P1: lattices 1.3-2.1 (40 x 30^3 7.2 / 5.0); shuffled within 32 vertices 2 (7.2 / 7.2, 20 x 40^3 11.3 /
//    10.4); within 128 4.9 (7.2 / 7.7, 11.3 / 11.3); within 512 8.6 (7.3 / 8.5, 11.5 / 12.8), 2-D 20 x 300^2 4.2
//    (10.2 / 9.0); within 4096, 2-D 5.6 (10.4 / 13.3); all 14 (9.8 / 20.4, 16.7 / 31.1), 2-D 6.1 (13.2 / 28.5).
//  * ... but not for problems whose z L1 holds (300 x 12^3, 2197 rows, all shuffled 2.7 / 2.05; 150 x 16^3, 4913 rows,
//    3.5 / 4.1), nor for few rows in all, where the waits count (all shuffled: 40 x 16^3, 197,000 rows, 2.3 / 1.5, 20 x
//    20^3, 185,000, 2.5 / 2.2, 7 x 30^3, 209,000, 4.4 / 3.6; 14 x 30^3, 417,000, 5.7 / 7.1).
constexpr double kSpreadLines = 4.5;  // a row
constexpr int64_t kSmallRows = 2560, kFewRows = 200000;

bool batch_sets_fit(const femk_plan* p, int32_t nprob, const int64_t* row_off) {
  if (!p->persist_ok || !p->use_sell || !p->sell_cols) return false;
  int64_t rows = 0;
  for (int32_t k = 0; k < nprob; ++k) rows = std::max(rows, row_off[k + 1] - row_off[k]);
  // testing the bounded waits: here only a group of the grid waits so, which one large problem is sure to get
  if (p->skip_arrival >= 0 && (nprob > 1 || rows <= 2 * 32 * 32 * kMaxCluster)) return false;
  const double mean = (double)p->n / nprob;
  if (mean < 96.0 && nprob > 20.0 * p->n_sm * std::max(1.0, mean / 32.0)) return false;
  if (rows > kSmallRows && p->n > kFewRows && (double)p->sell_lines > kSpreadLines * (double)p->n) return false;
  return (double)rows * operator_bytes(p) <= (double)kPersistBytes * p->n;
}

int batch_sets(femk_plan* p, int32_t nprob, const int64_t* row_off, const double* vals, const double* b, double* x,
               const double* dinv, double tol, double atol, int32_t maxiter, int32_t* iters_out, double* relres_out,
               int32_t* status_out, cudaStream_t s) {
  FEMK_TRY(ensure_workspace(p));
  FEMK_TRY(ensure_sell_values(p, false));
  // the problems by falling size, and the set of blocks that each runs on (the same for a run of them)
  const double row_bytes = (double)operator_bytes(p) / (double)p->n;
  std::vector<int32_t> order(nprob), cls(nprob);
  std::iota(order.begin(), order.end(), 0);
  auto rows = [&](int32_t k) { return row_off[k + 1] - row_off[k]; };
  std::stable_sort(order.begin(), order.end(), [&](int32_t i, int32_t j) { return rows(i) > rows(j); });
  // its work: CG steps go with the side of a cube
  auto work = [&](int32_t k) { return std::pow((double)rows(k), 4.0 / 3.0); };
  double total = 0.0;
  for (int32_t k = 0; k < nprob; ++k) total += work(k);
  for (int32_t i = 0; i < nprob; ++i) {
    const int32_t k = order[i];
    cls[i] = problem_class(p, nprob, rows(k), row_bytes * (double)rows(k), work(k) / total);
    if (i) cls[i] = std::min(cls[i], cls[i - 1]);
  }
  std::vector<double> large;
  for (int32_t i = 0; i < nprob && cls[i] >= kClusterClasses; ++i) large.push_back((double)rows(order[i]));
  if (!large.empty()) {
    int split = 0, g1 = 1, g2 = 1;
    choose_groups(p, large, row_bytes, &split, &g1, &g2);
    for (int32_t i = 0; i < (int32_t)large.size(); ++i) cls[i] = kClasses - (i < split ? g1 : g2);
  }
  // one buffer: results | row offsets, order, a queue a class | the groups' words
  const int64_t nout = sizeof(BatchOut) * (int64_t)nprob, nint = 2 * (int64_t)nprob + 1 + kClasses;
  const int64_t words0 = (nout + 4 * nint + 255) & ~int64_t(255), bytes = words0 + kMaxGroups * sizeof(GridWords);
  if (p->batch_queue_bytes < bytes) {
    if (p->batch_queue) cudaFree(p->batch_queue);
    p->batch_queue = nullptr;
    p->batch_queue_bytes = 0;
    FEMK_CUDA_TRY(cudaMalloc(&p->batch_queue, bytes));
    p->batch_queue_bytes = bytes;
  }
  std::vector<char> host(nout + 4 * nint, 0);
  BatchOut* out = (BatchOut*)host.data();
  int32_t* ints = (int32_t*)(host.data() + nout);
  for (int32_t k = 0; k < nprob; ++k) out[k].status = FEMK_TIMEOUT;
  for (int32_t k = 0; k <= nprob; ++k) ints[k] = (int32_t)row_off[k];
  std::copy(order.begin(), order.end(), ints + nprob + 1);
  char* base = (char*)p->batch_queue;
  FEMK_CUDA_TRY(cudaMemcpyAsync(base, host.data(), host.size(), cudaMemcpyHostToDevice, s));
  FEMK_TRY(launch_sell_values(p, vals, false, s));
  SetArgs a{};
  a.sptr = p->sell_ptr;
  a.cols = p->sell_cu   ? (const void*)p->sell_cu
           : p->sell_ct ? (const void*)p->sell_ct
                        : (p->sell_c16 ? (const void*)p->sell_c16 : (const void*)p->sell_cols);
  a.svals = p->sell_vals;
  a.tptr = p->sell_cu ? p->sell_cuptr : p->sell_ctptr;
  a.runs = p->sell_runs;
  a.off = (const int32_t*)(base + nout);
  a.words = (GridWords*)(base + words0);
  a.limit = p->barrier_spin;
  a.skip = p->skip_arrival;
  a.b = b;
  a.x = x;
  a.dinv = dinv;
  a.z = p->work;
  a.work = p->work + p->vstride;
  a.vstride = p->vstride;
  a.smem = kSetSmem;
  a.tol2 = tol * tol;
  a.atol2 = atol * atol;
  a.maxiter = maxiter;
  a.out = (BatchOut*)base;
  // A launch a class, by falling size, those of clusters on streams of their own: the blocks that one has no more
  // problems for go to the next. The groups of a grid wait for one another and run before, one launch at a time.
  bool forked = false;
  int sides = 0;
  auto launch_all = [&]() -> int {
    if (cls[0] != cls[nprob - 1]) {
      if (!p->batch_ev) FEMK_CUDA_TRY(cudaEventCreateWithFlags(&p->batch_ev, cudaEventDisableTiming));
      for (cudaStream_t& t : p->batch_side)
        if (!t) FEMK_CUDA_TRY(cudaStreamCreateWithFlags(&t, cudaStreamNonBlocking));
    }
    for (int32_t i = 0, j = 0; i < nprob; i = j) {
      const int c = cls[i], size = class_size(p, c);
      while (j < nprob && cls[j] == c) ++j;
      const int sets = std::min<int>(j - i, class_sets(p, c));
      const bool groups = c >= kClusterClasses;
      a.nprob = j - i;
      a.order = a.off + nprob + 1 + i;
      a.queue = (unsigned int*)(a.off + 2 * nprob + 1 + c);
      a.group = size;
      if (groups) FEMK_CUDA_TRY(cudaMemsetAsync(a.words, 0, kMaxGroups * sizeof(GridWords), s));
      cudaStream_t t = s;
      if (forked) {
        t = p->batch_side[sides++];
        FEMK_CUDA_TRY(cudaStreamWaitEvent(t, p->batch_ev, 0));
      } else if (j < nprob && (!groups || cls[j] < kClusterClasses)) {  // the launches after this one run beside it
        FEMK_CUDA_TRY(cudaEventRecord(p->batch_ev, s));
        forked = true;
      }
      FEMK_TRY(groups   ? launch_columns<kGrid>(p, a, size, sets, t)
               : c == 0 ? launch_columns<kOneBlock>(p, a, size, sets, t)
                        : launch_columns<kOneCluster>(p, a, size, sets, t));
    }
    return FEMK_OK;
  };
  const int rc = launch_all();
  // The caller's stream waits for the others also when a call failed: what was launched uses the caller's arrays.
  cudaError_t joined = cudaSuccess;
  for (int k = 0; k < sides; ++k) {
    cudaError_t e = cudaEventRecord(p->batch_ev, p->batch_side[k]);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(s, p->batch_ev, 0);
    if (e == cudaSuccess) continue;
    cudaStreamSynchronize(p->batch_side[k]);
    joined = e;
  }
  FEMK_TRY(rc);
  FEMK_CUDA_TRY(joined);
  FEMK_CUDA_TRY(cudaMemcpyAsync(out, a.out, nout, cudaMemcpyDeviceToHost, s));
  FEMK_CUDA_TRY(cudaStreamSynchronize(s));
  p->batch_graph_used = 0;
  int worst = FEMK_OK;
  for (int32_t k = 0; k < nprob; ++k) {
    if (iters_out) iters_out[k] = out[k].iter;
    if (relres_out) relres_out[k] = out[k].relres;
    if (status_out) status_out[k] = out[k].status;
    if (out[k].status != FEMK_OK && worst != FEMK_TIMEOUT) worst = out[k].status;
  }
  if (worst == FEMK_TIMEOUT) {
    set_error("femk_pcg_batched: a grid barrier gave up waiting");
    return FEMK_TIMEOUT;
  }
  if (worst != FEMK_OK) {
    set_error("femk_pcg_batched: at least one problem did not solve (see status_out)");
    return worst;
  }
  return FEMK_OK;
}

}  // namespace femk
