// The solver's copy of the operator (sliced ELL, SELL-32): its row order, its slices and its column tables.
//
// Row order. P1 plans keep the DOF order. A P2 plan numbers its edge midpoints as the cells first meet them, so
// consecutive rows belong to different kinds of edges: rows of unequal length share a slice (12 % padding at
// P2 64^3), and no two neighbouring rows have columns at the same offsets, so every entry carries a 4-byte column
// and every gather of a slice touches up to 32 sectors. When the edges fall into few classes by the distance of
// their end vertices' numbers (a lattice has 7 in 3-D, 3 in 2-D), the solver's rows are the vertices and then
// the edges class by class, each in the order of the lower end: neighbouring rows of a class then have the same
// length and the same column offsets along a mesh line. The solvers permute b, x and D^-1 on entry and x on
// exit; nothing outside them sees the order. B200, us a product: P2 64^3 in FP32 99.5 -> 50.5 (544 -> 250 MB), P2
// 37x45x41 in FP64 39.8 -> 26.8 (215 -> 132 MB): 5.0 TB/s of the measured 6.5.
//
// Column tables. A slice mostly has one or two runs of rows with the same column offsets (one mesh line, or the end of
// one and the start of the next), which it stores once a run: 16-bit offsets where those fit (P1 lattices; the
// 16-entry ring of femk_bulk.cuh reads them), 32-bit ones otherwise (P2 in the order above; sell_wide_rows). With one
// offset sequence a slice at most, the 28 % of P1 128^3's slices that hold a line's end kept 2 bytes an entry:
// 18 of the 309 MB of a product (53.9 -> 51.8 us a CG step), and nearly every slice did where lines are shorter than
// two slices.
#include <algorithm>
#include <climits>
#include <new>
#include <utility>

#include "femk_element.cuh"
#include "femk_internal.cuh"
#include "femk_bulk.cuh"
#include "femk_spmv.cuh"

namespace femk {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxClasses = 16;

template <typename T>
int dev_alloc(T** p, int64_t count) {
  FEMK_CUDA_TRY(cudaMalloc((void**)p, sizeof(T) * (count > 0 ? count : 1)));
  return FEMK_OK;
}

struct Temp {
  void* p = nullptr;
  ~Temp() {
    if (p) cudaFree(p);
  }
};

int grid_for(const femk_plan* p, int64_t threads) { return blocks_for(threads, kThreads, p->n_sm * 64); }

// ---------------------------------------------------------------------------------------------
// row order
// ---------------------------------------------------------------------------------------------
// lower and upper end vertex of every edge midpoint (every cell writes the same)
template <int ND>
__global__ void k_edge_ends(const int32_t* __restrict__ cells, int64_t ntet, int64_t nvert, int2* __restrict__ ends) {
  constexpr int NV = Cell<ND>::NV, NE = ND - NV;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < ntet * NE;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = t / NE;
    const int e = (int)(t % NE);
    const int32_t a = cells[c * ND + cell_edge_a<NV>(e)], b = cells[c * ND + cell_edge_b<NV>(e)];
    ends[cells[c * ND + NV + e] - nvert] = make_int2(min(a, b), max(a, b));
  }
}

// the distinct distances upper - lower (at most kMaxClasses; cls[kMaxClasses] is raised when there are more)
__global__ void k_edge_classes(const int2* __restrict__ ends, int64_t nedge, int32_t* __restrict__ cls) {
  __shared__ int32_t seen[kMaxClasses];  // distances that the block has met in cls
  if (threadIdx.x < kMaxClasses) seen[threadIdx.x] = 0;
  __syncthreads();
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nedge; e += (int64_t)gridDim.x * blockDim.x) {
    const int2 v = ends[e];
    const int32_t d = v.y - v.x;
    bool found = false;
    for (int k = 0; k < kMaxClasses && !found; ++k) found = seen[k] == d;
    if (found) continue;
    if (*(volatile int32_t*)(cls + kMaxClasses)) return;  // there are too many already
    for (int k = 0; k < kMaxClasses && !found; ++k) {
      int32_t c = *(volatile int32_t*)(cls + k);
      if (c == 0) c = atomicCAS(cls + k, 0, d);  // 0: this thread took the place
      if ((found = c == 0 || c == d)) seen[k] = d;
    }
    if (!found) {
      cls[kMaxClasses] = 1;
      return;
    }
  }
}

__device__ __forceinline__ int class_of(const int32_t* __restrict__ cls, int nc, int32_t d) {
  int k = 0;
  while (k < nc - 1 && cls[k] != d) ++k;
  return k;
}

__global__ void k_class_flags(const int2* __restrict__ ends, int64_t nedge, const int32_t* __restrict__ cls, int nc,
                              int64_t nvert, int64_t* __restrict__ flag) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nedge; e += (int64_t)gridDim.x * blockDim.x) {
    const int2 v = ends[e];
    flag[class_of(cls, nc, v.y - v.x) * nvert + v.x] = 1;  // (class, lower end) names one edge
  }
}

__global__ void k_order(const int2* __restrict__ ends, int64_t nedge, const int32_t* __restrict__ cls, int nc,
                        int64_t nvert, const int64_t* __restrict__ rank, int32_t* __restrict__ perm,
                        int32_t* __restrict__ pos) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nvert + nedge;
       t += (int64_t)gridDim.x * blockDim.x) {
    int64_t at = t;
    if (t >= nvert) {
      const int2 v = ends[t - nvert];
      at = nvert + rank[class_of(cls, nc, v.y - v.x) * nvert + v.x];
    }
    perm[at] = (int32_t)t;
    pos[t] = (int32_t)at;
  }
}

struct Order {
  Temp ends_base;
  int2* ends = nullptr;
  int32_t* cls = nullptr;
  int classes = 0;  // 0: the DOF order
};

// the edge classes of a P2 plan, when there are few
int find_order(const femk_plan* p, Order* o, cudaStream_t s) {
  const int64_t nedge = p->n - p->nvert;
  if (p->order != 2 || !p->use_sell || nedge < 1) return FEMK_OK;
  FEMK_CUDA_TRY(cudaMalloc(&o->ends_base.p, sizeof(int2) * nedge + sizeof(int32_t) * (kMaxClasses + 1)));
  o->ends = (int2*)o->ends_base.p;
  o->cls = (int32_t*)(o->ends + nedge);
  FEMK_CUDA_TRY(cudaMemsetAsync(o->cls, 0, sizeof(int32_t) * (kMaxClasses + 1), s));
  if (p->nd == 10)
    k_edge_ends<10><<<counted_launch() + grid_for(p, p->ntet * 6), kThreads, 0, s>>>(p->cells, p->ntet, p->nvert,
                                                                                  o->ends);
  else
    k_edge_ends<6><<<counted_launch() + grid_for(p, p->ntet * 3), kThreads, 0, s>>>(p->cells, p->ntet, p->nvert,
                                                                                 o->ends);
  k_edge_classes<<<counted_launch() + grid_for(p, nedge), kThreads, 0, s>>>(o->ends, nedge, o->cls);
  FEMK_CUDA_TRY(cudaGetLastError());
  int32_t h[kMaxClasses + 1];
  FEMK_CUDA_TRY(cudaMemcpyAsync(h, o->cls, sizeof(h), cudaMemcpyDeviceToHost, s));
  FEMK_CUDA_TRY(cudaStreamSynchronize(s));
  if (h[kMaxClasses]) return FEMK_OK;
  while (o->classes < kMaxClasses && h[o->classes]) ++o->classes;
  std::sort(h, h + o->classes);  // they were found in no fixed order
  FEMK_CUDA_TRY(cudaMemcpyAsync(o->cls, h, sizeof(int32_t) * o->classes, cudaMemcpyHostToDevice, s));
  FEMK_CUDA_TRY(cudaStreamSynchronize(s));
  return FEMK_OK;
}

int fill_order(femk_plan* p, const Order& o, cudaStream_t s) {
  const int64_t nedge = p->n - p->nvert, m = o.classes * p->nvert;
  Temp base;  // a flag for every (class, lower end), then their exclusive scan
  FEMK_CUDA_TRY(cudaMalloc(&base.p, sizeof(int64_t) * 2 * (m + 1)));
  int64_t* flag = (int64_t*)base.p;
  int64_t* rank = flag + m + 1;
  FEMK_CUDA_TRY(cudaMemsetAsync(flag, 0, sizeof(int64_t) * (m + 1), s));
  k_class_flags<<<counted_launch() + grid_for(p, nedge), kThreads, 0, s>>>(o.ends, nedge, o.cls, o.classes, p->nvert,
                                                                           flag);
  FEMK_TRY(scan_exclusive_i64(flag, rank, m, s));
  k_order<<<counted_launch() + grid_for(p, p->n), kThreads, 0, s>>>(o.ends, nedge, o.cls, o.classes, p->nvert, rank,
                                                                    p->perm, p->pos);
  FEMK_CUDA_TRY(cudaGetLastError());
  FEMK_CUDA_TRY(cudaStreamSynchronize(s));  // temporaries are freed on return
  return FEMK_OK;
}

// ---------------------------------------------------------------------------------------------
// slices
// ---------------------------------------------------------------------------------------------
// Width of each 32-row slice (its longest row) and its entry count.
__global__ void k_sell_width(const int32_t* __restrict__ indptr, const int32_t* __restrict__ perm, int64_t n,
                             int64_t nslices, int64_t* __restrict__ len) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t sl = warp; sl < nslices; sl += nwarps) {
    int64_t row = sl * 32 + lane;
    const bool live = row < n;
    if (live && perm) row = perm[row];
    int w = live ? indptr[row + 1] - indptr[row] : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w = max(w, __shfl_xor_sync(0xffffffffu, w, o));
    if (lane == 0) len[sl] = (int64_t)w * 32;
  }
}

__global__ void k_sell_fill(const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices, int64_t n,
                            int64_t nslices, const int64_t* __restrict__ sptr, int32_t* __restrict__ cols,
                            int16_t* __restrict__ c16) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t sl = warp; sl < nslices; sl += nwarps) {
    const int64_t row = sl * 32 + lane;
    const int64_t w = (sptr[sl + 1] - sptr[sl]) / 32;
    const int32_t beg = row < n ? indptr[row] : 0;
    const int32_t len = row < n ? indptr[row + 1] - beg : 0;
    const int64_t self = row < n ? row : n - 1;
    for (int64_t k = 0; k < w; ++k) {
      const int64_t j = sptr[sl] + k * 32 + lane;
      const bool real = k < len;
      const int32_t col = real ? indices[beg + k] : (int32_t)self;
      cols[j] = col;
      if (c16) c16[j] = (int16_t)(col - self);
    }
  }
}

// The same with column tables, in the solver's row order (perm, pos; NULL: the DOF order). A warp takes a slice, a lane
// a row: the row's columns as solver rows, sorted. Going down the slice, rows whose offsets (column - row) are all among
// those of a longer row, or hold all of them, form a run and share that longest row's offsets, an entry for each
// (value 0 where a row has none): rows along a mesh line, its ends included. A slice with up to kRuns runs stores
// one offset sequence a run (16-bit offsets: run by run, each padded to 8; 32-bit ones: piece by piece of kPiece
// entries, each padded to 4); a slice with more stores every entry's offset. No shared offset leads outside [0, n).
// PASS 0: words[s], the table entries of slice s. PASS 1: columns (and 16-bit offsets), places in the CSR row, tables
// and run starts.
constexpr int kRowMax = 255;  // place of an entry that a row does not have (rows hold fewer entries)
constexpr int kRuns = 4;

template <int PASS, typename T>
__global__ void k_sell_order(const int32_t* __restrict__ indptr, const int32_t* __restrict__ indices,
                             const int32_t* __restrict__ perm, const int32_t* __restrict__ pos, int64_t n,
                             int64_t nslices, const int64_t* __restrict__ sptr, int32_t cap,
                             int64_t* __restrict__ words, int32_t* __restrict__ cols, int16_t* __restrict__ c16,
                             uint8_t* __restrict__ src, const int64_t* __restrict__ tptr, T* __restrict__ tab,
                             int32_t* __restrict__ runs) {
  constexpr int kPad = sizeof(T) == 2 ? 8 : 4;
  extern __shared__ long long order_buf[];  // 32 cap words a warp: (offset << 8) | place, entry k of lane l at 32 k + l
  const int lane = threadIdx.x & 31;
  long long* buf = order_buf + (int64_t)(threadIdx.x >> 5) * 32 * cap;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t sl = warp; sl < nslices; sl += nwarps) {
    const int64_t b0 = sptr[sl];
    const int32_t w = (int32_t)((sptr[sl + 1] - b0) >> 5), head = (w + kPad - 1) & ~(kPad - 1);
    const int32_t row = (int32_t)(sl * 32) + lane;
    const bool live = row < n;
    const int32_t dof = live ? (perm ? perm[row] : row) : 0;
    const int32_t beg = live ? indptr[dof] : 0;
    const int32_t len = live ? indptr[dof + 1] - beg : 0;
    for (int32_t k = 0; k < len; ++k) {  // insertion sort by offset
      const int32_t col = indices[beg + k];
      const long long v = ((long long)((pos ? pos[col] : col) - row) << 8) | k;
      int32_t q = k;
      for (; q > 0 && buf[32 * (q - 1) + lane] > v; --q) buf[32 * q + lane] = buf[32 * (q - 1) + lane];
      buf[32 * q + lane] = v;
    }
    __syncwarp();
    auto off = [&](int l, int32_t k) { return (int32_t)(buf[32 * k + l] >> 8); };
    // whether every offset of lane `a` is one of lane `b` (all lanes ask and get the same answer)
    auto within = [&](int a, int32_t na, int b, int32_t nb) {
      bool in = true;
      for (int32_t k = lane; k < na; k += 32) {
        const int32_t v = off(a, k);
        int32_t lo = 0, hi = nb;
        while (lo < hi) {
          const int32_t mid = (lo + hi) >> 1;
          if (off(b, mid) < v)
            lo = mid + 1;
          else
            hi = mid;
        }
        in = in && lo < nb && off(b, lo) == v;
      }
      return __all_sync(0xffffffffu, in) != 0;
    };
    int nruns = 1, rep[kRuns] = {0, 0, 0, 0}, start[kRuns] = {0, 32, 32, 32};
    for (int l = 1; l < 32 && nruns > 0; ++l) {
      const int32_t nl = __shfl_sync(0xffffffffu, len, l);
      int cur = rep[0];
#pragma unroll
      for (int q = 1; q < kRuns; ++q)
        if (q < nruns) cur = rep[q];
      const int32_t nr = __shfl_sync(0xffffffffu, len, cur);
      if (nl == 0 || within(l, nl, cur, nr)) continue;  // rows past n are in any run
      if (within(cur, nr, l, nl)) {
#pragma unroll
        for (int q = 0; q < kRuns; ++q)
          if (q == nruns - 1) rep[q] = l;
        continue;
      }
      if (nruns == kRuns) {
        nruns = 0;
        break;
      }
#pragma unroll
      for (int q = 1; q < kRuns; ++q)
        if (q == nruns) {
          rep[q] = l;
          start[q] = l;
        }
      ++nruns;
    }
    int mine = 0, lead = rep[0];
#pragma unroll
    for (int q = 1; q < kRuns; ++q)
      if (q < nruns && lane >= start[q]) {
        mine = q;
        lead = rep[q];
      }
    const int32_t nlead = __shfl_sync(0xffffffffu, len, lead);
    const bool inside = !live || nlead == 0 || (row + off(lead, 0) >= 0 && row + off(lead, nlead - 1) < n);
    if (!__all_sync(0xffffffffu, inside)) nruns = 0;
    if (PASS == 0) {
      if (lane == 0) words[sl] = nruns > 0 ? nruns * head : 32 * w;
      __syncwarp();
      continue;
    }
    // entries: a run's rows in the lead's slots, or in their own order
    T* t = tab + tptr[sl];
    for (int32_t k = 0, q = 0; k < w; ++k) {
      const int64_t j = b0 + 32 * (int64_t)k + lane;
      const bool have = q < len && (nruns == 0 || off(lane, q) == off(lead, k));
      const int32_t o = have ? off(lane, q) : 0;
      cols[j] = live ? row + o : (int32_t)(n - 1);
      if (c16) c16[j] = (int16_t)o;
      src[j] = have ? (uint8_t)(buf[32 * q + lane] & 255) : (uint8_t)kRowMax;
      if (nruns == 0) t[32 * k + lane] = (T)o;
      q += have;
    }
    int32_t nrep[kRuns];
#pragma unroll
    for (int q = 0; q < kRuns; ++q) nrep[q] = __shfl_sync(0xffffffffu, len, rep[q]);
    if (nruns > 0) {
      for (int32_t k = lane; k < head; k += 32) {
        // piece p of run q starts at nruns * kPiece * p + q * (the piece's padded entries)
        const int32_t k0 = sizeof(T) == 2 ? 0 : k / kPiece * kPiece;
        const int32_t pk = sizeof(T) == 2 ? head : min(kPiece, head - k0);
#pragma unroll
        for (int q = 0; q < kRuns; ++q) {
          if (q >= nruns) continue;
          t[nruns * k0 + q * pk + (k - k0)] = (T)(k < nrep[q] ? off(rep[q], k) : 0);
        }
      }
    }
    if (lane == 0) runs[sl] = nruns > 0 ? start[1] | (start[2] << 8) | (start[3] << 16) : -1;
    __syncwarp();
  }
}

// 128-byte lines that the gathers of a product touch, summed over entries and slices (an entry of a slice is one
// gather of 32 rows): how far apart the columns of neighbouring rows lie.
__global__ void k_gather_lines(const int64_t* __restrict__ sptr, const int32_t* __restrict__ cols, int64_t nslices,
                               unsigned long long* __restrict__ lines) {
  const int lane = threadIdx.x & 31;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  unsigned long long sum = 0;
  for (int64_t sl = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; sl < nslices; sl += nwarps)
    for (int64_t j = sptr[sl] + lane; j < sptr[sl + 1]; j += 32) {
      const unsigned int same = __match_any_sync(0xffffffffu, cols[j] >> 4);
      sum += __popc(__ballot_sync(0xffffffffu, __ffs(same) - 1 == lane));
    }
  if (lane == 0) atomicAdd(lines, sum);
}

template <typename T>
int fill_tables(femk_plan* p, int64_t* len, int64_t* tptr, T** tab, int64_t* total, cudaStream_t s) {
  const int threads = 64, smem = threads * p->max_row * (int)sizeof(long long);
  const int grid = blocks_for(p->n_slices * 32, threads, p->n_sm * 64);
  FEMK_CUDA_TRY(cudaFuncSetAttribute(k_sell_order<0, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  FEMK_CUDA_TRY(cudaFuncSetAttribute(k_sell_order<1, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  k_sell_order<0, T><<<counted_launch() + grid, threads, smem, s>>>(p->indptr, p->indices, p->perm, p->pos, p->n,
                                                                    p->n_slices, p->sell_ptr, p->max_row, len, nullptr,
                                                                    nullptr, nullptr, nullptr, nullptr, nullptr);
  FEMK_TRY(scan_exclusive_i64(len, tptr, p->n_slices, s));
  FEMK_CUDA_TRY(cudaMemcpyAsync(total, tptr + p->n_slices, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  FEMK_CUDA_TRY(cudaStreamSynchronize(s));
  FEMK_TRY(dev_alloc(tab, *total));
  k_sell_order<1, T><<<counted_launch() + grid, threads, smem, s>>>(
      p->indptr, p->indices, p->perm, p->pos, p->n, p->n_slices, p->sell_ptr, p->max_row, nullptr, p->sell_cols,
      p->sell_c16, p->sell_src, tptr, *tab, p->sell_runs);
  FEMK_CUDA_TRY(cudaGetLastError());
  return FEMK_OK;
}

void drop_slices(femk_plan* p) {
  for (void* q : {p->sell_base, (void*)p->sell_cols, (void*)p->sell_cu, (void*)p->sell_ct})
    if (q) cudaFree(q);
  p->sell_base = nullptr;
  p->sell_ptr = p->sell_cuptr = p->sell_ctptr = nullptr;
  p->perm = p->pos = p->sell_runs = p->sell_cols = p->sell_ct = nullptr;
  p->sell_c16 = p->sell_cu = nullptr;
  p->sell_src = nullptr;
}

int build_slices(femk_plan* p, const Order& o, cudaStream_t s) {
  const int64_t n = p->n, ns = (n + 31) / 32;
  p->n_slices = ns;
  const bool ordered = o.classes > 0;
  // few allocations (one takes 0.3 ms): what the slices' number sizes, what the stored entries' number does, the tables
  const int64_t words = ns + (ordered ? 2 * n : 0);
  FEMK_CUDA_TRY(cudaMalloc(&p->sell_base, sizeof(int64_t) * 3 * (ns + 1) + sizeof(int32_t) * words));
  p->sell_ptr = (int64_t*)p->sell_base;
  int64_t* tptr = p->sell_ptr + ns + 1;
  int64_t* len = tptr + ns + 1;
  p->sell_runs = (int32_t*)(len + ns + 1);
  if (ordered) {
    p->perm = p->sell_runs + ns;
    p->pos = p->perm + n;
    FEMK_TRY(fill_order(p, o, s));
  }
  const int sgrid = grid_for(p, ns * 32);
  k_sell_width<<<counted_launch() + sgrid, kThreads, 0, s>>>(p->indptr, p->perm, n, ns, len);
  FEMK_TRY(scan_exclusive_i64(len, p->sell_ptr, ns, s));
  FEMK_CUDA_TRY(cudaMemcpyAsync(&p->sell_nnz, p->sell_ptr + ns, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  FEMK_CUDA_TRY(cudaStreamSynchronize(s));
  if (p->sell_nnz >= INT32_MAX) {
    p->use_sell = 0;
    drop_slices(p);
    return FEMK_OK;
  }
  // 16-bit offsets always fit a system of at most 2^15 rows; past that only the DOF order's are known to
  const bool c16 = ordered ? n <= 32768 : p->cols16 != nullptr;
  const bool tables = ordered || (c16 && p->sell_uni);
  char* base = nullptr;
  FEMK_CUDA_TRY(cudaMalloc(&base, (p->sell_nnz > 0 ? p->sell_nnz : 1) * (4 + (c16 ? 2 : 0) + (tables ? 1 : 0))));
  p->sell_cols = (int32_t*)base;
  base += 4 * p->sell_nnz;  // slices hold 32 entries a column: every part starts on 32 bytes
  if (c16) {
    p->sell_c16 = (int16_t*)base;
    base += 2 * p->sell_nnz;
  }
  if (tables) p->sell_src = (uint8_t*)base;
  if (!tables) {
    k_sell_fill<<<counted_launch() + sgrid, kThreads, 0, s>>>(p->indptr, p->indices, n, ns, p->sell_ptr, p->sell_cols,
                                                              p->sell_c16);
  } else if (c16) {
    FEMK_TRY(fill_tables(p, len, tptr, &p->sell_cu, &p->sell_cu_len, s));
    p->sell_cuptr = tptr;
  } else {
    FEMK_TRY(fill_tables(p, len, tptr, &p->sell_ct, &p->sell_ct_len, s));
    p->sell_ctptr = tptr;
  }
  FEMK_CUDA_TRY(cudaMemsetAsync(len, 0, sizeof(int64_t), s));  // the slices' lengths are not needed any more
  k_gather_lines<<<counted_launch() + sgrid, kThreads, 0, s>>>(p->sell_ptr, p->sell_cols, ns, (unsigned long long*)len);
  FEMK_CUDA_TRY(cudaGetLastError());
  FEMK_CUDA_TRY(cudaMemcpyAsync(&p->sell_lines, len, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  FEMK_CUDA_TRY(cudaStreamSynchronize(s));
  return FEMK_OK;
}

// ---------------------------------------------------------------------------------------------
// values and vectors in the solver's order
// ---------------------------------------------------------------------------------------------
__global__ void k_permute_in(const int32_t* __restrict__ perm, int64_t n, const double* __restrict__ b,
                             const double* __restrict__ x, const double* __restrict__ d, double* __restrict__ bs,
                             double* __restrict__ xs, double* __restrict__ ds) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t j = perm[i];
    if (b) bs[i] = b[j];
    if (x) xs[i] = x[j];
    if (d) ds[i] = d[j];
  }
}

__global__ void k_permute_out(const int32_t* __restrict__ perm, int64_t n, const double* __restrict__ xs,
                              double* __restrict__ x) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[perm[i]] = xs[i];
}

}  // namespace

int build_sell(femk_plan* p, cudaStream_t s) {
  Order o;
  FEMK_TRY(find_order(p, &o, s));
  return build_slices(p, o, s);
}

// frees the plan's layouts
void drop_sell(femk_plan* p) {
  for (int i = 0; i < 2; ++i) {
    drop_slices(p);
    cudaFree(p->sell_vals);
    cudaFree(p->sell_vals32);
    p->sell_vals = nullptr;
    p->sell_vals32 = nullptr;
    if (!p->dof_order) break;
    static_cast<SellLayout&>(*p) = *p->dof_order;
    delete p->dof_order;
    p->dof_order = nullptr;
  }
}

DofOrder::DofOrder(femk_plan* plan, cudaStream_t s) : p(plan) {
  if (!p->perm) return;
  SellLayout& own = *p;
  if (!p->dof_order) {
    const SellLayout ordered = own;
    own = SellLayout{};
    status = build_slices(p, Order{}, s);
    if (status != FEMK_OK) drop_slices(p);
    SellLayout* built = status == FEMK_OK ? new (std::nothrow) SellLayout(own) : nullptr;
    if (status == FEMK_OK && !built) {
      drop_slices(p);
      set_error("femk_pcg_batched: out of host memory");
      status = FEMK_ENOMEM;
    }
    own = ordered;
    if (status != FEMK_OK) return;
    p->dof_order = built;
  }
  std::swap(own, *p->dof_order);
  swapped = true;
}

DofOrder::~DofOrder() {
  if (swapped) std::swap(static_cast<SellLayout&>(*p), *p->dof_order);
}

int permute_in(femk_plan* p, const double** b, double** x, const double** dinv, cudaStream_t s) {
  if (!p->perm_ws) FEMK_TRY(dev_alloc(&p->perm_ws, 3 * p->vstride));
  double* bs = p->perm_ws;
  double* xs = bs + p->vstride;
  double* ds = xs + p->vstride;
  k_permute_in<<<counted_launch() + blocks_for(p->n, kThreads, p->n_sm * 8), kThreads, 0, s>>>(
      p->perm, p->n, b ? *b : nullptr, x ? *x : nullptr, dinv ? *dinv : nullptr, bs, xs, ds);
  FEMK_CUDA_TRY(cudaGetLastError());
  if (b) *b = bs;
  if (x) *x = xs;
  if (dinv && *dinv) *dinv = ds;
  return FEMK_OK;
}

int permute_out(const femk_plan* p, const double* xs, double* x, cudaStream_t s) {
  k_permute_out<<<counted_launch() + blocks_for(p->n, kThreads, p->n_sm * 8), kThreads, 0, s>>>(p->perm, p->n, xs, x);
  FEMK_CUDA_TRY(cudaGetLastError());
  return FEMK_OK;
}

}  // namespace femk
