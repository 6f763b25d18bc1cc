// Building blocks of the single-launch (persistent, cooperatively launched) Krylov solvers for systems
// whose operator stays on the chip: shared memory first, L2 for the rest.
//
// Each block owns a run of consecutive 32-row slices of the sliced-ELL operator for the whole solve. As many
// of its slices as fit are copied into shared memory once (values and columns), the others are read from L2 in
// every product; the block's parts of the solver vectors live in shared memory too. Only what other blocks
// gather goes through global memory.
//
// Reductions double as barriers over the blocks, and every block ends up with the same bits:
//  * one block: __syncthreads;
//  * one cluster of up to 16 blocks (or each of a grid's, on its own): every block stores its partial sums into every
//    other block's shared memory and crosses the hardware cluster barrier (0.7-1.0 us measured with 2-16 blocks of 512
//    threads);
//  * a cooperative grid, one block an SM: every block stores its partials in global memory and adds one to a
//    counter (release), waits until the counter says that all have (acquire), and adds all partials itself in
//    block order: 2.1 us, the same for 2 and for 148 blocks. Words that carry the partial and a phase number
//    together, polled by all blocks, need no second read but took 1.0-5.4 us (the polls of 148 blocks contend),
//    and 3.0-3.8 us in mailboxes of each reader's own.
// Only the grid's wait is a spin, and it is bounded: a block that runs out of its clock64 budget gives up and
// arrives no more, so the others run out too; the kernel returns and the host reports FEMK_TIMEOUT. The time before
// all blocks run does not count: a cooperative grid starts as a whole (a grid of 148 blocks with a limit of 1 ms,
// launched beside a kernel that held one SM for 50 ms, or beside another grid that ran for 11, waited for its end and
// solved).
#pragma once

#include <stdint.h>

#include "femk_internal.cuh"

namespace femk {

enum BlockSet { kOneBlock = 0, kOneCluster = 1, kGrid = 2 };

constexpr int kSumValues = 3;    // values a phase can sum at once
constexpr int kMaxBlocks = 256;  // blocks of a grid
constexpr int kMaxCluster = 16;

// Global scratch of the grid form: the partials of two alternating phases and two alternating counters. A
// launch counts on counter[turn] and zeroes the other one, which the next launch uses.
struct GridWords {
  double part[2][kSumValues][kMaxBlocks];
  unsigned int counter[2][32];  // a line apart
};

__device__ __forceinline__ unsigned int cluster_rank() {
  unsigned int r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ unsigned int cluster_size() {
  unsigned int r;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// stores a double at the address that `p` (own shared memory) has in block `rank` of the cluster
__device__ __forceinline__ void st_cluster(const double* p, unsigned int rank, double v) {
  uint32_t a;
  const uint32_t own = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(own), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Sums of NV values a thread over all blocks, the same bits in every thread of every block, and a barrier:
// what any block wrote before the call is visible to all after it (plain loads included).
template <int SET, int THREADS>
struct BlockSum {
  GridWords* words;
  int turn;
  long long limit;
  int skip;            // testing: the block that never arrives (-1: none)
  unsigned int phase;  // sums done
  int rank, size;      // kGrid: this block among those that sum together (all of the grid, or a group with its words)

  // Every thread of every block, before anything else of this struct. A cluster's blocks store into each other's
  // shared memory, which exists only once all of them have started: that is waited for here, once a launch (below
  // 1 us).
  __device__ __forceinline__ BlockSum(GridWords* words, int turn, long long limit, int skip, int rank, int size)
      : words(words), turn(turn), limit(limit), skip(skip), phase(0u), rank(rank), size(size) {
    if (SET == kOneCluster) cluster_sync();
  }

  // one thread of the block: its writes and, after a __syncthreads, its block's are released, the others' acquired
  __device__ __forceinline__ int arrive() {
    unsigned int* c = &words->counter[turn][0];
    const unsigned int want = (unsigned int)size * phase;  // wraps with the counter
    if (rank != skip) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(c) : "memory");
    const long long t0 = clock64();
    unsigned int seen, polls = 0;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(c) : "memory");
      if ((int)(seen - want) >= 0) return 1;
      if ((++polls & 63u) == 0u && clock64() - t0 > limit) return 0;
    }
  }

  template <int NV>
  __device__ __forceinline__ bool sum(double (&v)[NV]) {
    constexpr int W = THREADS / 32;
    constexpr int NB = SET == kGrid ? kMaxBlocks / 32 : kMaxCluster;
    __shared__ double red[2][kSumValues][W];
    __shared__ double tot[2][kSumValues][NB];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int par = (int)(phase & 1);
    const int G = SET == kOneCluster ? (int)cluster_size() : size;
    ++phase;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      v[j] = warp_sum(v[j]);
      if (lane == 0) red[par][j][warp] = v[j];
    }
    __syncthreads();
    if (SET == kOneBlock) {
#pragma unroll
      for (int j = 0; j < NV; ++j) v[j] = warp_sum(lane < W ? red[par][j][lane] : 0.0);
      return true;
    }
    if (SET == kOneCluster) {
      if (warp == 0) {
        const unsigned int me = cluster_rank();
#pragma unroll
        for (int j = 0; j < NV; ++j) {
          const double t = warp_sum(lane < W ? red[par][j][lane] : 0.0);
          if (lane < G) st_cluster(&tot[par][j][me], lane, t);
        }
      }
      cluster_sync();
#pragma unroll
      for (int j = 0; j < NV; ++j) v[j] = warp_sum(lane < G ? tot[par][j][lane] : 0.0);
      return true;
    }
    int ok = 1;
    if (warp == 0) {
      double t[NV];
#pragma unroll
      for (int j = 0; j < NV; ++j) t[j] = warp_sum(lane < W ? red[par][j][lane] : 0.0);
      if (lane == 0) {
#pragma unroll
        for (int j = 0; j < NV; ++j) __stcg(&words->part[par][j][rank], t[j]);
        ok = arrive();
      }
    }
    ok = __syncthreads_and(ok);
    const int groups = (G + 31) >> 5;
    if (warp < groups) {
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        const double t = warp_sum((int)threadIdx.x < G ? __ldcg(&words->part[par][j][threadIdx.x]) : 0.0);
        if (lane == 0) tot[par][j][warp] = t;
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NV; ++j) v[j] = warp_sum(lane < groups ? tot[par][j][lane] : 0.0);
    return ok != 0;
  }

  // the barrier alone: what any block wrote before it is visible to all after it
  __device__ __forceinline__ bool barrier() {
    if (SET != kGrid) {
      if (SET == kOneBlock)
        __syncthreads();
      else
        cluster_sync();
      return true;
    }
    ++phase;
    __syncthreads();
    const int ok = threadIdx.x == 0 ? arrive() : 1;
    return __syncthreads_and(ok) != 0;
  }

  // before the kernel returns: no block of a cluster leaves while another may store into its shared memory
  __device__ __forceinline__ void leave() {
    if (SET == kOneCluster) cluster_sync();
  }
};

// One block's share of the operator: slices [s0, s0 + ns), of which the first `fit` are in shared memory. IDX: the
// type of the columns, an offset from the row (16 bits) or absolute (32); TAB: column tables (femk_order.cu), whose
// entries are offsets of either type, in place of a column an entry.
template <typename IDX, bool TAB>
struct BlockMatrix {
  int32_t s0, ns, fit;   // first slice, slices, slices held in shared memory
  int32_t tfit;          // TAB: slices whose tables are
  const int32_t* off;    // shared: ns + 1 entry offsets from the block's first entry
  const int32_t* toff;   // shared, TAB: ns + 1 table offsets from the block's first table entry
  const int32_t* runs;   // shared, TAB: run starts of each slice
  const double* sv;      // shared values and columns of the first `fit` slices (tables: of the first `tfit`)
  const IDX* sc;
  const double* gv;      // the block's entries (tables) in global memory
  const IDX* gc;
};

// bytes of shared memory for the offsets (and, TAB, the run starts) of ns slices
template <bool TAB>
__device__ __forceinline__ int32_t offset_bytes(int32_t ns) {
  return (4 * (ns + 1 + (TAB ? 2 * ns + 1 : 0)) + 15) & ~15;
}

// First of the nslices slices from sptr on that belongs to block b: the blocks get equal shares of the work, counted
// as the stored entries plus 8 a row for the vector updates (rows may be of unequal length). Every thread gets the
// same answer.
constexpr int kSliceWork = 8 * 32;
__device__ __forceinline__ int32_t block_slice(const int64_t* __restrict__ sptr, int32_t nslices, int b, int blocks) {
  const int64_t e0 = __ldg(sptr);
  const int64_t want = e0 + (__ldg(sptr + nslices) - e0 + (int64_t)kSliceWork * nslices) * b / blocks;
  int32_t lo = 0, hi = nslices;
  while (lo < hi) {
    const int32_t mid = (lo + hi) >> 1;
    if (__ldg(sptr + mid) + (int64_t)kSliceWork * mid < want)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// Row sum of one lane's row, entries 32 apart, up to B loads in flight; g(column) is the operand. The entries
// add in k order, as everywhere else.
template <int B, bool SHARED, typename IDX, typename G>
__device__ __forceinline__ double lane_row(const double* vb, const IDX* cb, int32_t w, int32_t row, const G& g) {
  double acc = 0.0;
  for (int32_t k0 = 0; k0 < w; k0 += B) {
    double v[B];
    int32_t c[B];
#pragma unroll
    for (int u = 0; u < B; ++u) {
      const int32_t j = (k0 + u) * 32;
      const bool ok = k0 + u < w;
      c[u] = ok ? (int32_t)(SHARED ? cb[j] : __ldg(cb + j)) : 0;
      v[u] = ok ? (SHARED ? vb[j] : __ldg(vb + j)) : 0.0;
      if (sizeof(IDX) == 2) c[u] += row;
    }
#pragma unroll
    for (int u = 0; u < B; ++u)
      if (k0 + u < w) acc += v[u] * g(c[u]);
  }
  return acc;
}

// The same with the offsets of the row's run (HELD: the table is in shared memory): run `run` of `nruns`, kPieceRow
// entries at a time (16-byte loads of the table, one address a run).
constexpr int kPieceRow = 16;
template <bool SHARED, bool HELD, typename T, typename G>
__device__ __forceinline__ double table_row(const double* vb, const T* tab, int32_t w, int run, int nruns, int32_t row,
                                            const G& g) {
  constexpr int kPad = sizeof(T) == 2 ? 8 : 4, kVec = 16 / (int)sizeof(T);
  const int32_t head = (w + kPad - 1) & ~(kPad - 1);
  double acc = 0.0;
  for (int32_t k0 = 0; k0 < w; k0 += kPieceRow) {
    const T* t = sizeof(T) == 2 ? tab + run * head + k0 : tab + nruns * k0 + run * min(kPieceRow, head - k0);
    double v[kPieceRow];
    int4 q[kPieceRow / kVec];
#pragma unroll
    for (int u = 0; u < kPieceRow / kVec; ++u) {
      q[u] = make_int4(0, 0, 0, 0);
      if (k0 + u * kVec < w)
        q[u] = HELD ? reinterpret_cast<const int4*>(t)[u] : __ldg(reinterpret_cast<const int4*>(t) + u);
    }
#pragma unroll
    for (int u = 0; u < kPieceRow; ++u) {
      const int32_t j = (k0 + u) * 32;
      v[u] = k0 + u < w ? (SHARED ? vb[j] : __ldg(vb + j)) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < kPieceRow; ++u)
      if (k0 + u < w) {
        const int4 f = q[u / kVec];
        int32_t c;
        if (sizeof(T) == 2) {
          const int h = u % 8 / 2;
          const int32_t word = h == 0 ? f.x : (h == 1 ? f.y : (h == 2 ? f.z : f.w));
          c = (u & 1) ? word >> 16 : (int32_t)(int16_t)(word & 0xffff);
        } else {
          const int h = u % 4;
          c = h == 0 ? f.x : (h == 1 ? f.y : (h == 2 ? f.z : f.w));
        }
        acc += v[u] * g(row + c);
      }
  }
  return acc;
}

// An entry's own offset (slices of a table plan with too many runs)
template <bool SHARED, typename T, typename G>
__device__ __forceinline__ double offset_row(const double* vb, const T* cb, int32_t w, int32_t row, const G& g) {
  double acc = 0.0;
  for (int32_t k0 = 0; k0 < w; k0 += 8) {
    double v[8];
    int32_t c[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int32_t j = (k0 + u) * 32;
      c[u] = k0 + u < w ? (int32_t)(SHARED ? cb[j] : __ldg(cb + j)) : 0;
      v[u] = k0 + u < w ? (SHARED ? vb[j] : __ldg(vb + j)) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (k0 + u < w) acc += v[u] * g(row + c[u]);
  }
  return acc;
}

// The block's share, its first slices copied into `mat` (room bytes of shared memory; off: offset_bytes of shared
// memory). The whole block calls this. Tables of lattices take 1/60 of their values' room, and a gather waits for its
// table entry: all of them are held if they fit a quarter of the room (us an iteration, P1 64^3 11.9 -> 11.6, 80^3
// 18.3 -> 17.4, P2 34^3 21.3 -> 20.4).
template <int THREADS, typename IDX, bool TAB>
__device__ __forceinline__ void hold_slices(BlockMatrix<IDX, TAB>& m, const int64_t* __restrict__ sptr,
                                            const void* cols, const double* svals, const int64_t* __restrict__ tptr,
                                            const int32_t* __restrict__ runs, int32_t* off, unsigned char* mat,
                                            int32_t room) {
  __shared__ int32_t fit_s;
  const int64_t e0 = __ldg(sptr + m.s0), t0 = TAB ? __ldg(tptr + m.s0) : e0;
  int32_t* toff = off + m.ns + 1;
  int32_t* rs = toff + m.ns + 1;
  for (int32_t s = threadIdx.x; s <= m.ns; s += THREADS) {
    off[s] = (int32_t)(__ldg(sptr + m.s0 + s) - e0);
    if (TAB) {
      toff[s] = (int32_t)(__ldg(tptr + m.s0 + s) - t0);
      if (s < m.ns) rs[s] = __ldg(runs + m.s0 + s);
    }
  }
  if (threadIdx.x == 0) fit_s = 0;
  __syncthreads();
  const int32_t tabs = TAB ? ((int32_t)sizeof(IDX) * toff[m.ns] + 15) & ~15 : 0;
  const bool all = TAB && tabs <= room / 4;
  for (int32_t s = threadIdx.x; s < m.ns; s += THREADS) {
    const int64_t with = all ? tabs : (int64_t)sizeof(IDX) * (TAB ? toff[s + 1] : off[s + 1]);
    if (8 * (int64_t)off[s + 1] + with <= room) atomicMax(&fit_s, s + 1);
  }
  __syncthreads();
  m.fit = fit_s;
  m.tfit = all ? m.ns : m.fit;
  m.off = off;
  m.toff = toff;
  m.runs = rs;
  m.gv = svals + e0;
  m.gc = reinterpret_cast<const IDX*>(cols) + t0;
  const int32_t held = off[m.fit], theld = TAB ? toff[m.tfit] : held;
  double* sv = reinterpret_cast<double*>(mat);
  IDX* sc = reinterpret_cast<IDX*>(sv + held);
  for (int32_t k = threadIdx.x; k < held; k += THREADS) sv[k] = __ldg(m.gv + k);
  for (int32_t k = threadIdx.x; k < theld; k += THREADS) sc[k] = __ldg(m.gc + k);
  m.sv = sv;
  m.sc = sc;
  __syncthreads();
}

template <typename IDX, bool TAB, typename G>
__device__ __forceinline__ double block_row(const BlockMatrix<IDX, TAB>& m, int32_t s, int lane, int32_t row,
                                            const G& g) {
  const int32_t o = m.off[s], w = (m.off[s + 1] - o) >> 5;
  if constexpr (!TAB) {
    if (s < m.fit) return lane_row<16, true>(m.sv + o + lane, m.sc + o + lane, w, row, g);
    return lane_row<16, false>(m.gv + o + lane, m.gc + o + lane, w, row, g);
  } else {
    const int32_t t = m.toff[s], first = m.runs[s];
    if (first >= 0) {
      const int s1 = first & 255, s2 = (first >> 8) & 255, s3 = first >> 16;
      const int run = (lane >= s1) + (lane >= s2) + (lane >= s3), nruns = 1 + (s1 < 32) + (s2 < 32) + (s3 < 32);
      if (s < m.fit) return table_row<true, true>(m.sv + o + lane, m.sc + t, w, run, nruns, row, g);
      if (s < m.tfit) return table_row<false, true>(m.gv + o + lane, m.sc + t, w, run, nruns, row, g);
      return table_row<false, false>(m.gv + o + lane, m.gc + t, w, run, nruns, row, g);
    }
    if (s < m.fit) return offset_row<true>(m.sv + o + lane, m.sc + t + lane, w, row, g);
    return offset_row<false>(m.gv + o + lane, m.gc + t + lane, w, row, g);
  }
}

}  // namespace femk
