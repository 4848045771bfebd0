// Parts shared by the kernels that run all steps of a call in one launch
// (fit_loop.cu: FP64 and FP32, fit_loop_comp.cu: the compensated state): the
// split of a grid into tiles, the lists of a tile's cells, the grid barrier.
#pragma once
#include <stdint.h>

#include "fit_rows.cuh"
#include "tma_util.cuh"

namespace wk {

constexpr int kLoopThreads = 512;
constexpr int kLoopMat = 64;              // materials staged in shared memory
constexpr int kLoopSmem = 226 * 1024;
constexpr int kLoopDim = 62;              // largest tile dimension (6-bit box coordinates)

// words of wk_fit_desc.sync, one per 128 bytes
constexpr int kSyncCount = 0, kSyncDone = 32, kSyncAbort = 64;

// Tile split of a grid: block (bx, by, bz) owns [bx Nx / nbx, (bx+1) Nx / nbx)
// and so on; the largest tile sets the shared-memory layout.
struct LoopTiling {
  int nbx, nby, nbz;
  int tx, ty, tz;
};

// List entries: box coordinates (6 bits each), the nine factor bits
// (RowBits), the three row bits and the class.
enum RowBits { bXO = 1, bXZ = 2, bXY = 4, bYO = 8, bYZ = 16, bYX = 32, bZO = 64, bZX = 128, bZY = 256 };
constexpr uint32_t kRegular = 0, kMasked = 1, kWrapped = 2;
__device__ __forceinline__ uint32_t loop_entry(int a, int b, int c, int cols, int rows,
                                               uint32_t cls) {
  return (uint32_t)a | (uint32_t)b << 6 | (uint32_t)c << 12 | (uint32_t)cols << 18 |
         (uint32_t)rows << 27 | cls << 30;
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* a) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a) : "memory");
  return v;
}
__device__ __forceinline__ void red_release(unsigned* a) {
  asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a) : "memory");
}

// Whether a count that wraps at 2^32 (29 million steps of 148 blocks) has reached
// the target, from which it is never further than a grid.
__host__ __device__ __forceinline__ bool loop_arrived(unsigned count, unsigned target) {
  return (int)(count - target) >= 0;
}
// Thread 0: wait until `target` arrivals were counted.  False when the wait
// ran out or another block gave up.
__device__ __forceinline__ bool loop_wait(unsigned* sync, unsigned target, long long limit_ns) {
  if (limit_ns < 0) return false;
  if (loop_arrived(ld_acquire(sync + kSyncCount), target)) return true;
  const unsigned long long t0 = globaltimer_ns();
  for (long long it = 0; it < kWaitPolls; it++) {
    if (loop_arrived(ld_acquire(sync + kSyncCount), target)) return true;
    if ((it & 63) == 63 && (ld_acquire(sync + kSyncAbort) != 0 ||
                            (long long)(globaltimer_ns() - t0) > limit_ns))
      return false;
  }
  return false;
}

// Factor bits of a cell's rows in direction DIR and whether a factor that is
// not 0, of a row that is not masked (`rows`), takes a length other than the
// cell's own.
template <typename T, int DIR>
__device__ __forceinline__ int loop_bits(const FitParams<T>& p, Cell c, int rows, bool& wrap) {
  ColumnInv<T, DIR> ci;
  ci.init(p, c.i, c.j);
  const RowCols<T> f = ci.at(p, c.k);
  auto bit = [](T v, int b) { return v != T(0) ? b : 0; };
  int m = bit(f.xO, bXO) | bit(f.xZ, bXZ) | bit(f.xY, bXY) | bit(f.yO, bYO) | bit(f.yZ, bYZ) |
          bit(f.yX, bYX) | bit(f.zO, bZO) | bit(f.zX, bZX) | bit(f.zY, bZY);
  const bool wx = DIR > 0 ? c.i == p.Nx - 1 : c.i == 0;
  wrap = (wx && (m & bYX) && (rows & 4)) || (ci.dkx && (m & bZX) && (rows & 2)) ||
         (ci.dky && (m & bZY) && (rows & 1));
  return m;
}

// One more entry of `key` for every thread of the warp with take: its place
// in counters[key] (the places of a warp's entries follow each other).  Called
// by whole warps.
__device__ __forceinline__ int loop_place(bool take, int key, int* counters) {
  const int lane = threadIdx.x & 31;
  const unsigned same = __match_any_sync(0xffffffffu, take ? key : -1);
  const int leader = __ffs(same) - 1;
  int base = 0;
  if (take && lane == leader) base = atomicAdd(counters + key, __popc(same));
  base = __shfl_sync(0xffffffffu, base, leader);
  return base + __popc(same & ((1u << lane) - 1));
}

// Division of 0 <= n < 2^20 by d through a rounded-up reciprocal (exact:
// the error n * 2^-32 * d / d stays below 1 / d).
struct LoopDiv {
  unsigned m;
  __device__ __forceinline__ explicit LoopDiv(int d) : m(d == 1 ? 0u : 0xffffffffu / (unsigned)d + 1u) {}
  __device__ __forceinline__ int div(int n) const { return m ? (int)__umulhi((unsigned)n, m) : n; }
};

// The lists of a block's cells, in one counting and one placing pass: for
// q < n, key = entry(q, e) gives the list entry e and its key (-1: none).  List
// 0 (H cells) holds keys 0 to 5 in this order, list 1 (E cells) keys 6 to 8,
// list 2 (the halo) key 9.  len[0..2]: entries; len[3]: those of keys 0 to 2.
// Called by all threads; count and len in shared memory.
template <typename FH, typename FE, typename FS>
__device__ __forceinline__ void loop_lists(int* count, int* len, int nh, FH h_entry, uint32_t* lh,
                                           int ne, FE e_entry, uint32_t* le, int ns, FS s_entry,
                                           uint32_t* ls) {
  const int tid = threadIdx.x;
  auto one = [&](int n, auto&& entry, uint32_t* list, bool place) {
    for (int q0 = 0; q0 < n; q0 += kLoopThreads) {
      uint32_t e = 0;
      const int key = q0 + tid < n ? entry(q0 + tid, e) : -1;
      const int at = loop_place(key >= 0, key, count);
      if (place && key >= 0) list[at] = e;
    }
  };
  if (tid < 10) count[tid] = 0;
  __syncthreads();
  for (int pass = 0; pass < 2; pass++) {
    one(nh, h_entry, lh, pass == 1);
    one(ne, e_entry, le, pass == 1);
    one(ns, s_entry, ls, pass == 1);
    __syncthreads();
    if (pass == 0 && tid == 0) {
      for (int g = 0; g < 3; g++) {           // counts to first places, per list
        const int lo = g == 0 ? 0 : (g == 1 ? 6 : 9), hi = g == 0 ? 6 : (g == 1 ? 9 : 10);
        int sum = 0;
        for (int q = lo; q < hi; q++) {
          const int c = count[q];
          count[q] = sum;
          sum += c;
        }
        len[g] = sum;
      }
      len[3] = count[3];
    }
    __syncthreads();
  }
}

// End of a launch: the last block to leave sets the words back for the next.
__device__ __forceinline__ void loop_leave(unsigned* sync) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(sync + kSyncDone, 1u) == gridDim.x - 1) {
      __threadfence();
      atomicExch(sync + kSyncCount, 0u);
      atomicExch(sync + kSyncAbort, 0u);
      atomicExch(sync + kSyncDone, 0u);
    }
  }
}

// SMs of the current device; 0 on an error.
int loop_sms();

// The split whose largest tile takes the fewest cell updates per step: H on
// the tile and its low halo, E on the tile, the halo's loads (x faces count
// twice: a sector per cell).  layout(tx, ty, tz) gives the figures of a tile
// (bytes, n_ext, n_own, n_shell).  nbx = 0 when no split fits.
template <typename Layout>
LoopTiling loop_search(int Nx, int Ny, int Nz, int sms, Layout layout) {
  LoopTiling best = {0, 0, 0, 0, 0, 0};
  double best_cost = 0;
  for (int nx = 1; nx <= sms && nx <= Nx; nx++)
    for (int ny = 1; nx * ny <= sms && ny <= Ny; ny++) {
      const int nz = sms / (nx * ny) < Nz ? sms / (nx * ny) : Nz;
      const int tx = (Nx + nx - 1) / nx, ty = (Ny + ny - 1) / ny, tz = (Nz + nz - 1) / nz;
      if (tx > kLoopDim || ty > kLoopDim || tz > kLoopDim) continue;
      const auto lay = layout(tx, ty, tz);
      if (lay.bytes > kLoopSmem) continue;
      const double cost = lay.n_ext + lay.n_own + 0.5 * lay.n_shell + 1.0 * ty * tz;
      if (best.nbx == 0 || cost < best_cost) {
        best = {nx, ny, nz, tx, ty, tz};
        best_cost = cost;
      }
    }
  return best;
}

}  // namespace wk
