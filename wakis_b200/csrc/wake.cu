// Wake potential and impedance kernels (sm_100a) and their C-ABI launchers.
//
// wk_wake_potential  calc_long_WP_3d / calc_long_WP (wakis/wakeSolver.py:
//                    310-554): a block per 32 s samples, the transverse
//                    positions in upstream order with the running-sum
//                    carry-over, and the z sum in upstream's sequential
//                    order, so WP matches upstream value for value.
// wk_trans_wake      calc_trans_WP (556-612): per s sample the prefix sum
//                    of WP_3d in numpy's pairwise summation order.
// wk_dft_bins        the kept bins 0 <= f < fmax of np.fft.fft(x, n=N)
//                    (calc_long_Z / calc_trans_Z, 679-766) as a direct DFT.
#include <stdint.h>

#include <mutex>

#include "../../include/wakis_b200.h"
#include "abi_internal.h"

namespace {

// History column that sample s reads for the z index k of the sum, -1 for none
// (and the row and sign of the coefficient follow from k alone).
struct WakeArgs {
  int nz, k_off, ns, counter_moving, n_win, carry, Nzh;
  long long hist_nt, nt;
  double v, zmin_v, zmax_v, t0, ti, dt, qnorm;
};
template <typename Idx>
__device__ __forceinline__ Idx wake_column(const WakeArgs& g, const double* __restrict__ z,
                                           const long long* __restrict__ key_order, double sn,
                                           int k) {
  const int kr = g.counter_moving ? g.nz - 1 - k : k;
  const double zk = __ldg(z + kr);
  const double ts =
      g.counter_moving
          ? __dadd_rn(__dsub_rn(__dsub_rn(__ddiv_rn(__dsub_rn(zk, sn), -g.v), g.zmax_v), g.t0), g.ti)
          : __dadd_rn(__dsub_rn(__dsub_rn(__ddiv_rn(__dadd_rn(zk, sn), g.v), g.zmin_v), g.t0), g.ti);
  long long it = (long long)__ddiv_rn(ts, g.dt);   // truncation toward zero, as int()
  if (it >= g.nt) return -1;
  if (it < 0) it += g.nt;                          // negative index wraps as in numpy
  if (it < 0) return -1;
  const long long t = __ldg(key_order + it);
  return t >= 0 && t < g.hist_nt ? (Idx)t : -1;    // -1: no such history column
}

// One block per 32 samples.  The sum over z is sequential, window after window
// (each starts from the one before), so the adds of a sample form one chain of
// n_win nz terms: warp 8 runs the chains of the block's samples, one per lane,
// and warps 0 to 7 form the terms, kWakeChunk at a time into one of two
// shared-memory buffers, the history entries of a chunk (consecutive columns
// of a row for the lanes of a warp) being read while the chunk before is
// formed.  A term that does not exist is -0, which leaves any sum as it is.
// The columns, two divisions each, are formed once per (sample, z) and kept in
// shared memory for the other windows when they fit (COLS).  Idx: long long
// where a column or a term's number does not fit an int.
// Bound by the latency of the history: two entries of two chunks are on their way
// in a forming thread, and a barrier ends every 16 terms, so that a term takes
// some 140 cycles of a sample's 3600, of which the dependent add about ten; the
// history's read is at 1.3 TB/s.  On B200, 9 windows of nz = 400, ns = 11700,
// FP64: 267 us (345 MB), nz = 120, ns = 4700 54 us; nz = 400, ns = 10618: 2632 with
// one thread per sample that formed the column of every term and waited for its
// entry, 1158 with one warp per block doing both parts; 4 terms per warp and chunk
// 257, and 85 for nz = 120.
constexpr int kWakeProd = 8, kWakeEach = 2, kWakeChunk = kWakeProd * kWakeEach;
template <typename H, bool COLS, typename Idx>
__global__ void __launch_bounds__((kWakeProd + 1) * 32)
k_wake_potential(const H* __restrict__ hist, const int* __restrict__ win_map,
                 const double* __restrict__ z, const double* __restrict__ dz,
                 const double* __restrict__ s, const long long* __restrict__ key_order,
                 WakeArgs g, double* __restrict__ WP3d) {
  extern __shared__ __align__(16) unsigned char wake_smem[];
  double* term = reinterpret_cast<double*>(wake_smem);              // [2][kWakeChunk][32]
  int* cols = reinterpret_cast<int*>(term + 2 * kWakeChunk * 32);   // [nz][32] (COLS)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = blockIdx.x * 32 + lane;
  const bool on = n < g.ns;
  const Idx terms = (Idx)g.n_win * g.nz;
  const Idx chunks = (terms + kWakeChunk - 1) / kWakeChunk;
  if (terms == 0) {                          // empty sums
    double acc = 0.0;
    for (int w = 0; w < g.n_win && warp == 0 && on; w++) {
      acc = __ddiv_rn(g.carry ? acc : 0.0, g.qnorm);
      WP3d[(long long)w * g.ns + n] = acc;
    }
    return;
  }
  if (warp < kWakeProd) {
    const double sn = s[on ? n : g.ns - 1];
    // entry and coefficient of term q (window q / nz, z index q % nz): the
    // columns of window 0 are formed here, the others find them in `cols`
    // (written three chunks before at least)
    struct Terms {
      double coef[kWakeEach];
      H entry[kWakeEach];
      bool have[kWakeEach];
    };
    auto read = [&](Idx chunk, Terms& v) {
      const Idx q0 = chunk * kWakeChunk + warp * kWakeEach;
      int w = (int)(q0 / g.nz), k = (int)(q0 - (Idx)w * g.nz);
#pragma unroll
      for (int u = 0; u < kWakeEach; u++) {
        v.have[u] = false;
        if (q0 + u < terms) {
          const Idx t = COLS && w > 0 ? cols[k * 32 + lane]
                                      : (on ? wake_column<Idx>(g, z, key_order, sn, k) : -1);
          if (COLS && w == 0) cols[k * 32 + lane] = t;
          const int kz = (g.counter_moving ? g.nz - 1 - k : k) + g.k_off;
          const double c = __ldg(dz + k);
          v.coef[u] = g.counter_moving ? -c : c;
          v.have[u] = t >= 0;
          v.entry[u] = v.have[u]
                           ? hist[((long long)__ldg(win_map + w) * g.Nzh + kz) * g.hist_nt + t]
                           : H(0);
        }
        if (++k == g.nz) { k = 0; w++; }
      }
    };
    auto put = [&](Idx chunk, const Terms& v) {
      double* out = term + (chunk & 1) * kWakeChunk * 32 + warp * kWakeEach * 32 + lane;
#pragma unroll
      for (int u = 0; u < kWakeEach; u++)
        out[u * 32] = v.have[u] ? __dmul_rn((double)v.entry[u], v.coef[u]) : -0.0;
      __syncthreads();                       // the chunk is formed, the one before summed
    };
    // the entries of two chunks are on their way while a third is formed
    Terms va, vb;
    read(0, va);
    read(1, vb);
    for (Idx c = 0; c < chunks; c += 2) {
      put(c, va);
      read(c + 2, va);
      if (c + 1 < chunks) {
        put(c + 1, vb);
        read(c + 3, vb);
      }
    }
  } else {
    double acc = 0.0;
    int w = 0, k = 0;
    for (Idx c = 0; c < chunks; c++) {
      __syncthreads();
      const double* in = term + (c & 1) * kWakeChunk * 32 + lane;
      if (k + kWakeChunk < g.nz) {           // no window ends in this chunk
        double v[kWakeChunk];
#pragma unroll
        for (int u = 0; u < kWakeChunk; u++) v[u] = in[u * 32];
#pragma unroll
        for (int u = 0; u < kWakeChunk; u++) acc = __dadd_rn(acc, v[u]);
        k += kWakeChunk;
      } else {
#pragma unroll 1
        for (int u = 0; u < kWakeChunk && c * kWakeChunk + u < terms; u++) {
          acc = __dadd_rn(acc, in[u * 32]);
          if (++k == g.nz) {
            acc = __ddiv_rn(acc, g.qnorm);
            if (on) WP3d[(long long)w * g.ns + n] = acc;
            if (!g.carry) acc = 0.0;
            k = 0;
            w++;
          }
        }
      }
    }
  }
}

// Largest nz whose columns are kept in shared memory; the least is such that a
// column is written at least one barrier before it is read.
constexpr int kWakeColsMax = 1024, kWakeColsMin = 4 * kWakeChunk;
constexpr int kWakeTermBytes = 2 * kWakeChunk * 32 * 8;

template <typename H>
cudaError_t launch_wake_potential(const H* hist, const int* win_map, const double* z,
                                  const double* dz, const double* s, const long long* key_order,
                                  const WakeArgs& g, double* WP3d, cudaStream_t st) {
  const int blocks = (g.ns + 31) / 32;
  const int threads = (kWakeProd + 1) * 32;
  const long long most = 0x7fffffffLL - 4 * kWakeChunk;
  if (g.hist_nt > most || (long long)g.n_win * g.nz > most) {
    k_wake_potential<H, false, long long><<<blocks, threads, kWakeTermBytes, st>>>(
        hist, win_map, z, dz, s, key_order, g, WP3d);
  } else if (g.nz >= kWakeColsMin && g.nz <= kWakeColsMax) {
    cudaError_t e = cudaFuncSetAttribute(k_wake_potential<H, true, int>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kWakeTermBytes + kWakeColsMax * 128);
    if (e != cudaSuccess) return e;
    k_wake_potential<H, true, int><<<blocks, threads, kWakeTermBytes + g.nz * 128, st>>>(
        hist, win_map, z, dz, s, key_order, g, WP3d);
  } else {
    k_wake_potential<H, false, int><<<blocks, threads, kWakeTermBytes, st>>>(
        hist, win_map, z, dz, s, key_order, g, WP3d);
  }
  return cudaGetLastError();
}

// numpy's pairwise summation (blocks of <= 128 with 8 accumulators, halves
// rounded down to a multiple of 8), evaluated with an explicit stack.
__device__ double pw_leaf(const double* a, long long n) {
  if (n < 8) {
    double r = -0.0;
    for (long long i = 0; i < n; i++) r = __dadd_rn(r, a[i]);
    return r;
  }
  double r[8];
  for (int j = 0; j < 8; j++) r[j] = a[j];
  long long i = 8;
  for (; i < n - (n % 8); i += 8)
    for (int j = 0; j < 8; j++) r[j] = __dadd_rn(r[j], a[i + j]);
  double res = __dadd_rn(__dadd_rn(__dadd_rn(r[0], r[1]), __dadd_rn(r[2], r[3])),
                         __dadd_rn(__dadd_rn(r[4], r[5]), __dadd_rn(r[6], r[7])));
  for (; i < n; i++) res = __dadd_rn(res, a[i]);
  return res;
}

__device__ __forceinline__ long long pw_half(long long n) {
  long long n2 = n / 2;
  return n2 - n2 % 8;
}

__device__ double pw_sum(const double* a, long long n) {
  long long lo_s[48], n_s[48];
  double left_s[48];
  int stage[48];
  int sp = 0;
  lo_s[0] = 0; n_s[0] = n; stage[0] = 0;
  while (true) {
    long long m = n_s[sp];
    if (m <= 128) {
      double result = pw_leaf(a + lo_s[sp], m);
      while (true) {
        if (sp == 0) return result;
        sp--;
        if (stage[sp] == 1) {
          left_s[sp] = result;
          stage[sp] = 2;
          long long n2 = pw_half(n_s[sp]);
          lo_s[sp + 1] = lo_s[sp] + n2;
          n_s[sp + 1] = n_s[sp] - n2;
          stage[sp + 1] = 0;
          sp++;
          break;
        }
        result = __dadd_rn(left_s[sp], result);
      }
    } else {
      stage[sp] = 1;
      lo_s[sp + 1] = lo_s[sp];
      n_s[sp + 1] = pw_half(m);
      stage[sp + 1] = 0;
      sp++;
    }
  }
}

// The same sums of [lo, lo + n) of four arrays by a group of 8 lanes (`mask`,
// lane j of the group holds accumulator j), the result in all of them.
struct Pw4 { double v[4]; };
__device__ __forceinline__ Pw4 pw_leaf4(const double* const* a, int lo, int n, int j,
                                        unsigned mask) {
  Pw4 r;
  if (n < 8) {
#pragma unroll
    for (int q = 0; q < 4; q++) r.v[q] = -0.0;
    for (int i = 0; i < n; i++)
#pragma unroll
      for (int q = 0; q < 4; q++) r.v[q] = __dadd_rn(r.v[q], a[q][lo + i]);
    return r;
  }
#pragma unroll
  for (int q = 0; q < 4; q++) r.v[q] = a[q][lo + j];
  int i = 8;
  for (; i < n - (n % 8); i += 8)
#pragma unroll
    for (int q = 0; q < 4; q++) r.v[q] = __dadd_rn(r.v[q], a[q][lo + i + j]);
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int x = 1; x < 8; x *= 2)
      r.v[q] = __dadd_rn(r.v[q], __shfl_xor_sync(mask, r.v[q], x));
  for (; i < n; i++)
#pragma unroll
    for (int q = 0; q < 4; q++) r.v[q] = __dadd_rn(r.v[q], a[q][lo + i]);
  return r;
}
// ... of at most 128 * 2^D values, by a tree of calls.
template <int D>
__device__ __noinline__ Pw4 pw_tree4(const double* const* a, int lo, int n, int j, unsigned mask) {
  if (n <= 128) return pw_leaf4(a, lo, n, j, mask);
  Pw4 r;
  if constexpr (D > 0) {
    const int n2 = (int)pw_half(n);
    const Pw4 left = pw_tree4<D - 1>(a, lo, n2, j, mask);
    r = pw_tree4<D - 1>(a, lo + n2, n - n2, j, mask);
#pragma unroll
    for (int q = 0; q < 4; q++) r.v[q] = __dadd_rn(left.v[q], r.v[q]);
  } else {
#pragma unroll
    for (int q = 0; q < 4; q++) r.v[q] = pw_sum(a[q] + lo, n);
  }
  return r;
}

// numpy's pairwise sums of a[q][0 .. n) by one warp (the results in lane 0):
// the first five splits give 32 nodes (the bits of a node's number, highest
// first, choose left or right), summed four at a time by the groups of 8 lanes,
// one per lane afterwards, and added pair by pair; a node that is a leaf before
// the fifth split is the one whose further bits are 0.
__device__ __forceinline__ Pw4 pw_warp4(const double* const* a, int n, int lane) {
  auto node = [&](int id, int& lo, int& len, int& depth) {
    lo = 0;
    len = n;
    depth = 0;
    bool there = true;
#pragma unroll
    for (int b = 4; b >= 0; b--) {
      const bool right = id >> b & 1;
      if (len > 128) {
        const int n2 = (int)pw_half(len);
        lo += right ? n2 : 0;
        len = right ? len - n2 : n2;
        depth++;
      } else if (right) {
        there = false;
      }
    }
    return there;
  };
  const int grp = lane >> 3, j = lane & 7;
  const unsigned mask = 0xffu << (8 * grp);
  Pw4 r = {{0.0, 0.0, 0.0, 0.0}};
  int lo, len, depth;
  for (int it = 0; it < 8; it++) {
    Pw4 v = {{0.0, 0.0, 0.0, 0.0}};
    if (node(it * 4 + grp, lo, len, depth))
      v = len <= 128 ? pw_leaf4(a, lo, len, j, mask) : pw_tree4<4>(a, lo, len, j, mask);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 4; q++) {
      // node it * 4 + g is in the lanes of group g, and wanted by lane it * 4 + g
      const double x = __shfl_sync(0xffffffffu, v.v[q], (lane & 3) * 8);
      if (lane >> 2 == it) r.v[q] = x;
    }
  }
  node(lane, lo, len, depth);
#pragma unroll
  for (int b = 0; b < 5; b++)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const double o = __shfl_down_sync(0xffffffffu, r.v[q], 1 << b);
      if (depth >= 5 - b) r.v[q] = __dadd_rn(r.v[q], o);
    }
  return r;
}

// Positions (+1,0) (-1,0) (0,+1) (0,-1) are w = 7, 1, 5, 3 of the 3x3 block;
// one warp forms the four prefix integrals of a sample.  O(ns^2) adds in
// numpy's order.  On B200, ns = 10618: 149 us; 1052 with one thread
// per sample, 623 with one node per lane (32 lines a load).
constexpr int kTransWarps = 8;
__global__ void __launch_bounds__(kTransWarps * 32)
k_trans_wake(const double* __restrict__ WP3d, int ns, double ds, double dxsum, double dysum,
             double* __restrict__ WPx, double* __restrict__ WPy) {
  // the longest prefixes first
  const int n = ns - 1 - (int)(blockIdx.x * kTransWarps + (threadIdx.x >> 5));
  if (n < 0) return;
  const double* const a[4] = {WP3d + 7LL * ns, WP3d + 1LL * ns, WP3d + 5LL * ns, WP3d + 3LL * ns};
  const Pw4 r = pw_warp4(a, n, threadIdx.x & 31);
  if ((threadIdx.x & 31) == 0) {
    WPx[n] = __ddiv_rn(-__dsub_rn(__dmul_rn(r.v[0], ds), __dmul_rn(r.v[1], ds)), dxsum);
    WPy[n] = __ddiv_rn(-__dsub_rn(__dmul_rn(r.v[2], ds), __dmul_rn(r.v[3], ds)), dysum);
  }
}

// Axes longer than the tree of calls reaches (128 * 2^9 samples): one thread per
// sample.  A warp per sample would walk the long nodes lane by lane: 90000
// samples 31.3 ms, so 11.3; with a deeper tree of calls (255 registers) 15.5,
// 200000 samples 78 and 35.  At 65536 the warps take 4.7 ms and the threads 6.5.
constexpr int kTransWarpMax = 65536;
__global__ void k_trans_wake_long(const double* __restrict__ WP3d, int ns, double ds, double dxsum,
                                  double dysum, double* __restrict__ WPx,
                                  double* __restrict__ WPy) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= ns) return;
  const double ixp = __dmul_rn(pw_sum(WP3d + 7LL * ns, n), ds);
  const double ixm = __dmul_rn(pw_sum(WP3d + 1LL * ns, n), ds);
  const double iyp = __dmul_rn(pw_sum(WP3d + 5LL * ns, n), ds);
  const double iym = __dmul_rn(pw_sum(WP3d + 3LL * ns, n), ds);
  WPx[n] = __ddiv_rn(-__dsub_rn(ixp, ixm), dxsum);
  WPy[n] = __ddiv_rn(-__dsub_rn(iyp, iym), dysum);
}

// ------------------------------------------------------------- streaming --
// The s sample index n and z index k of the sum for WP(s_n) read step
// it(n, k) = (long)(ts/dt) (same rounded expression as k_wake_potential).
__device__ __forceinline__ long long wp_it(double zk, double sn, double v, double zmin_v,
                                           double zmax_v, double t0, double ti, double dt,
                                           int counter_moving) {
  double ts;
  if (!counter_moving)
    ts = __dadd_rn(__dsub_rn(__dsub_rn(__ddiv_rn(__dadd_rn(zk, sn), v), zmin_v), t0), ti);
  else
    ts = __dadd_rn(__dsub_rn(__dsub_rn(__ddiv_rn(__dsub_rn(zk, sn), -v), zmax_v), t0), ti);
  return (long long)__ddiv_rn(ts, dt);
}

// One thread per (window w, z index k, step r of the chunk): the steps
// step0 .. step0+n_steps-1 of the Ez window history are in ring columns
// 0 .. n_steps-1.  Step m sits at position p = pos[m] of upstream's sorted
// key list (pos = NULL: p = m); it adds Ez(w, k, m) * coef_k to acc[w][n]
// for every s sample n whose sum reads position p, i.e. it(n, k) == p.
// it(n, k) = it(0, k) + n within one (the s axis steps by v*dt), so the
// candidates are n = p - it(0, k) + [-4, 4], each tested with the exact
// expression.
template <typename H>
__global__ void k_wake_accumulate(const H* __restrict__ ring, long long ring_nt, int Nzh,
                                  long long step0, int n_steps, const int* __restrict__ win_map,
                                  int n_win, const double* __restrict__ z,
                                  const double* __restrict__ dz, int nz, int k_off,
                                  const double* __restrict__ s, int ns,
                                  const long long* __restrict__ pos, long long nt, double v,
                                  double zmin, double zmax, double t0, double ti, double dt,
                                  int counter_moving, double* __restrict__ acc) {
  const long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long per_w = (long long)nz * n_steps;
  if (g >= per_w * n_win) return;
  const int w = (int)(g / per_w);
  const long long rem = g - w * per_w;
  const int k = (int)(rem / n_steps);
  const int r = (int)(rem - (long long)k * n_steps);
  const long long m = step0 + r;
  const long long p = pos ? pos[m] : m;
  if (p < 0 || p >= nt) return;
  const double zmin_v = __ddiv_rn(zmin, v);
  const double zmax_v = __ddiv_rn(zmax, -v);
  int kz;
  double zk, coef;
  if (!counter_moving) {
    zk = z[k]; kz = k + k_off; coef = dz[k];
  } else {
    const int kr = nz - 1 - k;
    zk = z[kr]; kz = kr + k_off; coef = -dz[k];
  }
  const double e = (double)ring[((long long)win_map[w] * Nzh + kz) * ring_nt + r];
  const long long it0 = wp_it(zk, s[0], v, zmin_v, zmax_v, t0, ti, dt, counter_moving);
  const long long n_est = p - it0;
  for (long long n = n_est - 4; n <= n_est + 4; n++) {
    if (n < 0 || n >= ns) continue;
    if (wp_it(zk, s[n], v, zmin_v, zmax_v, t0, ti, dt, counter_moving) == p)
      atomicAdd(acc + (long long)w * ns + n, __dmul_rn(e, coef));
  }
}

// WP_3d[w][n] = ((carry ? WP_3d[w-1][n] : 0) + acc[w][n]) / qnorm, the
// windows in order (upstream's carry-over, wakeSolver.py:485,536).
__global__ void k_wake_finalize(const double* __restrict__ acc, int n_win, int ns, int carry,
                                double qnorm, double* __restrict__ WP3d) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= ns) return;
  double prev = 0.0;
  for (int w = 0; w < n_win; w++) {
    const double a = __ddiv_rn(__dadd_rn(carry ? prev : 0.0, acc[(long long)w * ns + n]), qnorm);
    WP3d[(long long)w * ns + n] = a;
    prev = a;
  }
}

// -------------------------------------------------- transverse, by scans --
// Double-double running sums (TwoSum, Knuth): the prefix integrals of the
// Panofsky-Wenzel transverse wake to ~106 bits, rounded once, for long s
// axes where the per-sample pairwise sums of k_trans_wake (O(ns^2)) do not
// scale.  Positions w = 7, 1, 5, 3 of the 3x3 block.
struct DD { double hi, lo; };
__device__ __forceinline__ DD dd_add(DD a, double b) {
  const double s = __dadd_rn(a.hi, b);
  const double bb = __dsub_rn(s, a.hi);
  const double err = __dadd_rn(__dsub_rn(a.hi, __dsub_rn(s, bb)), __dsub_rn(b, bb));
  const double lo = __dadd_rn(a.lo, err);
  const double hi = __dadd_rn(s, lo);
  return {hi, __dsub_rn(lo, __dsub_rn(hi, s))};
}
__device__ __forceinline__ DD dd_add(DD a, DD b) {
  DD r = dd_add(a, b.hi);
  return dd_add(r, b.lo);
}

__device__ __forceinline__ DD dd_mul(double a, double b) {   // exact product
  const double p = __dmul_rn(a, b);
  return {p, __fma_rn(a, b, -p)};
}

constexpr int kScanThreads = 256;
__device__ __forceinline__ int trans_win(int q) { return q == 0 ? 7 : (q == 1 ? 1 : (q == 2 ? 5 : 3)); }

// Segment g of `seg` samples: its four window sums (double-double) into
// part[g][4] (scratch).  Deterministic: each thread sums a fixed stride,
// then a fixed-shape tree.
__global__ void k_trans_part(const double* __restrict__ WP3d, int ns, int seg,
                             DD* __restrict__ part) {
  __shared__ DD red[4][kScanThreads];
  const int g = blockIdx.x;
  const long long a = (long long)g * seg, b = min((long long)ns, a + seg);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    DD acc = {0.0, 0.0};
    const double* x = WP3d + (long long)trans_win(q) * ns;
    for (long long n = a + threadIdx.x; n < b; n += kScanThreads) acc = dd_add(acc, x[n]);
    red[q][threadIdx.x] = acc;
  }
  __syncthreads();
  for (int h = kScanThreads / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h)
#pragma unroll
      for (int q = 0; q < 4; q++) red[q][threadIdx.x] = dd_add(red[q][threadIdx.x], red[q][threadIdx.x + h]);
    __syncthreads();
  }
  if (threadIdx.x < 4) part[(long long)g * 4 + threadIdx.x] = red[threadIdx.x][0];
}

// Exclusive scan of the segment sums, in place (one thread per window).
__global__ void k_trans_part_scan(DD* __restrict__ part, int nseg) {
  const int q = threadIdx.x;
  if (q >= 4) return;
  DD run = {0.0, 0.0};
  for (int g = 0; g < nseg; g++) {
    const DD v = part[(long long)g * 4 + q];
    part[(long long)g * 4 + q] = run;
    run = dd_add(run, v);
  }
}

// Segment g: from the segment offsets, thread 0 walks windows 7 and 1
// (WPx), thread 1 windows 5 and 3 (WPy): the exclusive prefix of each
// sample, rounded once and times ds, then the difference quotient.
__global__ void k_trans_final(const double* __restrict__ WP3d, int ns, int seg,
                              const DD* __restrict__ part, double ds, double dxsum,
                              double dysum, double* __restrict__ WPx, double* __restrict__ WPy) {
  const int g = blockIdx.x;
  const int t = threadIdx.x;
  if (t >= 2) return;
  const long long a = (long long)g * seg, b = min((long long)ns, a + seg);
  const int qp = 2 * t, qm = 2 * t + 1;             // (7, 1) or (5, 3)
  const double* xp = WP3d + (long long)trans_win(qp) * ns;
  const double* xm = WP3d + (long long)trans_win(qm) * ns;
  double* out = t == 0 ? WPx : WPy;
  const double den = t == 0 ? dxsum : dysum;
  DD rp = part[(long long)g * 4 + qp], rm = part[(long long)g * 4 + qm];
  for (long long n = a; n < b; n++) {
    const double ip = __dmul_rn(__dadd_rn(rp.hi, rp.lo), ds);
    const double im = __dmul_rn(__dadd_rn(rm.hi, rm.lo), ds);
    out[n] = __ddiv_rn(-__dsub_rn(ip, im), den);
    rp = dd_add(rp, xp[n]);
    rm = dd_add(rm, xm[n]);
  }
}

// One block per (signal, bin).  With w = exp(-2 pi i m / N), thread t sums
// x[t + T a] w^(T a) over a and multiplies once by w^t, so that a bin takes
// about T + len / T exponentials instead of len; the exponentials w^(T a) come
// from shared memory, kDftChunk at a time.  Fixed-shape tree reduction
// (deterministic).  40 registers, six blocks an SM (without the bound 42: five,
// 4 signals 47.2 us for 45.1).  On B200, 984 bins of 11700 samples, 4 signals: 45
// us, 209 with one exponential per term.
constexpr int kDftThreads = 256, kDftChunk = 256;
// cos and sin of 2 pi m n / N, the angle brought within an eighth of a turn by
// exact integer quarter turns first (so that its rounding, relative to a small
// angle, stays far below the functions' own).
__device__ __forceinline__ void dft_unit(long long m, long long n, long long N, double* c,
                                         double* s) {
  const long long r = (m * n) % N;
  const long long q = (4 * r + N / 2) / N;            // quarter turns, 0 to 4
  double sn, cs;
  sincospi(__ddiv_rn((double)(4 * r - q * N), 2.0 * (double)N), &sn, &cs);
  const double c0 = q & 1 ? -sn : cs, s0 = q & 1 ? cs : sn;
  *c = q & 2 ? -c0 : c0;
  *s = q & 2 ? -s0 : s0;
}
// The bin term by term, for a sum that is not finite: an infinity times the two
// factors, or the error term of its product, is NaN, also where the sum is
// infinite.  `sre`, `sim`: kDftThreads words each, two apart.
__device__ __forceinline__ void dft_plain(const double* __restrict__ xs, long long len, int m,
                                       long long N, double* sre, double* sim, double* re_out,
                                       double* im_out) {
  const int t = threadIdx.x;
  double re = 0.0, im = 0.0, c, s;
  for (long long n = t; n < len; n += kDftThreads) {
    dft_unit(m, n, N, &c, &s);
    re = __dadd_rn(re, __dmul_rn(xs[n], c));
    im = __dsub_rn(im, __dmul_rn(xs[n], s));
  }
  __syncthreads();
  sre[2 * t] = re;
  sim[2 * t] = im;
  __syncthreads();
  for (int w = kDftThreads / 2; w > 0; w >>= 1) {
    if (t < w) {
      sre[2 * t] = __dadd_rn(sre[2 * t], sre[2 * (t + w)]);
      sim[2 * t] = __dadd_rn(sim[2 * t], sim[2 * (t + w)]);
    }
    __syncthreads();
  }
  *re_out = sre[0];
  *im_out = sim[0];
}
__global__ void __launch_bounds__(kDftThreads, 6)
k_dft_bins(const double* __restrict__ x, long long len, long long N, int nbins,
           double* __restrict__ out) {
  const int m = blockIdx.x, sig = blockIdx.y, t = threadIdx.x;
  const double* xs = x + (long long)sig * len;
  __shared__ double2 unit[kDftChunk];
  double re = 0.0, im = 0.0;
  const long long steps = (len + kDftThreads - 1) / kDftThreads;
  for (long long a0 = 0; a0 < steps; a0 += kDftChunk) {
    const int na = (int)min((long long)kDftChunk, steps - a0);
    if (t < na) dft_unit(m, (a0 + t) * kDftThreads, N, &unit[t].x, &unit[t].y);
    __syncthreads();
    for (int a = 0; a < na; a++) {
      const long long n = (a0 + a) * kDftThreads + t;
      if (n < len) {
        const double v = xs[n];
        re = __fma_rn(v, unit[a].x, re);
        im = __fma_rn(-v, unit[a].y, im);
      }
    }
    __syncthreads();
  }
  // (re + i im)(c - i s) and the tree in double-double: each bin is rounded once
  double c, s;
  dft_unit(m, t, N, &c, &s);
  __shared__ DD sre[kDftThreads], sim[kDftThreads];
  sre[t] = dd_add(dd_mul(re, c), dd_mul(im, s));
  sim[t] = dd_add(dd_mul(im, c), dd_mul(-re, s));
  __syncthreads();
  for (int w = kDftThreads / 2; w > 0; w >>= 1) {
    if (t < w) {
      sre[t] = dd_add(sre[t], sre[t + w]);
      sim[t] = dd_add(sim[t], sim[t + w]);
    }
    __syncthreads();
  }
  re = __dadd_rn(sre[0].hi, sre[0].lo);
  im = __dadd_rn(sim[0].hi, sim[0].lo);
  if (!isfinite(re) || !isfinite(im)) dft_plain(xs, len, m, N, &sre[0].hi, &sim[0].hi, &re, &im);
  if (t == 0) {
    out[((long long)sig * nbins + m) * 2] = re;
    out[((long long)sig * nbins + m) * 2 + 1] = im;
  }
}

}  // namespace

extern "C" int wk_wake_potential(const void* hist, int hist_dtype, long long hist_nt, int Nzh,
                                 const int* win_map, int n_win, int carry, const double* z,
                                 const double* dz, int nz, int k_off, const double* s, int ns,
                                 const long long* key_order, long long nt, double v,
                                 double zmin, double zmax, double t0, double ti, double dt,
                                 double qnorm, int counter_moving, double* WP3d, void* stream) {
  if (!hist || !win_map || !z || !dz || !s || !key_order || !WP3d)
    return wk_fail(WK_E_NULL, "wk_wake_potential: NULL pointer");
  if (hist_dtype != WK_F64 && hist_dtype != WK_F32)
    return wk_fail(WK_E_DTYPE, "wk_wake_potential: hist dtype %d", hist_dtype);
  if (ns < 0 || nz < 0 || n_win < 1 || hist_nt < 1 || Nzh < 1 || k_off < 0 ||
      k_off + nz > Nzh || nt > hist_nt)
    return wk_fail(WK_E_RANGE, "wk_wake_potential: sizes (ns %d nz %d nwin %d nt %lld)",
                   ns, nz, n_win, nt);
  if (ns == 0) return WK_OK;
  cudaStream_t st = (cudaStream_t)stream;
  WakeArgs g;
  g.nz = nz; g.k_off = k_off; g.ns = ns; g.counter_moving = counter_moving;
  g.n_win = n_win; g.carry = carry; g.Nzh = Nzh;
  g.hist_nt = hist_nt; g.nt = nt;
  g.v = v; g.zmin_v = zmin / v; g.zmax_v = zmax / -v; g.t0 = t0; g.ti = ti; g.dt = dt;
  g.qnorm = qnorm;
  const cudaError_t e =
      hist_dtype == WK_F64
          ? launch_wake_potential((const double*)hist, win_map, z, dz, s, key_order, g, WP3d, st)
          : launch_wake_potential((const float*)hist, win_map, z, dz, s, key_order, g, WP3d, st);
  if (e != cudaSuccess) return wk_fail(-(int)e, "wk_wake_potential: %s", cudaGetErrorString(e));
  return wk_check_launch("wk_wake_potential");
}

extern "C" int wk_trans_wake(const double* WP3d, int ns, double ds, double dxsum, double dysum,
                             double* WPx, double* WPy, void* stream) {
  if (!WP3d || !WPx || !WPy) return wk_fail(WK_E_NULL, "wk_trans_wake: NULL pointer");
  if (ns < 0) return wk_fail(WK_E_RANGE, "wk_trans_wake: ns %d", ns);
  if (ns == 0) return WK_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (ns > kTransWarpMax)
    k_trans_wake_long<<<(unsigned)((ns + 127LL) / 128), 128, 0, st>>>(WP3d, ns, ds, dxsum, dysum,
                                                                      WPx, WPy);
  else
    k_trans_wake<<<(ns + kTransWarps - 1) / kTransWarps, kTransWarps * 32, 0, st>>>(
        WP3d, ns, ds, dxsum, dysum, WPx, WPy);
  return wk_check_launch("wk_trans_wake");
}

extern "C" int wk_dft_bins(const double* x, int nsig, long long len, long long N, int nbins,
                           double* out, void* stream) {
  if (!x || !out) return wk_fail(WK_E_NULL, "wk_dft_bins: NULL pointer");
  if (nsig < 1 || len < 0 || nbins < 0 || N < 1 || len > N || nbins > N || nsig > 65535)
    return wk_fail(WK_E_RANGE, "wk_dft_bins: nsig %d len %lld N %lld nbins %d", nsig, len, N,
                   nbins);
  if (nbins == 0) return WK_OK;
  if ((double)N * (double)nbins > 9.0e18)
    return wk_fail(WK_E_RANGE, "wk_dft_bins: N*nbins overflows the index product");
  cudaStream_t st = (cudaStream_t)stream;
  dim3 grid(nbins, nsig);
  k_dft_bins<<<grid, kDftThreads, 0, st>>>(x, len, N, nbins, out);
  return wk_check_launch("wk_dft_bins");
}

extern "C" int wk_wake_accumulate(const void* ring, int ring_dtype, long long ring_nt, int Nzh,
                                  long long step0, int n_steps, const int* win_map, int n_win,
                                  const double* z, const double* dz, int nz, int k_off,
                                  const double* s, int ns, const long long* pos, long long nt,
                                  double v, double zmin, double zmax, double t0, double ti,
                                  double dt, int counter_moving, double* acc, void* stream) {
  if (!ring || !win_map || !z || !dz || !s || !acc)
    return wk_fail(WK_E_NULL, "wk_wake_accumulate: NULL pointer");
  if (ring_dtype != WK_F64 && ring_dtype != WK_F32)
    return wk_fail(WK_E_DTYPE, "wk_wake_accumulate: ring dtype %d", ring_dtype);
  if (ns < 0 || nz < 0 || n_win < 1 || n_steps < 0 || n_steps > ring_nt || Nzh < 1 ||
      k_off < 0 || k_off + nz > Nzh || step0 < 0 || nt < 0)
    return wk_fail(WK_E_RANGE, "wk_wake_accumulate: sizes (ns %d nz %d nwin %d steps %d)", ns,
                   nz, n_win, n_steps);
  if (ns == 0 || nz == 0 || n_steps == 0) return WK_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const long long total = (long long)n_win * nz * n_steps;
  const int threads = 256;
  const long long blocks = (total + threads - 1) / threads;
  if (blocks > 0x7fffffffLL) return wk_fail(WK_E_RANGE, "wk_wake_accumulate: too many steps");
  if (ring_dtype == WK_F64)
    k_wake_accumulate<double><<<(unsigned)blocks, threads, 0, st>>>(
        (const double*)ring, ring_nt, Nzh, step0, n_steps, win_map, n_win, z, dz, nz, k_off, s,
        ns, pos, nt, v, zmin, zmax, t0, ti, dt, counter_moving, acc);
  else
    k_wake_accumulate<float><<<(unsigned)blocks, threads, 0, st>>>(
        (const float*)ring, ring_nt, Nzh, step0, n_steps, win_map, n_win, z, dz, nz, k_off, s,
        ns, pos, nt, v, zmin, zmax, t0, ti, dt, counter_moving, acc);
  return wk_check_launch("wk_wake_accumulate");
}

extern "C" int wk_wake_finalize(const double* acc, int n_win, int ns, int carry, double qnorm,
                                double* WP3d, void* stream) {
  if (!acc || !WP3d) return wk_fail(WK_E_NULL, "wk_wake_finalize: NULL pointer");
  if (ns < 0 || n_win < 1) return wk_fail(WK_E_RANGE, "wk_wake_finalize: ns %d nwin %d", ns, n_win);
  if (ns == 0) return WK_OK;
  cudaStream_t st = (cudaStream_t)stream;
  k_wake_finalize<<<(ns + 127) / 128, 128, 0, st>>>(acc, n_win, ns, carry, qnorm, WP3d);
  return wk_check_launch("wk_wake_finalize");
}

// Segments of the scan: at most max_seg of them, each at least 1024 samples.
static int trans_seg_len(int ns, int max_seg) {
  long long seg = (ns + (long long)max_seg - 1) / max_seg;
  if (seg < 1024) seg = 1024;
  return (int)seg;
}

static int trans_scan_launch(const double* WP3d, int ns, double ds, double dxsum, double dysum,
                             double* WPx, double* WPy, DD* part, int max_seg, cudaStream_t st,
                             const char* where) {
  const int seg = trans_seg_len(ns, max_seg);
  const int nseg = (int)(((long long)ns + seg - 1) / seg);
  k_trans_part<<<nseg, kScanThreads, 0, st>>>(WP3d, ns, seg, part);
  k_trans_part_scan<<<1, 32, 0, st>>>(part, nseg);
  k_trans_final<<<nseg, 32, 0, st>>>(WP3d, ns, seg, part, ds, dxsum, dysum, WPx, WPy);
  return wk_check_launch(where);
}

extern "C" long long wk_trans_wake_scan_scratch_bytes(int ns) {
  if (ns <= 0) return 0;
  const int seg = trans_seg_len(ns, 1 << 20);
  const long long nseg = ((long long)ns + seg - 1) / seg;
  return nseg * 4 * (long long)sizeof(DD);
}

extern "C" int wk_trans_wake_scan(const double* WP3d, int ns, double ds, double dxsum,
                                  double dysum, double* WPx, double* WPy, void* scratch,
                                  long long scratch_bytes, void* stream) {
  if (!WP3d || !WPx || !WPy) return wk_fail(WK_E_NULL, "wk_trans_wake_scan: NULL pointer");
  if (ns < 0) return wk_fail(WK_E_RANGE, "wk_trans_wake_scan: ns %d", ns);
  if (ns == 0) return WK_OK;
  if (!scratch) return wk_fail(WK_E_NULL, "wk_trans_wake_scan: scratch is NULL");
  if (((uintptr_t)scratch % 16) != 0)
    return wk_fail(WK_E_ALIGN, "wk_trans_wake_scan: scratch not 16-byte aligned");
  const long long need = wk_trans_wake_scan_scratch_bytes(ns);
  if (scratch_bytes < need)
    return wk_fail(WK_E_RANGE, "wk_trans_wake_scan: scratch of %lld bytes, %lld needed",
                   scratch_bytes, need);
  return trans_scan_launch(WP3d, ns, ds, dxsum, dysum, WPx, WPy, (DD*)scratch, 1 << 20,
                           (cudaStream_t)stream, "wk_trans_wake_scan");
}

// ------------------------------------------------- without allocation ----
// wk_trans_wake_scan_noalloc keeps its segment sums in this file-scope
// device array instead of caller memory.  Every GPU that loads the library
// holds it (kNoAllocSegments x 4 double-double sums = 256 KiB) until the
// process exits; all calls share it.
constexpr int kNoAllocSegments = 4096;
constexpr long long kNoAllocMaxSamples = (long long)kNoAllocSegments * 65536;
static __device__ __align__(256) DD g_trans_scratch[kNoAllocSegments * 4];

// Device address of g_trans_scratch, looked up once per device (in host
// code the symbol names a host-side stand-in, not device memory).
static constexpr int kMaxDevices = 64;
static DD* g_trans_scratch_dev[kMaxDevices];
static cudaError_t g_trans_scratch_err[kMaxDevices];
static std::once_flag g_trans_scratch_once[kMaxDevices];

extern "C" int wk_trans_wake_scan_noalloc(const double* WP3d, int ns, double ds, double dxsum,
                                          double dysum, double* WPx, double* WPy,
                                          void* stream) {
  if (!WP3d || !WPx || !WPy)
    return wk_fail(WK_E_NULL, "wk_trans_wake_scan_noalloc: NULL pointer");
  if (ns < 0) return wk_fail(WK_E_RANGE, "wk_trans_wake_scan_noalloc: ns %d", ns);
  if ((long long)ns > kNoAllocMaxSamples)
    return wk_fail(WK_E_RANGE,
                   "wk_trans_wake_scan_noalloc: %d samples is above this entry point's "
                   "maximum of %lld (its built-in scratch holds %d segment sums of at most "
                   "65536 samples each); use wk_trans_wake_scan with caller scratch",
                   ns, kNoAllocMaxSamples, kNoAllocSegments);
  if (ns == 0) return WK_OK;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess)
    return wk_fail(-(int)e, "wk_trans_wake_scan_noalloc: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices)
    return wk_fail(WK_E_RANGE, "wk_trans_wake_scan_noalloc: device %d", dev);
  std::call_once(g_trans_scratch_once[dev], [dev] {
    void* ptr = nullptr;
    g_trans_scratch_err[dev] = cudaGetSymbolAddress(&ptr, g_trans_scratch);
    g_trans_scratch_dev[dev] = static_cast<DD*>(ptr);
  });
  if (g_trans_scratch_err[dev] != cudaSuccess || !g_trans_scratch_dev[dev])
    return wk_fail(-(int)(g_trans_scratch_err[dev] != cudaSuccess ? g_trans_scratch_err[dev]
                                                                  : cudaErrorInvalidSymbol),
                   "wk_trans_wake_scan_noalloc: device address of the scratch array: %s",
                   cudaGetErrorString(g_trans_scratch_err[dev]));
  return trans_scan_launch(WP3d, ns, ds, dxsum, dysum, WPx, WPy, g_trans_scratch_dev[dev],
                           kNoAllocSegments, (cudaStream_t)stream,
                           "wk_trans_wake_scan_noalloc");
}
