// Rows of the FIT update with the column factors given one by one (sm_100a),
// for kernels that take every cell of the grid, boundary cells included,
// through the same code: a cell's rows differ from the interior ones only in
// the factors of their columns.  A column factor is the primal (dual) length
// of the column's component at the column's cell, 0 where the PEC (PMC) mask
// removes that column; the column's cell is the flat-offset neighbour (a step
// past a row's end lands on the next row, past a plane's end on the next
// plane).  Same products and same order as h_row_acc / e_curl_acc without the
// leading "+0" of the sum (it can only change the sign of a zero).
#pragma once
#include "fit_common.cuh"

namespace wk {

// Column factors of one cell: component (x, y, z) at the cell itself (O) and
// at its x, y or z neighbour.
template <typename T>
struct RowCols {
  T xO, xZ, xY, yO, yZ, yX, zO, zX, zY;
};

// Plane-invariant part of the column factors of column (i, j), neighbours in
// direction DIR (+1: H rows, primal lengths and PEC mask; -1: E rows, dual
// lengths and PMC mask).
template <typename T, int DIR>
struct ColumnInv {
  T Lx, Ly, LyX;        // lengths at the cell, y length at the x neighbour
  int bits;             // mask values away from the z faces, one bit per factor
  int dkx, dky;         // plane steps of the x and y neighbours (0 or 1)
  enum { XO = 1, XY = 2, YO = 4, YX = 8, ZO = 16, ZX = 32, ZY = 64 };

  __device__ __forceinline__ void init(const FitParams<T>& p, int i, int j) {
    const int Nx = p.Nx, Ny = p.Ny;
    const T* lx = DIR > 0 ? p.Lx : p.tLx;
    const T* ly = DIR > 0 ? p.Ly : p.tLy;
    const bool has = DIR > 0 ? p.has_pec != 0 : p.has_pmc != 0;
    const int* f = DIR > 0 ? p.pec_face : p.pmc_face;
    const bool wx = DIR > 0 ? i == Nx - 1 : i == 0;
    const bool wy = DIR > 0 ? j == Ny - 1 : j == 0;
    const int in = wx ? (DIR > 0 ? 0 : Nx - 1) : i + DIR;
    const int jn = wy ? (DIR > 0 ? 0 : Ny - 1) : j + DIR;
    const int jx = wx ? jn : j;
    dkx = (wx && wy) ? 1 : 0;
    dky = wy ? 1 : 0;
    Lx = __ldg(lx + i);
    Ly = __ldg(ly + j);
    LyX = __ldg(ly + jx);
    if (!has) {
      bits = 127;
      return;
    }
    auto xface = [&](int a) { return a == Nx - 1 ? f[1] != 0 : (a == 0 ? f[0] != 0 : true); };
    auto yface = [&](int b) { return b == Ny - 1 ? f[3] != 0 : (b == 0 ? f[2] != 0 : true); };
    auto zcomp = [&](int a, int b) { return (b == 0 || b == Ny - 1) ? yface(b) : xface(a); };
    bits = (yface(j) ? XO : 0) | (yface(jn) ? XY : 0) | (xface(i) ? YO : 0) |
           (xface(in) ? YX : 0) | (zcomp(i, j) ? ZO : 0) | (zcomp(in, jx) ? ZX : 0) |
           (zcomp(i, jn) ? ZY : 0);
  }

  // Factors of plane k; lz: the z lengths.  The z faces replace the mask of
  // the x and y components on their planes.
  __device__ __forceinline__ RowCols<T> at(const FitParams<T>& p, int k) const {
    const int Nz = p.Nz;
    const T* lz = DIR > 0 ? p.Lz : p.tLz;
    const bool has = DIR > 0 ? p.has_pec != 0 : p.has_pmc != 0;
    const int* f = DIR > 0 ? p.pec_face : p.pmc_face;
    const int lo = f[4], hi = f[5];
    auto ov = [&](int kk, int bit) {
      const bool base = (bits & bit) != 0;
      if (!has) return true;
      return kk == Nz - 1 ? hi != 0 : (kk == 0 ? lo != 0 : base);
    };
    const int kx = k + DIR * dkx, ky = k + DIR * dky, kz = k + DIR;
    const T z = T(0);
    RowCols<T> c;
    c.xO = ov(k, XO) ? Lx : z;
    c.xZ = ov(kz, XO) ? Lx : z;
    c.xY = ov(ky, XY) ? Lx : z;
    c.yO = ov(k, YO) ? Ly : z;
    c.yZ = ov(kz, YO) ? Ly : z;
    c.yX = ov(kx, YX) ? LyX : z;
    const T l0 = __ldg(lz + k);
    c.zO = (bits & ZO) ? l0 : z;
    // a neighbour outside the grid contributes no term (its value reads as 0)
    c.zX = (bits & ZX) ? (dkx ? __ldg(lz + min(max(kx, 0), Nz - 1)) : l0) : z;
    c.zY = (bits & ZY) ? (dky ? __ldg(lz + min(max(ky, 0), Nz - 1)) : l0) : z;
    return c;
  }
};

// New H of one cell.  E values: *0 at n, y1/z1 at n+1, x2/z2 at n+Nx, x3/y3 at
// n+Nx*Ny; R* = iA*imu of the rows (0 where the PMC mask removes the row).
template <typename T>
__device__ __forceinline__ void h_rows(T dt, bool desc, T R0, T R1, T R2, const RowCols<T>& c,
                                       T ex0, T ey0, T ez0, T ey1, T ez1, T ex2, T ez2, T ex3,
                                       T ey3, T& hx, T& hy, T& hz) {
  auto term = [&](T R, T L, T v) { return mul(mul(dt, mul(R, L)), v); };
  {
    const T t0 = term(R0, c.yO, ey0), t1 = term(R0, c.yZ, ey3), t2 = term(R0, c.zO, ez0),
            t3 = term(R0, c.zY, ez2);
    hx = sub(hx, desc ? add(sub(sub(t3, t2), t1), t0) : add(sub(sub(t0, t1), t2), t3));
  }
  {
    const T t0 = term(R1, c.xO, ex0), t1 = term(R1, c.xZ, ex3), t2 = term(R1, c.zO, ez0),
            t3 = term(R1, c.zX, ez1);
    hy = sub(hy, desc ? sub(add(sub(t2, t3), t1), t0) : sub(add(sub(t1, t0), t2), t3));
  }
  {
    const T t0 = term(R2, c.xO, ex0), t1 = term(R2, c.xY, ex2), t2 = term(R2, c.yO, ey0),
            t3 = term(R2, c.yX, ey1);
    hz = sub(hz, desc ? add(sub(sub(t3, t2), t1), t0) : add(sub(sub(t0, t1), t2), t3));
  }
}

// Curl parts of the E rows of one cell.  H values: *0 at n, y1/z1 at n-1,
// x2/z2 at n-Nx, x3/y3 at n-Nx*Ny; R* = ieps*itA of the rows (0 where the PEC
// mask removes the row).
template <typename T>
__device__ __forceinline__ void e_rows(T R0, T R1, T R2, const RowCols<T>& c, T hx0, T hy0, T hz0,
                                       T hy1, T hz1, T hx2, T hz2, T hx3, T hy3, T& cx, T& cy,
                                       T& cz) {
  auto term = [&](T R, T L, T v) { return mul(mul(R, L), v); };
  cx = add(sub(sub(term(R0, c.yZ, hy3), term(R0, c.yO, hy0)), term(R0, c.zY, hz2)),
           term(R0, c.zO, hz0));
  cy = sub(add(sub(term(R1, c.xO, hx0), term(R1, c.xZ, hx3)), term(R1, c.zX, hz1)),
           term(R1, c.zO, hz0));
  cz = add(sub(sub(term(R2, c.xY, hx2), term(R2, c.xO, hx0)), term(R2, c.yX, hy1)),
           term(R2, c.yO, hy0));
}

}  // namespace wk
