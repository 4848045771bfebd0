// Many steps per launch for grids that fit the shared memory of all SMs
// (sm_100a).
//
// On a small grid a step is far shorter than the launches that make it up
// (one to four, each with its own start, fill and drain), and its state goes
// through L2 twice.  Here one cooperative launch of one block per SM runs all
// steps of a call: block b keeps E and H of its tile (a box of cells) in
// shared memory from the first step to the last, with a halo of E around the
// tile and of H on its low sides.  Per step a block
//   1. updates H on the tile and on the low halo (recomputed, as its owner
//      does it, so that H never travels),
//   2. updates E on the tile and writes the E of the tile's outer cells to the
//      ping-pong buffer in global memory,
//   3. arrives at a grid-wide barrier, updates the H of the next step where
//      it reads only the tile's own E, waits for the barrier and reads the E
//      of its halo from the neighbours' cells.
// So a step costs one barrier, and the barrier's latency is covered by the
// interior cells.  The last step writes the whole tile.
//
// Cells are addressed by flat index (n + a + b Nx + c Nx Ny for box position
// (a, b, c)): a halo position past a row's or plane's end is the cell that
// the flat-offset difference operators reach there, so every face (PEC, PMC,
// PML, ABC, periodic) and any row length is covered, with the rows of
// fit_rows.cuh.  Each block lists its cells once per launch, ordered by
// class: regular (the factors of the cell's own lengths), masked (some
// factors are 0) and wrapped (a neighbour's length differs: formed from the
// tables by the general code), so that warps rarely mix classes.
//
// Bound by shared-memory bandwidth in the phases (26 reads of a word per cell
// in E) and, on the smallest grids, by the barrier (about 2 us of fence,
// arrival and the halo's L2 loads).  Measured on B200, us per step, launches
// per step before / here: 16x16x24 FP64 10.3 / 2.9, 40x40x80 FP64 with open
// ends 25 / 6.9, 50x50x150 FP32 41 / 9.0, 55x61x110 FP64 48 / 14, 64x64x160
// FP32 31 / 15; the set-up of a launch takes 11 to 70 us (16x16x24 to
// 64x64x160).  512 threads: 384 and 768 were 5 to 10 % slower over these.
//
// The barrier counts arrivals in a caller-owned word (wk_fit_desc.sync):
// monotonic within a launch, set back to 0 by the last block to leave.  Every
// wait is bounded; on timeout a block sets the status word and the abort word
// and leaves, and the others leave at their next wait.
#include <stdint.h>

#include "../../include/wakis_b200.h"
#include "abi_internal.h"
#include "fit_common.cuh"
#include "fit_kernels.cuh"
#include "fit_loop.cuh"

namespace wk {

// Shared-memory layout of the largest tile, in bytes.
template <typename T>
struct LoopLayout {
  int e, h, tab, mat, lists, ids, bytes;
  int n_ext, n_own, n_shell;
  __host__ __device__ LoopLayout(int tx, int ty, int tz, int n_mat, int id_bytes) {
    const int es = (tx + 2) * (ty + 2) * (tz + 2), hs = (tx + 1) * (ty + 1) * (tz + 1);
    n_own = tx * ty * tz;
    n_ext = n_own + ty * tz + tx * tz + tx * ty;
    // halo cells with at most one low and one high coordinate
    n_shell = 2 * (ty * tz + tx * tz + tx * ty) + 2 * (tx + ty + tz);
    auto r16 = [](int b) { return (b + 15) / 16 * 16; };
    e = 0;
    h = e + r16(3 * es * (int)sizeof(T));
    tab = h + r16(3 * hs * (int)sizeof(T));
    // iA and itA faces (box coordinates 0 .. t), then six 1-D lengths
    const int faces = (ty + 1) * (tz + 1) + (tx + 1) * (tz + 1) + (tx + 1) * (ty + 1);
    mat = tab + r16((2 * faces + 2 * (tx + ty + tz + 3)) * (int)sizeof(T));
    lists = mat + r16(n_mat <= kLoopMat ? 9 * n_mat * (int)sizeof(T) : 0);
    ids = lists + r16((n_ext + n_own + n_shell) * 4);
    bytes = ids + r16((n_ext + n_own) * (id_bytes == 1 ? 1 : 2)) + 256;
  }
};

template <typename T, typename IdT, bool SMT>
__global__ void __launch_bounds__(kLoopThreads, 1)
k_loop(FitParams<T> p, LoopTiling tl, int n_steps, long long step0, unsigned* sync) {
  constexpr int TH = kLoopThreads;
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int s_len[4], s_count[10];
  const LoopLayout<T> lay(tl.tx, tl.ty, tl.tz, p.n_mat, (int)sizeof(IdT));
  const int tid = threadIdx.x;
  const int Nx = p.Nx, Ny = p.Ny, Nz = p.Nz, plane = (int)p.NxNy;
  const long long N = p.N;
  step0 = step_index(p, step0);
  int t = blockIdx.x;
  const int bx = t % tl.nbx;
  t /= tl.nbx;
  const int by = t % tl.nby, bz = t / tl.nby;
  auto part = [](int q, int n, int nb) { return (int)((long long)q * n / nb); };
  const int i0 = part(bx, Nx, tl.nbx), i1 = part(bx + 1, Nx, tl.nbx);
  const int j0 = part(by, Ny, tl.nby), j1 = part(by + 1, Ny, tl.nby);
  const int k0 = part(bz, Nz, tl.nbz), k1 = part(bz + 1, Nz, tl.nbz);
  const int tx = i1 - i0, ty = j1 - j0, tz = k1 - k0;
  const int EX = tx + 2, EP = EX * (ty + 2), EV = EP * (tz + 2);   // E box: row, plane, volume
  const int HX = tx + 1, HP = HX * (ty + 1), HV = HP * (tz + 1);   // H box
  T* Es = reinterpret_cast<T*>(sm + lay.e);
  T* Hs = reinterpret_cast<T*>(sm + lay.h);
  T* sAx = reinterpret_cast<T*>(sm + lay.tab);     // iAx at (b, c), rows of ty + 1
  T* sAy = sAx + (ty + 1) * (tz + 1);              // iAy at (a, c)
  T* sAz = sAy + HX * (tz + 1);                    // iAz at (a, b)
  T* tAx = sAz + HP;
  T* tAy = tAx + (ty + 1) * (tz + 1);
  T* tAz = tAy + HX * (tz + 1);
  T* sL = tAz + HP;                                // Lx Ly Lz tLx tLy tLz
  T *sLx = sL, *sLy = sLx + HX, *sLz = sLy + ty + 1, *stLx = sLz + tz + 1, *stLy = stLx + HX,
    *stLz = stLy + ty + 1;
  T* smat = reinterpret_cast<T*>(sm + lay.mat);
  uint32_t* lh = reinterpret_cast<uint32_t*>(sm + lay.lists);   // H cells: tile and low halo
  uint32_t* le = lh + lay.n_ext;                                // E cells: tile
  uint32_t* ls = le + lay.n_own;                                // E halo
  IdT* idh = reinterpret_cast<IdT*>(sm + lay.ids);
  IdT* ide = idh + lay.n_ext;
  // flat index of box position (0, 0, 0)
  const int nb = (i0 - 1) + (j0 - 1) * Nx + (k0 - 1) * plane;
  auto flat = [&](int a, int b, int c) { return nb + a + b * Nx + c * plane; };
  const T* mat = SMT ? smat : p.mat;

  // ---- set-up: state and tables by cp.async while the lists are formed
  const LoopDiv dEP(EP), dEX(EX), dHP(HP), dHX(HX), dY1(ty + 1), dTP(tx * ty), dTX(tx);
  for (int q = tid; q < EV; q += TH) {
    const int c = dEP.div(q), r = q - c * EP, b = dEX.div(r), a = r - b * EX;
    const int n = flat(a, b, c);
    const bool v = n >= 0 && n < N;
#pragma unroll
    for (int d = 0; d < 3; d++)
      cp_async<sizeof(T)>(Es + d * EV + q, p.E_in + (v ? d * N + n : 0), v);
  }
  for (int q = tid; q < HV; q += TH) {
    const int c = dHP.div(q), r = q - c * HP, b = dHX.div(r), a = r - b * HX;
    const int n = flat(a, b, c);
    const bool v = n >= 0 && n < N;
#pragma unroll
    for (int d = 0; d < 3; d++)
      cp_async<sizeof(T)>(Hs + d * HV + q, p.H_in + (v ? d * N + n : 0), v);
  }
  // tables at box coordinates; positions outside the grid are read by no
  // regular or masked cell
  auto put = [&](T* dst, const T* src) { cp_async<sizeof(T)>(dst, src, true); };
  for (int q = tid; q < (ty + 1) * (tz + 1); q += TH) {
    const int c = dY1.div(q), j = max(j0 - 1 + q - c * (ty + 1), 0), k = max(k0 - 1 + c, 0);
    put(sAx + q, p.iAx + j + (long long)k * Ny);
    put(tAx + q, p.itAx + j + (long long)k * Ny);
  }
  for (int q = tid; q < HX * (tz + 1); q += TH) {
    const int c = dHX.div(q), i = max(i0 - 1 + q - c * HX, 0), k = max(k0 - 1 + c, 0);
    put(sAy + q, p.iAy + i + (long long)k * Nx);
    put(tAy + q, p.itAy + i + (long long)k * Nx);
  }
  for (int q = tid; q < HP; q += TH) {
    const int c = dHX.div(q), i = max(i0 - 1 + q - c * HX, 0), j = max(j0 - 1 + c, 0);
    put(sAz + q, p.iAz + i + (long long)j * Nx);
    put(tAz + q, p.itAz + i + (long long)j * Nx);
  }
  if (tid < HX) { const int i = max(i0 - 1 + tid, 0); put(sLx + tid, p.Lx + i); put(stLx + tid, p.tLx + i); }
  if (tid < ty + 1) { const int j = max(j0 - 1 + tid, 0); put(sLy + tid, p.Ly + j); put(stLy + tid, p.tLy + j); }
  if (tid < tz + 1) { const int k = max(k0 - 1 + tid, 0); put(sLz + tid, p.Lz + k); put(stLz + tid, p.tLz + k); }
  cp_async_commit();
  if (SMT)
    for (int q = tid; q < 9 * p.n_mat; q += TH) smat[q] = p.mat[q];
  __syncthreads();
  // The three lists (loop_lists): H cells first those whose E is all the tile's
  // own (a < tx, b < ty, c < tz, no halo), each part ordered by class (keys 0
  // to 5), E cells by class (6 to 8), the halo's E (9).
  auto h_entry = [&](int q, uint32_t& e) -> int {
    const int c = dHP.div(q), r = q - c * HP, b = dHX.div(r), a = r - b * HX;
    const int n = flat(a, b, c);
    const int low = (a == 0) + (b == 0) + (c == 0);
    if (low > 1 || n < 0) return -1;
    const int outer = (low == 0 && a < tx && b < ty && c < tz) ? 0 : 3;
    if (lean_h<T>(i0 - 1 + a, j0 - 1 + b, k0 - 1 + c, Nx, Ny, Nz)) {
      e = loop_entry(a, b, c, 511, 7, kRegular);
      return outer;
    }
    const Cell cc = cell_of(n, Nx, Ny);
    if (low && p.has_pec) {
      // a halo cell whose H enters only masked E rows is left alone
      const Cell u = cell_of(n + (a == 0 ? 1 : (b == 0 ? Nx : plane)), Nx, Ny);
      const int normal = a == 0 ? 0 : (b == 0 ? 1 : 2);
      bool used = false;
      for (int d = 0; d < 3; d++)
        if (d != normal && face_val(p.pec_face, d, u.i, u.j, u.k, Nx, Ny, Nz)) used = true;
      if (!used) return -1;
    }
    int rows = 0;
    for (int d = 0; d < 3; d++)
      if (!p.has_pmc || face_val(p.pmc_face, d, cc.i, cc.j, cc.k, Nx, Ny, Nz)) rows |= 1 << d;
    bool wrap;
    const int m = loop_bits<T, 1>(p, cc, rows, wrap);
    wrap |= (a == 0 && i0 == 0) || (b == 0 && j0 == 0);
    const uint32_t cls = wrap ? kWrapped : (m == 511 && rows == 7 ? kRegular : kMasked);
    e = loop_entry(a, b, c, m, rows, cls);
    return outer + (int)cls;
  };
  auto e_entry = [&](int q, uint32_t& e) -> int {
    const int c = dTP.div(q), r = q - c * tx * ty, b = dTX.div(r), a = r - b * tx;
    const Cell cc = {i0 + a, j0 + b, k0 + c};
    if (lean_e<T>(cc.i, cc.j, cc.k, Nx, Ny, Nz)) {
      e = loop_entry(a + 1, b + 1, c + 1, 511, 7, kRegular);
      return 6;
    }
    int rows = 0;
    for (int d = 0; d < 3; d++)
      if (!p.has_pec || face_val(p.pec_face, d, cc.i, cc.j, cc.k, Nx, Ny, Nz)) rows |= 1 << d;
    bool wrap;
    const int m = loop_bits<T, -1>(p, cc, rows, wrap);
    const uint32_t cls = wrap ? kWrapped : (m == 511 && rows == 7 ? kRegular : kMasked);
    e = loop_entry(a + 1, b + 1, c + 1, m, rows, cls);
    return 6 + (int)cls;
  };
  auto s_entry = [&](int q, uint32_t& e) -> int {
    const int c = dEP.div(q), r = q - c * EP, b = dEX.div(r), a = r - b * EX;
    const int low = (a == 0) + (b == 0) + (c == 0);
    const int high = (a == tx + 1) + (b == ty + 1) + (c == tz + 1);
    const int n = flat(a, b, c);
    e = loop_entry(a, b, c, 0, 0, 0);
    return low + high > 0 && low <= 1 && high <= 1 && n >= 0 && n < N ? 9 : -1;
  };
  const int own = tx * ty * tz;
  loop_lists(s_count, s_len, HV, h_entry, lh, own, e_entry, le, EV, s_entry, ls);
  const int nh = s_len[0], ne = s_len[1], nsh = s_len[2], nh_own = s_len[3];
  auto id_of = [&](uint32_t e) -> IdT {
    return (IdT)load_id(p.mat_id, p.id_bytes, flat(e & 63, e >> 6 & 63, e >> 12 & 63));
  };
  auto fill_ids = [&](const uint32_t* list, IdT* out, int n) {
    for (int q0 = tid; q0 < n; q0 += 4 * TH) {
      IdT v[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (q0 + u * TH < n) v[u] = id_of(list[q0 + u * TH]);
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (q0 + u * TH < n) out[q0 + u * TH] = v[u];
    }
  };
  fill_ids(lh, idh, nh);
  fill_ids(le, ide, ne);
  cp_async_wait<0>();
  __syncthreads();

  // cell of a box position (one before the grid: the last column of the row
  // below, the last row of the plane below)
  auto true_cell = [&](int a, int b, int c) {
    Cell cc = {i0 - 1 + a, j0 - 1 + b, k0 - 1 + c};
    if (cc.i < 0) { cc.i = Nx - 1; cc.j--; }
    if (cc.j < 0) { cc.j += Ny; cc.k--; }
    return cc;
  };
  const bool desc = p.h_desc != 0;
  const T dt = p.dt;
  auto pick = [](uint32_t bits, int b, T v) { return (bits & b) ? v : T(0); };

  struct HCell {
    T h[3], ex0, ey0, ez0, ey1, ez1, ex2, ez2, ex3, ey3, R[3], L[3];
    int at;
  };
  auto h_read = [&](int q, uint32_t e, HCell& v) {
    const int a = e & 63, b = e >> 6 & 63, c = e >> 12 & 63;
    const T* E = Es + (c * EP + b * EX + a);
    v.at = c * HP + b * HX + a;
    const T* H = Hs + v.at;
    const T* m0 = mat + 9 * (int)idh[q];
    v.h[0] = H[0]; v.h[1] = H[HV]; v.h[2] = H[2 * HV];
    v.ex0 = E[0]; v.ey0 = E[EV]; v.ez0 = E[2 * EV];
    v.ey1 = E[EV + 1]; v.ez1 = E[2 * EV + 1];
    v.ex2 = E[EX]; v.ez2 = E[2 * EV + EX];
    v.ex3 = E[EP]; v.ey3 = E[EV + EP];
    v.R[0] = mul(sAx[c * (ty + 1) + b], m0[3]);
    v.R[1] = mul(sAy[c * HX + a], m0[4]);
    v.R[2] = mul(sAz[b * HX + a], m0[5]);
    v.L[0] = sLx[a]; v.L[1] = sLy[b]; v.L[2] = sLz[c];
  };
  auto h_update = [&](int q, uint32_t e, HCell& v) {
    const uint32_t cls = e >> 30;
    if (cls == kRegular) {
      h_lean(dt, desc, v.R[0], v.R[1], v.R[2], v.L[0], v.L[1], v.L[2], v.ex0, v.ey0, v.ez0, v.ey1,
             v.ez1, v.ex2, v.ez2, v.ex3, v.ey3, v.h[0], v.h[1], v.h[2]);
    } else {
      RowCols<T> f;
      if (cls == kMasked) {
        const uint32_t w = e >> 18;
        f = {pick(w, bXO, v.L[0]), pick(w, bXZ, v.L[0]), pick(w, bXY, v.L[0]),
             pick(w, bYO, v.L[1]), pick(w, bYZ, v.L[1]), pick(w, bYX, v.L[1]),
             pick(w, bZO, v.L[2]), pick(w, bZX, v.L[2]), pick(w, bZY, v.L[2])};
      } else {
        const Cell cc = true_cell(e & 63, e >> 6 & 63, e >> 12 & 63);
        const T* m0 = mat + 9 * (int)idh[q];
        v.R[0] = mul(__ldg(p.iAx + cc.j + (long long)cc.k * Ny), m0[3]);
        v.R[1] = mul(__ldg(p.iAy + cc.i + (long long)cc.k * Nx), m0[4]);
        v.R[2] = mul(__ldg(p.iAz + cc.i + (long long)cc.j * Nx), m0[5]);
        ColumnInv<T, 1> ci;
        ci.init(p, cc.i, cc.j);
        f = ci.at(p, cc.k);
      }
      const uint32_t rows = e >> 27;
      h_rows(dt, desc, pick(rows, 1, v.R[0]), pick(rows, 2, v.R[1]), pick(rows, 4, v.R[2]), f,
             v.ex0, v.ey0, v.ez0, v.ey1, v.ez1, v.ex2, v.ez2, v.ex3, v.ey3, v.h[0], v.h[1], v.h[2]);
    }
  };
  // H of the list's cells [q_lo, q_hi); a cell writes only its own H
  auto h_cells = [&](int q_lo, int q_hi) {
    for (int q = q_lo + tid; q < q_hi; q += TH) {
      HCell v;
      const uint32_t e = lh[q];
      h_read(q, e, v);
      h_update(q, e, v);
      Hs[v.at] = v.h[0];
      Hs[HV + v.at] = v.h[1];
      Hs[2 * HV + v.at] = v.h[2];
    }
  };

  // E of the tile's cells
  struct ECell {
    T e[3], hx0, hy0, hz0, hy1, hz1, hx2, hz2, hx3, hy3, R[3], L[3], ieps[3], sig[3];
    int at;
  };
  const bool jsig = p.j_mode == WK_J_SIGMA_E;
  // the source line, the capture window: in this tile?
  const bool src = (p.line_on || p.beam_on) && p.ixs >= i0 && p.ixs < i1 && p.iys >= j0 && p.iys < j1;
  const bool cap = p.cap_on && p.cap_i0 < i1 && p.cap_i0 + p.cap_ni > i0 && p.cap_j0 < j1 &&
                   p.cap_j0 + p.cap_nj > j0;
  auto e_read = [&](int q, uint32_t e, ECell& v) {
    const int a = e & 63, b = e >> 6 & 63, c = e >> 12 & 63;
    v.at = c * EP + b * EX + a;
    const T* E = Es + v.at;
    const T* H = Hs + (c * HP + b * HX + a);
    const T* m0 = mat + 9 * (int)ide[q];
    v.hx0 = H[0]; v.hy0 = H[HV]; v.hz0 = H[2 * HV];
    v.hy1 = H[HV - 1]; v.hz1 = H[2 * HV - 1];
    v.hx2 = H[-HX]; v.hz2 = H[2 * HV - HX];
    v.hx3 = H[-HP]; v.hy3 = H[HV - HP];
    v.e[0] = E[0]; v.e[1] = E[EV]; v.e[2] = E[2 * EV];
#pragma unroll
    for (int d = 0; d < 3; d++) {
      v.ieps[d] = m0[d];
      v.sig[d] = jsig ? m0[6 + d] : T(0);
    }
    v.R[0] = mul(v.ieps[0], tAx[c * (ty + 1) + b]);
    v.R[1] = mul(v.ieps[1], tAy[c * HX + a]);
    v.R[2] = mul(v.ieps[2], tAz[b * HX + a]);
    v.L[0] = stLx[a]; v.L[1] = stLy[b]; v.L[2] = stLz[c];
  };
  auto e_update = [&](uint32_t e, ECell& v, long long step) {
    const uint32_t cls = e >> 30;
    const int a = e & 63, b = e >> 6 & 63, c = e >> 12 & 63;
    const Cell cc = {i0 - 1 + a, j0 - 1 + b, k0 - 1 + c};
    T cu[3];
    if (cls == kRegular) {
      e_lean(v.R[0], v.R[1], v.R[2], v.L[0], v.L[1], v.L[2], v.hx0, v.hy0, v.hz0, v.hy1, v.hz1,
             v.hx2, v.hz2, v.hx3, v.hy3, cu[0], cu[1], cu[2]);
    } else {
      RowCols<T> f;
      if (cls == kMasked) {
        const uint32_t w = e >> 18;
        f = {pick(w, bXO, v.L[0]), pick(w, bXZ, v.L[0]), pick(w, bXY, v.L[0]),
             pick(w, bYO, v.L[1]), pick(w, bYZ, v.L[1]), pick(w, bYX, v.L[1]),
             pick(w, bZO, v.L[2]), pick(w, bZX, v.L[2]), pick(w, bZY, v.L[2])};
      } else {
        ColumnInv<T, -1> ci;
        ci.init(p, cc.i, cc.j);
        f = ci.at(p, cc.k);
      }
      const uint32_t rows = e >> 27;
      e_rows(pick(rows, 1, v.R[0]), pick(rows, 2, v.R[1]), pick(rows, 4, v.R[2]), f, v.hx0, v.hy0,
             v.hz0, v.hy1, v.hz1, v.hx2, v.hz2, v.hx3, v.hy3, cu[0], cu[1], cu[2]);
    }
    if (cap) capture(p, cc, 0, step, v.e[2]);
#pragma unroll
    for (int d = 0; d < 3; d++) {
      T jv = jsig ? mul(v.sig[d], v.e[d]) : T(0);
      if (d == 2 && src && cc.i == p.ixs && cc.j == p.iys)
        jv = j_in(p, d, cc, 0, step, v.e[d], v.sig[d]);
      v.e[d] = add(v.e[d], mul(dt, sub(cu[d], mul(v.ieps[d], jv))));
    }
  };
  auto e_store = [&](uint32_t e, const ECell& v, T* Eo, T* Hfinal) {
    const int a = e & 63, b = e >> 6 & 63, c = e >> 12 & 63;
    Es[v.at] = v.e[0];
    Es[EV + v.at] = v.e[1];
    Es[2 * EV + v.at] = v.e[2];
    const int n = flat(a, b, c);
    if (Hfinal || a == 1 || a == tx || b == 1 || b == ty || c == 1 || c == tz) {
      Eo[n] = v.e[0];
      Eo[N + n] = v.e[1];
      Eo[2 * N + n] = v.e[2];
    }
    if (Hfinal) {
      Hfinal[n] = v.hx0;
      Hfinal[N + n] = v.hy0;
      Hfinal[2 * N + n] = v.hz0;
    }
  };
  auto e_cells = [&](long long step, T* Eo, T* Hfinal) {
    for (int q = tid; q < ne; q += TH) {
      ECell v;
      const uint32_t e = le[q];
      e_read(q, e, v);
      e_update(e, v, step);
      e_store(e, v, Eo, Hfinal);
    }
  };

  const long long lim = p.wait_ns == 0 ? 20 * kWaitNs : p.wait_ns;
  T *Eo = p.E_out, *Ex = p.E_in;      // buffers of the next and the current step
  unsigned target = 0;
  bool ok = true;
  h_cells(0, nh_own);
  for (int s = 0; s < n_steps; s++) {
    // H of the cells that read the halo
    h_cells(nh_own, nh);
    __syncthreads();
    const bool last = s + 1 == n_steps;
    e_cells(step0 + s, Eo, last ? ((n_steps & 1) ? p.H_out : p.H_in) : nullptr);
    if (last) break;
    __syncthreads();
    if (tid == 0) red_release(sync + kSyncCount);
    target += gridDim.x;
    // H of the next step where it reads the tile's own E only
    h_cells(0, nh_own);
    if (tid == 0) {
      ok = loop_wait(sync, target, lim);
      if (!ok) {
        if (p.status) atomicExch(p.status, 1);
        atomicExch(sync + kSyncAbort, 1u);
      }
    }
    ok = __syncthreads_and(ok);
    if (!ok) break;
    for (int q = tid; q < nsh; q += TH) {
      const uint32_t e = ls[q];
      const int a = e & 63, b = e >> 6 & 63, c = e >> 12 & 63;
      const long long n = flat(a, b, c);
      T* E = Es + (c * EP + b * EX + a);
#pragma unroll
      for (int d = 0; d < 3; d++) E[d * EV] = Eo[d * N + n];
    }
    T* sw = Ex;
    Ex = Eo;
    Eo = sw;
    __syncthreads();
  }
  loop_leave(sync);
}

int loop_sms() {
  static int sms[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (sms[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    sms[dev] = n;
  }
  return sms[dev];
}

namespace {

// The tile split of a grid.  The search takes tens of microseconds, as long as
// several steps, so each thread keeps the answer of its last shape.
template <typename T>
LoopTiling loop_tiling(const FitParams<T>& p, int sms) {
  struct Last { int Nx, Ny, Nz, n_mat, sms; LoopTiling tl; };
  static thread_local Last last = {0, 0, 0, 0, 0, {0, 0, 0, 0, 0, 0}};
  const int mats = p.n_mat <= kLoopMat ? p.n_mat : (p.n_mat <= 256 ? 256 : 65536);
  if (last.Nx == p.Nx && last.Ny == p.Ny && last.Nz == p.Nz && last.n_mat == mats && last.sms == sms)
    return last.tl;
  const int idb = p.n_mat <= 256 ? 1 : 2;
  const LoopTiling best = loop_search(p.Nx, p.Ny, p.Nz, sms, [&](int tx, int ty, int tz) {
    return LoopLayout<T>(tx, ty, tz, p.n_mat, idb);
  });
  last = {p.Nx, p.Ny, p.Nz, mats, sms, best};
  return best;
}

template <typename T, typename IdT, bool SMT>
cudaError_t launch_loop_as(const FitParams<T>& p, const LoopTiling& tl, int n_steps,
                           long long step0, unsigned* sync, cudaStream_t st) {
  auto kern = k_loop<T, IdT, SMT>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kLoopSmem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tl.nbx * tl.nby * tl.nbz));
  cfg.blockDim = dim3(kLoopThreads);
  cfg.dynamicSmemBytes = LoopLayout<T>(tl.tx, tl.ty, tl.tz, p.n_mat, (int)sizeof(IdT)).bytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, p, tl, n_steps, step0, sync);
}
}  // namespace

template <typename T>
bool loop_supported(const FitParams<T>& p) {
  if (p.N >= (1LL << 28) || p.n_mat > 65536 || p.j_mode == WK_J_ARRAY) return false;
  return loop_tiling<T>(p, loop_sms()).nbx > 0;
}

template <typename T>
cudaError_t launch_loop(const FitParams<T>& p, int n_steps, long long step0, unsigned* sync,
                        cudaStream_t st) {
  const LoopTiling tl = loop_tiling<T>(p, loop_sms());
  if (tl.nbx == 0) return cudaErrorInvalidValue;
  if (p.n_mat <= kLoopMat) return launch_loop_as<T, uint8_t, true>(p, tl, n_steps, step0, sync, st);
  if (p.n_mat <= 256) return launch_loop_as<T, uint8_t, false>(p, tl, n_steps, step0, sync, st);
  return launch_loop_as<T, uint16_t, false>(p, tl, n_steps, step0, sync, st);
}

template bool loop_supported<double>(const FitParams<double>&);
template bool loop_supported<float>(const FitParams<float>&);
template cudaError_t launch_loop<double>(const FitParams<double>&, int, long long, unsigned*,
                                         cudaStream_t);
template cudaError_t launch_loop<float>(const FitParams<float>&, int, long long, unsigned*,
                                        cudaStream_t);

}  // namespace wk
