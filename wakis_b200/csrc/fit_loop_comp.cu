// Many steps per launch of the FP32-compensated step (sm_100a): the scheme of
// fit_loop.cu (one cooperative launch, every block keeps its tile in shared
// memory, one grid barrier per step, the halo's E exchanged through L2) on the
// state of float values and bf16 words (fit_comp.cuh).
//
// The rows are those of the compensated TMA step (fit_tma_comp.cuh), one cell
// at a time: float row sums from factors formed in FP64 and rounded once, the
// increment added by comp_add; with z faces that are not PEC-masked the planes
// 0, 1, Nz-2, Nz-1 take its FP64 shell rows, and
// the E of plane 2 reads the H of plane 1 that its tiles form with float rows
// (kept beside the stored one).  So a cell's values do not depend on which of
// the two kernels steps it.  Grids that the compensated TMA step does not take
// (Nx no multiple of 4) are stepped as the two-pass schedule steps them, value
// for value (WIDE): factors formed in FP64 from the row's area, material and
// length and rounded once, FP64 shell rows two cells deep on all faces.  The x/y
// faces are PEC-masked (an E entry tangential to a face it lies on enters no H
// row, an E row tangential to its face gets no curl); the compensation words
// of E travel only where a shell row reads them.
//
// Bound like fit_loop.cu.  Measured on B200 (us a step, launches per step
// before / here, the longest call's share of the set-up included): 16x16x32
// closed 11.3 / 2.7, 16x20x40 open ends 27.7 / 4.1, 40x40x80 open 28.7 / 5.8,
// 52x52x110 open 32.8 / 9.4, 64x60x100 absorber ends 14.4 / 9.9; WIDE: 31x29x60
// open 24.6 / 4.6, 33x40x70 lossy 33.0 / 5.8, 61x47x90 absorber 38.9 / 9.7.
#include <stdint.h>

#include "../../include/wakis_b200.h"
#include "abi_internal.h"
#include "fit_comp.cuh"
#include "fit_loop.cuh"

namespace wk {

namespace {

constexpr int kCompMat = 64;
// classes of the cells with FP64 rows: from the tables in shared memory, or by
// the general code where a neighbour's length differs from the cell's own
constexpr uint32_t kShell = 2, kShellGen = 3;

// Factors of the two columns of a row (float, dt folded in).
__device__ __forceinline__ float2 row_pair(double dt, double iA, double La, double Lb) {
  return make_float2((float)((dt * iA) * La), (float)((dt * iA) * Lb));
}

struct CompLayout {
  int e, h, ec, hc, h1, tab, mat, lists, ids, bytes;
  int n_ext, n_own, n_shell;
  __host__ __device__ CompLayout(int tx, int ty, int tz, int n_mat) {
    const int es = (tx + 2) * (ty + 2) * (tz + 2), hs = (tx + 1) * (ty + 1) * (tz + 1);
    n_own = tx * ty * tz;
    n_ext = n_own + ty * tz + tx * tz + tx * ty;
    n_shell = 2 * (ty * tz + tx * tz + tx * ty) + 2 * (tx + ty + tz);
    auto r16 = [](int b) { return (b + 15) / 16 * 16; };
    e = 0;
    h = e + r16(12 * es);
    ec = h + r16(12 * hs);
    hc = ec + r16(6 * es);
    h1 = hc + r16(6 * hs);
    tab = h1 + r16(8 * (tx + 1) * (ty + 1));   // factor pairs, areas and lengths
    const int faces = (ty + 1) * (tz + 1) + (tx + 1) * (tz + 1) + (tx + 1) * (ty + 1);
    mat = tab + r16((4 * faces + 2 * (tx + ty + tz + 3)) * 8);
    lists = mat + r16(n_mat * 136);
    ids = lists + r16((n_ext + n_own + n_shell) * 4);
    bytes = ids + r16(n_ext + n_own) + 256;
  }
};

template <bool SIG, bool WIDE>
__global__ void __launch_bounds__(kLoopThreads, 1)
k_loop_comp(const __grid_constant__ FitParams<double> p, CompState st, LoopTiling tl, int shell,
            int n_steps, long long step0, unsigned* sync) {
  constexpr int TH = kLoopThreads;
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int s_len[4], s_count[10];
  const CompLayout lay(tl.tx, tl.ty, tl.tz, p.n_mat);
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
  const int EX = tx + 2, EP = EX * (ty + 2), EV = EP * (tz + 2);
  const int HX = tx + 1, HP = HX * (ty + 1), HV = HP * (tz + 1);
  float* Es = reinterpret_cast<float*>(sm + lay.e);
  float* Hs = reinterpret_cast<float*>(sm + lay.h);
  comp_t* Ecs = reinterpret_cast<comp_t*>(sm + lay.ec);
  comp_t* Hcs = reinterpret_cast<comp_t*>(sm + lay.hc);
  float* H1 = reinterpret_cast<float*>(sm + lay.h1);     // Hx, Hy of plane 1 by float rows
  // factor pairs of the rows at box coordinates: H x (b, c), y (a, c), z (a, b), then E
  float2* fhx = reinterpret_cast<float2*>(sm + lay.tab);
  float2* fhy = fhx + (ty + 1) * (tz + 1);
  float2* fhz = fhy + HX * (tz + 1);
  float2* fex = fhz + HP;
  float2* fey = fex + (ty + 1) * (tz + 1);
  float2* fez = fey + HX * (tz + 1);
  float* mt = reinterpret_cast<float*>(sm + lay.mat);   // [n_mat][16] imu, ieps, dt ieps, dt ieps sigma
  uint32_t* lh = reinterpret_cast<uint32_t*>(sm + lay.lists);
  uint32_t* le = lh + lay.n_ext;
  uint32_t* ls = le + lay.n_own;
  uint8_t* idh = sm + lay.ids;
  uint8_t* ide = idh + lay.n_ext;
  const int nb = (i0 - 1) + (j0 - 1) * Nx + (k0 - 1) * plane;
  auto flat = [&](int a, int b, int c) { return nb + a + b * Nx + c * plane; };

  // areas, lengths and the material table in FP64
  double* ahx = reinterpret_cast<double*>(fez + HP);
  double* ahy = ahx + (ty + 1) * (tz + 1);
  double* ahz = ahy + HX * (tz + 1);
  double* aex = ahz + HP;
  double* aey = aex + (ty + 1) * (tz + 1);
  double* aez = aey + HX * (tz + 1);
  double* lx = aez + HP;
  double *ly = lx + HX, *lz = ly + ty + 1, *tlx = lz + tz + 1, *tly = tlx + HX, *tlz = tly + ty + 1;
  double* mw = reinterpret_cast<double*>(mt + 16 * p.n_mat);   // [n_mat][9]

  // ---- set-up
  const LoopDiv dEP(EP), dEX(EX), dHP(HP), dHX(HX), dY1(ty + 1), dTP(tx * ty), dTX(tx);
  for (int q = tid; q < EV; q += TH) {
    const int c = dEP.div(q), r = q - c * EP, b = dEX.div(r), a = r - b * EX;
    const int n = flat(a, b, c);
    const bool v = n >= 0 && n < N;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      cp_async<4>(Es + d * EV + q, st.E_in + (v ? d * N + n : 0), v);
      Ecs[d * EV + q] = v ? st.Ec_in[d * N + n] : (comp_t)0;
    }
  }
  for (int q = tid; q < HV; q += TH) {
    const int c = dHP.div(q), r = q - c * HP, b = dHX.div(r), a = r - b * HX;
    const int n = flat(a, b, c);
    const bool v = n >= 0 && n < N;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      cp_async<4>(Hs + d * HV + q, st.H_in + (v ? d * N + n : 0), v);
      Hcs[d * HV + q] = v ? st.Hc_in[d * N + n] : (comp_t)0;
    }
  }
  cp_async_commit();
  // factors; positions outside the grid are read by no cell with float rows
  for (int q = tid; q < (ty + 1) * (tz + 1); q += TH) {
    const int c = dY1.div(q), j = max(j0 - 1 + q - c * (ty + 1), 0), k = max(k0 - 1 + c, 0);
    const long long m = j + (long long)k * Ny;
    ahx[q] = p.iAx[m];
    aex[q] = p.itAx[m];
    if (!WIDE) {
      fhx[q] = row_pair(p.dt, p.iAx[m], p.Ly[j], p.Lz[k]);
      fex[q] = row_pair(p.dt, p.itAx[m], p.tLy[j], p.tLz[k]);
    }
  }
  for (int q = tid; q < HX * (tz + 1); q += TH) {
    const int c = dHX.div(q), i = max(i0 - 1 + q - c * HX, 0), k = max(k0 - 1 + c, 0);
    const long long m = i + (long long)k * Nx;
    ahy[q] = p.iAy[m];
    aey[q] = p.itAy[m];
    if (!WIDE) {
      fhy[q] = row_pair(p.dt, p.iAy[m], p.Lx[i], p.Lz[k]);
      fey[q] = row_pair(p.dt, p.itAy[m], p.tLx[i], p.tLz[k]);
    }
  }
  for (int q = tid; q < HP; q += TH) {
    const int c = dHX.div(q), i = max(i0 - 1 + q - c * HX, 0), j = max(j0 - 1 + c, 0);
    const long long m = i + (long long)j * Nx;
    ahz[q] = p.iAz[m];
    aez[q] = p.itAz[m];
    if (!WIDE) {
      fhz[q] = row_pair(p.dt, p.iAz[m], p.Lx[i], p.Ly[j]);
      fez[q] = row_pair(p.dt, p.itAz[m], p.tLx[i], p.tLy[j]);
    }
  }
  if (tid < HX) { const int i = max(i0 - 1 + tid, 0); lx[tid] = p.Lx[i]; tlx[tid] = p.tLx[i]; }
  if (tid < ty + 1) { const int j = max(j0 - 1 + tid, 0); ly[tid] = p.Ly[j]; tly[tid] = p.tLy[j]; }
  if (tid < tz + 1) { const int k = max(k0 - 1 + tid, 0); lz[tid] = p.Lz[k]; tlz[tid] = p.tLz[k]; }
  for (int q = tid; q < 9 * p.n_mat; q += TH) mw[q] = p.mat[q];
  for (int q = tid; q < p.n_mat * 3 && !WIDE; q += TH) {
    const int m = q / 3, d = q - m * 3;
    const double* m0 = p.mat + 9 * m;
    mt[m * 16 + d] = (float)m0[3 + d];
    mt[m * 16 + 4 + d] = (float)m0[d];
    mt[m * 16 + 8 + d] = (float)(p.dt * m0[d]);
    mt[m * 16 + 12 + d] = (float)((p.dt * m0[d]) * m0[6 + d]);
  }
  auto shell_cell = [&](Cell c) {
    if (WIDE && (c.i < 2 || c.i > Nx - 3 || c.j < 2 || c.j > Ny - 3 || c.k < 2 || c.k > Nz - 3))
      return true;
    return shell && (c.k < 2 || c.k >= Nz - 2);
  };
  auto row_bits = [&](Cell c) {
    int rows = 0;
    for (int d = 0; d < 3; d++)
      if (face_val(p.pec_face, d, c.i, c.j, c.k, Nx, Ny, Nz)) rows |= 1 << d;
    return rows;
  };
  auto h_entry = [&](int q, uint32_t& e) -> int {
    const int c = dHP.div(q), r = q - c * HP, b = dHX.div(r), a = r - b * HX;
    const int n = flat(a, b, c);
    const int low = (a == 0) + (b == 0) + (c == 0);
    if (low > 1 || n < 0) return -1;
    const int outer = (low == 0 && a < tx && b < ty && c < tz) ? 0 : 3;
    const Cell cc = cell_of(n, Nx, Ny);
    if (low) {
      // a halo cell whose H enters only masked E rows is left alone
      const Cell u = cell_of(n + (a == 0 ? 1 : (b == 0 ? Nx : plane)), Nx, Ny);
      if ((row_bits(u) & ~(1 << (a == 0 ? 0 : (b == 0 ? 1 : 2)))) == 0) return -1;
    }
    bool wrap;
    const int m = loop_bits<double, 1>(p, cc, 7, wrap);
    wrap |= (a == 0 && i0 == 0) || (b == 0 && j0 == 0);
    const uint32_t cls = shell_cell(cc) ? (wrap ? kShellGen : kShell)
                                        : (m == 511 ? kRegular : kMasked);
    e = loop_entry(a, b, c, m, 7, cls);
    return outer + min((int)cls, 2);
  };
  auto e_entry = [&](int q, uint32_t& e) -> int {
    const int c = dTP.div(q), r = q - c * tx * ty, b = dTX.div(r), a = r - b * tx;
    const Cell cc = {i0 + a, j0 + b, k0 + c};
    const int rows = row_bits(cc);
    bool wrap;
    loop_bits<double, -1>(p, cc, rows, wrap);
    const uint32_t cls = shell_cell(cc) ? (wrap ? kShellGen : kShell)
                                        : (rows == 7 ? kRegular : kMasked);
    e = loop_entry(a + 1, b + 1, c + 1, 511, rows, cls);
    return 6 + min((int)cls, 2);
  };
  auto s_entry = [&](int q, uint32_t& e) -> int {
    const int c = dEP.div(q), r = q - c * EP, b = dEX.div(r), a = r - b * EX;
    const int low = (a == 0) + (b == 0) + (c == 0);
    const int high = (a == tx + 1) + (b == ty + 1) + (c == tz + 1);
    const int n = flat(a, b, c);
    e = loop_entry(a, b, c, 0, 0, 0);
    return low + high > 0 && low <= 1 && high <= 1 && n >= 0 && n < N ? 9 : -1;
  };
  loop_lists(s_count, s_len, HV, h_entry, lh, tx * ty * tz, e_entry, le, EV, s_entry, ls);
  const int nh = s_len[0], ne = s_len[1], nsh = s_len[2], nh_own = s_len[3];
  auto id_of = [&](uint32_t e) {
    return (uint8_t)load_id(p.mat_id, p.id_bytes, flat(e & 63, e >> 6 & 63, e >> 12 & 63));
  };
  for (int q = tid; q < nh; q += TH) idh[q] = id_of(lh[q]);
  for (int q = tid; q < ne; q += TH) ide[q] = id_of(le[q]);
  cp_async_wait<0>();
  __syncthreads();

  const bool src = (p.line_on || p.beam_on) && p.ixs >= i0 && p.ixs < i1 && p.iys >= j0 && p.iys < j1;
  const bool cap = p.cap_on && p.cap_i0 < i1 && p.cap_i0 + p.cap_ni > i0 && p.cap_j0 < j1 &&
                   p.cap_j0 + p.cap_nj > j0;
  auto pick = [](uint32_t bits, int b, float v) { return (bits & b) ? v : 0.f; };
  const int eoff[4] = {0, 1, EX, EP}, hoff[4] = {0, 1, HX, HP};
  const bool desc = p.h_desc != 0;
  // factors of the two columns of a row: material f of the table, area and
  // lengths (WIDE), or the pair of the row times the float material
  auto wide = [&](double area, double mu, double La, double Lb) {
    const double R = area * mu;
    return make_float2((float)(p.dt * (R * La)), (float)(p.dt * (R * Lb)));
  };
  auto narrow = [&](float mu, float2 f) {
    return make_float2(__fmul_rn(mu, f.x), __fmul_rn(mu, f.y));
  };

  auto h_cells = [&](int q_lo, int q_hi) {
    for (int q = q_lo + tid; q < q_hi; q += TH) {
      const uint32_t e = lh[q];
      const int a = e & 63, b = e >> 6 & 63, c = e >> 12 & 63;
      const int at = c * HP + b * HX + a, ae = c * EP + b * EX + a;
      const uint32_t cls = e >> 30;
      const bool below = !WIDE && cls >= kShell && k0 - 1 + c == 1;   // plane 1: both forms
      if (cls < kShell || below) {
        const float* E = Es + ae;
        const int id = idh[q];
        float ex0 = E[0], ey0 = E[EV], ez0 = E[2 * EV], ey1 = E[EV + 1], ez1 = E[2 * EV + 1],
              ex2 = E[EX], ez2 = E[2 * EV + EX], ex3 = E[EP], ey3 = E[EV + EP];
        if (cls != kRegular) {
          const uint32_t w = e >> 18;
          ex0 = pick(w, bXO, ex0); ey0 = pick(w, bYO, ey0); ez0 = pick(w, bZO, ez0);
          ey1 = pick(w, bYX, ey1); ez1 = pick(w, bZX, ez1);
          ex2 = pick(w, bXY, ex2); ez2 = pick(w, bZY, ez2);
          ex3 = pick(w, bXZ, ex3); ey3 = pick(w, bYZ, ey3);
        }
        const int qx = c * (ty + 1) + b, qy = c * HX + a, qz = b * HX + a;
        const float* m0 = mt + 16 * id;
        const double* w0 = mw + 9 * id;
        const float2 fx = WIDE ? wide(ahx[qx], w0[3], ly[b], lz[c]) : narrow(m0[0], fhx[qx]);
        const float2 fy = WIDE ? wide(ahy[qy], w0[4], lx[a], lz[c]) : narrow(m0[1], fhy[qy]);
        const float2 fz = WIDE ? wide(ahz[qz], w0[5], lx[a], ly[b]) : narrow(m0[2], fhz[qz]);
        float s[3];
        if (WIDE) {
          s[0] = hsum_x(desc, fx.x, fx.y, ey0, ey3, ez0, ez2);
          s[1] = hsum_y(desc, fy.x, fy.y, ex0, ex3, ez0, ez1);
          s[2] = hsum_z(desc, fz.x, fz.y, ex0, ex2, ey0, ey1);
        } else {
          s[0] = __fmaf_rn(fx.x, __fsub_rn(ey0, ey3), __fmul_rn(fx.y, __fsub_rn(ez2, ez0)));
          s[1] = __fmaf_rn(fy.x, __fsub_rn(ex3, ex0), __fmul_rn(fy.y, __fsub_rn(ez0, ez1)));
          s[2] = __fmaf_rn(fz.x, __fsub_rn(ex0, ex2), __fmul_rn(fz.y, __fsub_rn(ey1, ey0)));
        }
#pragma unroll
        for (int d = 0; d < 3; d++) {
          float v;
          comp_t w;
          comp_add(Hs[d * HV + at], Hcs[d * HV + at], -s[d], v, w);
          if (below) {
            if (d < 2) H1[d * HP + b * HX + a] = v;
          } else {
            Hs[d * HV + at] = v;
            Hcs[d * HV + at] = w;
          }
        }
      }
      if (cls >= kShell) {
        auto ev = [&](int d, int kind) {
          const int m = d * EV + ae + eoff[kind];
          return comp_value(Es[m], Ecs[m]);
        };
        double h[3];
#pragma unroll
        for (int d = 0; d < 3; d++) h[d] = comp_value(Hs[d * HV + at], Hcs[d * HV + at]);
        const int id = idh[q];
        const double* m0 = mw + 9 * id;
        RowCols<double> f;
        double R0, R1, R2;
        if (cls == kShell) {
          const uint32_t w = e >> 18;
          auto has = [&](int bit, double L) { return (w & bit) ? L : 0.0; };
          const double Lx = lx[a], Ly = ly[b], Lz = lz[c];
          f = {has(bXO, Lx), has(bXZ, Lx), has(bXY, Lx), has(bYO, Ly), has(bYZ, Ly),
               has(bYX, Ly), has(bZO, Lz), has(bZX, Lz), has(bZY, Lz)};
          R0 = ahx[c * (ty + 1) + b];
          R1 = ahy[c * HX + a];
          R2 = ahz[b * HX + a];
        } else {
          Cell cc = {i0 - 1 + a, j0 - 1 + b, k0 - 1 + c};
          if (cc.i < 0) { cc.i = Nx - 1; cc.j--; }
          if (cc.j < 0) { cc.j += Ny; cc.k--; }
          ColumnInv<double, 1> ci;
          ci.init(p, cc.i, cc.j);
          f = ci.at(p, cc.k);
          R0 = __ldg(p.iAx + cc.j + (long long)cc.k * Ny);
          R1 = __ldg(p.iAy + cc.i + (long long)cc.k * Nx);
          R2 = __ldg(p.iAz + cc.i + (long long)cc.j * Nx);
        }
        h_rows(p.dt, desc, mul(R0, m0[3]), mul(R1, m0[4]), mul(R2, m0[5]), f, ev(0, 0),
               ev(1, 0), ev(2, 0), ev(1, 1), ev(2, 1), ev(0, 2), ev(2, 2), ev(0, 3), ev(1, 3), h[0],
               h[1], h[2]);
#pragma unroll
        for (int d = 0; d < 3; d++) comp_split(h[d], Hs[d * HV + at], Hcs[d * HV + at]);
      }
    }
  };

  auto e_cells = [&](long long step, float* Eo, comp_t* Eco, float* Hf, comp_t* Hcf) {
    for (int q = tid; q < ne; q += TH) {
      const uint32_t e = le[q];
      const int a = e & 63, b = e >> 6 & 63, c = e >> 12 & 63;
      const int at = c * EP + b * EX + a, ah = c * HP + b * HX + a;
      const int n = flat(a, b, c);
      const Cell cc = {i0 - 1 + a, j0 - 1 + b, k0 - 1 + c};
      const float* H = Hs + ah;
      const uint32_t cls = e >> 30;
      float v[3] = {Es[at], Es[EV + at], Es[2 * EV + at]};
      comp_t w[3] = {Ecs[at], Ecs[EV + at], Ecs[2 * EV + at]};
      if (cap) capture(p, cc, n, step, comp_value(v[2], w[2]));
      if (cls < kShell) {
        const int id = ide[q];
        const float* m0 = mt + 16 * id;
        const double* w0 = mw + 9 * id;
        const float hx0 = H[0], hy0 = H[HV], hz0 = H[2 * HV];
        const int qx = c * (ty + 1) + b, qy = c * HX + a, qz = b * HX + a;
        const float2 fx = WIDE ? wide(aex[qx], w0[0], tly[b], tlz[c]) : narrow(m0[4], fex[qx]);
        const float2 fy = WIDE ? wide(aey[qy], w0[1], tlx[a], tlz[c]) : narrow(m0[5], fey[qy]);
        const float2 fz = WIDE ? wide(aez[qz], w0[2], tlx[a], tly[b]) : narrow(m0[6], fez[qz]);
        const bool two = !WIDE && shell && cc.k == 2;
        const float hx3 = two ? H1[b * HX + a] : H[-HP], hy3 = two ? H1[HP + b * HX + a] : H[HV - HP];
        const float hy1 = H[HV - 1], hz1 = H[2 * HV - 1], hx2 = H[-HX], hz2 = H[2 * HV - HX];
        float cu[3];
        if (WIDE) {
          cu[0] = ecurl_x(fx.x, fx.y, hy0, hz2, hy3, hz0);
          cu[1] = ecurl_y(fy.x, fy.y, hx0, hz1, hx3, hz0);
          cu[2] = ecurl_z(fz.x, fz.y, hx0, hy1, hx2, hy0);
        } else {
          cu[0] = __fmaf_rn(fx.x, __fsub_rn(hy3, hy0), __fmul_rn(fx.y, __fsub_rn(hz0, hz2)));
          cu[1] = __fmaf_rn(fy.x, __fsub_rn(hx0, hx3), __fmul_rn(fy.y, __fsub_rn(hz1, hz0)));
          cu[2] = __fmaf_rn(fz.x, __fsub_rn(hx2, hx0), __fmul_rn(fz.y, __fsub_rn(hy0, hy1)));
        }
#pragma unroll
        for (int d = 0; d < 3; d++) {
          if (!(e >> 27 & 1 << d)) cu[d] = 0.f;
          float jt = 0.f;
          if (SIG)
            jt = WIDE ? (float)(p.dt * w0[d] * (w0[6 + d] * comp_value(v[d], w[d])))
                      : __fmul_rn(m0[12 + d], v[d]);
          if (d == 2 && src && cc.i == p.ixs && cc.j == p.iys) {
            const long long lt = step - p.line_step0;
            const double jb = p.line_on ? ((lt >= 0 && lt < p.line_nsteps)
                                               ? p.line[lt * Nz + cc.k] : 0.0)
                                        : beam_j(p, step, cc.k);
            jt = WIDE ? (float)(p.dt * w0[2] * jb) : (float)((double)m0[10] * jb);
          }
          comp_add(v[d], w[d], __fsub_rn(cu[d], jt), v[d], w[d]);
        }
      } else {
        auto hv = [&](int d, int kind) { return (double)H[d * HV - hoff[kind]]; };
        double x[3] = {comp_value(v[0], w[0]), comp_value(v[1], w[1]), comp_value(v[2], w[2])};
        const int id = ide[q];
        const double* m0 = mw + 9 * id;
        const uint32_t rows = e >> 27;
        auto row = [&](int d, double R) { return (rows >> d & 1) ? R : 0.0; };
        RowCols<double> f;
        if (cls == kShell) {
          const double tLx = tlx[a], tLy = tly[b], tLz = tlz[c];
          f = {tLx, tLx, tLx, tLy, tLy, tLy, tLz, tLz, tLz};
        } else {
          ColumnInv<double, -1> ci;
          ci.init(p, cc.i, cc.j);
          f = ci.at(p, cc.k);
        }
        double cu[3];
        e_rows(row(0, mul(m0[0], aex[c * (ty + 1) + b])), row(1, mul(m0[1], aey[c * HX + a])),
               row(2, mul(m0[2], aez[b * HX + a])), f, hv(0, 0), hv(1, 0), hv(2, 0), hv(1, 1),
               hv(2, 1), hv(0, 2), hv(2, 2), hv(0, 3), hv(1, 3), cu[0], cu[1], cu[2]);
#pragma unroll
        for (int d = 0; d < 3; d++) {
          double jv = SIG ? mul(m0[6 + d], x[d]) : 0.0;
          if (d == 2 && src && cc.i == p.ixs && cc.j == p.iys)
            jv = j_in(p, d, cc, n, step, x[d], m0[6 + d]);
          x[d] = comp_e_new(p.dt, m0[d], jv, cu[d], x[d]);
        }
#pragma unroll
        for (int d = 0; d < 3; d++) comp_split(x[d], v[d], w[d]);
      }
      const bool edge = a == 1 || a == tx || b == 1 || b == ty || c == 1 || c == tz;
      const bool word = Hf || (edge && (WIDE || (shell && (cc.k <= 2 || cc.k >= Nz - 2))));
#pragma unroll
      for (int d = 0; d < 3; d++) {
        Es[d * EV + at] = v[d];
        Ecs[d * EV + at] = w[d];
        if (Hf || edge) Eo[d * N + n] = v[d];
        if (word) Eco[d * N + n] = w[d];
        if (Hf) {
          Hf[d * N + n] = H[d * HV];
          Hcf[d * N + n] = Hcs[d * HV + ah];
        }
      }
    }
  };

  const long long lim = p.wait_ns == 0 ? 20 * kWaitNs : p.wait_ns;
  float *Eo = st.E_out, *Ex = const_cast<float*>(st.E_in);
  comp_t *Co = st.Ec_out, *Cx = const_cast<comp_t*>(st.Ec_in);
  unsigned target = 0;
  bool ok = true;
  h_cells(0, nh_own);
  for (int s = 0; s < n_steps; s++) {
    h_cells(nh_own, nh);
    __syncthreads();
    const bool last = s + 1 == n_steps;
    const bool odd = n_steps & 1;
    e_cells(step0 + s, Eo, Co,
            last ? (odd ? st.H_out : const_cast<float*>(st.H_in)) : nullptr,
            last ? (odd ? st.Hc_out : const_cast<comp_t*>(st.Hc_in)) : nullptr);
    if (last) break;
    __syncthreads();
    if (tid == 0) red_release(sync + kSyncCount);
    target += gridDim.x;
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
      const int n = flat(a, b, c), at = c * EP + b * EX + a;
#pragma unroll
      for (int d = 0; d < 3; d++) Es[d * EV + at] = Eo[d * N + n];
      if (WIDE || shell) {
        const int k = n / plane;
        if (WIDE || k <= 2 || k >= Nz - 2)
#pragma unroll
          for (int d = 0; d < 3; d++) Ecs[d * EV + at] = Co[d * N + n];
      }
    }
    float* sw = Ex; Ex = Eo; Eo = sw;
    comp_t* sc = Cx; Cx = Co; Co = sc;
    __syncthreads();
  }
  loop_leave(sync);
}

LoopTiling comp_tiling(const FitParams<double>& p, int sms) {
  struct Last { int Nx, Ny, Nz, n_mat, sms; LoopTiling tl; };
  static thread_local Last last = {0, 0, 0, 0, 0, {0, 0, 0, 0, 0, 0}};
  if (last.Nx == p.Nx && last.Ny == p.Ny && last.Nz == p.Nz && last.n_mat == p.n_mat &&
      last.sms == sms)
    return last.tl;
  const LoopTiling best = loop_search(p.Nx, p.Ny, p.Nz, sms, [&](int tx, int ty, int tz) {
    return CompLayout(tx, ty, tz, p.n_mat);
  });
  last = {p.Nx, p.Ny, p.Nz, p.n_mat, sms, best};
  return best;
}

}  // namespace

bool loop_comp_supported(const FitParams<double>& p) {
  if (p.N >= (1LL << 28) || p.n_mat > kCompMat || tma_comp_mode(p) == 0) return false;
  return comp_tiling(p, loop_sms()).nbx > 0;
}

cudaError_t launch_loop_comp(const wk_fit_desc* d, const FitParams<double>& p, int n_steps,
                             long long step0, cudaStream_t st) {
  const LoopTiling tl = comp_tiling(p, loop_sms());
  if (tl.nbx == 0) return cudaErrorInvalidValue;
  const bool sig = p.j_mode == WK_J_SIGMA_E;
  auto kern = tma_comp_supported(d, p) ? (sig ? k_loop_comp<true, false> : k_loop_comp<false, false>)
                                       : (sig ? k_loop_comp<true, true> : k_loop_comp<false, true>);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kLoopSmem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tl.nbx * tl.nby * tl.nbz));
  cfg.blockDim = dim3(kLoopThreads);
  cfg.dynamicSmemBytes = CompLayout(tl.tx, tl.ty, tl.tz, p.n_mat).bytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, p, comp_state(d, d->par), tl, (int)(tma_comp_mode(p) == 2),
                            n_steps, step0, d->sync);
}

}  // namespace wk
