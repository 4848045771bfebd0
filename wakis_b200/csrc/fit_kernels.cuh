// Helpers shared by the step kernels: Ez capture, J source of an E row,
// descriptor -> kernel parameter conversion, and the plane-marching kernel
// declaration.
#pragma once
#include "../../include/wakis_b200.h"
#include "fit_common.cuh"

namespace wk {

constexpr int kMarchThreads = 256;
constexpr int kShellBlock = 256;

// Shell decomposition of the two-pass and TMA schedules.  Blocks of 256 threads
// are decoded once per block (32-bit): planes k in {0,1,Nz-2,Nz-1} row by
// row (256 cells of a row per block), then rows j in {0,1,Ny-2,Ny-1} of the
// inner planes, then the columns i in {0,1,Nx-2,Nx-1} of the inner rows (4
// cells x 64 rows per block).  Cells that meet the single-coefficient
// condition take the lean rows; the rest the general row code.
struct ShellGrid {
  int cx, cy;          // 256-cell chunks per row, 64-row chunks per column
  int nbA, nbB, nbC;   // blocks of the three regions
};

inline ShellGrid shell_grid(int Nx, int Ny, int Nz, bool planes_only = false) {
  ShellGrid g;
  g.cx = (Nx + kShellBlock - 1) / kShellBlock;
  g.cy = (Ny - 4 + 63) / 64;
  g.nbA = 4 * Ny * g.cx;
  g.nbB = planes_only ? 0 : 4 * (Nz - 4) * g.cx;
  g.nbC = planes_only ? 0 : g.cy * (Nz - 4);
  return g;
}

__device__ __forceinline__ bool shell_cell_of(const ShellGrid& g, int b, int tid, int Nx, int Ny,
                                              int Nz, Cell& c) {
  if (b < g.nbA) {
    const int r = b / g.cx, ck = b - r * g.cx;
    const int kk = r / Ny;
    c.j = r - kk * Ny;
    c.k = kk < 2 ? kk : Nz - 4 + kk;
    c.i = ck * kShellBlock + tid;
    return c.i < Nx;
  }
  b -= g.nbA;
  if (b < g.nbB) {
    const int r = b / g.cx, ck = b - r * g.cx;
    const int jj = r & 3;
    c.k = 2 + (r >> 2);
    c.j = jj < 2 ? jj : Ny - 4 + jj;
    c.i = ck * kShellBlock + tid;
    return c.i < Nx;
  }
  b -= g.nbB;
  const int r = b / g.cy, cj = b - r * g.cy;
  const int ii = tid & 3;
  c.k = 2 + r;
  c.i = ii < 2 ? ii : Nx - 4 + ii;
  c.j = 2 + cj * 64 + (tid >> 2);
  return c.j <= Ny - 3;
}


template <typename T>
__device__ __forceinline__ void capture(const FitParams<T>& p, Cell c, long long n,
                                        long long step, T ez) {
  int a = c.i - p.cap_i0, b = c.j - p.cap_j0;
  const long long t = step - p.cap_step0;
  if (a >= 0 && a < p.cap_ni && b >= 0 && b < p.cap_nj && t >= 0 && t < p.cap_nt) {
    long long w = (long long)a * p.cap_nj + b;
    p.cap[(w * p.Nz + c.k) * p.cap_nt + t] = ez;
  }
}

// J value entering the E row of component d at cell n (before the update).
template <typename T>
__device__ __forceinline__ T j_in(const FitParams<T>& p, int d, Cell c, long long n,
                                  long long step, T e_old, T sigma) {
  if (d == 2 && c.i == p.ixs && c.j == p.iys) {
    if (p.line_on) {
      const long long t = step - p.line_step0;
      return (t >= 0 && t < p.line_nsteps) ? p.line[t * p.Nz + c.k] : T(0);
    }
    if (p.beam_on) return beam_j(p, step, c.k);
  }
  if (p.j_mode == WK_J_SIGMA_E) return mul(sigma, e_old);
  if (p.j_mode == WK_J_ARRAY) return p.J[(long long)d * p.N + n];
  return T(0);
}

template <typename T>
inline FitParams<T> make_params(const wk_fit_desc* d, int par) {
  FitParams<T> p;
  p.Nx = d->Nx; p.Ny = d->Ny; p.Nz = d->Nz;
  p.NxNy = (long long)d->Nx * d->Ny;
  p.N = p.NxNy * d->Nz;
  p.E_in = (T*)d->E[par]; p.H_in = (T*)d->H[par];
  p.E_out = (T*)d->E[par ^ 1]; p.H_out = (T*)d->H[par ^ 1];
  p.J = (T*)d->J;
  p.j_mode = d->j_mode; p.use_cond = d->use_conductivity;
  p.mat_id = d->mat_id; p.id_bytes = d->id_bytes;
  p.mat = (const T*)d->mat_table;
  p.n_mat = d->n_mat;
  p.Lx = (const T*)d->Lx; p.Ly = (const T*)d->Ly; p.Lz = (const T*)d->Lz;
  p.tLx = (const T*)d->tLx; p.tLy = (const T*)d->tLy; p.tLz = (const T*)d->tLz;
  p.iAx = (const T*)d->iAx; p.iAy = (const T*)d->iAy; p.iAz = (const T*)d->iAz;
  p.itAx = (const T*)d->itAx; p.itAy = (const T*)d->itAy; p.itAz = (const T*)d->itAz;
  for (int f = 0; f < 6; f++) { p.pec_face[f] = d->pec_face[f]; p.pmc_face[f] = d->pmc_face[f]; }
  p.has_pec = d->has_pec; p.has_pmc = d->has_pmc; p.h_desc = d->h_sum_desc;
  p.dt = (T)d->dt;
  p.dt64 = d->dt; p.dt32 = (float)d->dt; p.dt_is_f32 = d->dt_is_f32;
  p.beam_on = d->beam_on; p.ixs = d->ixs; p.iys = d->iys;
  p.b_qv = d->b_qv; p.b_v = d->b_v; p.b_v32 = (float)d->b_v; p.b_s0 = d->b_s0;
  p.b_c0 = d->b_c0; p.b_two_sig2 = d->b_two_sig2; p.b_dx = d->b_dx; p.b_dy = d->b_dy;
  p.zc = d->zc;
  p.line_on = d->line_on; p.line_step0 = d->line_step0; p.line_nsteps = d->line_nsteps;
  p.line = (const T*)d->line;
  p.cap_on = d->cap_on; p.cap_i0 = d->cap_i0; p.cap_j0 = d->cap_j0;
  p.cap_ni = d->cap_ni; p.cap_nj = d->cap_nj; p.cap_nt = d->cap_nt; p.cap_step0 = d->cap_step0;
  p.cap = (T*)d->cap;
  fast_div_magic((unsigned)d->Nx, &p.nx_mul, &p.nx_shift);
  p.status = d->status;
  p.step_dev = d->step_dev;
  p.faces_clean = d->faces_clean;
  p.wait_ns = d->wait_ns;
  p.steps_per_launch = d->steps_per_launch;
  return p;
}


// Cell of the idx-th shell cell (idx < shell_cells): planes k in {0, 1, Nz-2,
// Nz-1}, then rows j in {0, 1, Ny-2, Ny-1} of the inner planes, then columns i in
// {0, 1, Nx-2, Nx-1} of the inner rows (needs Nx, Ny, Nz >= 5, cells < 2^31).
inline long long shell_cells(int Nx, int Ny, int Nz, bool planes_only) {
  const long long planes = 4LL * Nx * Ny;
  return planes_only ? planes : planes + 4LL * (Nz - 4) * (Nx + Ny - 4);
}
// Whether cell n + off lies in a grid of N cells (0 <= n < N, 0 <= off <= N):
// the sum itself can pass 2^31 on the top planes of the largest grids.
__host__ __device__ __forceinline__ bool inside_after(int n, int off, int N) {
  return n < N - off;
}
__device__ __forceinline__ Cell shell_cell(int idx, int Nx, int Ny, int Nz) {
  Cell c;
  const int NxNy = Nx * Ny;
  if (idx < 4 * NxNy) {
    const int kk = idx / NxNy, rem = idx - kk * NxNy;
    c.k = kk < 2 ? kk : Nz - 4 + kk;
    c.j = rem / Nx;
    c.i = rem - c.j * Nx;
    return c;
  }
  idx -= 4 * NxNy;
  if (idx < 4 * Nx * (Nz - 4)) {
    const int t = idx / Nx;
    c.i = idx - t * Nx;
    c.j = (t & 3) < 2 ? (t & 3) : Ny - 4 + (t & 3);
    c.k = 2 + (t >> 2);
    return c;
  }
  idx -= 4 * Nx * (Nz - 4);
  c.i = (idx & 3) < 2 ? (idx & 3) : Nx - 4 + (idx & 3);
  const int t = idx >> 2, kk = t / (Ny - 4);
  c.k = 2 + kk;
  c.j = 2 + t - kk * (Ny - 4);
  return c;
}

// A launch that may start once every block of the kernel before it in the
// stream has passed pdl_trigger (or ended); pdl_wait ends when that kernel has
// ended and its writes are visible.  A kernel before it that was launched the
// ordinary way has seen everything earlier in the stream complete, so the
// blocks of both may read what those wrote.
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <typename... P, typename... A>
cudaError_t launch_beside(void (*kern)(P...), dim3 grid, int threads, int smem, cudaStream_t st,
                          A... args) {
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// Fused step of one cell with the general row code: the new H of the cell
// and of the three backward neighbours it needs is computed from the old
// state, then the new E of the cell.
template <typename T>
__device__ __forceinline__ void fused_cell_general(const FitParams<T>& p, long long step,
                                                   long long n, Cell c) {
  const long long N = p.N;
  int id = load_id(p.mat_id, p.id_bytes, n);
  if (p.cap_on) capture(p, c, n, step, p.E_in[2 * N + n]);
  T hn[3];
#pragma unroll
  for (int d = 0; d < 3; d++) hn[d] = h_row(p, p.E_in, p.H_in[d * N + n], d, c, n, id);
  T hm1[3], hmy[3], hmz[3];
  if (n >= 1) {
    Cell cm = minus_x(c, p.Nx, p.Ny); long long m = n - 1;
    int idm = load_id(p.mat_id, p.id_bytes, m);
    hm1[1] = h_row(p, p.E_in, p.H_in[N + m], 1, cm, m, idm);
    hm1[2] = h_row(p, p.E_in, p.H_in[2 * N + m], 2, cm, m, idm);
  } else { hm1[1] = hm1[2] = T(0); }
  hm1[0] = T(0);
  if (n >= p.Nx) {
    Cell cm = minus_y(c, p.Ny); long long m = n - p.Nx;
    int idm = load_id(p.mat_id, p.id_bytes, m);
    hmy[0] = h_row(p, p.E_in, p.H_in[m], 0, cm, m, idm);
    hmy[2] = h_row(p, p.E_in, p.H_in[2 * N + m], 2, cm, m, idm);
  } else { hmy[0] = hmy[2] = T(0); }
  hmy[1] = T(0);
  if (n >= p.NxNy) {
    Cell cm = c; cm.k--; long long m = n - p.NxNy;
    int idm = load_id(p.mat_id, p.id_bytes, m);
    hmz[0] = h_row(p, p.E_in, p.H_in[m], 0, cm, m, idm);
    hmz[1] = h_row(p, p.E_in, p.H_in[N + m], 1, cm, m, idm);
  } else { hmz[0] = hmz[1] = T(0); }
  hmz[2] = T(0);
  auto hv = [&](int e, int kind) -> T {
    if (kind == 0) return hn[e];
    if (kind == 1) return hm1[e];
    if (kind == 2) return hmy[e];
    return hmz[e];
  };
#pragma unroll
  for (int d = 0; d < 3; d++) {
    T ieps = p.mat[9 * id + d];
    T sigma = p.mat[9 * id + 6 + d];
    T eold = p.E_in[d * N + n];
    T jv = j_in(p, d, c, n, step, eold, sigma);
    T curl = e_curl_acc(p, d, c, n, ieps, hv);
    T enew = add(eold, mul(p.dt, sub(curl, mul(ieps, jv))));
    p.E_out[d * N + n] = enew;
    if (p.j_mode == WK_J_ARRAY && p.use_cond) p.J[d * N + n] = mul(sigma, enew);
  }
#pragma unroll
  for (int d = 0; d < 3; d++) p.H_out[d * N + n] = hn[d];
}

// Launch the two-pass schedule (H pass, then E pass; interior lean kernels
// and general shell kernels) of one step (fit_fused.cu); needs Nx, Ny, Nz >= 5.
// kb = planes per thread (1, 2 or 4).
template <typename T>
cudaError_t launch_two_pass(const FitParams<T>& p, long long step, cudaStream_t st, int kb);

// Step of the shell cells (planes_only: of the four z-boundary planes) from the
// old state, in one launch that lets a launch_beside one start with it
// (fit_fused.cu); needs Nx, Ny, Nz >= 5, cells < 2^31, separate old and new state.
template <typename T>
cudaError_t launch_shell_step(const FitParams<T>& p, long long step, cudaStream_t st,
                              bool planes_only);

// TMA-staged fused step (fit_tma.cu): interior tiles + shell launches.
template <typename T>
bool tma_supported(const FitParams<T>& p);
// Row and component pitch of 16 bytes.
template <typename T>
bool tma_pitch(const FitParams<T>& p);
template <typename T>
cudaError_t launch_tma(const FitParams<T>& p, long long step, cudaStream_t st, int KC,
                       int rows);

// All steps of a call in one launch, for small grids (fit_loop.cu): those whose
// state fits the shared memory of the SMs; every dimension >= 5.
template <typename T>
bool loop_supported(const FitParams<T>& p);
template <typename T>
cudaError_t launch_loop(const FitParams<T>& p, int n_steps, long long step0, unsigned* sync,
                        cudaStream_t st);

// A launch of launch_loop or launch_loop_comp refused because its blocks cannot
// all be resident (a context that is given fewer SMs than the device has):
// nothing was written, and the call runs step by step.  Clears the error.
inline bool loop_refused(cudaError_t e) {
  if (e != cudaErrorCooperativeLaunchTooLarge) return false;
  (void)cudaGetLastError();
  return true;
}

// Two steps per launch (fit_tma2.cu): k_tma2 covers grids whose faces are
// all PEC-masked and clean, with J = 0 or sigma*E.
template <typename T>
bool tma2_supported(const FitParams<T>& p);
template <typename T>
cudaError_t launch_tma2(const FitParams<T>& p, long long step, cudaStream_t st, int KC);

}  // namespace wk
