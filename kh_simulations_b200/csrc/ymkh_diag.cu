// ymkh_diag.cu — on-device diagnostics: energy (YM_Energy.cu:3-32), circular
// mode amplitudes (ymgpu2d/analysis/remote_timeseries.py:62-77,
// ymgpu2d/analysis/resolution_convergence.py:77-86) and the non-Abelian Gauss
// law residual.
//
// The reference checks the Gauss constraint offline, from 6-digit CSV snapshots
// (ymgpu2d/analysis/gauss_check.py:40-110):
//   G^a = (Ex^a - Ex^a[x-1]) / dx + (Ez^a - Ez^a[z-1]) / dz
//       + alpha (Az x Ezc)^a - (Q^a_A nA + Q^a_B nB),
//   Ezc^a = (Ez^a + Ez^a[z-1]) / 2, neighbours wrapping around in x and z.
// Here it runs on the FP64 state.  Each cell's terms are evaluated operand
// for operand as that script writes them.
//
// Every diagnostic is two kernels: partial sums over the grid, then one small
// kernel that reduces them (it is launched while the first runs and waits for
// it: griddepcontrol).  What bounds them: reading the arrays once on a large
// grid; on a small one the launches, and how many CTAs share the cells, so
// the cells per thread shrink with the grid.  The sums of energy and Gauss
// terms are compensated (Neumaier); all orders are fixed by the grid size
// alone.  The results go straight to the caller's page of pinned host memory.
//
// Measured (us per call with its result on the host) against a final kernel of
// one thread per value, amplitudes of one thread per column and results copied
// to pageable memory: at 256 x 768 energy 62 -> 24, amplitude 113 -> 26,
// weighted 230 -> 31, Gauss 55 -> 37; at 1024 x 2048 89 -> 64, 333 -> 32,
// 642 -> 39, 295 -> 133; at 4096 x 8192 658 -> 636 (6.3 TB/s), 2682 -> 118,
// 3898 -> 155, 4435 -> 1481.

#include "ymkh_common.cuh"

namespace ymkh {

namespace {

// Lets the stream's next kernel start its launch; the final kernels wait for
// the partial sums with dependency_wait.  They take those as plain pointers:
// const __restrict__ would promise memory that nobody writes while the kernel
// runs, whose loads may be moved in front of the wait.
__device__ __forceinline__ void dependency_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// (s, c) += (s2, c2), two compensated sums
__device__ __forceinline__ void neumaier_merge(double& s, double& c, double s2, double c2) {
  c += c2;
  neumaier_add(s, c, s2);
}

// Sum over the CTA of every thread's (s, c), in thread 0: a butterfly in each
// warp, then over the warps.
template <int NT>
__device__ __forceinline__ void neumaier_block(double& s, double& c) {
  __shared__ double ws[NT / 32][2];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1)
    neumaier_merge(s, c, __shfl_down_sync(0xffffffffu, s, d), __shfl_down_sync(0xffffffffu, c, d));
  if (lane == 0) {
    ws[w][0] = s;
    ws[w][1] = c;
  }
  __syncthreads();
  if (w == 0) {
    s = lane < NT / 32 ? ws[lane][0] : 0.0;
    c = lane < NT / 32 ? ws[lane][1] : 0.0;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
      neumaier_merge(s, c, __shfl_down_sync(0xffffffffu, s, d), __shfl_down_sync(0xffffffffu, c, d));
  }
}

// Cells per thread of the partial sums: `most` on a grid that gives every SM
// four CTAs that way, fewer below.  A constant, not the device's SMs: the order of
// the sums, and with it their last bits, depends on the grid size alone.
constexpr int DG_THREADS = 256;
constexpr int DG_CTAS = 148 * 4;
int cells_per_thread(size_t N, int most) {
  const size_t per = (N + (size_t)DG_THREADS * DG_CTAS - 1) / ((size_t)DG_THREADS * DG_CTAS);
  return per < 1 ? 1 : (per > (size_t)most ? most : (int)per);
}
int parts(size_t N, int per) { return (int)((N + (size_t)DG_THREADS * per - 1) / ((size_t)DG_THREADS * per)); }

// ---------------------------------------------------------------- energy
// Per-cell energy of YM_Energy.cu:3-21.  Each CTA sums a contiguous block of cells.
constexpr int EN_PER_THREAD = 16;

__global__ void __launch_bounds__(DG_THREADS)
    energy_partial_kernel(const __grid_constant__ State st, size_t N, int per, double* __restrict__ part) {
  dependency_launch();
  const size_t base = (size_t)blockIdx.x * DG_THREADS * per;
  double s = 0.0, c = 0.0;
#pragma unroll 2
  for (int k = 0; k < per; ++k) {
    const size_t i = base + (size_t)k * DG_THREADS + threadIdx.x;
    if (i >= N) break;
    const double nA = fmax(st.a[FN][i], 1e-10);
    const double nB = fmax(st.b[FN][i], 1e-10);
    const double pxA = st.a[FPX][i], pzA = st.a[FPZ][i], pxB = st.b[FPX][i], pzB = st.b[FPZ][i];
    const double keA = 0.5 * (pxA * pxA + pzA * pzA) / nA;
    const double keB = 0.5 * (pxB * pxB + pzB * pzB) / nB;
    double em2 = 0.0;
    em2 = st.f[EX1][i] * st.f[EX1][i];
    em2 = em2 + st.f[EX2][i] * st.f[EX2][i];
    em2 = em2 + st.f[EX3][i] * st.f[EX3][i];
    em2 = em2 + st.f[EZ1][i] * st.f[EZ1][i];
    em2 = em2 + st.f[EZ2][i] * st.f[EZ2][i];
    em2 = em2 + st.f[EZ3][i] * st.f[EZ3][i];
    em2 = em2 + st.f[BY1][i] * st.f[BY1][i];
    em2 = em2 + st.f[BY2][i] * st.f[BY2][i];
    em2 = em2 + st.f[BY3][i] * st.f[BY3][i];
    const double e = keA + keB + 0.5 * em2;
    neumaier_add(s, c, e);
  }
  neumaier_block<DG_THREADS>(s, c);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = s;
    part[2 * blockIdx.x + 1] = c;
  }
}

// *out = the total; with err, out[1] = the device error word.
constexpr int EF_THREADS = 1024;
__global__ void __launch_bounds__(EF_THREADS)
    energy_final_kernel(double* part, int nparts, double* out, const unsigned* err) {
  dependency_wait();
  double s = 0.0, c = 0.0;
  for (int i = threadIdx.x; i < nparts; i += EF_THREADS) neumaier_merge(s, c, part[2 * i], part[2 * i + 1]);
  neumaier_block<EF_THREADS>(s, c);
  if (threadIdx.x == 0) {
    out[0] = s + c;
    if (err) out[1] = (double)*err;
  }
}

// ------------------------------------------------------------ mode amplitude
// Per column x, F = sum_z (re + i im) e^{-2 pi i k z/nz} and Fc for re - i im
// (ymgpu2d/analysis/remote_timeseries.py:62-77 for re, im = Az2, Az3;
// ymgpu2d/analysis/resolution_convergence.py:83-86 for By2, By3).  A CTA takes
// 32 columns and a range of rows, eight rows at a time; the phase factors of
// 64 rows are formed once and shared by its columns.
constexpr int MA_ROWS = 64;
struct ModeShape {
  int tiles, splits, rows;  // 32-column tiles, row ranges, rows of a range
};
ModeShape mode_shape(int nx, int nz) {
  ModeShape m;
  m.tiles = (nx + 31) / 32;
  int splits = std::max(1, std::min((DG_CTAS + m.tiles - 1) / m.tiles, 32));
  splits = std::min(splits, (nz + MA_ROWS - 1) / MA_ROWS);
  m.rows = (nz + splits - 1) / splits;
  m.splits = (nz + m.rows - 1) / m.rows;
  return m;
}

// part[range][x] = (Re F, Im F, Re Fc, Im Fc) of the range's rows
__global__ void __launch_bounds__(256)
    mode_amp_kernel(const double* __restrict__ re, const double* __restrict__ im, int nx, int nz, int k, int rows,
                    double4* __restrict__ part) {
  dependency_launch();
  __shared__ double2 ph[MA_ROWS];
  __shared__ double sum[8][4][32];
  const int lane = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int x = blockIdx.x * 32 + lane, xr = min(x, nx - 1);
  const int z0 = blockIdx.y * rows, z1 = min(nz, z0 + rows);
  double fr = 0, fi = 0, cr = 0, ci = 0;
  for (int zt = z0; zt < z1; zt += MA_ROWS) {
    const int n = min(MA_ROWS, z1 - zt);
    __syncthreads();
    if (threadIdx.x < n) {
      double sn, cs;
      sincospi(-2.0 * (double)k * (double)(zt + threadIdx.x) / (double)nz, &sn, &cs);
      ph[threadIdx.x] = make_double2(cs, sn);
    }
    __syncthreads();
#pragma unroll 4
    for (int i = ty; i < n; i += 8) {
      const double2 p = ph[i];
      const double a = re[idx2(xr, zt + i, nx)], b = im[idx2(xr, zt + i, nx)];
      // (a + i b)(cs + i sn)
      fr += a * p.x - b * p.y;
      fi += a * p.y + b * p.x;
      // (a - i b)(cs + i sn)
      cr += a * p.x + b * p.y;
      ci += a * p.y - b * p.x;
    }
  }
  sum[ty][0][lane] = fr;
  sum[ty][1][lane] = fi;
  sum[ty][2][lane] = cr;
  sum[ty][3][lane] = ci;
  __syncthreads();
  if (ty < 4) {  // warp v sums component v over the eight rows of threads
    double v = sum[0][ty][lane];
#pragma unroll
    for (int j = 1; j < 8; ++j) v += sum[j][ty][lane];
    if (x < nx) reinterpret_cast<double*>(&part[(size_t)blockIdx.y * nx + x])[ty] = v;
  }
}

// Without a weight: (mean_x |F| / nz, mean_x |Fc| / nz), remote_timeseries.py:72-74.
// With one: (sum_x w[x] |F| / nz, sum_x w[x] |Fc| / nz), the shear-layer
// weighted average of resolution_convergence.py:83-86.
__global__ void __launch_bounds__(1024)
    mode_amp_final_kernel(double4* part, int splits, const double* __restrict__ w, int nx, int nz,
                          double* out) {
  dependency_wait();
  double s0 = 0, s1 = 0;
  for (int x = threadIdx.x; x < nx; x += 1024) {
    double4 f = part[x];
    for (int j = 1; j < splits; ++j) {
      const double4 g = part[(size_t)j * nx + x];
      f.x += g.x;
      f.y += g.y;
      f.z += g.z;
      f.w += g.w;
    }
    const double a = hypot(f.x, f.y), b = hypot(f.z, f.w);
    s0 += w ? w[x] * (a / nz) : a;
    s1 += w ? w[x] * (b / nz) : b;
  }
  __shared__ double r[32][2];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    s0 += __shfl_down_sync(0xffffffffu, s0, d);
    s1 += __shfl_down_sync(0xffffffffu, s1, d);
  }
  if (lane == 0) {
    r[wp][0] = s0;
    r[wp][1] = s1;
  }
  __syncthreads();
  if (wp == 0) {
    s0 = r[lane][0];
    s1 = r[lane][1];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      s0 += __shfl_down_sync(0xffffffffu, s0, d);
      s1 += __shfl_down_sync(0xffffffffu, s1, d);
    }
    if (lane == 0) {
      out[0] = w ? s0 : s0 / nx / nz;
      out[1] = w ? s1 : s1 / nx / nz;
    }
  }
}

// ------------------------------------------------------------------- Gauss
// A CTA has one group of threads per colour, all on the same cells: a thread
// then holds six compensated sums instead of sixteen, so more warps are
// resident to cover the loads (the cells' arrays come through L1 for the second
// and third colour; 1553 -> 1481 us at 4096 x 8192).
constexpr int GA_CELLS = 128, GA_THREADS = 3 * GA_CELLS;
constexpr int GA_PER_THREAD = 16;
constexpr int GA_NV = YMKH_GAUSS_NOUT;
// value slots: [0..2] G, [3..5] div E, [6..8] alpha (Az x Ezc), [9..11] rho,
// [12..14] div E + alpha (Az x Ezc), [15] |Ex1|+|Ex2|+|Ex3|+|Ez1|+|Ez2|+|Ez3|

// part[v][CTA] = (sum, compensation)
__global__ void __launch_bounds__(GA_THREADS, 2)
    gauss_partial_kernel(const __grid_constant__ State st, int nx, int nz, double dx, double dz, double rdx, double rdz,
                         double alpha, int per, double2* __restrict__ part) {
  dependency_launch();
  const int a = threadIdx.x / GA_CELLS, t = threadIdx.x - a * GA_CELLS;  // colour, cell
  const int a1 = a == 2 ? 0 : a + 1, a2 = a == 0 ? 2 : a - 1;
  double s[6], c[6];  // G, div E, alpha (Az x Ezc), rho, lhs of the colour; colour 0: the sum of magnitudes
#pragma unroll
  for (int v = 0; v < 6; ++v) s[v] = c[v] = 0.0;
  const size_t N = (size_t)nx * (size_t)nz;
  const double* const ex = st.f[EX1 + a];
  const double* const ez = st.f[EZ1 + a];
  const double* const ez1 = st.f[EZ1 + a1];
  const double* const ez2 = st.f[EZ1 + a2];
  const double* const az1 = st.f[AZ1 + a1];
  const double* const az2 = st.f[AZ1 + a2];
  const double* const qa = st.a[FQ1 + a];
  const double* const qb = st.b[FQ1 + a];
  // one division per thread: the cell's row and column then advance with it
  size_t i = (size_t)blockIdx.x * GA_CELLS * per + t;
  int z = (int)(i / (size_t)nx), x = (int)(i - (size_t)z * (size_t)nx);
  for (int k = 0; k < per && i < N; ++k) {
    const size_t iw = (x == 0) ? i + (size_t)(nx - 1) : i - 1;
    const size_t is = (z == 0) ? i + (size_t)(nz - 1) * (size_t)nx : i - (size_t)nx;
    const double ezi = ez[i], exi = ex[i];
    const double de = div_rn(exi - ex[iw], dx, rdx) + div_rn(ezi - ez[is], dz, rdz);
    const double p = ez1[i], q = ez2[i];
    const double e1 = 0.5 * (p + ez1[is]), e2 = 0.5 * (q + ez2[is]);
    const double nab = alpha * (az1[i] * e2 - az2[i] * e1);
    const double rho = qa[i] * st.a[FN][i] + qb[i] * st.b[FN][i];
    const double lhs = de + nab, g = lhs - rho;
    neumaier_add(s[0], c[0], g * g);
    neumaier_add(s[1], c[1], de * de);
    neumaier_add(s[2], c[2], nab * nab);
    neumaier_add(s[3], c[3], rho * rho);
    neumaier_add(s[4], c[4], lhs * lhs);
    if (a == 0) {  // here a1 and a2 are colours 2 and 3
      double alle = fabs(exi) + fabs(st.f[EX2][i]);
      alle = alle + fabs(st.f[EX3][i]);
      alle = alle + fabs(ezi);
      alle = alle + fabs(p);
      alle = alle + fabs(q);
      neumaier_add(s[5], c[5], alle * alle);
    }
    i += GA_CELLS;
    for (x += GA_CELLS; x >= nx; x -= nx) ++z;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int v = 0; v < 6; ++v)
      neumaier_merge(s[v], c[v], __shfl_down_sync(0xffffffffu, s[v], off), __shfl_down_sync(0xffffffffu, c[v], off));
  }
  __shared__ double2 ws[GA_THREADS / 32][6];
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int v = 0; v < 6; ++v) ws[threadIdx.x >> 5][v] = make_double2(s[v], c[v]);
  __syncthreads();
  if (threadIdx.x < GA_NV) {
    const int slot = threadIdx.x, v = slot == 15 ? 5 : slot / 3, w0 = (slot == 15 ? 0 : slot % 3) * (GA_CELLS / 32);
    double sv = 0.0, cv = 0.0;
    for (int w = 0; w < GA_CELLS / 32; ++w) neumaier_merge(sv, cv, ws[w0 + w][v].x, ws[w0 + w][v].y);
    part[(size_t)slot * gridDim.x + blockIdx.x] = make_double2(sv, cv);
  }
}

// One CTA per value: the CTA partials, then the root-mean-square over the N cells.
__global__ void __launch_bounds__(DG_THREADS)
    gauss_final_kernel(double2* part, int nparts, double n_cells, double* out) {
  dependency_wait();
  double s = 0.0, c = 0.0;
  for (int b = threadIdx.x; b < nparts; b += DG_THREADS) {
    const double2 p = part[(size_t)blockIdx.x * nparts + b];
    neumaier_merge(s, c, p.x, p.y);
  }
  neumaier_block<DG_THREADS>(s, c);
  if (threadIdx.x == 0) out[blockIdx.x] = sqrt((s + c) / n_cells);
}

}  // namespace

int energy_nparts(size_t N) { return parts(N, cells_per_thread(N, EN_PER_THREAD)); }

cudaError_t launch_energy(const State& st, size_t N, double* part, double* out, const unsigned* err, cudaStream_t s) {
  const int np = energy_nparts(N);
  energy_partial_kernel<<<np, DG_THREADS, 0, s>>>(st, N, cells_per_thread(N, EN_PER_THREAD), part);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return launch_dependent(energy_final_kernel, dim3(1), dim3(EF_THREADS), s, part, np, out, err);
}

size_t mode_amp_scratch(int nx, int nz) { return (size_t)4 * nx * mode_shape(nx, nz).splits; }

cudaError_t launch_mode_amp(const double* re, const double* im, int nx, int nz, int k, double* scratch,
                            const double* weight, double* out, cudaStream_t s) {
  const ModeShape m = mode_shape(nx, nz);
  double4* part = reinterpret_cast<double4*>(scratch);
  mode_amp_kernel<<<dim3(m.tiles, m.splits), 256, 0, s>>>(re, im, nx, nz, k, m.rows, part);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return launch_dependent(mode_amp_final_kernel, dim3(1), dim3(1024), s, part, m.splits, weight, nx, nz, out);
}

// Cells per thread of the Gauss sums, as cells_per_thread with its own CTAs.
static int gauss_per(size_t N) {
  const size_t per = (N + (size_t)GA_CELLS * DG_CTAS - 1) / ((size_t)GA_CELLS * DG_CTAS);
  return per < 1 ? 1 : (per > (size_t)GA_PER_THREAD ? GA_PER_THREAD : (int)per);
}
int gauss_nparts(size_t N) {
  const size_t per = (size_t)GA_CELLS * gauss_per(N);
  return (int)((N + per - 1) / per);
}

cudaError_t launch_gauss(const State& st, int nx, int nz, double dx, double dz, double alpha, double* part,
                         double* out, cudaStream_t s) {
  const size_t N = (size_t)nx * (size_t)nz;
  const int np = gauss_nparts(N);
  double2* p2 = reinterpret_cast<double2*>(part);
  gauss_partial_kernel<<<np, GA_THREADS, 0, s>>>(st, nx, nz, dx, dz, 1.0 / dx, 1.0 / dz, alpha, gauss_per(N), p2);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return launch_dependent(gauss_final_kernel, dim3(GA_NV), dim3(DG_THREADS), s, p2, np, (double)N, out);
}

}  // namespace ymkh
