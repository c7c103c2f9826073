// ymkh_column.cu — post-Maxwell stages that act along z or pointwise:
// sponge (YM_Physics.cu:161-182), xi_cut (:192-210), z-mean removal
// (:272-327), the DFT kz band filters (:349-584), z-hyperdiffusion (:228-259)
// and the colour-1 zeroing (ymgpu2d/main_ym.cu:443-447).  All update the new
// state buffer in place; none reads a neighbour another CTA writes.
//
// The band filter is written as two dense FP64 contractions per band, over
// all filtered arrays at once (21 arrays: the 15 EM/colour arrays of
// YM_Physics.cu:373-379 and n, px, pz of both beams):
//   C[j, x] = inv2 * sum_z W[z, j] G[z, x]          (coefficients A_m, B_m)
//   G[z, x] = G[z, x] - sum_j W[z, j] C[j, x]       (subtract the band)
// with W[z, 2i] = cosf(phase), W[z, 2i+1] = sinf(phase) the reference's FP32
// twiddles (YM_Physics.cu:387-388) widened to double and inv2 = 2.0f/nz
// (:425), summed in the reference's order (its warp-shuffle tree), so the
// filtered step is bit-identical to the reference's -fmad=false build.

#include "ymkh_common.cuh"

#include <mutex>

namespace ymkh {

// ---------------------------------------------------------------- twiddles
// W[z * ldw + 2*(m-lo) + {0,1}] for m in [lo, hi].
__global__ void twiddle_kernel(double* W, int nz, int lo, int hi, int ldw) {
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  const int m = lo + blockIdx.y;
  if (z >= nz || m > hi) return;
  float phase = 2.0f * (float)M_PI * m * z / (float)nz;
  float cz = cosf(phase), sz = sinf(phase);
  W[(size_t)z * ldw + 2 * (m - lo)] = (double)cz;
  W[(size_t)z * ldw + 2 * (m - lo) + 1] = (double)sz;
}

__global__ void twiddle_f32_kernel(float* c, float* s, int nz, int lo, int hi) {
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  const int m = lo + blockIdx.y;
  if (z >= nz || m > hi) return;
  float phase = 2.0f * (float)M_PI * m * z / (float)nz;
  c[(size_t)(m - lo) * nz + z] = cosf(phase);
  s[(size_t)(m - lo) * nz + z] = sinf(phase);
}

cudaError_t launch_twiddles(double* W, int nz, int lo, int hi, int ldw, cudaStream_t s) {
  dim3 grid((nz + 127) / 128, hi - lo + 1);
  twiddle_kernel<<<grid, 128, 0, s>>>(W, nz, lo, hi, ldw);
  return cudaGetLastError();
}
cudaError_t launch_twiddles_f32(float* c, float* sn, int nz, int lo, int hi, cudaStream_t s) {
  dim3 grid((nz + 127) / 128, hi - lo + 1);
  twiddle_f32_kernel<<<grid, 128, 0, s>>>(c, sn, nz, lo, hi);
  return cudaGetLastError();
}


// ---------------------------------------------------------- sponge / xicut
__global__ void sponge_xicut_kernel(const __grid_constant__ ArrayList a12, StepParams p, int cut) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  const int z = blockIdx.y;
  if (x >= p.nx) return;
  const double xc = (p.nx * p.dx) * 0.5;
  const double xi = fabs((x * p.dx - xc) / p.epsilon);
  const size_t i = idx2(x, z, p.nx);
  if (cut) {
    if (xi <= p.xi_cut) return;
#pragma unroll
    for (int k = 0; k < 12; ++k) a12.p[k][i] = 0.0;
  } else {
    if (xi <= p.xi_sponge) return;
    const double sig = p.sigma_sponge * (xi - p.xi_sponge);
    const double dec = exp(-sig * p.dt);
#pragma unroll
    for (int k = 0; k < 12; ++k) a12.p[k][i] *= dec;
  }
}

cudaError_t launch_sponge_xicut(const ArrayList& a12, const StepParams& p, int cut, cudaStream_t s) {
  dim3 grid((p.nx + 127) / 128, p.nz);
  sponge_xicut_kernel<<<grid, 128, 0, s>>>(a12, p, cut);
  return cudaGetLastError();
}

// -------------------------------------------------------------- z-mean
// Arrays [0, nmean) lose their z-mean; arrays [nmean, gridDim.y) are set to
// zero (the colour-1 fields, which the step zeroes once the z-mean is done:
// ymgpu2d/main_ym.cu:443-447; no stage in between reads or writes them).
// One CTA per (4 columns, array).  The column sum uses the reference's
// halving tree (YM_Physics.cu:301-308) so the mean is bit-identical.
constexpr int ZM_CX = 4;
constexpr size_t kColumnSmemMax = 200 * 1024;  // shared memory of the staged-column kernels
__global__ void zmean_kernel(const __grid_constant__ ArrayList arrs, int nx, int nz, int nmean,
                             double* __restrict__ means) {
  extern __shared__ double sm[];  // [nz][ZM_CX]
  const int x0 = blockIdx.x * ZM_CX;
  double* g = arrs.p[blockIdx.y];
  if ((int)blockIdx.y >= nmean) {
    for (int i = threadIdx.x; i < nz * ZM_CX; i += blockDim.x) {
      const int z = i / ZM_CX, c = i - z * ZM_CX;
      if (x0 + c < nx) g[idx2(x0 + c, z, nx)] = 0.0;
    }
    return;
  }
  for (int i = threadIdx.x; i < nz * ZM_CX; i += blockDim.x) {
    const int z = i / ZM_CX, c = i - z * ZM_CX;
    sm[i] = (x0 + c < nx) ? g[idx2(x0 + c, z, nx)] : 0.0;
  }
  __syncthreads();
  for (int st = nz >> 1; st > 0; st >>= 1) {
    for (int i = threadIdx.x; i < st * ZM_CX; i += blockDim.x) sm[i] += sm[i + st * ZM_CX];
    __syncthreads();
  }
  const double inv = 1.0 / (double)nz;
  if (means) {
    if (threadIdx.x < ZM_CX && x0 + threadIdx.x < nx) means[(size_t)blockIdx.y * nx + x0 + threadIdx.x] = sm[threadIdx.x] * inv;
    return;
  }
  for (int i = threadIdx.x; i < nz * ZM_CX; i += blockDim.x) {
    const int z = i / ZM_CX, c = i - z * ZM_CX;
    if (x0 + c < nx) {
      const size_t gi = idx2(x0 + c, z, nx);
      g[gi] -= sm[c] * inv;
    }
  }
}

// Power-of-two NZ = 32 M: one CTA per (32 columns, array), warp l holding the
// rows z = l + 32 j of its lane's column, so every load is one coalesced row
// segment.  The halving tree pairs z with z + NZ/2, then z + NZ/4, ...: its
// levels down to stride 32 stay inside a residue class z mod 32, where they
// form the same halving tree over j; each thread sums its class in that order
// with a pairwise binary counter over the leaves in bit-reversed j order
// (T(y) = T(y_even) + T(y_odd)), and the last five levels (strides 16 .. 1)
// are a shuffle tree over the 32 class sums.  The sum is therefore the
// halving tree's, bit for bit; the columns are then re-read (mostly from L2)
// and the mean subtracted.
template <int LOGM>
__global__ void __launch_bounds__(1024) zmean_p2_kernel(const __grid_constant__ ArrayList arrs, int nx, int nmean,
                                                        double* __restrict__ means) {
  constexpr int M = 1 << LOGM;
  __shared__ double part[32][33];
  __shared__ double mean[32];
  const int lane = threadIdx.x & 31, l = threadIdx.x >> 5;
  const int x = blockIdx.x * 32 + lane;
  double* g = arrs.p[blockIdx.y];
  const bool in = x < nx;
  if ((int)blockIdx.y >= nmean) {  // an array the step zeroes (zmean_kernel)
    if (in)
#pragma unroll 8
      for (int j = 0; j < M; ++j) g[(size_t)(l + 32 * j) * nx + x] = 0.0;
    return;
  }
  double st[LOGM + 1];
#pragma unroll
  for (int jj = 0; jj < M; ++jj) {
    int j = 0;
#pragma unroll
    for (int b = 0; b < LOGM; ++b) j |= ((jj >> b) & 1) << (LOGM - 1 - b);
    double carry = in ? g[(size_t)(l + 32 * j) * nx + x] : 0.0;
    int k = 0;
#pragma unroll
    for (int b = 0; b < LOGM; ++b) {
      if (((jj >> b) & 1) == 0) break;
      carry = st[b] + carry;
      k = b + 1;
    }
    st[k] = carry;
  }
  part[l][lane] = st[LOGM];
  __syncthreads();
  {
    double v = part[lane][l];  // warp l: column l of the tile, lane = residue class
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, d);
    if (lane == 0) mean[l] = v * (1.0 / (double)(32 * M));
  }
  __syncthreads();
  if (means) {
    if (in && l == 0) means[(size_t)blockIdx.y * nx + x] = mean[lane];
    return;
  }
  if (in) {
    const double mu = mean[lane];
#pragma unroll 8
    for (int j = 0; j < M; ++j) {
      const size_t gi = (size_t)(l + 32 * j) * nx + x;
      g[gi] -= mu;
    }
  }
}

cudaError_t launch_zmean(const ArrayList& arrs, int nmean, int nzero, int nx, int nz, double* means, cudaStream_t s) {
  const int narr = nmean + nzero;
  const dim3 g32((nx + 31) / 32, narr);
  switch (nz) {
    case 128: zmean_p2_kernel<2><<<g32, 1024, 0, s>>>(arrs, nx, nmean, means); return cudaGetLastError();
    case 256: zmean_p2_kernel<3><<<g32, 1024, 0, s>>>(arrs, nx, nmean, means); return cudaGetLastError();
    case 512: zmean_p2_kernel<4><<<g32, 1024, 0, s>>>(arrs, nx, nmean, means); return cudaGetLastError();
    case 1024: zmean_p2_kernel<5><<<g32, 1024, 0, s>>>(arrs, nx, nmean, means); return cudaGetLastError();
    case 2048: zmean_p2_kernel<6><<<g32, 1024, 0, s>>>(arrs, nx, nmean, means); return cudaGetLastError();
    case 4096: zmean_p2_kernel<7><<<g32, 1024, 0, s>>>(arrs, nx, nmean, means); return cudaGetLastError();
    case 8192: zmean_p2_kernel<8><<<g32, 1024, 0, s>>>(arrs, nx, nmean, means); return cudaGetLastError();
    default: break;
  }
  const size_t smem = (size_t)nz * ZM_CX * sizeof(double);
  if (smem > kColumnSmemMax) return cudaErrorInvalidValue;  // NZ > 6400 without a coalesced form
  dim3 grid((nx + ZM_CX - 1) / ZM_CX, narr);
  zmean_kernel<<<grid, 256, smem, s>>>(arrs, nx, nz, nmean, means);
  return cudaGetLastError();
}

// ---------------------------------------------------------- hyperdiffusion
// Race-free form of YM_Physics.cu:228-259: every stencil reads the values
// from before the update (the reference's in-place version reads a mix).
constexpr int HD_CX = 4;
__global__ void hyperdiff_kernel(const __grid_constant__ ArrayList a12, int nx, int nz, double mu) {
  extern __shared__ double sm[];  // [nz][HD_CX]
  const int x0 = blockIdx.x * HD_CX;
  double* g = a12.p[blockIdx.y];
  for (int i = threadIdx.x; i < nz * HD_CX; i += blockDim.x) {
    const int z = i / HD_CX, c = i - z * HD_CX;
    sm[i] = (x0 + c < nx) ? g[idx2(x0 + c, z, nx)] : 0.0;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nz * HD_CX; i += blockDim.x) {
    const int z = i / HD_CX, c = i - z * HD_CX;
    if (x0 + c >= nx) continue;
    const int zm1 = (z == 0) ? nz - 1 : z - 1;
    const int zm2 = (z <= 1) ? z - 2 + nz : z - 2;
    const int zp1 = (z == nz - 1) ? 0 : z + 1;
    const int zp2 = (z >= nz - 2) ? z + 2 - nz : z + 2;
    const double d4 = sm[zm2 * HD_CX + c] - 4.0 * sm[zm1 * HD_CX + c] + 6.0 * sm[i] - 4.0 * sm[zp1 * HD_CX + c] +
                      sm[zp2 * HD_CX + c];
    g[idx2(x0 + c, z, nx)] = sm[i] - mu * d4;
  }
}

// NZ a multiple of 32 (at least 64): one 1024-thread CTA per (32 columns,
// array); lane c holds column c and warp w the rows [w L, (w+1) L), L = NZ/32,
// so every access is a coalesced 256-byte row segment.  Each warp first reads
// the two rows on either side of its segment (periodic in z), then the CTA
// synchronises, and each warp updates its own rows in place from a five-row
// window of values read before any write: every stencil sees the values from
// before the update, as hyperdiff_kernel's shared copy gives, with the same
// arithmetic, so the result is the same bit for bit.
__global__ void __launch_bounds__(1024) hyperdiff_seg_kernel(const __grid_constant__ ArrayList a12, int nx, int nz,
                                                             double mu) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int x = blockIdx.x * 32 + lane;
  const bool in = x < nx;
  double* g = a12.p[blockIdx.y];
  const int L = nz >> 5, z0 = w * L;
  auto at = [&](int z) -> double {
    z = z < 0 ? z + nz : (z >= nz ? z - nz : z);
    return in ? g[(size_t)z * nx + x] : 0.0;
  };
  const double h0 = at(z0 - 2), h1 = at(z0 - 1);        // rows below the segment
  const double t0 = at(z0 + L), t1 = at(z0 + L + 1);    // rows above it
  __syncthreads();  // every warp holds its neighbours' rows before any write
  double w0 = h0, w1 = h1, w2 = at(z0), w3 = at(z0 + 1);
#pragma unroll 4
  for (int k = 0; k < L; ++k) {
    const double w4 = (k + 2 < L) ? at(z0 + k + 2) : (k + 2 == L ? t0 : t1);
    const double d4 = w0 - 4.0 * w1 + 6.0 * w2 - 4.0 * w3 + w4;
    if (in) g[(size_t)(z0 + k) * nx + x] = w2 - mu * d4;
    w0 = w1;
    w1 = w2;
    w2 = w3;
    w3 = w4;
  }
}

cudaError_t launch_hyperdiff(const ArrayList& a12, int nx, int nz, double mu, cudaStream_t s) {
  if (nz % 32 == 0 && nz >= 64) {
    hyperdiff_seg_kernel<<<dim3((nx + 31) / 32, 12), 1024, 0, s>>>(a12, nx, nz, mu);
    return cudaGetLastError();
  }
  const size_t smem = (size_t)nz * HD_CX * sizeof(double);
  if (smem > kColumnSmemMax) return cudaErrorInvalidValue;  // NZ > 6400 and not a multiple of 32
  dim3 grid((nx + HD_CX - 1) / HD_CX, 12);
  hyperdiff_kernel<<<grid, 256, smem, s>>>(a12, nx, nz, mu);
  return cudaGetLastError();
}

// The staged-column kernels (zmean_kernel, hyperdiff_kernel) keep a block of
// whole columns in shared memory.  The dynamic shared-memory limit is a
// property of the kernel, shared by every run in the process: it only ever
// grows (to the largest NZ seen), so a run with a smaller NZ never lowers it
// under a larger resident run.  Above kColumnSmemMax (NZ > 6400) nothing is
// set: such runs use the coalesced kernels, and a stage that would need a
// staged kernel there fails at its launch.
size_t column_smem(int nz) { return (size_t)nz * (ZM_CX > HD_CX ? ZM_CX : HD_CX) * sizeof(double); }

cudaError_t prepare_column(int nz) {
  static std::mutex mu;
  static size_t granted[64];  // per device
  const size_t smem = column_smem(nz);
  if (smem > kColumnSmemMax) return cudaSuccess;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(mu);
  if (smem > 48 * 1024 && smem > granted[dev]) {
    cudaError_t e = cudaFuncSetAttribute(zmean_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(hyperdiff_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    granted[dev] = smem;
  }
  return cudaSuccess;
}

// ------------------------------------------------------------- band filter
// The FP64 band filter in the reference's own summation order, so that a
// filtered step is bit-identical to the reference's kernels built with
// -fmad=false (YM_Physics.cu:349-455 for the 15 EM/colour arrays, :461-584
// for pz, px and n).  Two dense contractions per band and array, each
// blocked over (mode, column) or (z, column) tiles:
//
//   coefficients  C[j][x] = inv2 * S_j(x),
//     S_j(x) = sum over warps w, in order from 0.0, of the warp's lane-0
//     shuffle tree of the 32 products v[32w + i][x] * tw[j][32w + i]
//     (YM_Physics.cu:396-426);
//   apply         v[z][x] -= delta, delta = sum over modes m in order from
//     0.0 of (A_m * cos_m(z) + B_m * sin_m(z)) (YM_Physics.cu:429-450).
//
// Products and sums are rounded separately (no fused multiply-add), as the
// reference's -fmad=false build rounds them.

// Bound by the FP64 pipe: 4 operations per row, coefficient and column, none of
// them fused, so 2.77 ms at 1024 x 2048 with 18 arrays and modes 342..512.
// Both kernels keep the operand that belongs to a thread's columns in
// registers (32 rows x 2 columns of the array; 16 x 2 running sums) and read
// the twiddles, which all lanes share, as one 16-byte (cos, sin) load.  That
// load takes two shared-memory cycles: with one column a thread it could only
// feed four FP64 instructions and set the pace (81% of the load pipe, FP64
// 70%); with two, eight.  Measured there, with 21 arrays and under the profiler:
// 2.18 + 2.11 ms at 78% of the FP64 pipe each, against 2.70 + 2.68 ms for the two
// kernels that loaded both operands of a 2 x 4 and a 4 x 4 block from shared
// memory.  Staging the coefficients in shared memory too cost the apply kernel a
// CTA per SM.
//
// The reference's warp reduction (shfl_down by 16, 8, 4, 2, 1) leaves lane 0
// with root = T4(0) + T4(1), T4(i) = T3(i) + T3(i+2), T3(i) = T2(i) + T2(i+4),
// T2(i) = T1(i) + T1(i+8), T1(i) = a_i + a_{i+16} (every sum is commutative,
// so only the grouping matters).  Visited in bit-reversed order (0, 8, 4,
// 12, 2, ...), the sixteen T1 nodes form a balanced pairwise tree over
// consecutive visits, which a stack of four partial sums evaluates.
constexpr int BD_TX = 128;    // columns per CTA
constexpr int BD_CH = 32;     // z rows in registers: a warp of the reference
constexpr int BC_NC = 2, BC_NT = BD_TX / BC_NC;  // coefficients: columns threadIdx.x + n * BC_NT per thread
constexpr int BC_BM = 16;     // most modes of a coefficient CTA
constexpr int BA_BM = 16;     // modes per twiddle tile of the apply kernel

// Stages the twiddles of rows [z0, z0 + 32) and modes [m0, m0 + bm) as
// tw[z][bm] (cos, sin) pairs, zero past the last row or mode.
template <int NT>
__device__ __forceinline__ void stage_twiddles(double2* tw, const double* __restrict__ W, int ldw, int z0, int m0, int bm,
                                               int nz, int M) {
  for (int i = threadIdx.x; i < BD_CH * bm; i += NT) {
    const int z = i / bm, m = i - z * bm;
    if (z0 + z < nz && m0 + m < M) cp_async16(&tw[i], W + (size_t)(z0 + z) * ldw + 2 * (m0 + m));
    else tw[i] = make_double2(0.0, 0.0);
  }
  cp_async_commit();
}

// C[2m + {0, 1}][x] for modes [m0, m0 + bm) of one array: the running sums of
// the block's modes stay in shared memory, each thread's own.  NC columns a
// thread: one where 64 columns or fewer are left, so that no thread sums a column
// that is not there (2048 x 40, modes 683..1024: 722 us against 1182 with two;
// 1024 x 40 225 against 347).
template <int NC, bool AHEAD>
__device__ __forceinline__ void band_coef(const ArrayList& arrs, const double* __restrict__ W, int ldw, int M, int bm,
                                          double* __restrict__ C, int xb, int nx, int nz, double inv2,
                                          double2* band_smem) {
  constexpr int NT = BC_NT, TX = NC * NT;
  double2* const tw = band_smem;                                              // [2][BD_CH][bm]
  double2* const sum = band_smem + (size_t)2 * BD_CH * bm + threadIdx.x;      // [bm][TX]
  const int m0 = blockIdx.x * bm, x0 = xb + threadIdx.x, k = blockIdx.z;
  const double* g = arrs.p[k] + x0;
  bool in[NC];
#pragma unroll
  for (int n = 0; n < NC; ++n) in[n] = x0 + n * NT < nx;
  const int nm = min(bm, M - m0), nch = (nz + BD_CH - 1) / BD_CH;
  for (int m = 0; m < nm; ++m)
#pragma unroll
    for (int n = 0; n < NC; ++n) sum[m * TX + n * NT] = make_double2(0.0, 0.0);
  stage_twiddles<NT>(tw, W, ldw, 0, m0, bm, nz, M);
  auto rows = [&](double(&f)[NC][BD_CH], int ch) {
#pragma unroll
    for (int i = 0; i < BD_CH; ++i)
#pragma unroll
      for (int n = 0; n < NC; ++n) {
        const int z = ch * BD_CH + i;
        f[n][i] = (in[n] && z < nz) ? g[(size_t)z * nx + n * NT] : 0.0;
      }
  };
  double next[NC][BD_CH];
  if (AHEAD) rows(next, 0);
  for (int ch = 0; ch < nch; ++ch) {
    double f[NC][BD_CH];
    if (AHEAD) {
#pragma unroll
      for (int i = 0; i < BD_CH; ++i)
#pragma unroll
        for (int n = 0; n < NC; ++n) f[n][i] = next[n][i];
      if (ch + 1 < nch) rows(next, ch + 1);
    } else {
      rows(f, ch);
    }
    cp_async_wait<0>();
    __syncthreads();  // this chunk's twiddles are there, the other buffer is free
    if (ch + 1 < nch) stage_twiddles<NT>(tw + ((ch + 1) & 1) * BD_CH * bm, W, ldw, (ch + 1) * BD_CH, m0, bm, nz, M);
    const double2* t = tw + (ch & 1) * BD_CH * bm;
    for (int m = 0; m < nm; ++m, ++t) {
      double sc[NC][4], ss[NC][4];  // pending tree nodes of heights 1..4 (T2..T4 partial sums)
#pragma unroll
      for (int kk = 0; kk < 16; ++kk) {
        const int i = bitrev4(kk);
        const double2 w0 = t[i * bm], w1 = t[(i + 16) * bm];
#pragma unroll
        for (int n = 0; n < NC; ++n) {
          double c = f[n][i] * w0.x + f[n][i + 16] * w1.x;  // T1(i); products rounded (YM_Physics.cu:394)
          double s = f[n][i] * w0.y + f[n][i + 16] * w1.y;
          int lvl = 0;  // merge with the pending nodes: one level per trailing one bit of kk
#pragma unroll
          for (int L = 0; L < 4; ++L) {
            if (((kk >> L) & 1) && lvl == L) {
              c = sc[n][L] + c;
              s = ss[n][L] + s;
              ++lvl;
            }
          }
          if (lvl < 4) {
            sc[n][lvl] = c;
            ss[n][lvl] = s;
          } else {  // warp sums added in warp order from 0.0
            double2 S = sum[m * TX + n * NT];
            S.x = S.x + c;
            S.y = S.y + s;
            sum[m * TX + n * NT] = S;
          }
        }
      }
    }
  }
  double* Ck = C + (size_t)k * 2 * M * nx + (size_t)2 * m0 * nx + x0;
#pragma unroll
  for (int n = 0; n < NC; ++n)
    if (in[n])
      for (int m = 0; m < nm; ++m) {
        const double2 S = sum[m * TX + n * NT];
        Ck[(size_t)(2 * m) * nx + n * NT] = S.x * inv2;
        Ck[(size_t)(2 * m + 1) * nx + n * NT] = S.y * inv2;
      }
}

__global__ void __launch_bounds__(BC_NT)
    band_coef_kernel(const __grid_constant__ ArrayList arrs, const double* __restrict__ W, int ldw, int M, int bm,
                     double* __restrict__ C, int nx, int nz, double inv2) {
  extern __shared__ __align__(16) double2 band_smem[];
  const int xb = blockIdx.y * BD_TX;
  if (nx - xb <= BC_NT) band_coef<1, false>(arrs, W, ldw, M, bm, C, xb, nx, nz, inv2, band_smem);
  else band_coef<BC_NC, false>(arrs, W, ldw, M, bm, C, xb, nx, nz, inv2, band_smem);
}

// Blocks of 64 columns, each chunk's rows read while the one before is summed.
__global__ void __launch_bounds__(BC_NT)
    band_coef_ahead_kernel(const __grid_constant__ ArrayList arrs, const double* __restrict__ W, int ldw, int M, int bm,
                           double* __restrict__ C, int nx, int nz, double inv2) {
  extern __shared__ __align__(16) double2 band_smem[];
  band_coef<1, true>(arrs, W, ldw, M, bm, C, blockIdx.y * BC_NT, nx, nz, inv2, band_smem);
}

// v[z][x] -= sum over the band's modes in order of (A_m cos_m(z) + B_m sin_m(z)),
// 32 rows and 128 columns per CTA, 16 x 2 of them in a thread's registers: a
// twiddle pair then serves eight FP64 instructions.
constexpr int BA_NT = 128, BA_RZ = 16;
template <int BA_NC>  // columns per thread, as in band_coef
__device__ __forceinline__ void band_apply(const ArrayList& arrs, const double* __restrict__ W, int ldw, int M,
                                           const double* __restrict__ C, int nx, int nz, double2 (*tw)[BD_CH * BA_BM]) {
  const int zh = (threadIdx.x >> 6) * BA_RZ;
  const int z0 = blockIdx.x * BD_CH, x0 = blockIdx.y * BD_TX + (threadIdx.x & 63), k = blockIdx.z;
  const double* c = C + (size_t)k * 2 * M * nx;
  int xc[BA_NC];  // the columns whose coefficients are read
  // Coefficients are read two modes ahead: they come from L2, and a mode takes
  // a warp about as long as that.
  double d[BA_NC][BA_RZ], nxt[2][2][BA_NC];
  auto read = [&](int m) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const double* r = c + (size_t)2 * min(m + u, M - 1) * nx;
#pragma unroll
      for (int n = 0; n < BA_NC; ++n) {
        nxt[u][0][n] = r[xc[n]];
        nxt[u][1][n] = r[nx + xc[n]];
      }
    }
  };
  stage_twiddles<BA_NT>(tw[0], W, ldw, z0, 0, BA_BM, nz, M);
#pragma unroll
  for (int n = 0; n < BA_NC; ++n) {
    xc[n] = min(x0 + n * 64, nx - 1);
#pragma unroll
    for (int i = 0; i < BA_RZ; ++i) d[n][i] = 0.0;
  }
  read(0);
  const int nblk = (M + BA_BM - 1) / BA_BM;
  for (int b = 0; b < nblk; ++b) {
    cp_async_wait<0>();
    __syncthreads();
    if (b + 1 < nblk) stage_twiddles<BA_NT>(tw[(b + 1) & 1], W, ldw, z0, (b + 1) * BA_BM, BA_BM, nz, M);
    const double2* t = tw[b & 1] + zh * BA_BM;
    const int nm = min(BA_BM, M - b * BA_BM);
    for (int m = 0; m < nm; m += 2) {
      double cur[2][2][BA_NC];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int n = 0; n < BA_NC; ++n) {
          cur[u][0][n] = nxt[u][0][n];
          cur[u][1][n] = nxt[u][1][n];
        }
      read(b * BA_BM + m + 2);
#pragma unroll
      for (int u = 0; u < 2; ++u, ++t) {
        if (m + u >= nm) break;
#pragma unroll
        for (int i = 0; i < BA_RZ; ++i) {
          const double2 w = t[i * BA_BM];
#pragma unroll
          for (int n = 0; n < BA_NC; ++n) d[n][i] = d[n][i] + (cur[u][0][n] * w.x + cur[u][1][n] * w.y);  // YM_Physics.cu:433
        }
      }
    }
  }
  // A column's rows are all read before the first is written: the compiler may
  // not move a read past a write whose row it cannot tell apart, and one after
  // the other they took longer than a band of few modes (filter at 1024 x 768, one
  // mode: 108 us against 180, 13 modes 207 against 272).
  double* g = arrs.p[k] + x0;
#pragma unroll
  for (int n = 0; n < BA_NC; ++n)
    if (x0 + n * 64 < nx) {
      double v[BA_RZ];
#pragma unroll
      for (int i = 0; i < BA_RZ; ++i) v[i] = z0 + zh + i < nz ? g[(size_t)(z0 + zh + i) * nx + n * 64] : 0.0;
#pragma unroll
      for (int i = 0; i < BA_RZ; ++i)
        if (z0 + zh + i < nz) g[(size_t)(z0 + zh + i) * nx + n * 64] = v[i] - d[n][i];
    }
}

__global__ void __launch_bounds__(BA_NT)
    band_apply_kernel(const __grid_constant__ ArrayList arrs, const double* __restrict__ W, int ldw, int M,
                      const double* __restrict__ C, int nx, int nz) {
  __shared__ __align__(16) double2 tw[2][BD_CH * BA_BM];
  if (nx - (int)blockIdx.y * BD_TX <= 64) band_apply<1>(arrs, W, ldw, M, C, nx, nz, tw);
  else band_apply<2>(arrs, W, ldw, M, C, nx, nz, tw);
}

size_t band_coef_smem(int bm, int cols) { return sizeof(double2) * (size_t)bm * (2 * BD_CH + cols); }

cudaError_t launch_band(const ArrayList& arrs, int narr, const double* W, int ldw, int J, double* C, int nx, int nz,
                        double inv2, cudaStream_t s) {
  const int M = J / 2, nxb = (nx + BD_TX - 1) / BD_TX, nxc = (nx + BC_NT - 1) / BC_NT;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long slots = sms * 4;
  // Modes per CTA of the two-column form.  Four CTAs fit an SM and all take
  // equally long, so while they fill the SMs only a few times, the number whose
  // turns come to the fewest modes (us at 256 x 512, modes 86..128: 99 against 107
  // with four and 105 with sixteen; 512 x 512, modes 171..256 314 against 347 and
  // 342); beyond, the most that fit, which read the array least (1024 x 2048 3.65
  // ms against 3.91 with four).
  auto ctas = [&](int m, int blocks) { return (long long)((M + m - 1) / m) * blocks * narr; };
  auto turns = [&](int m) { return (ctas(m, nxb) + slots - 1) / slots; };
  int bm = std::min(BC_BM, M);
  if (turns(bm) <= 4)
    for (int m = bm - 1; m >= 4; --m)
      if (turns(m) * m < turns(bm) * bm) bm = m;
  // Few modes on a grid of few columns leave that form waiting for each chunk's
  // rows: there the one-column form that reads a chunk ahead, with the fewest
  // modes a CTA that keep four CTAs an SM (more of them read the array more often
  // than they save).  It is taken when the busiest SM then has less to do: its
  // column and mode costs 1.15 times as much, but the two-column form waits for
  // its rows about as long as it sums 150 (filter us, two- against one-column
  // form: 1024 x 128 13 modes 91 / 66, 8192 x 128 24 modes 813 / 585, 8192 x 448
  // 13 modes 1328 / 1005, 8192 x 192 32 modes 1230 / 948, 1024 x 192 40 modes
  // 183 / 158, but 1024 x 256 24 modes 129 / 137, 1024 x 768 13 modes 207 / 213,
  // 1024 x 512 64 modes 462 / 512, one mode 4096 x 40 136 / 150).
  int ba = 1;
  while (ba < bm && ctas(ba, nxc) > slots) ++ba;
  auto busiest = [&](int m, int blocks, int cols) { return (ctas(m, blocks) + sms - 1) / sms * m * cols; };
  const long long two = busiest(bm, nxb, nx <= BC_NT ? BC_NT : BD_TX), one = busiest(ba, nxc, BC_NT);
  if (ctas(ba, nxc) <= slots && one * 23 < (two + (nx > BC_NT ? 150 : 0)) * 20)
    band_coef_ahead_kernel<<<dim3((M + ba - 1) / ba, nxc, narr), BC_NT, band_coef_smem(ba, BC_NT), s>>>(arrs, W, ldw, M, ba,
                                                                                                     C, nx, nz, inv2);
  else
    band_coef_kernel<<<dim3((M + bm - 1) / bm, nxb, narr), BC_NT, band_coef_smem(bm, BD_TX), s>>>(arrs, W, ldw, M, bm, C, nx,
                                                                                               nz, inv2);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  band_apply_kernel<<<dim3((nz + BD_CH - 1) / BD_CH, nxb, narr), BA_NT, 0, s>>>(arrs, W, ldw, M, C, nx, nz);
  return cudaGetLastError();
}

}  // namespace ymkh
