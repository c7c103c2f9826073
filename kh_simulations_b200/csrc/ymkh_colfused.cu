// ymkh_colfused.cu — the column stages of a step in one launch, for grids of
// up to 512 rows (NZ a multiple of 32): sponge, xi_cut, z-mean removal with
// the colour-1 zeroing, the FP64 DFT band filters and z-hyperdiffusion
// (stages 6b to 6d, ymgpu2d/main_ym.cu:365-447; the kernels they replace are
// named in ymkh_column.cu).  Each of them treats every array on its own and
// works along z or pointwise, so one CTA can take 32 columns of one array
// through all of them: warp w holds the rows [32 w, 32 w + 32) of its lane's
// column in registers.
//
// What bounds it: below 512 rows the separate kernels (one to three a stage)
// are launches and half-empty waves of passes over L2-resident arrays; in a
// batch, a member's stages were up to five launches.  Here the members of a
// batch with the same NZ share one launch through a table.  The band filter's
// arithmetic stays bound by the FP64 pipe (ymkh_column.cu).
//
// Every sum keeps the order of the separate kernels, so the state is the same
// bit for bit: the z-mean is the reference's halving tree (levels that pair
// rows 32 or more apart pair warps, row by row; the last five are a tree over
// the 32 row sums), a coefficient is the warps' shuffle-tree roots added in
// warp order, and the hyperdiffusion stencils read values from before the update.

#include "ymkh_common.cuh"

namespace ymkh {

namespace {

constexpr int CF_BM = 8;  // modes per block of the band filter

__device__ __forceinline__ int find_col(const ColDesc* d, int n, int item) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (d[mid].item0 <= item) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Twiddles of this warp's 32 rows and modes [m0, m0 + CF_BM) into its own
// buffer [32][CF_BM], zero past the last mode.
__device__ __forceinline__ void stage_warp(double2* tw, const double* __restrict__ W, int M, int z0, int m0, int lane) {
#pragma unroll
  for (int u = 0; u < CF_BM; ++u) {
    const int e = lane + 32 * u, z = e / CF_BM, m = e % CF_BM;
    if (m0 + m < M) cp_async16(&tw[e], W + (size_t)(z0 + z) * 2 * M + 2 * (m0 + m));
    else tw[e] = make_double2(0.0, 0.0);
  }
  cp_async_commit();
}

// The row pitch behind an optimisation barrier, so that the 32 row addresses
// are formed anew at each use instead of being kept (and spilled) between them.
__device__ __forceinline__ size_t fresh(int nx) {
  asm volatile("" : "+r"(nx));
  return (size_t)nx;
}

}  // namespace

__global__ void __launch_bounds__(512, 1) column_kernel(const ColDesc* __restrict__ descs, int ndesc) {
  extern __shared__ __align__(16) double2 col_smem[];
  __shared__ ColDesc cd;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  {
    const int which = find_col(descs, ndesc, (int)blockIdx.x);
    const unsigned long long* s = reinterpret_cast<const unsigned long long*>(&descs[which]);
    unsigned long long* d = reinterpret_cast<unsigned long long*>(&cd);
    for (int i = tid; i < (int)(sizeof(ColDesc) / 8); i += blockDim.x) d[i] = s[i];
  }
  __syncthreads();
  const int nx = cd.nx, nz = cd.nz, nch = nz >> 5;
  const int local = (int)blockIdx.x - cd.item0;
  const int k = cd.k0 + local / cd.ncb;  // array of the list of 21; 3..14 are colours 2 and 3
  const int x = (local % cd.ncb) * 32 + lane;
  const bool in = x < nx;
  const bool c23 = k >= 3 && k < 15;
  double* const g = cd.arr[k] + (size_t)(32 * w) * nx + (in ? x : 0);  // this thread's rows: g[i * nx]

  if (k < 3 && cd.kz0) {  // colour 1 (ymgpu2d/main_ym.cu:443-447)
    if (in)
      for (int i = 0; i < 32; ++i) g[(size_t)i * nx] = 0.0;
    return;
  }

  double f[32];
  {
    const size_t pitch = fresh(nx);
#pragma unroll
    for (int i = 0; i < 32; ++i) f[i] = in ? g[i * pitch] : 0.0;
  }
  bool dirty = false;  // f differs from what memory holds

  if (c23 && (cd.sponge || cd.cut)) {  // YM_Physics.cu:161-210
    const double xc = (nx * cd.dx) * 0.5;
    const double xi = fabs((x * cd.dx - xc) / cd.epsilon);
    if (cd.sponge && xi > cd.xi_sponge) {
      const double sig = cd.sigma_sponge * (xi - cd.xi_sponge);
      const double dec = exp(-sig * cd.dt);
#pragma unroll
      for (int i = 0; i < 32; ++i) f[i] *= dec;
    }
    if (cd.cut && xi > cd.xi_cut) {
#pragma unroll
      for (int i = 0; i < 32; ++i) f[i] = 0.0;
    }
    dirty = true;
  }

  if (c23 && cd.kz0) {  // z-mean (YM_Physics.cu:301-308), NZ a power of two
    double t[16];
    if (nch == 1) {
#pragma unroll
      for (int i = 0; i < 16; ++i) t[i] = f[i] + f[i + 16];
    } else {
      double* const rows = reinterpret_cast<double*>(col_smem) + lane;  // [nch][32][32]
      double* const part = rows + nch * 1024;                           // [32][32] sums over the warps
#pragma unroll
      for (int i = 0; i < 32; ++i) rows[(w * 32 + i) * 32] = f[i];
      __syncthreads();
      const int h = nch >> 1;
      for (int i = w; i < 32; i += nch) {  // row i of all warps, halving tree over the warps
        double a[8];
        const double* r = rows + i * 32;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j < h) a[j] = r[j * 1024] + r[(j + h) * 1024];
#pragma unroll
        for (int s = 4; s > 0; s >>= 1)
          if (s < h)
#pragma unroll
            for (int j = 0; j < s; ++j) a[j] = a[j] + a[j + s];
        part[i * 32] = a[0];
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 16; ++i) t[i] = part[i * 32] + part[(i + 16) * 32];
      __syncthreads();  // the buffers are free again
    }
#pragma unroll
    for (int s = 8; s > 0; s >>= 1)
#pragma unroll
      for (int i = 0; i < s; ++i) t[i] = t[i] + t[i + s];
    const double mean = t[0] * (1.0 / (double)nz);
#pragma unroll
    for (int i = 0; i < 32; ++i) f[i] -= mean;
    dirty = true;
  }

  // band filters (YM_Physics.cu:349-584)
  double2* const tw = col_smem + w * (32 * CF_BM);   // [32][CF_BM], this warp's
  double2* const root = col_smem + nch * (32 * CF_BM);  // [nch][CF_BM][32]
  double2* const co = root + nch * CF_BM * 32 + lane;   // [M][32]
  for (int b = 0; b < cd.nb; ++b) {
    const double* const W = cd.W[b];
    const int M = cd.M[b];
    if (dirty && in) {
      const size_t pitch = fresh(nx);
#pragma unroll
      for (int i = 0; i < 32; ++i) g[i * pitch] = f[i];  // read back by the same thread below
    }
    for (int m0 = 0; m0 < M; m0 += CF_BM) {
      const int nm = min(CF_BM, M - m0);
      stage_warp(tw, W, M, 32 * w, m0, lane);
      cp_async_wait<0>();
      __syncwarp();
#pragma unroll 1
      for (int m = 0; m < nm; ++m) {
        const double2* t = tw + m;
        double sc[5], ss[5];  // pending tree nodes (band_coef_kernel)
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
          const int i = bitrev4(kk);
          const double2 w0 = t[i * CF_BM], w1 = t[(i + 16) * CF_BM];
          double c = f[i] * w0.x + f[i + 16] * w1.x;
          double s = f[i] * w0.y + f[i + 16] * w1.y;
          int lvl = 0;
#pragma unroll
          for (int L = 0; L < 4; ++L) {
            if (((kk >> L) & 1) && lvl == L) {
              c = sc[L] + c;
              s = ss[L] + s;
              ++lvl;
            }
          }
          sc[lvl] = c;
          ss[lvl] = s;
        }
        root[(w * CF_BM + m) * 32 + lane] = make_double2(sc[4], ss[4]);
      }
      __syncthreads();  // every warp's roots of the block
      for (int m = w; m < nm; m += nch) {
        double2 S = make_double2(0.0, 0.0);
        for (int j = 0; j < nch; ++j) {  // warp sums in warp order from 0.0
          const double2 r = root[(j * CF_BM + m) * 32 + lane];
          S.x = S.x + r.x;
          S.y = S.y + r.y;
        }
        co[(m0 + m) * 32] = make_double2(S.x * cd.inv2, S.y * cd.inv2);
      }
      __syncthreads();  // the roots are free again, the block's coefficients there
    }
    double d[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) d[i] = 0.0;
    for (int m0 = 0; m0 < M; m0 += CF_BM) {
      const int nm = min(CF_BM, M - m0);
      if (M > CF_BM) {  // (else the buffer still holds the only block)
        __syncwarp();
        stage_warp(tw, W, M, 32 * w, m0, lane);
        cp_async_wait<0>();
        __syncwarp();
      }
#pragma unroll 1
      for (int m = 0; m < nm; ++m) {
        const double2 ab = co[(m0 + m) * 32];
        const double2* t = tw + m;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const double2 v = t[i * CF_BM];
          d[i] = d[i] + (ab.x * v.x + ab.y * v.y);
        }
      }
    }
    const size_t pitch = fresh(nx);
#pragma unroll
    for (int i = 0; i < 32; ++i) f[i] = (in ? g[i * pitch] : 0.0) - d[i];
    dirty = true;
    __syncwarp();
  }

  if (c23 && cd.hyper) {  // YM_Physics.cu:228-259
    double* const edge = reinterpret_cast<double*>(col_smem);  // [nch][4][32]: first and last two rows of each warp
    __syncthreads();
    edge[(w * 4 + 0) * 32 + lane] = f[0];
    edge[(w * 4 + 1) * 32 + lane] = f[1];
    edge[(w * 4 + 2) * 32 + lane] = f[30];
    edge[(w * 4 + 3) * 32 + lane] = f[31];
    __syncthreads();
    const int wp = w == 0 ? nch - 1 : w - 1, wn = w == nch - 1 ? 0 : w + 1;
    double w0 = edge[(wp * 4 + 2) * 32 + lane], w1 = edge[(wp * 4 + 3) * 32 + lane];
    const double t0 = edge[(wn * 4 + 0) * 32 + lane], t1 = edge[(wn * 4 + 1) * 32 + lane];
    const double mu = cd.hyp_diff;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const double w2 = f[i], w3 = i < 31 ? f[i < 31 ? i + 1 : 31] : t0, w4 = i < 30 ? f[i < 30 ? i + 2 : 31] : (i == 30 ? t0 : t1);
      const double d4 = w0 - 4.0 * w1 + 6.0 * w2 - 4.0 * w3 + w4;
      f[i] = w2 - mu * d4;
      w0 = w1;
      w1 = w2;
    }
    dirty = true;
  }

  if (in && dirty) {
    const size_t pitch = fresh(nx);
#pragma unroll
    for (int i = 0; i < 32; ++i) g[i * pitch] = f[i];
  }
}

size_t column_fused_smem(int nz, int max_modes, int kz0) {
  const size_t nch = (size_t)nz / 32;
  const size_t band = max_modes ? nch * (2 * 32 * CF_BM) + (size_t)max_modes * 32 : 0;
  const size_t zmean = kz0 && nch > 1 ? nch * 512 + 512 : 0, edge = nch * 64;
  return sizeof(double2) * std::max(band, std::max(zmean, edge));
}

cudaError_t prepare_column_fused() {
  return cudaFuncSetAttribute(column_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kColumnFusedSmemMax);
}

cudaError_t launch_column_fused(const ColDesc* dev, int n, int items, int nz, size_t smem, cudaStream_t s) {
  column_kernel<<<items, nz, smem, s>>>(dev, n);
  return cudaGetLastError();
}

}  // namespace ymkh
