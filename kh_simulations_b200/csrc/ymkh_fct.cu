// ymkh_fct.cu — fused flux-corrected transport of both beams.
//
// One launch replaces, per time step, the reference's stages 1-4
// (ymgpu2d/main_ym.cu:324-355): velocities (YM_Fluid.cu:3-11), the four D2D
// state copies (YM_Fluid.cu:134-143), the periodic x-sweep with ghost padding
// (YM_FCT.cu:47-91) or the wall x-sweep (YM_FCT.cu:30-45), the transposed
// z-sweep (YM_FCT.cu:93-135, FCT_Sweeps.cu:12-177) and the density floor /
// wall boundary (YM_Fluid.cu:13-30), for all six swept variables
// (n, px, pz, Q1..Q3) of both beams.  The momentum and colour sources the
// reference stores at the end of the previous step (kernel_ym_lorentz,
// kernel_ym_precession, YM_Fluid.cu:32-108) are recomputed here from the
// start-of-step state, which is what they are a function of.
//
// Two forms: fct_strip_kernel (128-wide strips, one warp per variable, further
// down with its own comment) for all but the smallest grids and for batches,
// and fct_fused_kernel<32 | 64>, described here (32 for the smallest grids, 64
// where the caller or the tuner asks for it).
//
// Layout: work items are (x-strip, z-segment) pairs; each persistent CTA takes
// a contiguous block of them and runs each strip's part as one piece.  A strip
// emits TB-6 columns; thread t of a beam owns
// stage position t+1 (shear index x0-3+t), and every x-sweep phase is at
// most one position or interface per thread: interface quantities (eps, nu,
// mu, low-order fluxes) are formed once per interface.  Threads [0,TB)
// handle beam A, [TB,2TB) beam B; the beams synchronise only through their
// own named barriers.  Row data (12 fluid arrays plus the field rows the
// sources need) is staged in shared memory NST-1 rows ahead: TMA bulk row
// copies (cp.async.bulk, split at the periodic wrap), one per thread spread
// over all warps, complete on a per-stage mbarrier; wall boundaries use
// per-element cp.async with clamped indices.  For each row the x-sweep
// (FCT_Sweeps.cu:88-162) runs across the strip in shared memory; its result
// for the thread's own column feeds a register pipeline that performs the
// z-sweep along the stream, emitting row r-3 once row r arrives (halo 3,
// zero-gradient clamped z ends as FCT_Sweeps.cu:68-81).
//
// HBM traffic per cell: 24 arrays read (12 fluid + 12 fields), 12 written;
// row and column halos come from L2/shared memory.

#include "ymkh_common.cuh"

namespace ymkh {

namespace {

// Stage layout (units of W doubles); stage position sp holds shear index
// x = x0 - 4 + sp, sp in [0, W) with W = TB + 2.
constexpr int ST_FL = 0;     // fluid: (beam*6 + var)
constexpr int ST_EX = 12;    // Ex1..3 row zr
constexpr int ST_BY = 15;    // By1..3 row zr
constexpr int ST_BYM = 18;   // By1..3 row zm
constexpr int ST_EZ = 21;    // Ez1..3 row zr
constexpr int ST_EZM = 24;   // Ez1..3 row zm
constexpr int ST_AZ = 27;    // Az1..3 row zr
constexpr int ST_AZM = 30;   // Az1..3 row zm
constexpr int ST_NZP = 33;   // n (beam A, B) row zp (warm_T only)
constexpr int ST_NZM = 35;   // n (beam A, B) row zm (warm_T only)
constexpr int ST_SIZE = 37;

// Per-beam work arrays (units of W), by stage position / interface index
// (interface j+1/2 stored at j).  Fluxes F, D are dead after phase B, so the
// limited fluxes reuse their space.  WB_SZ holds the pz z-source of the last
// two rows (slot r & 1): the Q group forms it, the n/px/pz group uses it one
// row later, which keeps the two groups' work per row about equal.
constexpr int WB_F = 1, WB_D = 7, WB_FLIM = 1, WB_LOR = 13, WB_LNR = 19, WB_SZ = 25, WB_SIZE = 27;

// Named barrier of one (beam, half) thread group (ids 1..4; 0 is __syncthreads).
__device__ __forceinline__ void beam_bar(int group, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(nthreads) : "memory");
}

// apply_fct_limiter (FCT_DeviceMath.cuh:108-125) with the products by
// copysign(1, d0) written as flips of the sign bit: multiplying by -1 is an
// exact negation, i.e. the same bits.  The inner minima may differ from
// fmin's only in the sign of a zero, which max_sel(+0, .) removes.
__device__ __forceinline__ double flip_sign(double x, unsigned long long m) {
  return __longlong_as_double(__double_as_longlong(x) ^ m);
}
__device__ __forceinline__ double fct_limit_sel(double f, double dm1, double d0, double dp1) {
  const unsigned long long m = (unsigned long long)__double_as_longlong(d0) & 0x8000000000000000ull;
  const double r = max_sel(0.0, min_sel(flip_sign(dm1, m), min_sel(fabs(f), flip_sign(dp1, m))));
  return flip_sign(r, m);
}

}  // namespace

template <int TB>
constexpr size_t fct_smem_bytes(int nst) {
  return (size_t)(TB + 2) * sizeof(double) * (nst * ST_SIZE + 2 * WB_SIZE) + (size_t)(TB + 2) * sizeof(int) +
         (size_t)8 * nst + 16;
}


// The half of a thread group as a compile-time constant: the row loop is
// compiled once per half, with the swept variables' shared-memory offsets,
// which variables carry z-sources and which source each half forms fixed
// (1.0% faster at 4096 x 8192 than one loop that branches on the half).
template <int V>
struct HalfC {
  static constexpr int value = V;
};

// One TMA bulk row copy of a stage (the table in fct_fused_kernel).
struct RowCopy {
  const double* base;
  const double* base0;
  int dst, kind, len1, pad_;
};

// Per-thread z-pipeline state for the three swept variables of one half
// (H = 0: n, px, pz; H = 1: Q1, Q2, Q3) of one beam.
struct ZPipe {
  double V1[3], f1[3], d1[3], L2[3], N4[3], N3[3], N2[3], A2[3], F3[3], S1[3];
  double U1, mu1;
};

template <int TB, int NST>
__global__ void __launch_bounds__(4 * TB, 2)
    fct_fused_kernel(const __grid_constant__ RunTable T) {
  constexpr int W = TB + 2;
  constexpr int NT = 4 * TB;
  constexpr int TO = TB - 6;  // output columns per strip
  extern __shared__ __align__(16) double smem[];
  double* const stage = smem;
  double* const wk = smem + (size_t)NST * ST_SIZE * W;
  int* const xtab = reinterpret_cast<int*>(wk + (size_t)2 * WB_SIZE * W);
  uint64_t* const bars = reinterpret_cast<uint64_t*>(
      (reinterpret_cast<uintptr_t>(xtab + W) + 15) & ~static_cast<uintptr_t>(15));

  __shared__ RunDesc rd;
  __shared__ int s_run;
  __shared__ RowCopy cpt[40];
  const State& st = rd.in;
  const State& out = rd.out;
  const StepParams& p = rd.p;
  const int tid = threadIdx.x;
  const int grp = tid / TB;     // (beam, half) group, 0..3
  const int beam = grp >> 1;
  const int half = grp & 1;     // 0: n, px, pz   1: Q1, Q2, Q3
  const int t = tid - grp * TB;
  const int sp = t + 1;         // this thread's stage position
  double* const wb = wk + (size_t)beam * WB_SIZE * W;

  if (tid == 0) {
    for (int s = 0; s < NST; ++s) mbar_init(&bars[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  unsigned issued = 0, consumed = 0;  // rows issued / consumed by this CTA (all items)
  unsigned phase_bits = 0;            // per-stage mbarrier phase of the bulk path

  // Each CTA takes one contiguous block of the flattened items.  Within a run
  // the items are strip-major (a strip's z-segments consecutive), and
  // consecutive segments of one strip form one piece: the z pipeline warms up
  // (6 rows) once per piece instead of once per segment.  The host cuts the
  // blocks by cost.
  const int i_beg = T.fct_first[blockIdx.x], i_end = T.fct_first[blockIdx.x + 1];
  int next = i_beg;
  for (int item = i_beg; item < i_end; item = next) {
    __syncthreads();  // previous piece fully consumed
    if (tid == 0) s_run = find_run(T.runs, T.nruns, item, false);
    __syncthreads();
    load_desc(&rd, &T.runs[s_run]);
    __syncthreads();
    const int nx = p.nx, nz = p.nz;
    const bool warm = p.warm_T > 0.0;
    const bool wall = !p.periodic_x;
    const bool bulk = rd.fct_bulk == LOAD_BULK_ALL;  // TMA bulk rows on mbarriers (else per-element cp.async)
    const double dt = p.dt;
    const double dtdx = p.dt / p.dx;
    const double dtdz = p.dt / p.dz;
    const int nseg = (nz + rd.fct_seg - 1) / rd.fct_seg;
    const int local = item - rd.fct_item0;
    const int strip = local / nseg;
    const int seg0 = local - strip * nseg;
    next = min(i_end, rd.fct_item0 + (strip + 1) * nseg);  // past this piece's last segment
    const int zs = seg0 * rd.fct_seg;
    const int ze = min(nz, (seg0 + (next - item)) * rd.fct_seg);
    const int x0 = strip * TO;

    if (!bulk)
      for (int i = tid; i < W; i += NT) xtab[i] = stage_x(x0 - 4 + i, nx, p.periodic_x);
    // the pz source before the first row is zero, as the pipeline's start
    for (int i = tid; i < 2 * 2 * W; i += NT) wk[(size_t)(i / (2 * W)) * WB_SIZE * W + WB_SZ * W + i % (2 * W)] = 0.0;
    __syncthreads();

    // bulk rows: the row copies of the item, one per array of the stage
    // (source array at the strip's first column and at column 0 for the part
    // past the periodic wrap, stage slot offset, which row, length before the
    // wrap) in a shared table read by the issuing thread
    if (bulk && tid < 33 + (warm ? 4 : 0)) {
      const int a = tid;
      const double* base;
      int dst, kind_row = 0;
      if (a < 12) {
        base = a < 6 ? st.a[a] : st.b[a - 6];
        dst = ST_FL + a;
      } else if (a < 33) {
        const int kind = (a - 12) / 3, c = (a - 12) - kind * 3;  // EX, BY, BYM, EZ, EZM, AZ, AZM
        base = (kind == 0) ? st.f[EX1 + c] : (kind <= 2) ? st.f[BY1 + c] : (kind <= 4) ? st.f[EZ1 + c] : st.f[AZ1 + c];
        dst = ST_EX + (a - 12);
        kind_row = (kind == 2 || kind == 4 || kind == 6) ? 1 : 0;
      } else {
        const int w = a - 33;  // NZP A, NZP B, NZM A, NZM B
        base = (w & 1) ? st.b[FN] : st.a[FN];
        dst = ST_NZP + w;
        kind_row = (w >> 1) ? 1 : 2;
      }
      int x = (x0 - 4) % nx;
      x = x < 0 ? x + nx : x;
      cpt[a].base = base + x;
      cpt[a].base0 = base;
      cpt[a].dst = dst;
      cpt[a].kind = kind_row;
      cpt[a].len1 = min(W, nx - x);
    }
    __syncthreads();

    auto issue_row = [&](int r) {
      const int s = (int)(issued % NST);
      double* sb = stage + (size_t)s * ST_SIZE * W;
      const int zr = zclamp(r, nz);
      const int zm = (zr == 0) ? nz - 1 : zr - 1;
      const int zp = (zr == nz - 1) ? 0 : zr + 1;
      const size_t ro = (size_t)zr * nx, rom = (size_t)zm * nx, rop = (size_t)zp * nx;
      const int narr = 33 + (warm ? 4 : 0);
      if (bulk) {
        // one row copy per thread, spread over the warps (lane-major) so no
        // single warp serialises the issue; completions that land before
        // thread 0 arms the stage only drive its transaction count negative,
        // and the phase cannot complete before that arrival.  The copy's
        // array, slot and wrap split are fixed per item (cp_*).
        if (tid == 0) mbar_expect_tx(&bars[s], (unsigned)(narr * W * 8));
        const int ca = (tid & 31) * (NT / 32) + (tid >> 5);  // lane-major over the warps
        if (ca < narr) {
          const RowCopy& c = cpt[ca];
          const int len1 = c.len1;
          if (dbg_ok(zr >= 0 && zr < nz && zm >= 0 && zm < nz && zp >= 0 && zp < nz && len1 > 0 && W - len1 <= nx &&
                         c.dst >= 0 && c.dst < ST_SIZE, T.err)) {
            const size_t off = c.kind == 0 ? ro : (c.kind == 1 ? rom : rop);
            double* const dst = sb + c.dst * W;
            bulk_g2s(dst, c.base + off, (unsigned)len1 * 8u, &bars[s]);
            if (len1 < W) bulk_g2s(dst + len1, c.base0 + off, (unsigned)(W - len1) * 8u, &bars[s]);
          }
        }
      } else {
        const bool rows_ok = dbg_ok(zr >= 0 && zr < nz && zm >= 0 && zm < nz && zp >= 0 && zp < nz, T.err);
        for (int i = tid; i < 12 * (W - 1); i += NT) {
          const int a = i / (W - 1), q = 1 + (i - a * (W - 1));
          if (rows_ok && dbg_ok(xtab[q] >= 0 && xtab[q] < nx, T.err))
            cp_async8(sb + (ST_FL + a) * W + q, (a < 6 ? st.a[a] : st.b[a - 6]) + ro + xtab[q]);
        }
        for (int i = tid; i < 21 * (W - 1); i += NT) {
          const int a = i / (W - 1), q = 1 + (i - a * (W - 1));
          const int kind = a / 3, c = a - kind * 3;  // EX, BY, BYM, EZ, EZM, AZ, AZM
          const double* base = (kind == 0) ? st.f[EX1 + c]
                               : (kind <= 2) ? st.f[BY1 + c]
                               : (kind <= 4) ? st.f[EZ1 + c]
                                             : st.f[AZ1 + c];
          const size_t off = (kind == 2 || kind == 4 || kind == 6) ? rom : ro;
          if (rows_ok && dbg_ok(xtab[q] >= 0 && xtab[q] < nx, T.err))
            cp_async8(sb + (ST_EX + a) * W + q, base + off + xtab[q]);
        }
        if (warm) {
          for (int i = tid; i < 4 * (W - 1); i += NT) {
            const int a = i / (W - 1), q = 1 + (i - a * (W - 1));
            const double* base = (a & 1) ? st.b[FN] : st.a[FN];
            if (rows_ok && dbg_ok(xtab[q] >= 0 && xtab[q] < nx, T.err))
              cp_async8(sb + (ST_NZP + a) * W + q, base + ((a >> 1) ? rom : rop) + xtab[q]);
          }
        }
        cp_async_commit();
      }
      ++issued;
    };

    const int r_first = zs - 3, r_last = ze + 2;
    for (int k = 0; k < NST - 1; ++k)
      if (r_first + k <= r_last) issue_row(r_first + k);
      else if (!bulk) cp_async_commit();

    // the piece's rows, for this thread's half (a compile-time constant here)
    auto rows = [&](auto HC) {
      constexpr int half = decltype(HC)::value;
      constexpr int k0 = 3 * half;  // first swept variable of this half
      ZPipe zp;
#pragma unroll
      for (int j = 0; j < 3; ++j)
        zp.V1[j] = zp.f1[j] = zp.d1[j] = zp.L2[j] = zp.N4[j] = zp.N3[j] = zp.N2[j] = zp.A2[j] = zp.F3[j] = zp.S1[j] = 0.0;
      zp.U1 = zp.mu1 = 0.0;
      const int x_own = x0 - 4 + sp;
      const bool zthread = (t >= 3) && (t < TB - 3);  // owns an output column
      const bool owner = zthread && (x_own < nx);

      for (int r = r_first; r <= r_last; ++r) {
        const int s = (int)(consumed % NST);
        if (bulk) {  // one thread polls the stage's mbarrier; the CTA barrier below
          // releases the others after it (no spinning by every thread)
          if (tid == 0) mbar_wait(&bars[s], (phase_bits >> s) & 1u, T.err);
          phase_bits ^= 1u << s;
        } else {
          cp_async_wait<NST - 2>();
        }
        __syncthreads();  // row r staged for everyone; the previous row's stage is free
        ++consumed;
        if (r + NST - 1 <= r_last) issue_row(r + NST - 1);
        else if (!bulk) cp_async_commit();
        const double* sb = stage + (size_t)s * ST_SIZE * W;
        const double* fl = sb + (size_t)(ST_FL + beam * 6) * W;

        // ---- A: velocities at sp, sp+1 (YM_Fluid.cu:3-11); interface sp+1/2:
        // eps, nu, mu and the low-order fluxes of this half's variables
        // (FCT_Sweeps.cu:88-98); half 0 also forms the px source at sp
        // (YM_Fluid.cu:43-66, 71-80).
        double vz_own, ux_own, mu_if = 0.0, sx = 0.0;
        double Fo[3] = {0.0, 0.0, 0.0}, Do[3] = {0.0, 0.0, 0.0};  // this thread's interface fluxes
        {
          const double n0 = max_sel(fl[FN * W + sp], 0.05);
          ux_own = fl[FPX * W + sp] / n0;
          vz_own = fl[FPZ * W + sp] / n0;
          if (t < TB - 1) {
            const double n1 = max_sel(fl[FN * W + sp + 1], 0.05);
            const double u1 = fl[FPX * W + sp + 1] / n1;
            const double e = fct_eps(ux_own, u1, dtdx);
            double nu;
            fct_nu_mu(e, nu, mu_if);
#pragma unroll
            for (int j = 0; j < 3; ++j) {
              const int k = k0 + j;
              const double v0 = fl[k * W + sp], v1 = fl[k * W + sp + 1];
              Fo[j] = 0.5 * e * (v0 + v1);
              Do[j] = nu * (v1 - v0);
              wb[(WB_F + k) * W + sp] = Fo[j];
              wb[(WB_D + k) * W + sp] = Do[j];
            }
          }
          if (half == 0 && t >= 1 && t < TB - 1) {
            int ps = sp;  // at a wall the clamped ghost cells carry the edge cell's source
            if (wall) {
              const int xg = x0 - 4 + sp;
              ps = (xg < 0 ? 0 : (xg >= nx ? nx - 1 : xg)) - (x0 - 4);
            }
            const double vz = (ps == sp) ? vz_own : fl[FPZ * W + ps] / max_sel(fl[FN * W + ps], 0.05);
            double acc = 0.0;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              const double ex = 0.5 * (sb[(ST_EX + c) * W + ps] + sb[(ST_EX + c) * W + ps - 1]);
              const double by = 0.25 * (sb[(ST_BY + c) * W + ps] + sb[(ST_BY + c) * W + ps - 1] +
                                        sb[(ST_BYM + c) * W + ps] + sb[(ST_BYM + c) * W + ps - 1]);
              const double term = fl[(FQ1 + c) * W + ps] * (ex + vz * by);
              acc = (c == 0) ? term : acc + term;
            }
            sx = -acc;
            if (warm) {
              const double dndx = (fl[FN * W + ps + 1] - fl[FN * W + ps - 1]) / (2.0 * p.dx);
              sx -= p.warm_T * dndx;
            }
          }
        }
        beam_bar(grp, TB);

        // ---- B: lorhot / lnrhot at sp (FCT_Sweeps.cu:102-103), t in [1, TB-1).
        double Lo[3] = {0.0, 0.0, 0.0}, Ln[3] = {0.0, 0.0, 0.0};  // this thread's lorhot, lnrhot
        if (t >= 1 && t < TB - 1) {
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            const int k = k0 + j;
            const double v0 = fl[k * W + sp];
            const double fd = Fo[j] - wb[(WB_F + k) * W + sp - 1];
            const double dd = Do[j] - wb[(WB_D + k) * W + sp - 1];
            const double lo = (k == FPX) ? v0 + dt * sx - fd : v0 - fd;
            Lo[j] = lo;
            Ln[j] = lo + dd;
            wb[(WB_LOR + k) * W + sp] = lo;
            wb[(WB_LNR + k) * W + sp] = Ln[j];
          }
        }
        beam_bar(grp, TB);

        // ---- C: antidiffusive flux and limiter at interface sp+1/2
        // (FCT_Sweeps.cu:139-160), t in [2, TB-3).
        double Fl[3] = {0.0, 0.0, 0.0};  // this thread's limited flux
        if (t >= 2 && t < TB - 3) {
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            const int k = k0 + j;
            const double* lor = wb + (WB_LOR + k) * W;
            const double* lnr = wb + (WB_LNR + k) * W;
            const double l1 = lnr[sp + 1];
            const double fad = mu_if * (lor[sp + 1] - Lo[j]);
            Fl[j] = fct_limit_sel(fad, Ln[j] - lnr[sp - 1], l1 - Ln[j], lnr[sp + 2] - l1);
            wb[(WB_FLIM + k) * W + sp] = Fl[j];
          }
        }
        beam_bar(grp, TB);

        // ---- D: x-swept values of the own column, z-sources, z-pipeline.
        if (zthread) {
          double Vx[3], S[3];
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            const int k = k0 + j;
            Vx[j] = Ln[j] - (Fl[j] - wb[(WB_FLIM + k) * W + sp - 1]);
          }
          const double vz = vz_own;
          const double q1 = fl[FQ1 * W + sp], q2 = fl[FQ2 * W + sp], q3 = fl[FQ3 * W + sp];
          if (half == 0) {
            // the pz source of row r-1, formed by the Q group last row
            S[0] = 0.0;
            S[1] = 0.0;
            S[2] = 0.0;
            zp.S1[2] = wb[(WB_SZ + ((r - 1) & 1)) * W + sp];
          } else {
            // YM_Fluid.cu:67 (src.pz) and :76-79 (warm closure), for the other group
            const double vx = ux_own;
            double by[3], ezn[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
              by[c] = 0.25 * (sb[(ST_BY + c) * W + sp] + sb[(ST_BY + c) * W + sp - 1] + sb[(ST_BYM + c) * W + sp] +
                              sb[(ST_BYM + c) * W + sp - 1]);
              ezn[c] = 0.5 * (sb[(ST_EZ + c) * W + sp] + sb[(ST_EZM + c) * W + sp]);
            }
            double sz = -(q1 * (ezn[0] - vx * by[0]) + q2 * (ezn[1] - vx * by[1]) + q3 * (ezn[2] - vx * by[2]));
            if (warm) {
              const double dndz = (sb[(ST_NZP + beam) * W + sp] - sb[(ST_NZM + beam) * W + sp]) / (2.0 * p.dz);
              sz -= p.warm_T * dndz;
            }
            wb[(WB_SZ + (r & 1)) * W + sp] = sz;
            // YM_Fluid.cu:99-107 (colour precession)
            double azn[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) azn[c] = 0.5 * (sb[(ST_AZ + c) * W + sp] + sb[(ST_AZM + c) * W + sp]);
            S[0] = p.alpha * vz * (q2 * azn[2] - q3 * azn[1]);
            S[1] = p.alpha * vz * (q3 * azn[0] - q1 * azn[2]);
            S[2] = p.alpha * vz * (q1 * azn[1] - q2 * azn[0]);
          }

          const double e = fct_eps(zp.U1, vz, dtdz);
          double nu, mu;
          fct_nu_mu(e, nu, mu);
          double outv[3];
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            const bool has_src = (half == 1) || (j == 2);  // pz and Q1..Q3 carry z-sources
            const double fR = 0.5 * e * (zp.V1[j] + Vx[j]);
            const double dR = nu * (Vx[j] - zp.V1[j]);
            const double lo = has_src ? zp.V1[j] + dt * zp.S1[j] - (fR - zp.f1[j]) : zp.V1[j] - (fR - zp.f1[j]);
            const double ln = lo + (dR - zp.d1[j]);
            const double fad = zp.mu1 * (lo - zp.L2[j]);
            const double flim = fct_limit_sel(zp.A2[j], zp.N3[j] - zp.N4[j], zp.N2[j] - zp.N3[j], ln - zp.N2[j]);
            outv[j] = zp.N3[j] - (flim - zp.F3[j]);
            zp.V1[j] = Vx[j];
            zp.S1[j] = S[j];
            zp.f1[j] = fR;
            zp.d1[j] = dR;
            zp.L2[j] = lo;
            zp.N4[j] = zp.N3[j];
            zp.N3[j] = zp.N2[j];
            zp.N2[j] = ln;
            zp.A2[j] = fad;
            zp.F3[j] = flim;
          }
          zp.U1 = vz;
          zp.mu1 = mu;
          const int o = r - 3;
          if (owner && o >= zs && o < ze) {
            // YM_Fluid.cu:20-29 (density floor, wall momentum)
            if (half == 0) {
              if (outv[0] < 0.05) outv[0] = 0.05;
              if (wall && (x_own == 0 || x_own == nx - 1)) outv[1] = 0.0;
            }
            double* const* dst = beam ? out.b : out.a;
            const size_t gi = idx2(x_own, o, nx);
            if (dbg_ok(x_own >= 0 && x_own < nx && o >= 0 && o < nz && sp >= 1 && sp + 2 < W, T.err)) {
#pragma unroll
              for (int j = 0; j < 3; ++j) dst[k0 + j][gi] = outv[j];
            }
          }
        }
      }
    };
    if (half == 0) rows(HalfC<0>{});
    else rows(HalfC<1>{});
    if (!bulk) {  // the next piece may take the stages by TMA
      cp_async_wait<0>();
      if (T.nruns > 1) fence_proxy_async();  // (a run keeps to one kind of copy)
    }
  }
}

// ---------------------------------------------------------------------------
// The 128-wide form: one warp per swept variable.
//
// What bounds it: the FP64 and integer instructions of the 24 sweeps per cell,
// at four warps a scheduler.  fct_fused_kernel issues 114 warp instructions a
// cell: every phase of the x sweep goes through shared memory and a barrier,
// each thread group forms its own velocities, and each row costs 33 row
// copies.  Here it is 73:
// - Twelve sweep warps take one variable of one beam each.  A lane owns four
//   neighbouring columns, so most neighbours are its own registers and the
//   rest come by shuffles; there is no barrier between the phases, and the
//   four columns are independent work.
// - Four coefficient warps run a row ahead: velocities, the interface
//   coefficients of both directions and all sources, once per cell and beam
//   (the field averages once for both beams), handed over in shared memory
//   through mbarriers (co_full, co_free; two slots).
// - A row arrives as three TMA boxes of 12, 12 and 9 arrays, requested by one
//   thread four rows ahead (six more small ones where the window wraps).
// - While every input is finite and far from overflow, the limiter needs two
//   compares (fct_limit_fin); a row that is not sends the rest of the piece
//   through the NaN-exact form.
// - The sweep warps hold 72 registers of z history: setmaxnreg gives them 136
//   and the coefficient warps 104 of the 512 x 128 at launch.
// Measured (FCT, one step, against the 128-wide fct_fused_kernel that it took
// the place of): 3.12 ms against 5.17 at 4096 x 8192, 227 us against 366 at
// 1024 x 2048, 42 against 73 at 256 x 768; of that, blocks cut by cost
// (3.42 -> 3.12 ms together with boxes for the edge strips).  Tried and slower
// (ms against the 3.4 to 3.9 of the kernel at the time): the z history rotated
// through names by unrolling the row loop two or three times (no register
// moves, but spills and a loop past the instruction cache: 3.6 and 5.3),
// separate fast and slow row loops, a CTA barrier per row in place of the
// mbarriers, divisions in place of `velocities` (4% more).

namespace {

constexpr int F2_W = kFctBoxWidth;  // staged positions per row: position q holds shear index x0 - 4 + q
constexpr int F2_O = 120;    // output columns per strip: positions 4 .. 123 (lanes 1 .. 30, four each)
constexpr int F2_NT = 512;   // 12 sweep warps, 4 coefficient warps
constexpr int F2_SWEEP = 12;
constexpr int F2_NFL = 6;    // ring depth of the fluid rows
constexpr int F2_NFD = 4;    // ring depth of the field rows, read by the coefficient warps only
// field rows of a stage, in the state's array order: row z of Ex, Ez, By, Az,
// row z-1 of Ez, By, Az, and n at z+1 and z-1 (warm_T only)
constexpr int F2_EX = 0, F2_EZ = 3, F2_BY = 6, F2_AZ = 9, F2_EZM = 12, F2_BYM = 15, F2_AZM = 18, F2_NZP = 21, F2_NZM = 23;
constexpr int F2_FD = 25;
constexpr int F2_WRAP = 144;  // wrapped columns of a row: 33 arrays of 4 (in 128-byte aligned blocks of 12)

// Rows a coefficient warp hands to the sweep warps, per beam: x-interface
// 0.5*eps and nu, dt * px source; z-interface 0.5*eps and nu, mu of the
// previous z-interface, dt * (pz, Q1..Q3 source) of the previous row.
constexpr int HR_XH = 0, HR_XNU = 1, HR_XS = 2, HR_ZH = 3, HR_ZNU = 4, HR_ZMU = 5, HR_ZS = 6, HR_SIZE = 10;
// Layout of such a row: position q at pair (q >> 1) of the even or odd
// pairs, so that lane l's four positions are two 16-byte loads at stride 16
// (no bank conflict) and the writers' 8-byte stores conflict-free too (the
// odd pairs start 64 bytes past a 128-byte boundary).
constexpr int HR_ODD = 72, HR_W = 136;
__device__ __forceinline__ int hr_pos(int q) { return ((q >> 1) & 1) * HR_ODD + (q >> 2) * 2 + (q & 1); }

__device__ __forceinline__ void ld4(double (&v)[4], const double* p0, const double* p1) {
  const double2 a = *reinterpret_cast<const double2*>(p0), b = *reinterpret_cast<const double2*>(p1);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

constexpr int F2_NCO = 2;  // coefficient slots
static_assert(F2_NFL == 4 + F2_NCO && F2_NFD == 4, "row i+4 takes the fluid slot of row i-2 and the field slot of row i");

// Barrier of the coefficient warps (id 1; 0 is __syncthreads).
__device__ __forceinline__ void coef_bar() {
  asm volatile("bar.sync 1, %0;" ::"n"(F2_NT - 32 * F2_SWEEP) : "memory");
}

// The limiter for finite arguments: the same result as fct_limit_sel.  With
// s the sign of d0, max(0, min(s dm1, |f|, s dp1)) is zero when dm1 or dp1 has
// the other sign, else the smallest of the three magnitudes; s then gives it
// d0's sign.  Two compares instead of five, and no sign flips.
__device__ __forceinline__ double fct_limit_fin(double f, double dm1, double d0, double dp1) {
  const int h0 = __double2hiint(d0);
  const int differ = (__double2hiint(dm1) ^ h0) | (__double2hiint(dp1) ^ h0);  // sign bit
  double m = fabs(dp1) < fabs(dm1) ? dp1 : dm1;
  m = fabs(f) < fabs(m) ? f : m;
  const int lo = differ < 0 ? 0 : __double2loint(m);
  const int hi = differ < 0 ? 0 : __double2hiint(m);
  return __hiloint2double((hi & 0x7fffffff) | (h0 & (int)0x80000000), lo);
}

// Inputs below 2^100 and coefficients below 2^200 in magnitude keep every
// product and sum of a sweep far from overflow (at most 2^800 or so).
constexpr int F2_BIG_HI = (1023 + 100) << 20;
constexpr double F2_BIG = 0x1p200;

}  // namespace

constexpr size_t fct_strip_smem_bytes() {
  return sizeof(double) * ((size_t)F2_W * (F2_NFL * 12 + F2_NFD * F2_FD) + F2_NFD * F2_WRAP + F2_NCO * 2 * HR_SIZE * HR_W) +
         sizeof(int) * F2_W + 8 * (F2_NFL + 2 * F2_NCO + 1) + sizeof(double) * (4 * F2_W + 2);
}

__global__ void __launch_bounds__(F2_NT, 1) fct_strip_kernel(const __grid_constant__ RunTable T) {
  constexpr int W = F2_W;
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(128) double strip_smem[];
  double* const sfl = strip_smem;                              // [F2_NFL][12][W]
  double* const sfd = sfl + (size_t)F2_NFL * 12 * W;     // [F2_NFD][F2_FD][W]
  double* const wrap = sfd + (size_t)F2_NFD * F2_FD * W;  // [F2_NFD][F2_WRAP] wrapped columns
  double* const hlp = wrap + F2_NFD * F2_WRAP;  // [F2_NCO][2 beams][HR_SIZE][HR_W]
  int* const xtab = reinterpret_cast<int*>(hlp + F2_NCO * 2 * HR_SIZE * HR_W);
  uint64_t* const bars = reinterpret_cast<uint64_t*>(xtab + W);  // row staged [F2_NFL]
  uint64_t* const co_full = bars + F2_NFL;                        // coefficients written [F2_NCO]
  uint64_t* const co_free = co_full + F2_NCO;                     // row and coefficients read [F2_NCO]
  double* const uxr = reinterpret_cast<double*>(co_free + F2_NCO + 1);  // [2][2 beams][W] ux of the row

  __shared__ RunDesc rd;
  __shared__ int s_run, s_bad;
  __shared__ RowCopy cpt[40];
  const State& st = rd.in;
  const State& out = rd.out;
  const StepParams& p = rd.p;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  if (tid == 0) {
    for (int s = 0; s < F2_NFL; ++s) mbar_init(&bars[s], 1);
    for (int s = 0; s < F2_NCO; ++s) {
      mbar_init(&co_full[s], F2_NT / 32 - F2_SWEEP);
      mbar_init(&co_free[s], F2_SWEEP);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // sequence number of the piece's first row in the rings
  unsigned seq = 0;
  unsigned phase_bits = 0;  // per-barrier phase of the bulk path (one coefficient thread waits)

  // this CTA's items: a contiguous block, cut by cost on the host
  const int i_beg = T.fct_first[blockIdx.x], i_end = T.fct_first[blockIdx.x + 1];

  // The piece that starts at an item: its run, strip and rows.  Every thread
  // calls it once per piece; the barriers also end the previous piece.
  struct Piece {
    int x0, zs, ze, next;
    bool warm, wall, bulk, box, edge;
  };
  auto begin_piece = [&](int item) -> Piece {
    Piece c;
    __syncthreads();  // previous piece fully consumed
    if (tid == 0) {
      s_run = find_run(T.runs, T.nruns, item, false);
      s_bad = 0;
    }
    __syncthreads();
    load_desc(&rd, &T.runs[s_run]);
    __syncthreads();
    const int nx = p.nx, nz = p.nz;
    c.warm = p.warm_T > 0.0;
    c.wall = !p.periodic_x;
    c.bulk = rd.fct_bulk != LOAD_ELEM;
    const int nseg = (nz + rd.fct_seg - 1) / rd.fct_seg;
    const int local = item - rd.fct_item0;
    const int strip = local / nseg, seg0 = local - strip * nseg;
    c.next = min(i_end, rd.fct_item0 + (strip + 1) * nseg);  // past this piece's last segment
    c.zs = seg0 * rd.fct_seg;
    c.ze = min(nz, (seg0 + (c.next - item)) * rd.fct_seg);
    c.x0 = strip * F2_O;
    c.edge = c.x0 == 0 || c.x0 - 4 + W > nx;
    c.box = rd.fct_bulk == LOAD_BOX && !(c.warm && c.edge);
    return c;
  };

  if (warp < F2_SWEEP) {
    // -------------------------------------------------- a sweep warp: one variable of one beam
    asm volatile("setmaxnreg.inc.sync.aligned.u32 136;");
    const int beam = warp / 6, k = warp - beam * 6;
    const bool has_sx = (k == FPX), has_sz = (k >= FPZ);
    const double* const fl0 = sfl + (beam * 6 + k) * W + 4 * lane;
    const double* const fl_last = fl0 + (size_t)(F2_NFL - 1) * 12 * W;
    const double* const hlp0 = hlp + beam * (HR_SIZE * HR_W) + 2 * lane;
    const double* fl = fl0;  // this lane's columns of the row, in the ring
    unsigned gc = 0;         // rows read so far: coefficient slot and phase
    for (int item = i_beg; item < i_end;) {
      const Piece c = begin_piece(item);
      item = c.next;
      __syncthreads();  // the coefficient warps' row table
      const int nx = p.nx;
      const int nrow = c.ze - c.zs + 6;  // rows zs-3 .. ze+2
      double* dst = (beam ? out.b[k] : out.a[k]) + idx2(0, c.zs, nx);
      const int xo = c.x0 - 4 + 4 * lane;  // first of this lane's four columns
      const bool owner = lane >= 1 && lane <= 30 && xo < nx;
      const bool bulk = c.bulk;
      const int wall_x = (c.wall && k == FPX) ? nx - 1 : -1;  // px is zero at x = 0 and here
      double V1[4], f1[4], d1[4], L2[4], Na[4], Nb[4], Nc[4], A2[4], F3[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) V1[j] = f1[j] = d1[j] = L2[j] = Na[j] = Nb[j] = Nc[j] = A2[j] = F3[j] = 0.0;

      // Whether every input of row i is finite and small enough that no
      // later product or sum can overflow: then no NaN or infinity arises,
      // and the limiter may use plain compares.
      auto row_is_finite = [&] {
        double v[4];
        ld4(v, fl, fl + 2);
        const int m = max(max(__double2hiint(v[0]) & 0x7fffffff, __double2hiint(v[1]) & 0x7fffffff),
                          max(__double2hiint(v[2]) & 0x7fffffff, __double2hiint(v[3]) & 0x7fffffff));
        return !__any_sync(FULL, m >= F2_BIG_HI) && *(volatile int*)&s_bad == 0;
      };
      // Row i: x sweep of the row, then one step of the z sweep down the
      // lane's columns; N4, N3, N2 are the last three z lnrhot rows and N4
      // receives the new one.
      auto row = [&](bool fin, int i, double(&N4)[4], double(&N3)[4], double(&N2)[4]) {
        const double* const hr = hlp0 + (gc & 1u) * (2 * HR_SIZE * HR_W);
        // ---- x sweep (FCT_Sweeps.cu:88-162): interface j is between this lane's columns j and j+1
        double ln[4], fx[4];
        {
          double v[4], h[4], nu[4], F[4], D[4], lo[4], dd[4];
          ld4(v, fl, fl + 2);
          ld4(h, hr + HR_XH * HR_W, hr + HR_XH * HR_W + HR_ODD);
          ld4(nu, hr + HR_XNU * HR_W, hr + HR_XNU * HR_W + HR_ODD);
          const double vr = __shfl_down_sync(FULL, v[0], 1);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const double vn = j < 3 ? v[j + 1] : vr;
            F[j] = h[j] * (v[j] + vn);
            D[j] = nu[j] * (vn - v[j]);
          }
          const double Fl = __shfl_up_sync(FULL, F[3], 1), Dl = __shfl_up_sync(FULL, D[3], 1);
          if (has_sx) {
            double s[4];
            ld4(s, hr + HR_XS * HR_W, hr + HR_XS * HR_W + HR_ODD);
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = v[j] + s[j];
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            lo[j] = v[j] - (F[j] - (j ? F[j - 1] : Fl));
            ln[j] = lo[j] + (D[j] - (j ? D[j - 1] : Dl));
          }
          const double lor = __shfl_down_sync(FULL, lo[0], 1), lnr = __shfl_down_sync(FULL, ln[0], 1);
#pragma unroll
          for (int j = 0; j < 4; ++j) dd[j] = (j < 3 ? ln[j + 1] : lnr) - ln[j];
          const double ddl = __shfl_up_sync(FULL, dd[3], 1), ddr = __shfl_down_sync(FULL, dd[0], 1);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const double mu = fma(-0.5, nu[j], 0.25);  // 0.25 - 0.5*nu: 0.5*nu is exact
            fx[j] = mu * ((j < 3 ? lo[j + 1] : lor) - lo[j]);
          }
          if (fin) {
#pragma unroll
            for (int j = 0; j < 4; ++j) fx[j] = fct_limit_fin(fx[j], j ? dd[j - 1] : ddl, dd[j], j < 3 ? dd[j + 1] : ddr);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) fx[j] = fct_limit_sel(fx[j], j ? dd[j - 1] : ddl, dd[j], j < 3 ? dd[j + 1] : ddr);
          }
        }
        const double fxl = __shfl_up_sync(FULL, fx[3], 1);
        // ---- z sweep: row i-3 leaves when row i arrives
        double ov[4];
        {
          double h[4], nu[4], mu1[4], s[4];
          ld4(h, hr + HR_ZH * HR_W, hr + HR_ZH * HR_W + HR_ODD);
          ld4(nu, hr + HR_ZNU * HR_W, hr + HR_ZNU * HR_W + HR_ODD);
          ld4(mu1, hr + HR_ZMU * HR_W, hr + HR_ZMU * HR_W + HR_ODD);
          if (has_sz) ld4(s, hr + (HR_ZS + k - FPZ) * HR_W, hr + (HR_ZS + k - FPZ) * HR_W + HR_ODD);
          double fl4[4], fad[4], lz[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const double Vx = ln[j] - (fx[j] - (j ? fx[j - 1] : fxl));
            const double fR = h[j] * (V1[j] + Vx);
            const double dR = nu[j] * (Vx - V1[j]);
            const double vs = has_sz ? V1[j] + s[j] : V1[j];
            const double lo = vs - (fR - f1[j]);
            lz[j] = lo + (dR - d1[j]);
            fad[j] = mu1[j] * (lo - L2[j]);
            V1[j] = Vx;
            f1[j] = fR;
            d1[j] = dR;
            L2[j] = lo;
          }
          if (fin) {
#pragma unroll
            for (int j = 0; j < 4; ++j) fl4[j] = fct_limit_fin(A2[j], N3[j] - N4[j], N2[j] - N3[j], lz[j] - N2[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) fl4[j] = fct_limit_sel(A2[j], N3[j] - N4[j], N2[j] - N3[j], lz[j] - N2[j]);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            ov[j] = N3[j] - (fl4[j] - F3[j]);
            F3[j] = fl4[j];
            A2[j] = fad[j];
            N4[j] = lz[j];
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&co_free[gc & 1u]);
        ++gc;
        fl = fl == fl_last ? fl0 : fl + 12 * W;
        if (i >= 6) {  // row zs + i - 6 (YM_Fluid.cu:20-29: density floor, wall momentum)
          if (k == FN) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (ov[j] < 0.05) ov[j] = 0.05;
          }
          if (owner && dbg_ok(xo >= 0 && c.zs + i - 6 < c.ze, T.err)) {
            if (bulk) {  // nx even, rows 16-byte aligned
              *reinterpret_cast<double2*>(dst + xo) = make_double2(ov[0], ov[1]);
              if (xo + 2 < nx) *reinterpret_cast<double2*>(dst + xo + 2) = make_double2(ov[2], ov[3]);
            } else {
#pragma unroll
              for (int j = 0; j < 4; ++j)
                if (xo + j < nx) dst[xo + j] = (wall_x >= 0 && (xo + j == 0 || xo + j == wall_x)) ? 0.0 : ov[j];
            }
          }
          dst += nx;
        }
      };

      // row i staged and its coefficients written / row i read
      auto wait_row = [&] { mbar_wait(&co_full[gc & 1u], (gc >> 1) & 1u, T.err); };
      bool fin = true;
      for (int i = 0; i < nrow; ++i) {
        wait_row();
        if (fin) fin = row_is_finite();
        row(fin, i, Na, Nb, Nc);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double t = Na[j];
          Na[j] = Nb[j];
          Nb[j] = Nc[j];
          Nc[j] = t;
        }
      }
    }
  } else {
    // -------------------------------------------------- a coefficient warp: 32 positions, both beams
    asm volatile("setmaxnreg.dec.sync.aligned.u32 104;");
    const int htid = tid - F2_SWEEP * 32;
    const int q = htid;
    const int hq = hr_pos(q);
    unsigned gc = 0;        // rows handed over so far: coefficient slot and phase
    int s6 = 0, s4 = 0;     // ring slots of the next row
    const int q_next = q < W - 1 ? 1 : 0;  // the last position has no interface
    for (int item = i_beg; item < i_end;) {
      const Piece c = begin_piece(item);
      item = c.next;
      const int nx = p.nx, nz = p.nz, x0 = c.x0;
      const bool warm = c.warm, bulk = c.bulk, box = c.box;
      const int narr = 33 + (warm ? 4 : 0);
      // Evenly spaced arrays (box): a row is three TMA boxes (and four for
      // warm_T).  Past the edges of the grid they read zeros, so where the
      // window wraps, the four wrapped columns next to the edge (all that the
      // strip's outputs need: those before x = 0 in the first strip, from
      // x = nx in the last) come as three narrow boxes and are put in their
      // places when the row is there.  With warm_T such a strip copies row by row.
      const TensorMap* const maps = rd.maps;  // boxes of 12, 9 and 1 arrays; 4-wide boxes of 12 and 9 arrays
      if (box && htid == 0) tensormap_acquire<kFctMaps>(maps);
      const bool patch_l = x0 == 0, patch = box && c.edge;
      const int patch_q = patch_l ? 0 : nx - (x0 - 4);  // position of the first wrapped column
      if (!bulk) xtab[q] = stage_x(x0 - 4 + q, nx, p.periodic_x);
      // row copies of the piece: source array, its row (z, z-1, z+1), its place in the fluid or field ring
      if (htid < narr) {
        const int a = htid;
        const double* base;
        int dst, kind_row = 0;
        if (a < 12) {
          base = a < 6 ? st.a[a] : st.b[a - 6];
          dst = a;
        } else if (a < 33) {  // fields 0..11 of row z, 3..11 of row z-1
          dst = a - 12;
          base = st.f[dst < 12 ? dst : dst - 9];
          kind_row = dst < 12 ? 0 : 1;
        } else {
          const int w = a - 33;  // n at z+1 (A, B), n at z-1 (A, B)
          base = (w & 1) ? st.b[FN] : st.a[FN];
          dst = F2_NZP + w;
          kind_row = (w >> 1) ? 1 : 2;
        }
        int x = (x0 - 4) % nx;
        x = x < 0 ? x + nx : x;
        cpt[a].base = base + x;
        cpt[a].base0 = base;
        cpt[a].dst = dst;
        cpt[a].kind = kind_row;
        cpt[a].len1 = min(W, nx - x);
      }
      __syncthreads();
      const int r_first = c.zs - 3;
      const int nrow = c.ze - c.zs + 6;

      // requests row i of the piece (coefficient warps only)
      auto issue_row = [&](int i) {
        const unsigned g = seq + (unsigned)i;
        double* const fl = sfl + (size_t)(g % F2_NFL) * 12 * W;
        double* const fd = sfd + (size_t)(g % F2_NFD) * F2_FD * W;
        uint64_t* const bar = &bars[g % F2_NFL];
        const int zr = zclamp(r_first + i, nz);
        const int zm = (zr == 0) ? nz - 1 : zr - 1;
        const int zp = (zr == nz - 1) ? 0 : zr + 1;
        const bool rows_ok = dbg_ok(zr >= 0 && zr < nz && zm >= 0 && zm < nz && zp >= 0 && zp < nz, T.err);
        if (box) {
          if (htid == 0) {
            mbar_expect_tx(bar, (unsigned)((narr * W + (patch ? 33 * 4 : 0)) * 8));
            if (rows_ok) {
              if (patch) {
                double* const wr = wrap + (g % F2_NFD) * F2_WRAP;
                const int xw = patch_l ? nx - 4 : 0;
                box_g2s(wr, maps + 3, xw, zr, 12, bar);
                box_g2s(wr + 48, maps + 3, xw, zr, 0, bar);
                box_g2s(wr + 96, maps + 4, xw, zm, 3, bar);
              }
              box_g2s(fl, maps, x0 - 4, zr, 12, bar);
              box_g2s(fd, maps, x0 - 4, zr, 0, bar);
              box_g2s(fd + F2_EZM * W, maps + 1, x0 - 4, zm, 3, bar);
              if (warm) {
                box_g2s(fd + F2_NZP * W, maps + 2, x0 - 4, zp, 12, bar);
                box_g2s(fd + (F2_NZP + 1) * W, maps + 2, x0 - 4, zp, 18, bar);
                box_g2s(fd + F2_NZM * W, maps + 2, x0 - 4, zm, 12, bar);
                box_g2s(fd + (F2_NZM + 1) * W, maps + 2, x0 - 4, zm, 18, bar);
              }
            }
          }
        } else if (bulk) {
          // one row copy per thread, spread over the warps (lane-major)
          if (htid == 0) mbar_expect_tx(bar, (unsigned)(narr * W * 8));
          const int ca = lane * (F2_NT / 32 - F2_SWEEP) + warp - F2_SWEEP;
          if (ca < narr) {
            const RowCopy& c = cpt[ca];
            const int len1 = c.len1;
            if (rows_ok && dbg_ok(len1 > 0 && c.dst >= 0 && c.dst < (ca < 12 ? 12 : F2_FD), T.err)) {
              const size_t off = (size_t)(c.kind == 0 ? zr : (c.kind == 1 ? zm : zp)) * nx;
              double* const dst = (ca < 12 ? fl : fd) + c.dst * W;
              bulk_g2s(dst, c.base + off, (unsigned)len1 * 8u, bar);
              for (int done = len1; done < W;) {  // past the periodic wrap (more than once if nx < W)
                const int len = min(W - done, nx);
                bulk_g2s(dst + done, c.base0 + off, (unsigned)len * 8u, bar);
                done += len;
              }
            }
          }
        } else {
          const int x = xtab[htid];
          if (rows_ok && dbg_ok(x >= 0 && x < nx, T.err))
            for (int a = 0; a < narr; ++a) {
              const RowCopy& c = cpt[a];
              const size_t off = (size_t)(c.kind == 0 ? zr : (c.kind == 1 ? zm : zp)) * nx;
              cp_async8((a < 12 ? fl : fd) + c.dst * W + htid, c.base0 + off + x);
            }
          cp_async_commit();
        }
      };

      int ps = q;  // at a wall the clamped ghost cells carry the edge cell's px source
      if (c.wall) {
        const int xg = x0 - 4 + q;
        ps = (xg < 0 ? 0 : (xg >= nx ? nx - 1 : xg)) - (x0 - 4);
      }
      ps = max(1, min(W - 2, ps));  // positions 0 and 127 are not used
      const double dt = p.dt;
      const double dtdx = p.dt / p.dx;
      const double dtdz = p.dt / p.dz;
      double U1[2] = {0.0, 0.0}, mu1[2] = {0.0, 0.0}, S1[2][4];
#pragma unroll
      for (int b = 0; b < 2; ++b) S1[b][0] = S1[b][1] = S1[b][2] = S1[b][3] = 0.0;
      for (int i = 0; i < 4; ++i)
        if (i < nrow) issue_row(i);
        else if (!bulk) cp_async_commit();
      // element e of the wrapped columns: column e & 3 of array e >> 2
      auto patch_row = [&](double* fl, double* fd, const double* src) {
        for (int e = htid; e < 33 * 4; e += W) {
          const int a = e >> 2, x = patch_q + (e & 3);
          if (x < W) (a < 12 ? fl + a * W : fd + (a - 12) * W)[x] = src[e];
        }
        fence_proxy_async();  // the slots go back to TMA
      };
      for (int i = 0; i < nrow; ++i) {
        // row i staged
        if (bulk) {
          const unsigned b = (seq + (unsigned)i) % F2_NFL;
          mbar_wait(&bars[b], (phase_bits >> b) & 1u, T.err);
          phase_bits ^= 1u << b;
        } else {
          cp_async_wait<3>();
          coef_bar();
        }
        if (patch) {
          patch_row(sfl + s6 * (12 * W), sfd + s4 * (F2_FD * W), wrap + s4 * F2_WRAP);
          coef_bar();
        }
        const double* const fl = sfl + s6 * (12 * W) + q;
        const double* const fd = sfd + s4 * (F2_FD * W) + ps;
        s6 = s6 == F2_NFL - 1 ? 0 : s6 + 1;
        s4 = (s4 + 1) & (F2_NFD - 1);
        double* const ur = uxr + (gc & 1u) * (2 * W) + q;
        double* const hr0 = hlp + (gc & 1u) * (2 * HR_SIZE * HR_W) + hq;
        // velocities (YM_Fluid.cu:3-11); the x interface also needs the next position's
        double ux[2], vz[2];
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          velocities(max_sel(fl[(b * 6 + FN) * W], 0.05), fl[(b * 6 + FPX) * W], fl[(b * 6 + FPZ) * W], ux[b], vz[b]);
          ur[b * W] = ux[b];
        }
        // field averages at the cell, shared by both beams (YM_Fluid.cu:43-66, 99-102)
        double ex[3], by[3], ez[3], az[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double* e = fd + c * W;
          ex[c] = 0.5 * (e[F2_EX * W] + e[F2_EX * W - 1]);
          by[c] = 0.25 * (e[F2_BY * W] + e[F2_BY * W - 1] + e[F2_BYM * W] + e[F2_BYM * W - 1]);
          ez[c] = 0.5 * (e[F2_EZ * W] + e[F2_EZM * W]);
          az[c] = 0.5 * (e[F2_AZ * W] + e[F2_AZM * W]);
        }
        double sx[2], sz[2], sq[2][3];
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          const double q1 = fl[(b * 6 + FQ1) * W], q2 = fl[(b * 6 + FQ2) * W], q3 = fl[(b * 6 + FQ3) * W];
          sx[b] = -(q1 * (ex[0] + vz[b] * by[0]) + q2 * (ex[1] + vz[b] * by[1]) + q3 * (ex[2] + vz[b] * by[2]));
          sz[b] = -(q1 * (ez[0] - ux[b] * by[0]) + q2 * (ez[1] - ux[b] * by[1]) + q3 * (ez[2] - ux[b] * by[2]));
          const double av = p.alpha * vz[b];  // YM_Fluid.cu:103-107
          sq[b][0] = dt * (av * (q2 * az[2] - q3 * az[1]));
          sq[b][1] = dt * (av * (q3 * az[0] - q1 * az[2]));
          sq[b][2] = dt * (av * (q1 * az[1] - q2 * az[0]));
        }
        if (warm) {  // YM_Fluid.cu:71-80
#pragma unroll
          for (int b = 0; b < 2; ++b) {
            const double* nn = fl + (b * 6 + FN) * W + (ps - q);
            const double* nz_ = fd + (q - ps) + b * W;
            sx[b] -= p.warm_T * ((nn[1] - nn[-1]) / (2.0 * p.dx));
            sz[b] -= p.warm_T * ((nz_[F2_NZP * W] - nz_[F2_NZM * W]) / (2.0 * p.dz));
          }
        }
        coef_bar();  // every position's ux written, the row's fields read: its field slot is free
        // the coefficient slot free: every sweep warp is past row i-2, whose fluid slot row i+4 takes
        mbar_wait(&co_free[gc & 1u], ((gc >> 1) & 1u) ^ 1u, T.err);
        if (i + 4 < nrow) issue_row(i + 4);
        else if (!bulk) cp_async_commit();
        double size = 0.0;  // of everything handed to the sweep warps
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          double* const hr = hr0 + b * (HR_SIZE * HR_W);
          const double e = fct_eps(ux[b], ur[b * W + q_next], dtdx);
          double nu, mu;
          fct_nu_mu(e, nu, mu);
          hr[HR_XH * HR_W] = 0.5 * e;
          hr[HR_XNU * HR_W] = nu;
          size += nu;
          const double ezi = fct_eps(U1[b], vz[b], dtdz);
          fct_nu_mu(ezi, nu, mu);
          hr[HR_ZH * HR_W] = 0.5 * ezi;
          hr[HR_ZNU * HR_W] = nu;
          hr[HR_ZMU * HR_W] = mu1[b];
          size += nu;
          U1[b] = vz[b];
          mu1[b] = mu;
          sx[b] = dt * sx[b];
          sz[b] = dt * sz[b];
          hr[HR_XS * HR_W] = sx[b];
#pragma unroll
          for (int v = 0; v < 4; ++v) hr[(HR_ZS + v) * HR_W] = S1[b][v];
          S1[b][0] = sz[b];
          S1[b][1] = sq[b][0];
          S1[b][2] = sq[b][1];
          S1[b][3] = sq[b][2];
          size += fabs(sx[b]) + fabs(sz[b]);
          size += (fabs(sq[b][0]) + fabs(sq[b][1])) + fabs(sq[b][2]);
        }
        if (!(size < F2_BIG)) s_bad = 1;
        __syncwarp();
        if (lane == 0) mbar_arrive(&co_full[gc & 1u]);
        ++gc;
      }
      if (!bulk) {  // the next piece may take the slots by TMA
        cp_async_wait<0>();
        if (T.nruns > 1) fence_proxy_async();  // (a run keeps to one kind of copy)
      }
      seq += (unsigned)nrow;
    }
  }
}

template <int TB, int NST>
static cudaError_t prepare_fct_t() {
  return cudaFuncSetAttribute(fct_fused_kernel<TB, NST>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)fct_smem_bytes<TB>(NST));
}

// Stage ring depth of fct_fused_kernel (rows in flight = NST - 1): with four
// stages two CTAs of 64-wide strips fit an SM's shared memory, with five one.
template <int TB>
constexpr int fct_nst() {
  return 4;
}

int fct_nstrips(int nx, int tb) {
  const int out = tb == 128 ? F2_O : tb - 6;
  return (nx + out - 1) / out;
}

int fct_bulk_ok(const StepParams& p, int tb) {
  return (p.periodic_x && (p.nx % 2) == 0 && (tb == 128 || p.nx >= tb + 2)) ? 1 : 0;
}

// The kernel reads start-of-step values across strip and segment halos while
// other CTAs write theirs, so each run's fluid goes to its second buffer
// (`out`); fields are only read.  grid_ctas persistent CTAs take contiguous
// blocks of the flattened (run, strip, segment) items, T.fct_first's.
cudaError_t launch_fct_table(const RunTable& T, int tb, int grid_ctas, cudaStream_t s) {
  const int grid = std::max(1, std::min(T.fct_items, grid_ctas));
  switch (tb) {
    case 32: fct_fused_kernel<32, fct_nst<32>()><<<grid, 128, fct_smem_bytes<32>(fct_nst<32>()), s>>>(T); break;
    case 64: fct_fused_kernel<64, fct_nst<64>()><<<grid, 256, fct_smem_bytes<64>(fct_nst<64>()), s>>>(T); break;
    case 128: fct_strip_kernel<<<grid, F2_NT, fct_strip_smem_bytes(), s>>>(T); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t prepare_fct(int tb) {
  switch (tb) {
    case 32: return prepare_fct_t<32, fct_nst<32>()>();
    case 64: return prepare_fct_t<64, fct_nst<64>()>();
    case 128:
      return cudaFuncSetAttribute(fct_strip_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fct_strip_smem_bytes());
    default: return cudaErrorInvalidValue;
  }
}

int fct_ctas_per_sm(int tb) {
  int n = 0;
  switch (tb) {
    case 32: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fct_fused_kernel<32, fct_nst<32>()>, 128, fct_smem_bytes<32>(fct_nst<32>())); break;
    case 64: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fct_fused_kernel<64, fct_nst<64>()>, 256, fct_smem_bytes<64>(fct_nst<64>())); break;
    case 128: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fct_strip_kernel, F2_NT, fct_strip_smem_bytes()); break;
    default: break;
  }
  return n;
}

}  // namespace ymkh
