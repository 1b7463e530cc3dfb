// Fused FP64 steps of the mixed-precision defect-correction loop.
//
// One pass over level 1 computes the FP64 residual r = b - A x with the
// same per-cell arithmetic as the residual operator, and in the same pass
//   * accumulates sum(msk r^2) and sum(msk r) per block (FP64; fixed
//     block-to-cell assignment, so the reduction is deterministic),
//   * writes the FP32 right-hand side of the correction equation,
//     (float)(r * scale), where scale is a power of two taken from the
//     previous residual norm (its only job is to keep FP32 far from
//     under- and overflow; exact in both directions).
// For the vertex-centred (Dirichlet) operator that is the whole FP64 work
// of an iteration besides the update x += e / scale. For the cell-centred
// (Neumann) operator the wet mean must come off first: the pass also keeps
// r in FP64 and a second pass writes the mean-free FP32 right-hand side.
#include <algorithm>

#include "ops_dev.cuh"

namespace cfmg {


// per-block partial sums -> 2 * kMxParts doubles: [sum r^2 | sum r]. With
// NEUMANN the FP64 r is kept for the mean-removing pass and sum r is
// Neumaier-compensated per thread; else the scaled FP32 right-hand side is
// written here and r64 is not stored.
template <int KIND, bool NEUMANN>
__global__ void __launch_bounds__(kMxThreads) k_resid_fused(double* __restrict__ r, const double* __restrict__ x,
                                                            const double* __restrict__ b, const double* __restrict__ d,
                                                            const uint8_t* __restrict__ m, Geom g, Box bx,
                                                            long long lo, long long n, const double* __restrict__ ds,
                                                            float* __restrict__ b32, float* __restrict__ r32,
                                                            double* __restrict__ partials) {
  dep_wait();
  const double scale = ds[0];
  double s2 = 0.0, s1 = 0.0, c1 = 0.0;
  const long long ni = bx.i1 - bx.i0 + 1, nj = bx.j1 - bx.j0 + 1;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    long long I;
    if (KIND == OPK_RESID9 || KIND == OPK_RESID7 || KIND == OPK_RESID19) {
      const int i = bx.i0 + (int)(t % ni);
      const long long q = t / ni;
      const int j = bx.j0 + (int)(q % nj);
      const int k = bx.k0 + (int)(q / nj);
      I = lin(g, i, j, k);
    } else {
      I = lo + t;
    }
    double v;
    if (KIND == OPK_RESID5) v = v_resid5(x, b, d, m, g.n1, I);
    else if (KIND == OPK_RESID9) v = v_resid9(x, b, d, m, g.n1, I);
    else if (KIND == OPK_RESID7) v = v_resid7(x, b, d, m, g.n1, g.n2, I);
    else v = v_resid19(x, b, d, m, g.n1, g.n2, I);
    s2 = __fma_rn(v, v, s2);  // v is a signed zero on dry cells
    if (NEUMANN) {
      r[I] = v;
      const double tt = __dadd_rn(s1, v);
      c1 = __dadd_rn(c1, (fabs(s1) >= fabs(v)) ? __dadd_rn(__dsub_rn(s1, tt), v) : __dadd_rn(__dsub_rn(v, tt), s1));
      s1 = tt;
    } else {
      const float f = (float)(v * scale);
      b32[I] = f;
      r32[I] = f;
    }
  }
  s1 = __dadd_rn(s1, c1);
  __shared__ double sh2[kMxThreads / 32], sh1[kMxThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s2 += __shfl_down_sync(0xffffffffu, s2, o);
    s1 += __shfl_down_sync(0xffffffffu, s1, o);
  }
  if ((threadIdx.x & 31) == 0) {
    sh2[threadIdx.x >> 5] = s2;
    sh1[threadIdx.x >> 5] = s1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0, c = 0.0;
    for (int w = 0; w < kMxThreads / 32; ++w) {
      a += sh2[w];
      c += sh1[w];
    }
    partials[blockIdx.x] = a;
    partials[kMxParts + blockIdx.x] = c;
  }
}

// Final reduction into the handle's scalars: S_NORM = sum msk r^2 (0 -> 1
// for the reference rule), S_RES = the residual ratio against *normb,
// S_MEAN2 = wet mean of r (when nwet is given). The scale the pass just
// applied (S_NEXT on entry) becomes S_CUR / S_ICUR, and the next scale
// 2^-round(log2(rms)) goes to S_NEXT (powers of two, exact both ways).
__global__ void __launch_bounds__(kMxParts) k_fused_final(const double* __restrict__ partials, double* ds,
                                                          const double* normb, const double* nwet, int norm_kind,
                                                          LoopTest lt, int q) {
  dep_wait();
  __shared__ double a[kMxParts], c[kMxParts];
  __shared__ __int128 ci[kMxParts];
  const bool exact = q != kFloatSums;
  a[threadIdx.x] = partials[threadIdx.x];
  c[threadIdx.x] = partials[kMxParts + threadIdx.x];
  if (exact)
    ci[threadIdx.x] = (__int128)(((unsigned __int128)(unsigned long long)__double_as_longlong(
                                      partials[2 * kMxParts + threadIdx.x])
                                  << 64) |
                                 (unsigned long long)__double_as_longlong(c[threadIdx.x]));
  __syncthreads();
  for (int w = kMxParts / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) {
      a[threadIdx.x] += a[threadIdx.x + w];
      if (exact) ci[threadIdx.x] += ci[threadIdx.x + w];
      else c[threadIdx.x] += c[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    double sum = a[0];
    const double raw = sum;
    if (norm_kind == CFMG_NORM_REF_SQUARED) {
      if (sum == 0.0) sum = 1.0;
      ds[S_NORM] = sum;
      ds[S_RES] = (*normb > 0.0) ? sum / *normb : 0.0;
    } else {
      ds[S_NORM] = sum;
      ds[S_RES] = (*normb > 0.0) ? sqrt(sum / *normb) : 0.0;
    }
    const double nw = (nwet && *nwet > 0) ? *nwet : 1.0;
    const double s1 = exact ? ldexp(int_to_double(ci[0]), -(fix_exponent(ds) + q)) : c[0];
    ds[S_MEAN2] = nwet ? s1 / nw : 0.0;
    const double used = ds[S_NEXT];
    ds[S_CUR] = used;
    ds[S_ICUR] = 1.0 / used;
    const double rms = sqrt(raw / (nwet && *nwet > 0 ? *nwet : 1.0));
    int e = 0;
    if (rms > 0 && isfinite(rms)) frexp(rms, &e);
    ds[S_NEXT] = ldexp(1.0, -e);
    ds[S_MAXX] = ds[S_MAXO];  // the next update collects max |x| from max |x| outside U
    // the wet mean in units of the right-hand side, as an FP32 value
    *reinterpret_cast<float*>(ds + S_SHIFT) = (float)(ds[S_MEAN2] * used);
    if (lt.on) loop_test(lt, ds[S_RES], *normb);
  }
}

// The FP32 right-hand side (r - mean) * scale on wet cells, four cells a
// thread with their loads in flight. The FP64 pipe bounds it: the conversion
// is done by integer operations, which leaves that pipe two of three a cell
// (2048^2: 26 us with all three; 15.2 now). r32: where the cycle reads it.
__global__ void __launch_bounds__(256) k_rhs32(const double* __restrict__ r, const uint8_t* __restrict__ m,
                                               const double* __restrict__ mean_at,
                                               const double* __restrict__ scale_at, float* __restrict__ b32,
                                               float* __restrict__ r32, long long n) {
  dep_wait();
  const double mean = *mean_at, scale = *scale_at;
  const long long I0 = (long long)blockIdx.x * 1024 + threadIdx.x;
  double v[4];
  bool wet[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const long long I = I0 + 256 * q;
    wet[q] = I < n && m[I] != 0;
    v[q] = I < n ? r[I] : 0.0;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const long long I = I0 + 256 * q;
    const float f = wet[q] ? d2f(__dmul_rn(__dsub_rn(v[q], mean), scale)) : 0.f;
    if (I < n) {
      b32[I] = f;
      if (r32) r32[I] = f;
    }
  }
}

// x += e * iscale (the FP64 solution update), four cells a thread: e is
// converted by integer operations, which leaves the FP64 pipe the FMA and the
// pass its memory traffic (2048^2: 18.3 us with the conversion on that pipe,
// 12.2 now)
__global__ void __launch_bounds__(256) k_update_scaled(double* __restrict__ x, const float* __restrict__ e,
                                                       const double* __restrict__ iscale, long long n) {
  dep_wait();
  const double is = *iscale;
  const long long I0 = (long long)blockIdx.x * 1024 + threadIdx.x;
  double v[4];
  float d[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const long long I = I0 + 256 * q;
    v[q] = I < n ? x[I] : 0.0;
    d[q] = I < n ? e[I] : 0.f;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const long long I = I0 + 256 * q;
    if (I < n) x[I] = __fma_rn(f2d_pow2(d[q], 0, 1.0), is, v[q]);
  }
}

// ----------------------------------------------------------------------
// Integer form of the fused pass. The FP64 pipe of a GB300 runs at 1/64 of
// the FP32 rate, and the FP64 stencil arithmetic above keeps it busy
// (about 13 FP64 operations a cell). Here x and b are read as FP64 but
// converted with integer operations to 64-bit fixed point, v * 2^k rounded
// to an integer, with k = 58 - E for max(|x|, |b|) < 2^E (S_MAXX, S_MAXB).
// The residual Q*r = Q*(diag*x + b) - (stencil sum), with Q = 4 for the
// 9-point weights 1/2 and 1/4 and Q = 1 otherwise, is then an exact
// integer (|Q r| 2^k < 2^63), so it carries no rounding at all: its error
// is that of representing x on the 2^-k grid, below 2^-58 max|x| per cell
// (FP64 arithmetic on the same x rounds at 2^-53 |x| per operation). The
// FP64 pipe is left with two conversions and one FMA a cell: sum r^2 in
// FP64 and the FP32 right-hand side. The cell-centred sum r is kept exact
// in 128-bit integers per thread.
//
// dq[I] = Q*diag[I] (an integer in 0..127) on wet cells, -128 on dry ones.

template <int KIND>
__device__ __forceinline__ long long fix_resid(const double* __restrict__ x, const double* __restrict__ b, int dq,
                                               int k, long long n1, long long n2, long long I) {
  if (dq < 0) return 0;
  const long long X = to_fix(x[I], k), B = to_fix(b[I], k);
  if (KIND == OPK_RESID9) {
    const long long F = to_fix(x[I - 1], k) + to_fix(x[I + 1], k) + to_fix(x[I - n1], k) + to_fix(x[I + n1], k);
    const long long D = to_fix(x[I - 1 - n1], k) + to_fix(x[I + 1 - n1], k) + to_fix(x[I - 1 + n1], k) +
                        to_fix(x[I + 1 + n1], k);
    return (long long)dq * X + 4 * B - 2 * F - D;
  } else if (KIND == OPK_RESID7) {
    const long long F = to_fix(x[I - 1], k) + to_fix(x[I + 1], k) + to_fix(x[I - n1], k) + to_fix(x[I + n1], k) +
                        to_fix(x[I - n2], k) + to_fix(x[I + n2], k);
    return (long long)dq * X + B - F;
  } else {
    const long long F = to_fix(x[I - 1], k) + to_fix(x[I + 1], k) + to_fix(x[I - n1], k) + to_fix(x[I + n1], k);
    return (long long)dq * X + B - F;
  }
}

// per-block partial sums: partials[blk] = sum r^2, partials[kMxParts + blk]
// = sum r. NEUMANN: b32 = (float)(r * scale) here, the mean comes off in a
// second pass (which also writes r32); else b32 and, when r32 != nullptr,
// r32 get the right-hand side.
template <int KIND, bool NEUMANN>
__global__ void __launch_bounds__(kMxThreads) k_resid_int(const double* __restrict__ x, const double* __restrict__ b,
                                                          const int8_t* __restrict__ dq, Geom g, Box bx, long long lo,
                                                          long long n, const double* __restrict__ ds,
                                                          float* __restrict__ b32, float* __restrict__ r32,
                                                          double* __restrict__ partials) {
  dep_wait();
  constexpr int q = (KIND == OPK_RESID9) ? 2 : 0;  // Q = 2^q
  const int k = fix_exponent(ds);
  const float fm = (float)ldexp(ds[S_NEXT], -(k + q));  // power of two: R -> r * scale
  double s2 = 0.0;
  __int128 s1 = 0;
  const long long ni = bx.i1 - bx.i0 + 1, nj = bx.j1 - bx.j0 + 1;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    long long I;
    if (KIND == OPK_RESID5) {
      I = lo + t;
    } else {
      const int i = bx.i0 + (int)(t % ni);
      const long long qq = t / ni;
      I = lin(g, i, bx.j0 + (int)(qq % nj), bx.k0 + (int)(qq / nj));
    }
    const long long R = fix_resid<KIND>(x, b, dq[I], k, g.n1, g.n2, I);
    const double rd = __ll2double_rn(R);
    s2 = __fma_rn(rd, rd, s2);
    const float f = __fmul_rn(__ll2float_rn(R), fm);
    b32[I] = f;
    if (NEUMANN) s1 += (__int128)R;
    else if (r32) r32[I] = f;
  }
  int_partials<KIND == OPK_RESID7>(s2, s1, -2 * (k + q), k + q, partials);
}

// Strips of rows (2D, and 3D plane by plane): the same residual with every
// x converted once. A warp owns 30 consecutive linear indices of a row
// (lanes 1..30; lanes 0 and 31 hold the values on either side, which at the
// ends of a row are the wrap-around neighbours of the linear 5-point range)
// and walks down `rows` rows, keeping each converted row's centre and
// west + east sum in registers; the west and east values come from the
// adjacent lanes. Integer sums are exact, so each row's west + east sum
// serves as the start of its faces (as centre row) and of the diagonals of
// the rows above and below. The loop body covers 6 rows, so the rotation of
// the row window (period 3) costs no moves. x, b and dq come through a ring in
// shared memory that each lane fills for itself with asynchronous copies, three
// rows ahead: loads into registers that far ahead waited for one another on the
// few scoreboards a warp has, and the one-byte loads of dq, a row ahead, held
// each row up (4096^2: 114 us with those, 107 now, 99 without dq at all). The
// residual norm is summed from the FP32 right-hand-side values f = r*scale
// (exact squares via FMA, double-float accumulation per thread, FP64
// across threads), so the FP64 pipe does one conversion a cell. The grid is
// one wave of warps, each taking several equal tasks.
//
// x is the level-1 array of the handle's arena. The lanes around the index
// space read up to 31 elements before its start and after its end, into the
// device scalars before it and into y after it; those values are not used.
constexpr int kIntCols = 30;  // output columns per warp strip
static_assert(kIntCols + 1 < kResidIntReach, "a warp reaches kIntCols + 1 columns beyond its strip's first");
constexpr int kIntUnroll = 6;  // rows per loop body; rows per task is a multiple
constexpr int kIntRing = 3;    // rows in flight; a ring of kIntRing + 1 slots (a power of two)

struct StripSpace {
  long long len;   // array length
  long long row0;  // linear index of column 0 of the first row (of the first plane)
  long long n2;    // plane stride (7-point: the k +- 1 neighbours)
  int nplanes;     // planes of the index space (1 in 2D)
  int c0, ncols;   // columns of the index space: c0 .. c0+ncols-1 (0-based linear offsets in a row)
  int nrows;       // rows of the index space
  int nstrips;     // ceil(ncols / kIntCols)
  int rows;        // rows per warp task (a multiple of kIntUnroll)
  long long n1;
};

// sflag (optional): 1 for each (plane, row, strip) whose 30 columns hold a
// wet cell; a task whose rows are all dry in its strip is skipped (its b32 is
// +0 already, its residuals would add exact zeros to the sums).
template <int KIND, bool NEUMANN>
__global__ void __launch_bounds__(kMxThreads) k_resid_int2d(const double* __restrict__ x, const double* __restrict__ b,
                                                            const int8_t* __restrict__ dq, StripSpace sp,
                                                            const double* __restrict__ ds, float* __restrict__ b32,
                                                            float* __restrict__ r32, double* __restrict__ partials,
                                                            const uint8_t* __restrict__ sflag) {
  dep_wait();
  constexpr int q = (KIND == OPK_RESID9) ? 2 : 0;  // Q = 2^q
  const int k = fix_exponent(ds);
  const double scale = ds[S_NEXT];
  const float fm = (float)ldexp(scale, -(k + q));  // power of two: R -> r * scale
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const int nchunks = (sp.nrows + sp.rows - 1) / sp.rows;
  const long long per_plane = (long long)sp.nstrips * nchunks;
  const long long ntasks = per_plane * sp.nplanes;
  const long long n1 = sp.n1;
  __shared__ double2 ring[kMxThreads / 32][kIntRing + 1][32];
  __shared__ int dring[kMxThreads / 32][kIntRing + 1][32];
  float hi = 0.f, lo = 0.f;  // double-float sum of f^2
  __int128 s1 = 0;
  for (long long task = warp0; task < ntasks; task += nwarps) {
    const int plane = (int)(task / per_plane);
    const long long pt = task - plane * per_plane;
    const int strip = (int)(pt % sp.nstrips);
    const int chunk = (int)(pt / sp.nstrips);
    // lanes 1..30 own the strip's 30 columns; lanes 0 and 31 hold the
    // columns on either side, so every x is converted by exactly one lane
    const int c = sp.c0 + strip * kIntCols + lane - 1;  // this lane's column
    const bool col_ok = lane >= 1 && lane <= kIntCols && c < sp.c0 + sp.ncols;
    const int ra = chunk * sp.rows, rb = min(ra + sp.rows, sp.nrows);
    if (sflag) {  // warp-uniform: the task's rows of this strip, a lane a row
      unsigned any = 0;
      for (int r = ra + lane; r < rb; r += 32) any |= sflag[((long long)plane * sp.nrows + r) * sp.nstrips + strip];
      if (!__any_sync(0xffffffffu, any != 0)) continue;
    }
    const long long I0 = sp.row0 + plane * sp.n2 + (long long)ra * n1 + c;  // row ra, this lane
    const double* xp = x + I0;
    // rows ra-1 and ra converted; x of rows ra+1, ra+2 and b, dq of row ra in flight
    long long Cm = to_fix(xp[-n1], k), C0 = to_fix(xp[0], k);
    long long rsm = __shfl_up_sync(0xffffffffu, Cm, 1) + __shfl_down_sync(0xffffffffu, Cm, 1);
    long long rs0 = __shfl_up_sync(0xffffffffu, C0, 1) + __shfl_down_sync(0xffffffffu, C0, 1);
    // copy j: x of row ra+1+j, b of row ra+j and the word that holds its dq, into slot j of the lane's ring
    auto request = [&](int j) {
      const long long I = I0 + (long long)j * n1;
      double2* at = &ring[threadIdx.x >> 5][j & kIntRing][lane];
      if (ra + j < rb) {
        cp_async<8>(&at->x, x + I + n1);
        if (col_ok) {
          cp_async<8>(&at->y, b + I);
          cp_async<4>(&dring[threadIdx.x >> 5][j & kIntRing][lane], dq + (I & ~3LL));
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int j = 0; j < kIntRing; ++j) request(j);
    double za = 0.0, zb = 0.0;  // 7-point: x of the planes below and above, row ra
    if (KIND == OPK_RESID7 && col_ok) {
      za = xp[-sp.n2];
      zb = xp[sp.n2];
    }
    // one row of the strip (r < rb): the rotation of the row window is the
    // last step, so in the unguarded 6-row groups it costs no register moves
    auto row_step = [&](int r) {
      const long long I = I0 + (long long)(r - ra) * n1;
      // row r+1 converted; the rows kIntRing further on requested
      asm volatile("cp.async.wait_group %0;" ::"n"(kIntRing - 1) : "memory");
      const double2 v = ring[threadIdx.x >> 5][(r - ra) & kIntRing][lane];
      const int dw = dring[threadIdx.x >> 5][(r - ra) & kIntRing][lane];
      request(r - ra + kIntRing);
      const long long Cp = to_fix(v.x, k);
      const long long rsp = __shfl_up_sync(0xffffffffu, Cp, 1) + __shfl_down_sync(0xffffffffu, Cp, 1);
      const double cb = v.y, clo = za, chi = zb;
      const int d = col_ok ? (dw << (24 - 8 * (int)(I & 3))) >> 24 : -1;
      if (r + 1 < rb) {
        if (KIND == OPK_RESID7 && col_ok) {
          za = x[I + n1 - sp.n2];
          zb = x[I + n1 + sp.n2];
        }
      }
      const long long B = to_fix(cb, k);
      long long R;
      if (KIND == OPK_RESID9)
        R = (long long)d * C0 + 4 * B - 2 * (rs0 + Cm + Cp) - (rsm + rsp);
      else if (KIND == OPK_RESID7)
        R = (long long)d * C0 + B - (rs0 + Cm + Cp + to_fix(clo, k) + to_fix(chi, k));
      else
        R = (long long)d * C0 + B - (rs0 + Cm + Cp);
      R = d >= 0 ? R : 0LL;  // dry cells and lanes outside the strip
      const float f = __fmul_rn(__ll2float_rn(R), fm);
      if (col_ok) {
        b32[I] = f;
        if (!NEUMANN && r32) r32[I] = f;
      }
      if (NEUMANN) s1 += (__int128)R;
      // p + e = f^2 exactly; (hi, lo) += p + e by TwoSum (explicit _rn
      // operations: a contracted hi + f*f would break the error terms);
      // f = 0 outside the strip adds exactly nothing
      const float p = __fmul_rn(f, f), e = __fmaf_rn(f, f, -p);
      const float sn = __fadd_rn(hi, p), bp = __fsub_rn(sn, hi);
      lo = __fadd_rn(lo, __fadd_rn(__fadd_rn(__fsub_rn(hi, __fsub_rn(sn, bp)), __fsub_rn(p, bp)), e));
      hi = sn;
      Cm = C0; rsm = rs0;
      C0 = Cp; rs0 = rsp;
    };
    int r0 = ra;
    for (; r0 + kIntUnroll <= rb; r0 += kIntUnroll) {
#pragma unroll
      for (int u = 0; u < kIntUnroll; ++u) row_step(r0 + u);
    }
    for (; r0 < rb; ++r0) row_step(r0);
  }
  // sum f^2 -> sum r^2 = sum f^2 / scale^2 (exact power of two)
  int_partials<KIND == OPK_RESID7>(((double)hi + (double)lo) / (scale * scale), s1, 0, k + q, partials);
}

template <int KIND, bool NEUMANN>
static int int2d_grid() {
  // one wave: resident blocks per SM x SMs, at most kMxParts; made by one thread
  // (another that saw it before the cut launched more blocks than there are partials)
  static const int blocks = [] {
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_resid_int2d<KIND, NEUMANN>, kMxThreads, 0);
    return std::min(kMxParts, sm_count() * std::max(per, 1));
  }();
  return blocks;
}

// the strips of the 2D (and 3D strip-form) residual: false when the form
// does not apply
static bool strip_space(int kind, const Geom& g, const Box& bx, StripSpace& sp) {
  sp.n1 = g.n1;
  sp.n2 = g.n2;
  sp.len = g.len;
  sp.nplanes = 1;
  if (kind == OPK_RESID7) {  // interior box ic x jc x kc (rloop3d!)
    sp.row0 = (long long)(bx.j0 - 1) * g.n1 + (long long)(bx.k0 - 1) * g.n2;
    sp.c0 = bx.i0 - 1;
    sp.ncols = bx.i1 - bx.i0 + 1;
    sp.nrows = bx.j1 - bx.j0 + 1;
    sp.nplanes = bx.k1 - bx.k0 + 1;
  } else if (g.tz != 1) {
    return false;
  } else if (kind == OPK_RESID5) {  // linear range 1+n1 .. len-n1: rows 2..ty-1, every column
    sp.row0 = g.n1;
    sp.c0 = 0;
    sp.ncols = g.tx;
    sp.nrows = g.ty - 2;
  } else if (kind == OPK_RESID9) {  // interior box of the single layer
    sp.row0 = (long long)(bx.j0 - 1) * g.n1;
    sp.c0 = bx.i0 - 1;
    sp.ncols = bx.i1 - bx.i0 + 1;
    sp.nrows = bx.j1 - bx.j0 + 1;
  } else {
    return false;
  }
  if (sp.nrows <= 0 || sp.ncols <= 0 || sp.nplanes <= 0) return false;
  sp.nstrips = (sp.ncols + kIntCols - 1) / kIntCols;
  return true;
}

bool launch_resid_int2d(int kind, const double* x, const double* b, const int8_t* dq, const Geom& g, const Box& bx,
                        const double* ds, float* b32, float* r32, bool neumann, double* partials, cudaStream_t s,
                        const uint8_t* sflag) {
  StripSpace sp;
  if (!strip_space(kind, g, bx, sp)) return false;
#define CFMG_INT2(K)                                                                                        \
  if (kind == K) {                                                                                          \
    const int grid = neumann ? int2d_grid<K, true>() : int2d_grid<K, false>();                             \
    /* about 4 tasks per warp of the wave, 6 to 96 rows each */                                             \
    const long long warp_rows = (long long)sp.nstrips * sp.nrows * sp.nplanes;                              \
    long long rows = warp_rows / (4LL * grid * (kMxThreads / 32));                                          \
    rows = rows < kIntUnroll ? kIntUnroll : (rows > 96 ? 96 : rows);                                        \
    sp.rows = (int)((rows + kIntUnroll - 1) / kIntUnroll * kIntUnroll);                                     \
    if (neumann)                                                                                            \
      launch_dep(k_resid_int2d<K, true>, grid, kMxThreads, 0, s, x, b, dq, sp, ds, b32, r32, partials, sflag);      \
    else                                                                                                    \
      launch_dep(k_resid_int2d<K, false>, grid, kMxThreads, 0, s, x, b, dq, sp, ds, b32, r32, partials, sflag);     \
    return true;                                                                                            \
  }
  CFMG_INT2(OPK_RESID5)
  CFMG_INT2(OPK_RESID9)
  CFMG_INT2(OPK_RESID7)
#undef CFMG_INT2
  return false;
}

// ---- wet sum of r for the operators without a fused pass (variable
// coefficient, x-periodic), per block into partials[kNormParts]. Each r is
// taken to fixed point with 94 bits below the bound |r| <= sqrt(sum r^2) that
// the norm just gave (ds[S_NORM]) and added exactly in 128-bit integers: an r
// above 2^-41 of the bound keeps all its bits, a smaller one loses less than
// 2^-94 of it. A thread's sum is then right to the last bit of a double, as
// the compensated FP64 sum that this replaces was (with 58 bits it was off by
// up to 2^-59 of the bound a cell, which is sqrt(n) times the rms of r). That
// sum issued six FP64 operations a cell: 66 us at 2048^2 against 15.
// v 2^k for |v| 2^k < 2^95, towards zero; zero and subnormal v give 0 (k <= 1022)
__device__ __forceinline__ __int128 to_fix_wide(double v, int k) {
  const int hi = __double2hiint(v);
  const unsigned lo = (unsigned)__double2loint(v);
  const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
  const int n = min(max(1117 - k - (int)(((unsigned)hi << 1) >> 21), 0), 127);
  // the significand, 42 bits up
  const unsigned long long top = __funnelshift_l(lo, mh, 10), low = (unsigned long long)(lo << 10) << 32;
  const __int128 m = (__int128)((((unsigned __int128)top << 64) | low) >> n);
  return hi < 0 ? -m : m;
}
__global__ void __launch_bounds__(256) k_mean_fix(const double* __restrict__ r, const uint8_t* __restrict__ m,
                                                  long long n, const double* __restrict__ ds,
                                                  double* __restrict__ partials) {
  dep_wait();
  int e2 = 0;
  const double sq = ds[S_NORM];
  if (sq > 0 && isfinite(sq)) frexp(sq, &e2);  // sum r^2 < 2^e2
  const int k = 94 - ((e2 + 1) >> 1);
  __int128 s = 0;
  const long long st = (long long)kNormParts * 256;
  long long I = (long long)blockIdx.x * 256 + threadIdx.x;
  for (; I + 3 * st < n; I += 4 * st) {  // four cells' loads in flight
    const double v0 = r[I], v1 = r[I + st], v2 = r[I + 2 * st], v3 = r[I + 3 * st];
    const uint8_t m0 = m[I], m1 = m[I + st], m2 = m[I + 2 * st], m3 = m[I + 3 * st];
    if (m0) s += to_fix_wide(v0, k);
    if (m1) s += to_fix_wide(v1, k);
    if (m2) s += to_fix_wide(v2, k);
    if (m3) s += to_fix_wide(v3, k);
  }
  for (; I < n; I += st)
    if (m[I]) s += to_fix_wide(r[I], k);
  double v = int_to_double(s);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  __shared__ double sh[8];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0;
    for (int w = 0; w < 8; ++w) a += sh[w];
    partials[blockIdx.x] = ldexp(a, -k);
  }
}
void launch_mean_fix(const double* r, const uint8_t* m, long long n, const double* ds, double* partials,
                     cudaStream_t s) {
  launch_dep(k_mean_fix, kNormParts, 256, 0, s, r, m, n, ds, partials);
}

// ---- 3D 19-point form. A block owns a 32 x 8 column tile of the interior box
// and marches along k. Each x of the tile and its one-cell rim is converted
// once into shared memory (340 conversions for 256 cells); a thread reads its
// 3 x 3 neighbourhood there and keeps, per plane, the cell C, its four faces
// F and its four diagonals D. The 19-point sum at plane k needs no more than
//   faces = F(k) + C(k-1) + C(k+1),  edges = D(k) + F(k-1) + F(k+1),
// exact in any order, so the planes k -+ 1 come from registers: 9 shared loads
// and 11 additions of 64-bit integers a cell, where the FP64 form
// (k_resid_fused) issues 21 FP64 operations on a pipe 1/64 as fast. The next
// plane's x, b and dq are loaded before this plane is summed; two tile
// buffers, so one barrier a plane. The sum of 52 |x| Q weights reaches
// 52 * 2^57, so the grid is one bit coarser (k = 57 - E) than the 2D forms'.
// Tasks (tile, run of planes) are dealt to one wave of blocks; the run length
// is the one with the least planes for the busiest block, two rim planes a
// task counted. sum r^2 is taken in FP64 from the exact R (two FP64-pipe
// instructions a cell), as exactly as the FP64 form's. An x or b far below the
// largest holds fewer bits here than as a double, but nothing is rounded after:
// against exact arithmetic r is off by 0.6e-16 to 0.8e-16 in the rms and 2.5e-16
// at most where the FP64 form is off by 1.7e-16 to 3.2e-16 and 1.3e-15 to 2.5e-15
// (balls of 48 x 48 x 32 to 96 x 96 x 48, after 1 to 12 cycles; |b| about 1). At
// 192 x 192 x 128: 56 us (cold) against 255-270 us for the FP64 form.
constexpr int kR19W = 32, kR19H = 8, kR19Rim = (kR19W + 2) * (kR19H + 2);
template <bool NEUMANN>
__global__ void __launch_bounds__(kMxThreads, 4) k_resid_int19(const double* __restrict__ x,
                                                               const double* __restrict__ b,
                                                               const int8_t* __restrict__ dq, Geom g, Box bx,
                                                               const double* __restrict__ ds, float* __restrict__ b32,
                                                               float* __restrict__ r32, double* __restrict__ partials,
                                                               int nti, int ntj, int nch, int run) {
  dep_wait();
  __shared__ long long T[2][kR19H + 2][kR19W + 2];
  constexpr int q = 2;  // Q = 4
  const int k = fix_exponent(ds) - 1;
  const float fm = (float)ldexp(ds[S_NEXT], -(k + q));  // power of two: R -> r * scale
  const int tid = threadIdx.x, li = tid & 31, lj = tid >> 5;
  const bool second = tid < kR19Rim - kMxThreads;
  const int r0 = tid / (kR19W + 2), c0 = tid - r0 * (kR19W + 2);
  const int e1 = tid + kMxThreads, r1 = second ? e1 / (kR19W + 2) : 0, c1 = second ? e1 - r1 * (kR19W + 2) : 0;
  double s2 = 0.0;  // sum R^2: the conversion and the FMA are all the FP64 pipe does per cell
  __int128 s1 = 0;
  for (int task = blockIdx.x; task < nti * ntj * nch; task += gridDim.x) {
    const int ti = task % nti, tj = task / nti % ntj, tc = task / (nti * ntj);
    const int i0 = bx.i0 + ti * kR19W, j0 = bx.j0 + tj * kR19H;  // 1-based
    const int ka = bx.k0 + tc * run, kb = min(ka + run - 1, bx.k1);
    const bool ok = i0 + li <= bx.i1 && j0 + lj <= bx.j1;
    // rim cells beyond the array (tiles past the box) are clamped: no cell of the box reads them
    const long long o0 = (long long)(min(i0 - 1 + c0, g.tx) - 1) + g.n1 * (min(j0 - 1 + r0, g.ty) - 1);
    const long long o1 = (long long)(min(i0 - 1 + c1, g.tx) - 1) + g.n1 * (min(j0 - 1 + r1, g.ty) - 1);
    const long long oc = (long long)(i0 + li - 1) + g.n1 * (j0 + lj - 1);
    const double* xp = x + g.n2 * (ka - 2);  // plane ka - 1
    double xa = xp[o0], xb = second ? xp[o1] : 0.0, bn = 0.0;
    int dn = -1;
    long long Cm = 0, Fm = 0, C0 = 0, F0 = 0, D0 = 0;
    __syncthreads();  // the last task's readers are done with both buffers
    for (int p = ka - 1; p <= kb + 1; ++p) {
      long long(*t)[kR19W + 2] = T[p & 1];
      t[r0][c0] = to_fix(xa, k);
      if (second) t[r1][c1] = to_fix(xb, k);
      const double bc = bn;
      const int dc = dn;
      if (p <= kb) {
        xp += g.n2;
        xa = xp[o0];
        if (second) xb = xp[o1];
        if (ok && p >= ka) {
          const long long I = oc + g.n2 * (p - 1);
          bn = b[I];
          dn = dq[I];
        }
      }
      __syncthreads();
      const long long W = t[lj + 1][li], C = t[lj + 1][li + 1], E = t[lj + 1][li + 2];
      const long long F = W + E + t[lj][li + 1] + t[lj + 2][li + 1];
      const long long D = t[lj][li] + t[lj][li + 2] + t[lj + 2][li] + t[lj + 2][li + 2];
      if (p > ka) {  // the residual at plane p - 1
        const long long B = to_fix(bc, k);
        long long R = (long long)dc * C0 + 4 * B - 2 * (F0 + Cm + C) - (D0 + Fm + F);
        R = dc >= 0 ? R : 0LL;  // dry cells and lanes outside the box
        const float f = __fmul_rn(__ll2float_rn(R), fm);
        if (ok) {
          const long long I = oc + g.n2 * (p - 2);
          b32[I] = f;
          if (!NEUMANN && r32) r32[I] = f;
        }
        if (NEUMANN) s1 += (__int128)R;
        const double rd = __ll2double_rn(R);
        s2 = __fma_rn(rd, rd, s2);
      }
      Cm = C0; Fm = F0;
      C0 = C; F0 = F; D0 = D;
    }
  }
  int_partials<false>(s2, s1, -2 * (k + q), k + q, partials);
}

void launch_resid_int19(const double* x, const double* b, const int8_t* dq, const Geom& g, const Box& bx,
                        const double* ds, float* b32, float* r32, bool neumann, double* partials, cudaStream_t s) {
  static const int wave = [] {
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return std::min(kMxParts, std::max(1, 4 * nsm));
  }();
  const int nti = (bx.i1 - bx.i0 + kR19W) / kR19W, ntj = (bx.j1 - bx.j0 + kR19H) / kR19H, nk = bx.k1 - bx.k0 + 1;
  int best = 1;
  long long cost = -1;
  for (int c = 1; c <= nk; ++c) {
    const int run = (nk + c - 1) / c;
    const long long tasks = (long long)nti * ntj * ((nk + run - 1) / run);
    const long long v = (tasks + wave - 1) / wave * (run + 2);
    if (cost < 0 || v < cost) {
      cost = v;
      best = c;
    }
  }
  const int run = (nk + best - 1) / best, nch = (nk + run - 1) / run;
  const long long tasks = (long long)nti * ntj * nch;
  const unsigned grid = (unsigned)std::min<long long>(wave, std::max<long long>(1, tasks));
  if (neumann)
    launch_dep(k_resid_int19<true>, grid, kMxThreads, 0, s, x, b, dq, g, bx, ds, b32, r32, partials, nti, ntj, nch, run);
  else
    launch_dep(k_resid_int19<false>, grid, kMxThreads, 0, s, x, b, dq, g, bx, ds, b32, r32, partials, nti, ntj, nch, run);
}

// sflag[(plane * nrows + row) * nstrips + strip] = 1 when the strip's
// columns of that row hold a wet cell
__global__ void k_make_sflag(const uint8_t* __restrict__ m, uint8_t* __restrict__ sflag, StripSpace sp) {
  const long long T = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n = (long long)sp.nplanes * sp.nrows * sp.nstrips;
  if (T >= n) return;
  const int strip = (int)(T % sp.nstrips);
  const long long pr = T / sp.nstrips;
  const int row = (int)(pr % sp.nrows), plane = (int)(pr / sp.nrows);
  const long long base = sp.row0 + plane * sp.n2 + (long long)row * sp.n1;
  const int c0 = sp.c0 + strip * kIntCols, c1 = min(c0 + kIntCols, sp.c0 + sp.ncols);
  unsigned any = 0;
  for (int c = c0; c < c1; ++c) any |= m[base + c];
  sflag[T] = any ? 1 : 0;
}

long long resid_sflag_size(int kind, const Geom& g, const Box& bx) {
  StripSpace sp;
  if (!strip_space(kind, g, bx, sp)) return 0;
  return (long long)sp.nplanes * sp.nrows * sp.nstrips;
}

void launch_make_sflag(int kind, const uint8_t* m, uint8_t* sflag, const Geom& g, const Box& bx, cudaStream_t s) {
  StripSpace sp;
  if (!strip_space(kind, g, bx, sp)) return;
  const long long n = (long long)sp.nplanes * sp.nrows * sp.nstrips;
  k_make_sflag<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(m, sflag, sp);
}

// cell-centred second pass: b32 = r32 = msk ? b32 - mean * scale : 0 with
// ms = ds + S_MEAN2 (the FP32 shift sits in S_SHIFT, made once by k_fused_final)
__global__ void k_rhs32_shift(const uint8_t* __restrict__ m, const double* __restrict__ ms, float* __restrict__ b32,
                              float* __restrict__ r32, long long n) {
  dep_wait();
  long long I = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (I >= n) return;
  const float sh = *reinterpret_cast<const float*>(ms + (S_SHIFT - S_MEAN2));  // (float)(mean * scale)
  const float f = m[I] ? __fsub_rn(b32[I], sh) : 0.f;
  b32[I] = f;
  if (r32) r32[I] = f;  // only the F-cycle restricts level 1's r before forming it
}

// the same, 16 cells a thread in 16-byte accesses (m, b32, r32 16-byte
// aligned); the last n % 16 cells by the scalar form in the final thread
template <bool SKIP>
__global__ void __launch_bounds__(256) k_rhs32_shift16(const uint8_t* __restrict__ m, const double* __restrict__ ms,
                                                       float* __restrict__ b32, float* __restrict__ r32,
                                                       long long n) {
  dep_wait();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long ng = n >> 4;
  if (t > ng) return;
  const float sh = *reinterpret_cast<const float*>(ms + (S_SHIFT - S_MEAN2));
  if (t == ng) {
    for (long long I = ng << 4; I < n; ++I) {
      const float f = m[I] ? __fsub_rn(b32[I], sh) : 0.f;
      b32[I] = f;
      if (r32) r32[I] = f;
    }
    return;
  }
  const uint4 mv = reinterpret_cast<const uint4*>(m)[t];
  // SKIP: 16 dry cells hold b32 = +0 already (the residual pass writes 0 there)
  if (SKIP && (mv.x | mv.y | mv.z | mv.w) == 0u) return;
  float4* bp = reinterpret_cast<float4*>(b32) + 4 * t;
  float4 v[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) v[u] = bp[u];
  const unsigned mw[4] = {mv.x, mv.y, mv.z, mv.w};
#pragma unroll
  for (int u = 0; u < 4; ++u) {  // mask bytes of cells 4u .. 4u+3, little-endian
    v[u].x = (mw[u] & 0xffu) ? __fsub_rn(v[u].x, sh) : 0.f;
    v[u].y = (mw[u] & 0xff00u) ? __fsub_rn(v[u].y, sh) : 0.f;
    v[u].z = (mw[u] & 0xff0000u) ? __fsub_rn(v[u].z, sh) : 0.f;
    v[u].w = (mw[u] & 0xff000000u) ? __fsub_rn(v[u].w, sh) : 0.f;
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) bp[u] = v[u];
  if (r32) {
    float4* rp = reinterpret_cast<float4*>(r32) + 4 * t;
#pragma unroll
    for (int u = 0; u < 4; ++u) rp[u] = v[u];
  }
}

// dq from diag and msk; *ok is cleared when a wet cell's Q*diag is not an
// integer in 0..most or a mask value is not 0/1
__global__ void k_make_dq(const double* __restrict__ diag, const uint8_t* __restrict__ m, double Q, double most,
                          int8_t* dq, long long n, int* ok) {
  dep_wait();
  long long I = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (I >= n) return;
  int8_t v = -128;
  if (m[I] == 1) {
    const double qd = diag[I] * Q;
    if (qd >= 0.0 && qd <= most && qd == floor(qd)) v = (int8_t)qd;
    else atomicAnd(ok, 0);
  } else if (m[I] != 0) {
    atomicAnd(ok, 0);
  }
  dq[I] = v;
}

// max |x| and max |b| (as the bit patterns of non-negative doubles, which
// order like the values) into ds[S_MAXX], ds[S_MAXB], and max |x| over the
// cells outside the box U = [ui0, ui1] x [uj0, uj1] of every layer (1-based;
// tx, ty the array's row and plane extents) into ds[S_MAXO]; all start at 0
__global__ void k_maxabs2(const double* __restrict__ x, const double* __restrict__ b, long long n, int tx, int ty,
                          int ui0, int ui1, int uj0, int uj1, double* ds, const uint8_t* __restrict__ m) {
  dep_wait();
  unsigned long long mx = 0, mb = 0, mo = 0;
  const long long nrows = n / tx;  // rows of all layers
  for (long long row = blockIdx.x; row < nrows; row += gridDim.x) {
    const int j = (int)(row % ty) + 1;
    const bool row_u = j >= uj0 && j <= uj1;
    const double* xr = x + row * tx;
    const double* br = b + row * tx;
    for (int i0 = threadIdx.x; i0 < tx; i0 += blockDim.x) {
      const unsigned long long ux = (unsigned long long)__double_as_longlong(xr[i0]) & 0x7FFFFFFFFFFFFFFFULL;
      const unsigned long long ub = (unsigned long long)__double_as_longlong(br[i0]) & 0x7FFFFFFFFFFFFFFFULL;
      const bool in_u = m ? m[row * tx + i0] != 0 : (row_u && i0 + 1 >= ui0 && i0 + 1 <= ui1);
      mx = ux > mx ? ux : mx;
      mb = ub > mb ? ub : mb;
      mo = (!in_u && ux > mo) ? ux : mo;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long ox = __shfl_down_sync(0xffffffffu, mx, o), ob = __shfl_down_sync(0xffffffffu, mb, o);
    const unsigned long long oo = __shfl_down_sync(0xffffffffu, mo, o);
    mx = ox > mx ? ox : mx;
    mb = ob > mb ? ob : mb;
    mo = oo > mo ? oo : mo;
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax((unsigned long long*)(ds + S_MAXX), mx);
    atomicMax((unsigned long long*)(ds + S_MAXB), mb);
    if (mo) atomicMax((unsigned long long*)(ds + S_MAXO), mo);
  }
}

// x += e * iscale, with max |x| of the result into ds[S_MAXX] (reset by the
// fused pass's final reduction): a grid-stride pass of 4 blocks per SM,
// one atomic per block
__global__ void __launch_bounds__(kMxThreads) k_update_scaled_max(double* __restrict__ x, const float* __restrict__ e,
                                                                  const double* __restrict__ ds, long long n,
                                                                  double* dsw) {
  dep_wait();
  const double is = ds[S_ICUR];
  const int pe = pow2_exponent(is);  // iscale = 2^pe
  unsigned long long mx = 0;
  const long long st = (long long)gridDim.x * blockDim.x;
  for (long long I0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; I0 < n; I0 += 4 * st) {
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {  // loads of 4 cells in flight
      const long long I = I0 + u * st;
      if (I < n) v[u] = __dadd_rn(x[I], f2d_pow2(e[I], pe, is));
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long I = I0 + u * st;
      if (I < n) {
        x[I] = v[u];
        const unsigned long long ub = (unsigned long long)__double_as_longlong(v[u]) & 0x7FFFFFFFFFFFFFFFULL;
        mx = ub > mx ? ub : mx;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long ox = __shfl_down_sync(0xffffffffu, mx, o);
    mx = ox > mx ? ox : mx;
  }
  __shared__ unsigned long long sh[kMxThreads / 32];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kMxThreads / 32; ++w) mx = sh[w] > mx ? sh[w] : mx;
    if (mx) atomicMax((unsigned long long*)(dsw + S_MAXX), mx);
  }
}

// the same with 16-byte accesses (x and e 16-byte aligned): 4 cells a
// group, two groups of a thread in flight; the last n % 4 cells by block 0
//
// msk (optional): a group of 4 dry cells is skipped (e = +0 there, so x stays
// as it is up to the sign of a zero); the max |x| of the dry cells, which no
// update changes, is in S_MAXO, from which S_MAXX starts.
__global__ void __launch_bounds__(kMxThreads) k_update_scaled_max4(double* __restrict__ x, const float* __restrict__ e,
                                                                   const double* __restrict__ ds, long long n,
                                                                   double* dsw, const uint8_t* __restrict__ msk) {
  dep_wait();
  const double is = ds[S_ICUR];
  const int pe = pow2_exponent(is);  // iscale = 2^pe
  unsigned long long mx = 0;
  auto upd = [&](double xo, float ev) {
    const double v = __dadd_rn(xo, f2d_pow2(ev, pe, is));
    const unsigned long long ub = (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFULL;
    mx = ub > mx ? ub : mx;
    return v;
  };
  const long long ng = n >> 2;
  const long long st = (long long)gridDim.x * blockDim.x;
  const float4* e4 = reinterpret_cast<const float4*>(e);
  double2* x2 = reinterpret_cast<double2*>(x);
  for (long long g0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; g0 < ng; g0 += 2 * st) {
    float4 ev[2];
    double2 xa[2], xb[2];
    bool act[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const long long g = g0 + u * st;
      act[u] = g < ng;
      if (act[u] && msk) {
        const uchar4 mm = reinterpret_cast<const uchar4*>(msk)[g];
        act[u] = (mm.x | mm.y | mm.z | mm.w) != 0;
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const long long g = g0 + u * st;
      if (act[u]) {
        ev[u] = e4[g];
        xa[u] = x2[2 * g];
        xb[u] = x2[2 * g + 1];
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const long long g = g0 + u * st;
      if (act[u]) {
        double2 ra, rb;
        ra.x = upd(xa[u].x, ev[u].x);
        ra.y = upd(xa[u].y, ev[u].y);
        rb.x = upd(xb[u].x, ev[u].z);
        rb.y = upd(xb[u].y, ev[u].w);
        x2[2 * g] = ra;
        x2[2 * g + 1] = rb;
      }
    }
  }
  if (blockIdx.x == 0 && threadIdx.x < (n & 3)) {
    const long long I = (ng << 2) + threadIdx.x;
    x[I] = upd(x[I], e[I]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long ox = __shfl_down_sync(0xffffffffu, mx, o);
    mx = ox > mx ? ox : mx;
  }
  __shared__ unsigned long long sh[kMxThreads / 32];
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kMxThreads / 32; ++w) mx = sh[w] > mx ? sh[w] : mx;
    if (mx) atomicMax((unsigned long long*)(dsw + S_MAXX), mx);
  }
}

void launch_resid_int(int kind, const double* x, const double* b, const int8_t* dq, const Geom& g, const Box& bx,
                      long long lo, long long n, const double* ds, float* b32, float* r32, bool neumann,
                      double* partials, cudaStream_t s) {
#define CFMG_INT(K)                                                                                        \
  if (kind == K) {                                                                                         \
    if (neumann)                                                                                           \
      launch_dep(k_resid_int<K, true>, kMxParts, kMxThreads, 0, s, x, b, dq, g, bx, lo, n, ds, b32, r32, partials); \
    else                                                                                                   \
      launch_dep(k_resid_int<K, false>, kMxParts, kMxThreads, 0, s, x, b, dq, g, bx, lo, n, ds, b32, r32, partials); \
    return;                                                                                                \
  }
  CFMG_INT(OPK_RESID5)
  CFMG_INT(OPK_RESID9)
  CFMG_INT(OPK_RESID7)
#undef CFMG_INT
}

void launch_rhs32_shift(const uint8_t* m, const double* mean_scale, float* b32, float* r32, long long n,
                        cudaStream_t s, bool skip_dry) {
  const bool a16 = ((uintptr_t)m | (uintptr_t)b32 | (uintptr_t)r32) % 16 == 0;
  if (a16) {
    const long long nt = (n >> 4) + 1;  // groups of 16, and one thread for the rest
    if (skip_dry && !r32)
      launch_dep(k_rhs32_shift16<true>, (unsigned)((nt + 255) / 256), 256, 0, s, m, mean_scale, b32, r32, n);
    else
      launch_dep(k_rhs32_shift16<false>, (unsigned)((nt + 255) / 256), 256, 0, s, m, mean_scale, b32, r32, n);
  } else {
    launch_dep(k_rhs32_shift, (unsigned)((n + 255) / 256), 256, 0, s, m, mean_scale, b32, r32, n);
  }
}

// most: |x| and |b| are at most 2^58 steps (2^57 in the 19-point form), so a
// sum of dq x, Q b and the neighbours' weights in units of 1/Q stays below 2^63
// while dq + Q + weights <= 31 (63); the setup's own diag gives 4, 6, 12 and 24
void launch_make_dq(int kind, const double* diag, const uint8_t* m, int8_t* dq, long long n, int* ok,
                    cudaStream_t s) {
  const bool q4 = kind == OPK_RESID9 || kind == OPK_RESID19;
  const int others = kind == OPK_RESID5 ? 1 + 4 : kind == OPK_RESID7 ? 1 + 6 : kind == OPK_RESID9 ? 4 + 12 : 4 + 24;
  const int most = (kind == OPK_RESID19 ? 63 : 31) - others;
  launch_dep(k_make_dq, (unsigned)((n + 255) / 256), 256, 0, s, diag, m, q4 ? 4.0 : 1.0, (double)most, dq, n, ok);
}

void launch_maxabs2(const double* x, const double* b, long long n, int tx, int ty, int ui0, int ui1, int uj0, int uj1,
                    double* ds, cudaStream_t s, const uint8_t* m) {
  launch_dep(k_maxabs2, 1024, 256, 0, s, x, b, n, tx, ty, ui0, ui1, uj0, uj1, ds, m);
}

void launch_update_scaled_max(double* x, const float* e, double* ds, long long n, cudaStream_t s,
                              const uint8_t* msk) {
  static int nsm = 0;
  if (!nsm) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  }
  if (((uintptr_t)x | (uintptr_t)e) % 16 == 0 && (uintptr_t)msk % 4 == 0)
    launch_dep(k_update_scaled_max4, nsm * 4, kMxThreads, 0, s, x, e, ds, n, ds, msk);
  else
    launch_dep(k_update_scaled_max, nsm * 4, kMxThreads, 0, s, x, e, ds, n, ds);  // 4 blocks per SM: measured 4 % faster than 8
}

void launch_resid_fused(int kind, double* r, const double* x, const double* b, const double* d, const uint8_t* m,
                        const Geom& g, const Box& bx, long long lo, long long n, const double* scale, float* b32,
                        float* r32, bool neumann, double* partials, cudaStream_t s) {
#define CFMG_FUSED(K)                                                                                            \
  if (kind == K) {                                                                                               \
    if (neumann)                                                                                                 \
      launch_dep(k_resid_fused<K, true>, kMxParts, kMxThreads, 0, s, r, x, b, d, m, g, bx, lo, n, scale, b32, r32, partials); \
    else                                                                                                         \
      launch_dep(k_resid_fused<K, false>, kMxParts, kMxThreads, 0, s, r, x, b, d, m, g, bx, lo, n, scale, b32, r32, partials); \
    return;                                                                                                      \
  }
  CFMG_FUSED(OPK_RESID5)
  CFMG_FUSED(OPK_RESID9)
  CFMG_FUSED(OPK_RESID7)
  CFMG_FUSED(OPK_RESID19)
#undef CFMG_FUSED
}

void launch_fused_final(const double* partials, double* ds, const double* normb, const double* nwet, int norm_kind,
                        cudaStream_t s, const LoopTest* lt, int q) {
  launch_dep(k_fused_final, 1, kMxParts, 0, s, partials, ds, normb, nwet, norm_kind, lt ? *lt : LoopTest{}, q);
}

void launch_rhs32(const double* r, const uint8_t* m, const double* mean, const double* scale, float* b32, float* r32,
                  long long n, cudaStream_t s) {
  launch_dep(k_rhs32, (unsigned)((n + 1023) / 1024), 256, 0, s, r, m, mean, scale, b32, r32, n);
}

void launch_update_scaled(double* x, const float* e, const double* iscale, long long n, cudaStream_t s) {
  launch_dep(k_update_scaled, (unsigned)((n + 1023) / 1024), 256, 0, s, x, e, iscale, n);
}

}  // namespace cfmg
