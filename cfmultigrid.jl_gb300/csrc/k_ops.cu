// Per-level multigrid operators: Jacobi sweeps, residuals, restriction,
// prolongation, periodic halo fill and the masked norm.
//
// Instantiated for double (the FP64 drop-in) and float (the cycles of the
// mixed-precision form). Every sum and product goes through the _rn
// intrinsics so that nvcc cannot contract a multiply and an add into one
// FMA: the FP64 instantiation rounds exactly where the Julia reference
// rounds, and is bit-identical to it. The only FMAs used are ones whose
// product is exact (a multiplication by 1/2, 1/4, 2, 4 or 8), which round
// once on the same exact value as the reference's two-step form.
//
// These kernels are single-pass and keep the reference's own loop ranges,
// halo cells included; they are FP64-issue bound on GB300 (the FP64 pipe
// runs at 1/64 of the FP32 rate), so their memory traffic is not the limit.
#include "ops_dev.cuh"

namespace cfmg {

constexpr int kThreads = 256;

inline unsigned nblocks(long long n, int per = kThreads) { return (unsigned)((n + per - 1) / per); }

// FP64 instances with ZS: a warp whose lanes all have zero operands stores the
// signed zero that the operator gives and is done (see ZeroAcc).
#define CFMG_ZERO_WARP(dst, test)                                    \
  if constexpr (ZS) {                                    \
    double z = 0.0;                                                  \
    const bool zr = test;                                            \
    if (__all_sync(__activemask(), zr)) {                            \
      dst = z;                                                       \
      return;                                                        \
    }                                                                \
  }

// ----------------------------------------------------------------- sweeps
// sloop2d! (src/laplacian.jl:66-73): y = (1-w)x - (w*idiag)*(b - s4) over
// the linear range 1+n1 .. length-n1.
template <class T, bool ZS>
__global__ void __launch_bounds__(kThreads) k_sweep5_2d(const T* __restrict__ x, T* __restrict__ y,
                                                        const T* __restrict__ b, const T* __restrict__ w, T cff,
                                                        long long n1, long long lo, long long hi) {
  dep_wait();
  long long I = lo + (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (I >= hi) return;
  CFMG_ZERO_WARP(y[I], (zero_sweep<ZS_5>(x, b, w, x, x, cff, n1, 0, I, z)))
  d_sweep5(x, y, b, w, cff, n1, I);
}

// sloop3d_v1! (src/laplacian.jl:11-20): 7-point, linear range 1+n2 .. length-n2.
template <class T, bool ZS>
__global__ void __launch_bounds__(kThreads) k_sweep7_3d(const T* __restrict__ x, T* __restrict__ y,
                                                        const T* __restrict__ b, const T* __restrict__ w, T cff,
                                                        long long n1, long long n2, long long lo, long long hi) {
  dep_wait();
  long long I = lo + (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (I >= hi) return;
  CFMG_ZERO_WARP(y[I], (zero_sweep<ZS_7>(x, b, w, x, x, cff, n1, n2, I, z)))
  d_sweep7(x, y, b, w, cff, n1, n2, I);
}

// Thread mapping of a box kernel: x over i, y over j, z over k.
struct BoxIdx {
  int i, j, k;
  bool ok;
};
__device__ __forceinline__ BoxIdx box_idx(const Box& bx) {
  BoxIdx r;
  r.i = bx.i0 + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  r.j = bx.j0 + (int)(blockIdx.y * blockDim.y + threadIdx.y);
  r.k = bx.k0 + (int)blockIdx.z;
  r.ok = r.i <= bx.i1 && r.j <= bx.j1 && r.k <= bx.k1;
  return r;
}
inline dim3 box_grid(const Box& bx, dim3 blk) {
  int ni = bx.i1 - bx.i0 + 1, nj = bx.j1 - bx.j0 + 1, nk = bx.k1 - bx.k0 + 1;
  return dim3((unsigned)((ni + blk.x - 1) / blk.x), (unsigned)((nj + blk.y - 1) / blk.y), (unsigned)nk);
}
inline long long box_cells(const Box& bx) {
  return (long long)(bx.i1 - bx.i0 + 1) * (bx.j1 - bx.j0 + 1) * (bx.k1 - bx.k0 + 1);
}
// The test for zero operands pays where the FP64 pipe bounds a pass: from
// half a million cells. At 512^2 a 9-point sweep took 9.9 us with it and 9.5
// without, at 128^2 4.3 and 3.6 (it lengthens the chain of a launch that is
// all latency); at 104 x 88 x 56 (620 000 cells of a basin, a third wet) 10.2
// and 13.6.
constexpr long long kZeroMin = 1LL << 19;
// The FP64 9-point operators' integer form (k_fix.cu) pays from a quarter of a
// million cells: at 512^2 a sweep took 10.5 us with it and 12.6 without, at
// 384^2 9.8 and 9.9.
constexpr long long kFixMin = 1LL << 18;
#define CFMG_ZS(K, N, ...)                                                                     \
  do {                                                                                         \
    if (sizeof(T) == 8 && (N) >= kZeroMin) launch_dep(K<T, sizeof(T) == 8>, __VA_ARGS__);      \
    else launch_dep(K<T, false>, __VA_ARGS__);                                                 \
  } while (0)
inline bool box_empty(const Box& bx) { return bx.i1 < bx.i0 || bx.j1 < bx.j0 || bx.k1 < bx.k0; }
static const dim3 kBoxBlk(64, 4, 1);

template <class T>
__global__ void __launch_bounds__(kThreads) k_sweep9_2d(const T* __restrict__ x, T* __restrict__ y,
                                                        const T* __restrict__ b, const T* __restrict__ w, T cff,
                                                        Geom g, Box bx) {
  dep_wait();
  BoxIdx q = box_idx(bx);
  if (!q.ok) return;
  const long long I = lin(g, q.i, q.j, q.k);
  d_sweep9(x, y, b, w, cff, g.n1, I);
}

template <class T, bool ZS>
__global__ void __launch_bounds__(kThreads) k_sweep19_3d(const T* __restrict__ x, T* __restrict__ y,
                                                         const T* __restrict__ b, const T* __restrict__ w, T cff,
                                                         Geom g, Box bx) {
  dep_wait();
  BoxIdx q = box_idx(bx);
  if (!q.ok) return;
  const long long I = lin(g, q.i, q.j, q.k);
  CFMG_ZERO_WARP(y[I], (zero_sweep<ZS_19>(x, b, w, x, x, cff, g.n1, g.n2, I, z)))
  d_sweep19(x, y, b, w, cff, g.n1, g.n2, I);
}

template <class T, bool ZS>
__global__ void __launch_bounds__(kThreads) k_sweep_vc_2d(const T* __restrict__ x, T* __restrict__ y,
                                                          const T* __restrict__ b, const T* __restrict__ w,
                                                          const T* __restrict__ cE, const T* __restrict__ cN, T cff,
                                                          long long n1, long long lo, long long hi) {
  dep_wait();
  long long I = lo + (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (I >= hi) return;
  CFMG_ZERO_WARP(y[I], (zero_sweep<ZS_VC>(x, b, w, cE, cN, cff, n1, 0, I, z)))
  d_sweepvc(x, y, b, w, cE, cN, cff, n1, I);
}

// -------------------------------------------------------------- residuals
// rloop2d! (src/laplacian.jl:87-93): r = msk*((diag*x + b) - s4).
template <class T, bool ZS>
__global__ void __launch_bounds__(kThreads) k_resid5_2d(T* __restrict__ r, const T* __restrict__ x,
                                                        const T* __restrict__ b, const T* __restrict__ d,
                                                        const uint8_t* __restrict__ m, long long n1, long long lo,
                                                        long long hi) {
  dep_wait();
  long long I = lo + (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (I >= hi) return;
  CFMG_ZERO_WARP(r[I], (zero_resid<ZS_5>(x, b, d, x, x, n1, 0, I, z)))
  d_resid5(r, x, b, d, m, n1, I);
}

// rloop3d! (src/laplacian.jl:43-51): interior box only.
template <class T, bool ZS>
__global__ void __launch_bounds__(kThreads) k_resid7_3d(T* __restrict__ r, const T* __restrict__ x,
                                                        const T* __restrict__ b, const T* __restrict__ d,
                                                        const uint8_t* __restrict__ m, Geom g, Box bx) {
  dep_wait();
  BoxIdx q = box_idx(bx);
  if (!q.ok) return;
  const long long I = lin(g, q.i, q.j, q.k);
  CFMG_ZERO_WARP(r[I], (zero_resid<ZS_7>(x, b, d, x, x, g.n1, g.n2, I, z)))
  d_resid7(r, x, b, d, m, g.n1, g.n2, I);
}

// residual of the 2D 9-point extension, interior box.
template <class T>
__global__ void __launch_bounds__(kThreads) k_resid9_2d(T* __restrict__ r, const T* __restrict__ x,
                                                        const T* __restrict__ b, const T* __restrict__ d,
                                                        const uint8_t* __restrict__ m, Geom g, Box bx) {
  dep_wait();
  BoxIdx q = box_idx(bx);
  if (!q.ok) return;
  const long long I = lin(g, q.i, q.j, q.k);
  d_resid9(r, x, b, d, m, g.n1, I);
}

// residual_laplacian9! (src/laplacian9.jl:49-73), interior box.
template <class T, bool ZS>
__global__ void __launch_bounds__(kThreads) k_resid19_3d(T* __restrict__ r, const T* __restrict__ x,
                                                         const T* __restrict__ b, const T* __restrict__ d,
                                                         const uint8_t* __restrict__ m, Geom g, Box bx) {
  dep_wait();
  BoxIdx q = box_idx(bx);
  if (!q.ok) return;
  const long long I = lin(g, q.i, q.j, q.k);
  CFMG_ZERO_WARP(r[I], (zero_resid<ZS_19>(x, b, d, x, x, g.n1, g.n2, I, z)))
  d_resid19(r, x, b, d, m, g.n1, g.n2, I);
}

template <class T, bool ZS>
__global__ void __launch_bounds__(kThreads) k_resid_vc_2d(T* __restrict__ r, const T* __restrict__ x,
                                                          const T* __restrict__ b, const T* __restrict__ d,
                                                          const T* __restrict__ cE, const T* __restrict__ cN,
                                                          const uint8_t* __restrict__ m, long long n1, long long lo,
                                                          long long hi) {
  dep_wait();
  long long I = lo + (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (I >= hi) return;
  CFMG_ZERO_WARP(r[I], (zero_resid<ZS_VC>(x, b, d, cE, cN, n1, 0, I, z)))
  d_residvc(r, x, b, d, cE, cN, m, n1, I);
}

// ------------------------------------------------------------ restriction

// Thread per coarse interior cell (ii, jj, kk); the coarse b is written.
template <class T, int KIND, bool ZS>
__global__ void __launch_bounds__(kThreads) k_restrict(const T* __restrict__ x, T* __restrict__ xc,
                                                       const T* __restrict__ coef, Geom gf, Geom gc, Box cb) {
  dep_wait();
  BoxIdx q = box_idx(cb);
  if (!q.ok) return;
  const long long C = lin(gc, q.i, q.j, q.k);
  CFMG_ZERO_WARP(xc[C], (zero_restrict<KIND>(x, coef[C], gf, gc, q.i, q.j, q.k, z)))
  d_restrict<T, KIND>(x, xc, coef, gf, gc, q.i, q.j, q.k);
}

// ----------------------------------------------------------- prolongation

// Thread per fine parent (i, j, k) = (nh+1+2p, nh+1+2q, ...); each parent
// updates its 4 (2D) or 8 (3D) children, which no other thread touches.
// fmsk (optional, FP32 cycles): a parent whose children are all dry is
// skipped; a dry fine cell holds +0 and has Pcoef = 0, so the update would
// leave it +0.
template <class T, int KIND, bool ASSIGN, bool ZS>
__global__ void __launch_bounds__(kThreads) k_prolong(T* __restrict__ xf, const T* __restrict__ x,
                                                      const T* __restrict__ coef, Geom gf, Geom gc, int np_i,
                                                      int np_j, int kf0, int kf1, int np_k,
                                                      const uint8_t* __restrict__ fmsk) {
  dep_wait();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  const int qj = blockIdx.y * blockDim.y + threadIdx.y;
  const int qk = blockIdx.z;
  if (p >= np_i || qj >= np_j || qk >= np_k) return;
  if (fmsk) {
    const int nh = gf.nh;
    const bool t3 = KIND == 1 || KIND == 3;
    const long long F = lin(gf, nh + 1 + 2 * p, nh + 1 + 2 * qj, t3 ? nh + 1 + 2 * qk : kf0 + qk);
    const long long f1 = gf.n1, f2 = gf.n2;
    unsigned any = fmsk[F] | fmsk[F + 1] | fmsk[F + f1] | fmsk[F + 1 + f1];
    if (t3) any |= fmsk[F + f2] | fmsk[F + 1 + f2] | fmsk[F + f1 + f2] | fmsk[F + 1 + f1 + f2];
    if (!any) return;
  }
  if constexpr (ZS && !ASSIGN) {
    const bool dry = zero_prolong<KIND>(xf, x, coef, gf, gc, p, qj, qk, kf0);
    if (__all_sync(__activemask(), dry)) return;
  }
  d_prolong<T, KIND, ASSIGN>(xf, x, coef, gf, gc, p, qj, qk, kf0);
}

// ------------------------------------------ residual + restriction, 3D
// rloop3d! (src/laplacian.jl:43-51) at the eight children of each coarse
// interior cell and the cell-centred 3D restriction of those residuals
// (rcloop3d!, src/RP_on_centers.jl:62-82) into the coarse b, in one pass of
// the FP32 7-point level: the fine r is not stored and read back. diag is
// read as its one-byte code (an integer diag for the 7-point weights, the
// float exactly). Each child's residual and the sum of the eight are
// computed as v_resid7 and v_restrict<KIND 1> do, so the coarse b is the
// same bits. Every child must lie in the fine interior box (checked by the
// caller). skip_dry: a coarse cell whose eight children are dry gets +0
// without the residual's loads (the masked residuals are signed zeros, so
// the restricted value is a zero, of whichever sign).
__global__ void __launch_bounds__(256) k_resid_restrict7c(const float* __restrict__ x, const float* __restrict__ b,
                                                          const uint8_t* __restrict__ dc,
                                                          const uint8_t* __restrict__ m,
                                                          const float* __restrict__ rcoef, float* __restrict__ bc,
                                                          Geom gf, Geom gc, Box cb, bool skip_dry) {
  dep_wait();
  const BoxIdx q = box_idx(cb);
  if (!q.ok) return;
  typedef Ar<float> A;
  const int nh = gc.nh;
  const long long n1 = gf.n1, n2 = gf.n2;
  const long long F = lin(gf, c2f(q.i, nh), c2f(q.j, nh), c2f(q.k, nh));
  if (skip_dry && (m[F] | m[F + 1] | m[F + n1] | m[F + 1 + n1] | m[F + n2] | m[F + 1 + n2] | m[F + n1 + n2] |
                   m[F + 1 + n1 + n2]) == 0) {
    bc[lin(gc, q.i, q.j, q.k)] = 0.f;
    return;
  }
  auto r = [&](long long I) {
    return mask_mul(m[I], A::sub(A::add(A::mul((float)dc[I], x[I]), b[I]), faces6(x, I, n1, n2)));
  };
  float s = A::add(r(F), r(F + 1));
  s = A::add(s, r(F + n1));
  s = A::add(s, r(F + 1 + n1));
  s = A::add(s, r(F + n2));
  s = A::add(s, r(F + 1 + n2));
  s = A::add(s, r(F + n1 + n2));
  s = A::add(s, r(F + 1 + n1 + n2));
  const long long C = lin(gc, q.i, q.j, q.k);
  bc[C] = A::mul(rcoef[C], s);
}
void launch_resid_restrict7c(const float* x, const float* b, const uint8_t* dc, const uint8_t* m, const float* rcoef,
                             float* bc, const Geom& gf, const Geom& gc, const Box& cb, cudaStream_t s,
                             bool skip_dry) {
  if (box_empty(cb)) return;
  launch_dep(k_resid_restrict7c, box_grid(cb, kBoxBlk), kBoxBlk, 0, s, x, b, dc, m, rcoef, bc, gf, gc, cb,
             skip_dry);
}

// in-order global loads (asm volatile keeps them ahead of the arithmetic
// that follows, so that all of a thread's loads are in flight together)
__device__ __forceinline__ float ld_nc_ordered(const float* p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_ordered(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

// pcloop3d! (src/RP_on_centers.jl:84-114) in FP32 with every load of a
// parent issued before its arithmetic: the 25 coarse values (the centre and
// the 8 in-plane neighbours of each of the planes kc-1, kc, kc+1 that the
// eight children's `square` terms use), the 8 Pcoef values and, unless
// ASSIGN, the 8 fine x values. d_prolong<float, 1>'s arithmetic in its order.
// The thread-per-parent form compiled to 32 registers with its loads spread
// over the arithmetic; its warps waited on memory 85-90 % of the time.
// fmsk (optional): a parent whose eight children are all dry is skipped; a
// dry fine cell holds +0 and has Pcoef = 0, so the update would leave it +0.
template <bool ASSIGN>
__global__ void __launch_bounds__(256) k_prolong3c_f(float* __restrict__ xf, const float* __restrict__ x,
                                                     const float* __restrict__ coef, Geom gf, Geom gc, int np_i,
                                                     int np_j, int np_k, const uint8_t* __restrict__ fmsk) {
  dep_wait();
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  const int q = blockIdx.y * blockDim.y + threadIdx.y;
  const int qk = blockIdx.z;
  if (p >= np_i || q >= np_j || qk >= np_k) return;
  typedef Ar<float> A;
  const int nh = gf.nh;
  const int i = nh + 1 + 2 * p, j = nh + 1 + 2 * q, k = nh + 1 + 2 * qk;
  const long long c1 = gc.n1, c2 = gc.n2, f1 = gf.n1, f2 = gf.n2;
  const long long C = lin(gc, f2c(i, nh), f2c(j, nh), f2c(k, nh)), F = lin(gf, i, j, k);
  if (fmsk) {
    unsigned any = 0;
#pragma unroll
    for (int t = 0; t < 8; ++t) any |= fmsk[F + (t & 1) + ((t >> 1) & 1) * f1 + (t >> 2) * f2];
    if (!any) return;
  }
  // xs[dk][d]: plane C + (dk-1)*c2, offsets d = W, E, S, N, SW, SE, NW, NE
  const long long off[8] = {-1, 1, -c1, c1, -1 - c1, 1 - c1, -1 + c1, 1 + c1};
  float xs[3][8];
#pragma unroll
  for (int dk = 0; dk < 3; ++dk)
#pragma unroll
    for (int d = 0; d < 8; ++d) xs[dk][d] = ld_nc_ordered(x + C + (dk - 1) * c2 + off[d]);
  const float x0 = ld_nc_ordered(x + C);
  float cf[8], xo[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) {  // child t: di = t & 1, dj = (t >> 1) & 1, dk = t >> 2
    const long long Fi = F + (t & 1) + ((t >> 1) & 1) * f1 + (t >> 2) * f2;
    cf[t] = ld_nc_ordered(coef + Fi);
    xo[t] = ASSIGN ? 0.f : ld_ordered(xf + Fi);
  }
  const float x28 = A::mul(x0, 28.f);
#pragma unroll
  for (int dj = 0; dj <= 1; ++dj)
#pragma unroll
    for (int di = 0; di <= 1; ++di) {
      const int dI = di, dJ = 2 + dj, dIJ = 4 + di + 2 * dj;  // W/E, S/N, the corner
      auto sq = [&](int pl) { return A::add(A::mul(3.f, A::add(xs[pl][dI], xs[pl][dJ])), xs[pl][dIJ]); };
      const float a = sq(0);
      const float bb = A::mul(sq(1), 3.f);
      const float c = sq(2);
      const int t0 = di + 2 * dj, t1 = t0 + 4;
      const long long F0 = F + di + dj * f1, F1 = F0 + f2;
      xf[F0] = A::add(xo[t0], A::mul(cf[t0], A::add(A::add(bb, a), x28)));
      xf[F1] = A::add(xo[t1], A::mul(cf[t1], A::add(A::add(bb, c), x28)));
    }
}

// ------------------------------------------- small level in shared memory
// A smoothing call of npairs pairs on a level whose x, y, b and omega*idiag
// fit one block's shared memory (the coarsest solve: 2*ndeepest sweeps on a
// few hundred cells): one block loads the four arrays, runs every sweep with
// a block barrier between sweeps, and writes x and y back. Launched as the
// engine's separate Ops, each sweep would cost a cluster barrier and the
// round trip through L2. The sweep ranges and the per-cell arithmetic are
// smooth_t's: the linear range n1 .. len-n1 with v_sweep5 (2D 5-point), the
// box icp x jcp then the interior with v_sweep9 (2D 9-point), the linear
// range n2 .. len-n2 with v_sweep7 (3D 7-point); Jacobi sweeps, so the order
// of the cells within a sweep does not matter, and the bits are the same.
constexpr int kSmallThreads = 1024;
template <class T>
__global__ void __launch_bounds__(kSmallThreads) k_small_smooth(SmallSm s) {
  dep_wait();
  extern __shared__ __align__(16) unsigned char ssm_raw[];
  const long long len = s.g.len;
  T* X = reinterpret_cast<T*>(ssm_raw);
  T* Y = X + len;
  T* B = Y + len;
  T* W = B + len;
  for (long long t = threadIdx.x; t < len; t += blockDim.x) {
    X[t] = static_cast<const T*>(s.x)[t];
    Y[t] = static_cast<const T*>(s.y)[t];
    B[t] = static_cast<const T*>(s.b)[t];
    W[t] = static_cast<const T*>(s.w)[t];
  }
  __syncthreads();
  const T cff = (T)s.cff;
  const long long n1 = s.g.n1, n2 = s.g.n2;
  auto sweep = [&](const T* src, T* dst, bool first) {
    if (s.stencil == 5) {
      for (long long I = n1 + threadIdx.x; I < len - n1; I += blockDim.x) dst[I] = v_sweep5(src, B, W, cff, n1, I);
    } else if (s.stencil == 7) {
      for (long long I = n2 + threadIdx.x; I < len - n2; I += blockDim.x) dst[I] = v_sweep7(src, B, W, cff, n1, n2, I);
    } else {
      const Box& bx = first ? s.ext : s.in;
      const int ni = bx.i1 - bx.i0 + 1, nj = bx.j1 - bx.j0 + 1;
      const long long n = (long long)ni * nj * (bx.k1 - bx.k0 + 1);
      for (long long t = threadIdx.x; t < n; t += blockDim.x) {
        const int i = bx.i0 + (int)(t % ni);
        const long long q = t / ni;
        const long long I = lin(s.g, i, bx.j0 + (int)(q % nj), bx.k0 + (int)(q / nj));
        dst[I] = v_sweep9(src, B, W, cff, n1, I);
      }
    }
    __syncthreads();
  };
  for (int p = 0; p < s.npairs; ++p) {
    sweep(X, Y, true);
    sweep(Y, X, false);
  }
  for (long long t = threadIdx.x; t < len; t += blockDim.x) {
    static_cast<T*>(s.x)[t] = X[t];
    static_cast<T*>(s.y)[t] = Y[t];
  }
}
// The same on kSmallCtas SMs (FP64, where one SM's FP64 pipe bounds the
// one-block form): a cluster whose CTAs each hold the whole level in their
// shared memory and sweep one contiguous share of the swept cells, storing
// each new value into their own copy and, through distributed shared memory,
// into every other CTA's copy; a cluster barrier (release/acquire) ends each
// sweep, after which every copy is the full new iterate. Each CTA writes its
// share of x and y back. The cells and their arithmetic are the one-block
// form's.
constexpr int kSmallCtas = 8, kSmallCluThreads = 256;
__device__ __forceinline__ unsigned small_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void small_cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void st_remote(double* local, unsigned rank, double v) {
  unsigned a = (unsigned)__cvta_generic_to_shared(local), ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(v) : "memory");
}
__global__ void __launch_bounds__(kSmallCluThreads) k_small_smooth_cluster(SmallSm s) {
  dep_wait();
  typedef double T;
  extern __shared__ __align__(16) unsigned char ssm_raw[];
  const long long len = s.g.len;
  T* X = reinterpret_cast<T*>(ssm_raw);
  T* Y = X + len;
  T* B = Y + len;
  T* W = B + len;
  for (long long t = threadIdx.x; t < len; t += blockDim.x) {
    X[t] = static_cast<const T*>(s.x)[t];
    Y[t] = static_cast<const T*>(s.y)[t];
    B[t] = static_cast<const T*>(s.b)[t];
    W[t] = static_cast<const T*>(s.w)[t];
  }
  small_cluster_barrier();  // every copy loaded before any CTA stores into another's
  const unsigned rank = small_rank();
  const T cff = (T)s.cff;
  const long long n1 = s.g.n1, n2 = s.g.n2;
  // the swept cells of a sweep as an index space 0 .. n-1 -> cell I
  auto space = [&](bool first, long long& n) {
    if (s.stencil == 5) n = len - 2 * n1;
    else if (s.stencil == 7) n = len - 2 * n2;
    else {
      const Box& bx = first ? s.ext : s.in;
      n = (long long)(bx.i1 - bx.i0 + 1) * (bx.j1 - bx.j0 + 1) * (bx.k1 - bx.k0 + 1);
    }
  };
  auto cell = [&](bool first, long long t) -> long long {
    if (s.stencil == 5) return n1 + t;
    if (s.stencil == 7) return n2 + t;
    const Box& bx = first ? s.ext : s.in;
    const int ni = bx.i1 - bx.i0 + 1, nj = bx.j1 - bx.j0 + 1;
    const long long q = t / ni;
    return lin(s.g, bx.i0 + (int)(t % ni), bx.j0 + (int)(q % nj), bx.k0 + (int)(q / nj));
  };
  auto sweep = [&](const T* src, T* dst, bool first) {
    long long n;
    space(first, n);
    const long long a = n * rank / kSmallCtas, e = n * (rank + 1) / kSmallCtas;
    for (long long t = a + threadIdx.x; t < e; t += blockDim.x) {
      const long long I = cell(first, t);
      const T v = s.stencil == 5 ? v_sweep5(src, B, W, cff, n1, I)
                                 : (s.stencil == 7 ? v_sweep7(src, B, W, cff, n1, n2, I) : v_sweep9(src, B, W, cff, n1, I));
      for (unsigned r = 0; r < kSmallCtas; ++r) {
        if (r == rank) dst[I] = v;
        else st_remote(dst + I, r, v);
      }
    }
    small_cluster_barrier();
  };
  for (int p = 0; p < s.npairs; ++p) {
    sweep(X, Y, true);
    sweep(Y, X, false);
  }
  // each CTA writes back the cells it swept (the others are unchanged)
  for (int f = 0; f < 2; ++f) {
    long long n;
    space(f == 0, n);
    const long long a = n * rank / kSmallCtas, e = n * (rank + 1) / kSmallCtas;
    for (long long t = a + threadIdx.x; t < e; t += blockDim.x) {
      const long long I = cell(f == 0, t);
      if (f == 0) static_cast<T*>(s.y)[I] = Y[I];
      else static_cast<T*>(s.x)[I] = X[I];
    }
  }
}

template <class T>
void launch_small_smooth(const SmallSm& s, cudaStream_t st) {
  const size_t smem = 4 * (size_t)s.g.len * sizeof(T);
  static bool attr = false, attr_c = false;
  if (!attr) {
    cudaFuncSetAttribute(k_small_smooth<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmemMax);
    attr = true;
  }
  if (sizeof(T) == 8 && s.g.len >= kSmallCluMinCells) {
    if (!attr_c) {
      cudaFuncSetAttribute(k_small_smooth_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmemMax);
      attr_c = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kSmallCtas, 1, 1);
    cfg.blockDim = dim3(kSmallCluThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kSmallCtas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = tl_dep_launch ? 2 : 1;
    cudaLaunchKernelEx(&cfg, k_small_smooth_cluster, s);
    return;
  }
  launch_dep(k_small_smooth<T>, 1, kSmallThreads, smem, st, s);
}
template void launch_small_smooth<double>(const SmallSm&, cudaStream_t);
template void launch_small_smooth<float>(const SmallSm&, cudaStream_t);

// ------------------------------------------------------------------- halo
// fill! for :xperio (src/halo.jl:6-9). One thread per (j,k) line copies the
// nh columns through registers, so the copies of each statement read
// before they write, as Julia's sliced assignment does.
template <class T>
__global__ void __launch_bounds__(kThreads) k_fill_xperio(T* __restrict__ x, int tx, int nh, long long nlines) {
  dep_wait();
  long long L = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (L < nlines) d_fill_line(x + L * tx, tx, nh);
}

// ------------------------------------------------------------------- norm
// Deterministic two-stage reduction in one launch: block b of (up to)
// kNormParts sums the elements b, b+P, b+2P, ... strided by the whole grid of
// kNormParts blocks; the block that finishes last (a counter, back at 0 when
// it is done) adds the kNormParts partials in a fixed tree, so the sum does
// not depend on which block that is. Fields of fewer than kNormParts blocks'
// cells launch only the blocks that hold some; the other partials are 0.
// With `lt` (the solve loop's last kernel) it also tests the stopping rule.
// As two launches and a test kernel these were 3 of the 18 nodes of a 64^2
// FP64 solve's iteration (see launch_norm).
// msk*v^2 for a mask that is neither 0 nor 1: out of line, since inline the
// compiler issued its conversion and three operations for every cell, five on
// the FP64 pipe instead of the one FMA (39 us against 16 at 2048^2)
static __device__ __noinline__ double weighted_square(uint8_t mm, double v, double s) {
  return __dadd_rn(s, __dmul_rn((double)mm, __dmul_rn(v, v)));
}
// s: each thread's sum
__device__ __forceinline__ void norm_finish(double s, double* __restrict__ partials, unsigned* counter, double* out,
                                            const double* normb, int norm_kind, const LoopTest& lt) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s = __dadd_rn(s, __shfl_down_sync(0xffffffffu, s, o));
  __shared__ double ws[kThreads / 32];
  __shared__ bool last;
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = threadIdx.x < kThreads / 32 ? ws[threadIdx.x] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = __dadd_rn(s, __shfl_down_sync(0xffffffffu, s, o));
    if (threadIdx.x == 0) {
      partials[blockIdx.x] = s;
      __threadfence();
      last = atomicInc(counter, gridDim.x - 1) == gridDim.x - 1;
    }
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  __shared__ double sh[kNormParts];
  for (int t = threadIdx.x; t < kNormParts; t += kThreads) sh[t] = t < (int)gridDim.x ? __ldcg(partials + t) : 0.0;
  __syncthreads();
  for (int w = kNormParts / 2; w > 0; w >>= 1) {
    for (int t = threadIdx.x; t < w; t += kThreads) sh[t] = __dadd_rn(sh[t], sh[t + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    double sum = sh[0];
    if (norm_kind == CFMG_NORM_REF_SQUARED && sum == 0.0) sum = 1.0;
    out[0] = sum;
    if (normb) {
      const double nb = *normb;
      const double q = nb > 0.0 ? sum / nb : 0.0;
      const double res = norm_kind == CFMG_NORM_REF_SQUARED ? q : sqrt(q);
      out[1] = res;
      if (lt.on) loop_test(lt, res, nb);
    }
  }
}
template <class T>
__global__ void __launch_bounds__(kThreads) k_norm(const T* __restrict__ x, const uint8_t* __restrict__ m, long long n,
                                                   double* __restrict__ partials, unsigned* counter, double* out,
                                                   const double* normb, int norm_kind, LoopTest lt) {
  dep_wait();
  double s = 0.0;
  const long long st = (long long)kNormParts * kThreads;
  auto add = [&](uint8_t mm, T xv) {
    if (mm) {
      const double v = (double)xv;
      if (mm == 1) s = __fma_rn(v, v, s);
      else s = weighted_square(mm, v, s);
    }
  };
  long long I = (long long)blockIdx.x * kThreads + threadIdx.x;
  for (; I + 3 * st < n; I += 4 * st) {  // four elements' loads in flight, added in their order
    const uint8_t m0 = m[I], m1 = m[I + st], m2 = m[I + 2 * st], m3 = m[I + 3 * st];
    const T x0 = x[I], x1 = x[I + st], x2 = x[I + 2 * st], x3 = x[I + 3 * st];
    add(m0, x0);
    add(m1, x1);
    add(m2, x2);
    add(m3, x3);
  }
  for (; I < n; I += st) add(m[I], x[I]);
  norm_finish(s, partials, counter, out, normb, norm_kind, lt);
}
__global__ void k_loop_start(LoopTest lt) {
  lt.ds[S_NITE] = 0.0;
  loop_test(lt, lt.ds[S_RES], lt.ds[S_NORMB]);
}
void launch_loop_start(const LoopTest& lt, cudaStream_t s) { k_loop_start<<<1, 1, 0, s>>>(lt); }

// An FP64 level's residual and its norm in one launch, for levels of at most
// one cell a thread of the norm (kNormParts blocks: 262 144 cells), whose two
// launches are latency: the cell's residual as the separate kernel stores it
// (cells out of its range keep their r), then the norm's own sums. A 64^2 FP64
// solve takes 909 us with it and 963 with two launches.
template <int KIND>
__global__ void __launch_bounds__(kThreads) k_resid_norm(double* __restrict__ r, const double* __restrict__ x,
                                                         const double* __restrict__ b, const double* __restrict__ d,
                                                         const double* __restrict__ cE, const double* __restrict__ cN,
                                                         const uint8_t* __restrict__ m, Geom g, Box bx, long long lo,
                                                         long long hi, long long n, double* __restrict__ partials,
                                                         unsigned* counter, double* out, const double* normb,
                                                         int norm_kind, LoopTest lt) {
  dep_wait();
  const long long I = (long long)blockIdx.x * kThreads + threadIdx.x;
  double s = 0.0;
  if (I < n) {
    bool in;
    if (KIND == OPK_RESID5 || KIND == OPK_RESIDVC) {
      in = I >= lo && I < hi;
    } else {
      const int k = (int)(I / g.n2), q = (int)(I - k * g.n2), j = q / (int)g.n1, i = q - j * (int)g.n1;
      in = i + 1 >= bx.i0 && i + 1 <= bx.i1 && j + 1 >= bx.j0 && j + 1 <= bx.j1 && k + 1 >= bx.k0 && k + 1 <= bx.k1;
    }
    const uint8_t mm = m[I];
    double v = 0.0;
    if (in) {
      if (KIND == OPK_RESID5) v = v_resid5(x, b, d, m, g.n1, I);
      if (KIND == OPK_RESID7) v = v_resid7(x, b, d, m, g.n1, g.n2, I);
      if (KIND == OPK_RESID9) v = v_resid9(x, b, d, m, g.n1, I);
      if (KIND == OPK_RESID19) v = v_resid19(x, b, d, m, g.n1, g.n2, I);
      if (KIND == OPK_RESIDVC) v = v_residvc(x, b, d, cE, cN, m, g.n1, I);
      r[I] = v;
    } else if (mm) {
      v = r[I];
    }
    if (mm == 1) s = __fma_rn(v, v, s);
    else if (mm) s = weighted_square(mm, v, s);
  }
  norm_finish(s, partials, counter, out, normb, norm_kind, lt);
}
bool launch_resid_norm(int kind, double* r, const double* x, const double* b, const double* d, const double* cE,
                       const double* cN, const uint8_t* m, const Geom& g, const Box& bx, double* partials,
                       unsigned* counter, double* out, const double* normb, int norm_kind, cudaStream_t s,
                       const LoopTest* lt) {
  const long long n = g.len;
  const unsigned nb = nblocks(n);
  switch (kind) {
#define CFMG_RN(K)                                                                                              \
  case K:                                                                                                       \
    launch_dep(k_resid_norm<K>, nb, kThreads, 0, s, r, x, b, d, cE, cN, m, g, bx, g.n1, g.len - g.n1, n, partials, \
               counter, out, normb, norm_kind, lt ? *lt : LoopTest{});                                         \
    return true;
    CFMG_RN(OPK_RESID5)
    CFMG_RN(OPK_RESID7)
    CFMG_RN(OPK_RESID9)
    CFMG_RN(OPK_RESID19)
    CFMG_RN(OPK_RESIDVC)
#undef CFMG_RN
    default: return false;
  }
}

// --------------------------------------------------------------- launchers
template <class T>
void launch_sweep5_2d(const T* x, T* y, const T* b, const T* w, T cff, const Geom& g, cudaStream_t s) {
  long long lo = g.n1, hi = g.len - g.n1;
  if (hi <= lo) return;
  CFMG_ZS(k_sweep5_2d, hi - lo, nblocks(hi - lo), kThreads, 0, s, x, y, b, w, cff, g.n1, lo, hi);
}
template <class T>
void launch_sweep7_3d(const T* x, T* y, const T* b, const T* w, T cff, const Geom& g, cudaStream_t s) {
  long long lo = g.n2, hi = g.len - g.n2;
  if (hi <= lo) return;
  CFMG_ZS(k_sweep7_3d, hi - lo, nblocks(hi - lo), kThreads, 0, s, x, y, b, w, cff, g.n1, g.n2, lo, hi);
}
// The FP32 7-point sweep of a 3D level (the linear range n2 .. len-n2 of
// sloop3d_v1!, src/laplacian.jl:11-20: every (i, j) of the planes k = 2 ..
// tz-1), register-blocked along k: a thread owns one (i, j) column and a
// run of kKRun planes, carries x at k-1, k and k+1 in registers from one
// plane to the next, and takes the four in-plane neighbours from L1 (the
// block covers 32 x 8 columns). omega*idiag is read as a one-byte code into
// a 256-entry table (L1-resident): 13 instead of 16 bytes of traffic per
// cell. The per-cell arithmetic and its order are k_sweep7_3d<float>'s
// (faces6, then cff*x - w*(b - faces)), so the bits are the same.
constexpr int kKRun = 8;
__global__ void __launch_bounds__(256) k_sweep7_3d_q(const float* __restrict__ x, float* __restrict__ y,
                                                     const float* __restrict__ b, const uint8_t* __restrict__ wq,
                                                     const float* __restrict__ wtab, float cff, int tx, int ty,
                                                     int tz) {
  dep_wait();
  const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y;
  const int k0 = 1 + blockIdx.z * kKRun;  // 0-based planes k0 .. k1-1 of 1 .. tz-2
  if (i >= tx || j >= ty || k0 > tz - 2) return;
  const int k1 = min(k0 + kKRun, tz - 1);
  typedef Ar<float> A;
  const long long n1 = tx, n2 = (long long)tx * ty;
  long long I = (long long)i + n1 * j + n2 * k0;
  float xm = x[I - n2], xc = x[I];
  for (int k = k0; k < k1; ++k, I += n2) {
    const float xp = x[I + n2];
    const float f = A::add(A::add(A::add(A::add(A::add(x[I - 1], x[I + 1]), x[I - n1]), x[I + n1]), xm), xp);
    const float w = __ldg(wtab + wq[I]);
    y[I] = A::sub(A::mul(cff, xc), A::mul(w, A::sub(b[I], f)));
    xm = xc;
    xc = xp;
  }
}
// The same sweep four cells at a time: a thread owns a quad of consecutive
// linear indices of a plane (16-byte loads of x at k and k +- 1, of b and of
// the four codes; the j -+ 1 rows as two 8-byte loads each, since an even
// row length tx leaves them 8-byte aligned only; the two cells beside the
// quad as single loads) and a run of kQRun planes, with the code table in
// shared memory. It needs n2 = tx*ty a multiple of 4, tx even and 16-byte
// aligned arrays. A 512x512x256 sweep (tx = ty = 518): 193 -> 140 us, 0.96 of
// the measured HBM copy bandwidth for its 13 bytes a cell (against four
// times as many load instructions in the one-cell form, whose warps stalled
// on the load queue). Each cell's arithmetic is the one-cell form's.
// ZERO: x is known to hold +0 in every cell (the first sweep of a cycle's
// level-1 pre-smoothing): it is not read, and the same formula on +0
// operands gives the same bits.
//
// qact (optional): a quad whose cells are dry in every plane of the run is
// skipped. In the mixed form's FP32 fields a dry cell holds +0 in x, y and b
// and has omega*idiag = 0, so the sweep would write +0 over +0 there.
//
// run: planes a thread sweeps, kQRun or 1. A run reads each plane once instead
// of three times but takes its planes one after the other; a level that gives
// fewer than kQBlocks blocks an SM in runs is bound by that chain of loads, and
// takes a plane a thread (70 x 70 x 38 and below of a 512 x 512 x 256 solve:
// 7.4-7.9 -> 4.3-5.1 us a sweep).
constexpr int kQRun = kQRunPlanes;
constexpr int kQBlocks = 4;  // an SM
template <bool ZERO>
__global__ void __launch_bounds__(256) k_sweep7_3d_q4(const float* __restrict__ x, float* __restrict__ y,
                                                      const float* __restrict__ b, const uint8_t* __restrict__ wq,
                                                      const float* __restrict__ wtab, float cff, long long n1,
                                                      long long n2, int tz, const uint8_t* __restrict__ qact,
                                                      int run) {
  __shared__ float tab[256];
  dep_wait();
  const long long t = (long long)blockIdx.x * 256 + threadIdx.x;  // quad of the plane
  const int k0 = 1 + blockIdx.y * run;
  const bool live = 4 * t < n2 && k0 <= tz - 2 && (!qact || qact[(long long)((k0 - 1) / kQRun) * (n2 >> 2) + t]);
  if (!__syncthreads_or(live)) return;  // a block of dry quads reads nothing more
  tab[threadIdx.x] = wtab[threadIdx.x];
  __syncthreads();
  if (!live) return;
  const int k1 = min(k0 + run, tz - 1);
  typedef Ar<float> A;
  long long I = 4 * t + n2 * k0;
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const float2 z2 = make_float2(0.f, 0.f);
  auto ld4 = [&](long long J) { return ZERO ? z4 : *reinterpret_cast<const float4*>(x + J); };
  auto ld2 = [&](long long J) { return ZERO ? z2 : *reinterpret_cast<const float2*>(x + J); };
  float4 xm = ld4(I - n2), xc = ld4(I);
  for (int k = k0; k < k1; ++k, I += n2) {
    const float4 xp = ld4(I + n2);
    const float xw = ZERO ? 0.f : x[I - 1], xe = ZERO ? 0.f : x[I + 4];
    const float2 s0 = ld2(I - n1), s1 = ld2(I - n1 + 2);
    const float2 u0 = ld2(I + n1), u1 = ld2(I + n1 + 2);
    const float4 bb = *reinterpret_cast<const float4*>(b + I);
    const uchar4 q = *reinterpret_cast<const uchar4*>(wq + I);
    const float f0 = A::add(A::add(A::add(A::add(A::add(xw, xc.y), s0.x), u0.x), xm.x), xp.x);
    const float f1 = A::add(A::add(A::add(A::add(A::add(xc.x, xc.z), s0.y), u0.y), xm.y), xp.y);
    const float f2 = A::add(A::add(A::add(A::add(A::add(xc.y, xc.w), s1.x), u1.x), xm.z), xp.z);
    const float f3 = A::add(A::add(A::add(A::add(A::add(xc.z, xe), s1.y), u1.y), xm.w), xp.w);
    const float w0 = tab[q.x], w1 = tab[q.y], w2 = tab[q.z], w3 = tab[q.w];
    float4 o;
    o.x = A::sub(A::mul(cff, xc.x), A::mul(w0, A::sub(bb.x, f0)));
    o.y = A::sub(A::mul(cff, xc.y), A::mul(w1, A::sub(bb.y, f1)));
    o.z = A::sub(A::mul(cff, xc.z), A::mul(w2, A::sub(bb.z, f2)));
    o.w = A::sub(A::mul(cff, xc.w), A::mul(w3, A::sub(bb.w, f3)));
    *reinterpret_cast<float4*>(y + I) = o;
    xm = xc;
    xc = xp;
  }
}
bool sweep7_quad_ok(const Geom& g, const void* x, const void* y, const void* b, const void* wq) {
  return g.n2 % 4 == 0 && g.n1 % 2 == 0 && ((uintptr_t)x | (uintptr_t)y | (uintptr_t)b) % 16 == 0 &&
         (uintptr_t)wq % 4 == 0;
}
void launch_sweep7_3d_q(const float* x, float* y, const float* b, const uint8_t* wq, const float* wtab, float cff,
                        const Geom& g, cudaStream_t s, bool x_zero, const uint8_t* qact) {
  if (g.tz < 3) return;
  if (sweep7_quad_ok(g, x, y, b, wq)) {
    const long long nb = (g.n2 / 4 + 255) / 256;
    const int run = nb * ((g.tz - 2 + kQRun - 1) / kQRun) < kQBlocks * sm_count() ? 1 : kQRun;
    const dim3 grid((unsigned)nb, (unsigned)((g.tz - 2 + run - 1) / run));
    if (x_zero)
      launch_dep(k_sweep7_3d_q4<true>, grid, 256, 0, s, x, y, b, wq, wtab, cff, g.n1, g.n2, g.tz, qact, run);
    else
      launch_dep(k_sweep7_3d_q4<false>, grid, 256, 0, s, x, y, b, wq, wtab, cff, g.n1, g.n2, g.tz, qact, run);
    return;
  }
  if (x_zero) cudaMemsetAsync(const_cast<float*>(x), 0, (size_t)g.len * sizeof(float), s);  // the one-cell form reads x
  const dim3 grid((unsigned)((g.tx + 31) / 32), (unsigned)((g.ty + 7) / 8), (unsigned)((g.tz - 2 + kKRun - 1) / kKRun));
  launch_dep(k_sweep7_3d_q, grid, dim3(32, 8, 1), 0, s, x, y, b, wq, wtab, cff, g.tx, g.ty, g.tz);
}

// The FP32 19-point sweep (smooth_laplacian9!'s body, src/laplacian9.jl:14-44)
// four cells a thread, over a box: a thread owns a quad of consecutive
// linear indices of a plane and a run of kQ19Run planes, carrying the quad's
// neighbourhood of planes k-1, k and k+1 in registers (x of its row as a
// 16-byte load and the cells beside it, the rows j -/+ 1 as 8-byte pairs and
// their cells beside). Cells of the quad outside the box are computed but not
// stored. v_sweep19's arithmetic, in its order. Needs n2 = tx*ty a multiple
// of 4, tx even, 16-byte aligned arrays and a halo of at least 3 (every read
// then stays inside the array).
constexpr int kQ19Run = 4;
struct Q19Plane {
  float4 c;        // row j: the quad
  float cw, ce;    // row j: beside the quad
  float4 s, n;     // rows j-1 and j+1 under the quad
  float sw, se, nw, ne;
};
__device__ __forceinline__ Q19Plane q19_load(const float* __restrict__ x, long long P, long long n1) {
  Q19Plane r;
  r.c = *reinterpret_cast<const float4*>(x + P);
  r.cw = x[P - 1];
  r.ce = x[P + 4];
  const float2 s0 = *reinterpret_cast<const float2*>(x + P - n1), s1 = *reinterpret_cast<const float2*>(x + P - n1 + 2);
  const float2 u0 = *reinterpret_cast<const float2*>(x + P + n1), u1 = *reinterpret_cast<const float2*>(x + P + n1 + 2);
  r.s = make_float4(s0.x, s0.y, s1.x, s1.y);
  r.n = make_float4(u0.x, u0.y, u1.x, u1.y);
  r.sw = x[P - n1 - 1];
  r.se = x[P - n1 + 4];
  r.nw = x[P + n1 - 1];
  r.ne = x[P + n1 + 4];
  return r;
}
__device__ __forceinline__ float q4at(const float4& v, int c) { return c == 0 ? v.x : c == 1 ? v.y : c == 2 ? v.z : v.w; }
__global__ void __launch_bounds__(256) k_sweep19_3d_q4(const float* __restrict__ x, float* __restrict__ y,
                                                       const float* __restrict__ b, const float* __restrict__ w,
                                                       float cff, long long n1, long long n2, Box bx, long long q0,
                                                       long long nq, int run) {
  dep_wait();
  const long long qi = q0 + (long long)blockIdx.x * 256 + threadIdx.x;  // quad of the plane
  const int k0 = (bx.k0 - 1) + (int)blockIdx.y * run;                   // 0-based planes k0 .. k1-1
  if (qi >= q0 + nq || k0 > bx.k1 - 1) return;
  const int k1 = min(k0 + run, bx.k1);
  const long long Lp = 4 * qi;
  const int jq = (int)(Lp / n1), iq = (int)(Lp - (long long)jq * n1);
  bool inb[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    int i = iq + c, j = jq;
    if (i >= n1) {
      i -= (int)n1;
      ++j;
    }
    inb[c] = i >= bx.i0 - 1 && i <= bx.i1 - 1 && j >= bx.j0 - 1 && j <= bx.j1 - 1;
  }
  if (!(inb[0] || inb[1] || inb[2] || inb[3])) return;
  const bool all = inb[0] && inb[1] && inb[2] && inb[3];
  typedef Ar<float> A;
  long long I = Lp + n2 * k0;
  Q19Plane pm = q19_load(x, I - n2, n1), pc = q19_load(x, I, n1);
  for (int k = k0; k < k1; ++k, I += n2) {
    const Q19Plane pp = q19_load(x, I + n2, n1);
    const float4 bb = *reinterpret_cast<const float4*>(b + I), ww = *reinterpret_cast<const float4*>(w + I);
    float o[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float xw = c == 0 ? pc.cw : q4at(pc.c, c - 1), xe = c == 3 ? pc.ce : q4at(pc.c, c + 1);
      const float sw = c == 0 ? pc.sw : q4at(pc.s, c - 1), se = c == 3 ? pc.se : q4at(pc.s, c + 1);
      const float nw = c == 0 ? pc.nw : q4at(pc.n, c - 1), ne = c == 3 ? pc.ne : q4at(pc.n, c + 1);
      const float mw = c == 0 ? pm.cw : q4at(pm.c, c - 1), me = c == 3 ? pm.ce : q4at(pm.c, c + 1);
      const float pw = c == 0 ? pp.cw : q4at(pp.c, c - 1), pe = c == 3 ? pp.ce : q4at(pp.c, c + 1);
      const float f = A::add(A::add(A::add(A::add(A::add(xw, xe), q4at(pc.s, c)), q4at(pc.n, c)), q4at(pm.c, c)),
                             q4at(pp.c, c));
      float e = A::add(sw, se);
      e = A::add(e, nw);
      e = A::add(e, ne);
      e = A::add(e, mw);
      e = A::add(e, me);
      e = A::add(e, pw);
      e = A::add(e, pe);
      e = A::add(e, q4at(pm.s, c));
      e = A::add(e, q4at(pm.n, c));
      e = A::add(e, q4at(pp.s, c));
      e = A::add(e, q4at(pp.n, c));
      float t = A::fmx(f, -0.5f, q4at(bb, c));
      t = A::fmx(e, -0.25f, t);
      o[c] = A::sub(A::mul(cff, q4at(pc.c, c)), A::mul(q4at(ww, c), t));
    }
    if (all) {
      *reinterpret_cast<float4*>(y + I) = make_float4(o[0], o[1], o[2], o[3]);
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (inb[c]) y[I + c] = o[c];
    }
    pm = pc;
    pc = pp;
  }
}
bool launch_sweep19_3d_q4(const float* x, float* y, const float* b, const float* w, float cff, const Geom& g,
                          const Box& bx, cudaStream_t s) {
  if (g.n2 % 4 != 0 || g.n1 % 2 != 0 || g.nh < 3 || ((uintptr_t)x | (uintptr_t)y | (uintptr_t)b | (uintptr_t)w) % 16)
    return false;
  if (box_empty(bx)) return true;
  const long long q0 = (g.n1 * (bx.j0 - 1)) / 4, qe = (g.n1 * bx.j1 + 3) / 4;  // quads covering rows j0 .. j1
  const long long nq = qe - q0;
  const long long nb = (nq + 255) / 256;
  const int nk = bx.k1 - bx.k0 + 1, run = nb * ((nk + kQ19Run - 1) / kQ19Run) < kQBlocks * sm_count() ? 1 : kQ19Run;
  const dim3 grid((unsigned)nb, (unsigned)((nk + run - 1) / run));
  launch_dep(k_sweep19_3d_q4, grid, 256, 0, s, x, y, b, w, cff, g.n1, g.n2, bx, q0, nq, run);
  return true;
}

template <class T>
void launch_sweep9_2d(const T* x, T* y, const T* b, const T* w, T cff, const Geom& g, const Box& bx,
                      cudaStream_t s) {
  if (box_empty(bx)) return;
  if constexpr (sizeof(T) == 8) {
    if (g.tz == 1 && box_cells(bx) >= kFixMin) return launch_fix_sweep9(x, y, b, w, cff, g, bx, s);
  }
  launch_dep(k_sweep9_2d<T>, box_grid(bx, kBoxBlk), kBoxBlk, 0, s, x, y, b, w, cff, g, bx);
}
template <class T>
void launch_sweep19_3d(const T* x, T* y, const T* b, const T* w, T cff, const Geom& g, const Box& bx,
                       cudaStream_t s) {
  if (box_empty(bx)) return;
  CFMG_ZS(k_sweep19_3d, box_cells(bx), box_grid(bx, kBoxBlk), kBoxBlk, 0, s, x, y, b, w, cff, g, bx);
}
template <class T>
void launch_sweep_vc_2d(const T* x, T* y, const T* b, const T* w, const T* cE, const T* cN, T cff, const Geom& g,
                        cudaStream_t s) {
  long long lo = g.n1, hi = g.len - g.n1;
  if (hi <= lo) return;
  CFMG_ZS(k_sweep_vc_2d, hi - lo, nblocks(hi - lo), kThreads, 0, s, x, y, b, w, cE, cN, cff, g.n1, lo, hi);
}
template <class T>
void launch_resid5_2d(T* r, const T* x, const T* b, const T* d, const uint8_t* m, const Geom& g, cudaStream_t s) {
  long long lo = g.n1, hi = g.len - g.n1;
  if (hi <= lo) return;
  CFMG_ZS(k_resid5_2d, hi - lo, nblocks(hi - lo), kThreads, 0, s, r, x, b, d, m, g.n1, lo, hi);
}
template <class T>
void launch_resid7_3d(T* r, const T* x, const T* b, const T* d, const uint8_t* m, const Geom& g, const Box& bx,
                      cudaStream_t s) {
  if (box_empty(bx)) return;
  CFMG_ZS(k_resid7_3d, box_cells(bx), box_grid(bx, kBoxBlk), kBoxBlk, 0, s, r, x, b, d, m, g, bx);
}
template <class T>
void launch_resid9_2d(T* r, const T* x, const T* b, const T* d, const uint8_t* m, const Geom& g, const Box& bx,
                      cudaStream_t s) {
  if (box_empty(bx)) return;
  if constexpr (sizeof(T) == 8) {
    if (g.tz == 1 && box_cells(bx) >= kFixMin) return launch_fix_resid9(r, x, b, d, m, g, bx, s);
  }
  launch_dep(k_resid9_2d<T>, box_grid(bx, kBoxBlk), kBoxBlk, 0, s, r, x, b, d, m, g, bx);
}
template <class T>
void launch_resid19_3d(T* r, const T* x, const T* b, const T* d, const uint8_t* m, const Geom& g, const Box& bx,
                       cudaStream_t s) {
  if (box_empty(bx)) return;
  CFMG_ZS(k_resid19_3d, box_cells(bx), box_grid(bx, kBoxBlk), kBoxBlk, 0, s, r, x, b, d, m, g, bx);
}
template <class T>
void launch_resid_vc_2d(T* r, const T* x, const T* b, const T* d, const T* cE, const T* cN, const uint8_t* m,
                        const Geom& g, cudaStream_t s) {
  long long lo = g.n1, hi = g.len - g.n1;
  if (hi <= lo) return;
  CFMG_ZS(k_resid_vc_2d, hi - lo, nblocks(hi - lo), kThreads, 0, s, r, x, b, d, cE, cN, m, g.n1, lo, hi);
}
template <class T>
void launch_restrict(int kind, const T* xf, T* bc, const T* Rcoef, const Geom& gf, const Geom& gc, const Box& cb,
                     cudaStream_t s) {
  if (box_empty(cb)) return;
  dim3 grid = box_grid(cb, kBoxBlk);
  // the fine cells that it reads decide (see kZeroMin)
  const bool zs = sizeof(T) == 8 && gf.len >= kZeroMin;
#define CFMG_RES(K)                                                                                     \
  case K:                                                                                               \
    if (zs) launch_dep(k_restrict<T, K, sizeof(T) == 8>, grid, kBoxBlk, 0, s, xf, bc, Rcoef, gf, gc, cb); \
    else launch_dep(k_restrict<T, K, false>, grid, kBoxBlk, 0, s, xf, bc, Rcoef, gf, gc, cb);           \
    break;
  switch (kind) {
    CFMG_RES(0)
    CFMG_RES(1)
    CFMG_RES(2)
    default:
    CFMG_RES(3)
  }
#undef CFMG_RES
}
template <class T>
void launch_prolong(int kind, T* xf, const T* xc, const T* Pcoef, const Geom& gf, const Geom& gc, int nxf, int nyf,
                    int nzf, int kf0, int kf1, bool assign, cudaStream_t s, const uint8_t* fmsk) {
  // parents: i = nh+1 : 2 : nx+nh (likewise j, and k in 3D)
  const int np_i = (nxf + 1) / 2, np_j = (nyf + 1) / 2;
  const bool threed = (kind == 1 || kind == 3);
  const int np_k = threed ? (nzf + 1) / 2 : (kf1 - kf0 + 1);
  if (np_i <= 0 || np_j <= 0 || np_k <= 0) return;
  dim3 blk(64, 4, 1);
  dim3 grid((unsigned)((np_i + 63) / 64), (unsigned)((np_j + 3) / 4), (unsigned)np_k);
  if (sizeof(T) == 4 && kind == 1) {
    if (assign)
      launch_dep(k_prolong3c_f<true>, grid, blk, 0, s, (float*)xf, (const float*)xc, (const float*)Pcoef, gf, gc, np_i,
                 np_j, np_k, fmsk);
    else
      launch_dep(k_prolong3c_f<false>, grid, blk, 0, s, (float*)xf, (const float*)xc, (const float*)Pcoef, gf, gc,
                 np_i, np_j, np_k, fmsk);
    return;
  }
  const bool zs = sizeof(T) == 8 && gf.len >= kZeroMin;
#define CFMG_PRO_L(K, A, Z) \
  launch_dep(k_prolong<T, K, A, Z>, grid, blk, 0, s, xf, xc, Pcoef, gf, gc, np_i, np_j, kf0, kf1, np_k, fmsk)
#define CFMG_PRO(K)                                       \
  case K:                                                 \
    if (assign) CFMG_PRO_L(K, true, false);               \
    else if (zs) CFMG_PRO_L(K, false, sizeof(T) == 8);    \
    else CFMG_PRO_L(K, false, false);                     \
    break;
  switch (kind) {
    CFMG_PRO(0)
    CFMG_PRO(1)
    CFMG_PRO(2)
    default:
    CFMG_PRO(3)
  }
#undef CFMG_PRO
#undef CFMG_PRO_L
}
template <class T>
void launch_fill_xperio(T* x, const Geom& g, cudaStream_t s) {
  long long nlines = (long long)g.ty * g.tz;
  launch_dep(k_fill_xperio<T>, nblocks(nlines), kThreads, 0, s, x, g.tx, g.nh, nlines);
}
template <class T>
void launch_norm(const T* x, const uint8_t* m, size_t n, double* partials, unsigned* counter, double* out,
                 const double* normb, int norm_kind, cudaStream_t s, const LoopTest* lt) {
  const long long nb = ((long long)n + kThreads - 1) / kThreads;
  launch_dep(k_norm<T>, (unsigned)(nb < kNormParts ? nb : kNormParts), kThreads, 0, s, x, m, (long long)n, partials,
             counter, out, normb, norm_kind, lt ? *lt : LoopTest{});
}

#define CFMG_INST(T)                                                                                             \
  template void launch_sweep5_2d<T>(const T*, T*, const T*, const T*, T, const Geom&, cudaStream_t);            \
  template void launch_sweep7_3d<T>(const T*, T*, const T*, const T*, T, const Geom&, cudaStream_t);            \
  template void launch_sweep9_2d<T>(const T*, T*, const T*, const T*, T, const Geom&, const Box&, cudaStream_t); \
  template void launch_sweep19_3d<T>(const T*, T*, const T*, const T*, T, const Geom&, const Box&,              \
                                     cudaStream_t);                                                              \
  template void launch_sweep_vc_2d<T>(const T*, T*, const T*, const T*, const T*, const T*, T, const Geom&,      \
                                      cudaStream_t);                                                             \
  template void launch_resid5_2d<T>(T*, const T*, const T*, const T*, const uint8_t*, const Geom&, cudaStream_t); \
  template void launch_resid7_3d<T>(T*, const T*, const T*, const T*, const uint8_t*, const Geom&, const Box&,   \
                                    cudaStream_t);                                                               \
  template void launch_resid9_2d<T>(T*, const T*, const T*, const T*, const uint8_t*, const Geom&, const Box&,   \
                                    cudaStream_t);                                                               \
  template void launch_resid19_3d<T>(T*, const T*, const T*, const T*, const uint8_t*, const Geom&, const Box&,  \
                                     cudaStream_t);                                                              \
  template void launch_resid_vc_2d<T>(T*, const T*, const T*, const T*, const T*, const T*, const uint8_t*,      \
                                      const Geom&, cudaStream_t);                                                \
  template void launch_restrict<T>(int, const T*, T*, const T*, const Geom&, const Geom&, const Box&,            \
                                   cudaStream_t);                                                                \
  template void launch_prolong<T>(int, T*, const T*, const T*, const Geom&, const Geom&, int, int, int, int, int, \
                                  bool, cudaStream_t, const uint8_t*);                                           \
  template void launch_fill_xperio<T>(T*, const Geom&, cudaStream_t);                                            \
  template void launch_norm<T>(const T*, const uint8_t*, size_t, double*, unsigned*, double*, const double*, int,    \
                               cudaStream_t, const LoopTest*);

CFMG_INST(double)
CFMG_INST(float)
template void launch_fill_xperio<uint8_t>(uint8_t*, const Geom&, cudaStream_t);

}  // namespace cfmg

namespace cfmg {

__global__ void k_f32_to_f64(const float* a, double* out, long long n) {
  dep_wait();
  long long I = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (I < n) out[I] = (double)a[I];
}
__global__ void k_f64_to_f32(const double* a, float* out, long long n) {
  dep_wait();
  long long I = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (I < n) out[I] = (float)a[I];
}

// One Op as a standalone kernel (fine levels).
template <class T>
static void launch_op_t(const Op& op, cudaStream_t s) {
  const T* x = (const T*)op.x;
  const T* b = (const T*)op.b;
  const T* w = (const T*)op.w;
  const T* d = (const T*)op.d;
  T* y = (T*)op.y;
  const T cff = (T)op.cff;
  switch (op.kind) {
    case OPK_SWEEP5: launch_sweep5_2d<T>(x, y, b, w, cff, op.g, s); break;
    case OPK_SWEEP7:
      if (sizeof(T) == 4 && op.wq)
        launch_sweep7_3d_q((const float*)x, (float*)y, (const float*)b, op.wq, op.wtab, (float)cff, op.g, s,
                           op.assign != 0, op.qact);
      else
        launch_sweep7_3d<T>(x, y, b, w, cff, op.g, s);
      break;
    case OPK_SWEEP9: launch_sweep9_2d<T>(x, y, b, w, cff, op.g, op.box, s); break;
    case OPK_SWEEP19:
      if (!(sizeof(T) == 4 && launch_sweep19_3d_q4((const float*)x, (float*)y, (const float*)b, (const float*)w,
                                                   (float)cff, op.g, op.box, s)))
        launch_sweep19_3d<T>(x, y, b, w, cff, op.g, op.box, s);
      break;
    case OPK_SWEEPVC: launch_sweep_vc_2d<T>(x, y, b, w, (const T*)op.cE, (const T*)op.cN, cff, op.g, s); break;
    case OPK_RESID5: launch_resid5_2d<T>(y, x, b, d, op.m, op.g, s); break;
    case OPK_RESID7: launch_resid7_3d<T>(y, x, b, d, op.m, op.g, op.box, s); break;
    case OPK_RESID9: launch_resid9_2d<T>(y, x, b, d, op.m, op.g, op.box, s); break;
    case OPK_RESID19: launch_resid19_3d<T>(y, x, b, d, op.m, op.g, op.box, s); break;
    case OPK_RESIDVC: launch_resid_vc_2d<T>(y, x, b, d, (const T*)op.cE, (const T*)op.cN, op.m, op.g, s); break;
    case OPK_RESTRICT0:
    case OPK_RESTRICT1:
    case OPK_RESTRICT2:
    case OPK_RESTRICT3:
      launch_restrict<T>(op.kind - OPK_RESTRICT0, x, y, (const T*)op.coef, op.g, op.gc, op.box, s);
      break;
    case OPK_PROLONG0:
    case OPK_PROLONG1:
    case OPK_PROLONG2:
    case OPK_PROLONG3: {
      const int kind = op.kind - OPK_PROLONG0;
      const bool t3 = (kind == 1 || kind == 3);
      // launch_prolong derives the parent counts from (nx, ny, nz) of the fine level
      launch_prolong<T>(kind, y, x, (const T*)op.coef, op.g, op.gc, 2 * op.np_i, 2 * op.np_j,
                        t3 ? 2 * (op.kf1 - op.kf0 + 1) : 1, op.kf0, op.kf1, op.assign != 0, s, op.m);
      break;
    }
    case OPK_FILL: launch_fill_xperio<T>(y, op.g, s); break;
    case OPK_ZERO: cudaMemsetAsync(y, 0, op.n * sizeof(T), s); break;
    default: break;
  }
}

void launch_op(const Op& op, cudaStream_t s) {
  if (op.kind == OPK_F32TO64) {
    launch_dep(k_f32_to_f64, nblocks(op.n), kThreads, 0, s, (const float*)op.x, (double*)op.y, op.n);
    return;
  }
  if (op.kind == OPK_F64TO32) {
    launch_dep(k_f64_to_f32, nblocks(op.n), kThreads, 0, s, (const double*)op.x, (float*)op.y, op.n);
    return;
  }
  if (op.prec == 0) launch_op_t<double>(op, s);
  else launch_op_t<float>(op, s);
}

}  // namespace cfmg
