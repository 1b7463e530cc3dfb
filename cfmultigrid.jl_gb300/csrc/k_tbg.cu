// Descent and ascent steps of FP64 2D levels in one launch each (closed
// topology, one layer, 5-point, 9-point and variable-coefficient operators).
//
// A mid-size FP64 level (1500 to 150 000 cells) takes 12 launches a cycle
// (4 sweeps, residual, restriction, zeroing, prolongation, 4 sweeps) whose
// own work is below a microsecond each: launch and load latency, 2.1 us a
// graph node, is what they cost. Here a block loads a tile with a halo wide
// enough for the whole step into shared memory and runs it there:
//   descent: x = +0, or x = Pcoef P(coarse x) after an F-cycle's prolongation;
//            np pairs of sweeps; residual; restriction into the coarse b, the
//            coarse x zeroed
//   ascent:  x = x + Pcoef P(coarse x), np pairs of sweeps
// Each sweep covers the tile's cells that later ones need: sweep s leaves a
// margin of s + 1 cells. The tiles overlap, so a step must not read what it
// writes: a descent reads no x at all, and leaves a copy of its result in the
// level's scratch array, which is what the ascent reads. Level 1 starts from
// the caller's x; its descent writes the scratch only, and the ascent x and y.
//
// Every cell of the tile is updated by the same formula, which rests on the
// coefficients that setup_operators made (the caller checks that they are)
// and on omega <= 1: outside the wet interior x, y and the coarse levels' x
// hold +0 and omega*idiag, Pcoef are +0, so the formula leaves +0 there. (On
// level 1 x may hold anything there: with omega*idiag = +0 the formula is the
// reference's (1-omega) x in its sweep range, and cells out of range matter to
// no cell with omega*idiag != 0; the 9-point operator's second sweep, over the
// interior only, leaves the others alone.) The
// arithmetic per cell is that of the separate kernels, and x, y, r and the
// coarse b and x receive what those would leave: the same bits.
//
// The FP64 pipe of one SM does a tile's work, so the tile size is the one
// with the least work for the busiest SM (tbg_tile): small tiles for levels
// that would leave SMs idle, at the price of a wider relative halo. A warp
// whose cells are all land (zeros) skips the arithmetic.
#include <algorithm>

#include "ops_dev.cuh"

namespace cfmg {

namespace {

constexpr int kGThreads = 256;
constexpr int kGMaxTile = 40;

// cell t of an n x n square: row t / n by a multiplication exact for t < 4096, n <= 64
struct Sq {
  unsigned n, inv;
  __device__ __forceinline__ explicit Sq(int nn) : n(nn), inv((1u << 20) / nn + 1) {}
  __device__ __forceinline__ void at(int t, int& i, int& j) const {
    const unsigned q = ((unsigned)t * inv) >> 20;
    j = (int)q;
    i = t - (int)(q * n);
  }
};

template <int ST>
__device__ __forceinline__ double g_cell(const double* x, int L, int S, double b, double w, double cff,
                                         const double* cE, const double* cN) {
  typedef Ar<double> A;
  double t;
  if (ST == TAIL_9) {
    t = A::fmx(sum4(x, L, S), -0.5, b);
    t = A::fmx(diags4(x, L, S), -0.25, t);
  } else if (ST == TAIL_VC) {
    t = A::sub(b, vc_sum(x, cE, cN, L, S));
  } else {
    t = A::sub(b, sum4(x, L, S));
  }
  return A::sub(A::mul(cff, x[L]), A::mul(w, t));
}

// x = b = +-0, w = +0 and every neighbour a zero: the update of an x of +0 is +0
template <int ST>
__device__ __forceinline__ bool g_land(const double* x, int L, int S, double b, double w) {
  ZeroAcc z;
  z.add(b);
  z.add(x[L - 1]);
  z.add(x[L + 1]);
  z.add(x[L - S]);
  z.add(x[L + S]);
  if (ST == TAIL_9) {
    z.add(x[L - 1 - S]);
    z.add(x[L + 1 - S]);
    z.add(x[L - 1 + S]);
    z.add(x[L + 1 + S]);
  }
  return z.zero() && (__double_as_longlong(x[L]) | __double_as_longlong(w)) == 0ll;
}

// MODE 0: descent from x = +0; 1: descent from x = Pcoef P(xc); 2: ascent.
// KIND 0: cell centres, 2: vertices (restriction and prolongation).
template <int ST, int MODE, int KIND>
__global__ void __launch_bounds__(kGThreads) k_step2d(TbgArgs a, int S, int core) {
  dep_wait();
  typedef Ar<double> A;
  extern __shared__ double gsm[];
  const int n2 = S * S, np = a.np, H = (S - core) / 2, tid = threadIdx.x;
  double* X = gsm;
  double* Y = X + n2;
  double* B = Y + n2;
  double* W = B + n2;
  double* E = W + n2;
  double* N = E + n2;
  const int i0 = 1 + (int)blockIdx.x * core - H, j0 = 1 + (int)blockIdx.y * core - H;  // 1-based tile origin
  const int tx = a.tx, ty = a.ty, nh = a.nh;
  const Sq all(S);
  for (int t = tid; t < n2; t += kGThreads) {
    int i, j;
    all.at(t, i, j);
    const int gi = i0 + i, gj = j0 + j;
    const bool in = gi >= 1 && gi <= tx && gj >= 1 && gj <= ty;
    const long long I = in ? (long long)(gi - 1) + (long long)tx * (gj - 1) : 0;
    double xv = 0.0;
    if ((MODE == 2 || a.xs) && in) xv = a.xs[I];
    B[t] = in ? a.b[I] : 0.0;
    W[t] = in ? a.w[I] : 0.0;
    if (ST == TAIL_VC) {
      E[t] = in ? a.cE[I] : 0.0;
      N[t] = in ? a.cN[I] : 0.0;
    }
    if (MODE != 0) {
      // parents (p, q) update their children; the others keep x
      const int p = gi - nh - 1, q = gj - nh - 1;
      const bool fam = p >= 0 && p < 2 * a.np_i && q >= 0 && q < 2 * a.np_j;
      const double pc = fam ? a.pc[I] : 0.0;
      const bool live = __double_as_longlong(pc) != 0ll;
      if (__any_sync(__activemask(), live) && live) {
        const long long C = (long long)((p >> 1) + nh) + (long long)a.ctx * ((q >> 1) + nh);
        const double v = prolong_child<double, KIND>(a.xc, C, a.ctx, 0, (p & 1) | ((q & 1) << 1));
        xv = A::add(xv, A::mul(pc, v));
      }
    }
    X[t] = xv;
    Y[t] = 0.0;
  }
  __syncthreads();
  for (int s = 0; s < 2 * np; ++s) {
    const double* src = (s & 1) ? Y : X;
    double* dst = (s & 1) ? X : Y;
    const int n = S - 2 * (s + 1);
    const Sq sq(n);
    for (int t = tid; t < n * n; t += kGThreads) {
      int i, j;
      sq.at(t, i, j);
      const int L = (j + s + 1) * S + i + s + 1;
      const double b = B[L], w = W[L];
      if (ST == TAIL_9 && (s & 1)) {  // the interior only
        const int gi = i0 + i + s + 1, gj = j0 + j + s + 1;
        if (gi <= nh || gi > tx - nh || gj <= nh || gj > ty - nh) continue;
      }
      double v = 0.0;
      if (!__all_sync(__activemask(), g_land<ST>(src, L, S, b, w))) v = g_cell<ST>(src, L, S, b, w, a.cff, E, N);
      dst[L] = v;
    }
    __syncthreads();
  }
  // the core of x (and of y, the last odd sweep's result), over the ranges of
  // the reference's sweeps: rows 2 .. ty-1, or ext and interior boxes
  const Sq cs(core);
  for (int t = tid; t < core * core; t += kGThreads) {
    int i, j;
    cs.at(t, i, j);
    const int gi = i0 + H + i, gj = j0 + H + j, L = (j + H) * S + i + H;
    if (gi > tx || gj > ty) continue;
    const long long I = (long long)(gi - 1) + (long long)tx * (gj - 1);
    const bool r1 = ST == TAIL_9 ? gi >= nh && gi <= tx - nh + 1 && gj >= nh && gj <= ty - nh + 1
                                 : gj >= 2 && gj <= ty - 1;
    const bool r2 = ST == TAIL_9 ? gi > nh && gi <= tx - nh && gj > nh && gj <= ty - nh : r1;
    if (r1 && a.y) a.y[I] = Y[L];
    if (r2 && a.x) a.x[I] = X[L];
    if (MODE != 2 && (r2 || a.xs)) a.s[I] = X[L];  // level 1's x out of range counts too
  }
  if (MODE == 2) return;
  __syncthreads();
  // residual of the smoothed x into Y, one cell beyond the core
  const int m = H - 1, nr = core + 2;
  const Sq rs(nr);
  for (int t = tid; t < nr * nr; t += kGThreads) {
    int i, j;
    rs.at(t, i, j);
    const int L = (j + m) * S + i + m, gi = i0 + m + i, gj = j0 + m + j;
    const bool in = gi >= 1 && gi <= tx && gj >= 2 && gj <= ty - 1 &&
                    (ST != TAIL_9 || (gi > nh && gi <= tx - nh && gj > nh && gj <= ty - nh));
    double v = 0.0;
    if (in) {
      const long long I = (long long)(gi - 1) + (long long)tx * (gj - 1);
      const double d = a.d[I];
      v = A::add(A::mul(d, X[L]), B[L]);
      if (ST == TAIL_9) {
        v = A::fmx(sum4(X, L, S), -0.5, v);
        v = A::fmx(diags4(X, L, S), -0.25, v);
      } else if (ST == TAIL_VC) {
        v = A::sub(v, vc_sum(X, E, N, L, S));
      } else {
        v = A::sub(v, sum4(X, L, S));
      }
      v = mask_mul(a.m[I], v);
      if (i > 0 && i <= core && j > 0 && j <= core) a.r[I] = v;
    }
    Y[L] = v;
  }
  __syncthreads();
  // coarse cells anchored in the core
  const int ci0 = i0 + H, cj0 = j0 + H;  // first core cell
  const int ii0 = max(nh + 1, ((ci0 - nh - 1 + 1) >> 1) + nh + 1), jj0 = max(nh + 1, ((cj0 - nh - 1 + 1) >> 1) + nh + 1);
  const int ii1 = min(a.ctx - nh, ((ci0 + core - 1 - nh - 1) >> 1) + nh + 1);
  const int jj1 = min(a.cty - nh, ((cj0 + core - 1 - nh - 1) >> 1) + nh + 1);
  const int ni = ii1 - ii0 + 1, nj = jj1 - jj0 + 1;
  if (ni <= 0 || nj <= 0) return;
  const Sq rq(ni);
  for (int t = tid; t < ni * nj; t += kGThreads) {
    int i, j;
    rq.at(t, i, j);
    const int ii = ii0 + i, jj = jj0 + j;
    const int L = (c2f(jj, nh) - j0) * S + c2f(ii, nh) - i0;
    double v;
    if (KIND == 0) {
      v = A::add(A::add(A::add(Y[L], Y[L + 1]), Y[L + S]), Y[L + 1 + S]);
    } else {  // 1-2-1 x 1-2-1
      v = A::fmx(Y[L - S], 2.0, Y[L - 1 - S]);
      v = A::add(v, Y[L + 1 - S]);
      v = A::fmx(Y[L - 1], 2.0, v);
      v = A::fmx(Y[L], 4.0, v);
      v = A::fmx(Y[L + 1], 2.0, v);
      v = A::add(v, Y[L - 1 + S]);
      v = A::fmx(Y[L + S], 2.0, v);
      v = A::add(v, Y[L + 1 + S]);
    }
    const long long C = (long long)(ii - 1) + (long long)a.ctx * (jj - 1);
    a.bc[C] = A::mul(a.rc[C], v);
    a.xcz[C] = 0.0;
  }
}

// the core side with the least FP64 work for the busiest of 152 SMs
int tbg_tile(int tx, int ty, int np, bool descent) {
  const int H = 2 * np + (descent ? 2 : 0);
  int best = 4;
  double cost = 0.0;
  for (int core = 4; core + 2 * H <= kGMaxTile; core += 2) {
    const int S = core + 2 * H;
    const long long tiles = (long long)((tx + core - 1) / core) * ((ty + core - 1) / core);
    double w = 200.0 + 0.3 * S * S;  // loads and barriers, in cells of a sweep
    for (int s = 0; s < 2 * np; ++s) w += (S - 2 * (s + 1)) * (S - 2 * (s + 1));
    if (descent) w += 1.2 * (core + 2) * (core + 2);
    else w += S * S;
    w *= (double)((tiles + 151) / 152);
    if (cost == 0.0 || w < cost) {
      cost = w;
      best = core;
    }
  }
  return best;
}

template <int ST, int MODE, int KIND>
void launch_step(const TbgArgs& a, cudaStream_t s) {
  const int core = tbg_tile(a.tx, a.ty, a.np, MODE != 2), S = core + 2 * (2 * a.np + (MODE != 2 ? 2 : 0));
  const size_t smem = (size_t)(ST == TAIL_VC ? 6 : 4) * S * S * sizeof(double);
  static const cudaError_t attr = cudaFuncSetAttribute(
      k_step2d<ST, MODE, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, 6 * kGMaxTile * kGMaxTile * 8);
  (void)attr;
  const dim3 grid((unsigned)((a.tx + core - 1) / core), (unsigned)((a.ty + core - 1) / core));
  launch_dep(k_step2d<ST, MODE, KIND>, grid, kGThreads, smem, s, a, S, core);
}
template <int ST, int MODE>
void launch_step_k(const TbgArgs& a, bool vertices, cudaStream_t s) {
  if (vertices) launch_step<ST, MODE, 2>(a, s);
  else launch_step<ST, MODE, 0>(a, s);
}
template <int ST>
void launch_step_m(const TbgArgs& a, int mode, bool vertices, cudaStream_t s) {
  if (mode == 0) launch_step_k<ST, 0>(a, vertices, s);
  else if (mode == 1) launch_step_k<ST, 1>(a, vertices, s);
  else launch_step_k<ST, 2>(a, vertices, s);
}

}  // namespace

void launch_step2d(const TbgArgs& a, int stencil, int mode, bool vertices, cudaStream_t s) {
  if (stencil == TAIL_9) launch_step_m<TAIL_9>(a, mode, vertices, s);
  else if (stencil == TAIL_VC) launch_step_m<TAIL_VC>(a, mode, vertices, s);
  else launch_step_m<TAIL_5>(a, mode, vertices, s);
}

}  // namespace cfmg
