// Descent and ascent steps of 2D levels in one launch each (closed topology,
// one layer): FP64 levels of the 5-point, 9-point and variable-coefficient
// operators, and FP32 levels of the variable-coefficient operator.
//
// A mid-size FP64 level (600 to 114 285 cells of the 5-point operator, 72 727 of
// the others; about half of that on level 1) takes 12 launches a cycle
// (4 sweeps, residual, restriction, zeroing, prolongation, 4 sweeps) whose
// own work is below a microsecond each: launch and load latency, 2.1 us a
// graph node, is what they cost. Here a block loads a tile with a halo wide
// enough for the whole step into shared memory and runs it there:
//   descent: x = +0, or x = Pcoef P(coarse x) after an F-cycle's prolongation;
//            np pairs of sweeps; residual; restriction into the coarse b; from
//            x = +0 also the coarse x zeroed
//   ascent:  x = x + Pcoef P(coarse x), np pairs of sweeps
//   smoothing: np pairs of sweeps from x into the scratch, or back (a long
//            smoothing of the last level, pass after pass)
// Each sweep covers the tile's cells that later ones need: sweep s leaves a
// margin of s + 1 cells. The tiles overlap, so a step must not read what it
// writes: a descent reads no x at all, and leaves a copy of its result in the
// level's scratch array, which is what the ascent reads. Level 1 starts from
// the caller's x; its descent writes the scratch only, and the ascent x and y.
// A descent from Pcoef P(coarse x) reads coarse cells in its neighbours' cores,
// so it leaves the coarse x as it is: the caller zeroes it in a launch of its
// own where the next level reads it before writing it.
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

// FP64: 8 warps keep the pipe busy; FP32: two blocks of 16 an SM
template <class T>
constexpr int g_threads() { return sizeof(T) == 8 ? 256 : 512; }
// largest tile side, for its 6 arrays
template <class T>
constexpr int g_max_tile() { return sizeof(T) == 8 ? 40 : 64; }

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

__device__ __forceinline__ bool plus_zero(double v) { return __double_as_longlong(v) == 0ll; }
__device__ __forceinline__ bool plus_zero(float v) { return __float_as_uint(v) == 0u; }

template <class T, int ST>
__device__ __forceinline__ T g_cell(const T* x, int L, int S, T b, T w, T cff, const T* cE, const T* cN) {
  typedef Ar<T> A;
  T t;
  if (ST == TAIL_9) {
    t = A::fmx(sum4(x, L, S), T(-0.5), b);
    t = A::fmx(diags4(x, L, S), T(-0.25), t);
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

// MODE 0: descent from x = +0; 1: descent from x = Pcoef P(xc); 2: ascent; 3:
// np pairs of sweeps from xs into x or s, the other null.
// KIND 0: cell centres, 2: vertices (restriction and prolongation).
template <class T, int ST, int MODE, int KIND>
__global__ void __launch_bounds__(g_threads<T>()) k_step2d(TbgArgs<T> a, int S, int core) {
  dep_wait();
  typedef Ar<T> A;
  constexpr int NT = g_threads<T>();
  extern __shared__ __align__(16) unsigned char gsm_raw[];
  T* gsm = reinterpret_cast<T*>(gsm_raw);
  const int n2 = S * S, np = a.np, H = (S - core) / 2, tid = threadIdx.x;
  T* X = gsm;
  T* Y = X + n2;
  T* B = Y + n2;
  T* W = B + n2;
  T* E = W + n2;
  T* N = E + n2;
  const int i0 = 1 + (int)blockIdx.x * core - H, j0 = 1 + (int)blockIdx.y * core - H;  // 1-based tile origin
  const int tx = a.tx, ty = a.ty, nh = a.nh;
  const Sq all(S);
  for (int t = tid; t < n2; t += NT) {
    int i, j;
    all.at(t, i, j);
    const int gi = i0 + i, gj = j0 + j;
    const bool in = gi >= 1 && gi <= tx && gj >= 1 && gj <= ty;
    const long long I = in ? (long long)(gi - 1) + (long long)tx * (gj - 1) : 0;
    T xv = T(0);
    if ((MODE == 2 || a.xs) && in) xv = a.xs[I];
    B[t] = in ? a.b[I] : T(0);
    W[t] = in ? a.w[I] : T(0);
    if (ST == TAIL_VC) {
      E[t] = in ? a.cE[I] : T(0);
      N[t] = in ? a.cN[I] : T(0);
    }
    if (MODE == 1 || MODE == 2) {
      // parents (p, q) update their children; the others keep x
      const int p = gi - nh - 1, q = gj - nh - 1;
      const bool fam = p >= 0 && p < 2 * a.np_i && q >= 0 && q < 2 * a.np_j;
      const T pc = fam ? a.pc[I] : T(0);
      const bool live = !plus_zero(pc);
      if (__any_sync(__activemask(), live) && live) {
        const long long C = (long long)((p >> 1) + nh) + (long long)a.ctx * ((q >> 1) + nh);
        const T v = prolong_child<T, KIND>(a.xc, C, a.ctx, 0, (p & 1) | ((q & 1) << 1));
        xv = A::add(xv, A::mul(pc, v));
      }
    }
    X[t] = xv;
    Y[t] = T(0);
  }
  __syncthreads();
  for (int s = 0; s < 2 * np; ++s) {
    const T* src = (s & 1) ? Y : X;
    T* dst = (s & 1) ? X : Y;
    const int n = S - 2 * (s + 1);
    const Sq sq(n);
    for (int t = tid; t < n * n; t += NT) {
      int i, j;
      sq.at(t, i, j);
      const int L = (j + s + 1) * S + i + s + 1;
      const T b = B[L], w = W[L];
      if (ST == TAIL_9 && (s & 1)) {  // the interior only
        const int gi = i0 + i + s + 1, gj = j0 + j + s + 1;
        if (gi <= nh || gi > tx - nh || gj <= nh || gj > ty - nh) continue;
      }
      T v = T(0);
      bool land = false;
      if constexpr (sizeof(T) == 8) land = __all_sync(__activemask(), g_land<ST>(src, L, S, b, w));
      if (!land) v = g_cell<T, ST>(src, L, S, b, w, a.cff, E, N);
      dst[L] = v;
    }
    __syncthreads();
  }
  // the core of x (and of y, the last odd sweep's result), over the ranges of
  // the reference's sweeps: rows 2 .. ty-1, or ext and interior boxes
  const Sq cs(core);
  for (int t = tid; t < core * core; t += NT) {
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
    if (MODE != 2 && a.s && (r2 || a.xs)) a.s[I] = X[L];  // level 1's x out of range counts too
  }
  if (MODE >= 2) return;
  __syncthreads();
  // residual of the smoothed x into Y, one cell beyond the core
  const int m = H - 1, nr = core + 2;
  const Sq rs(nr);
  for (int t = tid; t < nr * nr; t += NT) {
    int i, j;
    rs.at(t, i, j);
    const int L = (j + m) * S + i + m, gi = i0 + m + i, gj = j0 + m + j;
    const bool in = gi >= 1 && gi <= tx && gj >= 2 && gj <= ty - 1 &&
                    (ST != TAIL_9 || (gi > nh && gi <= tx - nh && gj > nh && gj <= ty - nh));
    T v = T(0);
    if (in) {
      const long long I = (long long)(gi - 1) + (long long)tx * (gj - 1);
      const T d = a.d[I];
      v = A::add(A::mul(d, X[L]), B[L]);
      if (ST == TAIL_9) {
        v = A::fmx(sum4(X, L, S), T(-0.5), v);
        v = A::fmx(diags4(X, L, S), T(-0.25), v);
      } else if (ST == TAIL_VC) {
        v = A::sub(v, vc_sum(X, E, N, L, S));
      } else {
        v = A::sub(v, sum4(X, L, S));
      }
      v = mask_mul(a.m[I], v);
      if (a.r && i > 0 && i <= core && j > 0 && j <= core) a.r[I] = v;
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
  for (int t = tid; t < ni * nj; t += NT) {
    int i, j;
    rq.at(t, i, j);
    const int ii = ii0 + i, jj = jj0 + j;
    const int L = (c2f(jj, nh) - j0) * S + c2f(ii, nh) - i0;
    T v;
    if (KIND == 0) {
      v = A::add(A::add(A::add(Y[L], Y[L + 1]), Y[L + S]), Y[L + 1 + S]);
    } else {  // 1-2-1 x 1-2-1
      v = A::fmx(Y[L - S], T(2), Y[L - 1 - S]);
      v = A::add(v, Y[L + 1 - S]);
      v = A::fmx(Y[L - 1], T(2), v);
      v = A::fmx(Y[L], T(4), v);
      v = A::fmx(Y[L + 1], T(2), v);
      v = A::add(v, Y[L - 1 + S]);
      v = A::fmx(Y[L + S], T(2), v);
      v = A::add(v, Y[L + 1 + S]);
    }
    const long long C = (long long)(ii - 1) + (long long)a.ctx * (jj - 1);
    a.bc[C] = A::mul(a.rc[C], v);
    if (MODE == 0) a.xcz[C] = T(0);  // MODE 1: other tiles may still read it
  }
}

// the core side with the least work (FP64 instructions, or cells) for the busiest SM
int tbg_tile(int max_tile, int tx, int ty, int np, int mode) {
  const bool descent = mode < 2;
  const int H = 2 * np + (descent ? 2 : 0);
  const int nsm = sm_count();
  int best = 4;
  double cost = 0.0;
  for (int core = 4; core + 2 * H <= max_tile; core += 2) {
    const int S = core + 2 * H;
    const long long tiles = (long long)((tx + core - 1) / core) * ((ty + core - 1) / core);
    double w = 200.0 + 0.3 * S * S;  // loads and barriers, in cells of a sweep
    for (int s = 0; s < 2 * np; ++s) w += (S - 2 * (s + 1)) * (S - 2 * (s + 1));
    if (descent) w += 1.2 * (core + 2) * (core + 2);
    else if (mode == 2) w += S * S;
    w *= (double)((tiles + nsm - 1) / nsm);
    if (cost == 0.0 || w < cost) {
      cost = w;
      best = core;
    }
  }
  return best;
}

template <class T, int ST, int MODE, int KIND>
void launch_step(const TbgArgs<T>& a, cudaStream_t s) {
  constexpr int mt = g_max_tile<T>();
  const int core = tbg_tile(mt, a.tx, a.ty, a.np, MODE), S = core + 2 * (2 * a.np + (MODE < 2 ? 2 : 0));
  const size_t smem = (size_t)(ST == TAIL_VC ? 6 : 4) * S * S * sizeof(T);
  static const cudaError_t attr = cudaFuncSetAttribute(
      k_step2d<T, ST, MODE, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, 6 * mt * mt * (int)sizeof(T));
  (void)attr;
  const dim3 grid((unsigned)((a.tx + core - 1) / core), (unsigned)((a.ty + core - 1) / core));
  launch_dep(k_step2d<T, ST, MODE, KIND>, grid, g_threads<T>(), smem, s, a, S, core);
}
template <class T, int ST, int KIND>
void launch_step_m(const TbgArgs<T>& a, int mode, cudaStream_t s) {
  if (mode == 0) launch_step<T, ST, 0, KIND>(a, s);
  else if (mode == 1) launch_step<T, ST, 1, KIND>(a, s);
  else if (mode == 2) launch_step<T, ST, 2, KIND>(a, s);
  else if constexpr (sizeof(T) == 8) launch_step<T, ST, 3, KIND>(a, s);
}

}  // namespace

void launch_step2d(const TbgArgs<double>& a, int stencil, int mode, bool vertices, cudaStream_t s) {
  if (stencil == TAIL_VC) launch_step_m<double, TAIL_VC, 0>(a, mode, s);
  else if (stencil == TAIL_9) vertices ? launch_step_m<double, TAIL_9, 2>(a, mode, s)
                                       : launch_step_m<double, TAIL_9, 0>(a, mode, s);
  else vertices ? launch_step_m<double, TAIL_5, 2>(a, mode, s) : launch_step_m<double, TAIL_5, 0>(a, mode, s);
}
// FP32, variable coefficient, levels that fill the GPU: the same steps with
// the coefficients in registers. A block of 64 x 8 threads holds a 64 x 48
// tile; a thread owns 6 rows of a column with their b, omega*idiag and face
// coefficients (31 registers) and slides a window down them, so a cell update
// is 11 operations on 3 shared loads and a store, where k_step2d's index
// arithmetic and 11 shared loads make it 45 instructions. Every sweep covers
// the whole tile (cells near its edge hold values that nothing in the core
// reads); x is in shared memory twice, inside a border of zeros. Two blocks an
// SM, so one tile's loads overlap the other's sweeps. 2048^2, 2 pairs: descent
// 52 us, ascent 56 (k_step2d 96 and 73, the separate kernels 105 and 86).
// Levels below kVCells give it too few tiles.
constexpr long long kVCells = 150000;
constexpr int kVW = 64, kVG = 8, kVR = 6, kVH = kVG * kVR, kVS = kVW + 2;

template <int MODE>
__global__ void __launch_bounds__(kVW * kVG, 2) k_step2d_vc(TbgArgs<float> a) {
  dep_wait();
  typedef Ar<float> A;
  extern __shared__ __align__(16) unsigned char gsm_raw[];
  constexpr bool EPI = MODE != 2;
  float* P0 = reinterpret_cast<float*>(gsm_raw);
  float* P1 = P0 + (kVH + 2) * kVS;
  float* Ds = P1 + (kVH + 2) * kVS;
  uint8_t* Ms = reinterpret_cast<uint8_t*>(Ds + kVH * kVW);
  const int np = a.np, H = 2 * np + (EPI ? 2 : 0), cw = kVW - 2 * H, ch = kVH - 2 * H;
  const int lx = threadIdx.x, r0 = threadIdx.y * kVR, tid = threadIdx.y * kVW + lx;
  const int i0 = 1 + (int)blockIdx.x * cw - H, j0 = 1 + (int)blockIdx.y * ch - H;  // 1-based tile origin
  const int tx = a.tx, ty = a.ty, nh = a.nh;
  const int gi = i0 + lx;
  const bool col_in = gi >= 1 && gi <= tx;
  float B[kVR], W[kVR], cw_[kVR], ce[kVR], cn[kVR + 1];
#pragma unroll
  for (int r = 0; r < kVR; ++r) {
    const int gj = j0 + r0 + r;
    const bool in = col_in && gj >= 1 && gj <= ty;
    const long long I = in ? (long long)(gi - 1) + (long long)tx * (gj - 1) : 0;
    B[r] = in ? a.b[I] : 0.f;
    W[r] = in ? a.w[I] : 0.f;
    ce[r] = in ? a.cE[I] : 0.f;
    cw_[r] = in && I > 0 ? a.cE[I - 1] : 0.f;
    cn[r + 1] = in ? a.cN[I] : 0.f;
    if (r == 0) cn[0] = in && gj > 1 ? a.cN[I - tx] : 0.f;
    float xv = 0.f;
    if (MODE == 2) xv = in ? a.xs[I] : 0.f;
    if (MODE != 0) {
      const int p = gi - nh - 1, q = gj - nh - 1;
      const bool fam = p >= 0 && p < 2 * a.np_i && q >= 0 && q < 2 * a.np_j;
      const float pc = fam ? a.pc[I] : 0.f;
      if (pc != 0.f) {
        const long long C = (long long)((p >> 1) + nh) + (long long)a.ctx * ((q >> 1) + nh);
        xv = A::add(xv, A::mul(pc, prolong_child<float, 0>(a.xc, C, a.ctx, 0, (p & 1) | ((q & 1) << 1))));
      }
    }
    P0[(r0 + r + 1) * kVS + lx + 1] = xv;
    if (EPI) {
      Ds[(r0 + r) * kVW + lx] = in ? a.d[I] : 0.f;
      Ms[(r0 + r) * kVW + lx] = in ? a.m[I] : 0;
    }
  }
  for (int c = tid; c < kVS; c += kVW * kVG) {
    P0[c] = P1[c] = 0.f;
    P0[(kVH + 1) * kVS + c] = P1[(kVH + 1) * kVS + c] = 0.f;
  }
  for (int r = tid; r < kVH + 2; r += kVW * kVG) P0[r * kVS] = P1[r * kVS] = P0[r * kVS + kVS - 1] = P1[r * kVS + kVS - 1] = 0.f;
  __syncthreads();
  const float cff = a.cff;
  const int base = r0 * kVS + lx + 1;  // row above the thread's first, its column
  // the stencil sum of the thread's row r: centre rows xm, x0, xp, row pointer s
  auto sum = [&](const float* s, int r, float xm, float xp) {
    const float t = A::add(A::mul(cw_[r], s[-1]), A::mul(ce[r], s[1]));
    return A::add(A::add(t, A::mul(cn[r], xm)), A::mul(cn[r + 1], xp));
  };
#pragma unroll 1
  for (int k = 0; k < 2 * np; ++k) {
    const float* src = ((k & 1) ? P1 : P0) + base;
    float* dst = ((k & 1) ? P0 : P1) + base;
    float xm = src[0], x0 = src[kVS];
#pragma unroll
    for (int r = 0; r < kVR; ++r) {
      const float xp = src[(r + 2) * kVS];
      const float t = A::sub(B[r], sum(src + (r + 1) * kVS, r, xm, xp));
      dst[(r + 1) * kVS] = A::sub(A::mul(cff, x0), A::mul(W[r], t));
      xm = x0;
      x0 = xp;
    }
    __syncthreads();
  }
  // the core of x, rows 2 .. ty-1
  if (lx >= H && lx < kVW - H && col_in) {
#pragma unroll
    for (int r = 0; r < kVR; ++r) {
      const int lj = r0 + r, gj = j0 + lj;
      if (lj < H || lj >= kVH - H || gj < 2 || gj > ty - 1) continue;
      const long long I = (long long)(gi - 1) + (long long)tx * (gj - 1);
      const float v = P0[base + (r + 1) * kVS];
      a.x[I] = v;
      if (EPI) a.s[I] = v;
    }
  }
  if (!EPI) return;
  {
    const float* src = P0 + base;
    float xm = src[0], x0 = src[kVS];
#pragma unroll
    for (int r = 0; r < kVR; ++r) {
      const float xp = src[(r + 2) * kVS];
      const int gj = j0 + r0 + r;
      const float v = A::sub(A::add(A::mul(Ds[(r0 + r) * kVW + lx], x0), B[r]), sum(src + (r + 1) * kVS, r, xm, xp));
      P1[base + (r + 1) * kVS] = col_in && gj >= 2 && gj <= ty - 1 ? mask_mul(Ms[(r0 + r) * kVW + lx], v) : 0.f;
      xm = x0;
      x0 = xp;
    }
  }
  __syncthreads();
  // coarse cells anchored in the core: at most cw/2 x ch/2 of them
  const int ci0 = i0 + H, cj0 = j0 + H;
  const int ii0 = max(nh + 1, ((ci0 - nh) >> 1) + nh + 1), jj0 = max(nh + 1, ((cj0 - nh) >> 1) + nh + 1);
  const int ii1 = min(a.ctx - nh, ((ci0 + cw - 2 - nh) >> 1) + nh + 1);
  const int jj1 = min(a.cty - nh, ((cj0 + ch - 2 - nh) >> 1) + nh + 1);
  const int ni = ii1 - ii0 + 1, nj = jj1 - jj0 + 1;
  if (ni <= 0 || nj <= 0) return;
  const Sq rq(ni);
  for (int t = tid; t < ni * nj; t += kVW * kVG) {
    int i, j;
    rq.at(t, i, j);
    const int ii = ii0 + i, jj = jj0 + j;
    const float* y = P1 + (c2f(jj, nh) - j0 + 1) * kVS + c2f(ii, nh) - i0 + 1;
    const float v = A::add(A::add(A::add(y[0], y[1]), y[kVS]), y[kVS + 1]);
    const long long C = (long long)(ii - 1) + (long long)a.ctx * (jj - 1);
    a.bc[C] = A::mul(a.rc[C], v);
    if (MODE == 0) a.xcz[C] = 0.f;
  }
}

template <int MODE>
static void launch_vc(const TbgArgs<float>& a, cudaStream_t s) {
  const int H = 2 * a.np + (MODE != 2 ? 2 : 0), cw = kVW - 2 * H, ch = kVH - 2 * H;
  const size_t smem = 2 * (kVH + 2) * kVS * sizeof(float) + kVH * kVW * (sizeof(float) + 1);
  static const cudaError_t attr =
      cudaFuncSetAttribute(k_step2d_vc<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  (void)attr;
  const dim3 grid((unsigned)((a.tx + cw - 1) / cw), (unsigned)((a.ty + ch - 1) / ch));
  launch_dep(k_step2d_vc<MODE>, grid, dim3(kVW, kVG), smem, s, a);
}

// FP32: the variable-coefficient operator (the others have k_tb.cu's packed passes)
void launch_step2d(const TbgArgs<float>& a, int, int mode, bool, cudaStream_t s) {
  if ((long long)a.tx * a.ty >= kVCells) {
    if (mode == 0) launch_vc<0>(a, s);
    else if (mode == 1) launch_vc<1>(a, s);
    else launch_vc<2>(a, s);
    return;
  }
  launch_step_m<float, TAIL_VC, 0>(a, mode, s);
}

}  // namespace cfmg
