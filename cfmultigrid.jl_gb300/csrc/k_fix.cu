// The FP64 sweep and residual of the 9-point operator on large levels, their
// sums of neighbours taken on the integer pipes.
//
// The FP64 pipe takes a warp instruction in some 70 clocks per quarter of an
// SM, an integer pipe in 2: an FP64 addition done in some 15 integer
// instructions costs half as much, and the two pipes run side by side. Six of
// a cell's 11 FP64 operations are sums of neighbours; here they are integer
// ones, of which one is shared with the next row, and 5 (4 in the residual's
// case) stay on the FP64 pipe. A 2048^2 sweep takes 51 us where the plain form
// takes 74 to 92 (74 on a hierarchy's own data, where it skips land), at 1024^2
// 20 and 30, at 512^2 10.5 and 12.6; below that neither is ahead. (The 5- and
// 7-point operators have 3 and 5 sums of 7 and 9 operations and gained 3 to
// 8 % in sweeps over a basin and lost 10 to 20 % in residuals.)
//
// Every result is the one the separate FP64 operations give, bit for bit. A
// warp's strip of x is held as 96-bit integers, in units that hold every x
// down to 2^-15 of the strip's largest exactly with 12 zero bits below; sums
// of it do not overflow, and each addition is rounded to 53 bits, ties to
// even, as the FP64 one is. A strip with anything else in it (a smaller x, a
// NaN or an infinity, a sum below 2^-16 of the largest that is not 0) is
// recomputed with the general operators, which also serve smaller levels.
#include "ops_dev.cuh"

namespace cfmg {
namespace {

struct Fx {  // two's complement
  unsigned l, m, h;
};
constexpr int kSpan = 15;  // a value may be this many exponents below the strip's largest
constexpr int kLow = 12;   // zero bits below the last one of the smallest

// x in units of 2^(e0 - 1023 - 52): its 53 bits start between kLow and
// kLow + kSpan = 27. By multiplications, which leave the adders' pipe free.
__device__ __forceinline__ Fx fx_of(double x, int e0) {
  const unsigned lo = (unsigned)__double2loint(x), hi = (unsigned)__double2hiint(x);
  const unsigned s = (2u * hi - ((unsigned)e0 << 21)) >> 21;
  const unsigned mh = ((hi << 1) | lo) == 0u ? 0u : ((hi & 0xfffffu) | 0x100000u);
  const int pw = (int)((unsigned)(((int)hi >> 31) | 1) << (s & 31u));  // +-2^s
  const unsigned long long t = (unsigned long long)lo * (unsigned)pw;
  const unsigned m = (unsigned)(t >> 32) - (pw < 0 ? lo : 0u);
  const long long hm = (long long)(int)mh * pw + (int)m;
  return {(unsigned)t, (unsigned)hm, (unsigned)(hm >> 32)};
}
// a + b rounded to 53 bits, ties to even. q: the sum's first bit is 64 + q and
// its 53rd 12 + q; ~0 when the sum is below 2^64, which needs no rounding (no
// sum has bits below kLow).
__device__ __forceinline__ Fx fx_add(const Fx& a, const Fx& b, unsigned& q) {
  Fx v, r;
  asm("add.cc.u32 %0, %3, %6;\n\taddc.cc.u32 %1, %4, %7;\n\taddc.u32 %2, %5, %8;"
      : "=r"(v.l), "=r"(v.m), "=r"(v.h)
      : "r"(a.l), "r"(a.m), "r"(a.h), "r"(b.l), "r"(b.m), "r"(b.h));
  asm("bfind.s32 %0, %1;" : "=r"(q) : "r"(v.h));
  const unsigned half = __funnelshift_l(0x800u, 0x800u, q), rest = 2u * half - 1u;  // q = ~0: below kLow
  asm("add.cc.u32 %0, %3, %6;\n\taddc.cc.u32 %1, %4, 0;\n\taddc.u32 %2, %5, 0;"
      : "=r"(r.l), "=r"(r.m), "=r"(r.h)
      : "r"(v.l), "r"(v.m), "r"(v.h), "r"(half));
  const bool tie = (r.l & rest) == 0u;
  r.l &= ~rest;
  if (tie) r.l &= ~(2u * half);
  return r;
}
// a sum of fx_add with its q, as a double; bad when it is below 2^64 and not 0
__device__ __forceinline__ double fx_back(const Fx& a, unsigned q, int e0, bool& bad) {
  const unsigned n = (unsigned)((int)a.h >> 31), p = q + 12u;
  const unsigned dl = __funnelshift_r(a.l, a.m, p), dh = __funnelshift_r(a.m, a.h, p);
  // the magnitude; 2^53 where the rounding carried (or for -2^k), which adds 1 to the exponent
  const unsigned long long d = (((unsigned long long)(dh ^ n) << 32) | (dl ^ n)) - (((unsigned long long)n << 32) | n);
  const unsigned hi = (n & 0x80000000u) | ((unsigned)(d >> 32) + ((p + (unsigned)e0 - 1u) << 20));
  const bool z = q == ~0u;
  bad = bad || (z && (a.l | a.m | a.h) != 0u);
  return z ? 0.0 : __hiloint2double((int)hi, (int)(unsigned)d);
}
__device__ __forceinline__ Fx shfl_up(const Fx& a) {
  Fx r;
  r.l = __shfl_up_sync(~0u, a.l, 1);
  r.m = __shfl_up_sync(~0u, a.m, 1);
  r.h = __shfl_up_sync(~0u, a.h, 1);
  return r;
}
__device__ __forceinline__ Fx shfl_down(const Fx& a) {
  Fx r;
  r.l = __shfl_down_sync(~0u, a.l, 1);
  r.m = __shfl_down_sync(~0u, a.m, 1);
  r.h = __shfl_down_sync(~0u, a.h, 1);
  return r;
}
__device__ __forceinline__ bool is_zero(double v) { return ((__double2hiint(v) << 1) | __double2loint(v)) == 0; }
__device__ __forceinline__ bool neg_zero(double v) { return __double_as_longlong(v) == (long long)(1ull << 63); }
// What a strip's values are like: each one's magnitude as its upper word, with
// bit 0 for the lower one, so that 0 is 0
struct Span {
  unsigned top = 0, low = ~0u, neg = 0;  // largest; smallest that is not 0, less 1; whether there is a -0
  __device__ __forceinline__ unsigned see(double v) {
    const unsigned hi = (unsigned)__double2hiint(v);
    const unsigned key = (hi & 0x7fffffffu) | min((unsigned)__double2loint(v), 1u);
    top = max(top, key);
    low = min(low, key - 1u);
    if (key == 0u) neg |= hi;
    return key;
  }
  // over the warp; false when its values can't be held
  __device__ __forceinline__ bool close(int& e0) {
    top = __reduce_max_sync(~0u, top);
    low = __reduce_min_sync(~0u, low);
    neg = __any_sync(~0u, neg != 0u);
    e0 = (int)(top >> 20) - (kSpan + kLow);
    return top == 0u || (e0 >= 64 && e0 <= 2000 && (int)((low + 1u) >> 20) >= e0 + kLow);
  }
};

// The cells to write: columns c0..c1-1 of rows r0..r1-1 of an array n1 wide
// and len cells long
struct FixRange {
  long long n1, len;
  int c0, c1, r0, r1;
};
struct FixArgs {
  const double *x, *b, *w;  // w: omega*idiag of a sweep, diag of a residual
  double* y;
  const uint8_t* m;
  double cff;
};

// what is left for the FP64 pipe (v_sweep9, v_resid9 with the sums given)
template <bool RES>
__device__ __forceinline__ double fix_end(const FixArgs& a, double x, double b, double w, double s, double d,
                                          long long I) {
  typedef Ar<double> A;
  double t = RES ? A::add(A::mul(w, x), b) : b;
  t = A::fmx(s, -0.5, t);
  t = A::fmx(d, -0.25, t);
  return RES ? mask_mul(a.m[I], t) : A::sub(A::mul(a.cff, x), A::mul(w, t));
}
// A cell whose x and neighbours are zeros (fneg, dneg: the faces, the
// diagonals all are -0): true where b and the coefficient make the result a
// zero, whose sign follows from theirs, without an operation. b - faces/2 -
// diagonals/4 is -0 only from -0 less sums that are +0.
template <bool RES>
__device__ __forceinline__ bool fix_zero(const FixArgs& a, double x, double b, double w, bool fneg, bool dneg,
                                         double& out) {
  const bool t = is_neg(b) && !fneg && !dneg;
  out = signed_zero(RES ? (is_neg(w) != is_neg(x)) && t : is_neg(x) && !t);
  return is_zero(b) && (RES ? is_fin(w) : __double_as_longlong(w) == 0ll && a.cff >= 0.0 && !is_neg(a.cff));
}

// A warp takes 30 columns (and the one on either side) by kRows rows. Each x
// is converted once by its lane, and its neighbours have it by shuffles; the
// sum of a row's two neighbours of a column serves the row's faces and the
// next row's diagonals. Rows of zeros (land) skip all of it. Of 4 to 12 rows a
// warp, 4 was fastest: longer strips convert less twice, but their code and
// their last wave are longer (2048^2: 54.9 us at 4, 58.9 at 6, 61.1 at 8; a
// form that walks 16 rows in a loop 61).
constexpr int kRows = 4, kT = 128;
template <bool RES>
__global__ void __launch_bounds__(kT) k_fix9(const __grid_constant__ FixArgs a,
                                             const __grid_constant__ FixRange g) {
  dep_wait();
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int c = g.c0 + 30 * (int)blockIdx.x - 1 + lane;
  const int r = g.r0 + (kT / 32 * (int)blockIdx.y + wp) * kRows;
  if (r >= g.r1) return;
  const long long I0 = (long long)r * g.n1 + c;
  double x[kRows + 2];
  Span sp;
  unsigned some = 0;  // bit q: row q has a value that is not 0
#pragma unroll
  for (int q = 0; q < kRows + 2; ++q) {
    const long long I = I0 + (q - 1) * g.n1;
    x[q] = r - 1 + q <= g.r1 && I >= 0 && I < g.len ? a.x[I] : 0.0;
  }
#pragma unroll
  for (int q = 0; q < kRows + 2; ++q) some |= sp.see(x[q]) ? 1u << q : 0u;
  some = __reduce_or_sync(~0u, some);
  int e0;
  bool bad = !sp.close(e0);
  const bool cok = lane >= 1 && lane <= 30 && c < g.c1;
  const Fx zero = {0u, 0u, 0u};
  unsigned u;  // a sum's q that is not needed
  Fx hm = zero, h = zero, cm = zero, cc = zero;
  if (some & 1u) {
    cm = fx_of(x[0], e0);
    hm = fx_add(shfl_up(cm), shfl_down(cm), u);
  }
  if (some & 2u) {
    cc = fx_of(x[1], e0);
    h = fx_add(shfl_up(cc), shfl_down(cc), u);
  }
  auto inside = [&](int q) { return cok && r + q < g.r1; };
  double bn = inside(0) ? a.b[I0] : 0.0, wn = inside(0) ? a.w[I0] : 0.0;  // a row ahead
#pragma unroll
  for (int q = 0; q < kRows; ++q) {
    const long long I = I0 + q * g.n1;
    const bool ok = inside(q);
    const double bv = bn, wv = wn;
    if (q + 1 < kRows) {
      bn = inside(q + 1) ? a.b[I + g.n1] : 0.0;
      wn = inside(q + 1) ? a.w[I + g.n1] : 0.0;
    }
    Fx cp = zero, hp = zero, xl = zero, xr = zero;
    if (some >> (q + 2) & 1u) {
      cp = fx_of(x[q + 2], e0);
      xl = shfl_up(cp);
      xr = shfl_down(cp);
      hp = fx_add(xl, xr, u);
    }
    bool fneg = false, dneg = false;  // the sum of zeros that are all -0 is -0
    if (sp.neg) {
      const unsigned z0 = __ballot_sync(~0u, neg_zero(x[q])), z1 = __ballot_sync(~0u, neg_zero(x[q + 1])),
                     z2 = __ballot_sync(~0u, neg_zero(x[q + 2]));
      fneg = ((z1 << 1) & (z1 >> 1) & z0 & z2) >> lane & 1u;
      dneg = ((z0 << 1) & (z0 >> 1) & (z2 << 1) & (z2 >> 1)) >> lane & 1u;
    }
    double s = 0.0, d = 0.0;
    bool dry = false;
    if (some >> q & 7u) {
      unsigned qs;
      const Fx f = fx_add(fx_add(h, cm, u), cp, qs);
      s = fx_back(f, qs, e0, bad);
      const Fx e = fx_add(fx_add(hm, xl, u), xr, qs);
      d = fx_back(e, qs, e0, bad);
    } else {
      double z;
      dry = __all_sync(~0u, (fix_zero<RES>(a, x[q + 1], bv, wv, fneg, dneg, z)));
      if (dry && ok) a.y[I] = z;
    }
    if (!dry) {
      if (fneg) s = -0.0;
      if (dneg) d = -0.0;
      if (ok) a.y[I] = fix_end<RES>(a, x[q + 1], bv, wv, s, d, I);
    }
    hm = h;
    h = hp;
    cm = cc;
    cc = cp;
  }
  if (__any_sync(~0u, bad)) {
#pragma unroll 1
    for (int q = 0; q < kRows; ++q)
      if (inside(q)) {
        if (RES) d_resid9(a.y, a.x, a.b, a.w, a.m, g.n1, I0 + q * g.n1);
        else d_sweep9(a.x, a.y, a.b, a.w, a.cff, g.n1, I0 + q * g.n1);
      }
  }
}

template <bool RES>
void launch_fix9(const FixArgs& a, const Geom& g, const Box& bx, cudaStream_t s) {
  const FixRange r = {g.n1, g.len, bx.i0 - 1, bx.i1, bx.j0 - 1, bx.j1};
  const dim3 grid((unsigned)((r.c1 - r.c0 + 29) / 30),
                  (unsigned)((r.r1 - r.r0 + kT / 32 * kRows - 1) / (kT / 32 * kRows)));
  launch_dep(k_fix9<RES>, grid, dim3(kT), 0, s, a, r);
}

}  // namespace

void launch_fix_sweep9(const double* x, double* y, const double* b, const double* w, double cff, const Geom& g,
                       const Box& bx, cudaStream_t s) {
  launch_fix9<false>({x, b, w, y, nullptr, cff}, g, bx, s);
}
void launch_fix_resid9(double* r, const double* x, const double* b, const double* d, const uint8_t* m, const Geom& g,
                       const Box& bx, cudaStream_t s) {
  launch_fix9<true>({x, b, d, r, m, 0.0}, g, bx, s);
}

}  // namespace cfmg
