// Per-cell arithmetic of the multigrid operators, shared by the standalone
// kernels (k_ops.cu) and the coarse-level program engine (k_coarse.cu), so
// that both paths round identically.
//
// Every sum and product goes through the _rn intrinsics so that nvcc
// cannot contract a multiply and an add into one FMA: the FP64
// instantiation rounds exactly where the Julia reference rounds. The only
// FMAs used are ones whose product is exact (a multiplication by 1/2, 1/4,
// 2, 4 or 8), which round once on the same exact value as the reference's
// two-step form.
#pragma once

#include "cfmg_internal.h"

namespace cfmg {

template <class T>
struct Ar;
template <>
struct Ar<double> {
  static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
  static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
  static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
  // a*w + c with w a power of two (exact product): one rounding, same value
  static __device__ __forceinline__ double fmx(double a, double w, double c) { return __fma_rn(a, w, c); }
};
template <>
struct Ar<float> {
  static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
  static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ float fmx(float a, float w, float c) { return __fmaf_rn(a, w, c); }
};

// msk*v for a UInt8 mask, as the reference's promote-and-multiply: 1 -> v,
// 0 -> a zero carrying v's sign, other values -> (double)m*v.
template <class T>
__device__ __forceinline__ T mask_mul(uint8_t m, T v) {
  if (m == 1) return v;
  if (m == 0) return copysign(T(0), v);
  return Ar<T>::mul(T(m), v);
}

__device__ __forceinline__ long long lin(const Geom& g, int i, int j, int k) {
  return (long long)(i - 1) + g.n1 * ((long long)(j - 1) + (long long)g.ty * (k - 1));
}

__device__ __forceinline__ int c2f(int i, int nh) { return (i - nh - 1) * 2 + nh + 1; }  // src/gmg_types.jl:25
__device__ __forceinline__ int f2c(int i, int nh) { return (i - nh - 1) / 2 + nh + 1; }  // src/gmg_types.jl:26

// ------------------------------------------------------------- stencils
template <class T>
__device__ __forceinline__ T sum4(const T* x, long long I, long long n1) {
  typedef Ar<T> A;
  return A::add(A::add(A::add(x[I - 1], x[I + 1]), x[I - n1]), x[I + n1]);
}
template <class T>
__device__ __forceinline__ T diags4(const T* x, long long I, long long n1) {
  typedef Ar<T> A;
  return A::add(A::add(A::add(x[I - 1 - n1], x[I + 1 - n1]), x[I - 1 + n1]), x[I + 1 + n1]);
}
template <class T>
__device__ __forceinline__ T faces6(const T* x, long long I, long long n1, long long n2) {
  typedef Ar<T> A;
  return A::add(A::add(A::add(A::add(A::add(x[I - 1], x[I + 1]), x[I - n1]), x[I + n1]), x[I - n2]), x[I + n2]);
}
template <class T>
__device__ __forceinline__ T edges12(const T* x, long long I, long long n1, long long n2) {
  typedef Ar<T> A;
  T e = A::add(x[I - 1 - n1], x[I + 1 - n1]);
  e = A::add(e, x[I - 1 + n1]);
  e = A::add(e, x[I + 1 + n1]);
  e = A::add(e, x[I - 1 - n2]);
  e = A::add(e, x[I + 1 - n2]);
  e = A::add(e, x[I - 1 + n2]);
  e = A::add(e, x[I + 1 + n2]);
  e = A::add(e, x[I - n1 - n2]);
  e = A::add(e, x[I + n1 - n2]);
  e = A::add(e, x[I - n1 + n2]);
  e = A::add(e, x[I + n1 + n2]);
  return e;
}
template <class T>
__device__ __forceinline__ T vc_sum(const T* x, const T* cE, const T* cN, long long I, long long n1) {
  typedef Ar<T> A;
  T s = A::add(A::mul(cE[I - 1], x[I - 1]), A::mul(cE[I], x[I + 1]));
  s = A::add(s, A::mul(cN[I - n1], x[I - n1]));
  return A::add(s, A::mul(cN[I], x[I + n1]));
}

// ---------------------------------------------------------- sweeps at I
// v_* return the new value at I, d_* store it.
// sloop2d! (src/laplacian.jl:66-73): y = (1-w)x - (w*idiag)*(b - s4)
template <class T>
__device__ __forceinline__ T v_sweep5(const T* x, const T* b, const T* w, T cff, long long n1, long long I) {
  typedef Ar<T> A;
  return A::sub(A::mul(cff, x[I]), A::mul(w[I], A::sub(b[I], sum4(x, I, n1))));
}
// sloop3d_v1! (src/laplacian.jl:11-20)
template <class T>
__device__ __forceinline__ T v_sweep7(const T* x, const T* b, const T* w, T cff, long long n1, long long n2,
                                      long long I) {
  typedef Ar<T> A;
  return A::sub(A::mul(cff, x[I]), A::mul(w[I], A::sub(b[I], faces6(x, I, n1, n2))));
}
// in-plane laplacian9 (2D 9-point extension): b - faces/2 - diagonals/4
template <class T>
__device__ __forceinline__ T v_sweep9(const T* x, const T* b, const T* w, T cff, long long n1, long long I) {
  typedef Ar<T> A;
  T t = A::fmx(sum4(x, I, n1), T(-0.5), b[I]);
  t = A::fmx(diags4(x, I, n1), T(-0.25), t);
  return A::sub(A::mul(cff, x[I]), A::mul(w[I], t));
}
// smooth_laplacian9! body (src/laplacian9.jl:14-44)
template <class T>
__device__ __forceinline__ T v_sweep19(const T* x, const T* b, const T* w, T cff, long long n1, long long n2,
                                       long long I) {
  typedef Ar<T> A;
  T t = A::fmx(faces6(x, I, n1, n2), T(-0.5), b[I]);
  t = A::fmx(edges12(x, I, n1, n2), T(-0.25), t);
  return A::sub(A::mul(cff, x[I]), A::mul(w[I], t));
}
template <class T>
__device__ __forceinline__ T v_sweepvc(const T* x, const T* b, const T* w, const T* cE, const T* cN, T cff,
                                       long long n1, long long I) {
  typedef Ar<T> A;
  return A::sub(A::mul(cff, x[I]), A::mul(w[I], A::sub(b[I], vc_sum(x, cE, cN, I, n1))));
}
template <class T>
__device__ __forceinline__ void d_sweep5(const T* x, T* y, const T* b, const T* w, T cff, long long n1, long long I) {
  y[I] = v_sweep5(x, b, w, cff, n1, I);
}
template <class T>
__device__ __forceinline__ void d_sweep7(const T* x, T* y, const T* b, const T* w, T cff, long long n1, long long n2,
                                         long long I) {
  y[I] = v_sweep7(x, b, w, cff, n1, n2, I);
}
template <class T>
__device__ __forceinline__ void d_sweep9(const T* x, T* y, const T* b, const T* w, T cff, long long n1, long long I) {
  y[I] = v_sweep9(x, b, w, cff, n1, I);
}
template <class T>
__device__ __forceinline__ void d_sweep19(const T* x, T* y, const T* b, const T* w, T cff, long long n1, long long n2,
                                          long long I) {
  y[I] = v_sweep19(x, b, w, cff, n1, n2, I);
}
template <class T>
__device__ __forceinline__ void d_sweepvc(const T* x, T* y, const T* b, const T* w, const T* cE, const T* cN, T cff,
                                          long long n1, long long I) {
  y[I] = v_sweepvc(x, b, w, cE, cN, cff, n1, I);
}

// ------------------------------------------------------- residuals at I
// v_* return the residual value, d_* store it.
// rloop2d! (src/laplacian.jl:87-93): r = msk*((diag*x + b) - s4)
template <class T>
__device__ __forceinline__ T v_resid5(const T* x, const T* b, const T* d, const uint8_t* m, long long n1, long long I) {
  typedef Ar<T> A;
  return mask_mul(m[I], A::sub(A::add(A::mul(d[I], x[I]), b[I]), sum4(x, I, n1)));
}
// rloop3d! (src/laplacian.jl:43-51)
template <class T>
__device__ __forceinline__ T v_resid7(const T* x, const T* b, const T* d, const uint8_t* m, long long n1, long long n2,
                                      long long I) {
  typedef Ar<T> A;
  return mask_mul(m[I], A::sub(A::add(A::mul(d[I], x[I]), b[I]), faces6(x, I, n1, n2)));
}
template <class T>
__device__ __forceinline__ T v_resid9(const T* x, const T* b, const T* d, const uint8_t* m, long long n1, long long I) {
  typedef Ar<T> A;
  T v = A::add(A::mul(d[I], x[I]), b[I]);
  v = A::fmx(sum4(x, I, n1), T(-0.5), v);
  v = A::fmx(diags4(x, I, n1), T(-0.25), v);
  return mask_mul(m[I], v);
}
// residual_laplacian9! (src/laplacian9.jl:49-73)
template <class T>
__device__ __forceinline__ T v_resid19(const T* x, const T* b, const T* d, const uint8_t* m, long long n1,
                                       long long n2, long long I) {
  typedef Ar<T> A;
  T v = A::add(A::mul(d[I], x[I]), b[I]);
  v = A::fmx(faces6(x, I, n1, n2), T(-0.5), v);
  v = A::fmx(edges12(x, I, n1, n2), T(-0.25), v);
  return mask_mul(m[I], v);
}
template <class T>
__device__ __forceinline__ void d_resid5(T* r, const T* x, const T* b, const T* d, const uint8_t* m, long long n1,
                                         long long I) {
  r[I] = v_resid5(x, b, d, m, n1, I);
}
template <class T>
__device__ __forceinline__ void d_resid7(T* r, const T* x, const T* b, const T* d, const uint8_t* m, long long n1,
                                         long long n2, long long I) {
  r[I] = v_resid7(x, b, d, m, n1, n2, I);
}
template <class T>
__device__ __forceinline__ void d_resid9(T* r, const T* x, const T* b, const T* d, const uint8_t* m, long long n1,
                                         long long I) {
  r[I] = v_resid9(x, b, d, m, n1, I);
}
template <class T>
__device__ __forceinline__ void d_resid19(T* r, const T* x, const T* b, const T* d, const uint8_t* m, long long n1,
                                          long long n2, long long I) {
  r[I] = v_resid19(x, b, d, m, n1, n2, I);
}
template <class T>
__device__ __forceinline__ T v_residvc(const T* x, const T* b, const T* d, const T* cE, const T* cN, const uint8_t* m,
                                       long long n1, long long I) {
  typedef Ar<T> A;
  return mask_mul(m[I], A::sub(A::add(A::mul(d[I], x[I]), b[I]), vc_sum(x, cE, cN, I, n1)));
}
template <class T>
__device__ __forceinline__ void d_residvc(T* r, const T* x, const T* b, const T* d, const T* cE, const T* cN,
                                          const uint8_t* m, long long n1, long long I) {
  r[I] = v_residvc(x, b, d, cE, cN, m, n1, I);
}

// ------------------------------------------------ FP64 on zero operands
// The FP64 pipe bounds every FP64 operator (one warp instruction in 76 clocks
// per quarter of an SM), and over land and halo its operands are zeros. When
// a whole warp's are, the standalone kernels take the result from the sign
// bits instead: IEEE sums of zeros are +0 unless every term is -0. These
// return false (the caller computes) unless every operand is a zero and the
// coefficients are finite; zero_sweep also needs omega*idiag = +0 and
// 1-omega >= +0, as dry cells have for omega <= 1.
struct ZeroAcc {
  unsigned o = 0, l = 0, a = ~0u;
  __device__ __forceinline__ void add(double v) {
    const unsigned h = (unsigned)__double2hiint(v);
    o |= h;
    l |= (unsigned)__double2loint(v);
    a &= h;
  }
  __device__ __forceinline__ bool zero() const { return ((o << 1) | l) == 0u; }
  __device__ __forceinline__ bool neg() const { return (a >> 31) != 0u; }  // the sum of the zeros is -0
};
__device__ __forceinline__ bool is_neg(double v) { return __double2hiint(v) < 0; }
__device__ __forceinline__ bool is_fin(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }
__device__ __forceinline__ double signed_zero(bool neg) { return neg ? -0.0 : 0.0; }
enum ZeroStencil { ZS_5, ZS_7, ZS_19, ZS_VC };
// faces (and for the 19-point operator diagonals) of cell I; false when a value is not a zero
template <int ST>
__device__ __forceinline__ bool zero_nb(const double* x, const double* cE, const double* cN, long long I, long long n1,
                                        long long n2, bool& fneg, bool& dneg) {
  ZeroAcc f, d;
  f.add(x[I - 1]);
  f.add(x[I + 1]);
  f.add(x[I - n1]);
  f.add(x[I + n1]);
  bool ok = true;
  if (ST == ZS_7 || ST == ZS_19) {
    f.add(x[I - n2]);
    f.add(x[I + n2]);
  }
  if (ST == ZS_19) {
    d.add(x[I - 1 - n1]);
    d.add(x[I + 1 - n1]);
    d.add(x[I - 1 + n1]);
    d.add(x[I + 1 + n1]);
    d.add(x[I - 1 - n2]);
    d.add(x[I + 1 - n2]);
    d.add(x[I - 1 + n2]);
    d.add(x[I + 1 + n2]);
    d.add(x[I - n1 - n2]);
    d.add(x[I + n1 - n2]);
    d.add(x[I - n1 + n2]);
    d.add(x[I + n1 + n2]);
  }
  if (ST == ZS_VC) {  // products with face coefficients >= +0 keep the sign
    const double c[4] = {cE[I - 1], cE[I], cN[I - n1], cN[I]};
#pragma unroll
    for (int q = 0; q < 4; ++q) ok = ok && !is_neg(c[q]) && is_fin(c[q]);
  }
  fneg = f.neg();
  dneg = d.neg();
  return ok && f.zero() && (ST == ZS_19 ? d.zero() : true);
}
template <int ST>
__device__ __forceinline__ bool zero_sweep(const double* x, const double* b, const double* w, const double* cE,
                                           const double* cN, double cff, long long n1, long long n2, long long I,
                                           double& out) {
  bool fneg, dneg;
  ZeroAcc c;
  const double xv = x[I], bv = b[I];
  c.add(xv);
  c.add(bv);
  if (!zero_nb<ST>(x, cE, cN, I, n1, n2, fneg, dneg) || !c.zero() || __double_as_longlong(w[I]) != 0ll ||
      !(cff >= 0.0) || is_neg(cff))
    return false;
  // b - faces (- diagonals) is -0 only from -0 minus sums that are all +0
  bool tneg = is_neg(bv) && !fneg;
  if (ST == ZS_19) tneg = tneg && !dneg;
  out = signed_zero(is_neg(xv) && !tneg);
  return true;
}
template <int ST>
__device__ __forceinline__ bool zero_resid(const double* x, const double* b, const double* d, const double* cE,
                                           const double* cN, long long n1, long long n2, long long I, double& out) {
  bool fneg, dneg;
  ZeroAcc c;
  const double xv = x[I], bv = b[I], dv = d[I];
  c.add(xv);
  c.add(bv);
  if (!zero_nb<ST>(x, cE, cN, I, n1, n2, fneg, dneg) || !c.zero() || !is_fin(dv)) return false;
  bool v = (is_neg(dv) != is_neg(xv)) && is_neg(bv) && !fneg;  // (d x + b) - faces
  if (ST == ZS_19) v = v && !dneg;
  out = signed_zero(v);  // whatever the mask: it keeps the sign of a zero
  return true;
}

// ---------------------------------------------------------- restriction
// Coarse interior cell (ii, jj, kk) of kind 0 centres 2D (rcloop2d!,
// src/RP_on_centers.jl:117-133), 1 centres 3D (rcloop3d!, :5-23),
// 2 vertices 2D (rvloop2d!, src/RP_on_vertices.jl:96-115), 3 vertices 3D
// (restriction_vertices!, :1-32).
template <class T, int KIND>
__device__ __forceinline__ T v_restrict(const T* x, const T* coef, const Geom& gf, const Geom& gc, int ii, int jj,
                                        int kk, long long& C) {
  typedef Ar<T> A;
  const int nh = gc.nh;
  const int i = c2f(ii, nh), j = c2f(jj, nh);
  const long long n1 = gf.n1, n2 = gf.n2;
  T s;
  if (KIND == 0) {
    long long F = lin(gf, i, j, kk);
    s = A::add(A::add(A::add(x[F], x[F + 1]), x[F + n1]), x[F + 1 + n1]);
  } else if (KIND == 1) {
    long long F = lin(gf, i, j, c2f(kk, nh));
    s = A::add(x[F], x[F + 1]);
    s = A::add(s, x[F + n1]);
    s = A::add(s, x[F + 1 + n1]);
    s = A::add(s, x[F + n2]);
    s = A::add(s, x[F + 1 + n2]);
    s = A::add(s, x[F + n1 + n2]);
    s = A::add(s, x[F + 1 + n1 + n2]);
  } else if (KIND == 2) {  // 1-2-1 x 1-2-1
    long long F = lin(gf, i, j, kk);
    s = A::fmx(x[F - n1], T(2), x[F - 1 - n1]);
    s = A::add(s, x[F + 1 - n1]);
    s = A::fmx(x[F - 1], T(2), s);
    s = A::fmx(x[F], T(4), s);
    s = A::fmx(x[F + 1], T(2), s);
    s = A::add(s, x[F - 1 + n1]);
    s = A::fmx(x[F + n1], T(2), s);
    s = A::add(s, x[F + 1 + n1]);
  } else {  // 27 points, weights 1-2-4-8, left fold in source order
    long long F = lin(gf, i, j, c2f(kk, nh));
    bool first = true;
    s = T(0);
#pragma unroll
    for (int dk = -1; dk <= 1; ++dk)
#pragma unroll
      for (int dj = -1; dj <= 1; ++dj)
#pragma unroll
        for (int di = -1; di <= 1; ++di) {
          const int w = (2 - (di < 0 ? -di : di)) * (2 - (dj < 0 ? -dj : dj)) * (2 - (dk < 0 ? -dk : dk));
          T v = x[F + di + dj * n1 + dk * n2];
          if (first) {
            s = (w == 1) ? v : A::mul(T(w), v);
            first = false;
          } else {
            s = (w == 1) ? A::add(s, v) : A::fmx(v, T(w), s);
          }
        }
  }
  C = lin(gc, ii, jj, kk);
  return A::mul(coef[C], s);
}
template <class T, int KIND>
__device__ __forceinline__ void d_restrict(const T* x, T* xc, const T* coef, const Geom& gf, const Geom& gc, int ii,
                                           int jj, int kk) {
  long long C;
  const T v = v_restrict<T, KIND>(x, coef, gf, gc, ii, jj, kk, C);
  xc[C] = v;
}

// the restriction of zeros under a finite Rcoef (see ZeroAcc): the fold is -0 only when every child is
template <int KIND>
__device__ __forceinline__ bool zero_restrict(const double* x, double coef, const Geom& gf, const Geom& gc, int ii,
                                              int jj, int kk, double& out) {
  const int nh = gc.nh;
  const long long n1 = gf.n1, n2 = gf.n2;
  const bool t3 = KIND == 1 || KIND == 3;
  const long long F = lin(gf, c2f(ii, nh), c2f(jj, nh), t3 ? c2f(kk, nh) : kk);
  ZeroAcc a;
  constexpr int lo = KIND >= 2 ? -1 : 0;
#pragma unroll
  for (int dk = t3 ? lo : 0; dk <= (t3 ? 1 : 0); ++dk)
#pragma unroll
    for (int dj = lo; dj <= 1; ++dj)
#pragma unroll
      for (int di = lo; di <= 1; ++di) a.add(x[F + di + dj * n1 + dk * n2]);
  if (!a.zero() || !is_fin(coef)) return false;
  out = signed_zero(a.neg() != is_neg(coef));
  return true;
}

// --------------------------------------------------------- prolongation
// square (src/RP_on_centers.jl:1-3): 3*(x[i+di,j,k+dk]+x[i,j+dj,k+dk]) + x[i+di,j+dj,k+dk]
template <class T>
__device__ __forceinline__ T square3(const T* x, long long C, long long di, long long dj, long long dk) {
  typedef Ar<T> A;
  return A::add(A::mul(T(3), A::add(x[C + di + dk], x[C + dj + dk])), x[C + di + dj + dk]);
}

// Fine parent (p, q, qk): i = nh+1+2p, j = nh+1+2q, and k = kf0+qk (2D) or
// nh+1+2qk (3D). The parent updates its 4 (2D) or 8 (3D) children, which no
// other parent touches. Kinds as in d_restrict: pcloop2d!
// (src/RP_on_centers.jl:146-163), pcloop3d! (:84-104), pvloop2d!
// (src/RP_on_vertices.jl:117-137), prolongation_vertices! (:34-72).
// ASSIGN: the fine x is known to hold +0 at every updated cell, so it is
// not read: x = +0 + coef*v gives the same value and the same zero sign.
template <class T, int KIND, bool ASSIGN = false>
__device__ __forceinline__ void d_prolong(T* xf, const T* x, const T* coef, const Geom& gf, const Geom& gc, int p,
                                          int q, int qk, int kf0) {
  typedef Ar<T> A;
  const int nh = gf.nh;
  const int i = nh + 1 + 2 * p, j = nh + 1 + 2 * q;
  const int ic = f2c(i, nh), jc = f2c(j, nh);
  const long long c1 = gc.n1, c2 = gc.n2, f1 = gf.n1, f2 = gf.n2;
  if (KIND == 0) {
    const int k = kf0 + qk;
    const long long C = lin(gc, ic, jc, k), F = lin(gf, i, j, k);
    const T x9 = A::mul(x[C], T(9));
    // every load of the four children before the first store, so that they
    // are in flight together (the compiler cannot move a load of one child
    // above the store of another: the arrays might alias)
    T bb[4], cf[4], xo[4];
#pragma unroll
    for (int dj = 0; dj <= 1; ++dj)
#pragma unroll
      for (int di = 0; di <= 1; ++di) {
        const int c = 2 * dj + di;
        const long long Fi = F + di + dj * f1;
        bb[c] = square3(x, C, (long long)(2 * di - 1), (2 * dj - 1) * c1, 0LL);
        cf[c] = coef[Fi];
        xo[c] = ASSIGN ? T(0) : xf[Fi];
      }
#pragma unroll
    for (int dj = 0; dj <= 1; ++dj)
#pragma unroll
      for (int di = 0; di <= 1; ++di) {
        const int c = 2 * dj + di;
        xf[F + di + dj * f1] = A::add(xo[c], A::mul(cf[c], A::add(bb[c], x9)));
      }
  } else if (KIND == 1) {
    const int k = nh + 1 + 2 * qk;
    const int kc = f2c(k, nh);
    const long long C = lin(gc, ic, jc, kc), F = lin(gf, i, j, k);
    const T x28 = A::mul(x[C], T(28));
#pragma unroll
    for (int dj = 0; dj <= 1; ++dj)
#pragma unroll
      for (int di = 0; di <= 1; ++di) {
        const long long ddi = 2 * di - 1, ddj = (2 * dj - 1) * c1;
        T a = square3(x, C, ddi, ddj, -c2);
        T bb = A::mul(square3(x, C, ddi, ddj, 0LL), T(3));
        T c = square3(x, C, ddi, ddj, c2);
        long long F0 = F + di + dj * f1, F1 = F0 + f2;
        xf[F0] = A::add(ASSIGN ? T(0) : xf[F0], A::mul(coef[F0], A::add(A::add(bb, a), x28)));
        xf[F1] = A::add(ASSIGN ? T(0) : xf[F1], A::mul(coef[F1], A::add(A::add(bb, c), x28)));
      }
  } else if (KIND == 2) {
    const int k = kf0 + qk;
    const long long C = lin(gc, ic, jc, k), F = lin(gf, i, j, k);
    const T x00 = x[C], x10 = x[C + 1], x01 = x[C + c1], x11 = x[C + 1 + c1];
    const long long o[4] = {0, 1, f1, 1 + f1};
    T cf[4], xo[4];  // loads of the four children first, as in KIND 0
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      cf[c] = coef[F + o[c]];
      xo[c] = ASSIGN ? T(0) : xf[F + o[c]];
    }
    xf[F] = A::add(xo[0], A::mul(cf[0], x00));
    xf[F + 1] = A::add(xo[1], A::mul(cf[1], A::add(x00, x10)));
    xf[F + f1] = A::add(xo[2], A::mul(cf[2], A::add(x00, x01)));
    xf[F + 1 + f1] = A::add(xo[3], A::mul(cf[3], A::add(A::add(A::add(x00, x10), x01), x11)));
  } else {
    const int k = nh + 1 + 2 * qk;
    const int kc = f2c(k, nh);
    const long long C = lin(gc, ic, jc, kc), F = lin(gf, i, j, k);
    const T x000 = x[C], x100 = x[C + 1], x010 = x[C + c1], x001 = x[C + c2];
    const T x110 = x[C + 1 + c1], x101 = x[C + 1 + c2], x011 = x[C + c1 + c2], x111 = x[C + 1 + c1 + c2];
    auto upd = [&](long long Fi, T v) { xf[Fi] = A::add(ASSIGN ? T(0) : xf[Fi], A::mul(coef[Fi], v)); };
    upd(F, x000);
    upd(F + 1, A::add(x000, x100));
    upd(F + f1, A::add(x000, x010));
    upd(F + f2, A::add(x000, x001));
    upd(F + 1 + f1, A::add(A::add(A::add(x000, x100), x010), x110));
    upd(F + 1 + f2, A::add(A::add(A::add(x000, x100), x001), x101));
    upd(F + f1 + f2, A::add(A::add(A::add(x000, x001), x010), x011));
    T s = A::add(x000, x100);
    s = A::add(s, x001);
    s = A::add(s, x101);
    s = A::add(s, x010);
    s = A::add(s, x110);
    s = A::add(s, x011);
    s = A::add(s, x111);
    upd(F + 1 + f1 + f2, s);
  }
}

// d_prolong's value of one child (di = ch & 1, dj = ch >> 1 & 1, dk = ch >> 2)
// of coarse cell C before its Pcoef, in d_prolong's order.
template <class T, int K>
__device__ __forceinline__ T prolong_child(const T* x, long long C, long long c1, long long c2, int ch) {
  typedef Ar<T> A;
  const int di = ch & 1, dj = (ch >> 1) & 1, dk = ch >> 2;
  if (K == 0) return A::add(square3(x, C, (long long)(2 * di - 1), (2 * dj - 1) * c1, 0LL), A::mul(x[C], T(9)));
  if (K == 1) {
    const long long ddi = 2 * di - 1, ddj = (2 * dj - 1) * c1;
    const T bb = A::mul(square3(x, C, ddi, ddj, 0LL), T(3));
    return A::add(A::add(bb, square3(x, C, ddi, ddj, dk ? c2 : -c2)), A::mul(x[C], T(28)));
  }
  T v = x[C];
  if (K == 2) {
    if (di) v = A::add(v, x[C + 1]);
    if (dj) v = A::add(v, x[C + c1]);
    return di && dj ? A::add(v, x[C + 1 + c1]) : v;
  }
  const T x100 = x[C + 1], x010 = x[C + c1], x001 = x[C + c2];
  switch (ch) {
    case 0: return v;
    case 1: return A::add(v, x100);
    case 2: return A::add(v, x010);
    case 4: return A::add(v, x001);
    case 3: return A::add(A::add(A::add(v, x100), x010), x[C + 1 + c1]);
    case 5: return A::add(A::add(A::add(v, x100), x001), x[C + 1 + c2]);
    case 6: return A::add(A::add(A::add(v, x001), x010), x[C + c1 + c2]);
    default: break;
  }
  v = A::add(v, x100);
  v = A::add(v, x001);
  v = A::add(v, x[C + 1 + c2]);
  v = A::add(v, x010);
  v = A::add(v, x[C + 1 + c1]);
  v = A::add(v, x[C + c1 + c2]);
  return A::add(v, x[C + 1 + c1 + c2]);
}
// FP64 parent whose update changes nothing: its children's Pcoef and fine x
// are all +0, and every coarse value it reads is finite with room for the
// weights (below 2^1009), so +0 + 0*v = +0
template <int KIND>
__device__ __forceinline__ bool zero_prolong(const double* xf, const double* x, const double* coef, const Geom& gf,
                                             const Geom& gc, int p, int q, int qk, int kf0) {
  const int nh = gf.nh;
  const int i = nh + 1 + 2 * p, j = nh + 1 + 2 * q;
  const bool t3 = KIND == 1 || KIND == 3;
  const int k = t3 ? nh + 1 + 2 * qk : kf0 + qk;
  const long long F = lin(gf, i, j, k), f1 = gf.n1, f2 = gf.n2;
  unsigned long long o = 0;
#pragma unroll
  for (int c = 0; c < (t3 ? 8 : 4); ++c) {
    const long long Fi = F + (c & 1) + ((c >> 1) & 1) * f1 + (c >> 2) * f2;
    o |= (unsigned long long)__double_as_longlong(coef[Fi]) | (unsigned long long)__double_as_longlong(xf[Fi]);
  }
  if (o) return false;
  const long long C = lin(gc, f2c(i, nh), f2c(j, nh), t3 ? f2c(k, nh) : k), c1 = gc.n1, c2 = gc.n2;
  constexpr int lo = KIND < 2 ? -1 : 0;
  int big = 0;
#pragma unroll
  for (int dk = t3 ? lo : 0; dk <= (t3 ? 1 : 0); ++dk)
#pragma unroll
    for (int dj = lo; dj <= 1; ++dj)
#pragma unroll
      for (int di = lo; di <= 1; ++di) big = max(big, __double2hiint(x[C + di + dj * c1 + dk * c2]) & 0x7fffffff);
  return big < 0x7f000000;
}

// ------------------------------------------------------- fixed point
// Integer form of the mixed loop's level-1 residual (k_mixed.cu, k_batch.cu).
// N bytes to shared memory behind the thread's back (cp.async)
template <int N>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "n"(N)
               : "memory");
}

// round(v * 2^k) for |v| 2^k < 2^59, ties away from zero; zero and
// subnormal v give 0. Branch-free: with M = m << 10 (m the 53-bit
// significand, v = m 2^(ex-1075)) and y = M >> n for n = 1084 - ex - k, the
// magnitude is (y + 1) >> 1 and its negative (-y) >> 1 = (~y + 1) >> 1, so one
// exclusive or serves the sign. The range bound keeps n >= 4; n is capped at
// 63, where y = 0 as for any shift past the significand, and as for ex = 0
// with k <= 1021 (fix_k).
__device__ __forceinline__ long long to_fix(double v, int k) {
  const int hi = __double2hiint(v);
  const unsigned lo = (unsigned)__double2loint(v);
  const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
  const int n = min(max(1084 - k - (int)(((unsigned)hi << 1) >> 21), 0), 63);
  const unsigned long long M = ((unsigned long long)__funnelshift_l(lo, mh, 10) << 32) | (lo << 10);
  return (((long long)(M >> n) ^ (long long)(hi >> 31)) + 1LL) >> 1;
}
// 58 - E for values below 2^E. The bound at -963 (k <= 1021) shows in no result:
// where max(|x|, |b|) is below 2^-963, or below 2^-537 already, the squares of b
// and r are zeros, so |b| and the residual are reported as 0 (or the reference
// rule's 1) and the FP32 right-hand side, at the scale that they give, is 0.
__device__ __forceinline__ int fix_k(int E) { return 58 - max(E, -963); }
// k for max(|x|, |b|) (device scalars S_MAXX, S_MAXB)
__device__ __forceinline__ int fix_exponent(const double* ds) {
  const double mx = fmax(ds[S_MAXX], ds[S_MAXB]);
  int e = 0;
  if (mx > 0 && isfinite(mx)) frexp(mx, &e);  // mx < 2^e
  return fix_k(e);
}

__device__ __forceinline__ double int_to_double(__int128 v) {
  return __dadd_rn(__dmul_rn((double)(long long)(v >> 64), 18446744073709551616.0), (double)(unsigned long long)v);
}
// The end of the fixed-point residual passes, for blocks of kMxThreads: the
// block's sum r^2 (s2 of each thread, times 2^e2) into partials[blk] and its
// sum r (s1 of each thread, exact, in units of 2^-e1) into partials[kMxParts +
// blk], both combined in FP64. EXACT (the 7-point passes): sum r stays an
// integer, its low word there and its high word in partials[2 kMxParts + blk],
// so that the split of the cells over threads does not show in the wet mean,
// which is rounding noise of a sum that cancels. Unused ones are cleared for
// the final pass.
template <bool EXACT>
__device__ __forceinline__ void int_partials(double s2, __int128 s1, int e2, int e1, double* __restrict__ partials) {
  __shared__ double sh2[kMxThreads / 32], sd[EXACT ? 1 : kMxThreads / 32];
  __shared__ __int128 si[EXACT ? kMxThreads / 32 : 1];
  double d1 = EXACT ? 0.0 : ldexp(int_to_double(s1), -e1);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s2 += __shfl_down_sync(0xffffffffu, s2, o);
    if (EXACT) {
      const unsigned long long l = __shfl_down_sync(0xffffffffu, (unsigned long long)s1, o);
      const long long h = __shfl_down_sync(0xffffffffu, (long long)(s1 >> 64), o);
      s1 += (__int128)(((unsigned __int128)(unsigned long long)h << 64) | l);
    } else {
      d1 += __shfl_down_sync(0xffffffffu, d1, o);
    }
  }
  if ((threadIdx.x & 31) == 0) {
    sh2[threadIdx.x >> 5] = s2;
    if (EXACT) si[threadIdx.x >> 5] = s1;
    else sd[threadIdx.x >> 5] = d1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double u = 0.0, v = 0.0;
    __int128 vi = 0;
    for (int w = 0; w < kMxThreads / 32; ++w) {
      u += sh2[w];
      if (EXACT) vi += si[w];
      else v += sd[w];
    }
    partials[blockIdx.x] = ldexp(u, e2);
    partials[kMxParts + blockIdx.x] = EXACT ? __longlong_as_double((long long)vi) : v;
    if (EXACT) partials[2 * kMxParts + blockIdx.x] = __longlong_as_double((long long)(vi >> 64));
    for (int i = gridDim.x + blockIdx.x; i < kMxParts; i += gridDim.x) {
      partials[i] = partials[kMxParts + i] = 0.0;
      if (EXACT) partials[2 * kMxParts + i] = 0.0;
    }
  }
}

// e * 2^p as a double, exactly, with integer operations on the bits of the
// float (the FP64 pipe then only adds: x + e*2^p rounds once, as
// fma((double)e, 2^p, x) does). Zeros keep their sign; subnormal, infinite
// and NaN e, and a result outside the normal range, take the FP64 path
// (s2p = 2^p as a double).
// the FP64 product for the rare e that the bit assembly does not cover; out
// of line, so that it stays a branch that only warps holding such an e take
// (inline, the compiler predicates it and every cell pays the FP64 pipe)
static __device__ __noinline__ double f2d_pow2_slow(float e, double s2p) { return __dmul_rn((double)e, s2p); }
__device__ __forceinline__ double f2d_pow2(float e, int p, double s2p) {
  // zero and normal e by integer operations on the bits, with no branch:
  // a divergent branch here had the compiler issue the caller's FP64 add on
  // both paths
  const unsigned u = __float_as_uint(e);
  const unsigned long long sgn = (unsigned long long)(u >> 31) << 63;
  const int ex = (int)((u >> 23) & 0xffu);
  const int dex = ex - 127 + 1023 + p;
  const bool zero = (u & 0x7fffffffu) == 0u;
  const bool normal = ex != 0 && ex != 255 && dex > 0 && dex < 2047;
  const unsigned long long bits =
      sgn | ((unsigned long long)(unsigned)dex << 52) | ((unsigned long long)(u & 0x7fffffu) << 29);
  double v = __longlong_as_double((long long)(zero ? sgn : bits));
  if (!zero && !normal) v = f2d_pow2_slow(e, s2p);
  return v;
}
// v as a float, to nearest even, with integer operations on the bits where v
// and the result are zero or normal; else on the FP64 pipe, out of line
static __device__ __noinline__ float d2f_slow(double v) { return (float)v; }
__device__ __forceinline__ float d2f(double v) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const int fe = (int)((hi >> 20) & 0x7ffu) - 1023 + 127;
  const unsigned m = ((hi & 0xfffffu) << 3) | (lo >> 29);
  const unsigned up = ((lo & 0x1fffffffu) + 0x0fffffffu + (m & 1u)) >> 29;  // past half, or half and odd
  const bool zero = ((hi << 1) | lo) == 0u;
  float f = __uint_as_float((hi & 0x80000000u) | (zero ? 0u : ((unsigned)fe << 23) + m + up));
  if (!zero && (fe < 1 || fe > 253)) f = d2f_slow(v);
  return f;
}
// the exponent p of a power of two 2^p held in a double
__device__ __forceinline__ int pow2_exponent(double v) {
  return (int)(((unsigned long long)__double_as_longlong(v) >> 52) & 0x7ffULL) - 1023;
}

// The solve! loop's test (src/gmg_solver.jl:29-39): hist[nite] = res after
// every residual, and another iteration while res > tol and nite < maxite
// (the count moves before the iteration runs).
__device__ __forceinline__ void loop_test(const LoopTest& lt, double res, double normb) {
  const int nite = (int)lt.ds[S_NITE];
  lt.hist[nite] = res;
  // a NaN or Inf in b or in the residual ends the loop (reported as
  // CFMG_ERR_NONFINITE): an infinite |b| would otherwise give res = 0
  const bool more = isfinite(normb) && isfinite(res) && res > lt.tol && nite < lt.maxite;
  if (more) lt.ds[S_NITE] = (double)(nite + 1);
  cudaGraphSetConditional(lt.hc, more ? 1u : 0u);
}

// ------------------------------------------------------------------ halo
// fill! for :xperio (src/halo.jl:6-9) on one (j,k) line. Each statement's
// right-hand columns are read before any is written, as Julia's sliced
// assignment does (this matters when nx < nh).
constexpr int kMaxNh = 8;
template <class T>
__device__ __forceinline__ void d_fill_line(T* row, int tx, int nh) {
  T tmp[kMaxNh];
#pragma unroll
  for (int i = 0; i < kMaxNh; ++i)
    if (i < nh) tmp[i] = row[tx - 2 * nh + i];
#pragma unroll
  for (int i = 0; i < kMaxNh; ++i)
    if (i < nh) row[i] = tmp[i];
#pragma unroll
  for (int i = 0; i < kMaxNh; ++i)
    if (i < nh) tmp[i] = row[nh + i];
#pragma unroll
  for (int i = 0; i < kMaxNh; ++i)
    if (i < nh) row[tx - nh + i] = tmp[i];
}

}  // namespace cfmg
