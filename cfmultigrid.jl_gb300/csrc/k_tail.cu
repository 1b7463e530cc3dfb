// Coarse tail of a cycle in one block's shared memory.
//
// Below some level a cycle is a chain of operators on a few hundred to a few
// thousand cells: what it costs is the hand-over between two operators, not
// their work. As Ops of the cluster engine (k_coarse.cu) each took 2.2-2.5 us:
// fetching the Op, loading its operands from L2 and a cluster barrier whose
// release waits for the stores. Here one block loads the arrays of every
// level of the tail into shared memory once, runs the whole chain there (a
// block barrier between two operators, a barrier of the warps that hold work
// inside a smoothing call) and writes back what it changed.
//
// A smoothing call sweeps a list of the level's cells that can change: those
// with omega*idiag, Pcoef or the mask not 0 (k_tail_lists, remade when a
// coefficient changes). Any other cell of the sweep range holds +0 in x and y
// (checked once a launch, at the level's first call) and
// (1-omega)*(+0) - 0*t = +0 keeps it there for any finite t, so leaving it
// out changes no bit. On the coarsest levels most of the range is halo and
// land (a 4^2 level: 16 of 80 cells), and the FP64 pipe (one warp instruction
// in 76 clocks per quarter of an SM, measured) is what bounds a sweep there.
// A level that fails the check, one with a NaN or an infinity in x, y or b
// (t is not finite then), or omega > 1 (whose zeros change sign), sweeps its
// whole range as the reference does. The residual below level 1
// is formed at the listed cells; the others, whose mask is 0, get +0.
//
// The per-cell arithmetic and ranges are those of the standalone kernels
// (ops_dev.cuh), so the results are the same bits.
//
// Measured, engine Ops against this, per cycle: the tail of a 1152 x 608
// x-periodic mixed solve (levels 72 x 38 and below, with their coarsest FP64
// solve) 352 us of 443 against about 80 of 245; of a 64^2 FP64 solve (32^2
// and below) 118 of 157 against 68 of 108. What is left there is the FP64
// pipe (a 680-cell sweep: 3.5k clocks of the block's 4 quarters) and 0.2-0.4
// us an operator for its descriptor, its first loads and the barrier. 512
// threads: 128 registers each, and no more than 4 warps a quarter wait at a
// barrier.
#include "ops_dev.cuh"

namespace cfmg {

namespace {

constexpr int kTT = kTailThreads;
// list entries: cell index, bit 15 set when the cell is outside the second
// sweep's box (9- and 19-point operators)
constexpr unsigned kOut2 = 0x8000u;
// the block's dynamic shared memory
extern __shared__ __align__(16) unsigned char sm[];

// the value of one sweep at I; b and omega*idiag of the cell come in registers
template <class T, int ST>
__device__ __forceinline__ T tail_cell(const T* x, int I, int n1, int n2, T bI, T wI, T cff, const T* cE,
                                       const T* cN) {
  typedef Ar<T> A;
  const long long L = I, N1 = n1, N2 = n2;
  T t;
  if (ST == TAIL_5) t = A::sub(bI, sum4(x, L, N1));
  else if (ST == TAIL_7) t = A::sub(bI, faces6(x, L, N1, N2));
  else if (ST == TAIL_9) {
    t = A::fmx(sum4(x, L, N1), T(-0.5), bI);
    t = A::fmx(diags4(x, L, N1), T(-0.25), t);
  } else if (ST == TAIL_19) {
    t = A::fmx(faces6(x, L, N1, N2), T(-0.5), bI);
    t = A::fmx(edges12(x, L, N1, N2), T(-0.25), t);
  } else t = A::sub(bI, vc_sum(x, cE, cN, L, N1));
  return A::sub(A::mul(cff, x[I]), A::mul(wI, t));
}

// barrier of the first nw warps of the block
__device__ __forceinline__ void bar_warps(int nw) {
  if (nw == 1) __syncwarp();
  else asm volatile("bar.sync 1, %0;" ::"r"(nw * 32) : "memory");
}

// npairs pairs of sweeps over the listed cells. fill (x-periodic): fill! after
// each pair, as the second sweep's writers of the nh columns at either end
// writing their images in the halo (whose own cells are not swept then); a
// fill of every line in a step of its own, with its barrier, took as long as
// the two sweeps of a small level. whole: the list is the whole range (or
// nx < nh): fills as the reference does.
template <class T, int ST>
__device__ __forceinline__ void tail_smooth(int ctxi, int npairs, bool fill, bool whole, int nact) {
  const TailCtx& c = reinterpret_cast<const TailCtx*>(sm)[ctxi];
  T* x = reinterpret_cast<T*>(sm + c.ox);
  T* y = reinterpret_cast<T*>(sm + c.oy);
  const T* b = reinterpret_cast<const T*>(sm + c.ob);
  const T* w = reinterpret_cast<const T*>(sm + c.ow);
  const T* cE = reinterpret_cast<const T*>(sm + c.oE);
  const T* cN = reinterpret_cast<const T*>(sm + c.oN);
  const unsigned short* list = reinterpret_cast<const unsigned short*>(sm + c.olist + kTailListHdr);
  const T cff = (T)c.cff;
  const int n1 = c.n1, n2 = c.n2, tid = threadIdx.x;
  if (nact <= 0 && !fill) return;
  const bool img = fill && !whole && c.nx >= c.nh;
  const int nx = c.nx, nh = c.nh;
  // where the second sweep's value of cell I goes: bit 0 itself, 1 its image at I + nx, 2 at I - nx
  auto dest = [&](int I) -> unsigned {
    if (!img) return 1u;
    const int col = (int)((unsigned)I % (unsigned)n1);
    if (col < nh || col >= nh + nx) return 0u;
    return 1u | (col < 2 * nh ? 2u : 0u) | (col >= nx ? 4u : 0u);
  };
  auto put = [&](int I, T v, unsigned d) {
    if (d & 1u) x[I] = v;
    if (d & 2u) x[I + nx] = v;
    if (d & 4u) x[I - nx] = v;
  };
  auto fill_lines = [&]() {
    for (int t = tid; t < c.lines; t += kTT) d_fill_line(x + t * c.n1, c.n1, c.nh);
  };
  if ((!fill || img) && nact <= kTT) {  // one cell a thread, the warps that hold cells only
    const int nw = (nact + 31) >> 5;
    if ((tid >> 5) < nw) {
      const bool on = tid < nact;
      const unsigned e = list[on ? tid : 0];
      const int I = (int)(e & (kOut2 - 1));
      const bool on2 = on && !(e & kOut2);
      const T bI = b[I], wI = w[I];
      const unsigned d2 = on2 ? dest(I) : 0u;
      for (int p = 0; p < npairs; ++p) {
        T v = tail_cell<T, ST>(x, I, n1, n2, bI, wI, cff, cE, cN);
        if (on) y[I] = v;
        bar_warps(nw);
        v = tail_cell<T, ST>(y, I, n1, n2, bI, wI, cff, cE, cN);
        put(I, v, d2);
        bar_warps(nw);
      }
    }
    if (fill) {  // the lines out of the sweeps' range
      __syncthreads();
      fill_lines();
    }
    return;
  }
  for (int p = 0; p < npairs; ++p) {
    for (int t = tid; t < nact; t += kTT) {
      const int I = (int)(list[t] & (kOut2 - 1));
      y[I] = tail_cell<T, ST>(x, I, n1, n2, b[I], w[I], cff, cE, cN);
    }
    __syncthreads();
    for (int t = tid; t < nact; t += kTT) {
      const unsigned e = list[t];
      if (e & kOut2) continue;
      const int I = (int)e;
      put(I, tail_cell<T, ST>(y, I, n1, n2, b[I], w[I], cff, cE, cN), dest(I));
    }
    __syncthreads();
    if (fill && (!img || p == npairs - 1)) {
      fill_lines();
      __syncthreads();
    }
  }
}

template <class T>
__device__ __forceinline__ bool nonzero_bits(T v);
template <>
__device__ __forceinline__ bool nonzero_bits(float v) { return __float_as_uint(v) != 0u; }
template <>
__device__ __forceinline__ bool nonzero_bits(double v) { return __double_as_longlong(v) != 0ll; }

__device__ __forceinline__ bool finite_bits(float v) { return (__float_as_uint(v) & 0x7f800000u) != 0x7f800000u; }
__device__ __forceinline__ bool finite_bits(double v) { return is_fin(v); }

// whether the level must sweep its whole range: a cell that the context's list
// leaves out holds something in x or y or a NaN or an infinity in b, or (where
// x was not zeroed in the program) any cell of the array one in x or y: the
// sweeps carry them on
template <class T>
__device__ __forceinline__ bool tail_dirty(const TailCtx& c, int nact, int nrange) {
  const T* x = reinterpret_cast<const T*>(sm + c.ox);
  const T* y = reinterpret_cast<const T*>(sm + c.oy);
  const T* b = reinterpret_cast<const T*>(sm + c.ob);
  const unsigned short* list = reinterpret_cast<const unsigned short*>(sm + c.olist + kTailListHdr);
  bool bad = false;
  for (int t = nact + (int)threadIdx.x; t < nrange; t += kTT) {
    const int I = list[t] & (kOut2 - 1);
    bad |= nonzero_bits(x[I]) || nonzero_bits(y[I]) || !finite_bits(b[I]);
  }
  if (c.scan)
    for (int I = threadIdx.x; I < c.lines * c.n1; I += kTT) bad |= !finite_bits(x[I]) || !finite_bits(y[I]);
  return bad;
}

// operand of a TailOp: an offset into the block's shared memory (kTailSmem set) or a global address
template <class T>
__device__ __forceinline__ T* tail_ptr(unsigned long long p) {
  return (p & kTailSmem) ? reinterpret_cast<T*>(sm + (unsigned)p) : reinterpret_cast<T*>(p);
}

struct TailBox {  // box decoding in 32-bit arithmetic
  unsigned ni, nj;
  Box b;
  __device__ TailBox(const Box& bb) : ni(bb.i1 - bb.i0 + 1), nj(bb.j1 - bb.j0 + 1), b(bb) {}
  __device__ void at(unsigned t, int& i, int& j, int& k) const {
    const unsigned q = t / ni, r = q / nj;
    i = b.i0 + (int)(t - q * ni);
    j = b.j0 + (int)(q - r * nj);
    k = b.k0 + (int)r;
  }
};

__device__ __forceinline__ Geom tail_geom(int tx, int ty, int tz, int nh) {
  Geom g;
  g.tx = tx; g.ty = ty; g.tz = tz; g.nh = nh;
  g.n1 = tx; g.n2 = (long long)tx * ty; g.len = g.n2 * tz;
  return g;
}

template <class T, int ST>
__device__ __forceinline__ void tail_resid(const TailOp& op) {
  const T* x = tail_ptr<const T>(op.x);
  const T* b = tail_ptr<const T>(op.b);
  const T* d = tail_ptr<const T>(op.d);
  const T* cE = tail_ptr<const T>(op.cE);
  const T* cN = tail_ptr<const T>(op.cN);
  const uint8_t* m = tail_ptr<const uint8_t>(op.m);
  T* y = tail_ptr<T>(op.y);
  const Geom g = tail_geom(op.tx, op.ty, op.tz, op.nh);
  auto cell = [&](long long I) {
    if (ST == TAIL_5) d_resid5(y, x, b, d, m, g.n1, I);
    else if (ST == TAIL_VC) d_residvc(y, x, b, d, cE, cN, m, g.n1, I);
    else if (ST == TAIL_7) d_resid7(y, x, b, d, m, g.n1, g.n2, I);
    else if (ST == TAIL_9) d_resid9(y, x, b, d, m, g.n1, I);
    else d_resid19(y, x, b, d, m, g.n1, g.n2, I);
  };
  if (op.ctxi >= 0) {  // below level 1: the listed cells; +0 at the others (their mask is 0)
    const TailCtx& c = reinterpret_cast<const TailCtx*>(sm)[op.ctxi];
    const int* hdr = reinterpret_cast<const int*>(sm + c.olist);
    const unsigned short* list = reinterpret_cast<const unsigned short*>(sm + c.olist + kTailListHdr);
    const int nact = hdr[0], nrange = hdr[1];
    const unsigned n1 = (unsigned)op.tx, nj = (unsigned)op.ty;
    for (int t = threadIdx.x; t < nrange; t += kTT) {
      const unsigned e = list[t];
      if (e & kOut2) continue;  // the residual's range is the second sweep's
      if (ST == TAIL_7) {       // whose sweeps cover whole planes, the residual the interior box
        const unsigned r = e / n1, k = r / nj;
        const int i = (int)(e - r * n1) + 1, j = (int)(r - k * nj) + 1, kk = (int)k + 1;
        if (i < op.box.i0 || i > op.box.i1 || j < op.box.j0 || j > op.box.j1 || kk < op.box.k0 || kk > op.box.k1)
          continue;
      }
      if (t < nact) cell((long long)e);
      else y[e] = T(0);
    }
    return;
  }
  if (ST == TAIL_5 || ST == TAIL_VC) {
    for (int t = threadIdx.x; t < op.n; t += kTT) cell(op.lo + t);
  } else {
    const TailBox q(op.box);
    for (int t = threadIdx.x; t < op.n; t += kTT) {
      int i, j, k;
      q.at(t, i, j, k);
      cell(lin(g, i, j, k));
    }
  }
}

template <class T, int K>
__device__ __forceinline__ void tail_restrict(const TailOp& op) {
  const T* x = tail_ptr<const T>(op.x);
  const T* coef = tail_ptr<const T>(op.coef);
  T* y = tail_ptr<T>(op.y);
  const Geom g = tail_geom(op.tx, op.ty, op.tz, op.nh), gc = tail_geom(op.ctx, op.cty, op.tz, op.nh);
  const TailBox q(op.box);
  for (int t = threadIdx.x; t < op.n; t += kTT) {
    int i, j, k;
    q.at(t, i, j, k);
    d_restrict<T, K>(x, y, coef, g, gc, i, j, k);
  }
}

// a thread per child instead of per parent: a parent's 29 FP64 instructions in
// one warp took 1.1 us on a level of 16 parents
template <class T, int K>
__device__ __forceinline__ void tail_prolong(const TailOp& op) {
  const T* x = tail_ptr<const T>(op.x);
  const T* coef = tail_ptr<const T>(op.coef);
  T* y = tail_ptr<T>(op.y);
  const Geom g = tail_geom(op.tx, op.ty, op.tz, op.nh), gc = tail_geom(op.ctx, op.cty, op.tz, op.nh);
  constexpr bool t3 = K == 1 || K == 3;
  constexpr int nch = t3 ? 8 : 4;
  const unsigned ni = op.np_i, nj = op.np_j;
  const int nh = op.nh;
  for (int s = threadIdx.x; s < op.n * nch; s += kTT) {
    const unsigned ch = s % nch, t = s / nch, q = t / ni, r = q / nj;
    const int i = nh + 1 + 2 * (int)(t - q * ni), j = nh + 1 + 2 * (int)(q - r * nj);
    const int k = t3 ? nh + 1 + 2 * (int)r : op.kf0 + (int)r;
    const long long C = lin(gc, f2c(i, nh), f2c(j, nh), t3 ? f2c(k, nh) : k);
    const long long F = lin(g, i + (int)(ch & 1), j + (int)((ch >> 1) & 1), k + (int)(ch >> 2));
    y[F] = Ar<T>::add(y[F], Ar<T>::mul(coef[F], prolong_child<T, K>(x, C, gc.n1, gc.n2, (int)ch)));
  }
}

template <class T, int ST, int K>
__device__ __forceinline__ void tail_exec(const TailOp& op) {
  if (op.kind >= OPK_RESTRICT0 && op.kind <= OPK_RESTRICT3) {
    tail_restrict<T, K>(op);
  } else if (op.kind >= OPK_PROLONG0 && op.kind <= OPK_PROLONG3) {
    tail_prolong<T, K>(op);
  } else if (op.kind == OPK_FILL) {
    T* y = tail_ptr<T>(op.y);
    for (int t = threadIdx.x; t < op.n; t += kTT) d_fill_line(y + (long long)t * op.tx, op.tx, op.nh);
  } else if (op.kind == OPK_ZERO) {
    T* y = tail_ptr<T>(op.y);
    for (int t = threadIdx.x; t < op.n; t += kTT) y[t] = T(0);
  } else {
    tail_resid<T, ST>(op);
  }
}

}  // namespace

// One program, run by one block. A kernel per stencil ST and transfer kind K:
// with all operators in one kernel, each reached by an indirect call, a lone
// warp spent some 1900 clocks around a smoothing call of a small level.
template <int ST, int K>
__device__ __forceinline__ void tail_run(const unsigned char* __restrict__ blob, int blob_bytes, int nctx, int nstore,
                                         int ncopy, int nops) {
  __shared__ int full[kTailMaxCtx];  // -1: not looked at in this launch; 1: the context sweeps its whole range
  const int tid = threadIdx.x;
  // the program was uploaded before the launch: no kernel writes it
  for (int o = tid * 16; o < blob_bytes; o += kTT * 16)
    *reinterpret_cast<uint4*>(sm + o) = *reinterpret_cast<const uint4*>(blob + o);
  const TailCtx* ctx = reinterpret_cast<const TailCtx*>(sm);
  const TailCopy* cp = reinterpret_cast<const TailCopy*>(ctx + nctx);
  const TailOp* ops = reinterpret_cast<const TailOp*>(cp + ncopy);
  if (tid < kTailMaxCtx) full[tid] = -1;
  __syncthreads();
  dep_wait();
  // pieces of at most 16 bytes a thread, so that one pass over them keeps every load in flight
  const unsigned sb = (unsigned)__cvta_generic_to_shared(sm);
#pragma unroll 4
  for (int q = 0; q < ncopy; ++q)
    if (tid * 16 < (int)cp[q].bytes)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sb + cp[q].off + tid * 16),
                   "l"(reinterpret_cast<const unsigned char*>(cp[q].g) + tid * 16)
                   : "memory");
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  for (int o = 0; o < nops; ++o) {
    const TailOp& op = ops[o];
    if (op.kind == TAIL_SMOOTH) {
      const int q = op.ctxi;
      const TailCtx& c = ctx[q];
      const int* hdr = reinterpret_cast<const int*>(sm + c.olist);
      const int nact = hdr[0], nrange = hdr[1];
      int fl = full[q];
      if (fl < 0) {
        // nx < nh: the periodic halo of so narrow a level is not the image of its coefficients, and
        // fill! brings values to cells that the list leaves out
        const bool bad = c.cff < 0.0 || (op.fill && c.nx < c.nh) || (c.prec ? tail_dirty<float>(c, nact, nrange) : tail_dirty<double>(c, nact, nrange));
        fl = __syncthreads_or(bad) ? 1 : 0;
        if (tid == 0) full[q] = fl;
      }
      const int n = fl ? nrange : nact;
      if (c.prec) tail_smooth<float, ST>(q, op.npairs, op.fill != 0, fl != 0, n);
      else tail_smooth<double, ST>(q, op.npairs, op.fill != 0, fl != 0, n);
    } else if (op.kind == OPK_F32TO64) {
      const float* x = tail_ptr<const float>(op.x);
      double* y = tail_ptr<double>(op.y);
      for (int t = tid; t < op.n; t += kTT) y[t] = (double)x[t];
    } else if (op.kind == OPK_F64TO32) {
      const double* x = tail_ptr<const double>(op.x);
      float* y = tail_ptr<float>(op.y);
      for (int t = tid; t < op.n; t += kTT) y[t] = (float)x[t];
    } else if (op.prec) {
      tail_exec<float, ST, K>(op);
    } else {
      tail_exec<double, ST, K>(op);
    }
    if (!op.nobar) __syncthreads();
  }
  __syncthreads();
  // write back (the last 16 bytes may reach into the array's own padding, whose bytes were loaded with it)
#pragma unroll 4
  for (int q = 0; q < nstore; ++q)
    if (tid * 16 < (int)cp[q].bytes)
      *reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(cp[q].g) + tid * 16) =
          *reinterpret_cast<const uint4*>(sm + cp[q].off + tid * 16);
}

template <int ST, int K>
__global__ void __launch_bounds__(kTT, 1) k_tail(const unsigned char* __restrict__ blob, int blob_bytes, int nctx,
                                                 int nstore, int ncopy, int nops) {
  tail_run<ST, K>(blob, blob_bytes, nctx, nstore, ncopy, nops);
}

// batched solver: a block per program of the table, for instances still iterating
template <int ST, int K>
__global__ void __launch_bounds__(kTT, 1) k_tail_batch(const unsigned char* __restrict__ store,
                                                       const TailProg* __restrict__ tab,
                                                       const int* __restrict__ active) {
  const TailProg p = tab[blockIdx.x];  // uploaded before the launch
  dep_wait();
  if (!active[p.inst]) return;
  tail_run<ST, K>(store + p.off, p.bytes, p.nctx, p.nstore, p.ncopy, p.nops);
}

// The cell lists of the levels, one block a level: {live cells, cells of the
// first sweep's range}, then the live cells in rising order, then the others
// of the range; bit 15 marks a cell outside the second sweep's range.
__global__ void __launch_bounds__(1024) k_tail_lists(TailListArgs a) {
  dep_wait();
  const TailListLevel& l = a.lev[blockIdx.x];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = 32;
  __shared__ int cl[32], cd[32];
  const bool box = l.box != 0;
  const int n2 = l.n1 * l.nj;
  auto range = [&](int I) {  // 0: outside, 1: first sweep only, 2: both
    if (!box) return I >= l.lo && I < l.hi ? 2 : 0;
    const int k = I / n2, r = I - k * n2, j = r / l.n1, i = r - j * l.n1;
    auto in = [&](const Box& b) {
      return i >= b.i0 - 1 && i <= b.i1 - 1 && j >= b.j0 - 1 && j <= b.j1 - 1 && k >= b.k0 - 1 && k <= b.k1 - 1;
    };
    return in(l.ext) ? (in(l.in) ? 2 : 1) : 0;
  };
  auto live1 = [&](int I) { return nonzero_bits(l.w[I]) || nonzero_bits(l.pc[I]) || l.m[I] != 0; };
  auto live = [&](int I) {
    if (live1(I)) return true;
    if (!l.nx) return false;
    // x-periodic: fill! copies between a cell and its images, so they are listed together
    const int col = (int)((unsigned)I % (unsigned)l.n1);
    return ((col < 2 * l.nh && I + l.nx < l.len && live1(I + l.nx)) || (col >= l.nx && I >= l.nx && live1(I - l.nx)));
  };
  const int words = (l.len + 31) >> 5, per = (words + nw - 1) / nw;
  const int w0 = wid * per, w1 = min(words, (wid + 1) * per);
  int a0 = 0, a1 = 0;
  for (int wd = w0; wd < w1; ++wd) {
    const int I = wd * 32 + lane;
    const bool in = I < l.len && range(I) != 0, lv = in && live(I);
    a0 += __popc(__ballot_sync(0xffffffffu, lv));
    a1 += __popc(__ballot_sync(0xffffffffu, in && !lv));
  }
  if (lane == 0) {
    cl[wid] = a0;
    cd[wid] = a1;
  }
  __syncthreads();
  int bl = 0, bd = 0, tl = 0, td = 0;
  for (int v = 0; v < nw; ++v) {
    if (v < wid) {
      bl += cl[v];
      bd += cd[v];
    }
    tl += cl[v];
    td += cd[v];
  }
  bd += tl;
  unsigned short* list = reinterpret_cast<unsigned short*>(l.out + kTailListHdr);
  for (int wd = w0; wd < w1; ++wd) {
    const int I = wd * 32 + lane;
    const int rg = I < l.len ? range(I) : 0;
    const bool lv = rg && live(I);
    const unsigned b0 = __ballot_sync(0xffffffffu, lv), b1 = __ballot_sync(0xffffffffu, rg && !lv);
    const unsigned below = (1u << lane) - 1u;
    const unsigned short e = (unsigned short)(I | (rg == 1 ? kOut2 : 0u));
    if (lv) list[bl + __popc(b0 & below)] = e;
    else if (rg) list[bd + __popc(b1 & below)] = e;
    bl += __popc(b0);
    bd += __popc(b1);
  }
  if (threadIdx.x == 0) {
    int* hdr = reinterpret_cast<int*>(l.out);
    hdr[0] = tl;
    hdr[1] = tl + td;
  }
}

template <int ST, int K>
static void launch_tail_k(const void* blob, int blob_bytes, int nctx, int nstore, int ncopy, int nops, size_t smem,
                          cudaStream_t s) {
  static const cudaError_t attr =
      cudaFuncSetAttribute(k_tail<ST, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailSmemMax);
  (void)attr;
  launch_dep(k_tail<ST, K>, 1, kTT, smem, s, (const unsigned char*)blob, blob_bytes, nctx, nstore, ncopy, nops);
}
bool launch_tail(int stencil, int kind, const void* blob, int blob_bytes, int nctx, int nstore, int ncopy, int nops,
                 size_t smem, cudaStream_t s) {
#define CFMG_TAIL(ST, K)                                                           \
  if (stencil == ST && kind == K) {                                                \
    launch_tail_k<ST, K>(blob, blob_bytes, nctx, nstore, ncopy, nops, smem, s);    \
    return true;                                                                   \
  }
  CFMG_TAIL(TAIL_5, 0)
  CFMG_TAIL(TAIL_5, 2)
  CFMG_TAIL(TAIL_9, 0)
  CFMG_TAIL(TAIL_9, 2)
  CFMG_TAIL(TAIL_VC, 0)
  CFMG_TAIL(TAIL_7, 1)
  CFMG_TAIL(TAIL_7, 3)
  CFMG_TAIL(TAIL_19, 1)
  CFMG_TAIL(TAIL_19, 3)
#undef CFMG_TAIL
  return false;
}
template <int ST, int K>
static void launch_tail_batch_k(const void* store, const TailProg* tab, int n, size_t smem, const int* active,
                                cudaStream_t s) {
  static const cudaError_t attr =
      cudaFuncSetAttribute(k_tail_batch<ST, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTailSmemMax);
  (void)attr;
  launch_dep(k_tail_batch<ST, K>, (unsigned)n, kTT, smem, s, (const unsigned char*)store, tab, active);
}
bool launch_tail_batch(int stencil, int kind, const void* store, const TailProg* tab, int n, size_t smem,
                       const int* active, cudaStream_t s) {
  if (n <= 0) return true;
#define CFMG_TAIL(ST, K)                                                 \
  if (stencil == ST && kind == K) {                                      \
    launch_tail_batch_k<ST, K>(store, tab, n, smem, active, s);          \
    return true;                                                         \
  }
  CFMG_TAIL(TAIL_5, 0)
  CFMG_TAIL(TAIL_5, 2)
  CFMG_TAIL(TAIL_9, 0)
  CFMG_TAIL(TAIL_9, 2)
#undef CFMG_TAIL
  return false;
}

void launch_tail_lists(const TailListArgs& a, int n, cudaStream_t s) {
  if (n > 0) launch_dep(k_tail_lists, (unsigned)n, 1024, 0, s, a);
}

}  // namespace cfmg
