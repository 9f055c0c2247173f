// x-y plane passes of the stick-and-plane FFTs: the phases that one CTA runs
// over one z-plane in shared memory.
//
// Both directions use the four-step split N = A x B with every step in place:
//   columns (y) inverse: a) A-point DFTs over y = B n1 + n2, twiddles, rows
//                           B k1 + n2 of the plane;
//                        b) B-point DFTs over rows B k1 + n2; row B k1 + k2
//                           then holds y = k1 + A k2;
//   rows (x) inverse:    a) A-point over x = B n1 + n2, b) B-point over
//                           B k1 + n2, whose outputs x = k1 + A k2 are real
//                           space, in the registers of the thread that owns k1.
// The forward transforms run the transposed split (B, A): the B outputs of a
// thread in real space are the inputs of its forward B-point DFT, so real
// space never goes through shared memory, and each later step reads and writes
// the positions that the inverse step before it used.  No step ever permutes:
// the plane's rows stay at ys = B k1 + k2 for y = k1 + A k2 between the two
// column passes, and the arrays in real space (V(r), psi_v(r), dv(r)) are kept
// as [z][x][ys], so that the threads of a warp, which hold consecutive ys of
// one x, read them contiguously.
//
// Threads: consecutive threads take consecutive LINES (ys in the row phases,
// active columns in the column phases) at the same position along the line.
// With an odd row stride every access of a half- or quarter-warp then falls on
// distinct banks in all phases and both element sizes, and a warp's twiddles
// are one address, read from the constant bank (a 16-byte shared-memory load
// costs four wavefronts even when all lanes want the same element: 4,000 of
// 17,600 per FP64 108 x 108 plane).  The column phases take the sticks straight from
// global memory and give them back to it through cmap, so the plane is never
// zeroed, scattered to or gathered from.
#pragma once
#include "wb_fft.cuh"

namespace wb {

// Geometry of a plane.  Compiled cubic boxes: everything constant but the
// active columns of an unpruned one.  PR: the sphere lies in the outer quarters
// and A % 4 == 0, so dead inputs and outputs are known at compile time.
template <int N_, bool PR_>
struct CPlane {
  static constexpr int N = N_, A = FftSplit<N>::N1, B = FftSplit<N>::N2, RS = N | 1;
  static constexpr bool PR = PR_ && N % 4 == 0 && A % 4 == 0;
  static constexpr int SIZE = N * RS;
  int ncols_, nlow_;
  WB_DEV CPlane(int ncols, int nlow) : ncols_(ncols), nlow_(nlow) {}
  WB_DEV int ncols() const { return PR ? N / 2 : ncols_; }
  WB_DEV int nlow() const { return PR ? N / 4 : nlow_; }
  WB_DEV int nx() const { return N; }
  WB_DEV int ny() const { return N; }
  WB_DEV int ax() const { return A; }
  WB_DEV int bx() const { return B; }
  WB_DEV int ay() const { return A; }
  WB_DEV int by() const { return B; }
  WB_DEV int rs() const { return RS; }
  WB_DEV int div_cols(int i) const { return i / ncols(); }
  WB_DEV int div_rows(int i) const { return i / N; }
  // n1 of an A-point step whose elements are all zero (inverse) or unused (forward)
  WB_DEV static constexpr bool dead(int n1) { return PR && !(n1 < A / 4 || n1 >= A - A / 4); }
};

// Geometry of any other box: edges and splits taken at run time, no pruning
// beyond the active columns.
struct RPlane {
  static constexpr bool PR = false;
  int nx_, ny_, ax_, bx_, ay_, by_, ncols_, nlow_;
  unsigned mcols_, mrows_;  // ceil(2^32 / d): i / d = mulhi(i, m) for i d < 2^32
  WB_DEV int ncols() const { return ncols_; }
  WB_DEV int nlow() const { return nlow_; }
  WB_DEV int nx() const { return nx_; }
  WB_DEV int ny() const { return ny_; }
  WB_DEV int ax() const { return ax_; }
  WB_DEV int bx() const { return bx_; }
  WB_DEV int ay() const { return ay_; }
  WB_DEV int by() const { return by_; }
  WB_DEV int rs() const { return nx_ | 1; }
  WB_DEV int div_cols(int i) const { return (int)__umulhi((unsigned)i, mcols_); }
  WB_DEV int div_rows(int i) const { return (int)__umulhi((unsigned)i, mrows_); }
  WB_DEV static constexpr bool dead(int) { return false; }
};

// Step factors W_N^(k1 n2) at k1 B + n2 as a kernel parameter.
template <int N, class C>
struct TwParam {
  C t[N];
  WB_DEV C operator()(int i) const { return t[i]; }
};

// x of active column c, and whether x is one
template <class G>
WB_DEV int col_x(const G& g, int c) { return c < g.nlow() ? c : c + g.nx() - g.ncols(); }
template <class G>
WB_DEV bool live_x(const G& g, int x) { return x < g.nlow() || x >= g.nx() - (g.ncols() - g.nlow()); }

// columns, inverse a): sticks of the plane -> plane
template <int A, class G, class TW, class C>
WB_DEV void plane_col_in(C* pl, const TW& ty, const C* sz, const int* __restrict__ cmap, const G& g, int nt) {
  const int B = g.by(), nc = g.ncols(), rs = g.rs();
  for (int it = threadIdx.x; it < nc * B; it += nt) {
    const int n2 = g.div_cols(it), c = it - n2 * nc;
    int idx[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) idx[n1] = G::dead(n1) ? -1 : __ldg(cmap + (B * n1 + n2) * nc + c);
    C v[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) {
      v[n1] = mkc<C>(0, 0);
      if (!G::dead(n1) && idx[n1] >= 0) v[n1] = sz[idx[n1]];
    }
    rdft<A, +1>(v);
    C* p = pl + n2 * rs + col_x(g, c);
    p[0] = v[0];
#pragma unroll
    for (int k1 = 1; k1 < A; ++k1) p[B * k1 * rs] = ctw<+1>(v[k1], ty(k1 * B + n2));
  }
}
// columns, inverse b)
template <int B, class G, class C>
WB_DEV void plane_col_mid_inv(C* pl, const G& g, int nt) {
  const int A = g.ay(), nc = g.ncols(), rs = g.rs();
  for (int it = threadIdx.x; it < nc * A; it += nt) {
    const int k1 = g.div_cols(it), c = it - k1 * nc;
    C* p = pl + B * k1 * rs + col_x(g, c);
    C v[B];
#pragma unroll
    for (int i = 0; i < B; ++i) v[i] = p[i * rs];
    rdft<B, +1>(v);
#pragma unroll
    for (int i = 0; i < B; ++i) p[i * rs] = v[i];
  }
}
// columns, forward: B-point step and twiddles
template <int B, class G, class TW, class C>
WB_DEV void plane_col_mid_fwd(C* pl, const TW& ty, const G& g, int nt) {
  const int A = g.ay(), nc = g.ncols(), rs = g.rs();
  for (int it = threadIdx.x; it < nc * A; it += nt) {
    const int k1 = g.div_cols(it), c = it - k1 * nc;
    C* p = pl + B * k1 * rs + col_x(g, c);
    C v[B];
#pragma unroll
    for (int i = 0; i < B; ++i) v[i] = p[i * rs];
    rdft<B, -1>(v);
    p[0] = v[0];
#pragma unroll
    for (int q = 1; q < B; ++q) p[q * rs] = ctw<-1>(v[q], ty(k1 * B + q));
  }
}
// columns, forward: A-point step, plane -> sticks
template <int A, class G, class C>
WB_DEV void plane_col_out(const C* pl, C* sz, const int* __restrict__ cmap, const G& g, int nt) {
  const int B = g.by(), nc = g.ncols(), rs = g.rs();
  for (int it = threadIdx.x; it < nc * B; it += nt) {
    const int q = g.div_cols(it), c = it - q * nc;
    const C* p = pl + q * rs + col_x(g, c);
    int idx[A];
#pragma unroll
    for (int k = 0; k < A; ++k) idx[k] = G::dead(k) ? -1 : __ldg(cmap + (B * k + q) * nc + c);
    C v[A];
#pragma unroll
    for (int n = 0; n < A; ++n) v[n] = p[B * n * rs];
    rdft<A, -1>(v);
#pragma unroll
    for (int k = 0; k < A; ++k)
      if (!G::dead(k) && idx[k] >= 0) sz[idx[k]] = v[k];
  }
}
// rows, inverse a)
template <int A, class G, class TW, class C>
WB_DEV void plane_row_in(C* pl, const TW& tx, const G& g, int nt) {
  const int B = g.bx(), ny = g.ny(), rs = g.rs();
  for (int it = threadIdx.x; it < ny * B; it += nt) {
    const int n2 = g.div_rows(it), y = it - n2 * ny;
    C* p = pl + y * rs + n2;
    C v[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) {
      v[n1] = mkc<C>(0, 0);
      if (!G::dead(n1) && (G::PR || live_x(g, B * n1 + n2))) v[n1] = p[B * n1];
    }
    rdft<A, +1>(v);
    p[0] = v[0];
#pragma unroll
    for (int k1 = 1; k1 < A; ++k1) p[B * k1] = ctw<+1>(v[k1], tx(k1 * B + n2));
  }
}
// rows, inverse b): B real-space values x = k1 + A k2 of row y in v
template <int B, class C>
WB_DEV void row_to_real(const C* p, C* v) {
#pragma unroll
  for (int i = 0; i < B; ++i) v[i] = p[i];
  rdft<B, +1>(v);
}
// and back: forward B-point step and twiddles
template <int B, class TW, class C>
WB_DEV void row_from_real(C* p, C* v, const TW& tx, int k1) {
  rdft<B, -1>(v);
  p[0] = v[0];
#pragma unroll
  for (int q = 1; q < B; ++q) p[q] = ctw<-1>(v[q], tx(k1 * B + q));
}
// rows: inverse b), V(r) / N and the forward B-point step; vz = V of the plane, [x][ys]
template <int B, class G, class TW, class C>
WB_DEV void plane_row_vloc(C* pl, const TW& tx, const real_t<C>* __restrict__ vz, const G& g, int nt) {
  const int A = g.ax(), ny = g.ny(), rs = g.rs();
  for (int it = threadIdx.x; it < ny * A; it += nt) {
    const int k1 = g.div_rows(it), y = it - k1 * ny;
    C* p = pl + y * rs + B * k1;
    const real_t<C>* vr = vz + k1 * ny + y;
    real_t<C> w[B];
#pragma unroll
    for (int i = 0; i < B; ++i) w[i] = __ldg(vr + A * i * ny);
    C v[B];
    row_to_real<B>(p, v);
#pragma unroll
    for (int i = 0; i < B; ++i) v[i] = cscale(v[i], w[i]);
    row_from_real<B>(p, v, tx, k1);
  }
}
// rows: inverse b) to global memory, o = the plane's box, [x][ys]
template <int B, class G, class C>
WB_DEV void plane_row_box(const C* pl, C* __restrict__ o, const G& g, int nt) {
  const int A = g.ax(), ny = g.ny(), rs = g.rs();
  for (int it = threadIdx.x; it < ny * A; it += nt) {
    const int k1 = g.div_rows(it), y = it - k1 * ny;
    C v[B];
    row_to_real<B>(pl + y * rs + B * k1, v);
#pragma unroll
    for (int i = 0; i < B; ++i) o[(k1 + A * i) * ny + y] = v[i];
  }
}
// rows: inverse b) and the density sum += occ psi(r) dpsi(r) of a band pair, in
// global memory, one element per thread throughout (first: the sum starts here)
template <int B, class G, class C>
WB_DEV void plane_row_density(const C* pl, const C* __restrict__ ps, real_t<C>* __restrict__ sum, real_t<C> o1,
                              real_t<C> o2, bool first, const G& g, int nt) {
  const int A = g.ax(), ny = g.ny(), rs = g.rs();
  for (int it = threadIdx.x; it < ny * A; it += nt) {
    const int k1 = g.div_rows(it), y = it - k1 * ny;
    C v[B];
    row_to_real<B>(pl + y * rs + B * k1, v);
#pragma unroll
    for (int i = 0; i < B; ++i) {
      const int e = (k1 + A * i) * ny + y;
      const C s = ps[e];
      const real_t<C> d = fma(o1 * s.x, v[i].x, o2 * s.y * v[i].y);
      sum[e] = first ? d : sum[e] + d;
    }
  }
}
// rows: two real arrays (a + i b) scale -> forward B-point step
template <int B, class G, class TW, class C>
WB_DEV void plane_row_pair(C* pl, const TW& tx, const real_t<C>* a, const real_t<C>* b, real_t<C> scale, const G& g,
                           int nt) {
  const int A = g.ax(), ny = g.ny(), rs = g.rs();
  for (int it = threadIdx.x; it < ny * A; it += nt) {
    const int k1 = g.div_rows(it), y = it - k1 * ny;
    C v[B];
#pragma unroll
    for (int i = 0; i < B; ++i) {
      const int e = (k1 + A * i) * ny + y;
      v[i] = mkc<C>(a[e] * scale, b ? b[e] * scale : real_t<C>(0));
    }
    row_from_real<B>(pl + y * rs + B * k1, v, tx, k1);
  }
}
// rows: psi(r) dv(r) scale (dv: the real or the imaginary part of d) -> forward B-point step
template <int B, class G, class TW, class C>
WB_DEV void plane_row_rhs(C* pl, const TW& tx, const C* __restrict__ ps, const C* __restrict__ d, bool hi,
                          real_t<C> scale, const G& g, int nt) {
  const int A = g.ax(), ny = g.ny(), rs = g.rs();
  const real_t<C>* dr = reinterpret_cast<const real_t<C>*>(d) + (hi ? 1 : 0);
  for (int it = threadIdx.x; it < ny * A; it += nt) {
    const int k1 = g.div_rows(it), y = it - k1 * ny;
    C v[B];
    real_t<C> w[B];
#pragma unroll
    for (int i = 0; i < B; ++i) {
      const int e = (k1 + A * i) * ny + y;
      v[i] = ps[e];
      w[i] = dr[2 * e];
    }
#pragma unroll
    for (int i = 0; i < B; ++i) v[i] = cscale(v[i], w[i] * scale);
    row_from_real<B>(pl + y * rs + B * k1, v, tx, k1);
  }
}
// rows, forward: A-point step; only the active columns are written
template <int A, class G, class C>
WB_DEV void plane_row_out(C* pl, const G& g, int nt) {
  const int B = g.bx(), ny = g.ny(), rs = g.rs();
  for (int it = threadIdx.x; it < ny * B; it += nt) {
    const int q = g.div_rows(it), y = it - q * ny;
    C* p = pl + y * rs + q;
    C v[A];
#pragma unroll
    for (int n = 0; n < A; ++n) v[n] = p[B * n];
    rdft<A, -1>(v);
#pragma unroll
    for (int k = 0; k < A; ++k)
      if (!G::dead(k) && (G::PR || live_x(g, B * k + q))) p[B * k] = v[k];
  }
}

}  // namespace wb
