// Runtime-size stick-and-plane FFTs: the path for boxes without a compiled
// edge (non-cubic boxes, and the 2, 3, 5, 7-smooth edges outside the compiled
// list).  Same decomposition and Gamma pack/unpack as wb_fft_kernels.cu (z
// passes over stick pairs, one z-plane per CTA for the x-y passes, the
// caller's pointwise work between the inverse and the forward transforms),
// with line lengths, radix stages and twiddles taken at run time.
//
// A line is transformed in place, one radix stage at a time over the whole
// CTA: the inverse (QE invfft sign) by decimation in frequency, which leaves
// the result at digit-reversed positions, the forward by decimation in time
// over the same stages in reverse order, which takes digit-reversed input and
// returns natural order.  No permutation pass is ever run: real-space data
// live at digit-reversed positions in all three directions, they are only
// multiplied point by point with each other and with V(r), which the host
// stores in the same permuted layout.
//
// The x-y pass of most boxes (edges a * b with radices up to 16, the full plane
// in shared memory) runs the phases of wb_plane.cuh with the radices dispatched
// per phase: 45 x 54 planes take 1.2 us per FP64 item and z-plane set instead of
// 5.2 with the staged kernels.  The others (125, 128 x 128 in FP64, ...) keep only
// the plane's active columns (the x values of the sticks) in shared memory,
// column-major with an odd column stride; rows are transformed in chunks of full
// length through a row scratch area.
#include <algorithm>

#include <cmath>

#include "wb_internal.h"
#include "wb_plane.cuh"

namespace wb {

RtPlan rt_plan(int n) {
  RtPlan p{};
  p.n = n;
  p.ns = 0;
  int m = n;
  for (int r : {8, 4, 2, 3, 5, 7})
    while (m % r == 0 && p.ns < kRtMaxStages) {
      p.r[p.ns++] = r;
      m /= r;
    }
  if (m != 1 || n < 2) p.ns = 0;
  return p;
}

int rt_digit_reverse(const RtPlan& pl, int p) {
  int block = pl.n, mult = 1, k = 0, rem = p;
  for (int s = 0; s < pl.ns; ++s) {
    const int R = pl.r[s], m = block / R;
    k += (rem / m) * mult;
    rem %= m;
    mult *= R;
    block = m;
  }
  return k;
}

constexpr int kRtZsg = 8;      // stick pairs per z-pass CTA
constexpr int kRtZnt = 128;
constexpr int kRtPnt = 256;
constexpr int kRtMaxRows = 16; // rows per chunk of the row passes

size_t rt_plane_smem(const RtGeo& g, int elem_bytes, int* rows_per_chunk) {
  const size_t base = (size_t)elem_bytes * (g.nx + g.ny + (size_t)g.ncols * g.cs);
  const size_t cap = 227u * 1024u;
  if (base + (size_t)elem_bytes * g.nx > cap) return 0;
  int rc = (int)std::min<size_t>((cap - base) / ((size_t)elem_bytes * g.nx), (size_t)kRtMaxRows);
  rc = std::min(rc, g.ny);
  if (rows_per_chunk) *rows_per_chunk = rc;
  return base + (size_t)elem_bytes * rc * g.nx;
}

template <class C>
WB_DEV const C* rt_table(const double2* t64, const float2* t32) {
  if constexpr (sizeof(C) == 16) return reinterpret_cast<const C*>(t64);
  else return reinterpret_cast<const C*>(t32);
}

// One butterfly of radix R over legs base + q m (element stride es): DIF does
// the R-point DFT then the twiddles W_L^(q j), DIT the twiddles then the DFT;
// L = m R, W_L^(q j) = tw[q j ts] with ts = n / L (q j < L, so no wrap).
template <int R, int DIR, bool DIF, class C>
WB_DEV void rt_bfly(C* p, int es, int base, int m, int j, int ts, const C* tw) {
  C v[R];
#pragma unroll
  for (int q = 0; q < R; ++q) v[q] = p[(base + q * m) * es];
  if (!DIF && j) {
#pragma unroll
    for (int q = 1; q < R; ++q) v[q] = ctw<DIR>(v[q], tw[q * j * ts]);
  }
  rdft<R, DIR>(v);
  if (DIF && j) {
#pragma unroll
    for (int q = 1; q < R; ++q) v[q] = ctw<DIR>(v[q], tw[q * j * ts]);
  }
#pragma unroll
  for (int q = 0; q < R; ++q) p[(base + q * m) * es] = v[q];
}

// nlines lines (line l starts at data + loff(l), element stride es), all
// threads of the CTA; ends with a barrier
template <int DIR, bool DIF, class C, class Off>
WB_DEV void rt_lines(C* data, Off loff, int es, int nlines, const RtPlan& pl, const C* tw) {
  const int n = pl.n;
  int blk = DIF ? n : 1;
  for (int st = 0; st < pl.ns; ++st) {
    const int s = DIF ? st : pl.ns - 1 - st;
    const int R = pl.r[s];
    const int m = DIF ? blk / R : blk;
    const int ts = n / (m * R);
    const int nb = n / R;
    for (int it = threadIdx.x; it < nlines * nb; it += blockDim.x) {
      const int line = it / nb, b = it - line * nb;
      const int bi = b / m, j = b - bi * m;
      C* p = data + loff(line);
      const int base = bi * m * R + j;
      switch (R) {
        case 2: rt_bfly<2, DIR, DIF>(p, es, base, m, j, ts, tw); break;
        case 3: rt_bfly<3, DIR, DIF>(p, es, base, m, j, ts, tw); break;
        case 4: rt_bfly<4, DIR, DIF>(p, es, base, m, j, ts, tw); break;
        case 5: rt_bfly<5, DIR, DIF>(p, es, base, m, j, ts, tw); break;
        case 7: rt_bfly<7, DIR, DIF>(p, es, base, m, j, ts, tw); break;
        default: rt_bfly<8, DIR, DIF>(p, es, base, m, j, ts, tw); break;
      }
    }
    __syncthreads();
    blk = DIF ? m : m * R;
  }
}

struct RtOff {
  int stride;
  WB_DEV int operator()(int l) const { return l * stride; }
};

template <class C>
WB_DEV C* rt_smem() {
  extern __shared__ __align__(16) unsigned char smraw[];
  return reinterpret_cast<C*>(smraw);
}

// ---------------------------------------------------------------------------
// z passes: line side * kRtZsg + i of the work area is that stick of pair q0 + i
// ---------------------------------------------------------------------------
WB_DEV int rt_line(int l) { return (l & 1) * kRtZsg + (l >> 1); }

template <class C>
__global__ void __launch_bounds__(kRtZnt) k_zinv_rt(const C* __restrict__ src, long ld,
                                                    const int2* __restrict__ items, StickTab st, RtGeo g,
                                                    C* __restrict__ out, const int* dn) {
  if (dn && (int)blockIdx.y >= dev_count<true>(dn, 0)) return;
  const int N = g.nz, LS = N | 1;
  C* tw = rt_smem<C>();
  C* zb = tw + N;
  const C* twg = rt_table<C>(g.twz, g.twz32);
  const int q0 = blockIdx.x * kRtZsg, item = blockIdx.y;
  const int nq = min(kRtZsg, st.nsp - q0);
  const int2 it = items[item];
  const C* a = src + (long)it.x * ld;
  const C* b = src + (long)(it.y >= 0 ? it.y : it.x) * ld;
  const bool two = it.y >= 0;
  const int g0 = st.sp_gstart[q0], g1 = st.sp_gstart[q0 + nq];
  for (int i = threadIdx.x; i < N; i += kRtZnt) tw[i] = twg[i];
  for (int i = threadIdx.x; i < 2 * kRtZsg * LS; i += kRtZnt) zb[i] = mkc<C>(0, 0);
  __syncthreads();
  for (int gi = g0 + threadIdx.x; gi < g1; gi += kRtZnt) {
    const int2 qz = st.g_qz[gi];
    const C a1 = a[gi], a2 = two ? b[gi] : mkc<C>(0, 0);
    const C pos = mkc<C>(a1.x - a2.y, a1.y + a2.x);  // a1 + i a2
    const C neg = mkc<C>(a1.x + a2.y, a2.x - a1.y);  // conj(a1 - i a2)
    const int z = qz.y;
    if (qz.x < 2) {  // the (0,0) stick is its own mirror
      if (z != 0) { zb[(z + N) % N] = pos; zb[(N - z) % N] = neg; }
      else zb[0] = neg;  // G = 0: the -G store wins, as in the reference loop
    } else {
      const int l = rt_line(qz.x - 2 * q0);  // its mirror is l ^ kRtZsg
      zb[l * LS + (z + N) % N] = pos;
      zb[(l ^ kRtZsg) * LS + (N - z) % N] = neg;
    }
  }
  __syncthreads();
  rt_lines<+1, true>(zb, RtOff{LS}, 1, 2 * kRtZsg, g.pz, tw);
  C* o = out + (long)item * N * st.nst + q0;
  for (int e = threadIdx.x; e < 2 * kRtZsg * N; e += kRtZnt) {
    const int l = e % (2 * kRtZsg), pz = e / (2 * kRtZsg);
    if (l % kRtZsg < nq) o[(long)pz * st.nst + (l / kRtZsg) * st.hs + l % kRtZsg] = zb[l * LS + pz];
  }
}

template <class C, class Epi>
__global__ void __launch_bounds__(kRtZnt) k_zfwd_rt(const C* __restrict__ sticks, const int2* __restrict__ items,
                                                    StickTab st, RtGeo g, Epi epi, const int* dn) {
  if (dn && (int)blockIdx.y >= dev_count<true>(dn, 0)) return;
  using T = real_t<C>;
  const int N = g.nz, LS = N | 1;
  C* tw = rt_smem<C>();
  C* zb = tw + N;
  const C* twg = rt_table<C>(g.twz, g.twz32);
  const int q0 = blockIdx.x * kRtZsg, item = blockIdx.y;
  const int nq = min(kRtZsg, st.nsp - q0);
  const C* s0 = sticks + (long)item * N * st.nst + q0;
  for (int e = threadIdx.x; e < 2 * kRtZsg * N; e += kRtZnt) {
    const int l = e % (2 * kRtZsg), pz = e / (2 * kRtZsg);
    if (l % kRtZsg < nq) cp_async_elem(zb + l * LS + pz, s0 + (long)pz * st.nst + (l / kRtZsg) * st.hs + l % kRtZsg);
  }
  for (int i = threadIdx.x; i < N; i += kRtZnt) tw[i] = twg[i];
  cp_async_wait_all();
  __syncthreads();
  rt_lines<-1, false>(zb, RtOff{LS}, 1, 2 * kRtZsg, g.pz, tw);
  const int2 it = items[item];
  const int g0 = st.sp_gstart[q0], g1 = st.sp_gstart[q0 + nq];
  for (int gi = g0 + threadIdx.x; gi < g1; gi += kRtZnt) {
    const int2 qz = st.g_qz[gi];
    const typename Epi::Pre pr = epi.pre(gi, it);
    const int z = qz.y;
    C ap, am;
    if (qz.x < 2) {
      ap = zb[(z + N) % N];
      am = zb[(N - z) % N];
    } else {
      const int l = rt_line(qz.x - 2 * q0);
      ap = zb[l * LS + (z + N) % N];
      am = zb[(l ^ kRtZsg) * LS + (N - z) % N];
    }
    const C fp = mkc<C>(T(0.5) * (ap.x + am.x), T(0.5) * (ap.y + am.y));
    const C fm = mkc<C>(T(0.5) * (ap.x - am.x), T(0.5) * (ap.y - am.y));
    epi(gi, it, pr, mkc<C>(fp.x, fm.y), mkc<C>(fp.y, -fm.x));
  }
}

// ---------------------------------------------------------------------------
// x-y passes: half plane H[c][y] (active columns, stride cs) + row scratch
// ---------------------------------------------------------------------------
template <class C>
struct RtPlane {
  C *twx, *twy, *H, *Rb;
  WB_DEV RtPlane(const RtGeo& g) {
    twx = rt_smem<C>();
    twy = twx + g.nx;
    H = twy + g.ny;
    Rb = H + (size_t)g.ncols * g.cs;
  }
  WB_DEV void load_tw(const RtGeo& g) const {
    const C* tx = rt_table<C>(g.twx, g.twx32);
    const C* ty = rt_table<C>(g.twy, g.twy32);
    for (int i = threadIdx.x; i < g.nx; i += blockDim.x) twx[i] = tx[i];
    for (int i = threadIdx.x; i < g.ny; i += blockDim.x) twy[i] = ty[i];
  }
  // sticks -> H (zero elsewhere), then the inverse column transforms
  WB_DEV void sticks_in(const RtGeo& g, const StickTab& st, const C* __restrict__ sz) const {
    for (int e = threadIdx.x; e < g.ncols * g.cs; e += blockDim.x) H[e] = mkc<C>(0, 0);
    __syncthreads();
    for (int s = threadIdx.x; s < st.nst; s += blockDim.x) {
      const int p = g.spos[s];
      if (p >= 0) H[p] = sz[s];
    }
    __syncthreads();
    rt_lines<+1, true>(H, RtOff{g.cs}, 1, g.ncols, g.py, twy);
  }
  // forward column transforms, then H -> sticks
  WB_DEV void sticks_out(const RtGeo& g, const StickTab& st, C* __restrict__ sz) const {
    rt_lines<-1, false>(H, RtOff{g.cs}, 1, g.ncols, g.py, twy);
    for (int s = threadIdx.x; s < st.nst; s += blockDim.x) {
      const int p = g.spos[s];
      sz[s] = p >= 0 ? H[p] : mkc<C>(0, 0);
    }
  }
  // rows [y0, y0 + nr) of H -> Rb (full rows, zero at inactive x), inverse row transforms
  WB_DEV void rows_in(const RtGeo& g, int y0, int nr) const {
    for (int e = threadIdx.x; e < nr * g.nx; e += blockDim.x) Rb[e] = mkc<C>(0, 0);
    __syncthreads();
    for (int e = threadIdx.x; e < nr * g.ncols; e += blockDim.x) {
      const int r = e / g.ncols, c = e - r * g.ncols;
      Rb[r * g.nx + __ldg(g.colx + c)] = H[c * g.cs + y0 + r];
    }
    __syncthreads();
    rt_lines<+1, true>(Rb, RtOff{g.nx}, 1, nr, g.px, twx);
  }
  // forward row transforms of Rb, active columns back into H rows [y0, y0 + nr)
  WB_DEV void rows_out(const RtGeo& g, int y0, int nr) const {
    rt_lines<-1, false>(Rb, RtOff{g.nx}, 1, nr, g.px, twx);
    for (int e = threadIdx.x; e < nr * g.ncols; e += blockDim.x) {
      const int r = e / g.ncols, c = e - r * g.ncols;
      H[c * g.cs + y0 + r] = Rb[r * g.nx + __ldg(g.colx + c)];
    }
    __syncthreads();
  }
};

// psi -> V(r) psi(r) -> back, in place on the sticks of plane pz of item
template <class C>
__global__ void __launch_bounds__(kRtPnt) k_plane_vloc_rt(C* __restrict__ sticks, StickTab st, RtGeo g,
                                                          const real_t<C>* __restrict__ vs, int rc, const int* dn) {
  if (dn && (int)blockIdx.y >= dev_count<true>(dn, 0)) return;
  const RtPlane<C> P(g);
  const int pz = blockIdx.x, item = blockIdx.y;
  C* sz = sticks + ((long)item * g.nz + pz) * st.nst;
  P.load_tw(g);
  P.sticks_in(g, st, sz);
  const real_t<C>* vz = vs + (long)pz * g.nx * g.ny;
  for (int y0 = 0; y0 < g.ny; y0 += rc) {
    const int nr = min(rc, g.ny - y0);
    P.rows_in(g, y0, nr);
    for (int e = threadIdx.x; e < nr * g.nx; e += blockDim.x) P.Rb[e] = cscale(P.Rb[e], vz[(long)y0 * g.nx + e]);
    __syncthreads();
    P.rows_out(g, y0, nr);
  }
  P.sticks_out(g, st, sz);
}

// sticks -> real-space box (permuted layout), no scaling
__global__ void __launch_bounds__(kRtPnt) k_plane_inv_box_rt(const double2* __restrict__ sticks, StickTab st,
                                                             RtGeo g, double2* __restrict__ box, int rc) {
  const RtPlane<double2> P(g);
  const int pz = blockIdx.x, item = blockIdx.y;
  P.load_tw(g);
  P.sticks_in(g, st, sticks + ((long)item * g.nz + pz) * st.nst);
  double2* o = box + ((long)item * g.nz + pz) * g.nx * g.ny;
  for (int y0 = 0; y0 < g.ny; y0 += rc) {
    const int nr = min(rc, g.ny - y0);
    P.rows_in(g, y0, nr);
    for (int e = threadIdx.x; e < nr * g.nx; e += blockDim.x) o[(long)y0 * g.nx + e] = P.Rb[e];
    __syncthreads();
  }
}

// RHS (dfpt_module.f90:245-260): (psi_v1 + i psi_v2)(r) dv_p(r) / N -> forward
// -> sticks, one CTA per (plane, perturbation) over the band pairs
__global__ void __launch_bounds__(kRtPnt) k_plane_rhs_rt(const double2* __restrict__ evcr,
                                                         const double2* __restrict__ dvbox, int npv, StickTab st,
                                                         RtGeo g, double2* __restrict__ sticks, int rc) {
  const RtPlane<double2> P(g);
  const int pz = blockIdx.x, p = blockIdx.y;
  const long plane = (long)g.nx * g.ny;
  const double inv = 1.0 / ((double)plane * g.nz);
  const double2* dv = dvbox + ((long)(p >> 1) * g.nz + pz) * plane;
  const bool hi = p & 1;
  P.load_tw(g);
  for (int k = 0; k < npv; ++k) {
    const double2* ps = evcr + ((long)k * g.nz + pz) * plane;
    for (int y0 = 0; y0 < g.ny; y0 += rc) {
      const int nr = min(rc, g.ny - y0);
      for (int e = threadIdx.x; e < nr * g.nx; e += blockDim.x) {
        const long o = (long)y0 * g.nx + e;
        const double2 d = dv[o];
        P.Rb[e] = cscale(ps[o], (hi ? d.y : d.x) * inv);
      }
      __syncthreads();
      P.rows_out(g, y0, nr);
    }
    const long item = (long)p * npv + k;
    P.sticks_out(g, st, sticks + (item * g.nz + pz) * st.nst);
    __syncthreads();
  }
}

// density response (dfpt_module.f90:403-423, :478): drho_p = sum_v occ_v
// psi_v(r) dpsi_v(r) for the two perturbations of pair pp, accumulated in the
// CTA's own slice of acc (one element per thread throughout), then
// (drho_p1 + i drho_p2) scale -> forward -> sticks
__global__ void __launch_bounds__(kRtPnt, 1) k_plane_drho_rt(const double2* __restrict__ dsticks,
                                                          const double2* __restrict__ evcr,
                                                          const double* __restrict__ occ, int nocc, int mb,
                                                          StickTab st, RtGeo g, double2* __restrict__ acc,
                                                          double scale, double2* __restrict__ osticks, int rc) {
  const RtPlane<double2> P(g);
  const int pz = blockIdx.x, pp = blockIdx.y;
  const int npv = (nocc + 1) / 2;
  const long plane = (long)g.nx * g.ny;
  double2* ac = acc + ((long)pp * g.nz + pz) * plane;
  P.load_tw(g);
  for (int pi = 0; pi < 2; ++pi) {
    const int p = 2 * pp + pi;
    if (p >= mb) {  // odd batch: the second density of the last pair is zero
      for (long e = threadIdx.x; e < plane; e += blockDim.x) ac[e].y = 0.0;
      continue;
    }
    for (int k = 0; k < npv; ++k) {
      const long item = (long)p * npv + k;
      P.sticks_in(g, st, dsticks + (item * g.nz + pz) * st.nst);
      const double o1 = occ[2 * k];
      const double o2 = (2 * k + 1 < nocc) ? occ[2 * k + 1] : 0.0;
      const double2* ps = evcr + ((long)k * g.nz + pz) * plane;
      for (int y0 = 0; y0 < g.ny; y0 += rc) {
        const int nr = min(rc, g.ny - y0);
        P.rows_in(g, y0, nr);
        for (int e = threadIdx.x; e < nr * g.nx; e += blockDim.x) {
          const long o = (long)y0 * g.nx + e;
          const double2 d = P.Rb[e], s = ps[o];
          const double v = fma(o1 * s.x, d.x, o2 * s.y * d.y);
          double* a = pi ? &ac[o].y : &ac[o].x;
          *a = (k == 0) ? v : *a + v;
        }
        __syncthreads();
      }
    }
  }
  __syncthreads();
  for (int y0 = 0; y0 < g.ny; y0 += rc) {
    const int nr = min(rc, g.ny - y0);
    for (int e = threadIdx.x; e < nr * g.nx; e += blockDim.x) {
      const double2 a = ac[(long)y0 * g.nx + e];
      P.Rb[e] = make_double2(a.x * scale, a.y * scale);
    }
    __syncthreads();
    P.rows_out(g, y0, nr);
  }
  P.sticks_out(g, st, osticks + ((long)pp * g.nz + pz) * st.nst);
}

// ---------------------------------------------------------------------------
// x-y passes by the phases of wb_plane.cuh, radices dispatched per phase
// ---------------------------------------------------------------------------
// The edge's split: both radices in the list, the larger first, as even as
// possible (fewer points per thread leave more threads per SM).
static bool rt_radix(int r) {
  for (int q : {3, 4, 5, 6, 7, 8, 9, 10, 12, 15, 16})
    if (q == r) return true;
  return false;
}
void rt_split(int n, int* a, int* b) {
  *a = *b = 0;
  for (int q = 3; q * q <= n; ++q)
    if (n % q == 0 && rt_radix(q) && rt_radix(n / q)) { *a = n / q; *b = q; }
}
static size_t rt_fast_smem(int nx, int ny, size_t elem) { return elem * (size_t)ny * (nx | 1); }
bool rt_fast_setup(int nx, int ny, RtFast* f) {
  if (nx > kRtMaxEdge || ny > kRtMaxEdge || rt_fast_smem(nx, ny, 16) > 227u * 1024u) return false;
  rt_split(nx, &f->ax, &f->bx);
  rt_split(ny, &f->ay, &f->by);
  if (!f->ax || !f->ay) return false;
  f->max_radix = std::max(std::max(f->ax, f->bx), std::max(f->ay, f->by));
  auto fill = [](int n, int b, double2* t, float2* t32) {
    for (int i = 0; i < n; ++i) {
      const long double w = 2.0L * 3.14159265358979323846264338327950288L * (long double)((i / b) * (i % b) % n) / n;
      t[i] = make_double2((double)cosl(w), (double)sinl(w));
      t32[i] = make_float2((float)t[i].x, (float)t[i].y);
    }
  };
  fill(nx, f->bx, f->tx, f->tx32);
  fill(ny, f->by, f->ty, f->ty32);
  return true;
}

template <class C>
struct RtTw {
  C x[kRtMaxEdge], y[kRtMaxEdge];
};
// one dimension's step factors in the constant bank
template <class C, bool Y>
struct RtTwOf {
  const RtTw<C>& t;
  WB_DEV C operator()(int i) const { return Y ? t.y[i] : t.x[i]; }
};
template <int R> struct Radix { static constexpr int value = R; };
// f(Radix<r>) for the run-time radix r <= MAXR (uniform over the CTA)
template <int MAXR, class F>
WB_DEV void with_radix(int r, F f) {
  switch (r) {
    case 3: f(Radix<3>{}); break;
    case 4: f(Radix<4>{}); break;
    case 5: f(Radix<5>{}); break;
    case 6: f(Radix<6>{}); break;
    case 7: f(Radix<7>{}); break;
    case 8: f(Radix<8>{}); break;
    case 9: f(Radix<9>{}); break;
    case 10: f(Radix<10>{}); break;
    default:
      if constexpr (MAXR > 10) {
        if (r == 12) f(Radix<12>{});
        else if (r == 15) f(Radix<15>{});
        else f(Radix<16>{});
      }
  }
}
#define WB_RADIX(r, call) with_radix<MAXR>(r, [&](auto radix_) { constexpr int R = decltype(radix_)::value; call; })

template <int MAXR, class C>
WB_DEV void rtf_inverse(C* pl, const RtTw<C>& tw, const C* sz, const StickTab& st, const RPlane& g) {
  const int nt = blockDim.x;
  const RtTwOf<C, false> tx{tw};
  const RtTwOf<C, true> ty{tw};
  WB_RADIX(g.ay_, (plane_col_in<R>(pl, ty, sz, st.cmap, g, nt)));
  __syncthreads();
  WB_RADIX(g.by_, (plane_col_mid_inv<R>(pl, g, nt)));
  __syncthreads();
  WB_RADIX(g.ax_, (plane_row_in<R>(pl, tx, g, nt)));
  __syncthreads();
}
template <int MAXR, class C>
WB_DEV void rtf_forward(C* pl, const RtTw<C>& tw, C* sz, const StickTab& st, const RPlane& g) {
  const int nt = blockDim.x;
  const RtTwOf<C, true> ty{tw};
  __syncthreads();
  WB_RADIX(g.ax_, (plane_row_out<R>(pl, g, nt)));
  __syncthreads();
  WB_RADIX(g.by_, (plane_col_mid_fwd<R>(pl, ty, g, nt)));
  __syncthreads();
  WB_RADIX(g.ay_, (plane_col_out<R>(pl, sz, st.cmap, g, nt)));
}

// Two builds of each kernel.  Radices up to 10 and planes of which three or more
// fit an SM: 80 registers, blocks of 192 threads where four planes fit (45 x 54:
// 1.24 us per FP64 item against 1.32 with three of 256 and 1.52 with two), else of
// 256.  The others: 128 registers, two blocks of 256 or one of 512.
template <int MAXR>
constexpr int rtf_max_threads() { return MAXR <= 10 ? 256 : 512; }
template <int MAXR>
constexpr int rtf_blocks() { return MAXR <= 10 ? 3 : 1; }
struct RtfShape {
  bool small;
  int threads;
};
static RtfShape rtf_shape(const RtGeo& g, size_t elem) {
  const int fit = (int)(227u * 1024u / (rt_fast_smem(g.nx, g.ny, elem) + 1024));
  const bool small = g.fast->max_radix <= 10 && fit >= 3;
  return {small, small ? (fit >= 4 ? 192 : 256) : (fit >= 2 ? 256 : 512)};
}

// psi -> V(r) psi(r) / N -> back, in place on the sticks of plane pz of item
template <int MAXR, class C>
__global__ void __launch_bounds__(rtf_max_threads<MAXR>(), rtf_blocks<MAXR>()) k_plane_vloc_rtf(
    C* __restrict__ sticks, StickTab st, const __grid_constant__ RPlane g, const real_t<C>* __restrict__ vs,
    const __grid_constant__ RtTw<C> tw, const int* dn) {
  if (dn && (int)blockIdx.y >= dev_count<true>(dn, 0)) return;
  C* pl = rt_smem<C>();
  const int nt = blockDim.x;
  C* sz = sticks + ((long)blockIdx.y * gridDim.x + blockIdx.x) * st.nst;
  const RtTwOf<C, false> tx{tw};
  rtf_inverse<MAXR>(pl, tw, sz, st, g);
  WB_RADIX(g.bx_, (plane_row_vloc<R>(pl, tx, vs + (long)blockIdx.x * g.nx_ * g.ny_, g, nt)));
  rtf_forward<MAXR>(pl, tw, sz, st, g);
}

// sticks -> real-space box, no scaling
template <int MAXR>
__global__ void __launch_bounds__(rtf_max_threads<MAXR>(), rtf_blocks<MAXR>()) k_plane_inv_box_rtf(
    const double2* __restrict__ sticks, StickTab st, const __grid_constant__ RPlane g, double2* __restrict__ box,
    const __grid_constant__ RtTw<double2> tw) {
  double2* pl = rt_smem<double2>();
  const long plane = (long)blockIdx.y * gridDim.x + blockIdx.x;
  rtf_inverse<MAXR>(pl, tw, sticks + plane * st.nst, st, g);
  WB_RADIX(g.bx_, (plane_row_box<R>(pl, box + plane * g.nx_ * g.ny_, g, (int)blockDim.x)));
}

// RHS (dfpt_module.f90:245-260), one CTA per (plane, perturbation, band pair)
template <int MAXR>
__global__ void __launch_bounds__(rtf_max_threads<MAXR>(), rtf_blocks<MAXR>()) k_plane_rhs_rtf(
    const double2* __restrict__ evcr, const double2* __restrict__ dvbox, int npv, StickTab st,
    const __grid_constant__ RPlane g, double2* __restrict__ sticks, const __grid_constant__ RtTw<double2> tw) {
  double2* pl = rt_smem<double2>();
  const int pz = blockIdx.x, nz = gridDim.x, p = blockIdx.y, nt = blockDim.x;
  const long plane = (long)g.nx_ * g.ny_;
  const double inv = 1.0 / ((double)plane * nz);
  const double2* dv = dvbox + ((long)(p >> 1) * nz + pz) * plane;
  const RtTwOf<double2, false> tx{tw};
  for (int k = 0; k < npv; ++k) {
    __syncthreads();  // the previous band pair's column pass is done with the plane
    WB_RADIX(g.bx_, (plane_row_rhs<R>(pl, tx, evcr + ((long)k * nz + pz) * plane, dv, (p & 1) != 0, inv, g, nt)));
    rtf_forward<MAXR>(pl, tw, sticks + (((long)p * npv + k) * nz + pz) * st.nst, st, g);
  }
}

// density response (dfpt_module.f90:403-423, :478) of the perturbations 2 pp and
// 2 pp + 1, summed over the bands in the CTA's own slice of acc
template <int MAXR>
__global__ void __launch_bounds__(rtf_max_threads<MAXR>(), rtf_blocks<MAXR>()) k_plane_drho_rtf(
    const double2* __restrict__ dsticks, const double2* __restrict__ evcr, const double* __restrict__ occ, int nocc,
    int mb, StickTab st, const __grid_constant__ RPlane g, double2* __restrict__ acc, double scale,
    double2* __restrict__ osticks, const __grid_constant__ RtTw<double2> tw) {
  double2* pl = rt_smem<double2>();
  const int pz = blockIdx.x, nz = gridDim.x, pp = blockIdx.y, nt = blockDim.x;
  const int npv = (nocc + 1) / 2;
  const long plane = (long)g.nx_ * g.ny_;
  double* sum = reinterpret_cast<double*>(acc + ((long)pp * nz + pz) * plane);
  const RtTwOf<double2, false> tx{tw};
  for (int p = 2 * pp; p < min(mb, 2 * pp + 2); ++p)
    for (int k = 0; k < npv; ++k) {
      __syncthreads();
      rtf_inverse<MAXR>(pl, tw, dsticks + (((long)p * npv + k) * nz + pz) * st.nst, st, g);
      const double o1 = occ[2 * k], o2 = (2 * k + 1 < nocc) ? occ[2 * k + 1] : 0.0;
      WB_RADIX(g.bx_, (plane_row_density<R>(pl, evcr + ((long)k * nz + pz) * plane, sum + (p & 1) * plane, o1, o2,
                                            k == 0, g, nt)));
    }
  __syncthreads();
  // an odd batch: the second density of the last pair is zero
  WB_RADIX(g.bx_, (plane_row_pair<R>(pl, tx, sum, 2 * pp + 1 < mb ? sum + plane : nullptr, scale, g, nt)));
  rtf_forward<MAXR>(pl, tw, osticks + ((long)pp * nz + pz) * st.nst, st, g);
}

static RPlane rtf_plane(const RtGeo& g, const StickTab& st) {
  const RtFast& f = *g.fast;
  auto magic = [](int d) { return (unsigned)((0x100000000ull + d - 1) / d); };
  return RPlane{g.nx, g.ny, f.ax, f.bx, f.ay, f.by, st.ncols, st.xhi + 1, magic(st.ncols), magic(g.ny)};
}
template <class C>
static RtTw<C> rtf_tw(const RtGeo& g) {
  RtTw<C> t;
  for (int i = 0; i < kRtMaxEdge; ++i) {
    if constexpr (sizeof(C) == 16) { t.x[i] = g.fast->tx[i]; t.y[i] = g.fast->ty[i]; }
    else { t.x[i] = g.fast->tx32[i]; t.y[i] = g.fast->ty32[i]; }
  }
  return t;
}
// ---------------------------------------------------------------------------
// epilogues of the forward z pass (the same operations as wb_fft_kernels.cu's)
// ---------------------------------------------------------------------------
struct RtEpiStore {
  double2* dst;
  long ld;
  struct Pre {};
  WB_DEV Pre pre(int, int2) const { return {}; }
  WB_DEV void operator()(int gi, int2 it, const Pre&, double2 b1, double2 b2) const {
    dst[(long)it.x * ld + gi] = b1;
    if (it.y >= 0) dst[(long)it.y * ld + gi] = b2;
  }
};

// T = (V psi + g2kin psi with Im(G=0) = 0) - e psi
template <class C>
struct RtEpiHpsi {
  using T = real_t<C>;
  const C* P;
  C* Tv;
  long ld;
  const T* g2kin;
  const T* ecol;
  struct Pre {
    C p1, p2;
    T k;
  };
  WB_DEV Pre pre(int gi, int2 it) const {
    Pre r;
    r.p1 = P[(long)it.x * ld + gi];
    r.p2 = it.y >= 0 ? P[(long)it.y * ld + gi] : mkc<C>(0, 0);
    r.k = g2kin[gi];
    return r;
  }
  WB_DEV void one(int gi, int c, C p, T k, C vp) const {
    C h = mkc<C>(fma(k, p.x, vp.x), fma(k, p.y, vp.y));
    if (gi == 0) h.y = T(0);
    const T e = ecol[c];
    Tv[(long)c * ld + gi] = mkc<C>(fma(-e, p.x, h.x), fma(-e, p.y, h.y));
  }
  WB_DEV void operator()(int gi, int2 it, const Pre& pr, C b1, C b2) const {
    one(gi, it.x, pr.p1, pr.k, b1);
    if (it.y >= 0) one(gi, it.y, pr.p2, pr.k, b2);
  }
};

// dng(perm(g), p) = sqvc(g) drho_G(g), G = 0 zeroed
struct RtEpiDng {
  double2* dng;
  long ld;
  const int* perm;
  const double* sqvc;
  struct Pre {
    double s;
    int r;
  };
  WB_DEV Pre pre(int gi, int2) const { return {(gi == 0) ? 0.0 : sqvc[gi], perm[gi]}; }
  WB_DEV void operator()(int, int2 it, const Pre& pr, double2 b1, double2 b2) const {
    const long r = pr.r;
    dng[(long)it.x * ld + r] = make_double2(pr.s * b1.x, pr.s * b1.y);
    if (it.y >= 0) dng[(long)it.y * ld + r] = make_double2(pr.s * b2.x, pr.s * b2.y);
  }
};

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
template <class C>
static size_t rt_zsmem(const RtGeo& g) { return sizeof(C) * (g.nz + 2 * kRtZsg * (g.nz | 1)); }
static dim3 rt_zgrid(const StickTab& st, int nitems) { return dim3((st.nsp + kRtZsg - 1) / kRtZsg, nitems); }

// The kernels serve contexts of several boxes, so each is opted in to all the
// shared memory a CTA can have rather than to one box's size.
constexpr int kRtMaxSmem = 227 * 1024;
template <class... K>
static void opt_in(K*... k) {
  (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kRtMaxSmem), ...);
}
template <int MAXR>
static void rtf_setup() {
  opt_in(k_plane_vloc_rtf<MAXR, double2>, k_plane_vloc_rtf<MAXR, float2>, k_plane_inv_box_rtf<MAXR>,
         k_plane_rhs_rtf<MAXR>, k_plane_drho_rtf<MAXR>);
}
void rt_setup() {
  opt_in(k_zinv_rt<double2>, k_zinv_rt<float2>, k_zfwd_rt<double2, RtEpiStore>, k_zfwd_rt<double2, RtEpiHpsi<double2>>,
         k_zfwd_rt<float2, RtEpiHpsi<float2>>, k_zfwd_rt<double2, RtEpiDng>, k_plane_vloc_rt<double2>,
         k_plane_vloc_rt<float2>, k_plane_inv_box_rt, k_plane_rhs_rt, k_plane_drho_rt);
  rtf_setup<10>();
  rtf_setup<16>();
}

template <class C, class F>
static void zinv_rt_t(const F& f, const C* src, long ld, const int2* items, int nitems, C* sticks) {
  if (nitems <= 0) return;
  k_zinv_rt<C><<<rt_zgrid(f.st, nitems), kRtZnt, rt_zsmem<C>(*f.rt), f.stream>>>(src, ld, items, f.st, *f.rt,
                                                                                  sticks, f.dcount);
}
template <class C, class F, class Epi>
static void zfwd_rt_t(const F& f, const C* sticks, const int2* items, int nitems, Epi epi) {
  if (nitems <= 0) return;
  k_zfwd_rt<C, Epi><<<rt_zgrid(f.st, nitems), kRtZnt, rt_zsmem<C>(*f.rt), f.stream>>>(sticks, items, f.st, *f.rt,
                                                                                      epi, f.dcount);
}
template <class C, class F>
static void vloc_rt_t(const F& f, C* sticks, int nitems, const real_t<C>* vs) {
  if (nitems <= 0) return;
  if (f.rt->fast) {
    const RtfShape sh = rtf_shape(*f.rt, sizeof(C));
    auto k = sh.small ? k_plane_vloc_rtf<10, C> : k_plane_vloc_rtf<16, C>;
    k<<<dim3(f.rt->nz, nitems), sh.threads, rt_fast_smem(f.rt->nx, f.rt->ny, sizeof(C)), f.stream>>>(
        sticks, f.st, rtf_plane(*f.rt, f.st), vs, rtf_tw<C>(*f.rt), f.dcount);
    return;
  }
  int rc = 1;
  const size_t sm = rt_plane_smem(*f.rt, sizeof(C), &rc);
  k_plane_vloc_rt<C><<<dim3(f.rt->nz, nitems), kRtPnt, sm, f.stream>>>(sticks, f.st, *f.rt, vs, rc, f.dcount);
}

void rt_zinv(const FftArgs& f, const double2* src, long ld, const int2* items, int nitems, double2* sticks) {
  zinv_rt_t<double2>(f, src, ld, items, nitems, sticks);
}
void rt_zinv32(const FftArgs32& f, const float2* src, long ld, const int2* items, int nitems, float2* sticks) {
  zinv_rt_t<float2>(f, src, ld, items, nitems, sticks);
}
void rt_zfwd_store(const FftArgs& f, const double2* sticks, const int2* items, int nitems, double2* dst, long ld) {
  zfwd_rt_t<double2>(f, sticks, items, nitems, RtEpiStore{dst, ld});
}
void rt_zfwd_hpsi(const FftArgs& f, const double2* sticks, const int2* items, int nitems, const double2* P,
                  double2* T, long ld, const double* g2kin, const double* ecol) {
  zfwd_rt_t<double2>(f, sticks, items, nitems, RtEpiHpsi<double2>{P, T, ld, g2kin, ecol});
}
void rt_zfwd_hpsi32(const FftArgs32& f, const float2* sticks, const int2* items, int nitems, const float2* P,
                    float2* T, long ld, const float* g2kin, const float* ecol) {
  zfwd_rt_t<float2>(f, sticks, items, nitems, RtEpiHpsi<float2>{P, T, ld, g2kin, ecol});
}
void rt_zfwd_dng(const FftArgs& f, const double2* sticks, const int2* items, int nitems, double2* dng, long ld,
                 const int* perm, const double* sqvc) {
  zfwd_rt_t<double2>(f, sticks, items, nitems, RtEpiDng{dng, ld, perm, sqvc});
}
void rt_plane_vloc(const FftArgs& f, double2* sticks, int nitems, const double* vs) {
  vloc_rt_t<double2>(f, sticks, nitems, vs);
}
void rt_plane_vloc32(const FftArgs32& f, float2* sticks, int nitems, const float* vs) {
  vloc_rt_t<float2>(f, sticks, nitems, vs);
}
void rt_plane_inv_box(const FftArgs& f, const double2* sticks, int nitems, double2* box) {
  if (nitems <= 0) return;
  if (f.rt->fast) {
    const RtfShape sh = rtf_shape(*f.rt, 16);
    auto k = sh.small ? k_plane_inv_box_rtf<10> : k_plane_inv_box_rtf<16>;
    k<<<dim3(f.rt->nz, nitems), sh.threads, rt_fast_smem(f.rt->nx, f.rt->ny, 16), f.stream>>>(
        sticks, f.st, rtf_plane(*f.rt, f.st), box, rtf_tw<double2>(*f.rt));
    return;
  }
  int rc = 1;
  const size_t sm = rt_plane_smem(*f.rt, 16, &rc);
  k_plane_inv_box_rt<<<dim3(f.rt->nz, nitems), kRtPnt, sm, f.stream>>>(sticks, f.st, *f.rt, box, rc);
}
void rt_plane_rhs(const FftArgs& f, const double2* evcr, const double2* dvbox, int npv, int mb, double2* sticks) {
  if (mb <= 0) return;
  if (f.rt->fast) {
    const RtfShape sh = rtf_shape(*f.rt, 16);
    auto k = sh.small ? k_plane_rhs_rtf<10> : k_plane_rhs_rtf<16>;
    k<<<dim3(f.rt->nz, mb), sh.threads, rt_fast_smem(f.rt->nx, f.rt->ny, 16), f.stream>>>(
        evcr, dvbox, npv, f.st, rtf_plane(*f.rt, f.st), sticks, rtf_tw<double2>(*f.rt));
    return;
  }
  int rc = 1;
  const size_t sm = rt_plane_smem(*f.rt, 16, &rc);
  k_plane_rhs_rt<<<dim3(f.rt->nz, mb), kRtPnt, sm, f.stream>>>(evcr, dvbox, npv, f.st, *f.rt, sticks, rc);
}
void rt_plane_drho(const FftArgs& f, const double2* dsticks, const double2* evcr, const double* occ, int nocc,
                   int mb, double2* acc, double scale, double2* osticks) {
  if (mb <= 0) return;
  if (f.rt->fast) {
    const RtfShape sh = rtf_shape(*f.rt, 16);
    auto k = sh.small ? k_plane_drho_rtf<10> : k_plane_drho_rtf<16>;
    k<<<dim3(f.rt->nz, (mb + 1) / 2), sh.threads, rt_fast_smem(f.rt->nx, f.rt->ny, 16), f.stream>>>(
        dsticks, evcr, occ, nocc, mb, f.st, rtf_plane(*f.rt, f.st), acc, scale, osticks, rtf_tw<double2>(*f.rt));
    return;
  }
  int rc = 1;
  const size_t sm = rt_plane_smem(*f.rt, 16, &rc);
  k_plane_drho_rt<<<dim3(f.rt->nz, (mb + 1) / 2), kRtPnt, sm, f.stream>>>(dsticks, evcr, occ, nocc, mb, f.st,
                                                                          *f.rt, acc, scale, osticks, rc);
}

}  // namespace wb
