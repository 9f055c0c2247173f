// Stick-and-plane 3D FFTs of the Gamma-only response operator.
//
// The G sphere is cut into sticks along z.  A "stick pair" is the stick at
// (x, y) of the stored half sphere together with its mirror at (-x, -y), which
// holds the -G partners; the (0,0) stick is its own mirror.  Inside the
// library G vectors are ordered stick pair by stick pair, z ascending, so
// every stick pair reads one contiguous run of coefficients.
//
// One complex 3D FFT carries two real functions (FFT_kernel/fft_at_gamma.f90):
//   inverse: box(+G) = a1 + i a2, box(-G) = conj(a1 - i a2)          (:55-64)
//   forward: fp = (A(G) + A(-G))/2, fm = (A(G) - A(-G))/2,
//            b1 = (Re fp, Im fm), b2 = (Im fp, -Re fm)                 (:98-111)
// Both are fused into the z-pass kernels.  The x-y passes run one plane per
// CTA in shared memory, with the pointwise work of the caller (local
// potential, RHS product, density accumulation) fused between the inverse and
// forward transforms.
//
// Stick buffer layout: [item][z][side][pair], sides hs sticks apart: stick
// side * hs + q is the stored (side 0) or mirrored (side 1) stick of pair q, the
// pairs in (y, x) order, so that sticks next to each other in x are neighbours
// in memory for the column passes; the mirror slot of (0,0) and the sticks that
// round hs up are dummies.  g_qz of a stored G is (2q + side, z), side = which
// of the two sticks of the pair holds it.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "wb_internal.h"
#include "wb_plane.cuh"

namespace wb {

// z passes: 8 stick pairs per CTA of 128 threads (measured against 16/256 and
// 4/64 at 64^3: more, smaller CTAs overlap one CTA's loads with another's
// transform and stores; zfwd 0.30 instead of 0.34 us per FP64 item)
constexpr int ZSG = 8;
constexpr int ZNT = 128;

// step-1 factor table of a line (wb_fft.cuh) into shared memory
template <int N, class C>
WB_DEV void load_tw(C* tw, const C* twg) {
  for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = twg[i];
}

// ---------------------------------------------------------------------------
// z pass, inverse: sphere coefficients of a pair of columns -> sticks
// ---------------------------------------------------------------------------
// One unit = stick pairs [ZSG qg, ZSG qg + ZSG) of band-pair item `item`.
// Shared memory of every unit: the twiddles (N), then the work area.
// Line side * ZSG + i of the work area is that stick of pair q0 + i.  A unit
// takes its pointers from the dynamic shared array itself so that a unit body
// compiled as a separate function still addresses shared memory directly.
template <class C>
WB_DEV C* smem_tw() {
  extern __shared__ __align__(16) unsigned char smraw[];
  return reinterpret_cast<C*>(smraw);
}

// Twiddles of one thread, held in registers so that their global loads are
// issued with the unit's other loads and stored to shared memory after the zero
// fill.
template <int N, class C>
struct TwRegs {
  static constexpr int PER = (N + ZNT - 1) / ZNT;
  C v[PER];
  WB_DEV void load(const C* __restrict__ twg) {
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int i = threadIdx.x + ZNT * k;
      if (i < N) v[k] = twg[i];
    }
  }
  WB_DEV void store(C* tw) const {
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int i = threadIdx.x + ZNT * k;
      if (i < N) tw[i] = v[k];
    }
  }
};

// G coefficients prefetched per thread before the zero fill (the rest of a
// stick group's G vectors, if any, are read in a second loop).
constexpr int kZPre = 2;

static_assert((ZSG & (ZSG - 1)) == 0, "z_line's mirror flips one bit");
// line of pair-and-side 2 i + side of a stick group
WB_DEV int z_line(int l) { return (l & 1) * ZSG + (l >> 1); }

template <int N, bool PR, class C>
__global__ void __launch_bounds__(ZNT) k_zinv(const C* __restrict__ src, long ld,
                                              const int2* __restrict__ items, StickTab st,
                                              C* __restrict__ out,
                                              const C* __restrict__ twg, const int* dn) {
  if (dn && (int)blockIdx.y >= dev_count<true>(dn, 0)) return;  // beyond the device item count
  constexpr int LS = LinePad<N>::LEN | 1;  // odd line stride: conflict-free transposes
  using LP = LinePad<N>;
  C* tw = smem_tw<C>();
  C* zb = smem_tw<C>() + N;
  const int qg = blockIdx.x, item = blockIdx.y;
  const int q0 = qg * ZSG;
  const int nq = min(ZSG, st.nsp - q0);
  const int2 it = items[item];
  const C* a = src + (long)it.x * ld;
  const C* b = src + (long)(it.y >= 0 ? it.y : it.x) * ld;
  const bool two = it.y >= 0;
  const int g0 = st.sp_gstart[q0], g1 = st.sp_gstart[q0 + nq];
  TwRegs<N, C> twr;
  twr.load(twg);
  C pa[kZPre], pb[kZPre];
  int2 pq[kZPre];
#pragma unroll
  for (int k = 0; k < kZPre; ++k) {
    const int g = g0 + threadIdx.x + k * ZNT;
    if (g < g1) {
      pq[k] = st.g_qz[g];
      pa[k] = a[g];
      pb[k] = two ? b[g] : mkc<C>(0, 0);
    }
  }
  // zero what step 1 reads: with pruning only the live inputs (the sphere's z
  // lie in the outer quarters), otherwise the whole lines
  if constexpr (PR && Prune<N>::IN_OK) {
    constexpr int N1 = FftSplit<N>::N1, N2 = FftSplit<N>::N2, NLIVE = N1 / 2;
    for (int e = threadIdx.x; e < 2 * ZSG * NLIVE * N2; e += ZNT) {
      const int l = e / (NLIVE * N2), r = e % (NLIVE * N2);
      const int h = r / N2, n2 = r % N2;
      const int n1 = h < NLIVE / 2 ? h : N1 - NLIVE + h;
      zb[l * LS + LP::off_blk(n1, n2)] = mkc<C>(0, 0);
    }
  } else {
    for (int i = threadIdx.x; i < 2 * ZSG * LS; i += ZNT) zb[i] = mkc<C>(0, 0);
  }
  twr.store(tw);
  __syncthreads();
  auto put = [&](int2 qz, C a1, C a2) {
    // pos = a1 + i a2 ; neg = conj(a1 - i a2)
    const C pos = mkc<C>(a1.x - a2.y, a1.y + a2.x);
    const C neg = mkc<C>(a1.x + a2.y, a2.x - a1.y);
    const int z = qz.y;
    if (qz.x < 2) {  // the (0,0) stick is its own mirror
      if (z != 0) { zb[LP::off((z + N) % N)] = pos; zb[LP::off((N - z) % N)] = neg; }
      else zb[0] = neg;  // G = 0: the -G store wins, as in the reference loop
    } else {
      const int l = z_line(qz.x - 2 * q0);  // line of the stick holding G; its mirror is l ^ ZSG
      zb[l * LS + LP::off((z + N) % N)] = pos;
      zb[(l ^ ZSG) * LS + LP::off((N - z) % N)] = neg;
    }
  };
#pragma unroll
  for (int k = 0; k < kZPre; ++k)
    if (g0 + (int)threadIdx.x + k * ZNT < g1) put(pq[k], pa[k], pb[k]);
  for (int g = g0 + threadIdx.x + kZPre * ZNT; g < g1; g += ZNT)
    put(st.g_qz[g], a[g], two ? b[g] : mkc<C>(0, 0));
  __syncthreads();
  fft_lines<N, +1, ZNT, PR ? PRUNE_IN : PRUNE_NONE>(zb, LS, 2 * ZSG, tw);
  C* o = out + (long)item * N * st.nst + q0;
  for (int e = threadIdx.x; e < 2 * ZSG * N; e += ZNT) {
    const int l = e % (2 * ZSG), z = e / (2 * ZSG);
    if (l % ZSG < nq) o[(long)z * st.nst + (l / ZSG) * st.hs + l % ZSG] = zb[l * LS + LinePad<N>::off(z)];
  }
}

// ---------------------------------------------------------------------------
// z pass, forward: sticks -> sphere with the Gamma unpack, then an epilogue
// ---------------------------------------------------------------------------
// An epilogue reads its per-G inputs through Epi::pre (prefetching them
// before the transform was measured slower: the extra registers cost more
// occupancy than the hidden latency gained).
template <int N, bool PR, class C, class Epi>
__global__ void __launch_bounds__(ZNT) k_zfwd(const C* __restrict__ sticks,
                                              const int2* __restrict__ items, StickTab st,
                                              const C* __restrict__ twg, Epi epi, const int* dn) {
  if (dn && (int)blockIdx.y >= dev_count<true>(dn, 0)) return;
  constexpr int LS = LinePad<N>::LEN | 1;
  using LP = LinePad<N>;
  using T = real_t<C>;
  C* tw = smem_tw<C>();
  C* zb = smem_tw<C>() + N;
  const int qg = blockIdx.x, item = blockIdx.y;
  const int q0 = qg * ZSG;
  const int nq = min(ZSG, st.nsp - q0);
  const C* s0 = sticks + (long)item * N * st.nst + q0;
  // asynchronous copies: all of a CTA's reads are in flight at once, without
  // registers (a loop of loads and stores left the kernel waiting for each)
  for (int e = threadIdx.x; e < 2 * ZSG * N; e += ZNT) {
    const int l = e % (2 * ZSG), z = e / (2 * ZSG);
    if (l % ZSG < nq)
      cp_async_elem(zb + l * LS + LinePad<N>::off(z), s0 + (long)z * st.nst + (l / ZSG) * st.hs + l % ZSG);
  }
  load_tw<N>(tw, twg);
  const int2 it = items[item];
  const int g0 = st.sp_gstart[q0], g1 = st.sp_gstart[q0 + nq];
  cp_async_wait_all();
  __syncthreads();
  fft_lines<N, -1, ZNT, PR ? PRUNE_OUT : PRUNE_NONE>(zb, LS, 2 * ZSG, tw);
  auto take = [&](int g, int2 qz, const typename Epi::Pre& pr) {
    const int z = qz.y;
    C ap, am;
    if (qz.x < 2) {
      ap = zb[LP::off((z + N) % N)];
      am = zb[LP::off((N - z) % N)];
    } else {
      const int l = z_line(qz.x - 2 * q0);
      ap = zb[l * LS + LP::off((z + N) % N)];
      am = zb[(l ^ ZSG) * LS + LP::off((N - z) % N)];
    }
    const C fp = mkc<C>(T(0.5) * (ap.x + am.x), T(0.5) * (ap.y + am.y));
    const C fm = mkc<C>(T(0.5) * (ap.x - am.x), T(0.5) * (ap.y - am.y));
    epi(g, it, pr, mkc<C>(fp.x, fm.y), mkc<C>(fp.y, -fm.x));
  };
  for (int g = g0 + threadIdx.x; g < g1; g += ZNT) take(g, st.g_qz[g], epi.pre(g, it));
}

struct EpiStore {
  double2* dst;
  long ld;
  struct Pre {};
  WB_DEV Pre pre(int, int2) const { return {}; }
  WB_DEV void operator()(int g, int2 it, const Pre&, double2 b1, double2 b2) const {
    dst[(long)it.x * ld + g] = b1;
    if (it.y >= 0) dst[(long)it.y * ld + g] = b2;
  }
};

// T = (V psi + g2kin psi with Im(G=0) = 0) - e psi   (h_psi then
// apply_sternheimerop_to_m_wfcs.f90:65-74; KB and alpha Pv follow as GEMMs)
template <class C>
struct EpiHpsiT {
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
  WB_DEV Pre pre(int g, int2 it) const {
    Pre r;
    r.p1 = P[(long)it.x * ld + g];
    r.p2 = it.y >= 0 ? P[(long)it.y * ld + g] : mkc<C>(0, 0);
    r.k = g2kin[g];
    return r;
  }
  WB_DEV void one(int g, int c, C p, T k, C vp) const {
    C h = mkc<C>(fma(k, p.x, vp.x), fma(k, p.y, vp.y));
    if (g == 0) h.y = T(0);
    const T e = ecol[c];
    Tv[(long)c * ld + g] = mkc<C>(fma(-e, p.x, h.x), fma(-e, p.y, h.y));
  }
  WB_DEV void operator()(int g, int2 it, const Pre& pr, C b1, C b2) const {
    one(g, it.x, pr.p1, pr.k, b1);
    if (it.y >= 0) one(g, it.y, pr.p2, pr.k, b2);
  }
};
using EpiHpsi = EpiHpsiT<double2>;
using EpiHpsi32 = EpiHpsiT<float2>;

// dng(perm(g), p) = sqvc(g) * drho_G(g), G = 0 zeroed
// (dfpt_module.f90:485-487,502-503 and apply_operator.f90:63-67)
struct EpiDng {
  double2* dng;
  long ld;
  const int* perm;
  const double* sqvc;
  struct Pre {
    double s;
    int r;
  };
  WB_DEV Pre pre(int g, int2) const { return {(g == 0) ? 0.0 : sqvc[g], perm[g]}; }
  WB_DEV void operator()(int g, int2 it, const Pre& pr, double2 b1, double2 b2) const {
    const double s = pr.s;
    const long r = pr.r;
    dng[(long)it.x * ld + r] = make_double2(s * b1.x, s * b1.y);
    if (it.y >= 0) dng[(long)it.y * ld + r] = make_double2(s * b2.x, s * b2.y);
  }
};

// ---------------------------------------------------------------------------
// x-y plane passes (phases and layout: wb_plane.cuh)
// ---------------------------------------------------------------------------
constexpr size_t kMaxSmem = 227 * 1024;  // shared memory of one CTA
template <int N, class C>
constexpr size_t psmem() { return sizeof(C) * CPlane<N, true>::SIZE; }

// Threads per CTA of the plane kernels, sized so that the row phases (N A and
// N B items) fill whole rounds of the block and the CTAs that fit an SM's
// shared memory keep 64 to 128 registers per thread; and the CTAs per SM that
// the compiler must leave registers for.
template <int N, class C>
constexpr int plane_threads() {
  if (N <= 16) return 64;
  if (N <= 20) return 128;
  if (N <= 24) return 160;
  if (N <= 32) return 128;
  if (N <= 48) return 192;
  if (N <= 64) return 256;
  if (N <= 72) return 352;
  if (N <= 80) return 416;
  if (N <= 96) return sizeof(C) == 16 ? 576 : 512;
  return 512;
}
template <int N, class C>
constexpr int plane_blocks() {
  const int by_smem = (int)(227 * 1024 / (psmem<N, C>() + 1024));
  const int by_regs = 65536 / (plane_threads<N, C>() * (sizeof(C) == 16 ? 72 : 64));
  const int b = by_smem < by_regs ? by_smem : by_regs;
  return b < 1 ? 1 : b;
}
// Threads of the RHS and density kernels, which hold a share of the plane in
// registers over the band loop (N^2 / threads doubles): fewer for the large
// boxes, so that none spills; and the rounds of the block over the row items
// that hold real space.
template <int N>
constexpr int rd_threads() { return N <= 80 ? plane_threads<N, double2>() : N <= 96 ? 288 : 384; }
template <int N>
constexpr int real_rounds() { return (N * FftSplit<N>::N1 + rd_threads<N>() - 1) / rd_threads<N>(); }

// sticks of a plane -> inverse column transforms and the rows' first step; ends
// with the plane ready for row_to_real
template <class G, class TW, class C>
WB_DEV void plane_inverse(C* pl, const TW& tw, const C* sz, const StickTab& st, const G& g, int nt) {
  plane_col_in<G::A>(pl, tw, sz, st.cmap, g, nt);
  __syncthreads();
  plane_col_mid_inv<G::B>(pl, g, nt);
  __syncthreads();
  plane_row_in<G::A>(pl, tw, g, nt);
  __syncthreads();
}
// from row_from_real to the sticks
template <class G, class TW, class C>
WB_DEV void plane_forward(C* pl, const TW& tw, C* sz, const StickTab& st, const G& g, int nt) {
  __syncthreads();
  plane_row_out<G::A>(pl, g, nt);
  __syncthreads();
  plane_col_mid_fwd<G::B>(pl, tw, g, nt);
  __syncthreads();
  plane_col_out<G::A>(pl, sz, st.cmap, g, nt);
}

// psi -> V(r) psi(r) / N^3 -> back, in place on the sticks (QE vloc_psi_gamma);
// one CTA = plane z of item `item`.  Bound by the shared-memory pipe up to 80^3
// (64^3 FP64: about 4,800 wavefronts of a plane's 5,900 cycles) and by the FP64
// pipe in the 9- and 12-point row steps of 108^3 (5,700 of the 7,250 cycles that
// the largest phase takes).  Per band-pair item on one B200, against kernels that
// zeroed, scattered and gathered the plane and read their twiddles from shared
// memory per lane: 64^3 1.30 us (was 1.65) in FP64, 0.71 (0.92) in FP32; 80^3
// 3.1 (5.2) in FP64; 108^3 9.8 (14.0) and 4.8 (7.0); 48^3 1.1 (1.8).
//
// STAGED: a persistent CTA that runs over the units (plane, item) with the next
// unit's sticks copied into a shared-memory stage while it works on one, where
// one CTA fills an SM and the stage fits beside its plane.  Without it each CTA
// begins with two dependent trips to L2 or DRAM (3,500 of an FP64 108^3 plane's
// 24,400 cycles) and ends in a launch gap that nothing hides: 9.77 -> 9.14 us per
// item.  With several CTAs per SM the others hide both and the stage only costs
// (FP32 64^3 0.71 -> 0.76 us, 108^3 4.77 -> 4.92).
template <int N, bool PR, class C, bool STAGED>
__global__ void __launch_bounds__(plane_threads<N, C>(), plane_blocks<N, C>()) k_plane_vloc(
    C* __restrict__ sticks, StickTab st, const real_t<C>* __restrict__ vs, const __grid_constant__ TwParam<N, C> tw,
    int nitems, const int* dn) {
  constexpr int NT = plane_threads<N, C>();
  C* pl = smem_tw<C>();
  const CPlane<N, PR> g(st.ncols, st.xhi + 1);
  if constexpr (STAGED) {
    const int units = dev_count<true>(dn, nitems) * N;  // unit = item * N + z
    C* stage = pl + CPlane<N, PR>::SIZE;
    auto fetch = [&](int u) {
      const unsigned char* src = reinterpret_cast<const unsigned char*>(sticks + (long)u * st.nst);
      unsigned char* dst = reinterpret_cast<unsigned char*>(stage);
      for (int b = threadIdx.x * 16; b < st.nst * (int)sizeof(C); b += NT * 16)
        cp_async_elem(reinterpret_cast<double2*>(dst + b), reinterpret_cast<const double2*>(src + b));
    };
    int u = blockIdx.x;
    if (u < units) fetch(u);
    for (; u < units; u += gridDim.x) {
      cp_async_wait_all();
      __syncthreads();  // the stage is full; the last unit's column pass is done with the plane
      plane_col_in<FftSplit<N>::N1>(pl, tw, stage, st.cmap, g, NT);
      __syncthreads();
      if (u + (int)gridDim.x < units) fetch(u + gridDim.x);
      plane_col_mid_inv<FftSplit<N>::N2>(pl, g, NT);
      __syncthreads();
      plane_row_in<FftSplit<N>::N1>(pl, tw, g, NT);
      __syncthreads();
      plane_row_vloc<FftSplit<N>::N2>(pl, tw, vs + (long)(u % N) * N * N, g, NT);
      plane_forward(pl, tw, sticks + (long)u * st.nst, st, g, NT);
    }
  } else {
    if (dn && (int)blockIdx.y >= dev_count<true>(dn, 0)) return;
    const int z = blockIdx.x, item = blockIdx.y;
    C* sz = sticks + ((long)item * N + z) * st.nst;
    plane_inverse(pl, tw, sz, st, g, NT);
    plane_row_vloc<FftSplit<N>::N2>(pl, tw, vs + (long)z * N * N, g, NT);
    plane_forward(pl, tw, sz, st, g, NT);
  }
}

// sticks -> full real-space box (complex: two real functions), no scaling
template <int N, bool PR>
__global__ void __launch_bounds__(plane_threads<N, double2>(), plane_blocks<N, double2>()) k_plane_inv_box(
    const double2* __restrict__ sticks, StickTab st, double2* __restrict__ box, const __grid_constant__ TwParam<N, double2> tw) {
  constexpr int NT = plane_threads<N, double2>();
  double2* pl = smem_tw<double2>();
  const CPlane<N, PR> g(st.ncols, st.xhi + 1);
  const long plane = (long)blockIdx.y * N + blockIdx.x;
  plane_inverse(pl, tw, sticks + plane * st.nst, st, g, NT);
  plane_row_box<FftSplit<N>::N2>(pl, box + plane * N * N, g, NT);
}

// RHS of the Sternheimer equation, dfpt_module.f90:245-260:
// (psi_v1(r) + i psi_v2(r)) * dv_p(r) / N^3 -> forward -> sticks
// One CTA per (plane z, perturbation p) loops over the band pairs with its
// thread's share of dv_p(r) in registers; the psi planes come from L2.
template <int N, bool PR>
__global__ void __launch_bounds__(rd_threads<N>(), 1) k_plane_rhs(
    const double2* __restrict__ evcr, const double2* __restrict__ dvbox, int npv, StickTab st,
    double2* __restrict__ sticks, const __grid_constant__ TwParam<N, double2> tw) {
  constexpr int NT = rd_threads<N>(), B = FftSplit<N>::N2, A = FftSplit<N>::N1;
  constexpr int ROUNDS = real_rounds<N>();
  double2* pl = smem_tw<double2>();
  const CPlane<N, PR> g(st.ncols, st.xhi + 1);
  const int z = blockIdx.x, p = blockIdx.y;
  constexpr double inv = 1.0 / ((double)N * N * N);
  const double2* dv = dvbox + ((long)(p >> 1) * N + z) * N * N;
  const bool hi = p & 1;
  double w[ROUNDS][B];
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const int it = threadIdx.x + r * NT, k1 = it / N, y = it % N;
#pragma unroll
    for (int i = 0; i < B; ++i) {
      w[r][i] = 0.0;
      if (it < N * A) {
        const double2 d = dv[(k1 + A * i) * N + y];
        w[r][i] = (hi ? d.y : d.x) * inv;
      }
    }
  }
  for (int k = 0; k < npv; ++k) {
    const double2* ps = evcr + ((long)k * N + z) * N * N;
    __syncthreads();  // the previous band pair's column pass is done with the plane
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
      const int it = threadIdx.x + r * NT, k1 = it / N, y = it % N;
      if (it < N * A) {
        double2 v[B];
#pragma unroll
        for (int i = 0; i < B; ++i) v[i] = ps[(k1 + A * i) * N + y];
#pragma unroll
        for (int i = 0; i < B; ++i) v[i] = cscale(v[i], w[r][i]);
        row_from_real<B>(pl + y * g.rs() + B * k1, v, tw, k1);
      }
    }
    const long item = (long)p * npv + k;
    plane_forward(pl, tw, sticks + (item * N + z) * st.nst, st, g, NT);
  }
}

// Density response, dfpt_module.f90:403-423 and :478:
// drho_p(r) = sum_v occ_v psi_v(r) dpsi_v(r), two perturbations per CTA,
// then (drho_p1 + i drho_p2) * scale -> forward -> sticks.
// Real space stays in registers: a thread sums its share of the density over
// the bands where the inverse rows leave it, and starts the forward rows from
// there.  acc is per-CTA scratch in global memory that parks the first
// perturbation's density.
template <int N, bool PR>
__global__ void __launch_bounds__(rd_threads<N>(), 1) k_plane_drho(
    const double2* __restrict__ dsticks, const double2* __restrict__ evcr, const double* __restrict__ occ, int nocc,
    int mb, StickTab st, double2* __restrict__ acc, double scale, double2* __restrict__ osticks,
    const __grid_constant__ TwParam<N, double2> tw) {
  constexpr int NT = rd_threads<N>(), B = FftSplit<N>::N2, A = FftSplit<N>::N1;
  constexpr int ROUNDS = real_rounds<N>();
  double2* pl = smem_tw<double2>();
  const CPlane<N, PR> g(st.ncols, st.xhi + 1);
  const int z = blockIdx.x, pp = blockIdx.y;
  const int npv = (nocc + 1) / 2;
  double* ac = reinterpret_cast<double*>(acc + ((long)pp * N + z) * N * N);
  double a[ROUNDS][B];
  for (int pi = 0; pi < 2; ++pi) {
    const int p = 2 * pp + pi;
    if (pi == 1) {
#pragma unroll
      for (int r = 0; r < ROUNDS; ++r)
#pragma unroll
        for (int i = 0; i < B; ++i)
          if (threadIdx.x + r * NT < N * A) ac[(r * B + i) * NT + threadIdx.x] = a[r][i];
    }
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r)
#pragma unroll
      for (int i = 0; i < B; ++i) a[r][i] = 0.0;
    for (int k = 0; p < mb && k < npv; ++k) {
      const long item = (long)p * npv + k;
      __syncthreads();
      plane_inverse(pl, tw, dsticks + (item * N + z) * st.nst, st, g, NT);
      const double o1 = occ[2 * k];
      const double o2 = (2 * k + 1 < nocc) ? occ[2 * k + 1] : 0.0;
      const double2* ps = evcr + ((long)k * N + z) * N * N;
#pragma unroll
      for (int r = 0; r < ROUNDS; ++r) {
        const int it = threadIdx.x + r * NT, k1 = it / N, y = it % N;
        if (it < N * A) {
          double2 v[B];
          row_to_real<B>(pl + y * g.rs() + B * k1, v);
#pragma unroll
          for (int i = 0; i < B; ++i) {
            const double2 s = ps[(k1 + A * i) * N + y];
            a[r][i] += fma(o1 * s.x, v[i].x, o2 * s.y * v[i].y);
          }
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const int it = threadIdx.x + r * NT, k1 = it / N, y = it % N;
    if (it < N * A) {
      double2 v[B];
#pragma unroll
      for (int i = 0; i < B; ++i) v[i] = make_double2(ac[(r * B + i) * NT + threadIdx.x] * scale, a[r][i] * scale);
      row_from_real<B>(pl + y * g.rs() + B * k1, v, tw, k1);
    }
  }
  plane_forward(pl, tw, osticks + ((long)pp * N + z) * st.nst, st, g, NT);
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
template <int N, class C = double2>
static constexpr size_t zsmem() { return sizeof(C) * (N + 2 * ZSG * (LinePad<N>::LEN | 1)); }

// exp(+2 pi i j / n), accurate host values
static double2 unit_root(int j, int n) {
  const long double a = 2.0L * 3.14159265358979323846264338327950288L * (long double)(j % n) / (long double)n;
  return make_double2((double)cosl(a), (double)sinl(a));
}
template <int N, class C>
static TwParam<N, C> make_tw_param() {
  TwParam<N, C> t{};
  for (int k1 = 0; k1 < FftSplit<N>::N1; ++k1)
    for (int n2 = 0; n2 < FftSplit<N>::N2; ++n2) {
      const double2 w = unit_root(k1 * n2, N);
      t.t[k1 * FftSplit<N>::N2 + n2].x = (real_t<C>)w.x;
      t.t[k1 * FftSplit<N>::N2 + n2].y = (real_t<C>)w.y;
    }
  return t;
}

template <int N>
struct FftN {
  static constexpr int PT = plane_threads<N, double2>();
  // the plane kernels' twiddles, computed on the host once
  template <class C>
  static const TwParam<N, C>& tw_param() {
    static const TwParam<N, C> table = make_tw_param<N, C>();
    return table;
  }
  template <class K>
  static void smem(K* k, size_t bytes) {
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  }
  template <bool PR>
  static void setup_pr() {
    smem(k_zinv<N, PR, double2>, zsmem<N>());
    smem(k_zfwd<N, PR, double2, EpiStore>, zsmem<N>());
    smem(k_zfwd<N, PR, double2, EpiHpsi>, zsmem<N>());
    smem(k_zfwd<N, PR, double2, EpiDng>, zsmem<N>());
    smem(k_plane_vloc<N, PR, double2, false>, psmem<N, double2>());
    if constexpr (plane_blocks<N, double2>() == 1) smem(k_plane_vloc<N, PR, double2, true>, kMaxSmem);
    if constexpr (plane_blocks<N, float2>() == 1) smem(k_plane_vloc<N, PR, float2, true>, kMaxSmem);
    smem(k_plane_inv_box<N, PR>, psmem<N, double2>());
    smem(k_plane_rhs<N, PR>, psmem<N, double2>());
    smem(k_plane_drho<N, PR>, psmem<N, double2>());
    smem(k_zinv<N, PR, float2>, zsmem<N, float2>());
    smem(k_zfwd<N, PR, float2, EpiHpsi32>, zsmem<N, float2>());
    smem(k_plane_vloc<N, PR, float2, false>, psmem<N, float2>());
  }
  static void setup() {
    setup_pr<false>();
    setup_pr<true>();
  }
  static dim3 zgrid(const StickTab& st, int nitems) { return dim3((st.nsp + ZSG - 1) / ZSG, nitems); }
  // Local-potential transforms of the PCG operator, FP64 (C = double2) or the
  // FP32 inner solves (C = float2): one CTA per (stick group or plane, item);
  // with a device count (graph replays) nitems is the bound the grid is sized
  // for and the CTAs beyond the device count return at once.
  template <class C, class F>
  static void zinv_t(const F& f, const C* src, long ld, const int2* items, int nitems, C* sticks) {
    if (nitems <= 0) return;
    constexpr size_t zs = zsmem<N, C>();
    if (f.st.prune)
      k_zinv<N, true, C><<<zgrid(f.st, nitems), ZNT, zs, f.stream>>>(src, ld, items, f.st, sticks, f.tw, f.dcount);
    else
      k_zinv<N, false, C><<<zgrid(f.st, nitems), ZNT, zs, f.stream>>>(src, ld, items, f.st, sticks, f.tw, f.dcount);
  }
  template <class C, class F>
  static void vloc_t(const F& f, C* sticks, int nitems, const real_t<C>* vs) {
    if (nitems <= 0) return;
    constexpr size_t ps = psmem<N, C>();
    constexpr int nt = plane_threads<N, C>();
    if constexpr (plane_blocks<N, C>() == 1) {
      const size_t staged = ps + sizeof(C) * f.st.nst;
      if (staged <= kMaxSmem) {
        const int grid = std::min(nitems * N, sm_count());
        auto k = f.st.prune ? k_plane_vloc<N, true, C, true> : k_plane_vloc<N, false, C, true>;
        k<<<grid, nt, staged, f.stream>>>(sticks, f.st, vs, tw_param<C>(), nitems, f.dcount);
        return;
      }
    }
    auto k = f.st.prune ? k_plane_vloc<N, true, C, false> : k_plane_vloc<N, false, C, false>;
    k<<<dim3(N, nitems), nt, ps, f.stream>>>(sticks, f.st, vs, tw_param<C>(), nitems, f.dcount);
  }
  template <class C, class F, class Epi>
  static void zfwd_t(const F& f, const C* sticks, const int2* items, int nitems, Epi epi) {
    if (nitems <= 0) return;
    constexpr size_t zs = zsmem<N, C>();
    if (f.st.prune)
      k_zfwd<N, true, C, Epi><<<zgrid(f.st, nitems), ZNT, zs, f.stream>>>(sticks, items, f.st, f.tw, epi, f.dcount);
    else
      k_zfwd<N, false, C, Epi><<<zgrid(f.st, nitems), ZNT, zs, f.stream>>>(sticks, items, f.st, f.tw, epi, f.dcount);
  }
  static void zinv32(const FftArgs32& f, const float2* src, long ld, const int2* items, int nitems, float2* sticks) {
    zinv_t<float2>(f, src, ld, items, nitems, sticks);
  }
  static void vloc32(const FftArgs32& f, float2* sticks, int nitems, const float* vs) {
    vloc_t<float2>(f, sticks, nitems, vs);
  }
  static void zfwd_hpsi32(const FftArgs32& f, const float2* sticks, const int2* items, int nitems, EpiHpsi32 epi) {
    zfwd_t<float2>(f, sticks, items, nitems, epi);
  }
  static void zinv(const FftArgs& f, const double2* src, long ld, const int2* items, int nitems, double2* sticks) {
    zinv_t<double2>(f, src, ld, items, nitems, sticks);
  }
  template <class Epi>
  static void zfwd(const FftArgs& f, const double2* sticks, const int2* items, int nitems, Epi epi) {
    zfwd_t<double2>(f, sticks, items, nitems, epi);
  }
  static void vloc(const FftArgs& f, double2* sticks, int nitems, const double* vs) {
    vloc_t<double2>(f, sticks, nitems, vs);
  }
  static void inv_box(const FftArgs& f, const double2* sticks, int nitems, double2* box) {
    if (nitems <= 0) return;
    const dim3 g(N, nitems);
    if (f.st.prune) k_plane_inv_box<N, true><<<g, PT, psmem<N, double2>(), f.stream>>>(sticks, f.st, box, tw_param<double2>());
    else k_plane_inv_box<N, false><<<g, PT, psmem<N, double2>(), f.stream>>>(sticks, f.st, box, tw_param<double2>());
  }
  static void rhs(const FftArgs& f, const double2* evcr, const double2* dvbox, int npv, int mb, double2* sticks) {
    if (mb <= 0) return;
    const dim3 g(N, mb);
    if (f.st.prune)
      k_plane_rhs<N, true><<<g, rd_threads<N>(), psmem<N, double2>(), f.stream>>>(evcr, dvbox, npv, f.st, sticks,
                                                                                tw_param<double2>());
    else
      k_plane_rhs<N, false><<<g, rd_threads<N>(), psmem<N, double2>(), f.stream>>>(evcr, dvbox, npv, f.st, sticks,
                                                                                tw_param<double2>());
  }
  static void drho(const FftArgs& f, const double2* dsticks, const double2* evcr, const double* occ, int nocc,
                   int mb, double2* acc, double scale, double2* osticks) {
    if (mb <= 0) return;
    const dim3 g(N, (mb + 1) / 2);
    if (f.st.prune)
      k_plane_drho<N, true><<<g, rd_threads<N>(), psmem<N, double2>(), f.stream>>>(dsticks, evcr, occ, nocc, mb, f.st, acc,
                                                                          scale, osticks, tw_param<double2>());
    else
      k_plane_drho<N, false><<<g, rd_threads<N>(), psmem<N, double2>(), f.stream>>>(dsticks, evcr, occ, nocc, mb, f.st, acc,
                                                                           scale, osticks, tw_param<double2>());
  }
};

#define WB_FOR_EACH_N(X) X(16) X(20) X(24) X(32) X(36) X(40) X(48) X(60) X(64) X(72) X(80) X(96) X(100) X(108)

void fft_split(int n, int* a, int* b) {
  *a = *b = 0;
  switch (n) {
#define X(n)                   \
  case n:                      \
    *a = FftSplit<n>::N1;      \
    *b = FftSplit<n>::N2;      \
    break;
    WB_FOR_EACH_N(X)
#undef X
    default: break;
  }
}

bool fft_supported(int n) {
  switch (n) {
#define X(n) case n: return true;
    WB_FOR_EACH_N(X)
#undef X
    default: return false;
  }
}

void fft_setup(int n) {
  switch (n) {
#define X(n) case n: FftN<n>::setup(); break;
    WB_FOR_EACH_N(X)
#undef X
    default: break;
  }
}

#define WB_DISPATCH(n, call) \
  switch (n) {               \
    WB_FOR_EACH_N(X)         \
    default: break;          \
  }

void fft_zinv(const FftArgs& f, const double2* src, long ld, const int2* items, int nitems, double2* sticks) {
  if (f.rt) return rt_zinv(f, src, ld, items, nitems, sticks);
#define X(n) case n: FftN<n>::zinv(f, src, ld, items, nitems, sticks); break;
  WB_DISPATCH(f.n, )
#undef X
}
void fft_zfwd_store(const FftArgs& f, const double2* sticks, const int2* items, int nitems, double2* dst, long ld) {
  if (f.rt) return rt_zfwd_store(f, sticks, items, nitems, dst, ld);
#define X(n) case n: FftN<n>::zfwd(f, sticks, items, nitems, EpiStore{dst, ld}); break;
  WB_DISPATCH(f.n, )
#undef X
}
void fft_zfwd_hpsi(const FftArgs& f, const double2* sticks, const int2* items, int nitems, const double2* P,
                   double2* T, long ld, const double* g2kin, const double* ecol) {
  if (f.rt) return rt_zfwd_hpsi(f, sticks, items, nitems, P, T, ld, g2kin, ecol);
#define X(n) case n: FftN<n>::zfwd(f, sticks, items, nitems, EpiHpsi{P, T, ld, g2kin, ecol}); break;
  WB_DISPATCH(f.n, )
#undef X
}
void fft_zfwd_dng(const FftArgs& f, const double2* sticks, const int2* items, int nitems, double2* dng, long ld,
                  const int* perm, const double* sqvc) {
  if (f.rt) return rt_zfwd_dng(f, sticks, items, nitems, dng, ld, perm, sqvc);
#define X(n) case n: FftN<n>::zfwd(f, sticks, items, nitems, EpiDng{dng, ld, perm, sqvc}); break;
  WB_DISPATCH(f.n, )
#undef X
}
void fft_zinv32(const FftArgs32& f, const float2* src, long ld, const int2* items, int nitems, float2* sticks) {
  if (f.rt) return rt_zinv32(f, src, ld, items, nitems, sticks);
#define X(n) case n: FftN<n>::zinv32(f, src, ld, items, nitems, sticks); break;
  WB_DISPATCH(f.n, )
#undef X
}
void fft_plane_vloc32(const FftArgs32& f, float2* sticks, int nitems, const float* vs) {
  if (f.rt) return rt_plane_vloc32(f, sticks, nitems, vs);
#define X(n) case n: FftN<n>::vloc32(f, sticks, nitems, vs); break;
  WB_DISPATCH(f.n, )
#undef X
}
void fft_zfwd_hpsi32(const FftArgs32& f, const float2* sticks, const int2* items, int nitems, const float2* P,
                     float2* T, long ld, const float* g2kin, const float* ecol) {
  if (f.rt) return rt_zfwd_hpsi32(f, sticks, items, nitems, P, T, ld, g2kin, ecol);
#define X(n) case n: FftN<n>::zfwd_hpsi32(f, sticks, items, nitems, EpiHpsi32{P, T, ld, g2kin, ecol}); break;
  WB_DISPATCH(f.n, )
#undef X
}
void fft_plane_vloc(const FftArgs& f, double2* sticks, int nitems, const double* vs) {
  if (f.rt) return rt_plane_vloc(f, sticks, nitems, vs);
#define X(n) case n: FftN<n>::vloc(f, sticks, nitems, vs); break;
  WB_DISPATCH(f.n, )
#undef X
}
void fft_plane_inv_box(const FftArgs& f, const double2* sticks, int nitems, double2* box) {
  if (f.rt) return rt_plane_inv_box(f, sticks, nitems, box);
#define X(n) case n: FftN<n>::inv_box(f, sticks, nitems, box); break;
  WB_DISPATCH(f.n, )
#undef X
}
void fft_plane_rhs(const FftArgs& f, const double2* evcr, const double2* dvbox, int npv, int mb, double2* sticks) {
  if (f.rt) return rt_plane_rhs(f, evcr, dvbox, npv, mb, sticks);
#define X(n) case n: FftN<n>::rhs(f, evcr, dvbox, npv, mb, sticks); break;
  WB_DISPATCH(f.n, )
#undef X
}
void fft_plane_drho(const FftArgs& f, const double2* dsticks, const double2* evcr, const double* occ, int nocc,
                    int mb, double2* acc, double scale, double2* osticks) {
  if (f.rt) return rt_plane_drho(f, dsticks, evcr, occ, nocc, mb, acc, scale, osticks);
#define X(n) case n: FftN<n>::drho(f, dsticks, evcr, occ, nocc, mb, acc, scale, osticks); break;
  WB_DISPATCH(f.n, )
#undef X
}

}  // namespace wb
