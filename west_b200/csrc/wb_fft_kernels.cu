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

// ---------------------------------------------------------------------------
// z passes
// ---------------------------------------------------------------------------
// One unit = stick pairs [ZSG qg, ZSG qg + ZSG) of band-pair item `item`; line
// side * ZSG + i of its work area is that stick of pair q0 + i.  The four-step
// transforms keep everything but the exchange between the two steps in
// registers: the inverse's first step takes the sphere's coefficients straight
// from global memory (consecutive threads along a stick, whose coefficients are
// one run) and its second stores the sticks (consecutive threads over sticks);
// the forward's first step reads the sticks the same way, and in its second a
// thread owns z = k1 + A k2 of a stick and -z of its mirror, which is what the
// Gamma unpack of those G needs.
// Two steps of shared memory and one barrier per transform, where a zeroed and
// scattered work area, in-place steps and a separate unpack took five and three.
// Bound by DRAM latency and bandwidth: per item on one B200, inverse and forward,
// 64^3 FP32 0.143 and 0.170 us (0.188 and 0.199 before; 0.08 and 0.10 at 6.65
// TB/s), FP64 0.237 and 0.271 (0.238 and 0.302; 0.16 and 0.20); 108^3 FP64 1.42
// and 1.61 (1.53 and 1.76), FP32 0.70 and 0.84 (0.82 and 0.90).
constexpr int ZSG = kZGroup;

template <class C>
WB_DEV C* smem_tw() {
  extern __shared__ __align__(16) unsigned char smraw[];
  return reinterpret_cast<C*>(smraw);
}
// step factor table of a line (wb_fft.cuh) into shared memory
template <int N, class C>
WB_DEV void load_tw(C* tw, const C* twg) {
  for (int i = threadIdx.x; i < N; i += blockDim.x) tw[i] = twg[i];
}
// threads: the inverse's first step has ZSG B items; the forward's has 2 ZSG B
template <int N>
constexpr int z_threads() {
  constexpr int m = FftSplit<N>::N1 > FftSplit<N>::N2 ? FftSplit<N>::N1 : FftSplit<N>::N2;
  return (ZSG * m + 31) / 32 * 32;
}
// items, except where those threads would each hold two FP64 DFTs of 10 or more
// points in the second (80^3: 160 threads 0.91 us per item, 96 threads 0.78)
template <int N, class C>
constexpr int zf_threads() {
  return sizeof(C) == 16 && FftSplit<N>::N2 >= 10 ? z_threads<N>() : (2 * ZSG * FftSplit<N>::N2 + 31) / 32 * 32;
}

// The G vector behind element zi of the side-0 stick of pair q: g, or -1; flip:
// the sphere stores -G instead (for pair 0, its own mirror, also at G = 0, where
// the -G store wins as in the reference loop).  Without MAP each pair's
// coefficients are one ascending run of side 0, as in every sphere cut by planes;
// MAP reads a table instead (any half of the sphere).
template <int N, bool MAP>
WB_DEV int z_lookup(const StickTab& st, int q, int zi, bool* flip) {
  if constexpr (MAP) {
    const int e = __ldg(st.zmap + (long)q * N + zi);
    *flip = e & 1;
    return e >> 1;  // -1 stays -1
  } else {
    int z = zi < (N + 1) / 2 ? zi : zi - N;
    const int g0 = __ldg(st.sp_gstart + q), n = __ldg(st.sp_gstart + q + 1) - g0;
    *flip = q == 0 && z <= 0;
    if (q == 0) z = z < 0 ? -z : z;
    const int i = z - __ldg(st.zlo + q);
    return i >= 0 && i < n ? g0 + i : -1;
  }
}

template <int N, bool PR, class C, bool MAP>
__global__ void __launch_bounds__(z_threads<N>()) k_zinv(const C* __restrict__ src, long ld,
                                                         const int2* __restrict__ items, StickTab st,
                                                         C* __restrict__ out, const C* __restrict__ twg,
                                                         const int* dn) {
  if (dn && (int)blockIdx.y >= dev_count<true>(dn, 0)) return;  // beyond the device item count
  constexpr int A = FftSplit<N>::N1, B = FftSplit<N>::N2, NT = z_threads<N>();
  constexpr int LS = LinePad<N>::LEN | 1;  // odd: the second step's lanes over lines hit distinct banks
  using LP = LinePad<N>;
  using P = Prune<N>;
  constexpr bool PIN = PR && P::IN_OK;
  C* tw = smem_tw<C>();
  C* zb = tw + N;
  const int q0 = blockIdx.x * ZSG, item = blockIdx.y;
  const int nq = min(ZSG, st.nsp - q0);
  const int2 it2 = items[item];
  const C* a = src + (long)it2.x * ld;
  const bool two = it2.y >= 0;
  const C* b = src + (long)(two ? it2.y : it2.x) * ld;
  load_tw<N>(tw, twg);
  __syncthreads();
  for (int it = threadIdx.x; it < nq * B; it += NT) {
    const int i = it / B, n2 = it % B, q = q0 + i;
    C v0[A], v1[A];  // element B n1 + n2 of side 0, and of side 1 at its negative
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) {
      v0[n1] = v1[n1] = mkc<C>(0, 0);
      if (!PIN || P::in_live(n1)) {
        bool flip;
        const int g = z_lookup<N, MAP>(st, q, B * n1 + n2, &flip);
        if (g >= 0) {
          const C a1 = a[g], a2 = two ? b[g] : mkc<C>(0, 0);
          const C pos = mkc<C>(a1.x - a2.y, a1.y + a2.x);  // a1 + i a2
          const C neg = mkc<C>(a1.x + a2.y, a2.x - a1.y);  // conj(a1 - i a2)
          v0[n1] = flip ? neg : pos;
          v1[n1] = flip ? pos : neg;
        }
      }
    }
    C w[A];
#pragma unroll
    for (int j = 0; j < A; ++j) w[j] = n2 == 0 ? v1[(A - j) % A] : v1[A - 1 - j];
    C* p = zb + i * LS;
    rdft<A, +1>(v0);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) p[LP::off_blk(k1, n2)] = k1 ? ctw<+1>(v0[k1], tw[k1 * B + n2]) : v0[0];
    const int m2 = n2 == 0 ? 0 : B - n2;
    p += ZSG * LS;
    rdft<A, +1>(w);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) p[LP::off_blk(k1, m2)] = k1 ? ctw<+1>(w[k1], tw[k1 * B + m2]) : w[0];
  }
  __syncthreads();
  C* o = out + (long)item * N * st.nst + q0;
  for (int it = threadIdx.x; it < 2 * ZSG * A; it += NT) {
    const int l = it % (2 * ZSG), k1 = it / (2 * ZSG);
    if (l % ZSG >= nq) continue;
    const C* p = zb + l * LS;
    C v[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) v[n2] = p[LP::off_blk(k1, n2)];
    rdft<B, +1>(v);
    C* os = o + (l / ZSG) * st.hs + l % ZSG;
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) os[(long)(k1 + A * k2) * st.nst] = v[k2];
  }
}

// sticks -> sphere with the Gamma unpack, then an epilogue per G.  The columns an
// epilogue reads are copied to shared memory behind the first step (one run of G
// for the whole stick group), so that it waits for none of them.
template <int N, bool PR, class C, class Epi, bool MAP>
__global__ void __launch_bounds__(zf_threads<N, C>()) k_zfwd(const C* __restrict__ sticks,
                                                         const int2* __restrict__ items, StickTab st,
                                                         const C* __restrict__ twg, Epi epi, const int* dn) {
  if (dn && (int)blockIdx.y >= dev_count<true>(dn, 0)) return;
  constexpr int A = FftSplit<N>::N1, B = FftSplit<N>::N2, NT = zf_threads<N, C>();
  constexpr int LS = LinePad<N>::LEN | 1;
  using LP = LinePad<N>;
  using T = real_t<C>;
  using P = Prune<N>;
  constexpr bool POUT = PR && P::OUT_OK;
  C* tw = smem_tw<C>();
  C* zb = tw + N;
  const int q0 = blockIdx.x * ZSG, item = blockIdx.y;
  const int nq = min(ZSG, st.nsp - q0);
  const C* s0 = sticks + (long)item * N * st.nst + q0;
  const int2 it2 = items[item];
  const int g0 = st.sp_gstart[q0], ng = st.sp_gstart[q0 + nq] - g0;
  C* ps = zb + 2 * ZSG * LS;
  if constexpr (Epi::STAGED)
    for (int i = threadIdx.x; i < ng; i += NT) {
      cp_async_elem(ps + i, epi.P + (long)it2.x * epi.ld + g0 + i);
      if (it2.y >= 0) cp_async_elem(ps + ng + i, epi.P + (long)it2.y * epi.ld + g0 + i);
    }
  load_tw<N>(tw, twg);
  __syncthreads();
  for (int it = threadIdx.x; it < 2 * ZSG * B; it += NT) {
    const int l = it % (2 * ZSG), n2 = it / (2 * ZSG);
    if (l % ZSG >= nq) continue;
    const C* is = s0 + (l / ZSG) * st.hs + l % ZSG;
    C v[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) v[n1] = is[(long)(B * n1 + n2) * st.nst];
    rdft<A, -1>(v);
    C* p = zb + l * LS;
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) p[LP::off_blk(k1, n2)] = k1 ? ctw<-1>(v[k1], tw[k1 * B + n2]) : v[0];
  }
  if constexpr (Epi::STAGED) cp_async_wait_all();
  __syncthreads();
  for (int it = threadIdx.x; it < nq * A; it += NT) {
    const int i = it / A, k1 = it % A, q = q0 + i;
    const int m1 = k1 == 0 ? 0 : A - k1;
    const C* p0 = zb + i * LS;
    const C* p1 = q == 0 ? p0 : p0 + ZSG * LS;  // the (0,0) stick is its own mirror
    C v[B], u[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
      v[n2] = p0[LP::off_blk(k1, n2)];
      u[n2] = p1[LP::off_blk(m1, n2)];
    }
    rdft<B, -1>(v);
    rdft<B, -1>(u);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) {
      if (POUT && !P::out_live(k2)) continue;
      const int zi = k1 + A * k2;
      bool flip;
      const int g = z_lookup<N, MAP>(st, q, zi, &flip);
      if (g < 0 || (q == 0 && flip && zi != 0)) continue;  // pair 0: each G once
      const C s = k1 == 0 ? u[(B - k2) % B] : u[B - 1 - k2];
      const C ap = flip ? s : v[k2], am = flip ? v[k2] : s;
      const C fp = mkc<C>(T(0.5) * (ap.x + am.x), T(0.5) * (ap.y + am.y));
      const C fm = mkc<C>(T(0.5) * (ap.x - am.x), T(0.5) * (ap.y - am.y));
      epi(g, it2, epi.pre(g, it2, ps + (g - g0), ng), mkc<C>(fp.x, fm.y), mkc<C>(fp.y, -fm.x));
    }
  }
}

struct EpiStore {
  double2* dst;
  long ld;
  static constexpr bool STAGED = false;
  struct Pre {};
  WB_DEV Pre pre(int, int2, const double2*, int) const { return {}; }
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
  static constexpr bool STAGED = true;
  WB_DEV Pre pre(int g, int2 it, const C* ps, int ng) const {
    Pre r;
    r.p1 = ps[0];
    r.p2 = it.y >= 0 ? ps[ng] : mkc<C>(0, 0);
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
  static constexpr bool STAGED = false;
  WB_DEV Pre pre(int g, int2, const double2*, int) const { return {(g == 0) ? 0.0 : sqvc[g], perm[g]}; }
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
  template <bool PR, bool MAP>
  static void setup_z() {
    smem(k_zinv<N, PR, double2, MAP>, zsmem<N>());
    smem(k_zfwd<N, PR, double2, EpiStore, MAP>, zsmem<N>());
    smem(k_zfwd<N, PR, double2, EpiHpsi, MAP>, zsmem<N>() + 2 * sizeof(double2) * ZSG * N);
    smem(k_zfwd<N, PR, double2, EpiDng, MAP>, zsmem<N>());
    smem(k_zinv<N, PR, float2, MAP>, zsmem<N, float2>());
    smem(k_zfwd<N, PR, float2, EpiHpsi32, MAP>, zsmem<N, float2>() + 2 * sizeof(float2) * ZSG * N);
  }
  template <bool PR>
  static void setup_pr() {
    setup_z<PR, false>();
    smem(k_plane_vloc<N, PR, double2, false>, psmem<N, double2>());
    if constexpr (plane_blocks<N, double2>() == 1) smem(k_plane_vloc<N, PR, double2, true>, kMaxSmem);
    if constexpr (plane_blocks<N, float2>() == 1) smem(k_plane_vloc<N, PR, float2, true>, kMaxSmem);
    smem(k_plane_inv_box<N, PR>, psmem<N, double2>());
    smem(k_plane_rhs<N, PR>, psmem<N, double2>());
    smem(k_plane_drho<N, PR>, psmem<N, double2>());
    smem(k_plane_vloc<N, PR, float2, false>, psmem<N, float2>());
  }
  static void setup() {
    setup_pr<false>();
    setup_pr<true>();
    setup_z<false, true>();
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
    // a half sphere without runs takes the table form, unpruned
    auto k = f.st.zmap ? k_zinv<N, false, C, true> : f.st.prune ? k_zinv<N, true, C, false> : k_zinv<N, false, C, false>;
    k<<<zgrid(f.st, nitems), z_threads<N>(), zs, f.stream>>>(src, ld, items, f.st, sticks, f.tw, f.dcount);
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
    auto k = f.st.zmap ? k_zfwd<N, false, C, Epi, true>
                       : f.st.prune ? k_zfwd<N, true, C, Epi, false> : k_zfwd<N, false, C, Epi, false>;
    const size_t staged = Epi::STAGED ? 2 * sizeof(C) * f.st.gmax : 0;
    k<<<zgrid(f.st, nitems), zf_threads<N, C>(), zs + staged, f.stream>>>(sticks, items, f.st, f.tw, epi, f.dcount);
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
