// Dense and streaming kernels of the response operator: the Gamma bra-ket
// GEMMs on FP64 tensor cores (DMMA), the masked preconditioned CG steps, and
// small pointwise passes.
//
// Complex arrays of length npw are treated as real arrays of length 2*npw
// (Re, Im interleaved), exactly as WEST passes them to DGEMM at Gamma
// (glbrak.f90:37-40, apply_alpha_pc_to_m_wfcs.f90:65-72).
#include "wb_common.cuh"
#include <algorithm>

#include "wb_internal.h"

namespace wb {

int sm_count() {
  static const int nsm = [] {  // contexts of several threads may ask first
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 148;
    return n;
  }();
  return nsm;
}

WB_DEV void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// cp.async of 16 bytes (a pair of k: every operand is a column of double2) or 8; zeros
// when !ok.  Copies are committed in groups, one per stage of a ring.
WB_DEV void cp_pair(double* smem, const double* gmem, bool ok) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(ok ? 16 : 0) : "memory");
}
WB_DEV void cp_one(double* smem, const double* gmem, bool ok) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(ok ? 8 : 0) : "memory");
}
WB_DEV void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int LEFT>
WB_DEV void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(LEFT) : "memory"); }

// ---------------------------------------------------------------------------
// part[s][j][r] = sum_{k in split s} W[r][k] X[col j][k]        (A^T B, split K)
// A CTA takes 32 rows r x 32 columns j; its four warps interleave k and are summed at
// the end.  Stages of 32 k's of both operands stream through a ring of three buffers
// in shared memory by cp.async, so a CTA has two stages in flight whatever its warps
// do, and four CTAs fit an SM.  Rows of 36 doubles put the fragments of a half-warp
// (4 rows x 4 k) on distinct banks.  K is even and a stage reads pairs of k.
// One tile for every size.  Bound by the FP64 tensor pipe (36.9 TFLOP/s) and its own
// latency.  Against two larger ones with a warp per k, us and TFLOP/s: 64 rows, 2,048
// columns, K = 16,880 152 and 29 (64 x 64: 142); 112 rows, 384 columns, K = 33,800 111
// and 26 (112 x 64: 97), 208 rows, 384 columns, K = 74,774 411 and 29 (112 x 64: 416); but
// 80 rows, 256 columns, K = 4,800 15 (112 x 64: 34), 32 rows, 2,048 columns, K = 16,880 83
// (64 x 64: 140).  Their chains of additions are four times as long: error against sums
// in extended precision 1.4e-15 and 1.9e-15 at the first and third size, here 5.2e-16
// and 8.6e-16.
// ---------------------------------------------------------------------------
constexpr int TN_T = 32, TN_K = 32, TN_ST = 3, TN_LD = TN_K + 4, TN_STAGE = 2 * TN_T * TN_LD;
constexpr int TN_SMEM = (int)sizeof(double) * TN_STAGE * TN_ST;
static_assert(TN_STAGE * TN_ST >= 4 * TN_T * TN_T, "the ring holds the four warps' sums");

__global__ void __launch_bounds__(128, 4) k_gemm_tn(const double* __restrict__ W, long ldw, int M,
                                                    const double* __restrict__ X, long ldx,
                                                    const int* __restrict__ cols, int ncol_host, const int* dn, int K,
                                                    int kchunk, int trows, double* __restrict__ part) {
  extern __shared__ __align__(16) double tn_sm[];
  const int ncol = dev_count(dn, ncol_host);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lr = lane >> 2, lk = lane & 3;
  const int r0 = blockIdx.x * trows, j0 = blockIdx.y * TN_T, split = blockIdx.z;
  const int rend = min(M, r0 + trows);
  if (j0 >= ncol) return;
  if (dn) {  // the split plan of this column count
    const int ns = gemm_tn_plan(M, ncol, K);
    if (split >= ns) return;
    kchunk = gemm_tn_chunk(K, ns);
  }
  const int kb = split * kchunk, ke = min(K, kb + kchunk);
  // copies: TN_K/2 pairs of k per row; a thread's pair index is fixed, its rows step
  constexpr int PR = TN_K / 2, RSTEP = 128 / PR, NROW = 2 * TN_T / RSTEP;
  const int kp = (tid % PR) * 2, row0 = tid / PR;
  const double* src[NROW];
  unsigned okm = 0;
#pragma unroll
  for (int i = 0; i < NROW; ++i) {
    const int row = row0 + i * RSTEP;
    src[i] = W;
    if (row < TN_T) {
      const int r = r0 + row;
      if (r < rend) { src[i] = W + (long)r * ldw; okm |= 1u << i; }
    } else {
      const int j = j0 + row - TN_T;
      if (j < ncol) { src[i] = X + (long)(cols ? cols[j] : j) * ldx; okm |= 1u << i; }
    }
  }
  auto fetch = [&](int st, int k0) {
    double* d = tn_sm + st * TN_STAGE + row0 * TN_LD + kp;
    const int k = k0 + kp;
    const bool kok = k < ke;
#pragma unroll
    for (int i = 0; i < NROW; ++i)
      cp_pair(d + i * RSTEP * TN_LD, src[i] + (kok ? k : 0), kok && (okm >> i & 1u));
  };
  // fragments of eight rows or columns beyond M or ncol are skipped, CTA-uniformly
  const int nr = (rend - r0 + 7) / 8, nj = min(4, (ncol - j0 + 7) / 8);
  double acc[4][4][2];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
#pragma unroll
  for (int st = 0; st < TN_ST - 1; ++st) {
    if (kb + st * TN_K < ke) fetch(st, kb + st * TN_K);
    cp_commit();
  }
  int st = 0;
  for (int k0 = kb; k0 < ke; k0 += TN_K) {
    cp_wait<TN_ST - 2>();
    __syncthreads();  // the stage is here, and the last one is read by every warp
    const double* sw = tn_sm + st * TN_STAGE + lr * TN_LD + warp * 4 + lk;
    const double* sx = sw + TN_T * TN_LD;
    if (nr >= 3 && nj == 4) {  // at most one fragment of zero rows
#pragma unroll
      for (int kk = 0; kk < TN_K; kk += 16) {
        double av[4], bv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          av[i] = sw[i * 8 * TN_LD + kk];
          bv[i] = sx[i * 8 * TN_LD + kk];
        }
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) dmma(acc[a][b][0], acc[a][b][1], av[a], bv[b]);
      }
    } else {
#pragma unroll
      for (int kk = 0; kk < TN_K; kk += 16) {
        double bv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) bv[i] = sx[i * 8 * TN_LD + kk];
#pragma unroll
        for (int a = 0; a < 4; ++a)
          if (a < nr) {
            const double av = sw[a * 8 * TN_LD + kk];
#pragma unroll
            for (int b = 0; b < 4; ++b)
              if (b < nj) dmma(acc[a][b][0], acc[a][b][1], av, bv[b]);
          }
      }
    }
    const int kn = k0 + (TN_ST - 1) * TN_K;
    if (kn < ke) fetch(st == 0 ? TN_ST - 1 : st - 1, kn);
    cp_commit();
    st = st == TN_ST - 1 ? 0 : st + 1;
  }
  cp_wait<0>();
  __syncthreads();  // the ring becomes the warps' sums, [warp][j][r]
  double* red = tn_sm + warp * TN_T * TN_T;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int h = 0; h < 2; ++h) red[(b * 8 + 2 * lk + h) * TN_T + a * 8 + lr] = acc[a][b][h];
  __syncthreads();
  for (int e = tid; e < TN_T * TN_T; e += 128) {
    const int r = r0 + e % TN_T, j = j0 + e / TN_T;
    if (r >= rend || j >= ncol) continue;
    double sum = 0.0;
#pragma unroll
    for (int w = 0; w < 4; ++w) sum += tn_sm[w * TN_T * TN_T + e];
    part[((long)split * ncol + j) * M + r] = sum;
  }
}

size_t gemm_tn_part_doubles(int M, int nsys, int K) {
  size_t best = 0;
  for (int t = 1; t <= (nsys + 31) / 32; ++t) {  // the plan changes with the column tiles
    const int n = std::min(nsys, t * 32);
    best = std::max(best, (size_t)gemm_tn_plan(M, n, K) * n * M);
  }
  return best;
}
int gemm_tn_plan_max(int M, int ncol, int K) {
  const int first = bucket_systems(ncol) == kBucketSystems ? 1 : bucket_systems(ncol) / 2 + 1;
  int best = 1;
  for (int t = (first + 31) / 32; t <= (ncol + 31) / 32; ++t) best = std::max(best, gemm_tn_plan(M, t * 32, K));
  return best;
}

void gemm_tn(const double* W, long ldw, int M, const double* X, long ldx, const int* cols, int ncol, int K,
             int nsplit, double* part, cudaStream_t s, const int* dn) {
  if (ncol <= 0 || M <= 0) return;
  if (dn) nsplit = gemm_tn_plan_max(M, ncol, K);
  const int tiles = (M + TN_T - 1) / TN_T, trows = ((M + tiles - 1) / tiles + 7) / 8 * 8;
  dim3 grid(tiles, (ncol + TN_T - 1) / TN_T, nsplit);
  k_gemm_tn<<<grid, 128, TN_SMEM, s>>>(W, ldw, M, X, ldx, cols, ncol, dn, K, gemm_tn_chunk(K, nsplit), trows, part);
}

// The reductions of the bra-kets, FP64 (split plan of k_gemm_tn) and FP32 (of the
// tcgen05 bra-ket): S = 2 sum_s part - W0 X0, then C = D S for the projectors, alpha S
// for the bands.
template <class T>
WB_DEV int red_splits(int nsplit, const int* dn, int M, int ncol, int K, int ctas) {
  if constexpr (sizeof(T) == 8) {
    return dn ? gemm_tn_plan(M, ncol, K) : nsplit;
  } else {
    int per;
    if (dn && ctas > 0) umma_braket_plan(ncol, K, &nsplit, &per, ctas);
    return nsplit;
  }
}

// One CTA per column.  GROUPS (up to 512 columns): groups of threads share out a row's
// splits (eight partial sums each), then a row's projectors q of D, and are summed in
// order through shared memory, since the time is the chain of loads; without it a thread
// has a row to itself (four partial sums), and more columns are in flight.  us, with
// groups and without: 64 rows, 64 columns of 74 splits 6.6 and 17, 2,048 columns of 19
// splits 17 and 11; 208 rows, 64 columns of 42 splits 11 and 19, 2,048 columns 47 and 36.
// Several columns per CTA, to read D less often, lost to the longer chain: 64 rows, 1,024
// columns 7 with one, 13 with two, 15 with four.
template <class T, int NT, bool GROUPS>
__global__ void __launch_bounds__(NT) k_gamma_reduce(const T* __restrict__ part, int nsplit, int M, int ncol_host,
                                                     const int* dn, const T* __restrict__ W, long ldw,
                                                     const T* __restrict__ X, long ldx, const int* __restrict__ cols,
                                                     const T* __restrict__ D, int nkb, T alpha, T* __restrict__ C,
                                                     int K, int ctas) {
  extern __shared__ __align__(16) unsigned char red_sm[];
  T* S = reinterpret_cast<T*>(red_sm);
  const int ncol = dev_count(dn, ncol_host);
  const int j = blockIdx.x;
  if (j >= ncol) return;
  nsplit = red_splits<T>(nsplit, dn, M, ncol, K, ctas);
  const int col = cols ? cols[j] : j;
  const T x0 = X[(long)col * ldx];
  const T* pj = part + (long)j * M;
  const long step = (long)ncol * M;
  T* cj = C + (long)j * M;
  if constexpr (GROUPS) {
    __shared__ T scratch[NT];
    int rw = 32;
    while (rw < M && rw < NT) rw *= 2;
    const int ng = NT / rw, g = threadIdx.x / rw, rt = threadIdx.x % rw;
    auto group_sum = [&](T mine) {  // of row rt, in group 0
      scratch[threadIdx.x] = mine;
      __syncthreads();
      T sum = 0;
      if (g == 0)
        for (int q = 0; q < ng; ++q) sum += scratch[q * rw + rt];
      __syncthreads();
      return sum;
    };
    for (int r0 = 0; r0 < M; r0 += rw) {
      const int r = r0 + rt;
      T s[8] = {};
      if (r < M) {
        int i = g;
        for (; i + 7 * ng < nsplit; i += 8 * ng) {
#pragma unroll
          for (int q = 0; q < 8; ++q) s[q] += pj[(i + q * ng) * step + r];
        }
#pragma unroll
        for (int q = 0; q < 7; ++q)
          if (i + q * ng < nsplit) s[q] += pj[(i + q * ng) * step + r];
      }
      const T sum = group_sum(((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7])));
      if (g == 0 && r < M) S[r] = T(2) * sum - W[(long)r * ldw] * x0;
    }
    __syncthreads();
    for (int r0 = 0; r0 < M; r0 += rw) {
      const int r = r0 + rt;
      T c0 = 0, c1 = 0, c2 = 0, c3 = 0;
      if (r < nkb) {
        const T* d = D + r;
        int q = g;
        for (; q + 3 * ng < nkb; q += 4 * ng) {
          c0 = fma(d[(long)q * nkb], S[q], c0);
          c1 = fma(d[(long)(q + ng) * nkb], S[q + ng], c1);
          c2 = fma(d[(long)(q + 2 * ng) * nkb], S[q + 2 * ng], c2);
          c3 = fma(d[(long)(q + 3 * ng) * nkb], S[q + 3 * ng], c3);
        }
        for (; q < nkb; q += ng) c0 = fma(d[(long)q * nkb], S[q], c0);
      }
      const T c = group_sum((c0 + c1) + (c2 + c3));
      if (g == 0 && r < M) cj[r] = r < nkb ? c : alpha * S[r];
    }
  } else {
    for (int r = threadIdx.x; r < M; r += NT) {
      const T w0 = W[(long)r * ldw];
      T s0 = 0, s1 = 0, s2 = 0, s3 = 0;
      int i = 0;
      for (; i + 3 < nsplit; i += 4) {
        s0 += pj[i * step + r];
        s1 += pj[(i + 1) * step + r];
        s2 += pj[(i + 2) * step + r];
        s3 += pj[(i + 3) * step + r];
      }
      for (; i < nsplit; ++i) s0 += pj[i * step + r];
      S[r] = T(2) * ((s0 + s1) + (s2 + s3)) - w0 * x0;
    }
    __syncthreads();
    for (int r = threadIdx.x; r < M; r += NT) {
      T c = 0;
      if (r < nkb) {
#pragma unroll 8
        for (int q = 0; q < nkb; ++q) c = fma(D[r + (long)q * nkb], S[q], c);
      }
      cj[r] = r < nkb ? c : alpha * S[r];
    }
  }
}

// GROUPS decides the order of the sums and follows the count's bucket (512 is one's
// bound, see bucket_systems); the number of threads without it does not.
template <class T>
static void gamma_reduce_t(const T* part, int nsplit, int M, int ncol, const T* W, long ldw, const T* X, long ldx,
                           const int* cols, const T* D, int nkb, T alpha, T* C, cudaStream_t s, const int* dn, int K,
                           int ctas) {
  if (ncol <= 0 || M <= 0) return;
  auto go = [&](auto k, int nt) {
    k<<<ncol, nt, sizeof(T) * M, s>>>(part, nsplit, M, ncol, dn, W, ldw, X, ldx, cols, D, nkb, alpha, C, K, ctas);
  };
  if (ncol <= 8 * kBucketSystems) go(k_gamma_reduce<T, 512, true>, 512);
  else if (M <= 128) go(k_gamma_reduce<T, 128, false>, 128);
  else go(k_gamma_reduce<T, 256, false>, 256);
}
void gamma_reduce(const double* part, int nsplit, int M, int ncol, const double* W, long ldw, const double* X,
                  long ldx, const int* cols, const double* D, int nkb, double alpha, double* C, cudaStream_t s,
                  const int* dn, int K) {
  gamma_reduce_t<double>(part, nsplit, M, ncol, W, ldw, X, ldx, cols, D, nkb, alpha, C, s, dn, K, 0);
}
void gamma_reduce32(const float* part, int nsplit, int M, int ncol, const float* W, long ldw, const float* X, long ldx,
                    const int* cols, const float* D, int nkb, float alpha, float* C, cudaStream_t s, const int* dn,
                    int K, int umma_ctas) {
  gamma_reduce_t<float>(part, nsplit, M, ncol, W, ldw, X, ldx, cols, D, nkb, alpha, C, s, dn, K, umma_ctas);
}

// ---------------------------------------------------------------------------
// Y[col j][k] = beta Y[col j][k] + sum_r W[r][k] C[j][r]
// CTA: 4 warps x 32 k, 32 columns j; stages of 16 projectors r of W and C stream
// through a ring of three buffers by cp.async.  With beta != 0 a thread loads its
// share of Y into registers before the ring starts, so that those reads are in
// flight during the whole product and the epilogue only adds.  Row strides 132
// and 20: the fragments of a half-warp fall on distinct banks.
// ---------------------------------------------------------------------------
constexpr int NN_R = 16, NN_ST = 3, NN_WLD = 132, NN_CLD = 20;
constexpr int NN_STAGE = NN_R * NN_WLD + 32 * NN_CLD;

__global__ void __launch_bounds__(128, 3) k_gemm_nn(const double* __restrict__ W, long ldw, int M,
                                                 const double* __restrict__ C, double* __restrict__ Y, long ldy,
                                                 const int* __restrict__ cols, int ncol_host, const int* dn, int K,
                                                 double beta) {
  extern __shared__ __align__(16) double nn_sm[];
  const int ncol = dev_count(dn, ncol_host);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lr = lane >> 2, lk = lane & 3;
  const int kbase = blockIdx.x * 128, j0 = blockIdx.y * 32;
  if (j0 >= ncol) return;
  auto fetch = [&](int st, int rb) {
    double* sw = nn_sm + st * NN_STAGE;
    double* sc = sw + NN_R * NN_WLD;
    const int kp = (tid & 63) * 2, k = kbase + kp;  // K is even: a pair never straddles it
#pragma unroll
    for (int i = 0; i < NN_R / 2; ++i) {
      const int rr = (tid >> 6) + 2 * i, r = rb + rr;
      const bool ok = r < M && k < K;
      cp_pair(sw + rr * NN_WLD + kp, W + (ok ? (long)r * ldw + k : 0), ok);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = tid & 15, jl = (tid >> 4) + 8 * i, r = rb + rr, j = j0 + jl;
      const bool ok = r < M && j < ncol;
      cp_one(sc + jl * NN_CLD + rr, C + (ok ? (long)j * M + r : 0), ok);
    }
  };
#pragma unroll
  for (int st = 0; st < NN_ST - 1; ++st) {
    if (st * NN_R < M) fetch(st, st * NN_R);
    cp_commit();
  }
  const int k0 = kbase + warp * 32 + lr;
  double y[4][4][2];
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = j0 + b * 8 + 2 * lk + h;
      const bool jok = beta != 0.0 && j < ncol;
      const double* yc = Y + (jok ? (long)(cols ? cols[j] : j) * ldy : 0);
#pragma unroll
      for (int a = 0; a < 4; ++a) y[a][b][h] = jok && k0 + a * 8 < K ? yc[k0 + a * 8] : 0.0;
    }
  double acc[4][4][2];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
  int st = 0;
  for (int rb = 0; rb < M; rb += NN_R) {
    cp_wait<NN_ST - 2>();
    __syncthreads();
    const int rn = rb + (NN_ST - 1) * NN_R;
    if (rn < M) fetch(st == 0 ? NN_ST - 1 : st - 1, rn);
    cp_commit();
    const double* sw = nn_sm + st * NN_STAGE + lk * NN_WLD + warp * 32 + lr;
    const double* sc = nn_sm + st * NN_STAGE + NN_R * NN_WLD + lr * NN_CLD + lk;
#pragma unroll
    for (int r = 0; r < NN_R; r += 4) {
      if (rb + r >= M) break;
      double av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        av[i] = sw[r * NN_WLD + i * 8];
        bv[i] = sc[i * 8 * NN_CLD + r];
      }
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) dmma(acc[a][b][0], acc[a][b][1], av[a], bv[b]);
    }
    st = st == NN_ST - 1 ? 0 : st + 1;
  }
  cp_wait<0>();
#pragma unroll
  for (int b = 0; b < 4; ++b)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = j0 + b * 8 + 2 * lk + h;
      if (j >= ncol) continue;
      double* yc = Y + (long)(cols ? cols[j] : j) * ldy;
#pragma unroll
      for (int a = 0; a < 4; ++a)
        if (k0 + a * 8 < K) yc[k0 + a * 8] = beta * y[a][b][h] + acc[a][b][h];
    }
}

void gemm_nn(const double* W, long ldw, int M, const double* C, double* Y, long ldy, const int* cols, int ncol,
             int K, double beta, cudaStream_t s, const int* dn) {
  if (ncol <= 0 || M <= 0) return;
  constexpr int SM = (int)sizeof(double) * NN_STAGE * NN_ST;
  dim3 grid((K + 127) / 128, (ncol + 31) / 32);
  k_gemm_nn<<<grid, 128, SM, s>>>(W, ldw, M, C, Y, ldy, cols, ncol, dn, K, beta);
}

void la_setup() {
  cudaFuncSetAttribute(k_gemm_tn, cudaFuncAttributeMaxDynamicSharedMemorySize, TN_SMEM);
  cudaFuncSetAttribute(k_gemm_nn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)sizeof(double) * NN_STAGE * NN_ST);
  // S of all projectors beside the kernel's static scratch, which together pass the
  // 48 KB that a launch has without this: up to 6,144 projectors
  cudaFuncSetAttribute(k_gamma_reduce<double, 512, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 48 * 1024);
}

// ---------------------------------------------------------------------------
// pointwise passes
// ---------------------------------------------------------------------------
// aux(i, p) = dvg(perm(i), p) * sqvc(i)      (apply_operator.f90:49-53)
__global__ void k_permute_scale(const double2* __restrict__ dvg, long ld_in, const int* __restrict__ perm,
                                const double* __restrict__ sqvc, int npw, double2* __restrict__ aux, long ld_out) {
  const int p = blockIdx.y;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npw; i += gridDim.x * blockDim.x)
    aux[(long)p * ld_out + i] = cscale(dvg[(long)p * ld_in + perm[i]], sqvc[i]);
}
void permute_scale(const double2* dvg, long ld_in, const int* perm, const double* sqvc, int npw, int m,
                   double2* aux, long ld_out, cudaStream_t s) {
  if (m <= 0) return;
  k_permute_scale<<<dim3((npw + 255) / 256, m), 256, 0, s>>>(dvg, ld_in, perm, sqvc, npw, aux, ld_out);
}

// 1 / max(1, g2kin / eprec_v) per band and G: the preconditioner of
// precondition_m_wfcts.f90:35-51 and linsolve_sternheimer_m_wfcts.f90:150-160,
// applied by multiplication.
__global__ void k_make_iprec(const double* __restrict__ g2kin, const double* __restrict__ eprec, int npw, int nocc,
                             double* __restrict__ iprec) {
  const int v = blockIdx.y;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npw; i += gridDim.x * blockDim.x)
    iprec[(long)v * npw + i] = 1.0 / fmax(1.0, g2kin[i] / eprec[v]);
}
void make_iprec(const double* g2kin, const double* eprec, int npw, int nocc, double* iprec, cudaStream_t s) {
  k_make_iprec<<<dim3((npw + 255) / 256, nocc), 256, 0, s>>>(g2kin, eprec, npw, nocc, iprec);
}

// pf = f / max(1, g2kin / eprec)         (precondition_m_wfcts.f90:35-51)
__global__ void k_precondition(const double2* __restrict__ f, double2* __restrict__ pf,
                               const double* __restrict__ iprec, int nocc, int npw, long ld) {
  const int j = blockIdx.y;
  const double* ip = iprec + (long)(j % nocc) * npw;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npw; i += gridDim.x * blockDim.x) {
    const double2 v = f[(long)j * ld + i];
    pf[(long)j * ld + i] = make_double2(v.x * ip[i], v.y * ip[i]);
  }
}
void precondition(const double2* f, double2* pf, const double* iprec, int nocc, int npw, int ncol, long ld,
                  cudaStream_t s) {
  if (ncol <= 0) return;
  k_precondition<<<dim3((npw + 255) / 256, ncol), 256, 0, s>>>(f, pf, iprec, nocc, npw, ld);
}

__global__ void k_sub_into(const double2* __restrict__ a, const double2* __restrict__ b, double2* __restrict__ out,
                           int npw, long ld) {
  const int j = blockIdx.y;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npw; i += gridDim.x * blockDim.x)
    out[(long)j * ld + i] = csub(a[(long)j * ld + i], b[(long)j * ld + i]);
}
void sub_into(const double2* a, const double2* b, double2* out, int npw, int ncol, long ld, cudaStream_t s) {
  if (ncol <= 0) return;
  k_sub_into<<<dim3((npw + 255) / 256, ncol), 256, 0, s>>>(a, b, out, npw, ld);
}

// T = g2kin P (Im at G=0 zeroed) - e P     (k_psi.f90:51-77 then :65-74 of
// apply_sternheimerop_to_m_wfcs.f90)
__global__ void k_kinetic_hpsi(const double2* __restrict__ P, double2* __restrict__ T,
                               const double* __restrict__ g2kin, const double* __restrict__ ecol,
                               const int* __restrict__ cols, const int* dn, int npw, long ld) {
  if ((int)blockIdx.y >= dev_count(dn, gridDim.y)) return;
  const int c = cols ? cols[blockIdx.y] : blockIdx.y;
  const double e = ecol[c];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npw; i += gridDim.x * blockDim.x) {
    const double2 p = P[(long)c * ld + i];
    double2 h = cscale(p, g2kin[i]);
    if (i == 0) h.y = 0.0;
    T[(long)c * ld + i] = make_double2(fma(-e, p.x, h.x), fma(-e, p.y, h.y));
  }
}
void kinetic_hpsi(const double2* P, double2* T, const double* g2kin, const double* ecol, const int* cols, int ncol,
                  int npw, long ld, cudaStream_t s, const int* dn) {
  if (ncol <= 0) return;
  k_kinetic_hpsi<<<dim3((npw + 255) / 256, ncol), 256, 0, s>>>(P, T, g2kin, ecol, cols, dn, npw, ld);
}

__global__ void k_plane_layout(const double* __restrict__ in, double* __restrict__ out, int nx, int ny, long n, int a,
                               int b, double div) {
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x) {
    const int ys = (int)(e % ny), x = (int)(e / ny % nx);
    const long z = e / ((long)nx * ny);
    const int y = ys / b + a * (ys % b);
    out[e] = in[(z * ny + y) * nx + x] / div;
  }
}
void plane_layout(const double* in, double* out, int nx, int ny, int nz, int a, int b, double div, cudaStream_t s) {
  const long n = (long)nx * ny * nz;
  k_plane_layout<<<(int)std::min<long>((n + 255) / 256, 4096), 256, 0, s>>>(in, out, nx, ny, n, a, b, div);
}

// eprec_v = 1.35 sum_G |psi_v(G)|^2 g2kin(G)       (set_eprec.f90:40-53)
__global__ void __launch_bounds__(256) k_set_eprec(const double2* __restrict__ evc, const double* __restrict__ g2kin,
                                                   int npw, double* __restrict__ eprec) {
  __shared__ double red[8];
  const int v = blockIdx.x;
  double s = 0.0;
  for (int i = threadIdx.x; i < npw; i += 256) {
    const double2 c = evc[(long)v * npw + i];
    s += (c.x * c.x + c.y * c.y) * g2kin[i];
  }
  s = block_sum<256>(s, red);
  if (threadIdx.x == 0) eprec[v] = 1.35 * s;
}
void set_eprec(const double2* evc, const double* g2kin, int npw, int nocc, double* eprec, cudaStream_t s) {
  k_set_eprec<<<nocc, 256, 0, s>>>(evc, g2kin, npw, eprec);
}

__global__ void k_fill_columns(const double* __restrict__ pb, int nocc, int nsys, double* __restrict__ out) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nsys; j += gridDim.x * blockDim.x) out[j] = pb[j % nocc];
}
void fill_columns(const double* per_band, int nocc, int nsys, double* out, cudaStream_t s) {
  k_fill_columns<<<(nsys + 255) / 256, 256, 0, s>>>(per_band, nocc, nsys, out);
}

__global__ void k_frac_coefficients(const double* __restrict__ C, int nocc, int nsys, int nfull,
                                    const double* __restrict__ occ, const double* __restrict__ et,
                                    double* __restrict__ fc) {
  const int nfrac = nocc - nfull;
  const long n = (long)nsys * nfrac;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < n; e += (long)gridDim.x * blockDim.x) {
    const int j = (int)(e / nfrac), f = (int)(e % nfrac);
    const int i = j % nocc, r = nfull + f;
    double v = 0.0;
    const double docc = occ[i] - occ[r];
    if (r > i && fabs(docc) >= 1e-3) v = C[(long)j * nocc + r] * docc / occ[i] / (et[i] - et[r]);
    fc[e] = v;
  }
}
void frac_coefficients(const double* C, int nocc, int nsys, int nfull, const double* occ, const double* et,
                       double* fc, cudaStream_t s) {
  const long n = (long)nsys * (nocc - nfull);
  if (n <= 0) return;
  k_frac_coefficients<<<(int)std::min<long>((n + 255) / 256, 4096), 256, 0, s>>>(C, nocc, nsys, nfull, occ, et, fc);
}

// ---------------------------------------------------------------------------
// masked PCG (linsolve_sternheimer_m_wfcts.f90:146-330), one CTA per system
// ---------------------------------------------------------------------------
__global__ void k_cg_reset(unsigned char* conv, int nsys) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < nsys; j += gridDim.x * blockDim.x) conv[j] = 0;
}
void cg_reset(unsigned char* conv, int nsys, cudaStream_t s) {
  k_cg_reset<<<(nsys + 255) / 256, 256, 0, s>>>(conv, nsys);
}

// h = g / max(1, g2kin/eprec); rho = <h|g>_Gamma; converged if rho < thr_j
// (thr_j = max(tr2 * rel_j, floor) when rel != nullptr, else tr2); otherwise
// P = -h + (rho / rho_prev) P  (P = -h at the first iteration).  C is the
// vector type (double2, or float2 in the mixed form); scalars are FP64.
template <class C>
__global__ void __launch_bounds__(256) k_cg_prec_rho(const int* __restrict__ act, const int* dn, const C* __restrict__ g,
                                                     C* __restrict__ P, const double* __restrict__ iprec, int nocc,
                                                     double* rho_prev, unsigned char* conv, int iter_host,
                                                     const int* iter_dev, double tr2, const double* __restrict__ rel,
                                                     double floor, int npw, long ld) {
  using T = real_t<C>;
  __shared__ double red[16];
  const int n = dev_count(dn, gridDim.x);
  const int iter = iter_dev ? *iter_dev : iter_host;
  for (int b = blockIdx.x; b < n; b += gridDim.x) {
    const int j = act[b];
    const C* gj = g + (long)j * ld;
    C* pj = P + (long)j * ld;
    const double* ip = iprec + (long)(j % nocc) * npw;
    double t = 0.0, t0 = 0.0;
    for (int i = threadIdx.x; i < npw; i += 256) {
      const double w = ip[i];
      const C gv = gj[i];
      const double hx = (double)gv.x * w, hy = (double)gv.y * w;
      t = fma(hx, (double)gv.x, fma(hy, (double)gv.y, t));
      if (i == 0) t0 = hx * (double)gv.x;
    }
    const double2 s = block_sum2<256>(t, t0, red);
    const double rho = 2.0 * s.x - s.y;
    const double thr = rel ? fmax(tr2 * rel[j], floor) : tr2;
    if (rho < thr) {  // block-uniform
      if (threadIdx.x == 0) conv[j] = 1;
      continue;
    }
    const double beta = (iter == 1) ? 0.0 : rho / rho_prev[j];
    __syncthreads();
    if (threadIdx.x == 0) rho_prev[j] = rho;
    for (int i = threadIdx.x; i < npw; i += 256) {
      const double w = ip[i];
      const C gv = gj[i];
      const double hx = (double)gv.x * w, hy = (double)gv.y * w;
      if (iter == 1) {
        pj[i] = mkc<C>(T(-hx), T(-hy));
      } else {
        const C pv = pj[i];
        pj[i] = mkc<C>(T(fma(beta, (double)pv.x, -hx)), T(fma(beta, (double)pv.y, -hy)));
      }
    }
  }
}

// Grid of a per-system launch: one CTA per system; with a device count nmax
// bounds it (the CTAs beyond the count return at once).
static int sys_grid(int nmax, const int*) { return nmax; }

void cg_prec_rho(const int* act, int nact, const double2* g, double2* P, const double* iprec, int nocc,
                 double* rho_prev, unsigned char* conv, int iter, double tr2, int npw, long ld, cudaStream_t s,
                 const int* dn, const int* iter_dev) {
  if (nact <= 0) return;
  k_cg_prec_rho<double2><<<sys_grid(nact, dn), 256, 0, s>>>(act, dn, g, P, iprec, nocc, rho_prev, conv, iter, iter_dev,
                                                           tr2, nullptr, 0.0, npw, ld);
}
void cg_prec_rho32(const int* act, int nact, const float2* g, float2* P, const double* iprec, int nocc,
                   double* rho_prev, unsigned char* conv, int iter, double eta, const double* rel, double floor,
                   int npw, long ld, cudaStream_t s, const int* dn, const int* iter_dev) {
  if (nact <= 0) return;
  k_cg_prec_rho<float2><<<sys_grid(nact, dn), 256, 0, s>>>(act, dn, g, P, iprec, nocc, rho_prev, conv, iter, iter_dev,
                                                          eta, rel, floor, npw, ld);
}

// Active list in increasing system order (map_lbnd2ibnd, :356-382) and the
// Gamma FFT pairs (act[2k], act[2k+1]); one block of NT threads.  Returns the
// count in every thread.
template <int NT>
WB_DEV int compact_block(const unsigned char* conv, int nsys, int* act, int2* items, int* nact_out) {
  __shared__ int wsum[NT / 32];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  int base = 0;
  for (int c0 = 0; c0 < nsys; c0 += NT) {
    const int i = c0 + tid;
    const bool f = (i < nsys) && !__ldcg(conv + i);
    const unsigned bal = __ballot_sync(0xffffffffu, f);
    if (lane == 0) wsum[w] = __popc(bal);
    __syncthreads();
    int off = base, all = base;
    for (int q = 0; q < NT / 32; ++q) {
      if (q < w) off += wsum[q];
      all += wsum[q];
    }
    if (f) act[off + __popc(bal & ((1u << lane) - 1u))] = i;
    base = all;
    __syncthreads();
  }
  for (int k = tid; k < (base + 1) / 2; k += NT)
    items[k] = make_int2(act[2 * k], (2 * k + 1 < base) ? act[2 * k + 1] : -1);
  if (tid == 0) *nact_out = base;
  return base;
}
__global__ void __launch_bounds__(1024) k_cg_compact(const unsigned char* __restrict__ conv, int nsys_host,
                                                     const int* nsys_dev, int* act, int2* __restrict__ items,
                                                     int* __restrict__ nact_out) {
  compact_block<1024>(conv, dev_count(nsys_dev, nsys_host), act, items, nact_out);
}
void cg_compact(const unsigned char* conv, int nsys, int* act, int2* items, int* nact_dev, int* nact_host,
                cudaStream_t s, const int* nsys_dev) {
  k_cg_compact<<<1, 1024, 0, s>>>(conv, nsys, nsys_dev, act, items, nact_dev);
  if (nact_host) cudaMemcpyAsync(nact_host, nact_dev, sizeof(int), cudaMemcpyDeviceToHost, s);
}


// End of one PCG pass of the graph-captured loop, by the last CTA of the step
// kernel to finish: the active list of the next pass and, with ctl, the pass's
// counters and the loop test of k_loop_bucket and k_loop_ctl (a loop of one
// bucket needs no kernel of its own for either).
struct CgTail {
  int* ticket = nullptr;  // null: no tail; zero between launches
  const int* nsys = nullptr;
  int* act = nullptr;
  int2* items = nullptr;
  int* nact = nullptr;
  int* st = nullptr;
  cudaGraphConditionalHandle cond = 0;
  int ctl = 0, inner = 0;
};

WB_DEV void loop_count(int* st, int n) {
  if (n <= 0) return;
  *reinterpret_cast<long long*>(st + 4) += n;
  *reinterpret_cast<long long*>(st + 6) += 2 * ((n + 1) / 2);
  st[3] += 1;
}
WB_DEV void loop_test(cudaGraphConditionalHandle h, int n, int* st, int maxiter, int inner) {
  const int it = st[1];
  const bool more = n > 0 && it < maxiter;
  if (!inner && !more) st[2] = st[3] + (n == 0 ? 1 : 0);
  if (more) st[1] = it + 1;
  cudaGraphSetConditional(h, more ? 1u : 0u);
}

// Two sums over the block, then over the cluster's CTAs in rank order: the same
// bits in every thread of every CTA.  cl: [2][2] shared slots, used in turn (a
// CTA is never two reductions ahead of one that still reads).
template <int NT, int CS>
WB_DEV double2 cluster_sum2(double a, double b, double* red, double* cl, int& turn) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  constexpr int NW = NT / 32;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) { red[2 * w] = a; red[2 * w + 1] = b; }
  __syncthreads();
  a = l < NW ? red[2 * l] : 0.0;
  b = l < NW ? red[2 * l + 1] : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if constexpr (CS > 1) {
    double* slot = cl + 2 * turn;
    turn ^= 1;
    if (threadIdx.x == 0) { slot[0] = a; slot[1] = b; }
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    const unsigned mine = (unsigned)__cvta_generic_to_shared(slot);
    a = b = 0.0;
#pragma unroll
    for (int r = 0; r < CS; ++r) {
      unsigned peer;
      double pa, pb;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(mine), "r"(r));
      asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(pa) : "r"(peer) : "memory");
      asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(pb) : "r"(peer + 8) : "memory");
      a += pa;
      b += pb;
    }
  }
  return make_double2(a, b);
}

// One PCG step after the operator, in one kernel: the update of iteration
// `iter` (a = <P|g>, c = <P|T> with the Gamma dot, x -= a/c P, g -= a/c T;
// linsolve_sternheimer_m_wfcts.f90:253-329) and, unless iter == maxiter,
// iteration iter + 1's preconditioning, rho, test and direction (as
// k_cg_prec_rho: h = M g, rho = <h|g>, P = -h + rho/rho_prev P).
// One cluster of CS CTAs per system, each with its slice of the plane waves; the
// new g is preconditioned and its rho summed in the update's own pass, and the
// later passes re-read P, T and g (just written) from L1 and L2.
template <class C, int NT, int CS>
__global__ void __launch_bounds__(NT) k_cg_step(const int* act, const int* dn, int nhost,
                                                C* __restrict__ x, C* __restrict__ g, C* __restrict__ P,
                                                const C* __restrict__ T, const double* __restrict__ iprec, int nocc,
                                                double* rho_prev, unsigned char* conv, int iter_host,
                                                const int* iter_dev, int maxiter, double tr2,
                                                const double* __restrict__ rel, double floor, int npw, long ld,
                                                CgTail tail) {
  using R = real_t<C>;
  __shared__ double red[NT / 16];
  __shared__ double cl[4];
  __shared__ int last;
  const int n = dev_count(dn, nhost);
  const int iter = iter_dev ? *iter_dev : iter_host;
  const bool prec = iter + 1 <= maxiter;  // the reference leaves its loop before this preconditioning otherwise
  const int rank = CS > 1 ? (int)blockIdx.x % CS : 0;
  const int slice = (npw + CS - 1) / CS, lo = rank * slice, hi = min(npw, lo + slice);
  int turn = 0;
  for (int b = blockIdx.x / CS; b < n; b += gridDim.x / CS) {
    const int j = act[b];
    const C* tj = T + (long)j * ld;
    C* pj = P + (long)j * ld;
    C* gj = g + (long)j * ld;
    C* xj = x + (long)j * ld;
    const double* ip = iprec + (long)(j % nocc) * npw;
    const double rho_last = rho_prev[j];  // read before the reductions, after which rank 0 rewrites it
    double a = 0.0, c = 0.0;
    for (int i = lo + threadIdx.x; i < hi; i += NT) {
      const C p = pj[i], gv = gj[i], tv = tj[i];
      double da = fma((double)p.x, (double)gv.x, (double)p.y * (double)gv.y);
      double dc = fma((double)p.x, (double)tv.x, (double)p.y * (double)tv.y);
      if (i == 0) { da -= 0.5 * (double)p.x * (double)gv.x; dc -= 0.5 * (double)p.x * (double)tv.x; }
      a += da;
      c += dc;
    }
    const double2 s = cluster_sum2<NT, CS>(a, c, red, cl, turn);
    const R r = R((2.0 * s.x) / (2.0 * s.y));
    double tt = 0.0, t0 = 0.0;
    for (int i = lo + threadIdx.x; i < hi; i += NT) {
      const C p = pj[i], tv = tj[i];
      const C xv = xj[i], gv = gj[i];
      xj[i] = mkc<C>(fma(-r, p.x, xv.x), fma(-r, p.y, xv.y));
      const C gn = mkc<C>(fma(-r, tv.x, gv.x), fma(-r, tv.y, gv.y));
      gj[i] = gn;
      if (prec) {
        const double w = ip[i];
        const double hx = (double)gn.x * w, hy = (double)gn.y * w;
        tt = fma(hx, (double)gn.x, fma(hy, (double)gn.y, tt));
        if (i == 0) t0 = hx * (double)gn.x;
      }
    }
    if (!prec) continue;
    const double2 s2 = cluster_sum2<NT, CS>(tt, t0, red, cl, turn);
    const double rho = 2.0 * s2.x - s2.y;
    const double thr = rel ? fmax(tr2 * rel[j], floor) : tr2;
    if (rho < thr) {  // cluster-uniform
      if (rank == 0 && threadIdx.x == 0) conv[j] = 1;
      continue;
    }
    const double beta = rho / rho_last;  // iteration iter + 1 >= 2
    if (rank == 0 && threadIdx.x == 0) rho_prev[j] = rho;
    for (int i = lo + threadIdx.x; i < hi; i += NT) {
      const double w = ip[i];
      const C gv = gj[i], pv = pj[i];
      const double hx = (double)gv.x * w, hy = (double)gv.y * w;
      pj[i] = mkc<C>(R(fma(beta, (double)pv.x, -hx)), R(fma(beta, (double)pv.y, -hy)));
    }
  }
  if constexpr (CS > 1)  // no CTA leaves while another of its cluster may read its sums
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  if (!tail.ticket) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(tail.ticket, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int nn = compact_block<NT>(conv, *tail.nsys, tail.act, tail.items, tail.nact);
  if (threadIdx.x == 0) {
    *tail.ticket = 0;
    if (tail.ctl) {
      loop_count(tail.st, n);
      loop_test(tail.cond, nn, tail.st, maxiter, tail.inner);
    }
  }
}

// Threads per CTA and CTAs per system.  The choice and with it the order of the sums
// depends on the count's bucket alone (bucket_systems), not on the workspace's capacity
// or on how many systems are left of a bucket, so that a call has the same bits
// whatever ran on its context before, captured or not.  Measured on one B200, us a step:
//   up to 64 systems, 512 threads: the slices' serial passes are the time.  64^3 (8,440
//     plane waves) 24 systems FP64 12.8 with 4 CTAs, 16.9 with 2, 19.9 with 1; 64
//     systems 17.0, 16.9 and 20.8 (4 CTAs of 1024 threads 25.6: two waves).  Below
//     4,096 plane waves one CTA: 2,400 plane waves, 64 systems 8.8, with 4 CTAs 10.8.
//   more systems, one CTA each, while the systems in flight keep their four vectors in
//     L2 between the passes: two CTAs of 512 threads per SM up to 80 MB of vectors (256
//     systems FP64: 2,400 plane waves 12.9, one CTA of 1024 threads 17.0; 4,000 18.9 and
//     21.4; FP32: 5,200 16.9 and 21.0, 8,440 25.1 and 27.2, 10,500 38.2 and 39.4, but 1,024
//     systems of 8,440 150 and 143, of 10,500 206 and 174), then one of 1,024.
//   then the fewest CTAs per system with which one CTA per SM keeps to 96 MB.  2,048
//     systems FP64: 8,440 plane waves 437 with 1 CTA, 571 with 2; 16,900 1,085, 1,010 with
//     2, 1,325 with 4; 37,387 2,506, 2,649 and 2,396 with 4.  FP32: 16,900 566 with 1 and
//     642 with 2, 37,387 1,583 with 1, 1,373 with 2 and 1,604 with 4.
struct CgShape {
  int threads, ctas;
};
static CgShape cg_shape(int n, int npw, int elem) {
  if (npw <= 1024) return {256, 1};
  const int systems = bucket_systems(n);
  if (systems <= kBucketSystems && npw >= 4096) return {512, 4};
  const double vectors = 4.0 * elem * npw;
  if (vectors * 2 * sm_count() <= 80e6) return {512, 1};
  int cs = 1;
  while (cs < 8 && vectors * std::min(systems, sm_count() / cs) > 96e6) cs *= 2;
  return {1024, cs};
}
template <class C, int NT, int CS, class... A>
static void cg_step_launch(int nact, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  // one CTA per system: a persistent grid, so that no more systems than fit L2 are in flight
  cfg.gridDim = dim3(CS == 1 ? std::min(nact, sm_count() * (1024 / NT)) : nact * CS);
  cfg.blockDim = dim3(NT);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = CS;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = CS > 1 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k_cg_step<C, NT, CS>, args...);
}
static CgTail cg_tail(const CgLoop* l) {
  CgTail t;
  if (!l) return t;
  t.ticket = l->st + 8;
  t.nsys = l->st;
  t.act = l->act;
  t.items = l->items;
  t.nact = l->nact;
  t.st = l->st;
  t.cond = l->cond;
  t.ctl = l->ctl;
  t.inner = l->inner;
  return t;
}
template <class C>
static void cg_step_t(const int* act, int n, C* x, C* g, C* P, const C* T, const double* iprec, int nocc,
                      double* rho_prev, unsigned char* conv, int iter, int maxiter, double tr2, const double* rel,
                      double floor, int npw, long ld, cudaStream_t s, const int* dn, const int* iter_dev,
                      const CgLoop* loop) {
  if (n <= 0) return;
  const CgShape sh = cg_shape(n, npw, sizeof(C));
  auto go = [&](auto launch) {
    launch(n, s, act, dn, n, x, g, P, T, iprec, nocc, rho_prev, conv, iter, iter_dev, maxiter, tr2, rel, floor, npw,
           ld, cg_tail(loop));
  };
#define WB_STEP(NT, CS) \
  if (sh.threads == NT && sh.ctas == CS) return go([](int m, cudaStream_t q, auto... a) { cg_step_launch<C, NT, CS>(m, q, a...); })
  WB_STEP(256, 1);
  WB_STEP(512, 1);
  WB_STEP(512, 4);
  WB_STEP(1024, 1);
  WB_STEP(1024, 2);
  WB_STEP(1024, 4);
  WB_STEP(1024, 8);
#undef WB_STEP
}
void cg_step(const int* act, int nact, double2* x, double2* g, double2* P, const double2* T, const double* iprec,
             int nocc, double* rho_prev, unsigned char* conv, int iter, int maxiter, double tr2, int npw, long ld,
             cudaStream_t s, const int* dn, const int* iter_dev, const CgLoop* loop) {
  cg_step_t<double2>(act, nact, x, g, P, T, iprec, nocc, rho_prev, conv, iter, maxiter, tr2, nullptr, 0.0, npw, ld, s,
                     dn, iter_dev, loop);
}
void cg_step32(const int* act, int nact, float2* x, float2* g, float2* P, const float2* T, const double* iprec,
               int nocc, double* rho_prev, unsigned char* conv, int iter, int maxiter, double eta, const double* rel,
               double floor, int npw, long ld, cudaStream_t s, const int* dn, const int* iter_dev,
               const CgLoop* loop) {
  cg_step_t<float2>(act, nact, x, g, P, T, iprec, nocc, rho_prev, conv, iter, maxiter, eta, rel, floor, npw, ld, s, dn,
                    iter_dev, loop);
}

// ---------------------------------------------------------------------------
// FP64 iterative refinement around the FP32 PCG (mixed form)
// ---------------------------------------------------------------------------
// R = B - T (FP64); rho = <M^-1 R|R>_Gamma; converged if rho < tr2 (the test of
// linsolve_sternheimer_m_wfcts.f90:215-216 on the true FP64 residual).
// Otherwise the FP32 correction solve starts from d = 0 with g = -R.
__global__ void __launch_bounds__(256) k_refine_residual(const int* __restrict__ act, const double2* __restrict__ B,
                                                         const double2* __restrict__ T,
                                                         const double* __restrict__ iprec, int nocc, double tr2,
                                                         unsigned char* conv, double* rho0, float2* __restrict__ g32,
                                                         float2* __restrict__ d32, int npw, long ld) {
  __shared__ double red[16];
  const int j = act[blockIdx.x];
  const double2* bj = B + (long)j * ld;
  const double2* tj = T + (long)j * ld;
  const double* ip = iprec + (long)(j % nocc) * npw;
  double t = 0.0, t0 = 0.0;
  for (int i = threadIdx.x; i < npw; i += 256) {
    const double2 b = bj[i], a = tj[i];
    const double rx = b.x - a.x, ry = b.y - a.y;
    const double w = ip[i];
    t = fma(rx * w, rx, fma(ry * w, ry, t));
    if (i == 0) t0 = rx * w * rx;
  }
  const double2 s = block_sum2<256>(t, t0, red);
  const double rho = 2.0 * s.x - s.y;
  const bool c = rho < tr2;
  if (threadIdx.x == 0) { conv[j] = c ? 1 : 0; rho0[j] = rho; }
  if (c) return;
  float2* gj = g32 + (long)j * ld;
  float2* dj = d32 + (long)j * ld;
  for (int i = threadIdx.x; i < npw; i += 256) {
    const double2 b = bj[i], a = tj[i];
    gj[i] = make_float2((float)(a.x - b.x), (float)(a.y - b.y));
    dj[i] = make_float2(0.f, 0.f);
  }
}
void refine_residual(const int* act, int nact, const double2* B, const double2* T, const double* iprec, int nocc,
                     double tr2, unsigned char* conv, double* rho0, float2* g32, float2* d32, int npw, long ld,
                     cudaStream_t s) {
  if (nact <= 0) return;
  k_refine_residual<<<nact, 256, 0, s>>>(act, B, T, iprec, nocc, tr2, conv, rho0, g32, d32, npw, ld);
}

// x += d for the listed columns
__global__ void k_refine_accumulate(const int* __restrict__ act, double2* __restrict__ X,
                                    const float2* __restrict__ d32, int npw, long ld) {
  const int j = act[blockIdx.y];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npw; i += gridDim.x * blockDim.x) {
    const float2 d = d32[(long)j * ld + i];
    double2 x = X[(long)j * ld + i];
    X[(long)j * ld + i] = make_double2(x.x + (double)d.x, x.y + (double)d.y);
  }
}
void refine_accumulate(const int* act, int nact, double2* X, const float2* d32, int npw, long ld, cudaStream_t s) {
  if (nact <= 0) return;
  k_refine_accumulate<<<dim3((npw + 255) / 256, nact), 256, 0, s>>>(act, X, d32, npw, ld);
}

// FP32 T = g2kin P (Im at G=0 zeroed) - e P for the kinetic-only operator
__global__ void k_kinetic_hpsi32(const float2* __restrict__ P, float2* __restrict__ T, const float* __restrict__ g2kin,
                                 const float* __restrict__ ecol, const int* __restrict__ cols, const int* dn, int npw,
                                 long ld) {
  if ((int)blockIdx.y >= dev_count(dn, gridDim.y)) return;
  const int c = cols ? cols[blockIdx.y] : blockIdx.y;
  const float e = ecol[c];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npw; i += gridDim.x * blockDim.x) {
    const float2 p = P[(long)c * ld + i];
    float2 h = make_float2(p.x * g2kin[i], p.y * g2kin[i]);
    if (i == 0) h.y = 0.f;
    T[(long)c * ld + i] = make_float2(fmaf(-e, p.x, h.x), fmaf(-e, p.y, h.y));
  }
}
void kinetic_hpsi32(const float2* P, float2* T, const float* g2kin, const float* ecol, const int* cols, int ncol,
                    int npw, long ld, cudaStream_t s, const int* dn) {
  if (ncol <= 0) return;
  k_kinetic_hpsi32<<<dim3((npw + 255) / 256, ncol), 256, 0, s>>>(P, T, g2kin, ecol, cols, dn, npw, ld);
}

__global__ void k_to_float(const double* __restrict__ a, float* __restrict__ b, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) b[i] = (float)a[i];
}
void to_float(const double* a, float* b, long n, cudaStream_t s) {
  if (n <= 0) return;
  k_to_float<<<(int)std::min<long>((n + 255) / 256, 4096), 256, 0, s>>>(a, b, n);
}

// ---------------------------------------------------------------------------
// FP32 bra-ket GEMMs of the inner solve (SIMT FFMA, shared-memory tiles)
// ---------------------------------------------------------------------------
// part[s][j][r] = sum_{k in split s} W[r][k] X[col j][k]; tile 64 r x 64 j, k step 16
__global__ void __launch_bounds__(256) k_gemm_tn_f32(const float* __restrict__ W, long ldw, int M,
                                                     const float* __restrict__ X, long ldx,
                                                     const int* __restrict__ cols, int ncol_host, const int* dn,
                                                     int K, int kchunk, float* __restrict__ part) {
  __shared__ float Ws[16][64 + 4];
  __shared__ float Xs[16][64 + 4];
  const int ncol = dev_count(dn, ncol_host);
  const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  const int r0 = blockIdx.x * 64, j0 = blockIdx.y * 64, split = blockIdx.z;
  if (j0 >= ncol) return;
  const int kb = split * kchunk, ke = min(K, kb + kchunk);
  float acc[4][4] = {};
  // loader: 64 rows x 8 float2 per operand, two per thread
  const int lrow = tid / 8, lk = (tid % 8) * 2;
  const float* wrow[2];
  const float* xrow[2];
  bool wok[2], xok[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = r0 + lrow + 32 * h;
    wok[h] = r < M;
    wrow[h] = W + (long)(wok[h] ? r : 0) * ldw;
    const int j = j0 + lrow + 32 * h;
    xok[h] = j < ncol;
    const int cj = xok[h] ? (cols ? cols[j] : j) : 0;
    xrow[h] = X + (long)cj * ldx;
  }
  for (int k0 = kb; k0 < ke; k0 += 16) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = k0 + lk;
      float2 wv = make_float2(0.f, 0.f), xv = make_float2(0.f, 0.f);
      if (wok[h] && k < ke) wv = *reinterpret_cast<const float2*>(wrow[h] + k);
      if (xok[h] && k < ke) xv = *reinterpret_cast<const float2*>(xrow[h] + k);
      Ws[lk][lrow + 32 * h] = wv.x; Ws[lk + 1][lrow + 32 * h] = wv.y;
      Xs[lk][lrow + 32 * h] = xv.x; Xs[lk + 1][lrow + 32 * h] = xv.y;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { a[i] = Ws[kk][ty * 4 + i]; b[i] = Xs[kk][tx * 4 + i]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(a[i], b[q], acc[i][q]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = r0 + ty * 4 + i, j = j0 + tx * 4 + q;
      if (r < M && j < ncol) part[((long)split * ncol + j) * M + r] = acc[i][q];
    }
}

int gemm_tn_splits32(int M, int ncol, int K) {
  const int tiles = ((M + 63) / 64) * ((ncol + 63) / 64);
  int ns = (2 * 148 * 2 + tiles - 1) / tiles;
  const int maxs = (K + 511) / 512;
  if (ns > maxs) ns = maxs;
  if (ns < 1) ns = 1;
  return ns;
}

void gemm_tn32(const float* W, long ldw, int M, const float* X, long ldx, const int* cols, int ncol, int K, int nsplit,
               float* part, cudaStream_t s, const int* dn) {
  if (ncol <= 0 || M <= 0) return;
  int kchunk = (K + nsplit - 1) / nsplit;
  kchunk = (kchunk + 15) / 16 * 16;
  dim3 grid((M + 63) / 64, (ncol + 63) / 64, nsplit);
  k_gemm_tn_f32<<<grid, 256, 0, s>>>(W, ldw, M, X, ldx, cols, ncol, dn, K, kchunk, part);
}

// Y[col j][k] += sum_r W[r][k] C[j][r]; tile 128 k x 32 j, r step 16
__global__ void __launch_bounds__(256) k_gemm_nn_f32(const float* __restrict__ W, long ldw, int M,
                                                     const float* __restrict__ C, float* __restrict__ Y, long ldy,
                                                     const int* __restrict__ cols, int ncol_host, const int* dn,
                                                     int K) {
  __shared__ float Ws[16][128 + 4];
  __shared__ float Cs[16][32 + 1];
  const int ncol = dev_count(dn, ncol_host);
  const int tid = threadIdx.x, tx = tid % 32, ty = tid / 32;
  const int k0 = blockIdx.x * 128, j0 = blockIdx.y * 32;
  if (j0 >= ncol) return;
  float acc[4][4] = {};  // [k i][j q]: k = k0 + tx*4 + i, j = j0 + ty*4 + q
  for (int rb = 0; rb < M; rb += 16) {
    for (int e = tid; e < 16 * 64; e += 256) {           // W tile: 16 r x 64 float2
      const int rr = e / 64, kk = (e % 64) * 2;
      const int r = rb + rr, k = k0 + kk;
      float2 v = make_float2(0.f, 0.f);
      if (r < M && k < K) v = *reinterpret_cast<const float2*>(W + (long)r * ldw + k);
      Ws[rr][kk] = v.x; Ws[rr][kk + 1] = v.y;
    }
    for (int e = tid; e < 16 * 32; e += 256) {           // C tile: 16 r x 32 j
      const int rr = e % 16, jj = e / 16;
      const int r = rb + rr, j = j0 + jj;
      Cs[rr][jj] = (r < M && j < ncol) ? C[(long)j * M + r] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int rr = 0; rr < 16; ++rr) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { a[i] = Ws[rr][tx * 4 + i]; b[i] = Cs[rr][ty * 4 + i]; }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[i][q] = fmaf(a[i], b[q], acc[i][q]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int j = j0 + ty * 4 + q;
    if (j >= ncol) continue;
    const int col = cols ? cols[j] : j;
    float* y = Y + (long)col * ldy;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = k0 + tx * 4 + i;
      if (k < K) y[k] += acc[i][q];
    }
  }
}
void gemm_nn32_acc(const float* W, long ldw, int M, const float* C, float* Y, long ldy, const int* cols, int ncol, int K,
                   cudaStream_t s, const int* dn) {
  if (ncol <= 0 || M <= 0) return;
  dim3 grid((K + 127) / 128, (ncol + 31) / 32);
  k_gemm_nn_f32<<<grid, 256, 0, s>>>(W, ldw, M, C, Y, ldy, cols, ncol, dn, K);
}

// ---------------------------------------------------------------------------
// device-side loop control of the graph-captured PCG loops
// ---------------------------------------------------------------------------
// st[0] systems of the batch, st[1] iteration of the next pass, st[2] last
// iteration run, st[3] inner iterations run over all refinements (mixed form);
// st[4..5] active system-iterations and st[6..7] FFT boxes (64-bit counters);
// st[8] ticket of the step kernel's last CTA (zero between launches).
__global__ void k_loop_init(int* st, int nsys, int reset_totals) {
  st[0] = nsys;
  st[1] = 1;
  st[2] = 0;
  st[8] = 0;
  if (reset_totals) {
    st[3] = 0;
    *reinterpret_cast<long long*>(st + 4) = 0;
    *reinterpret_cast<long long*>(st + 6) = 0;
  }
}
void loop_init(int* st, int nsys, bool reset_totals, cudaStream_t s) {
  k_loop_init<<<1, 1, 0, s>>>(st, nsys, reset_totals ? 1 : 0);
}

// End of one PCG pass (operator, update of iteration st[1] and the
// preconditioning of iteration st[1] + 1, active list): linsolve's loop over
// iter = 1..n_dfpt_maxiter, left when no system is active
// (linsolve_sternheimer_m_wfcts.f90:146,222); every FP32 correction solve of
// the mixed form is bounded the same way.  Sets the WHILE condition of the
// graph; for the FP64 loop (inner = 0) it leaves the reference's iteration
// count in st[2]: the passes that did work, plus the one whose test found no
// system left.
__global__ void k_loop_ctl(cudaGraphConditionalHandle h, const int* nact, int* st, int maxiter, int inner) {
  loop_test(h, *nact, st, maxiter, inner);
}
void loop_ctl(cudaGraphConditionalHandle h, const int* nact, int* st, int maxiter, bool inner, cudaStream_t s) {
  k_loop_ctl<<<1, 1, 0, s>>>(h, nact, st, maxiter, inner ? 1 : 0);
}

// Start of a pass: counts the pass's work (st[3] passes with active systems,
// their active-system and FFT-item sums) and sets the SWITCH value: the
// smallest bucket k with min_items << k >= the active band-pair items (last
// bucket: the workspace capacity).
__global__ void k_loop_bucket(cudaGraphConditionalHandle h, const int* nact, int* st, int min_items, int nbuckets) {
  const int n = *nact;
  loop_count(st, n);
  const int items = (n + 1) / 2;
  int k = 0;
  while (k < nbuckets - 1 && (min_items << k) < items) ++k;
  cudaGraphSetConditional(h, (unsigned)k);
}
void loop_bucket(cudaGraphConditionalHandle h, const int* nact, int* st, int min_items, int nbuckets, cudaStream_t s) {
  k_loop_bucket<<<1, 1, 0, s>>>(h, nact, st, min_items, nbuckets);
}

__global__ void k_count_unconverged(const unsigned char* __restrict__ conv, int nocc, int mb, int* __restrict__ out) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= mb) return;
  int n = 0;
  for (int v = 0; v < nocc; ++v) n += conv[(long)p * nocc + v] ? 0 : 1;
  out[p] = n;
}
void count_unconverged(const unsigned char* conv, int nocc, int mb, int* out, cudaStream_t s) {
  if (mb <= 0) return;
  k_count_unconverged<<<(mb + 127) / 128, 128, 0, s>>>(conv, nocc, mb, out);
}

}  // namespace wb
