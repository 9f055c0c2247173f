// Internal interfaces between the west_b200 host code and its kernels.
#pragma once
#include <cuda_runtime.h>

#include <vector>

namespace wb {

// Stick decomposition of the Gamma half sphere (built on the host from nl).
constexpr int kZGroup = 8;  // stick pairs per CTA of the z passes
struct StickTab {
  int nsp;               // stick pairs; pair 0 is the (0,0) stick
  int nst;               // sticks in the buffer = 2 * hs
  int hs;                // stick side * hs + q is side 0 or 1 of pair q (hs >= nsp)
  const int* sp_gstart;  // [nsp + 1] first internal G index of each pair
  const int2* g_qz;      // [npw] (2 * pair + side, signed z) of each internal G
  int gmax;              // most G vectors of kZGroup consecutive pairs from a multiple of it
  const int* zlo;        // [nsp] lowest z of each pair (its coefficients are a run of side 0)
  const int* zmap;       // null, or where pairs have no such runs: [pair][z] 2 g + flip, -1 = none (z_lookup)
  const int* cmap;       // [y][active column] stick at (x, y), -1 = none
  int xhi;               // active plane columns: x in [0, xhi] and [N - (ncols - xhi - 1), N)
  int ncols;
  int prune;             // 1 if every |Miller index| < N/4 (sphere inside the outer quarters)
};

// Runtime-size transforms (boxes without a compiled edge: non-cubic boxes and
// the other 2, 3, 5, 7-smooth edges).  A line of length n is transformed in
// place by radix stages r[0..ns) (each 2, 3, 4, 5, 7 or 8): the inverse as
// decimation in frequency (natural input, output at digit-reversed positions),
// the forward as decimation in time over the same stages in reverse order
// (digit-reversed input, natural output).  Real-space data therefore sit at
// digit-reversed positions in every direction; they are only ever multiplied
// point by point, with V(r) stored in the same permuted layout.
// Boxes whose x and y edges split as a * b with radices up to 16 and whose full
// plane fits in shared memory run the plane phases of wb_plane.cuh instead, with
// the splits and twiddles below taken at run time (real space is then [pz][x][ys]).
constexpr int kRtMaxEdge = 160;
struct RtFast {
  int ax = 0, bx = 0, ay = 0, by = 0, max_radix = 0;
  double2 tx[kRtMaxEdge], ty[kRtMaxEdge];  // W_n^(k1 n2) at k1 b + n2
  float2 tx32[kRtMaxEdge], ty32[kRtMaxEdge];
};
// the split of an edge (0, 0 if it has none)
void rt_split(int n, int* a, int* b);
constexpr int kRtMaxStages = 16;
struct RtPlan {
  int n, ns;
  int r[kRtMaxStages];
};
struct RtGeo {
  int nx, ny, nz;            // box edges, x fastest
  RtPlan px, py, pz;
  int ncols;                 // active x columns of a plane (the sticks' x values)
  int cs;                    // column stride of the shared-memory half plane (>= ny, odd)
  const int* colx;           // [ncols] box x index of active column c
  const int* spos;           // [nst] half-plane offset c * cs + (y mod ny) of each stick, -1 = dummy
  const double2 *twx, *twy, *twz;  // exp(+2 pi i j / n) per direction
  const float2 *twx32, *twy32, *twz32;
  const RtFast* fast;        // host pointer; null: the staged kernels
};
// radix stages of n (empty if n has a prime factor above 7)
RtPlan rt_plan(int n);
// box index in a direction of the value stored at position p by the inverse
int rt_digit_reverse(const RtPlan& pl, int p);
// fills f and returns true if the box runs the phases of wb_plane.cuh
bool rt_fast_setup(int nx, int ny, RtFast* f);
// shared memory of the runtime plane kernels for the given geometry and element size
size_t rt_plane_smem(const RtGeo& g, int elem_bytes, int* rows_per_chunk);

// Launches that take a device count (dcount != nullptr, CUDA-graph replays)
// size their grid for the host count as a maximum and read the number of
// systems from *dcount; items are pairs of systems.
struct FftArgs {
  int n;                 // box edge (0 when the runtime-size path runs)
  StickTab st;
  const double2* tw;     // [n] step factors W_n^(k1 n2) at k1 N2 + n2 (wb_fft.cuh)
  cudaStream_t stream;
  const int* dcount = nullptr;
  const RtGeo* rt = nullptr;  // runtime-size path when set
};

// FP32 twin of FftArgs for the mixed-precision inner solves.
struct FftArgs32 {
  int n;
  StickTab st;
  const float2* tw;
  cudaStream_t stream;
  const int* dcount = nullptr;
  const RtGeo* rt = nullptr;
};

// runtime-size counterparts of the fft_* entry points below (f.rt set)
void rt_zinv(const FftArgs& f, const double2* src, long ld, const int2* items, int nitems, double2* sticks);
void rt_zinv32(const FftArgs32& f, const float2* src, long ld, const int2* items, int nitems, float2* sticks);
void rt_zfwd_store(const FftArgs& f, const double2* sticks, const int2* items, int nitems, double2* dst, long ld);
void rt_zfwd_hpsi(const FftArgs& f, const double2* sticks, const int2* items, int nitems, const double2* P,
                  double2* T, long ld, const double* g2kin, const double* ecol);
void rt_zfwd_hpsi32(const FftArgs32& f, const float2* sticks, const int2* items, int nitems, const float2* P,
                    float2* T, long ld, const float* g2kin, const float* ecol);
void rt_zfwd_dng(const FftArgs& f, const double2* sticks, const int2* items, int nitems, double2* dng, long ld,
                 const int* perm, const double* sqvc);
void rt_plane_vloc(const FftArgs& f, double2* sticks, int nitems, const double* vs);
void rt_plane_vloc32(const FftArgs32& f, float2* sticks, int nitems, const float* vs);
void rt_plane_inv_box(const FftArgs& f, const double2* sticks, int nitems, double2* box);
void rt_plane_rhs(const FftArgs& f, const double2* evcr, const double2* dvbox, int npv, int mb, double2* sticks);
void rt_plane_drho(const FftArgs& f, const double2* dsticks, const double2* evcr, const double* occ, int nocc,
                   int mb, double2* acc, double scale, double2* osticks);
void rt_setup();

// SMs of the current device
int sm_count();

bool fft_supported(int n);
// the split n = a * b of a compiled edge's line transforms: the plane kernels
// keep y = k1 + a k2 of real space at row b k1 + k2 (0, 0 for other edges)
void fft_split(int n, int* a, int* b);
// out[z][x][ys] = in[z][y][x] / div, ys = b (y mod a) + y / a: the plane
// kernels' real-space layout (wb_plane.cuh)
void plane_layout(const double* in, double* out, int nx, int ny, int nz, int a, int b, double div, cudaStream_t s);

// Davidson restart hand-off in WEST's layout (Wstat/davidson_restart.f90):
// <dir>/summary.json (dav_iter, notcnv, nbase, conv, ev, ew), <dir>/hr_vr.dat
// (Fortran unformatted: hr then vr, n_pdep_basis^2 doubles each) and the basis
// <dir>/V<j>.dat, N<j>.dat (j = 000001.., pdep file format) for j <= nbase.
// dvg/dng are host arrays [ld, nbase] complex in WEST's G order.
struct DavRestart {
  int dav_iter = 0, notcnv = 0, nbase = 0;
  std::vector<int> conv;
  std::vector<double> ev, ew, hr, vr;
};
int dav_restart_write(const char* dir, const DavRestart& r, int nvec, int nvecx, int npw, const double* dvg,
                      const double* dng, long ld);
int dav_restart_read(const char* dir, DavRestart& r, int nvec, int nvecx, int npw, double* dvg, double* dng,
                     long ld);
void dav_restart_clear(const char* dir, int nvecx);
void fft_zinv32(const FftArgs32& f, const float2* src, long ld, const int2* items, int nitems, float2* sticks);
void fft_plane_vloc32(const FftArgs32& f, float2* sticks, int nitems, const float* vs);
void fft_zfwd_hpsi32(const FftArgs32& f, const float2* sticks, const int2* items, int nitems, const float2* P,
                     float2* T, long ld, const float* g2kin, const float* ecol);
void fft_setup(int n);
void fft_zinv(const FftArgs& f, const double2* src, long ld, const int2* items, int nitems, double2* sticks);
void fft_zfwd_store(const FftArgs& f, const double2* sticks, const int2* items, int nitems, double2* dst, long ld);
void fft_zfwd_hpsi(const FftArgs& f, const double2* sticks, const int2* items, int nitems, const double2* P,
                   double2* T, long ld, const double* g2kin, const double* ecol);
void fft_zfwd_dng(const FftArgs& f, const double2* sticks, const int2* items, int nitems, double2* dng, long ld,
                  const int* perm, const double* sqvc);
void fft_plane_vloc(const FftArgs& f, double2* sticks, int nitems, const double* vs);
void fft_plane_inv_box(const FftArgs& f, const double2* sticks, int nitems, double2* box);
void fft_plane_rhs(const FftArgs& f, const double2* evcr, const double2* dvbox, int npv, int mb, double2* sticks);
void fft_plane_drho(const FftArgs& f, const double2* dsticks, const double2* evcr, const double* occ, int nocc,
                    int mb, double2* acc, double scale, double2* osticks);

// ---- dense kernels (wb_la.cu) ----
// part[s][j][r] = sum_{k in split s} W[r*ldw + k] * X[col(j)*ldx + k]
// The captured PCG loops have one branch per bucket of active systems: up to 64, 128,
// 256, ... (wb_api.cu, capture_loop).  bucket_systems: the bound of the bucket that
// serves n systems.  A captured launch is sized for that bound or, in the last bucket,
// for the workspace's capacity, an eager one for the live count: all three have the
// same bucket, so a launch shape that decides the order of a sum depends on it only.
constexpr int kBucketSystems = 64;
inline int bucket_systems(int n) {
  int b = kBucketSystems;
  while (b < n) b *= 2;
  return b;
}
// Split-K plans of the bra-ket GEMMs, host and device: a graph replay sizes its
// split grid for the largest plan and every CTA derives the plan of the device
// column count itself, so both paths split the same count the same way.
// gemm_tn_splits: splits of a caller with a fixed part buffer (about 2 * 148 *
// ctas_per_sm CTAs of 32 x 32 tiles, at least 512 k each).
__host__ __device__ inline int gemm_tn_splits(int M, int ncol, int K, int ctas_per_sm = 2) {
  const int tiles = ((M + 31) / 32) * ((ncol + 31) / 32);
  int ns = (2 * 148 * ctas_per_sm + tiles - 1) / (tiles > 0 ? tiles : 1);
  const int maxs = (K + 511) / 512;
  if (ns > maxs) ns = maxs;
  if (ns < 1) ns = 1;
  return ns;
}
// k's of one split: a multiple of the pair width and of 16
__host__ __device__ inline int gemm_tn_chunk(int K, int nsplit) { return ((K + nsplit - 1) / nsplit + 15) / 16 * 16; }
// gemm_tn_plan: splits of the PCG's bra-kets.  At most 896 k each (32 splits of a long K),
// because a split's k's are one chain of additions per warp and its error grows with the
// root of the chain's length; at least 384, below which the partial sums cost more than
// the rounds saved, or 192 where the grid would otherwise leave half of the GPU's CTA
// slots empty and a CTA's latency is the time.  Between these bounds four CTAs per SM,
// then the first count of eight whose last round over 148 SMs is at least 95% full.
// Bra-ket and reduction over 460 shapes (8 to 2,048 columns, 16 to 288 rows, K from 400 to
// 74,774) stay within 1.9% of the best split on average, 9% at the 97th percentile.
__host__ __device__ inline int gemm_tn_plan(int M, int ncol, int K) {
  int tiles = ((M + 31) / 32) * ((ncol + 31) / 32);
  if (tiles < 1) tiles = 1;
  int lo = (K + 895) / 896, hi = K / 384;
  if (lo > 32) lo = 32;
  if (lo < 1) lo = 1;
  if (hi < lo) hi = lo;
  if (tiles * hi < 296) {
    const int fill = 296 / tiles < K / 192 ? 296 / tiles : K / 192;
    if (hi < fill) hi = fill;
  }
  int ns = 592 / tiles;
  if (ns < lo) ns = lo;
  if (ns > hi) ns = hi;
  int best = ns;
  long best_ctas = 0, best_rounds = 0;
  for (int t = ns; t < ns + 8 && t <= hi; ++t) {
    const long ctas = (long)tiles * t, rounds = (ctas + 147) / 148;
    if (rounds * 148 * 20 <= ctas * 21) return t;
    if (!best_ctas || rounds * best_ctas < best_rounds * ctas) { best = t; best_ctas = ctas; best_rounds = rounds; }
  }
  return best;
}
// the largest plan of any count that a captured launch of bound ncol serves
int gemm_tn_plan_max(int M, int ncol, int K);
// part doubles for any column count up to nsys
size_t gemm_tn_part_doubles(int M, int nsys, int K);
// with dn the kernel takes the plan of the device count (nsplit is then ignored)
void gemm_tn(const double* W, long ldw, int M, const double* X, long ldx, const int* cols, int ncol, int K,
             int nsplit, double* part, cudaStream_t s, const int* dn = nullptr);
// opts the GEMM kernels into their shared memory on the current device
void la_setup();
// S = 2 sum_s part - W0 X0 (Gamma bra-ket, glbrak.f90:39-40), then
// C[j][r] = sum_{r'<nkb} D[r][r'] S[j][r'] for r < nkb, alpha S[j][r] otherwise
void gamma_reduce(const double* part, int nsplit, int M, int ncol, const double* W, long ldw, const double* X,
                  long ldx, const int* cols, const double* D, int nkb, double alpha, double* C, cudaStream_t s,
                  const int* dn = nullptr, int K = 0);
// Y[col(j)] = beta Y[col(j)] + W C[j]  over K real rows
void gemm_nn(const double* W, long ldw, int M, const double* C, double* Y, long ldy, const int* cols, int ncol,
             int K, double beta, cudaStream_t s, const int* dn = nullptr);

void permute_scale(const double2* dvg, long ld_in, const int* perm, const double* sqvc, int npw, int m,
                   double2* aux, long ld_out, cudaStream_t s);
// iprec[v][i] = 1 / max(1, g2kin[i] / eprec[v])
void make_iprec(const double* g2kin, const double* eprec, int npw, int nocc, double* iprec, cudaStream_t s);
// column j uses band j % nocc
void precondition(const double2* f, double2* pf, const double* iprec, int nocc, int npw, int ncol, long ld,
                  cudaStream_t s);
void sub_into(const double2* a, const double2* b, double2* out, int npw, int ncol, long ld, cudaStream_t s);
void kinetic_hpsi(const double2* P, double2* T, const double* g2kin, const double* ecol, const int* cols, int ncol,
                  int npw, long ld, cudaStream_t s, const int* dn = nullptr);
void set_eprec(const double2* evc, const double* g2kin, int npw, int nocc, double* eprec, cudaStream_t s);
void fill_columns(const double* per_band, int nocc, int nsys, double* out, cudaStream_t s);
// Fractional occupations (dfpt_module.f90:363-393): from C[j][r] = <psi_r|dV psi_i>
// (j = p nocc + i, r < nocc) the coefficients fc[j][f] of the bands r = nfull + f:
// 0 for r <= i or |occ_i - occ_r| < 1e-3, else C (occ_i - occ_r) / occ_i / (e_i - e_r)
void frac_coefficients(const double* C, int nocc, int nsys, int nfull, const double* occ, const double* et,
                       double* fc, cudaStream_t s);
void cg_reset(unsigned char* conv, int nsys, cudaStream_t s);
void cg_prec_rho(const int* act, int nact, const double2* g, double2* P, const double* iprec, int nocc,
                 double* rho_prev, unsigned char* conv, int iter, double tr2, int npw, long ld, cudaStream_t s,
                 const int* dn = nullptr, const int* iter_dev = nullptr);
// nact_host may be null (no host copy); nsys_dev, if given, overrides nsys
void cg_compact(const unsigned char* conv, int nsys, int* act, int2* items, int* nact_dev, int* nact_host,
                cudaStream_t s, const int* nsys_dev = nullptr);
// Loop state a captured PCG pass hands to its step kernel (wb_la.cu, CgTail):
// the active list it rebuilds and, with ctl, the WHILE condition it sets.
struct CgLoop {
  int* act;
  int2* items;
  int* nact;
  int* st;  // int[kLoopInts]
  cudaGraphConditionalHandle cond;
  int ctl, inner;
};
constexpr int kLoopInts = 12;
// One PCG step after the operator: the update of iteration `iter` and, unless
// iter == maxiter, the preconditioning / rho / convergence test / direction of
// iteration iter + 1 (the iteration comes from *iter_dev when given); with loop,
// also the end of the pass.
void cg_step(const int* act, int nact, double2* x, double2* g, double2* P, const double2* T, const double* iprec,
             int nocc, double* rho_prev, unsigned char* conv, int iter, int maxiter, double tr2, int npw, long ld,
             cudaStream_t s, const int* dn = nullptr, const int* iter_dev = nullptr, const CgLoop* loop = nullptr);
void cg_step32(const int* act, int nact, float2* x, float2* g, float2* P, const float2* T, const double* iprec,
               int nocc, double* rho_prev, unsigned char* conv, int iter, int maxiter, double eta, const double* rel,
               double floor, int npw, long ld, cudaStream_t s, const int* dn = nullptr,
               const int* iter_dev = nullptr, const CgLoop* loop = nullptr);
void count_unconverged(const unsigned char* conv, int nocc, int mb, int* out, cudaStream_t s);
// loop state of the graph-captured PCG loops: int st[kLoopInts] (wb_la.cu)
void loop_init(int* st, int nsys, bool reset_totals, cudaStream_t s);
void loop_ctl(cudaGraphConditionalHandle h, const int* nact, int* st, int maxiter, bool inner, cudaStream_t s);
void loop_bucket(cudaGraphConditionalHandle h, const int* nact, int* st, int min_items, int nbuckets, cudaStream_t s);

// ---- mixed form: FP32 inner PCG and FP64 refinement (wb_la.cu) ----
// inner test: rho < max(eta * rel[j], floor)
void cg_prec_rho32(const int* act, int nact, const float2* g, float2* P, const double* iprec, int nocc,
                   double* rho_prev, unsigned char* conv, int iter, double eta, const double* rel, double floor,
                   int npw, long ld, cudaStream_t s, const int* dn = nullptr, const int* iter_dev = nullptr);
void refine_residual(const int* act, int nact, const double2* B, const double2* T, const double* iprec, int nocc,
                     double tr2, unsigned char* conv, double* rho0, float2* g32, float2* d32, int npw, long ld,
                     cudaStream_t s);
void refine_accumulate(const int* act, int nact, double2* X, const float2* d32, int npw, long ld, cudaStream_t s);
void kinetic_hpsi32(const float2* P, float2* T, const float* g2kin, const float* ecol, const int* cols, int ncol,
                    int npw, long ld, cudaStream_t s, const int* dn = nullptr);
void to_float(const double* a, float* b, long n, cudaStream_t s);
int gemm_tn_splits32(int M, int ncol, int K);
void gemm_tn32(const float* W, long ldw, int M, const float* X, long ldx, const int* cols, int ncol, int K, int nsplit,
               float* part, cudaStream_t s, const int* dn = nullptr);
void gamma_reduce32(const float* part, int nsplit, int M, int ncol, const float* W, long ldw, const float* X, long ldx,
                    const int* cols, const float* D, int nkb, float alpha, float* C, cudaStream_t s,
                    const int* dn = nullptr, int K = 0, int umma_ctas = 0);
void gemm_nn32_acc(const float* W, long ldw, int M, const float* C, float* Y, long ldy, const int* cols, int ncol, int K,
                   cudaStream_t s, const int* dn = nullptr);

// split-BF16x3 tcgen05 GEMMs of the FP32 inner solve (wb_umma.cu)
bool umma_supported(int M);
int umma_np(int M);
void umma_setup();
__host__ __device__ inline void umma_braket_plan(int ncol, int K, int* nsplit, int* kb_per_split,
                                                 int ctas_per_sm = 2) {
  const int nkb = (K + 63) / 64;
  int tiles = (ncol + 127) / 128;
  if (tiles < 1) tiles = 1;
  int target = (ctas_per_sm * 148 + tiles - 1) / tiles;
  if (target < 1) target = 1;
  int per = (nkb + target - 1) / target;
  if (per < 2) per = 2;
  if (per > nkb) per = nkb;
  *kb_per_split = per;
  *nsplit = (nkb + per - 1) / per;
}
// part floats for any batch up to nsys and any ctas_per_sm up to kUmmaMaxCtas
constexpr int kUmmaMaxCtas = 3;
size_t umma_part_floats(int M, int nsys, int K);
size_t umma_braket_bytes(int M, int K);
size_t umma_update_bytes(int M, int K);
void umma_presplit(const double* W, long ldw, int M, int K, void* braket_tiles, void* update_tiles, cudaStream_t s);
// part[s][j][r] = sum over split s of W[r][k] X[cols[j]][k]; returns the number of splits
int umma_braket(const void* tiles, int M, const float* X, long ldx, const int* cols, int ncol, int K, float* part,
                int* err, cudaStream_t s, const int* dn = nullptr, int ctas_per_sm = 2);
// Y[cols[j]][k] += sum_r W[r][k] C[j][r]
// nj: systems per CTA (64 or 128; 0 = by projector count)
void umma_update(const void* tiles, int M, const float* C, float* Y, long ldy, const int* cols, int ncol, int K,
                 int* err, cudaStream_t s, const int* dn = nullptr, int nj = 0);

}  // namespace wb
