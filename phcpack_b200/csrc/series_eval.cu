// series_eval.cu -- batched evaluation and differentiation of polynomial
// systems at truncated power series (the Polynomials layer of PHCpack's GPU
// code, Polynomials/dbl2_polynomials_kernels.cu:1577, batched over systems).
//
// Two arrangements.  A warp per polynomial: one CTA per (system, group of up
// to 8 polynomials); the CTA stages the system's input series in shared
// memory (coalesced 16-byte loads), each warp keeps its monomial's forward
// and backward products in its own shared-memory slots and accumulates the
// polynomial's value and gradient rows in the output buffer, which it owns.
// A CTA per polynomial, for few polynomials: the warps share its monomials
// and the rows are summed in shared memory in the monomials' order.
//
// Bound by the FP64 pipe and the latency of its operations.  1024 systems
// (n = 32, 32 monomials, degree 31, complex double-double): 37.4 ms with the
// multiple-double operators, 29.9 with open accumulators (md::macc), 28.5
// with two-variable monomials in three products instead of four, 24.2 with
// one inlined product per kernel in chunks of three terms, 22.0 with the
// squares of the variables at hand: 77 % of the FP64 pipe's rate.  At 16 warps per SM; 24 (80 registers) measured 4 % slower, 8
// with 153 registers 25 %.
#include "common.cuh"
#include "series_eval.cuh"

namespace phc {

static const int kMaxWarpsPerBlock = 8;
static const int kMaxSmem = 227 * 1024;
static const int kSquareDims = 256;  // variables whose squares may be kept
// Polynomials up to which a CTA takes one: 8 warps each, so that one wave of
// CTAs still gives every SM 8 polynomials.  One system of 8 polynomials of 12
// monomials (degree 15, complex double-double): 68 us shared, 332 with a warp
// per polynomial; 512 polynomials at degree 95: 1.04 ms against 2.7.
// A monomial of one variable is one product (in double also two variables
// are little work): there the CTA's staging and summing outweigh the shared
// products beyond two CTAs per SM (960 polynomials of 6 one-variable
// monomials in double: 35 us shared, 33 with a warp per polynomial).
static const long kSplitPolys = 148 * 8, kSplitPolysShort = 148 * 2;

// Input series of a system, n doubles, into shared memory.
__device__ __forceinline__ void stage_inputs(const double *__restrict__ xin, double *Xs, int n) {
  if ((n & 1) == 0 && (reinterpret_cast<unsigned long long>(xin) & 15) == 0) {
    const double2 *src = reinterpret_cast<const double2 *>(xin);
    double2 *dst = reinterpret_cast<double2 *>(Xs);
    for (int i = threadIdx.x; i < n / 2; i += blockDim.x) dst[i] = src[i];
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) Xs[i] = xin[i];
  }
}

// The squares of the variables that have an exponent above 2 in the monomials
// m0..m1-1, into sq (dim series): a product each, one less wherever they
// occur.  Null when a coefficient of X (all variables, so that it does not
// depend on the polynomials of the CTA) is below 2^-400 or above 2^500: a
// square could leave the range, or lose lower limbs at its end, where c x x
// does not.  X in shared memory.  Called by the whole CTA; the caller
// synchronises before they are read.  (Which variables those are is marked in
// the squares' own places: static shared memory would count against the
// launches without squares too, whose scratch may take all there is.)
template <class N, bool BIG>
__device__ const double *needed_squares(int dim, int deg, int maxvar, int m0, int m1, const int *__restrict__ nvr,
                                        const int *__restrict__ idx, const int *__restrict__ exps, const double *X,
                                        double *sq) {
  const int S = (deg + 1) * N::width;
  for (int i = threadIdx.x; i < dim; i += blockDim.x) sq[i * S] = 0.0;
  __syncthreads();  // and X is in place
  bool outside = false;
  for (int i = threadIdx.x; i < dim * (deg + 1) * (N::width / N::tr::limbs); i += blockDim.x) {
    const double a = fabs(X[i * N::tr::limbs]);
    outside = outside || !(a == 0.0 || (a >= 0x1p-400 && a <= 0x1p500));
  }
  if (__syncthreads_or(outside)) return nullptr;
  for (int m = m0 + threadIdx.x; m < m1; m += blockDim.x) {
    const int k = nvr[m];
    if (k < 1 || k > maxvar) continue;
    for (int v = 0; v < k; ++v) {
      const int i = idx[(long)m * maxvar + v];
      if (i >= 0 && i < dim && exps[(long)m * maxvar + v] > 2) sq[i * S] = 1.0;
    }
  }
  __syncthreads();
  const typename wser<N, BIG>::map map(deg, threadIdx.x & 31, 0);
  for (int i = threadIdx.x >> 5; i < dim; i += blockDim.x >> 5) {
    if (sq[i * S] == 0.0) continue;
    const typename N::T z = wser<N, BIG>::conv(X + i * S, X + i * S, map);
    if (map.valid) md::stn(sq + i * S + map.kout() * N::width, z);
  }
  return sq;
}

// A warp per polynomial.  BIG (degrees 32..191): one more scratch series per
// warp (the value); the inputs are staged in shared memory when they fit
// beside the scratch and read from global memory otherwise.
template <class N, bool BIG>
__global__ void __launch_bounds__(kMaxWarpsPerBlock * 32, N::width <= 4 ? 2 : 1)
    k_system_evaldiff(int dim, int deg, int maxvar, int wpb, int stage, int squares, const int *__restrict__ mon_off,
                      const int *__restrict__ nvr, const int *__restrict__ idx, const int *__restrict__ exps,
                      const double *__restrict__ cst, const double *__restrict__ cff,
                      const double *__restrict__ input, double *__restrict__ output) {
  extern __shared__ __align__(16) double sm[];
  const int S = (deg + 1) * N::width;
  const int bps = (dim + wpb - 1) / wpb;
  const int s = blockIdx.x / bps;
  const int p0 = (blockIdx.x % bps) * wpb;
  const double *X = input + (long)s * dim * S;
  double *scr = sm;
  if (stage) {
    stage_inputs(X, sm, dim * S);
    X = sm;
    scr = sm + ((dim * S + 1) & ~1);
  }
  const int warp = threadIdx.x >> 5;
  const int p = p0 + warp;
  const long sp = (long)s * dim + p;
  const double *X2 = nullptr;
  if (squares) {
    X2 = needed_squares<N, BIG>(dim, deg, maxvar, mon_off[(long)s * dim + p0], mon_off[(long)s * dim + min(p0 + wpb, dim)],
                                nvr, idx, exps, X, scr);
    scr += (dim * S + 1) & ~1;
  }
  __syncthreads();
  if (p >= dim) return;
  scr += (long)warp * (warp_slots(maxvar) + (BIG ? 1 : 0)) * S;
  warp_poly_evaldiff<N, BIG>(dim, deg, maxvar, mon_off[sp], mon_off[sp + 1], nvr, idx, exps, cst + sp * S, cff, X, X2,
                             scr, output + sp * (dim + 1) * S);
}

// A CTA per polynomial, its monomials shared by the warps.
template <class N, bool BIG>
__global__ void __launch_bounds__(kMaxWarpsPerBlock * 32, N::width <= 4 ? 2 : 1)
    k_poly_evaldiff(int dim, int deg, int maxvar, int stage, int squares, const int *__restrict__ mon_off,
                    const int *__restrict__ nvr, const int *__restrict__ idx, const int *__restrict__ exps,
                    const double *__restrict__ cst, const double *__restrict__ cff, const double *__restrict__ input,
                    double *__restrict__ output) {
  extern __shared__ __align__(16) double sm[];
  const int S = (deg + 1) * N::width;
  const long sp = blockIdx.x;
  const double *X = input + (sp / dim) * dim * S;
  double *rows = sm;
  double *scr = sm + (((dim + 1) * S + 1) & ~1);
  if (stage) {
    stage_inputs(X, scr, dim * S);
    X = scr;
    scr += (dim * S + 1) & ~1;
  }
  const double *X2 = nullptr;
  if (squares) {
    X2 = needed_squares<N, BIG>(dim, deg, maxvar, mon_off[sp], mon_off[sp + 1], nvr, idx, exps, X, scr);
    scr += (dim * S + 1) & ~1;
  }
  __syncthreads();
  cta_poly_evaldiff<N, BIG>(dim, deg, maxvar, mon_off[sp], mon_off[sp + 1], nvr, idx, exps, cst + sp * S, cff, X, X2,
                            scr, rows, output + sp * (dim + 1) * S);
}

template <class N>
static int launch_system(int nsys, int dim, int deg, int maxvar, const int *mon_off, const int *nvr, const int *idx,
                         const int *exps, const double *cst, const double *cff, const double *input, double *output,
                         cudaStream_t stream) {
  const int S = (deg + 1) * N::width;
  const bool big = deg > 31;  // series longer than a warp
  const long series = (long)S * sizeof(double);
  const long xs = (long)((dim * S + 1) & ~1) * sizeof(double);
  // The squares of the variables beside the inputs, for short series, while
  // two CTAs of the built-in shape still share an SM (1024 systems n = 32
  // with exponents up to 3: one in nine products saved, 24.2 -> 22.2 ms;
  // exponents up to 2: 20.2 -> 20.5).  Decided by the sizes alone, so that
  // every arrangement forms the same products.
  const long warp8 = (dim < kMaxWarpsPerBlock ? dim : kMaxWarpsPerBlock) * (long)warp_slots(maxvar) * series;
  const int squares = !big && dim <= kSquareDims && warp8 + 2 * xs + 1024 <= 114 * 1024;
  // A warp per polynomial leaves most of the GPU idle on a few systems, and
  // each warp's products follow one another.  While the polynomials are
  // fewer than kSplitPolys a CTA takes one polynomial and shares its
  // monomials among its warps, when the rows fit in shared memory.  (Whatever
  // knob 0 says: it sizes the CTAs of the other arrangement, and what was
  // found for a large batch must not send the small ones there.)
  const bool short_work = maxvar == 1 || (maxvar == 2 && N::tr::limbs == 1);
  if ((long)nsys * dim <= (short_work ? kSplitPolysShort : kSplitPolys)) {
    const long per_warp = (warp_slots(maxvar) + maxvar + 1) * series;
    const long rows = (long)(((dim + 1) * S + 1) & ~1) * sizeof(double);
    int nw = kMaxWarpsPerBlock;
    const long fixed = rows + (squares ? 2 * xs : 0);
    while (nw > 2 && fixed + nw * per_warp > kMaxSmem - 1024) --nw;
    long smem = fixed + nw * per_warp;
    if (smem <= kMaxSmem - 1024) {
      const int stage = squares || smem + xs <= 200 * 1024;
      if (stage && !squares) smem += xs;
      auto kern = big ? k_poly_evaldiff<N, true> : k_poly_evaldiff<N, false>;
      PHC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      kern<<<(unsigned)(nsys * dim), nw * 32, smem, stream>>>(dim, deg, maxvar, stage, squares, mon_off, nvr, idx, exps,
                                                               cst, cff, input, output);
      PHC_CHECK_LAUNCH();
      return PHC_OK;
    }
  }
  // one warp per polynomial, up to 8 per CTA; monomials with many variables
  // need many scratch series per warp, so fewer warps share a CTA when the
  // shared memory would not hold the scratch of 8; the inputs are staged in
  // shared memory when they fit beside the scratch
  const long per_warp = (warp_slots(maxvar) + (big ? 1 : 0)) * series;
  int wpb = dim < kMaxWarpsPerBlock ? dim : kMaxWarpsPerBlock;
  const int tuned = tune_get(kTuneEvalWarps);  // warps per CTA chosen by the autotuner
  if (tuned > 0) wpb = tuned < dim ? tuned : dim;
  while (wpb > 1 && (long)wpb * per_warp > kMaxSmem) --wpb;
  const long scr = (long)wpb * per_warp;
  int stage = (scr + xs) <= 200 * 1024;
  const long smem = scr + (stage ? xs : 0) + (squares ? xs : 0);
  if (smem > kMaxSmem) {
    set_error("system_evaldiff: %ld bytes of shared memory needed (maxvar %d, degree %d)", smem, maxvar, deg);
    return PHC_ERR_LIMIT;
  }
  auto kern = big ? k_system_evaldiff<N, true> : k_system_evaldiff<N, false>;
  PHC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int bps = (dim + wpb - 1) / wpb;
  const long grid = (long)nsys * bps;
  kern<<<(unsigned)grid, wpb * 32, smem, stream>>>(dim, deg, maxvar, wpb, stage, squares, mon_off, nvr, idx, exps, cst, cff,
                                                   input, output);
  PHC_CHECK_LAUNCH();
  return PHC_OK;
}

int system_evaldiff(int prec, int cplx, int nsys, int dim, int deg, int maxvar, const int *mon_off, const int *nvr,
                    const int *idx, const int *exps, const double *cst, const double *cff, const double *input,
                    double *output, cudaStream_t stream) {
  PHC_REQUIRE(prec_ok(prec), "system_evaldiff: precision %d not in {1,2,4}", prec);
  PHC_REQUIRE(nsys >= 0 && dim >= 1 && deg >= 0 && maxvar >= 1, "system_evaldiff: bad sizes");
  if (deg > 191) {
    set_error("system_evaldiff: degree %d > 191", deg);
    return PHC_ERR_LIMIT;
  }
  if (nsys == 0) return PHC_OK;
  PHC_REQUIRE(mon_off && nvr && idx && exps && cst && cff && input && output, "system_evaldiff: null pointer");
#define PHC_SYS(R, C) \
  return launch_system<md::num<R, C> >(nsys, dim, deg, maxvar, mon_off, nvr, idx, exps, cst, cff, input, output, stream)
  if (!cplx) {
    if (prec == 1) PHC_SYS(double, false);
    if (prec == 2) PHC_SYS(md::dd, false);
    PHC_SYS(md::qd, false);
  } else {
    if (prec == 1) PHC_SYS(double, true);
    if (prec == 2) PHC_SYS(md::dd, true);
    PHC_SYS(md::qd, true);
  }
#undef PHC_SYS
}

}  // namespace phc
