// dense.cuh -- CTA-level multiple-double dense linear algebra: blocked
// Householder QR in WY form, inversion of the diagonal tiles of R and tiled
// back substitution, Q^H b, and the block lower-triangular Toeplitz solve of
// the power-series Newton step.
//
// One CTA owns one instance.  Matrices are row-major, limb-interleaved, in
// global memory (one instance's Q, R and WY panels stay resident in L2);
// shared memory holds the Householder vector, the reflector coefficients,
// the current solution vector and the reduction buffers.  Dot products are
// shared by groups of four or eight lanes; the norms of the skip rules are
// formed by every warp for itself.
#pragma once
#include "md.cuh"
#include "ozaki.cuh"

namespace phc {

template <class N>
__device__ __forceinline__ typename N::T ldn_at(const double *p, long i) {
  typename N::T a;
  md::ldn(p + i * N::width, a);
  return a;
}
template <class N>
__device__ __forceinline__ void stn_at(double *p, long i, const typename N::T &a) {
  md::stn(p + i * N::width, a);
}

template <class N>
__device__ __forceinline__ typename N::T warp_sum(typename N::T a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a = N::add(a, md::shfl_xor(a, o));
  return a;
}

__device__ __forceinline__ double warp_max(double a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a = fmax(a, __shfl_xor_sync(0xffffffffu, a, o));
  return a;
}

// Block-wide sum, every thread gets the result.  red: shared scratch of
// (blockDim/32) numbers of width N::width.
template <class N>
__device__ typename N::T block_sum(typename N::T a, double *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  a = warp_sum<N>(a);
  __syncthreads();
  if (lane == 0) stn_at<N>(red, warp, a);
  __syncthreads();
  typename N::T s = N::zero();
  for (int w = 0; w < nw; ++w) s = N::add(s, ldn_at<N>(red, w));
  __syncthreads();
  return s;
}

__device__ __forceinline__ double block_max(double a, double *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  a = warp_max(a);
  __syncthreads();
  if (lane == 0) red[warp] = a;
  __syncthreads();
  double s = 0.0;
  for (int w = 0; w < nw; ++w) s = fmax(s, red[w]);
  __syncthreads();
  return s;
}

// Block-wide minimum of one double per thread (any sign).
__device__ __forceinline__ double block_min(double a, double *red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a = fmin(a, __shfl_xor_sync(0xffffffffu, a, o));
  __syncthreads();
  if (lane == 0) red[warp] = a;
  __syncthreads();
  double s = red[0];
  for (int w = 1; w < nw; ++w) s = fmin(s, red[w]);
  __syncthreads();
  return s;
}

// max_i |leading limb| of v (complex: |re| + |im|): the "1-norm" of the
// reference's skip rules, Newton/dbl_onenorms_host.cpp:9,20.  Every warp
// forms it by itself (n is at most a few dozen: a CTA-wide reduction would
// cost three barriers for two loads per lane), so all threads get the result
// without a barrier.
template <class N>
__device__ __forceinline__ double warp_maxnorm(int n, const double *v) {
  double a = 0.0;
  for (int i = threadIdx.x & 31; i < n; i += 32) a = fmax(a, N::lead(ldn_at<N>(v, i)));
  return warp_max(a);
}

// Skip thresholds of the reference's least-squares solvers per precision:
// Newton/dbl_bals_host.cpp:36,199 (double: |b_0| + 1 == 1 in the head,
// 1e-15 in the tail), dbl2_bals_host.cpp:43,254 (1e-28),
// dbl4_bals_host.cpp:51,335 (1e-56).
template <class N>
__device__ __forceinline__ double skip_tol() {
  return N::tr::limbs == 1 ? 1.0e-15 : (N::tr::limbs == 2 ? 1.0e-28 : 1.0e-56);
}
template <class N>
__device__ __forceinline__ bool head_tiny(double nrm) {
  return N::tr::limbs == 1 ? (__dadd_rn(nrm, 1.0) == 1.0) : (nrm < skip_tol<N>());
}

// Shared-memory layout of one CTA (in doubles), sized by dense_smem_doubles.
struct dense_smem {
  double *v;     // Householder vector, n numbers
  double *w;     // n numbers: reflector products / right hand side
  double *x;     // n numbers: solution of one stage
  double *beta;  // szt reals (as numbers of width N::width)
  double *red;   // reduction scratch, 32 numbers
  double *misc;  // 8 numbers
};

template <class N>
__device__ dense_smem carve(double *sm, int n, int szt) {
  const int W = N::width;
  dense_smem s;
  s.v = sm;
  s.w = s.v + n * W;
  s.x = s.w + n * W;
  s.beta = s.x + n * W;
  s.red = s.beta + szt * W;
  s.misc = s.red + 32 * W;
  return s;
}
__host__ __device__ inline long dense_smem_doubles(int n, int szt, int W) { return (long)(3 * n + szt + 40) * W; }
// with the WY panels (Y, W, P, T) and the current column panel of R staged
// in shared memory as well
__host__ __device__ inline long dense_smem_doubles_staged(int n, int szt, int W) {
  return dense_smem_doubles(n, szt, W) + 5L * n * szt * W;
}

// Workspace in global memory per instance (numbers): Y, W, P (szt x n each),
// T (n x szt) and the inverted diagonal tiles of R (n x szt).
__host__ __device__ inline long dense_work_numbers(int n, int szt) { return 5L * n * szt; }

// Dot products shared by aligned groups of four lanes: output o of a pass
// is computed by the four lanes 4(o mod 8) .. +3 of warp o / 8, each summing
// every fourth term, then two xor shuffles add the four partial sums (the
// chains of dependent multiple-double operations are a quarter as long as
// with one thread per output).  All lanes of a warp take part in every pass.
template <class N>
__device__ __forceinline__ typename N::T group4_sum(typename N::T a) {
  a = N::add(a, md::shfl_xor(a, 1));
  return N::add(a, md::shfl_xor(a, 2));
}

// The same with groups of 8 lanes, for long chains.
template <class N>
__device__ __forceinline__ typename N::T group_sum(typename N::T a, int lanes) {
  a = group4_sum<N>(a);
  return lanes == 8 ? N::add(a, md::shfl_xor(a, 4)) : a;
}

// sum += (conj) a_l b_l over l = l0, l0 + step, ... < n with a at stride lda
// and b at stride ldb (numbers); the next pair is loaded before the products
// of the present one (rows of A and Q come from L2 or memory, 300 to 1000
// cycles away).  CONJ: conj(a); NEG: -a.
template <class N, bool CONJ, bool NEG>
__device__ __forceinline__ void dot_acc(md::msum<N> &sum, const double *a, long lda, const double *b, long ldb, int l0,
                                        int step, int n) {
  typedef typename N::T T;
  if (l0 >= n) return;
  T x = ldn_at<N>(a, (long)l0 * lda), y = ldn_at<N>(b, (long)l0 * ldb);
#pragma unroll 1
  for (int l = l0; l < n; l += step) {
    const int nl = l + step < n ? l + step : l;
    const T xn = ldn_at<N>(a, (long)nl * lda), yn = ldn_at<N>(b, (long)nl * ldb);
    if (CONJ)
      sum.cfma(x, y);
    else if (NEG)
      sum.fnma(x, y);
    else
      sum.fma(x, y);
    x = xn;
    y = yn;
  }
}

// ------------------------------------------------------------- Householder
// One column of a panel: the reflector of x = R[c.., c], m = n - c entries,
// in PHCpack's convention (Matrices/dbl2_factorizations.cpp:374 real, :436
// complex): v[0] = 1, beta = 2|v0|^2/(sigma + |v0|^2); the real case takes
// v0 = x0 - mu or -sigma/(x0 + mu), the complex case v0 = x0 - mu x0/|x0|;
// and R[c.., c..e) <- (I - beta v v^H) R[c.., c..e), w_j = beta sum_i
// conj(R_ij) v_i, R_ij -= v_i conj(w_j) (:534/:567).
//
// A reflector is a chain of dependent scalar operations (a square root and
// two divisions, most of a quad-double column's time) between two sweeps
// over the panel.  With v = (1, x_i / v0) the inner products split into
// conj(R_cj) + (1/v0) D_j, D_j = sum_{i>c} conj(R_ij) x_i, and D_c is sigma
// itself: the first sweep needs nothing of the chain and also replaces the
// norm's reduction, and the warps 0 and 1 form beta and 1/v0 side by side.
// Four barriers per column.
//
// Where sigma or x0 is near an end of the range the first sweep is done again
// with the column scaled by 2^-E, the power of two above the largest x_i below
// the diagonal (exact): unscaled, sigma and the D_j lose their lower limbs,
// and 1/v0 overflows, where small x_i stand below an x0 of order one.  (All
// columns scaled gives the same bits, at 5 to 10 % of a double or
// double-double QR.)  A column is left alone (beta = 0) where the reference's
// beta is zero: when the squares of all x_i underflow, or the square of v0
// does.
//
// Entry (i, j) of R sits at Rm[(i - r0) * ld + (j - c0)]: the whole matrix
// (r0 = c0 = 0, ld = ncols) or a panel of it staged in shared memory.  Leaves
// v in S.v (m numbers) and beta in S.misc[0] (a real number).
static const int kReflectUnder = -537;  // the square of a number below 2^-537 underflows

// High word of the larger of |re| and |im| of number i at p: orders numbers by
// size, a NaN above all.
template <class N>
__device__ __forceinline__ unsigned lead_word(const double *p, long i) {
  p += i * N::width;
  const unsigned a = (unsigned)__double2hiint(p[0]) & 0x7fffffffu;
  return N::is_complex ? max(a, (unsigned)__double2hiint(p[N::tr::limbs]) & 0x7fffffffu) : a;
}
// Exponent E of the scale of a column, mx and x0 the high words of its largest
// entry below the diagonal and of the diagonal one: the entries are below 2^E,
// and E is not so far below x0's that x0's square would overflow.
__device__ __forceinline__ int reflect_exponent(unsigned mx, unsigned x0) {
  if (mx == 0u) return 0;
  return max(min((int)(mx >> 20) - 1022, 1000), max((int)(x0 >> 20) - 1322, -1000));
}
__device__ __forceinline__ double pow2(int e) {  // 0 when it would not be a normal number
  return e < -1022 ? 0.0 : __hiloint2double((1023 + e) << 20, 0);
}
// every limb times a power of two
__device__ __forceinline__ double mul_pow2(double a, double s) { return __dmul_rn(a, s); }
__device__ __forceinline__ md::dd mul_pow2(const md::dd &a, double s) {
  return md::mk(__dmul_rn(a.hi, s), __dmul_rn(a.lo, s));
}
__device__ __forceinline__ md::qd mul_pow2(const md::qd &a, double s) {
  return md::mkq(__dmul_rn(a.x[0], s), __dmul_rn(a.x[1], s), __dmul_rn(a.x[2], s), __dmul_rn(a.x[3], s));
}
template <class R>
__device__ __forceinline__ md::cx<R> mul_pow2(const md::cx<R> &a, double s) {
  md::cx<R> r;
  r.re = mul_pow2(a.re, s);
  r.im = mul_pow2(a.im, s);
  return r;
}

// D_j for the nc columns from col's on, rows 1..m-1 of col, into w (D_0 =
// sigma); SCALED: with x 2^-E for x, down = 2^-E.  4 lanes per column, 8 when
// the columns are few and long.
template <class N, bool SCALED>
__device__ __forceinline__ void reflect_sums(int m, int nc, long ld, const double *col, double *w, double down) {
  typedef typename N::T T;
  const int G = (nc * 8 <= (int)blockDim.x && m > 16) ? 8 : 4;
  const int grp = threadIdx.x / G, part = threadIdx.x % G, ngrp = blockDim.x / G;
  for (int base = 0; base < nc; base += ngrp) {
    const int j = base + grp;
    md::msum<N> sum;
    sum.zero();
    if (j < nc)
      for (int i = 1 + part; i < m; i += G) {
        T x = ldn_at<N>(col, (long)i * ld), r = ldn_at<N>(col, (long)i * ld + j);
        if (SCALED) {
          x = mul_pow2(x, down);
          if (j == 0) r = x;
        }
        sum.cfma(r, x);
      }
    const T d = group_sum<N>(sum.value(), G);
    if (j < nc && part == 0) stn_at<N>(w, j, d);
  }
}

// beta (into misc[0]) and 1/v0 (into misc[2]) from sigma (w[0]) and x0 by the
// warps 0 and 1 side by side; SCALED: of the column times 2^-E.  Unscaled,
// misc[4] says whether sigma or x0 is near an end of the range.
template <class N, bool SCALED>
__device__ __forceinline__ void reflect_scalars(int m, const double *col, const double *w, double *misc, int E) {
  typedef typename N::T T;
  typedef typename N::real R;
  typedef md::num<R, false> RN;
  const int warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  if (warp >= 2) return;
  T x0 = ldn_at<N>(col, 0);
  if (SCALED) x0 = mul_pow2(x0, pow2(-E));
  R sigma;
  {
    const T d0 = ldn_at<N>(w, 0);
    if constexpr (N::is_complex)
      sigma = d0.re;
    else
      sigma = d0;
  }
  const bool do_beta = warp == 0, do_inv = warp == 1 || nwarp == 1;
  if (!SCALED && do_beta && (threadIdx.x & 31) == 0) {
    const double sig = md::lead(sigma);
    misc[4 * N::width] = (m == 1 || (sig >= 0x1p-120 && sig <= 0x1p600 && N::lead(x0) <= 0x1p400)) ? 0.0 : 1.0;
  }
  R beta = RN::zero();
  T inv = N::one();
  if (!md::is_zero(sigma) && !(SCALED && md::lead(sigma) < pow2(2 * (kReflectUnder - E)))) {
    T v0 = N::zero();
    if constexpr (N::is_complex) {
      const R sq0 = N::norm2(x0);
      const R rad0 = RN::tr::sqrt(sq0);
      R mu = RN::tr::sqrt(RN::add(sq0, sigma));
      if (md::is_zero(rad0)) {
        v0 = N::mkc(RN::neg(mu), RN::zero());
      } else {
        mu = RN::tr::div(mu, rad0);
        v0 = N::mkc(RN::sub(x0.re, RN::mul(mu, x0.re)), RN::sub(x0.im, RN::mul(mu, x0.im)));
      }
      const R v0sq = N::norm2(v0);
      const bool under = SCALED && md::lead(v0sq) < pow2(2 * (kReflectUnder - E));
      if (do_beta && !under) beta = md::mul_d(RN::tr::div(v0sq, RN::add(sigma, v0sq)), 2.0);
      if (do_inv) inv = N::mkc(RN::tr::div(v0.re, v0sq), RN::neg(RN::tr::div(v0.im, v0sq)));
    } else {
      const R mu = RN::tr::sqrt(RN::add(RN::mul(x0, x0), sigma));
      const bool cancel = !(md::lead(x0) <= 0.0);  // x0 - mu would cancel
      const R a = cancel ? RN::add(x0, mu) : RN::sub(x0, mu);
      const bool under = SCALED && cancel && md::lead(sigma) < __dmul_rn(md::lead(a), pow2(kReflectUnder - E));
      // sigma + v0^2 = -2 mu v0, so that beta = -v0 / mu: one division
      // beside the other warp's, none of them waiting for another
      if (do_inv) inv = cancel ? RN::neg(RN::tr::div(a, sigma)) : RN::tr::div(RN::one(), a);
      if (do_beta && !under) beta = cancel ? RN::tr::div(sigma, RN::mul(a, mu)) : RN::neg(RN::tr::div(a, mu));
    }
  }
  if ((threadIdx.x & 31) == 0) {
    if (do_beta) stn_at<RN>(misc, 0, beta);
    if (do_inv) stn_at<N>(misc + 2 * N::width, 0, inv);
  }
}

// The sums and scalars again with the column's scale; returns E (0 for a
// column of zeros below the diagonal: they stand).  Out of line: columns that
// need it are rare, and its code would take the others' instruction cache.
template <class N>
__device__ __noinline__ int reflect_rescaled(int m, int nc, long ld, const double *col, double *w, double *misc) {
  unsigned mx = 0u;  // the scale, by every warp for itself
  for (int i = 1 + (threadIdx.x & 31); i < m; i += 32) mx = max(mx, lead_word<N>(col, (long)i * ld));
  const int E = reflect_exponent(__reduce_max_sync(0xffffffffu, mx), lead_word<N>(col, 0));
  if (E == 0) return 0;
  reflect_sums<N, true>(m, nc, ld, col, w, pow2(-E));
  __syncthreads();
  reflect_scalars<N, true>(m, col, w, misc, E);
  __syncthreads();
  return E;
}

template <class N>
__device__ void block_reflect(int n, long ld, int c, int e, double *Rm, dense_smem &S, int r0, int c0) {
  typedef typename N::T T;
  typedef typename N::real R;
  typedef md::num<R, false> RN;
  const int m = n - c, nc = e - c;
  double *col = Rm + ((long)(c - r0) * ld + (c - c0)) * N::width;  // entry (c, c)
  reflect_sums<N, false>(m, nc, ld, col, S.w, 1.0);
  __syncthreads();
  reflect_scalars<N, false>(m, col, S.w, S.misc, 0);
  __syncthreads();
  int E = 0;
  if (S.misc[4 * N::width] != 0.0) E = reflect_rescaled<N>(m, nc, ld, col, S.w, S.misc);
  const R beta = ldn_at<RN>(S.misc, 0);
  const bool trivial = md::is_zero(beta);
  // v (as the reference leaves it when there is nothing to reflect) and w
  {
    const T inv = ldn_at<N>(S.misc + 2 * N::width, 0);
    for (int t = threadIdx.x; t < m + nc; t += blockDim.x) {
      if (t < m) {
        T v = N::one();
        if (t > 0) {
          v = ldn_at<N>(col, (long)t * ld);
          if (!trivial) v = N::mul(E != 0 ? mul_pow2(v, pow2(-E)) : v, inv);
        }
        stn_at<N>(S.v, t, v);
      } else if (!trivial) {
        const int j = t - m;
        const T dj = ldn_at<N>(S.w, j);  // D_j 2^-E, at j = 0 sigma 4^-E
        const T d = md::mul_add<N>(N::conj(ldn_at<N>(col, j)), inv, j == 0 && E != 0 ? mul_pow2(dj, pow2(E)) : dj);
        stn_at<N>(S.w, j, N::scale(d, beta));
      }
    }
  }
  __syncthreads();
  if (trivial) return;
  for (int t = threadIdx.x; t < m * nc; t += blockDim.x) {
    const int i = t / nc, j = t - i * nc;
    const long o = (long)i * ld + j;
    stn_at<N>(col, o, md::mul_sub<N>(ldn_at<N>(col, o), ldn_at<N>(S.v, i), N::conj(ldn_at<N>(S.w, j))));
  }
  __syncthreads();
}

// ------------------------------------------------------------- blocked QR
// A = Q R with Q n x n and R n x ncols (row-major), ncols = szt*nbt <= n.
// Matrices/dbl2_baqr_host.cpp:728 and dbl2_baqr_kernels.cu:3520: per tile
// the szt reflectors are applied to the panel column by column, then
// W = -B (I + W Y^H) Y column by column (:13), the trailing columns get
// R <- R + Y (W^H R) and Q <- Q + (Q W) Y^H.  R must hold A on entry.
// work: the WY panels Y, W, the product P and T (4 n szt numbers), in
// shared memory when the kernel staged them there, else in the instance's
// global workspace; panel: shared memory for the current column panel of R
// (n szt numbers: rows rowoff.., the tile's szt columns), or nullptr to
// factor the panel in place in global memory.  With OZ (real numbers only)
// the four trailing products run as Ozaki-split products on the FP64 tensor
// cores (ozaki.cuh) with the scratch oz (ozaki_work_doubles, global);
// complex numbers keep the CUDA-core products.
template <class N, bool OZ = false>
__device__ void block_houseqr(int n, int ncols, int szt, double *Q, double *Rm, double *work, double *oz,
                              dense_smem &S, double *panel = nullptr) {
  typedef typename N::T T;
  typedef typename N::real R;
  typedef md::num<R, false> RN;
  const int W = N::width;
  double *Y = work;                         // szt x n
  double *Wm = Y + (long)szt * n * W;       // szt x n
  double *P = Wm + (long)szt * n * W;       // szt x n
  double *Tm = P + (long)szt * n * W;       // n x szt
  const int nbt = ncols / szt;
  for (int t = threadIdx.x; t < n * n; t += blockDim.x) {
    const int i = t / n, j = t % n;
    stn_at<N>(Q, t, (i == j) ? N::one() : N::zero());
  }
  __syncthreads();
  for (int k = 0; k < nbt; ++k) {
    const int rowoff = k * szt;
    const int m = n - rowoff;
    const int endcol = (k + 1) * szt;
    if (panel) {  // the tile's columns, rows rowoff.., into shared memory
      for (int t = threadIdx.x; t < m * szt; t += blockDim.x)
        stn_at<N>(panel, t, ldn_at<N>(Rm, (long)(rowoff + t / szt) * ncols + rowoff + t % szt));
      __syncthreads();
    }
    for (int L = 0; L < szt; ++L) {
      const int c = rowoff + L;
      if (panel)
        block_reflect<N>(n, szt, c, endcol, panel, S, rowoff, rowoff);
      else
        block_reflect<N>(n, ncols, c, endcol, Rm, S, 0, 0);
      if (threadIdx.x == 0) stn_at<RN>(S.beta, L, ldn_at<RN>(S.misc, 0));
      for (int i = threadIdx.x; i < m; i += blockDim.x)
        stn_at<N>(Y, (long)L * m + i, (i < L) ? N::zero() : ldn_at<N>(S.v, i - L));
      __syncthreads();
    }
    if (panel) {
      for (int t = threadIdx.x; t < m * szt; t += blockDim.x)
        stn_at<N>(Rm, (long)(rowoff + t / szt) * ncols + rowoff + t % szt, ldn_at<N>(panel, t));
      __syncthreads();
    }
    // W from the betas and Y (Matrices/dbl2_baqr_host.cpp:13): w_j = -beta_j
    // (y_j + sum_{l<j} w_l (y_l^H y_j)).  The inner products y_l^H y_j do not
    // wait for the w: all of them first (in P and T, free until the trailing
    // products; szt^2 <= 2 n szt numbers), then the columns one after another
    // with 4 lanes per entry.  y_l starts at row l.
    {
      const int grp = threadIdx.x >> 2, part = threadIdx.x & 3, ngrp = blockDim.x >> 2;
      const int pairs = szt * (szt - 1) / 2;
      int j = 1, kk = grp;  // pair number grp: (kk, j), kk < j
      while (j < szt && kk >= j) kk -= j++;
      for (int base = 0; base < pairs; base += ngrp) {
        const bool on = base + grp < pairs;
        md::msum<N> sum;
        sum.zero();
        if (on)
          for (int i = j + part; i < m; i += 4)
            sum.cfma(ldn_at<N>(Y, (long)kk * m + i), ldn_at<N>(Y, (long)j * m + i));
        const T g = group4_sum<N>(sum.value());
        if (on && part == 0) stn_at<N>(P, (long)j * szt + kk, g);
        kk += ngrp;
        while (j < szt && kk >= j) kk -= j++;
      }
      const R b0 = ldn_at<RN>(S.beta, 0);
      for (int i = threadIdx.x; i < m; i += blockDim.x)
        stn_at<N>(Wm, i, N::neg(N::scale(ldn_at<N>(Y, i), b0)));
      __syncthreads();
      for (int jj = 1; jj < szt; ++jj) {
        const R bj = ldn_at<RN>(S.beta, jj);
        for (int base = 0; base < m; base += ngrp) {
          const int i = base + grp;
          md::msum<N> z;
          z.zero();
          if (i < m) {
            if (part == 0) z.set(ldn_at<N>(Y, (long)jj * m + i));
            for (int l = part; l < jj; l += 4) z.fma(ldn_at<N>(Wm, (long)l * m + i), ldn_at<N>(P, (long)jj * szt + l));
          }
          const T zz = group4_sum<N>(z.value());
          if (i < m && part == 0) stn_at<N>(Wm, (long)jj * m + i, N::neg(N::scale(zz, bj)));
        }
        __syncthreads();
      }
    }
    if constexpr (OZ && !N::is_complex) {
      if (k < nbt - 1) {
        const int nc = ncols - endcol;
        // P = W^T C, then C += Y^T P
        ozaki_gemm<R>(szt, nc, m, [&](int a, int b) { return ldn_at<N>(Wm, (long)a * m + b); },
                      [&](int a, int b) { return ldn_at<N>(Rm, (long)(rowoff + a) * ncols + endcol + b); },
                      [&](int a, int b, const R &v) { stn_at<N>(P, (long)a * nc + b, v); }, oz);
        ozaki_gemm<R>(m, nc, szt, [&](int a, int b) { return ldn_at<N>(Y, (long)b * m + a); },
                      [&](int a, int b) { return ldn_at<N>(P, (long)a * nc + b); },
                      [&](int a, int b, const R &v) {
                        const long o = (long)(rowoff + a) * ncols + endcol + b;
                        stn_at<N>(Rm, o, N::add(ldn_at<N>(Rm, o), v));
                      }, oz);
      }
      // T = Q[:, rowoff..] W^T, then Q[:, rowoff..] += T Y
      ozaki_gemm<R>(n, szt, m, [&](int a, int b) { return ldn_at<N>(Q, (long)a * n + rowoff + b); },
                    [&](int a, int b) { return ldn_at<N>(Wm, (long)b * m + a); },
                    [&](int a, int b, const R &v) { stn_at<N>(Tm, (long)a * szt + b, v); }, oz);
      ozaki_gemm<R>(n, m, szt, [&](int a, int b) { return ldn_at<N>(Tm, (long)a * szt + b); },
                    [&](int a, int b) { return ldn_at<N>(Y, (long)a * m + b); },
                    [&](int a, int b, const R &v) {
                      const long o = (long)a * n + rowoff + b;
                      stn_at<N>(Q, o, N::add(ldn_at<N>(Q, o), v));
                    }, oz);
      continue;
    }
    if (k < nbt - 1) {
      // R[rowoff.., endcol..] += Y (W^H C)
      const int nc = ncols - endcol;
      for (int t = threadIdx.x; t < szt * nc; t += blockDim.x) {
        const int kk = t / nc, j = t % nc;
        md::msum<N> acc;
        acc.zero();
        for (int i = 0; i < m; ++i)
          acc.cfma(ldn_at<N>(Wm, (long)kk * m + i), ldn_at<N>(Rm, (long)(rowoff + i) * ncols + endcol + j));
        stn_at<N>(P, (long)kk * nc + j, acc.value());
      }
      __syncthreads();
      for (int t = threadIdx.x; t < m * nc; t += blockDim.x) {
        const int i = t / nc, j = t % nc;
        const long o = (long)(rowoff + i) * ncols + endcol + j;
        md::msum<N> acc;
        acc.set(ldn_at<N>(Rm, o));
        for (int kk = 0; kk < szt; ++kk) acc.fma(ldn_at<N>(Y, (long)kk * m + i), ldn_at<N>(P, (long)kk * nc + j));
        stn_at<N>(Rm, o, acc.value());
      }
      __syncthreads();
    }
    // Q[:, rowoff..] += (Q[:, rowoff..] W) Y^H
    for (int t = threadIdx.x; t < n * szt; t += blockDim.x) {
      const int i = t / szt, kk = t % szt;
      if (k == 0) {  // Q is still the identity
        stn_at<N>(Tm, (long)i * szt + kk, ldn_at<N>(Wm, (long)kk * m + i));
        continue;
      }
      md::msum<N> acc;
      acc.zero();
      for (int l = 0; l < m; ++l) acc.fma(ldn_at<N>(Q, (long)i * n + rowoff + l), ldn_at<N>(Wm, (long)kk * m + l));
      stn_at<N>(Tm, (long)i * szt + kk, acc.value());
    }
    __syncthreads();
    for (int t = threadIdx.x; t < n * m; t += blockDim.x) {
      const int i = t / m, j = t % m;
      const long o = (long)i * n + rowoff + j;
      md::msum<N> acc;
      acc.set(ldn_at<N>(Q, o));
      for (int kk = 0; kk < szt; ++kk) acc.cfma(ldn_at<N>(Y, (long)kk * m + j), ldn_at<N>(Tm, (long)i * szt + kk));
      stn_at<N>(Q, o, acc.value());
    }
    __syncthreads();
  }
}

// ------------------------------------------------------ tiled back substitution
// Inverse of every szt x szt diagonal tile of the upper triangular U (dim x dim,
// leading dimension ldu) into Tinv (nbt tiles of szt x szt), four lanes per
// (tile, column): column j of the inverse solves T x = e_j by back
// substitution (Matrices/dbl2_tabs_host.cpp:31 CPU_dbl2_upper_inverse,
// dbl2_tabs_kernels.cu:397 dbl2_invert_tiles).  A column is a chain of szt
// rows; the rows' reciprocal pivots, a division each, are formed beforehand
// side by side (kept on the diagonal of Tinv until the row is reached by its
// own column, whose entry they are).
template <class N>
__device__ void block_invert_tiles(int dim, int szt, const double *U, int ldu, double *Tinv) {
  typedef typename N::T T;
  const int W = N::width;
  const long tile2 = (long)szt * szt;
  for (int t = threadIdx.x; t < dim; t += blockDim.x) {
    const int tile = t / szt, i = t - tile * szt;
    stn_at<N>(Tinv, tile * tile2 + (long)i * szt + i, N::div(N::one(), ldn_at<N>(U, (long)t * ldu + t)));
  }
  __syncthreads();
  const int grp = threadIdx.x >> 2, part = threadIdx.x & 3, ngrp = blockDim.x >> 2;
  for (int base = 0; base < dim; base += ngrp) {
    const int t = base + grp;
    const int tile = t / szt, j = t < dim ? t - tile * szt : 0;
    const int off = tile * szt;
    double *inv = Tinv + tile * tile2 * W;
    if (t < dim)
      for (int i = j + 1 + part; i < szt; i += 4) stn_at<N>(inv, (long)i * szt + j, N::zero());
    // rows above the diagonal entry, all groups of the warp in step
    for (int back = 1; back < szt; ++back) {
      const int i = j - back;
      const bool on = t < dim && i >= 0;
      md::msum<N> sum;
      sum.zero();
      if (on)
        for (int l = j - part; l > i; l -= 4)
          sum.fnma(ldn_at<N>(U, (long)(off + i) * ldu + off + l), ldn_at<N>(inv, (long)l * szt + j));
      const T acc = group4_sum<N>(sum.value());
      if (on && part == 0) stn_at<N>(inv, (long)i * szt + j, N::mul(acc, ldn_at<N>(inv, (long)i * szt + i)));
      __syncwarp();
    }
  }
  __syncthreads();
}

// x = U^{-1} b with the inverted diagonal tiles: for k = nbt-1..0,
// x_k = Tinv_k b_k, then b_j -= U_jk x_k for j < k
// (Matrices/dbl2_tabs_host.cpp:147).  b (shared or global) is overwritten.
template <class N>
__device__ void block_tiled_backsub(int dim, int szt, const double *U, int ldu, const double *Tinv, double *b,
                                    double *x) {
  typedef typename N::T T;
  const int nbt = dim / szt;
  const int grp = threadIdx.x >> 2, part = threadIdx.x & 3, ngrp = blockDim.x >> 2;
  for (int k = nbt - 1; k >= 0; --k) {
    const int off = k * szt;
    const double *inv = Tinv + (long)k * szt * szt * N::width;
    for (int base = 0; base < szt; base += ngrp) {
      const int i = base + grp;
      md::msum<N> sum;
      sum.zero();
      if (i < szt)
        dot_acc<N, false, false>(sum, inv + (long)i * szt * N::width, 1, b + off * N::width, 1, part, 4, szt);
      const T acc = group4_sum<N>(sum.value());
      if (i < szt && part == 0) stn_at<N>(x, off + i, acc);
    }
    __syncthreads();
    for (int base = 0; base < off; base += ngrp) {
      const int r = base + grp;
      md::msum<N> sum;
      sum.zero();
      if (r < off)
        dot_acc<N, false, false>(sum, U + ((long)r * ldu + off) * N::width, 1, x + off * N::width, 1, part, 4, szt);
      const T acc = group4_sum<N>(sum.value());
      if (r < off && part == 0) stn_at<N>(b, r, N::sub(ldn_at<N>(b, r), acc));
    }
    __syncthreads();
  }
}

// w = Q^H b (Newton/dbl2_bals_kernels.cu:22 dbl2_bals_qtb), four lanes per
// output
template <class N>
__device__ void block_qhb(int n, const double *Q, const double *b, double *w) {
  typedef typename N::T T;
  const int grp = threadIdx.x >> 2, part = threadIdx.x & 3, ngrp = blockDim.x >> 2;
  for (int base = 0; base < n; base += ngrp) {
    const int i = base + grp;
    md::msum<N> sum;
    sum.zero();
    if (i < n)
      dot_acc<N, true, false>(sum, Q + (long)i * N::width, n, b, 1, part, 4, n);
    const T acc = group4_sum<N>(sum.value());
    if (i < n && part == 0) stn_at<N>(w, i, acc);
  }
  __syncthreads();
}

// b -= A x over rows rows: those of the matrices A_k, A_{k+1}, ... and of the
// right hand sides b_j, b_{j+1}, ..., stacked and contiguous
// (Newton/dbl2_tail_kernels.cu:19 dbl2_bals_tail, the targets of one stage at
// once).
// Quad-double: a thread per row (its 450 FP64 cycles per product cover the
// uncoalesced loads), two or four when the rows would leave threads idle.
// Double and double-double: G lanes per row, so that a load instruction
// touches few lines (a thread per row was bound by the L1 cache's
// wavefronts), R rows to a group of lanes at a time with the next entries
// loaded ahead, so that the loads of a stage, from L2 or memory, overlap.
// Real double-double, dimension 64, degree 31: 4.87 ms with one row, 3.35
// with two; complex double-double lost 4 % with two.
template <class N>
struct tail_shape {
  static const int G = (N::tr::limbs == 1 && !N::is_complex) ? 8 : 4;
  static const int R = N::tr::limbs == 1 ? (N::is_complex ? 2 : 4) : (N::is_complex ? 1 : 2);
};
template <class N>
__device__ void block_tail_update(int n, int rows, const double *A, double *b, const double *x) {
  typedef typename N::T T;
  if constexpr (N::tr::limbs > 2) {
    const int G = rows * 4 <= (int)blockDim.x ? 4 : (rows * 2 <= (int)blockDim.x ? 2 : 1);
    const int grp = threadIdx.x / G, part = threadIdx.x % G, ngrp = blockDim.x / G;
    for (int base = 0; base < rows; base += ngrp) {
      const int r = base + grp;
      md::msum<N> sum;
      sum.zero();
      if (r < rows) {
        if (part == 0) sum.set(ldn_at<N>(b, r));
        dot_acc<N, false, true>(sum, A + (long)r * n * N::width, 1, x, 1, part, G, n);
      }
      T v = sum.value();
      if (G > 1) v = N::add(v, md::shfl_xor(v, 1));
      if (G > 2) v = N::add(v, md::shfl_xor(v, 2));
      if (r < rows && part == 0) stn_at<N>(b, r, v);
    }
  } else {
    const int G = tail_shape<N>::G, R = tail_shape<N>::R;
    const int grp = threadIdx.x / G, part = threadIdx.x % G, ngrp = blockDim.x / G;
    for (int base = 0; base < rows; base += R * ngrp) {
      md::msum<N> sum[R];
      const double *a[R];
      T e[R];
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const int r = base + u * ngrp + grp;
        sum[u].zero();
        a[u] = A + (long)(r < rows ? r : 0) * n * N::width;
        e[u] = part < n ? ldn_at<N>(a[u], part) : N::zero();
        if (part == 0 && r < rows) sum[u].set(ldn_at<N>(b, r));
      }
#pragma unroll 1
      for (int l = part; l < n; l += G) {
        const int nl = l + G < n ? l + G : l;
        const T xl = ldn_at<N>(x, l);
        T next[R];
#pragma unroll
        for (int u = 0; u < R; ++u) next[u] = ldn_at<N>(a[u], nl);
#pragma unroll
        for (int u = 0; u < R; ++u) {
          sum[u].fnma(e[u], xl);
          e[u] = next[u];
        }
      }
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const int r = base + u * ngrp + grp;
        const T v = group_sum<N>(sum[u].value(), G);
        if (part == 0 && r < rows) stn_at<N>(b, r, v);
      }
    }
  }
  __syncthreads();
}

}  // namespace phc
