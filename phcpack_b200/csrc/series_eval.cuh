// series_eval.cuh -- warp-level truncated power series products and the
// monomial / polynomial evaluation-differentiation built on them.
//
// The convolution z_k = sum_{i<=k} x_i y_{k-i}, k = 0..d, is the hot loop of
// PHCpack's Convolutions and Polynomials (dbl2_convolutions_kernels.cu:92,
// dbl2_polynomials_kernels.cu:25), where one thread owns one coefficient and
// thread k does k+1 of the d+1 padded steps.  Here one warp computes one
// product: coefficients k and d-k are paired (together d+2 terms), and the
// two lanes of a pair split those terms in halves, so every lane does
// ceil((d+2)/2) steps; one shuffle exchange adds the halves.  A warp holds 16
// pairs: series of up to 32 coefficients take one round, longer ones
// ceil((d+1)/32) rounds of the same number of steps.  Series live in shared
// memory, limb-interleaved.
#pragma once
#include "md.cuh"

namespace phc {

// Lane mapping of round r of a degree-deg product: lane 16 h + l is half h of
// pair p = 16 r + l.  Every lane does nch chunks of U terms.  Half 0 does
// the k1 + 1 terms of k1 in its first sw chunks, then the first cnt2 terms of
// k2; half 1 the rest of k2 from x_i0 y_j0 on.  (Chunks, so that a lane turns
// from k1 to k2 between straight-line blocks of U products; the last chunk
// of a part may be short.)  A middle coefficient (k1 = k2, even degree) is
// shared like a k2.
template <int U>
struct lanemap {
  int k1, k2, i0, j0, cnt, cnt2, sw, nch, h;
  bool alone;  // half 0 of a pair: its own coefficient k1 needs nothing from the other half
  bool valid;  // this lane owns output coefficient kout()
  __device__ __forceinline__ lanemap(int deg, int lane, int round) {
    const int np = (deg + 2) >> 1;
    const int pp = 16 * round + (lane & 15);
    const bool active = pp < np;
    const int p = active ? pp : 0;
    h = lane >> 4;
    k1 = p;
    k2 = deg - p;
    nch = ((deg + 2 + U) / 2 + U - 1) / U;  // 2 nch U >= deg + 1 - p + a for a <= p + U
    const bool mid = k1 == k2;
    const int a = mid ? 0 : (p + U) / U;  // chunks of k1
    const int n2 = k2 + 1;                // terms of k2
    const int first = mid ? (n2 + 1) >> 1 : min((nch - a) * U, n2);
    alone = h == 0 && !mid;
    cnt2 = first;
    cnt = !active ? 0 : (h == 0 ? (mid ? first : p + 1) : n2 - first);
    sw = (active && alone) ? a : -1;
    i0 = h == 0 ? 0 : first;
    j0 = (alone ? k1 : k2) - i0;
    valid = active && !(h == 1 && mid);
  }
  __device__ __forceinline__ int kout() const { return h == 0 ? k1 : k2; }
};

// Terms per chunk: quad-double's products are long enough by themselves; at
// degree 31 three take 18 terms per lane where one takes 17.
template <class N> struct conv_chunk { static const int U = N::tr::limbs == 4 ? 1 : 3; };

// Series of one warp.  BIG: longer than 32 coefficients, several rounds.
template <class N, bool BIG>
struct wser {
  typedef typename N::T T;
  static const int W = N::width;
  static const int U = conv_chunk<N>::U;
  typedef lanemap<U> map;
  int deg, n1, lane;

  __device__ __forceinline__ wser(int deg_, int lane_) : deg(deg_), n1(deg_ + 1), lane(lane_) {}

  // z = x*y (x, y series in shared memory); returns the coefficient this
  // lane owns (m.valid) at index m.kout().  All 32 lanes must call it.
  //
  // The products go into one open accumulator (msum).  A lane of the first
  // half sums its k1 terms first and puts that sum aside when it turns to
  // its share of k2 (at chunk m.sw).
  static __device__ __forceinline__ T conv(const double *x, const double *y, const map &m) {
    md::msum<N> acc, done;
    acc.zero();
    done.zero();
    const double *px = x + m.i0 * W, *py = y + m.j0 * W;
    int left = m.cnt;
#pragma unroll 1
    for (int c = 0; c < m.nch; ++c) {
      if (c == m.sw) {  // k1 is complete; on to x_0 y_k2 + ...
        done = acc;
        acc.zero();
        px = x;
        py = y + m.k2 * W;
        left = m.cnt2;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        T xi = N::zero(), yj = N::zero();
        if (left > u) {
          md::ldn(px + u * W, xi);
          md::ldn(py - u * W, yj);
        }
        acc.fma(xi, yj);
      }
      px += U * W;
      py -= U * W;
      left -= U;
    }
    if (m.sw == m.nch) {
      done = acc;
      acc.zero();
    }
    const T a = acc.value();
    const T o = md::shfl_xor(a, 16);
    return m.alone ? done.value() : N::add(a, o);
  }

  __device__ __forceinline__ int rounds() const { return BIG ? (n1 + 31) >> 5 : 1; }
  // f(k) for the coefficients k, lane k mod 32
  template <class F>
  __device__ __forceinline__ void coefs(F f) const {
    if constexpr (BIG) {
#pragma unroll 1
      for (int k = lane; k < n1; k += 32) f(k);
    } else {
      if (lane < n1) f(lane);
    }
  }
  __device__ __forceinline__ void copy(const double *src, double *dst) const {
    coefs([&](int k) {
      T v;
      md::ldn(src + k * W, v);
      md::stn(dst + k * W, v);
    });
  }
  __device__ __forceinline__ void clear(double *dst) const {
    coefs([&](int k) { md::stn(dst + k * W, N::zero()); });
  }
};

// Shared-memory series slots a warp needs for monomials of up to maxvar
// variables: the coefficient and a temporary (which takes b_0 after the
// common factors), f_0..f_{k-2}, b_1..b_{k-3}.
__host__ __device__ inline int warp_slots(int maxvar) {
  int s = 2 * maxvar - 2;
  return s < 3 ? 3 : s;
}

// One monomial by one warp: its value and its k partial derivatives go to
// the sink.  The common-factor method of Newton/dbl2_systems_host.cpp:18-110
// (coefficient c <- x^(e-1) c, derivative j scaled by e_j), then the forward,
// backward and cross products of Convolutions/dbl2_monomials_host.cpp:4-22
// (CPU_dbl2_evaldiff, :175), 3k - 3 of them:
//   f_j = f_{j-1} x_j (f_{-1} = c, j <= k-2; f_{k-2} is the derivative in x_{k-1});
//   the value f_{k-2} x_{k-1};
//   b_0 = x_{k-1} x_{k-2}, b_i = b_{i-1} x_{k-2-i} (i <= k-3);
//   the derivative in x_0, b_{k-3} c;
//   those in x_{i+1}: f_i b_{k-4-i} (i <= k-4) and f_{k-3} x_{k-1} (i = k-3);
//   two variables: c x_1 is the derivative in x_0, times x_0 the value, and
//   x_0 c the derivative in x_1.
// All products run through one loop with one inlined copy of the series
// product: a call per product would keep the caller's state in registers
// across it, which the product needs for independent operations in flight
// (FP64 latency, not the pipe, limited the evaluation), and a copy per kind
// of product would not fit the instruction cache.
// X: dim series (shared memory or global); X2: their squares where a monomial
// has an exponent above 2 (a factor x^2 is then one product), or null; scr: warp_slots(maxvar) series of
// shared memory.  A malformed monomial (variable count, index or exponent
// out of range) is skipped rather than read out of bounds; the host entry
// points reject such supports before any launch.  Returns the number of
// variables, 0 for a skipped monomial.
template <class N, bool BIG, class Sink>
__device__ __forceinline__ int warp_monomial(const wser<N, BIG> &ws, int dim, int maxvar, int k,
                                             const int *__restrict__ ix, const int *__restrict__ ex,
                                             const double *__restrict__ cffm, const double *X, const double *X2,
                                             double *scr, Sink &sink) {
  typedef typename N::T T;
  const int S = ws.n1 * N::width;
  bool ok = (k >= 1 && k <= maxvar);
  for (int v = 0; ok && v < k; ++v) ok = (ix[v] >= 0 && ix[v] < dim && ex[v] >= 1);
  if (!ok) return 0;
  double *const F = scr + 2 * S;                 // f_0 .. f_{k-2}
  double *const B = scr + maxvar * S;            // b_1 .. b_{k-3} (B + i S)
  ws.copy(cffm, scr);
  __syncwarp();
  int cslot = 0;         // c is scratch series 0 or 1
  int v = 0, r = 1;      // next common factor: the r-th of variable v
  int j = 0;             // next of the 3k - 3 products (1 when k = 1)
  const int nprod = k == 1 ? 1 : 3 * k - 3;
#pragma unroll 1
  for (;;) {
    const double *C = scr + cslot * S;
    double *const b0 = scr + (cslot ^ 1) * S;
    const double *x, *y;
    double *dst = nullptr;  // scratch series that takes the product
    int var = -1;           // variable whose derivative it is
    bool value = false;
    while (v < k && r >= ex[v]) {
      ++v;
      r = 1;
    }
    if (v < k) {
      const bool two = X2 != nullptr && r + 1 < ex[v];
      x = (two ? X2 : X) + ix[v] * S;
      y = C;
      cslot ^= 1;
      dst = scr + cslot * S;
      r += two ? 2 : 1;
    } else if (j < nprod) {
      if (j < k - 1) {
        x = j == 0 ? C : F + (j - 1) * S;
        y = X + ix[k == 2 ? 1 : j] * S;
        dst = F + j * S;
        if (j == k - 2) var = k == 2 ? 0 : k - 1;
      } else if (j == k - 1) {
        x = k == 1 ? C : F + (k - 2) * S;
        y = X + ix[k == 2 ? 0 : k - 1] * S;
        value = true;
      } else if (j < 2 * k - 2) {
        const int i = j - k;
        x = i == 0 ? X + ix[k - 1] * S : (i == 1 ? b0 : B + (i - 1) * S);
        y = X + ix[k - 2 - i] * S;
        dst = i == 0 ? b0 : B + i * S;
      } else if (j == 2 * k - 2) {
        x = k == 2 ? X + ix[0] * S : (k == 3 ? b0 : B + (k - 3) * S);
        y = C;
        var = k == 2 ? 1 : 0;
      } else {
        const int i = j - (2 * k - 1);
        x = F + i * S;
        y = i == k - 3 ? X + ix[k - 1] * S : (i == k - 4 ? b0 : B + (k - 4 - i) * S);
        var = i + 1;
      }
      ++j;
    } else {
      break;
    }
    const bool deriv = var >= 0;
    const int row = deriv ? ix[var] : 0, e = deriv ? ex[var] : 1;
    if (deriv) sink.open(row);
#pragma unroll 1
    for (int q = 0; q < ws.rounds(); ++q) {
      const typename wser<N, BIG>::map m(ws.deg, ws.lane, q);
      const T z = wser<N, BIG>::conv(x, y, m);
      if (m.valid) {
        const int kk = m.kout();
        if (dst) md::stn(dst + kk * N::width, z);
        if (value) sink.value(kk, z);
        if (deriv) sink.derivative(var, row, e, kk, z);
      }
    }
    __syncwarp();
  }
  if (k == 1) {  // the derivative is c itself
    const double *C = scr + cslot * S;
    sink.open(ix[0]);
    ws.coefs([&](int kk) {
      T z;
      md::ldn(C + kk * N::width, z);
      sink.derivative(0, ix[0], ex[0], kk, z);
    });
    __syncwarp();
  }
  return k;
}

// Sink of a warp that owns a polynomial: value and gradient accumulate in
// out (dim+1 series in global memory; row dim is the value).  The value of a
// short series is kept in registers (each lane its coefficient), that of a
// long one in the scratch series Vs, and written once.  A gradient row is
// stored at its first contribution and read, added to and written back only
// after that (a 64-bit mask records the rows 0..63 written so far; rows from
// 64 on are zeroed first and always accumulated).
template <class N, bool BIG>
struct row_sink {
  typedef typename N::T T;
  static const int W = N::width;
  const wser<N, BIG> &ws;
  double *out, *Vs;
  unsigned long long written;
  bool first;
  T vacc;
  __device__ __forceinline__ row_sink(const wser<N, BIG> &w, double *o, double *vs, int dim, const double *cst)
      : ws(w), out(o), Vs(vs), written(0ull), first(false) {
    vacc = N::zero();
    for (int r = 64; r < dim; ++r) ws.clear(out + (long)r * ws.n1 * W);
    // the value starts at the constant series
    if constexpr (BIG) {
      ws.copy(cst, Vs);
      __syncwarp();
    } else {
      const typename wser<N, BIG>::map m(ws.deg, ws.lane, 0);
      if (m.valid) md::ldn(cst + m.kout() * W, vacc);
    }
  }
  __device__ __forceinline__ bool first_touch(int r) {
    if (r >= 64) return false;
    const bool f = !((written >> r) & 1ull);
    written |= 1ull << r;
    return f;
  }
  __device__ __forceinline__ void value(int k, const T &z) {
    if constexpr (BIG) {
      T v;
      md::ldn(Vs + k * W, v);
      md::stn(Vs + k * W, N::add(v, z));
    } else {
      vacc = N::add(vacc, z);
    }
  }
  // a monomial is about to contribute to gradient row r
  __device__ __forceinline__ void open(int r) { first = first_touch(r); }
  // row[k] += e z, stored when it is the row's first contribution
  __device__ __forceinline__ void derivative(int, int r, int e, int k, const T &z) {
    double *row = out + ((long)r * ws.n1 + k) * W;
    T v = (e > 1) ? N::scale_d(z, (double)e) : z;
    if (!first) {
      T o;
      md::ldn(row, o);
      v = N::add(o, v);
    }
    md::stn(row, v);
  }
  // the value, and zeros in the rows no monomial reached
  __device__ __forceinline__ void finish(int dim) {
    double *row = out + (long)dim * ws.n1 * W;
    if constexpr (BIG) {
      ws.copy(Vs, row);
    } else {
      const typename wser<N, BIG>::map m(ws.deg, ws.lane, 0);
      if (m.valid) md::stn(row + m.kout() * W, vacc);
    }
    for (int r = 0; r < dim && r < 64; ++r)
      if (!((written >> r) & 1ull)) ws.clear(out + (long)r * ws.n1 * W);
  }
};

// Value and gradient of one polynomial of a system by one warp into out.
// A row's coefficients may be updated by different lanes in different
// monomials; a row is touched at most once per monomial, and a warp barrier
// ends each.
template <class N, bool BIG>
__device__ __forceinline__ void warp_poly_evaldiff(int dim, int deg, int maxvar, int m0, int m1,
                                                   const int *__restrict__ nvr, const int *__restrict__ idx,
                                                   const int *__restrict__ exps, const double *__restrict__ cst,
                                                   const double *__restrict__ cff, const double *X,
                                                   const double *X2, double *scr, double *out) {
  const wser<N, BIG> ws(deg, threadIdx.x & 31);
  const long S = (long)ws.n1 * N::width;
  row_sink<N, BIG> sink(ws, out, scr + warp_slots(maxvar) * S, dim, cst);
  for (int mon = m0; mon < m1; ++mon)
    warp_monomial<N, BIG>(ws, dim, maxvar, nvr[mon], idx + (long)mon * maxvar, exps + (long)mon * maxvar,
                          cff + mon * S, X, X2, scr, sink);
  sink.finish(dim);
}

// Sink of a warp that does one of a polynomial's monomials: the value and
// the derivatives, scaled, in the warp's own series (slot 0 the value, slot
// 1 + v the derivative in the monomial's variable v).
template <class N, bool BIG>
struct slot_sink {
  typedef typename N::T T;
  static const int W = N::width;
  const wser<N, BIG> &ws;
  double *slots;
  __device__ __forceinline__ slot_sink(const wser<N, BIG> &w, double *s) : ws(w), slots(s) {}
  __device__ __forceinline__ void value(int k, const T &z) { md::stn(slots + k * W, z); }
  __device__ __forceinline__ void open(int) {}
  __device__ __forceinline__ void derivative(int v, int, int e, int k, const T &z) {
    md::stn(slots + ((1 + v) * ws.n1 + k) * W, (e > 1) ? N::scale_d(z, (double)e) : z);
  }
};

// Value and gradient of one polynomial by all warps of a CTA, a monomial per
// warp and round.  After each round the threads add the round's values and
// derivatives to the rows (dim+1 series of shared memory) in the order of
// the monomials, a thread per coefficient of every ng-th row, so a result
// does not depend on the warps' timing.  scr: per warp warp_slots(maxvar)
// scratch series and maxvar + 1 result series.
template <class N, bool BIG>
__device__ __forceinline__ void cta_poly_evaldiff(int dim, int deg, int maxvar, int m0, int m1,
                                                  const int *__restrict__ nvr, const int *__restrict__ idx,
                                                  const int *__restrict__ exps, const double *__restrict__ cst,
                                                  const double *__restrict__ cff, const double *X,
                                                  const double *X2, double *scr, double *rows, double *out) {
  typedef typename N::T T;
  const int W = N::width;
  const wser<N, BIG> ws(deg, threadIdx.x & 31);
  const int S = ws.n1 * W;
  const int warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int per = warp_slots(maxvar) + maxvar + 1;  // series per warp
  double *mine = scr + (long)warp * per * S;
  __shared__ int kdone[32];
  for (int t = threadIdx.x; t < (dim + 1) * S; t += blockDim.x) rows[t] = t < dim * S ? 0.0 : cst[t - dim * S];
  // thread t adds coefficient t mod n1 (and + blockDim when a series is
  // longer than the CTA) of the rows g, g + ng, ...
  const int ng = (int)blockDim.x / ws.n1 > 0 ? (int)blockDim.x / ws.n1 : 1;
  const int g = (int)threadIdx.x / ws.n1;
  for (int b = m0; b < m1; b += nw) {
    const int mon = b + warp;
    int k = 0;
    if (mon < m1) {
      slot_sink<N, BIG> sink(ws, mine + warp_slots(maxvar) * S);
      k = warp_monomial<N, BIG>(ws, dim, maxvar, nvr[mon], idx + (long)mon * maxvar, exps + (long)mon * maxvar,
                                cff + (long)mon * S, X, X2, mine, sink);
    }
    if ((threadIdx.x & 31) == 0) kdone[warp] = k;
    __syncthreads();
    if (g < ng) {
      for (int c = (int)threadIdx.x - g * ws.n1; c < ws.n1; c += blockDim.x) {
        for (int w = 0; w < nw; ++w) {
          const int kw = kdone[w];
          const int *ix = idx + (long)(b + w) * maxvar;
          const double *res = scr + ((long)w * per + warp_slots(maxvar)) * S + c * W;
          for (int v = 0; v <= kw && kw > 0; ++v) {
            const int r = v == 0 ? dim : ix[v - 1];
            if (r % ng != g) continue;
            T o, z;
            double *row = rows + (long)r * S + c * W;
            md::ldn(row, o);
            md::ldn(res + (long)v * S, z);
            md::stn(row, N::add(o, z));
          }
        }
      }
    }
    __syncthreads();
  }
  for (int t = threadIdx.x; t < (dim + 1) * S; t += blockDim.x) out[t] = rows[t];
}

}  // namespace phc
