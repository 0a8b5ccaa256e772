// tail_i8.cuh -- blocks of the quad-double Toeplitz tail on the integer
// tensor cores: b_j -= sum_s A_{j-s} x_s for a block of up to 16 solved
// stages s and the targets j behind it, by one CTA.
//
// A quad-double product and sum is 223 FP64 operations (3.5 cycles of an
// SM's FP64 pipe per multiply-add at the pipe's full rate, ~6 in the solve).
// Here every row of A_m and every x_s is written as an integer multiple of
// 2^(E-222), E its own exponent (|a| < 2^E), in 28 signed base-256 digits;
// a product's digits p and q meet in order p + q, whose sum over the row is
// an exact 32-bit integer (28 * 64 * 2^14 < 2^25), formed by mma.sync
// m16n8k32 s8 (1950 multiply-adds per cycle and SM measured).  The orders
// 0..28 are kept: 433 digit products, 0.22 cycles per multiply-add.  Each A_m
// is converted once per block of stages (23 error-free cuts per number, ~150
// cycles per warp and number), so a block should be long: stages are
// collected in blocks of 4, 8 and 16 (k_bals_solve).
//
// Errors.  Digits below 2^-222 of the row's largest entry and of the largest
// x, and the orders behind 28, are dropped: an error relative to M = 2^(Ea +
// Eb), where the quad-double products err relative to S = sum |a x|.  In
// units of 2^-212 (150 sums each of 32 and 64 normal and uniform products):
// at most 0.0027 M, 0.0008 in the mean square; quad-double products, open
// sums: at most 0.033 S, 0.006; every product and sum rounded: 0.13 S, 0.026.
// M is S's size for rows and x of one scale (S = 0.8 M at least in those
// sums), but not when large a meet small x.  So every sum has its own lower
// bound of S, one more digit product of magnitudes (the leading digits, each
// less one), and where that is below M / 16 the quad-double products are
// formed instead (dot products of 64 entries with half the unknowns scaled
// by 2^60 and their columns by 2^-60 lost 15 digits to the cuts).
//
// tcgen05's integer form would want the digits in swizzled descriptors and
// its sums in TMEM; the digits are produced here in registers, where
// mma.sync reads them through shared memory in its own fragment order, and
// converting, not multiplying, is already the larger part.
#pragma once
#include "dense.cuh"

namespace phc {

static const int kI8Digits = 28;
static const int kI8Cols = 16;   // stages per block
static const int kI8MaxN = 64;
static const int kI8MinN = 32;   // below, padding to 16 x 32 tiles eats the gain

static const int kI8Bound = 4096 / 16;  // M / 16 in units of the leading digits' product

// Shared memory (bytes): the digits of 32 rows of A_m in fragment order
// ([digit][m tile][k half][register][lane]), on whose place the order sums
// and the magnitudes go afterwards; the digits of the x_s; the exponents of
// the rows and columns.
static const int kI8D = (kI8Digits + 3) * 512 * 4;   // [order][row][column], order 28 in two parts, magnitudes
static const int kI8X = (kI8Digits + 1) * 2 * 32 * 4 * 4;  // [digit][column group][lane][register]
static const int kI8Smem = kI8D + kI8X + 256;

// Four numbers a[0..3] (normalised quad-doubles below 2^E) as digits: out[p]
// holds digit p of the four, a byte each.  Returns false when a limb is
// larger than its place allows (a number that is not normalised, an
// infinity or a NaN).
__device__ __forceinline__ bool i8_digits4(const md::qd (&a)[4], int E, unsigned (&out)[kI8Digits]) {
  bool ok = true;
  unsigned w[4][7];
  // x 2^-E, so that the cuts below are constants
  const double sc = __hiloint2double((1023 - E) << 20, 0);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    double r[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) r[l] = __dmul_rn(a[e].x[l], sc);
    // the cuts of a limb start where the limbs above end
    ok = ok && fabs(r[0]) < 1.0 && fabs(r[1]) < 0x1p-50 && fabs(r[2]) < 0x1p-103 && fabs(r[3]) < 0x1p-156;
    int c[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      // chunk q: units of 2^(28 (7 - q) - 222), the multiple in the low word of r + 1.5 2^52 unit
      const double big = 0x1.8p52 * (q == 0 ? 0x1p-26 : q == 1 ? 0x1p-54 : q == 2 ? 0x1p-82 : q == 3 ? 0x1p-110
                                     : q == 4 ? 0x1p-138 : q == 5 ? 0x1p-166 : q == 6 ? 0x1p-194 : 0x1p-222);
      // + 0x80 in every digit: bytes become digits + 128
      int s = (q & 1) ? 0x0808080 : 0x8080808;
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        if (q >= (l == 0 ? 0 : l == 1 ? 1 : l == 2 ? 3 : 5)) {
          const double t = __dadd_rn(r[l], big);
          s += __double2loint(t);
          r[l] = __dsub_rn(r[l], __dsub_rn(t, big));
        }
      }
      c[q] = s;
    }
    // carries, 28 bits to a chunk, then 32-bit words (top first)
    unsigned u[8];
    int carry = 0;
#pragma unroll
    for (int q = 7; q >= 0; --q) {
      const int s = c[q] + carry;
      u[q] = (unsigned)s & 0xfffffffu;
      carry = s >> 28;
    }
#pragma unroll
    for (int i = 0; i < 7; ++i) w[e][i] = ((u[i] << (4 + 4 * i)) | (u[i + 1] >> (24 - 4 * i))) ^ 0x80808080u;
  }
  // bytes of the four numbers together, digit by digit (the top byte of a word is its first digit)
#pragma unroll
  for (int i = 0; i < 7; ++i) {
    const unsigned lo01 = __byte_perm(w[0][i], w[1][i], 0x5140), hi01 = __byte_perm(w[0][i], w[1][i], 0x7362);
    const unsigned lo23 = __byte_perm(w[2][i], w[3][i], 0x5140), hi23 = __byte_perm(w[2][i], w[3][i], 0x7362);
    out[4 * i + 3] = __byte_perm(lo01, lo23, 0x5410);
    out[4 * i + 2] = __byte_perm(lo01, lo23, 0x7632);
    out[4 * i + 1] = __byte_perm(hi01, hi23, 0x5410);
    out[4 * i + 0] = __byte_perm(hi01, hi23, 0x7632);
  }
  return ok;
}

// Smallest E with m < 2^E for a finite m > 0; kI8Zero for m = 0; kI8Not when
// m is not finite or so large or small that scaled parts would leave the
// range of a double.
static const int kI8Not = 100000, kI8Zero = -100000;
__device__ __forceinline__ int i8_exponent(double m) {
  if (m == 0.0) return kI8Zero;
  const int e = ((__double2hiint(m) >> 20) & 0x7ff) - 1022;
  return (e > -300 && e < 300) ? e : kI8Not;
}
// The exponent to cut by, where there is none of the numbers' own (a limb
// behind a leading limb of zero then shows as one out of place).
__device__ __forceinline__ int i8_cut(int E) { return E == kI8Not ? 0 : (E == kI8Zero ? -299 : E); }

// Leading digits -> their magnitudes less one (zero stays): below |a| 2^(6-E).
// Kept as a digit behind the last.
__device__ __forceinline__ unsigned i8_magnitudes(unsigned d) { return __vsubus4(__vabs4(d), 0x01010101u); }

__device__ __forceinline__ void imma_s8(int (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The digit products of MT m tiles (from mt0) and column group cg for the
// orders og, og + 4, ..., og + 24; in the last accumulator half of order 28
// (og = 0 and 1, whose orders are the shortest: the longest stay 112 digit
// products) or the magnitudes (og = 2).
template <int MT>
__device__ __forceinline__ void i8_products(const unsigned *A, const unsigned *X, int ks, int mt0, int cg, int og,
                                            int (&acc)[8][MT][4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int t = 0; t < MT; ++t)
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[i][t][u] = 0;
#pragma unroll 1
  for (int p = 0; p < kI8Digits; ++p) {
    unsigned a[2][MT][4];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int t = 0; t < MT; ++t)
#pragma unroll
        for (int u = 0; u < 4; ++u)
          a[h][t][u] = h < ks ? A[(((p * 2 + mt0 + t) * 2 + h) * 4 + u) * 32 + (lane ^ ((u & 2) << 3))] : 0u;
#pragma unroll
    for (int i = 0; i < 7; ++i) {
      const int q = 4 * i + og - p;
      if (q >= 0) {
        const uint4 b = *reinterpret_cast<const uint4 *>(X + ((q * 2 + cg) * 32 + lane) * 4);
#pragma unroll
        for (int t = 0; t < MT; ++t) {
          imma_s8(acc[i][t], a[0][t], b.x, b.y);
          if (ks > 1) imma_s8(acc[i][t], a[1][t], b.z, b.w);
        }
      }
    }
    if (og < 2 && (p & 1) == og && p > 0) {
      const uint4 b = *reinterpret_cast<const uint4 *>(X + (((kI8Digits - p) * 2 + cg) * 32 + lane) * 4);
#pragma unroll
      for (int t = 0; t < MT; ++t) {
        imma_s8(acc[7][t], a[0][t], b.x, b.y);
        if (ks > 1) imma_s8(acc[7][t], a[1][t], b.z, b.w);
      }
    }
  }
  if (og == 2) {
    const uint4 b = *reinterpret_cast<const uint4 *>(X + ((kI8Digits * 2 + cg) * 32 + lane) * 4);
#pragma unroll
    for (int t = 0; t < MT; ++t)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (h >= ks) break;
        unsigned a[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          a[u] = A[(((kI8Digits * 2 + mt0 + t) * 2 + h) * 4 + u) * 32 + (lane ^ ((u & 2) << 3))];
        imma_s8(acc[7][t], a, h ? b.z : b.x, h ? b.w : b.y);
      }
  }
}

// The accumulators of i8_products into D[order][row][column], from row and
// column on.
template <int MT>
__device__ __forceinline__ void i8_store(int *D, int og, int row, int col, const int (&acc)[8][MT][4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (i == 7 && og > 2) break;
#pragma unroll
    for (int t = 0; t < MT; ++t)
#pragma unroll
      for (int u = 0; u < 4; u += 2)
        *reinterpret_cast<int2 *>(D + (4 * i + og) * 512 + (row + 16 * t + g + 4 * u) * 16 + col + 2 * tg) =
            make_int2(acc[i][t][u], acc[i][t][u + 1]);
  }
}

// Exponent of the unit of a sum's orders; kI8Not for a sum that is not of
// digits (a row or column that has none, or magnitudes below the bound),
// kI8Zero for one of zeros.
__device__ __forceinline__ int i8_sum_exponent(int er, int ec, int magnitudes) {
  if (er == kI8Not || ec == kI8Not) return kI8Not;
  if (er == kI8Zero || ec == kI8Zero) return kI8Zero;
  return magnitudes >= kI8Bound ? er + ec : kI8Not;
}

// The sums of a group of 32 rows that are not of digits: b_j -= A_m x in
// quad-double, four lanes to a sum.  a: the group's first row, of rows; b: its
// entry of b_{m+s0}; x: x_{s0}; columns: a bit each.
static __device__ __noinline__ void i8_hard_sums(int n, int rows, unsigned columns, const double *a, double *b,
                                                 const double *x, const int *magnitudes, const int *ea,
                                                 const int *eb) {
  typedef md::num<md::qd, false> N;
  const int part = threadIdx.x & 3;
#pragma unroll 1
  for (int o = threadIdx.x >> 2; o < 512; o += 64) {
    const int row = o >> 4, c = o & 15;
    const bool on = row < rows && ((columns >> c) & 1u) && i8_sum_exponent(ea[row], eb[c], magnitudes[o]) == kI8Not;
    if (!__any_sync(0xffffffffu, on)) continue;
    md::msum<N> sum;
    sum.zero();
    if (on)
      dot_acc<N, false, true>(sum, a + (long)row * n * 4, 1, x + (long)c * n * 4, 1, part, 4, n);
    const md::qd v = group4_sum<N>(sum.value());
    double *bj = b + ((long)c * n + row) * 4;
    if (on && part == 0) md::stn(bj, ldn_at<N>(bj, 0) + v);
  }
}

// b_j -= sum over the columns c < ns with bit c of mask set of A_{j-s0-c}
// x_{s0+c}, for the targets j0 <= j < j1 (j0 >= s0 + ns), of an n x n system
// (kI8MinN <= n <= kI8MaxN) in real quad-double.  mat, rhs, sol as in
// k_bals_solve; i8: kI8Smem bytes of shared memory.  All 256 threads call it.
// Returns the first m whose A_m is left to the caller: j1 - s0, or less when
// too many of the sums with an A_m (a third, spread evenly) were not of digits.
static __device__ __noinline__ int block_tail_i8(int n, const double *mat, double *rhs, const double *sol, int s0,
                                                 int ns, unsigned mask, int j0, int j1, unsigned char *i8) {
  typedef md::num<md::qd, false> N;
  unsigned *A = reinterpret_cast<unsigned *>(i8);
  int *D = reinterpret_cast<int *>(i8);
  unsigned *X = reinterpret_cast<unsigned *>(i8 + kI8D);
  int *ea = reinterpret_cast<int *>(i8 + kI8D + kI8X);  // 32 rows
  int *eb = ea + 32;                                    // 16 columns
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ks = n > 32 ? 2 : 1;
  const int ncg = ns > 8 ? 2 : 1;
  __syncthreads();  // the x_s are in place
  // columns: 16 threads to a column, a group of four entries each
  {
    const int c = tid >> 4, kg = tid & 15;
    const bool on = c < ns && ((mask >> c) & 1u);
    md::qd v[4];
    double mx = 0.0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = 4 * kg + e;
      v[e] = (on && k < n) ? ldn_at<N>(sol, (long)(s0 + c) * n + k) : N::zero();
      const double m = fabs(v[e].x[0]);
      mx = m > mx || m != m ? m : mx;  // a NaN stays
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      const double m = __shfl_xor_sync(0xffffffffu, mx, o);
      mx = m > mx || m != m ? m : mx;
    }
    const int E = mx != mx ? kI8Not : i8_exponent(mx);
    unsigned d[kI8Digits];
    const bool ok = i8_digits4(v, i8_cut(E), d);
    const unsigned all = (__ballot_sync(0xffffffffu, ok) >> (lane & 16)) & 0xffffu;
    if (kg == 0) eb[c] = all == 0xffffu ? E : kI8Not;
    // column g = c mod 8 of group c / 8; k = 32 h + 16 b + 4 tg: register 2 h + b
    const int h = kg >> 3, b = (kg >> 2) & 1, tg = kg & 3;
#pragma unroll
    for (int p = 0; p <= kI8Digits; ++p)
      X[((p * 2 + (c >> 3)) * 32 + (c & 7) * 4 + tg) * 4 + 2 * h + b] = p < kI8Digits ? d[p] : i8_magnitudes(d[0]);
  }
  __syncthreads();
#pragma unroll 1
  for (int m = j0 - s0 - ns + 1; m <= j1 - 1 - s0; ++m) {
    bool many = false;
    // columns whose target m + s0 + c lies in [j0, j1)
    const int cl = max(0, j0 - m - s0), ch = min(ns, j1 - m - s0);
#pragma unroll 1
    for (int r0 = 0; r0 < n; r0 += 32) {
      {
        // rows: 8 threads to a row, two groups of four entries each
        const int row = tid >> 3, part = tid & 7;
        const double *a = mat + ((long)m * n + r0 + row) * n * 4;
        const bool on = r0 + row < n;
        double mx = 0.0;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int k = (e < 4 ? 4 * part : 4 * (part + 8)) + (e & 3);
          const double v = (on && k < n) ? fabs(a[4 * k]) : 0.0;
          mx = v > mx || v != v ? v : mx;
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
          const double v = __shfl_xor_sync(0xffffffffu, mx, o);
          mx = v > mx || v != v ? v : mx;
        }
        const int E = mx != mx ? kI8Not : i8_exponent(mx);
        bool ok = true;
        const int mt = row >> 4, hi8 = (row >> 3) & 1, g = row & 7;
#pragma unroll 1
        for (int h = 0; h < ks; ++h) {
          md::qd v[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int k = 4 * (part + 8 * h) + e;
            v[e] = (on && k < n) ? ldn_at<N>(a, k) : N::zero();
          }
          unsigned d[kI8Digits];
          if (!i8_digits4(v, i8_cut(E), d)) ok = false;
          const int b = part >> 2, tg = part & 3, u = 2 * b + hi8;
          const int at = ((mt * 2 + h) * 4 + u) * 32 + ((g * 4 + tg) ^ (b << 4));
#pragma unroll
          for (int p = 0; p < kI8Digits; ++p) A[p * 512 + at] = d[p];
          A[kI8Digits * 512 + at] = i8_magnitudes(d[0]);
        }
        const unsigned all = (__ballot_sync(0xffffffffu, ok) >> (lane & 24)) & 0xffu;
        if (part == 0) ea[row] = all == 0xffu ? E : kI8Not;
        __syncthreads();
        const int og = warp & 3;
        if (ncg == 2) {
          const int cg = warp >> 2;
          const bool in = cl < 8 * cg + 8 && ch > 8 * cg;
          int acc[8][2][4];
          if (in) i8_products<2>(A, X, ks, 0, cg, og, acc);
          __syncthreads();
          if (in) i8_store<2>(D, og, 0, 8 * cg, acc);
        } else {
          const int t = warp >> 2;
          int acc[8][1][4];
          i8_products<1>(A, X, ks, t, 0, og, acc);
          __syncthreads();
          i8_store<1>(D, og, 16 * t, 0, acc);
        }
        __syncthreads();
      }
      // the order sums leave the integers: entry (row, column), two per thread
      const unsigned columns = mask & ((1u << ch) - 1u) & ~((1u << cl) - 1u);
      const int c = tid & 15, ec = eb[c];
      bool hard = false;
      if ((columns >> c) & 1u) {
#pragma unroll 1
        for (int row = tid >> 4; row < min(32, n - r0); row += 16) {
          const int *d = D + row * 16 + c;
          const int E = i8_sum_exponent(ea[row], ec, d[(kI8Digits + 2) * 512]);
          if (E == kI8Not) hard = true;
          if (E == kI8Not || E == kI8Zero) continue;  // zeros subtract nothing
          double *bj = rhs + ((long)(m + s0 + c) * n + r0 + row) * 4;
          md::macc<md::qd> s;
          s.set(ldn_at<N>(bj, 0));
          // order r weighs 2^(E - 12 - 8 r): four orders to a double, exactly
          double wt = __hiloint2double((1023 + E - 36) << 20, 0);
#pragma unroll 1
          for (int i = 0; i < 7; ++i, d += 4 * 512) {
            double v = (double)d[0];
            v = __fma_rn(v, 256.0, (double)d[512]);
            v = __fma_rn(v, 256.0, (double)d[1024]);
            v = __fma_rn(v, 256.0, (double)d[1536]);
            double e = __dmul_rn(v, -wt);
            s.f0 = md::two_sum(s.f0, e, e);
            s.at1(e);
            wt = __dmul_rn(wt, 0x1p-32);
          }
          s.at3(__dmul_rn((double)(d[0] + d[512]), __dmul_rn(wt, -0x1p24)));
          md::stn(bj, s.value());
        }
      }
      const int count = __syncthreads_count(hard);
      if (count) {
        i8_hard_sums(n, n - r0, columns, mat + ((long)m * n + r0) * n * 4, rhs + ((long)(m + s0) * n + r0) * 4,
                     sol + (long)s0 * n * 4, D + (kI8Digits + 2) * 512, ea, eb);
        many = many || count >= 8 * (ch - cl);  // of 16 threads to a column
        __syncthreads();
      }
    }
    if (many) return m + 1;
  }
  return j1 - s0;
}

}  // namespace phc
