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
// 0..27 are kept: 406 digit products, 0.21 cycles per multiply-add.  What is
// dropped is about 2^-217 |A_m|_row |x_s|_max, below the rounding of the
// quad-double sum it replaces (0.025 2^-212 sum |a x| per sum, measured) by a
// factor of 20 for rows of 64 entries of one scale.  Each A_m is
// converted once per block of stages (23 error-free cuts per number, ~150
// cycles per warp and number), so a block should be long: stages are
// collected in blocks of 4, 8 and 16 (k_bals_solve).
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

// Shared memory (bytes): the digits of 32 rows of A_m in fragment order, on
// whose place the order sums go afterwards; the digits of the x_s; the
// exponents of the rows and columns; a flag word.
static const int kI8A = kI8Digits * 2 * 2 * 4 * 32 * 4;   // [digit][m tile][k half][register][lane]
static const int kI8X = kI8Digits * 2 * 32 * 4 * 4;       // [digit][column group][lane][register]
static const int kI8Smem = kI8A + kI8X + 256;

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

// Smallest E with m < 2^E for a finite m > 0 (0 for m = 0); 100000 when m is
// not finite or so large or small that scaled parts would leave the range of
// a double.
__device__ __forceinline__ int i8_exponent(double m) {
  if (m == 0.0) return 0;
  const int e = ((__double2hiint(m) >> 20) & 0x7ff) - 1022;
  return (e > -300 && e < 300) ? e : 100000;
}

__device__ __forceinline__ void imma_s8(int (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The digit products of MT m tiles (from mt0) and column group cg for the
// orders og, og + 4, ..., og + 24 into D[order][row][column].
template <int MT>
__device__ __forceinline__ void i8_products(const unsigned *A, const unsigned *X, int ks, int mt0, int cg, int og,
                                            int (&acc)[7][MT][4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 7; ++i)
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
  }
}

// b_j -= sum over the columns c < ns with bit c of mask set of A_{j-s0-c}
// x_{s0+c}, for the targets j0 <= j < j1 (j0 >= s0 + ns), of an n x n system
// (kI8MinN <= n <= kI8MaxN) in real quad-double.  mat, rhs, sol as in
// k_bals_solve; i8: kI8Smem bytes of shared memory.  All 256 threads call it.
static __device__ __noinline__ void block_tail_i8(int n, const double *mat, double *rhs, const double *sol, int s0,
                                                  int ns, unsigned mask, int j0, int j1, unsigned char *i8) {
  typedef md::num<md::qd, false> N;
  unsigned *A = reinterpret_cast<unsigned *>(i8);
  int *D = reinterpret_cast<int *>(i8);
  unsigned *X = reinterpret_cast<unsigned *>(i8 + kI8A);
  int *ea = reinterpret_cast<int *>(i8 + kI8A + kI8X);  // 32 rows
  int *eb = ea + 32;                                    // 16 columns
  int *bad = eb + 16;                                   // [0] a column, [1] a row group
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ks = n > 32 ? 2 : 1;
  const int ncg = ns > 8 ? 2 : 1;
  if (tid < 2) bad[tid] = 0;
  __syncthreads();
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
    const int E = mx != mx ? 100000 : i8_exponent(mx);
    bool ok = E < 100000;
    unsigned d[kI8Digits];
    if (!i8_digits4(v, ok ? E : 0, d)) ok = false;
    if (!ok) bad[0] = 1;
    if (kg == 0) eb[c] = E;
    // column g = c mod 8 of group c / 8; k = 32 h + 16 b + 4 tg: register 2 h + b
    const int h = kg >> 3, b = (kg >> 2) & 1, tg = kg & 3;
#pragma unroll
    for (int p = 0; p < kI8Digits; ++p) X[((p * 2 + (c >> 3)) * 32 + (c & 7) * 4 + tg) * 4 + 2 * h + b] = d[p];
  }
  __syncthreads();
#pragma unroll 1
  for (int m = j0 - s0 - ns + 1; m <= j1 - 1 - s0; ++m) {
    // columns whose target m + s0 + c lies in [j0, j1)
    const int cl = max(0, j0 - m - s0), ch = min(ns, j1 - m - s0);
#pragma unroll 1
    for (int r0 = 0; r0 < n; r0 += 32) {
      // rows: 8 threads to a row, two groups of four entries each
      {
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
        const int E = mx != mx ? 100000 : i8_exponent(mx);
        bool ok = E < 100000;
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
          if (!i8_digits4(v, E < 100000 ? E : 0, d)) ok = false;
          const int b = part >> 2, tg = part & 3, u = 2 * b + hi8;
          const int at = ((mt * 2 + h) * 4 + u) * 32 + ((g * 4 + tg) ^ (b << 4));
#pragma unroll
          for (int p = 0; p < kI8Digits; ++p) A[p * 512 + at] = d[p];
        }
        if (!ok) bad[1] = 1;
        if (part == 0) ea[row] = E;
      }
      __syncthreads();
      const bool plain = bad[0] != 0 || bad[1] != 0;
      if (!plain) {
        const int og = warp & 3, g = lane >> 2, tg = lane & 3;
        if (ncg == 2) {
          const int cg = warp >> 2;
          const bool on = cl < 8 * cg + 8 && ch > 8 * cg;
          int acc[7][2][4];
          if (on) i8_products<2>(A, X, ks, 0, cg, og, acc);
          __syncthreads();
          if (on)
#pragma unroll
            for (int i = 0; i < 7; ++i)
#pragma unroll
              for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int u = 0; u < 4; u += 2)
                  *reinterpret_cast<int2 *>(D + (4 * i + og) * 512 + (16 * t + g + 4 * u) * 16 + 8 * cg + 2 * tg) =
                      make_int2(acc[i][t][u], acc[i][t][u + 1]);
        } else {
          const int t = warp >> 2;
          int acc[7][1][4];
          i8_products<1>(A, X, ks, t, 0, og, acc);
          __syncthreads();
#pragma unroll
          for (int i = 0; i < 7; ++i)
#pragma unroll
            for (int u = 0; u < 4; u += 2)
              *reinterpret_cast<int2 *>(D + (4 * i + og) * 512 + (16 * t + g + 4 * u) * 16 + 2 * tg) =
                  make_int2(acc[i][0][u], acc[i][0][u + 1]);
        }
      }
      __syncthreads();
      // the order sums leave the integers: entry (row, column), two per thread
#pragma unroll 1
      for (int t = tid; t < 512; t += 256) {
        const int row = t >> 4, c = t & 15;
        if (r0 + row >= n || c < cl || c >= ch || !((mask >> c) & 1u)) continue;
        double *bj = rhs + ((long)(m + s0 + c) * n + r0 + row) * 4;
        md::macc<md::qd> s;
        s.set(ldn_at<N>(bj, 0));
        if (plain) {
          const double *a = mat + ((long)m * n + r0 + row) * n * 4;
          const double *x = sol + (long)(s0 + c) * n * 4;
          for (int k = 0; k < n; ++k) s.add(-ldn_at<N>(a, k), ldn_at<N>(x, k));
        } else {
          // order r weighs 2^(ea + eb - 12 - 8 r): four orders to a double, exactly
          double wt = __hiloint2double((1023 + ea[row] + eb[c] - 36) << 20, 0);
#pragma unroll 1
          for (int i = 0; i < 7; ++i) {
            const int *d = D + 4 * i * 512 + t;
            double v = (double)d[0];
            v = __fma_rn(v, 256.0, (double)d[512]);
            v = __fma_rn(v, 256.0, (double)d[1024]);
            v = __fma_rn(v, 256.0, (double)d[1536]);
            double e = __dmul_rn(v, -wt);
            s.f0 = md::two_sum(s.f0, e, e);
            s.at1(e);
            wt = __dmul_rn(wt, 0x1p-32);
          }
        }
        md::stn(bj, s.value());
      }
      __syncthreads();
      if (tid == 0) bad[1] = 0;
      // (the next group's rows set it after this barrier's reads; the
      // barrier below orders the reset before them)
      __syncthreads();
    }
  }
}

}  // namespace phc
