"""The running sums of products of the device arithmetic (md::macc of
phcpack_b200/csrc/md.cuh), compiled for the host with the rounded intrinsics
as plain operations, against exact rational arithmetic: random products, and
sums whose terms cancel down to their second, third or fourth limb or at
several scales, where the accumulators no longer decrease.  The bounds are
those of a product and a sum rounded to the precision each: a few units of
2^-106 (double-double) or 2^-212 (quad-double) of sum |ab|; one unit of
quad-double, eight of double-double (whose products are rounded by themselves)
is asked for."""
import ctypes
import os
import random
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "phcpack_b200", "csrc")

SHIM = """
#pragma once
#include <cmath>
#define __device__
#define __host__
#define __forceinline__ inline
struct alignas(16) double2 { double x, y; };
static inline double2 make_double2(double a, double b) { return {a, b}; }
static inline double __dadd_rn(double a, double b) { return a + b; }
static inline double __dsub_rn(double a, double b) { return a - b; }
static inline double __dmul_rn(double a, double b) { return a * b; }
static inline double __ddiv_rn(double a, double b) { return a / b; }
static inline double __dsqrt_rn(double a) { return std::sqrt(a); }
static inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
static inline double __shfl_sync(unsigned, double v, int) { return v; }
static inline double __shfl_xor_sync(unsigned, double v, int) { return v; }
"""

SOURCE = """
#include "md.cuh"
template <class R, int L> static void sum(int n, const double *a, const double *b, double *out) {
  md::macc<R> m;
  m.zero();
  for (int i = 0; i < n; ++i) {
    R x, y;
    double *px = reinterpret_cast<double *>(&x), *py = reinterpret_cast<double *>(&y);
    for (int l = 0; l < L; ++l) {
      px[l] = a[L * i + l];
      py[l] = b[L * i + l];
    }
    m.add(x, y);
  }
  const R s = m.value();
  for (int l = 0; l < L; ++l) out[l] = reinterpret_cast<const double *>(&s)[l];
}
extern "C" void sum2(int n, const double *a, const double *b, double *out) { sum<md::dd, 2>(n, a, b, out); }
extern "C" void sum4(int n, const double *a, const double *b, double *out) { sum<md::qd, 4>(n, a, b, out); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("md_sums")
    (d / "cuda_runtime.h").write_text(SHIM)
    (d / "sums.cpp").write_text(SOURCE)
    so = str(d / "sums.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-w", "-I", str(d), "-I", CSRC,
                    str(d / "sums.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def limbs(f, prec):
    out = []
    for _ in range(prec):
        out.append(float(f))
        f -= Fraction(out[-1])
    return out


def number(rng, scale=0):
    return Fraction(rng.getrandbits(230) - (1 << 229), 1 << 229) * Fraction(2) ** scale


def random_products(rng, prec):
    n = rng.randint(1, 40)
    return [number(rng) for _ in range(n)], [number(rng) for _ in range(n)]


def one_cancellation(rng, prec):
    """x and a number that cancels all but its limbs from l on, among smaller
    terms."""
    x = number(rng)
    q = limbs(x, prec)
    lo = rng.randint(1, prec)
    y = [-v for v in q]
    if lo < prec:
        y[lo] *= 1 + rng.random()
    a = [x, sum(map(Fraction, y))] + [number(rng, -rng.randint(0, 53 * prec - 13)) for _ in range(rng.randint(3, 6))]
    rng.shuffle(a)
    return a, [Fraction(1)] * len(a)


def several_cancellations(rng, prec):
    a = []
    for _ in range(rng.randint(1, 4)):
        x = number(rng, -rng.randint(0, 40 * prec))
        y = [-v for v in limbs(x, prec)]
        y[rng.randrange(prec)] *= 1 + 2.0 ** -rng.randint(1, 52)
        a += [x, sum(map(Fraction, y))]
    a += [number(rng, -rng.randint(0, 53 * prec)) for _ in range(rng.randint(0, 4))]
    rng.shuffle(a)
    return a, [Fraction(1)] * len(a)


@pytest.mark.parametrize("prec,units", [(2, 8.0), (4, 1.0)])
@pytest.mark.parametrize("draw,count", [(random_products, 300), (one_cancellation, 3000), (several_cancellations, 3000)])
def test_sums_of_products(lib, prec, units, draw, count):
    rng = random.Random(11)
    fn = lib.sum2 if prec == 2 else lib.sum4
    ptr = lambda v: v.ctypes.data_as(ctypes.c_void_p)
    for _ in range(count):
        x, y = draw(rng, prec)
        a, b = np.array([limbs(v, prec) for v in x]), np.array([limbs(v, prec) for v in y])
        exact = lambda v: sum(map(Fraction, v.tolist()))
        terms = [exact(p) * exact(q) for p, q in zip(a, b)]
        out = np.zeros(prec)
        fn(len(x), ptr(a), ptr(b), ptr(out))
        err = abs(exact(out) - sum(terms))
        assert err <= Fraction(units) * Fraction(2) ** (-53 * prec) * sum(map(abs, terms))
