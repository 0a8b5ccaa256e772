"""GPU test of the Householder reflectors at the ends of the range: a first
column (x0, t r_1, t r_2, ...) with t from 1e-30 down to where its squares
underflow.  Q and R must be finite, Q orthogonal and, in real arithmetic, Q R
= A, checked in exact rational arithmetic with the tolerance of
test_dense_gpu.py (1e3 eps of the largest entry of a column); away from 1e-90
< t < 1e-40, where the reference's own v0^2 loses its lower limbs, real
factors are also the oracle's (where those are numbers: it divides by v0 = 0
where sigma / x0 underflows).  (In complex arithmetic the reference's v0 =
x0 - mu x0/|x0| cancels for small t: its reflector is unitary, but what it
leaves below the diagonal is rounding.)"""
from fractions import Fraction

import numpy as np
import pytest

from mdcheck import absdiff
from oracle import pyoracle
from phcpack_b200 import dense
from phcpack_b200 import workloads as wl

pytestmark = pytest.mark.gpu
ORC = pyoracle.oracle()
EPS = {1: 1e-14, 2: 1e-28, 4: 1e-60}
N, SZT = 6, 3


def matrix(prec, cplx, x0, t):
    rng = np.random.default_rng(17)
    a = wl.random_numbers(rng, (N, N), prec, cplx, "normal").reshape(N, N, -1)
    a[1:, 0] *= 2.0 ** np.round(np.log2(t))
    a[0, 0] = 0.0
    a[0, 0, 0] = x0
    return a


def exact(a, prec, cplx):
    """Numbers -> lists of (re, im) Fractions."""
    def num(v):
        re = sum(map(Fraction, v[:prec].tolist()))
        return re, (sum(map(Fraction, v[prec:].tolist())) if cplx else Fraction(0))
    return [[num(v) for v in row] for row in np.asarray(a).reshape(N, N, -1)]


def product(x, y):
    mul = lambda a, b: (a[0] * b[0] - a[1] * b[1], a[0] * b[1] + a[1] * b[0])
    add = lambda a, b: (a[0] + b[0], a[1] + b[1])
    out = [[(Fraction(0), Fraction(0))] * N for _ in range(N)]
    for i in range(N):
        for j in range(N):
            for k in range(N):
                out[i][j] = add(out[i][j], mul(x[i][k], y[k][j]))
    return out


@pytest.mark.parametrize("x0", [1.0, -1.0, 0.0, 1e10])
@pytest.mark.parametrize("prec,cplx", [(1, False), (2, False), (4, False), (1, True), (2, True), (4, True)])
def test_small_entries_below_the_diagonal(prec, cplx, x0):
    for t in (1e-30, 1e-62, 1e-70, 1e-78, 1e-82, 1e-100, 1e-120, 1e-135, 1e-145, 1e-150, 1e-152, 1e-156, 1e-159, 1e-170):
        if x0 == 0.0 and t < 1e-158:
            continue  # the whole column's squares underflow: left alone, as in the reference
        a = matrix(prec, cplx, x0, t)
        Q, R = dense.blocked_houseqr_host(prec, cplx, a.reshape(-1), 1, N, N, SZT)
        assert np.isfinite(Q).all() and np.isfinite(R).all(), t
        q, r, ex = exact(Q, prec, cplx), exact(R, prec, cplx), exact(a, prec, cplx)
        qh = [[(q[j][i][0], -q[j][i][1]) for j in range(N)] for i in range(N)]
        tol = Fraction(1e3 * EPS[prec])
        gram = product(qh, q)
        for i in range(N):
            for j in range(N):
                if i > j:
                    r[i][j] = (Fraction(0), Fraction(0))
                assert abs(gram[i][j][0] - (i == j)) <= tol and abs(gram[i][j][1]) <= tol, t
        if cplx:
            continue
        qr = product(q, r)
        for j in range(N):
            big = max(abs(v) for i in range(N) for v in ex[i][j])
            for i in range(N):
                assert all(abs(u - v) <= tol * big for u, v in zip(qr[i][j], ex[i][j])), t
        if not 1e-90 < t < 1e-40 and x0 != 0.0:
            Qo, Ro = ORC.blocked_houseqr(prec, cplx, N, N, SZT, N // SZT, a.reshape(-1))
            if not np.isfinite(Qo).all():
                continue
            assert absdiff(Q, Qo, prec, cplx).max() <= 1e3 * EPS[prec], t
            assert absdiff(R, Ro, prec, cplx).max() <= 1e3 * EPS[prec] * max(3.0, abs(x0)), t


@pytest.mark.parametrize("prec", [1, 2, 4])
def test_solve_with_a_tiny_entry(prec):
    # a 2 x 2 head [[1, 0.3], [1e-156, 1]]
    n, degp1 = 2, 2
    mat = np.zeros((degp1, n, n, prec))
    mat[0, :, :, 0] = [[1.0, 0.3], [1e-156, 1.0]]
    mat[1, :, :, 0] = [[0.5, 0.25], [0.125, 1.0]]
    rhs = np.zeros((degp1, n, prec))
    rhs[..., 0] = [[1.0, 2.0], [3.0, 4.0]]
    sol = dense.bals_solve_host(prec, False, mat.reshape(-1), rhs.reshape(-1), 1, n, degp1, 1)[0]
    so = ORC.bals_solve(prec, False, n, degp1, 1, mat.reshape(-1), rhs.reshape(-1))[0]
    assert np.isfinite(sol).all() and absdiff(sol, so, prec, False).max() <= 1e4 * EPS[prec] * 4
