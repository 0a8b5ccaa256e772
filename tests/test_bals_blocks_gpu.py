"""GPU test of the blocked tail of the real quad-double least-squares solve
(dimension 32..64: blocks of 4, 8 and 16 stages as digit products on the
integer tensor cores).  Against the oracle with the tolerance of
test_dense_gpu.py (1e4 eps max(1, |x|) per block), at the edges: the smallest
and largest dimension, dimensions off the tiles of 16 and 32 rows and one
more than 32 columns, a tail one stage past a block of 4, 8, 16 and two of
16, a skipped stage inside a block, and the rows that the digits cannot hold
(limbs that overlap, entries near the ends of the range) or that are too far
above the sums they enter (unknowns in other units, sparse rows), which take
the quad-double products."""
import numpy as np
import pytest

from oracle import pyoracle
from phcpack_b200 import _lib, dense
from phcpack_b200 import workloads as wl
from test_dense_gpu import check_bals

pytestmark = pytest.mark.gpu
ORC = pyoracle.oracle()


def solve_both(mat, rhs, n, degp1, szt):
    sol, _, _, _, fl = dense.bals_solve_host(4, False, mat, rhs, 1, n, degp1, szt)
    so, _, _, _, flo = ORC.bals_solve(4, False, n, degp1, 1, mat, rhs)
    return sol, fl, so, flo


def inputs(seed, n, degp1):
    rng = np.random.default_rng(seed)
    mat = wl.random_numbers(rng, (degp1, n, n), 4, False, "normal").reshape(degp1, n, n, 4)
    rhs = wl.random_numbers(rng, (degp1, n), 4, False, "normal").reshape(degp1, n, 4)
    return mat, rhs


@pytest.mark.parametrize("n,szt,degp1", [(32, 8, 6), (33, 11, 9), (36, 12, 10), (48, 16, 18), (63, 21, 7),
                                         (64, 16, 17), (64, 32, 35)])
def test_blocked_tail_matches_oracle(n, szt, degp1):
    mat, rhs = inputs(n + degp1, n, degp1)
    mat *= 2.0 ** -np.arange(degp1)[:, None, None, None]  # a convergent series
    sol, fl, so, flo = solve_both(mat.reshape(-1), rhs.reshape(-1), n, degp1, szt)
    assert np.array_equal(fl, flo)
    assert check_bals(sol, so, 4, False, degp1, n)


@pytest.mark.parametrize("kind", ["skipped", "overlapping", "huge", "tiny"])
def test_blocked_tail_special_rows(kind):
    n, szt, degp1 = 40, 20, 12
    mat, rhs = inputs(7, n, degp1)
    mat *= 4.0 ** -np.arange(degp1)[:, None, None, None]
    if kind == "skipped":
        # only degrees 0, 4, 8 carry anything: the stages between vanish
        mat[[k for k in range(degp1) if k % 4]] = 0.0
        rhs[[k for k in range(degp1) if k % 4]] = 0.0
    elif kind == "overlapping":
        mat[2, 5, :, 1] = mat[2, 5, :, 0] * 2.0 ** -45
    elif kind == "huge":
        mat *= 2.0 ** 310
        rhs *= 2.0 ** 310
    else:
        mat[2, 3] *= 2.0 ** -310
    sol, fl, so, flo = solve_both(mat.reshape(-1), rhs.reshape(-1), n, degp1, szt)
    assert np.array_equal(fl, flo)
    assert check_bals(sol, so, 4, False, degp1, n)


def graded(n):
    """Powers of two 2^0, 2^60 for the unknowns, in no order."""
    g = np.random.default_rng(n).permutation(np.arange(n) % 2 * 60)
    return 2.0 ** g


@pytest.mark.parametrize("n,szt,degp1", [(32, 8, 9), (40, 20, 18), (64, 16, 20)])
def test_blocked_tail_other_units(n, szt, degp1):
    """The unknowns in other units (columns of every A_k times 2^-g, unknowns
    times 2^g): large entries meet small ones in every sum.  Every unknown has
    to be as exact in its own unit as in the plain system, by the tolerance
    above."""
    mat, rhs = inputs(n + degp1, n, degp1)
    mat *= 2.0 ** -np.arange(degp1)[:, None, None, None]
    d = graded(n)
    plain = solve_both(mat.reshape(-1), rhs.reshape(-1), n, degp1, szt)[0].reshape(degp1, n, 4)
    sol, fl, so, flo = solve_both((mat / d[:, None]).reshape(-1), rhs.reshape(-1), n, degp1, szt)
    assert np.array_equal(fl, flo)
    sol, so = sol.reshape(degp1, n, 4) / d[:, None], so.reshape(degp1, n, 4) / d[:, None]
    assert check_bals(sol.reshape(-1), so.reshape(-1), 4, False, degp1, n)
    assert check_bals(plain.reshape(-1), so.reshape(-1), 4, False, degp1, n)


def test_a_plain_system_takes_the_digits():
    """Every quad-double operation of the solve commutes with a change of the
    unknowns' units, so solutions that differ in their last bits show that the
    plain system took the digit products, which the other cannot.  (A_0
    dominant: the solution does not grow from stage to stage, so that what
    the blocks subtract is not lost behind what is subtracted after them.)"""
    n, szt, degp1 = 64, 16, 20
    mat, rhs = inputs(1, n, degp1)
    mat[0, range(n), range(n), 0] += 24.0
    d = graded(n)
    plain = solve_both(mat.reshape(-1), rhs.reshape(-1), n, degp1, szt)[0].reshape(degp1, n, 4)
    sol, _, so, _ = solve_both((mat / d[:, None]).reshape(-1), rhs.reshape(-1), n, degp1, szt)
    sol, so = sol.reshape(degp1, n, 4) / d[:, None], so.reshape(degp1, n, 4) / d[:, None]
    assert check_bals(sol.reshape(-1), so.reshape(-1), 4, False, degp1, n)
    assert check_bals(plain.reshape(-1), so.reshape(-1), 4, False, degp1, n)
    assert np.array_equal(plain[0], sol[0]) and not np.array_equal(plain[5:], sol[5:])


def test_blocked_tail_sparse_rows():
    # rows of zeros, and rows of one entry (some of whose unknowns are far
    # below the largest: a few sums of a warp by quad-double products)
    n, szt, degp1 = 48, 16, 14
    mat, rhs = inputs(3, n, degp1)
    mat *= 2.0 ** -np.arange(degp1)[:, None, None, None]
    keep = mat.copy()
    mat[1:, ::6] = 0.0
    mat[1:, 3::6] = 0.0
    for k in range(1, degp1):
        mat[k, 3::6, (5 * k) % n] = keep[k, 3::6, (5 * k) % n]
    sol, fl, so, flo = solve_both(mat.reshape(-1), rhs.reshape(-1), n, degp1, szt)
    assert np.array_equal(fl, flo)
    assert check_bals(sol, so, 4, False, degp1, n)


@pytest.mark.parametrize("n,szt,degp1", [(36, 4, 10), (64, 8, 19), (64, 16, 9)])
def test_staged_panels_do_not_change_the_tail(n, szt, degp1):
    # knob 3 moves panels between global and shared memory, whether the digits
    # fit in the place of the WY panels (tile 16) or not: bit for bit the same
    mat, rhs = inputs(n, n, degp1)
    mat *= 2.0 ** -np.arange(degp1)[:, None, None, None]
    out = []
    try:
        for stage in (1, 2):
            _lib.call("phc_tune_set", 3, stage)
            out.append(dense.bals_solve_host(4, False, mat.reshape(-1), rhs.reshape(-1), 1, n, degp1, szt))
    finally:
        _lib.call("phc_tune_set", 3, 0)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
