"""GPU test of the blocked tail of the real quad-double least-squares solve
(dimension 32..64: blocks of 4, 8 and 16 stages as digit products on the
integer tensor cores).  Against the oracle with the tolerance of
test_dense_gpu.py (1e4 eps max(1, |x|) per block), at the edges: the smallest
and largest dimension, dimensions off the tiles of 16 and 32 rows and one
more than 32 columns, a tail one stage past a block of 4, 8, 16 and two of
16, a skipped stage inside a block, and the rows that the digits cannot hold
(limbs that overlap, entries near the ends of the range), which take the
FP64 products."""
import numpy as np
import pytest

from oracle import pyoracle
from phcpack_b200 import dense
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
