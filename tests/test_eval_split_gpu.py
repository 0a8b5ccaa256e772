"""GPU test of the two arrangements of phc_system_evaldiff: a warp per
polynomial, and (few polynomials) a CTA per polynomial with its monomials
shared among the warps.  Both form every product and add the monomials'
contributions in the same order, so they agree to the rounding of a sum with
zero; each is held to the oracle with the tolerances of test_eval_gpu.py.
Sizes: around one and two rounds of a series product (degrees 31, 32, 33),
degrees without a full pair of coefficients, fewer monomials than warps, one
more than a round of warps, and more gradient rows than the 64 of the row
mask."""
import numpy as np
import pytest

from mdcheck import abs_batch, check_scaled
from oracle import pyoracle
from phcpack_b200 import _lib, series
from phcpack_b200 import workloads as wl

pytestmark = pytest.mark.gpu
ORC = pyoracle.oracle()
RTOL = {1: 1e-14, 2: 1e-28, 4: 1e-60}


def evaluate(b, knob):
    import torch
    _lib.call("phc_tune_set", 0, knob)
    try:
        out = series.DeviceBatch(b).evaldiff()
        torch.cuda.synchronize()
    finally:
        _lib.call("phc_tune_set", 0, 0)
    return out.cpu().numpy()


@pytest.mark.parametrize("prec,cplx,nsys,dim,deg,nmon,maxvar", [
    (1, False, 2, 3, 0, 9, 2), (1, True, 1, 5, 31, 17, 3), (2, True, 1, 4, 1, 1, 1), (2, True, 2, 7, 2, 8, 5),
    (2, False, 1, 6, 31, 9, 4), (2, True, 1, 6, 32, 3, 4), (2, False, 2, 5, 33, 16, 3), (2, True, 1, 70, 3, 2, 2),
    (4, False, 1, 5, 16, 9, 5), (4, True, 1, 3, 30, 4, 3), (4, False, 1, 4, 63, 5, 2)])
def test_shared_monomials_match_oracle(prec, cplx, nsys, dim, deg, nmon, maxvar):
    b = wl.eval_batch(300 + deg, nsys, dim, deg, nmon, maxvar, prec, cplx, expmax=3)
    ref = ORC.system_evaldiff(b)
    scale = ORC.system_evaldiff(abs_batch(b))
    for knob in (0, 4):  # shared; four polynomials per CTA
        assert check_scaled(evaluate(b, knob), ref, scale, prec, cplx, RTOL[prec]) <= 1.0


@pytest.mark.parametrize("prec,cplx,dim,deg,expmax", [(1, False, 3, 5, 6), (2, True, 9, 31, 5), (2, False, 5, 31, 3),
                                                      (4, False, 4, 9, 4), (2, True, 40, 2, 4)])
def test_squares_match_oracle(prec, cplx, dim, deg, expmax):
    # a warp per polynomial with the squares of the variables at hand:
    # exponents 3, 4, 5, ... are one, one and a half, two squares ..., and a
    # last group of polynomials smaller than the CTA
    b = wl.eval_batch(400 + dim, 1, dim, deg, 5, 3, prec, cplx, expmax=expmax)
    ref = ORC.system_evaldiff(b)
    scale = ORC.system_evaldiff(abs_batch(b))
    for knob in (2, 8):
        assert check_scaled(evaluate(b, knob), ref, scale, prec, cplx, RTOL[prec]) <= 1.0
