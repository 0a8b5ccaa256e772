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
from phcpack_b200 import _lib, autotune, series
from phcpack_b200 import workloads as wl

pytestmark = pytest.mark.gpu
ORC = pyoracle.oracle()
RTOL = {1: 1e-14, 2: 1e-28, 4: 1e-60}


def repeated(b):
    """The systems of b over again, until a CTA per polynomial is too many."""
    c = 1184 // (b.nsys * b.dim) + 1
    nm = len(b.nvr)
    off = np.concatenate([b.mon_off[:-1] + np.int32(i * nm) for i in range(c)] + [np.array([c * nm], np.int32)])
    tile = lambda a: np.tile(a, (c,) + (1,) * (a.ndim - 1))
    return c, wl.SystemBatch(c * b.nsys, b.dim, b.deg, b.maxvar, b.prec, b.cplx, off.astype(np.int32), tile(b.nvr),
                             tile(b.idx), tile(b.exps), tile(b.cst), tile(b.cff), tile(b.input))


def evaluate(b, knob):
    """knob 0: a CTA per polynomial.  Otherwise that many polynomials per CTA,
    a warp each; all copies of the systems have to agree."""
    import torch
    copies, batch = (1, b) if knob == 0 else repeated(b)
    _lib.call("phc_tune_set", 0, knob)
    try:
        out = series.DeviceBatch(batch).evaldiff()
        torch.cuda.synchronize()
    finally:
        _lib.call("phc_tune_set", 0, 0)
    out = out.cpu().numpy().reshape(copies, -1)
    assert np.array_equal(out, np.broadcast_to(out[0], out.shape), equal_nan=True)
    return out[0]


@pytest.mark.parametrize("prec,cplx", [(1, True), (2, False), (4, False)])
def test_polynomials_per_cta_agree(prec, cplx):
    # bit for bit: the same products, summed in the same order
    b = wl.eval_batch(29, 3, 11, 14, 10, 4, prec, cplx, expmax=3)
    out = [evaluate(b, knob) for knob in (1, 2, 4, 8)]
    for o in out[1:]:
        assert np.array_equal(o, out[0])


def test_few_polynomials_do_not_depend_on_the_knob():
    """The warps per CTA that the autotuner found for a large batch do not
    take the arrangement for few polynomials away from a small one: 8
    polynomials of 12 monomials take at most half as long again as by the
    built-in rule (a warp per polynomial: five times as long)."""
    import torch
    db = series.DeviceBatch(wl.eval_batch(5, 1, 8, 15, 12, 4, 2, True, expmax=2))
    stream = torch.cuda.current_stream()
    secs = {}
    try:
        for knob in (0, 2, 8):
            _lib.call("phc_tune_set", 0, knob)
            secs[knob] = min(autotune._time(torch, stream, db.evaldiff, reps=9) for _ in range(3))
    finally:
        _lib.call("phc_tune_set", 0, 0)
    assert max(secs.values()) <= 1.5 * secs[0], secs


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


def test_scratch_that_takes_all_shared_memory():
    # degree 148, 20 variables, double: five warps' scratch is 8 bytes short
    # of the 227 KB a CTA can have
    b = wl.eval_batch(21, 60, 20, 148, 2, 20, 1, False, minvar=18)
    out = series.DeviceBatch(b).evaldiff().cpu().numpy()
    scale = ORC.system_evaldiff(abs_batch(b))
    assert check_scaled(out, ORC.system_evaldiff(b), scale, 1, False, RTOL[1]) <= 1.0


@pytest.mark.parametrize("shift", [520, -560])
@pytest.mark.parametrize("prec,cplx", [(1, False), (2, True), (4, False)])
def test_squares_out_of_range(prec, cplx, shift):
    """x_0 so large or small that its square leaves the range, with
    coefficients that bring its powers back: c x x x is a number."""
    b = wl.eval_batch(77, 2, 5, 9, 6, 3, prec, cplx, expmax=4)
    b.input.reshape(2, 5, -1)[:, 0] *= 2.0 ** shift
    e = ((b.idx == 0) & (np.arange(3) < b.nvr[:, None])) * b.exps
    assert e.max() >= 3
    b.exps[e == 4] = 3
    e = np.minimum(e, 3).max(axis=1)
    b.cff.reshape(len(e), -1)[:] *= np.where(e > 0, 2.0 ** (-np.sign(shift) * 510.0 * np.maximum(e - 1, 0)), 1.0)[:, None]
    ref = ORC.system_evaldiff(b)
    assert np.isfinite(ref).all()
    scale = ORC.system_evaldiff(abs_batch(b))
    for knob in (0, 4):
        assert check_scaled(evaluate(b, knob), ref, scale, prec, cplx, RTOL[prec]) <= 1.0
