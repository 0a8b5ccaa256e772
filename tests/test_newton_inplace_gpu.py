"""Newton steps at the full degree read the constants and coefficients where
they lie.  Views that start off the 16 bytes which the evaluation loads at
once give the same series and flags, bit for bit, as aligned arrays."""
import numpy as np
import pytest

from newton_problems import exponential_test_system
from phcpack_b200 import newton

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", ["cst", "cff", "both"])
@pytest.mark.parametrize("prec,cplx", [(1, False), (1, True), (2, False), (4, True)])
def test_unaligned_arrays(prec, cplx, which):
    import torch
    b, _ = exponential_test_system(9, 2, 6, 9, 5, 3, prec, cplx)
    s = torch.cuda.current_stream()
    dn = newton.DeviceNewton(b, szt=3)
    dn.solve(3, s)
    ref = dn.result()
    for name in ("cst", "cff") if which == "both" else (which,):
        a = getattr(dn, name)
        room = torch.empty(a.numel() + 1, dtype=a.dtype, device=a.device)
        room[1:].copy_(a)
        assert room[1:].data_ptr() % 16 == 8
        setattr(dn, name, room[1:])
    dn.solve(3, s)
    for x, y in zip(dn.result(), ref):
        assert np.array_equal(x, y)
