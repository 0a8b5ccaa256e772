"""GPU test of the tracker's launch variants by batch size: at the edges of
the rule (one path, four per SM, one more) the end points and the counters
equal those of the 64-register variant bit for bit."""
import numpy as np
import pytest

from phcpack_b200 import _lib
from phcpack_b200 import homotopy as hm

pytestmark = pytest.mark.gpu


def track(pb, variant):
    import torch
    dt = hm.DeviceTracker(pb)
    _lib.call("phc_tune_set", 1, variant)
    try:
        dt.run(pmode=1, rmode=2)
        torch.cuda.synchronize()
    finally:
        _lib.call("phc_tune_set", 1, 0)
    return dt.xend.cpu().numpy(), dt.info.cpu().numpy(), dt.dinfo.cpu().numpy()


@pytest.mark.parametrize("extra", [None, 0, 1])
def test_variants_agree(extra):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    npaths = 1 if extra is None else min(4 * sms + extra, 1024)
    pb = hm.subset(hm.config4(seed=6), np.arange(npaths))
    for a, b in zip(track(pb, 0), track(pb, 1)):
        assert np.array_equal(a, b)
