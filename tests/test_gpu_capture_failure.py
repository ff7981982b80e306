"""A trajectory graph that cannot be made (here: instantiated while the caller captures another
stream, which the runtime refuses) is an error of that call alone and leaves no graph behind."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def hmc():
    import gauge_higgs_b200 as gh
    h = gh.GaugeHiggsHMC([4, 4, 4, 4], gh.FundamentalRep(3), seed=5, beta=5.7, kappa=0.1, lam=0.5, nmd=4, tau=0.2)
    h.hot(0.5)
    h.phi_gaussian(12345, 0.3)
    h.sync()
    return h


def test_next_trajectory_is_right():
    import torch
    import gauge_higgs_b200 as gh
    a, b = hmc(), hmc()
    want = a.run(3)
    x = torch.zeros(8, device="cuda")
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        g.capture_begin(capture_error_mode="global")
        x.add_(1)
        with pytest.raises(gh.GaugeHiggsError, match="(?i)graph ?instantiat"):
            b.run(1)
        try:
            g.capture_end()
        except RuntimeError:      # the refused call ends the caller's capture too
            pass
    torch.cuda.synchronize()
    assert np.array_equal(b.run(3), want)
    a.close()
    b.close()
