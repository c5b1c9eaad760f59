"""Mixed-precision solves with tiles beyond 4,352, whose vector segment and reduction
buffers together exceed 48 KB of shared memory: two tiles (FP64 and FP32 block below the
diagonal) up to 5,632 and one tile up to 5,888.

Tolerance: the mixed-precision contract, a relative error of 1e-6 against the FP64 oracle."""
import numpy as np
import pytest

import exageostatcpp_b200 as egs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dts,band", [(4700, 4608, 0), (5300, 5120, 1), (5900, 5632, 0), (5700, 5632, 1),
                                        (5800, 5888, 0)])
def test_mixed_solves_of_large_tiles(n, dts, band):
    theta = (1.0, 0.05, 0.5)
    x, y = egs.generate_locations(n, 3)
    z = np.sin(7.0 * x) + np.cos(5.0 * y)
    p = egs.Problem(n, dts)
    p.set_precision(egs.EGS_PRECISION_MIXED, band)
    p.set_locations(x, y)
    p.set_observations(z)
    assert p.ts == dts
    got = p.mle_eval(theta)
    ref = O.mle_loglik(x, y, z, theta, return_parts=True)
    assert np.allclose(got, ref, rtol=1e-6, atol=0.0)
    p.close()
