"""Row scales and slices of the solved panel at the edges of their split: the
smallest tile (128: one warp step covers a strip's columns), an odd number of
steps (640), and more columns than a strip holds in shared memory (3,200, 3,328).

Tolerances: the element-wise bound of the Ozaki update (1e-12 of |L_i||L_j|^T,
seven slices carry 49 bits of each row maximum), and the mixed form's 1e-6
against the plain FP64 evaluation of the same points.
"""
import pytest

import exageostatcpp_b200 as egs
from test_gpu_ozaki_band import RTOL, run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ts,nt,band,k", [(128, 4, 1, 0), (640, 3, 1, 0), (3200, 2, 0, 0)])
def test_band_update_at_the_edges_of_the_strip(ts, nt, band, k):
    assert run_case(ts, nt, band, k, seed=ts) < RTOL


@pytest.mark.parametrize("n,dts,band", [(1500, 256, 1), (9800, 3328, 0)])
def test_mixed_evaluation_at_the_edges_of_the_strip(n, dts, band):
    from oracle import oracle as O
    theta = (1.0, 0.05, 0.5)
    x, y = O.generate_locations(n, O.GlibcRand(4))
    p = egs.Problem(n, dts)
    p.set_locations(x, y)
    z = p.generate_observations(theta, 4)
    p.close()
    out = []
    for form in ((egs.EGS_PRECISION_MIXED, band), ()):
        p = egs.Problem(n, dts, *form)
        p.set_locations(x, y)
        p.set_observations(z)
        out.append(p.mle_eval(theta))
        p.close()
    for a, b in zip(out[0][1:], out[1][1:]):  # log-determinant and quadratic form
        assert abs(a - b) <= 1e-6 * abs(b)
