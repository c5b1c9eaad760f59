"""Kriging through the covariance block of the tabulated Matern function: block
edges (256 rows x 16 columns per CTA), every kind of smoothness, coincident points
and distances beyond the table.

Tolerance: the predictions are k^T C^-1 z with kappa(C) < 1e5 here, so the two FP64
solvers agree to sqrt(n) eps kappa < 1e-9 of the largest prediction."""
import numpy as np
import pytest

import exageostatcpp_b200 as egs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu,beta", [(0.5, 0.1), (1.5, 0.05), (0.8, 0.05), (1.0, 0.001), (2.3, 0.03), (8.5, 0.01)])
@pytest.mark.parametrize("n,m", [(1, 1), (255, 16), (300, 17), (513, 1)])
def test_kriging_block(n, m, nu, beta):
    x, y = egs.generate_locations(n + m, 11)
    pick = np.random.default_rng(n).permutation(n + m)
    obs, miss = np.sort(pick[:n]), np.sort(pick[n:])
    z = np.sin(9.0 * x) + y
    xm, ym = x[miss].copy(), y[miss].copy()
    xm[0], ym[0] = x[obs[0]], y[obs[0]]  # a target on an observation: distance 0
    got, mspe = egs.predict_host(x[obs], y[obs], z[obs], xm, ym, (1.0, beta, nu), 128, z[miss])
    ref, ref_mspe = O.predict(x[obs], y[obs], z[obs], xm, ym, (1.0, beta, nu), z[miss])
    scale = max(np.abs(ref).max(), 1e-30)
    assert np.abs(got - ref).max() <= 1e-9 * scale
    assert abs(got[0] - z[obs[0]]) <= 1e-9 * scale
    assert mspe == pytest.approx(ref_mspe, rel=1e-8)
