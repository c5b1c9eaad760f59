"""The 64-column panel step: factor, carried solve and failing pivots at the
sizes where its outer blocks, chunks and fallbacks change.

Tolerance: a backward-stable factor and solve agree with LAPACK's to about
sqrt(n) eps kappa relative to the largest entry; kappa < 1e4 for these inputs
(an exponential covariance at one to two grid spacings), n <= 1,500:
40 * 2.2e-16 * 1e4 < 1e-10."""
import numpy as np
import pytest
import scipy.linalg

import exageostatcpp_b200 as egs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dts", [(1, 64), (64, 64), (65, 64), (130, 128), (200, 192), (333, 320), (449, 448),
                                   (700, 640), (1100, 320), (963, 64)])
@pytest.mark.parametrize("scale", [1.0, 1e-295, 1e290])
def test_factor_and_carried_solve(n, dts, scale):
    # scale 1e-295 and 1e290 put every pivot outside the range of the fast rsqrt
    theta = [scale, 0.03, 0.5]
    x, y = egs.generate_locations(n, 3)
    z = np.random.default_rng(n).standard_normal(n)
    p = egs.Problem(n, dts)
    p.set_locations(x, y)
    p.set_observations(z)
    ll, logdet, dot = p.mle_eval(theta)
    L = np.linalg.cholesky(O.covariance(x, y, [1.0, 0.03, 0.5]))
    w = scipy.linalg.solve_triangular(L, z, lower=True)
    root = np.sqrt(scale)
    got = p.lower_matrix() / root
    assert np.abs(got - L).max() <= 1e-10 * np.abs(L).max()
    assert np.abs(p.observations() * root - w).max() <= 1e-10 * np.abs(w).max()
    ref = 2.0 * np.log(np.diag(L)).sum() + n * np.log(scale)
    assert abs(logdet - ref) <= 1e-10 * max(1.0, abs(ref))
    assert dot == pytest.approx(w @ w / scale, rel=1e-10)
    # the separate factorisation leaves the observations alone
    p.generate(theta)
    p.restore_observations()
    p.potrf()
    assert np.array_equal(p.observations(), z)
    assert np.array_equal(p.lower_matrix() / root, got)
    p.close()


@pytest.mark.parametrize("n,dts", [(1400, 320), (2700, 320), (3001, 960)])
def test_update_tile_shapes(n, dts):
    # trailing updates of fewer than 148, 148 to 591 and more 64 x 64 tiles
    theta = [1.0, 0.03, 0.5]
    x, y = egs.generate_locations(n, 3)
    p = egs.Problem(n, dts)
    p.set_locations(x, y)
    p.generate(theta)
    p.potrf()
    L = np.linalg.cholesky(O.covariance(x, y, theta))
    assert np.abs(p.lower_matrix() - L).max() <= 1e-10 * np.abs(L).max()
    p.close()


@pytest.mark.parametrize("n,dts,bad", [(300, 320, 0), (300, 320, 63), (300, 320, 64), (300, 320, 201), (700, 192, 390),
                                       (700, 192, 699)])
def test_failing_pivot_is_reported(n, dts, bad):
    x, y = egs.generate_locations(n, 4)
    p = egs.Problem(n, dts)
    p.set_locations(x, y)
    p.generate([1.0, 0.03, 0.5])
    k = bad // p.ts
    t = p.tile(k, k)
    t[bad % p.ts, bad % p.ts] = -1.0
    egs._check(p._lib.egs_set_tile(p._h, k, k, np.asfortranarray(t).ctypes.data_as(egs._D)), "set_tile")
    with pytest.raises(egs.NotPositiveDefinite) as e:
        p.potrf()
    assert e.value.status == bad + 1
    p.generate([1.0, 0.03, 0.5])
    p.potrf()
    p.close()


@pytest.mark.parametrize("n,dts,band", [(1000, 64, 3), (1500, 320, 2), (1300, 192, 7), (900, 128, 100)])
def test_band_update_in_one_launch(n, dts, band):
    theta = [1.0, 0.01, 0.5]
    x, y, z = O.load_data(n, 6, theta)
    p = egs.Problem(n, dts)
    p.set_band(band)
    p.set_locations(x, y)
    p.set_observations(z)
    ref = O.dst_loglik(x, y, z, theta, dts, band, return_parts=True)
    assert np.allclose(p.mle_eval(theta), ref, rtol=1e-10, atol=0.0)
    p.close()
