"""Triangular solves against a finished factor: one vector, forward and backward,
and many right-hand sides as rows (MLOE / MMOM).

Tolerance: a triangular solve is backward stable, so it agrees with LAPACK's to
about sqrt(n) eps kappa(L) relative to the largest entry; kappa(L) < 1e2 for these
inputs (an exponential covariance at one to two grid spacings), n <= 2,000:
45 * 2.2e-16 * 1e2 = 1e-12."""
import numpy as np
import pytest
import scipy.linalg

import exageostatcpp_b200 as egs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dts", [(1, 64), (64, 64), (65, 64), (129, 64), (700, 192), (1000, 960), (2000, 320)])
def test_vector_solves(n, dts):
    theta = [1.3, 0.03, 0.5]
    x, y = egs.generate_locations(n, 5)
    z = np.random.default_rng(n).standard_normal(n)
    p = egs.Problem(n, dts)
    p.set_locations(x, y)
    p.set_observations(z)
    p.generate(theta)
    p.potrf()
    L = p.lower_matrix()
    p.trsv()
    w = scipy.linalg.solve_triangular(L, z, lower=True)
    assert np.abs(p.observations() - w).max() <= 1e-12 * np.abs(w).max()
    egs._check(p._lib.egs_trsv_transpose(p._h), "trsv_transpose")
    v = scipy.linalg.solve_triangular(L, w, lower=True, trans="T")
    assert np.abs(p.observations() - v).max() <= 1e-12 * np.abs(v).max()
    p.close()


@pytest.mark.parametrize("n,m,dts", [(1, 1, 64), (63, 2, 64), (200, 64, 64), (333, 65, 192), (500, 513, 320),
                                     (300, 1100, 128)])
def test_mloe_mmom_target_groups(n, m, dts):
    tt, te = (1.0, 0.05, 0.5), (0.8, 0.06, 0.6)
    x, y = egs.generate_locations(n + m, 7)
    pick = np.random.default_rng(n).permutation(n + m)
    obs, miss = np.sort(pick[:n]), np.sort(pick[n:])
    got = egs.mloe_mmom_host(x[obs], y[obs], x[miss], y[miss], tt, te, dts)
    ref = O.mloe_mmom(x[obs], y[obs], x[miss], y[miss], tt, te)
    assert abs(got[0] - ref[0]) < 1e-10 and abs(got[1] - ref[1]) < 1e-10, (got, ref)


def test_mloe_mmom_reports_a_failing_covariance():
    # two coincident observations: both covariances are singular
    x, y = egs.generate_locations(100, 7)
    x[17], y[17] = x[16], y[16]
    with pytest.raises(egs.NotPositiveDefinite):
        egs.mloe_mmom_host(x[:90], y[:90], x[90:], y[90:], (1.0, 0.05, 1.5), (0.8, 0.06, 1.5), 64)


@pytest.mark.parametrize("n,dts,theta", [(1, 64, (1.0, 0.1, 0.5)), (64, 64, (1.0, 0.05, 1.5)), (65, 64, (0.7, 0.05, 0.3)),
                                         (500, 192, (1.2, 0.03, 1.0)), (700, 320, (1.0, 0.002, 0.8)),
                                         (300, 128, (1.0, 0.02, 6.9)), (300, 128, (1.0, 0.015, 7.5))])
def test_fisher_orders_and_sizes(n, dts, theta):
    # beta = 0.002 puts distances beyond the tables, nu + 1 > 8 turns them off;
    # 1e-7 is the bound of the Richardson derivative in the other Fisher tests
    x, y = egs.generate_locations(n, 9)
    if n == 1:  # one point: no information on beta and nu
        with pytest.raises(egs.EgsError):
            egs.fisher_host(x, y, theta, dts)
        return
    inv = egs.fisher_host(x, y, theta, dts)
    ref = O.fisher_inverse(x, y, theta)
    assert np.abs(inv - ref).max() <= 1e-7 * np.abs(ref).max(), (inv, ref)


@pytest.mark.parametrize("n,dts", [(129, 64), (200, 320), (1000, 960)])
def test_row_sweeps_end_at_the_last_real_block(n, dts):
    # tiles mostly of padding, which the sweeps leave out, and odd numbers of the
    # blocks that the symmetric sweep stops at; tolerances as above
    theta = (1.1, 0.04, 0.8)
    x, y = egs.generate_locations(n + 70, 11)
    inv, ref = egs.fisher_host(x[:n], y[:n], theta, dts), O.fisher_inverse(x[:n], y[:n], theta)
    assert np.abs(inv - ref).max() <= 1e-7 * np.abs(ref).max(), (inv, ref)
    args = (x[:n], y[:n], x[n:], y[n:], theta, (0.9, 0.05, 0.7))
    got, ref = egs.mloe_mmom_host(*args, dts), O.mloe_mmom(*args)
    assert abs(got[0] - ref[0]) < 1e-10 and abs(got[1] - ref[1]) < 1e-10, (got, ref)
