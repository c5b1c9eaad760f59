"""Fisher information against a reference that is good to 64 bits: K_nu and dK_nu/dnu by the
trapezoid rule on the integral of exp(-x cosh t) cosh(nu t), which converges geometrically.

Tolerance: the information matrices A, scaled to unit diagonal, so that no conditioning of A
enters.  dC/dnu is a six-point difference of table values good to 4e-15 (relative): the
weights give (90 + 18 + 2) / (60 h) 4e-15 = 3.7e-12 at h = 2e-3, its truncation
h^6 / 140 d^7 less than that; twice for a product of two derivatives, and 2e-12 for the
solves (kappa(C) < 1e3): 1e-11."""
import numpy as np
import pytest
import scipy.linalg
import scipy.special

import exageostatcpp_b200 as egs

pytestmark = pytest.mark.gpu


def _bessel(x, nu):
    """K_nu(x), dK_nu/dnu and K_nu+1(x)."""
    h, k, d, k1 = 0.125, 0.5 * np.exp(-x), np.zeros_like(x), 0.5 * np.exp(-x)
    for i in range(1, int((np.arccosh(110.0 / min(100.0, x.min())) + 0.5) / h) + 2):
        t = i * h
        e = np.exp(-x * np.cosh(t))
        k += e * np.cosh(nu * t)
        d += e * (t * np.sinh(nu * t))
        k1 += e * np.cosh((nu + 1.0) * t)
    return h * k, h * d, h * k1


def _information(x, y, theta):
    s2, beta, nu = theta
    off = ~np.eye(len(x), dtype=bool)
    r = (np.hypot(x[:, None] - x, y[:, None] - y) / beta)[off]
    k, dk, k1 = _bessel(r, nu)
    con, rn = 1.0 / (2.0 ** (nu - 1.0) * scipy.special.gamma(nu)), r ** nu
    der = [np.eye(len(x)), np.zeros((len(x), len(x))), np.zeros((len(x), len(x)))]
    der[0][off] = con * rn * k
    der[1][off] = s2 * con / beta * rn * (r * k1 - 2.0 * nu * k)
    der[2][off] = s2 * con * rn * ((np.log(r) - np.log(2.0) - scipy.special.digamma(nu)) * k + dk)
    c = scipy.linalg.cho_factor(s2 * der[0], lower=True)
    m = [scipy.linalg.cho_solve(c, d) for d in der]
    return np.array([[0.5 * np.sum(p * q.T) for q in m] for p in m])


@pytest.mark.parametrize("n,dts,theta", [(300, 128, (1.2, 0.03, 0.8)), (450, 192, (0.7, 0.02, 0.5)),
                                         (400, 320, (1.0, 0.015, 2.3)), (193, 64, (1.5, 0.05, 0.35))])
def test_information_to_eleven_digits(n, dts, theta):
    x, y = egs.generate_locations(n, 9)
    got = np.linalg.inv(egs.fisher_host(x, y, theta, dts))
    ref = _information(x, y, theta)
    scale = np.sqrt(np.diag(ref))
    assert np.abs((got - ref) / np.outer(scale, scale)).max() <= 1e-11
