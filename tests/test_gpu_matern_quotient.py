"""The generator's quotient dist / beta (a product with 1 / beta, corrected by its exact
residual) against the plugin entry's division: with nu = 1/2 both end in sigma^2 exp(-x),
so the entries are equal bit for bit if and, away from tiny x, only if the quotients are.
Distances inside the table's range and outside it, zero, and products with 1 / beta that
overflow or underflow."""
import ctypes

import numpy as np
import pytest

import exageostatcpp_b200 as egs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [0.1, 3.7e-3, 1.7e5, 1e-310, 5e-324, 1e300])
def test_entries_equal_those_of_the_division(beta):
    torch = pytest.importorskip("torch")
    n, lib = 640, egs.load_library()
    rng = np.random.default_rng(5)
    # x = dist / beta from 2^-40 to beyond the table, dense where exp(-x) shows the last bit
    scaled = np.concatenate([np.exp2(rng.uniform(-40.0, 12.0, n // 2)), rng.uniform(0.5, 700.0, n // 2)])
    with np.errstate(over="ignore"):
        x = np.minimum(scaled * beta, 1e306)
    y = np.zeros(n)
    x[7], x[8], x[9] = 0.0, 0.0, 1e-320
    theta = np.array([1.3, beta, 0.5])
    p = egs.Problem(n, 320)
    p.set_locations(x, y)
    p.generate(theta)
    got = p.lower_matrix()
    p.close()
    dx, dy = torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda")
    a = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in (a, dx, dy)]
    egs._check(lib.egs_matern_block(ptr[0], n, n, n, ptr[1], ptr[2], ptr[1], ptr[2], theta.ctypes.data_as(egs._D), 0,
                                    None), "egs_matern_block")
    torch.cuda.synchronize()
    ref = np.tril(a.cpu().numpy().reshape(n, n).T)
    assert np.all(np.isfinite(ref))
    assert np.array_equal(got, ref)
