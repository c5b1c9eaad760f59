"""The library's memory pool: what it keeps is bounded, reused memory changes no
result (bit for bit), and several threads can create and destroy problems."""
import functools
import threading

import numpy as np
import pytest

import exageostatcpp_b200 as egs
from oracle import oracle as O

pytestmark = pytest.mark.gpu

KEEP = 1 << 30


@functools.lru_cache(None)
def _points(n):  # the generator draws from the process-wide rand(): main thread only
    return egs.generate_locations(n, 3)


def _eval(n, dts, mixed=False):
    x, y = _points(n)
    p = egs.Problem(n, dts)
    if mixed:
        p.set_precision(egs.EGS_PRECISION_MIXED, 1)
    p.set_locations(x, y)
    p.set_observations(np.sin(7.0 * x) + np.cos(5.0 * y))
    out = [p.mle_eval([1.0, 0.05, 0.8]) for _ in range(2)]
    assert out[0] == out[1]
    p.close()
    return out[0]


def test_kept_memory_is_bounded():
    torch = pytest.importorskip("torch")
    _eval(300, 64)  # contexts, modules, the pool's first chunk
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for n in (20000, 9000, 20000):  # 1.7 GB and 0.35 GB of tiles
        _eval(n, 960)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] >= before - KEEP - (64 << 20)


def test_reused_memory_changes_no_result():
    cases = [(700, 128, False), (3000, 256, True), (1500, 320, False), (64, 64, False)]
    first = [_eval(*c) for c in cases]
    # leave NaN-producing contents behind: a failing factorisation
    p = egs.Problem(3000, 320)
    x, y = egs.generate_locations(3000, 3)
    p.set_locations(x, y)
    p.set_observations(x)
    with pytest.raises(egs.NotPositiveDefinite):
        p.mle_eval([1.0, 50.0, 2.5])
    p.close()
    assert [_eval(*c) for c in reversed(cases)] == first[::-1]
    x, y, z = O.load_data(1100, 5, (1.0, 0.1, 0.5))
    args = (x[:1000], y[:1000], x[1000:], y[1000:], (1.0, 0.1, 0.5), (0.8, 0.12, 0.6), 256)
    a = egs.mloe_mmom_host(*args)
    f = egs.fisher_host(x, y, (1.0, 0.1, 0.8), 320)
    _eval(2000, 192)
    assert egs.mloe_mmom_host(*args) == a
    assert np.array_equal(egs.fisher_host(x, y, (1.0, 0.1, 0.8), 320), f)


def test_threads_create_and_destroy():
    want = {n: _eval(n, 128) for n in (200, 900, 1700)}
    got, errors = [], []

    def work(i):
        try:
            for k in range(4):
                n = (200, 900, 1700)[(i + k) % 3]
                got.append(_eval(n, 128) == want[n])
        except Exception as e:  # reported below
            errors.append(e)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors and len(got) == 16 and all(got)
