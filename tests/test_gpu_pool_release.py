"""Freed memory that the library's pool holds on to is there for an allocation that would
otherwise fail, of this library (a batch) and of another one in the process (torch)."""
import numpy as np
import pytest

import exageostatcpp_b200 as egs

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.mark.parametrize("who", ["batch", "torch"])
def test_held_memory_does_not_refuse_an_allocation(who):
    torch = pytest.importorskip("torch")

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0] // MB

    torch.cuda.empty_cache()
    egs.Problem(14000, 960).close()  # 885 MB of tiles, freed into the pool
    fill = torch.empty((free() - 600) * MB, dtype=torch.uint8, device="cuda")
    assert free() <= 600
    try:
        if who == "torch":
            more = torch.empty(900 * MB, dtype=torch.uint8, device="cuda")
            del more
        else:
            x, y = egs.generate_locations(3200, 3)
            B = 20  # 45 MB of tiles each
            b = egs.Batch(np.full(B, 3200), np.tile(x, B), np.tile(y, B), np.tile(x, B), 320)
            assert b.info()["bytes"] > 850 * MB
            b.close()
    finally:
        del fill
        torch.cuda.empty_cache()
