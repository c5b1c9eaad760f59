"""MLOE / MMOM where the two factors fit on the device but the blocks of 512 targets
beside them do not: smaller groups of targets, the same results."""
import pytest

import exageostatcpp_b200 as egs

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_targets_in_smaller_groups_where_memory_is_short():
    torch = pytest.importorskip("torch")
    n, m = 8000, 500
    x, y = egs.generate_locations(n + m, 7)
    args = (x[:n], y[:n], x[n:], y[n:], (1.0, 0.02, 0.5), (0.8, 0.024, 0.6), 640)
    want = egs.mloe_mmom_host(*args)
    torch.cuda.synchronize()
    egs.Problem(14000, 960).close()  # what the pool holds now is one block, given back below
    free = torch.cuda.mem_get_info()[0] // MB
    # two factors of 298 MB, then 6 x 31 MB of targets with groups of 512, 6 x 4 MB with 64
    fill = []
    try:
        fill.append(torch.empty((free + 100) * MB, dtype=torch.uint8, device="cuda"))
        free = torch.cuda.mem_get_info()[0] // MB
        assert free > 720
        fill.append(torch.empty((free - 720) * MB, dtype=torch.uint8, device="cuda"))
        assert egs.mloe_mmom_host(*args) == want
    finally:
        fill.clear()
        torch.cuda.empty_cache()
