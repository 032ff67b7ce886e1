"""Triangle counts on a device with little free memory: where the probing plan
can count, so does the automatic choice, with the same result."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("directed", [False, True])
def test_triangles_without_room_for_the_hub_rows(directed):
    import torch
    from strata_b200 import Engine
    from strata_b200.gpu import OutOfMemory
    rng = np.random.default_rng(2)
    m, nodes = 400_000, 1 << 24  # ids spread over 2^24: the plan's label sort takes 16 bytes an id
    a, b = ((rng.random(m) ** 3 * 20_000).astype(np.uint32) for _ in range(2))
    ids = rng.permutation(nodes)[:20_000].astype(np.uint32)
    ids[0] = nodes - 1
    edges = (ids[np.minimum(a, b)], ids[np.maximum(a, b)])

    def count(probe):
        with Engine(0) as eng:  # its own pool: holds nothing yet
            eng.set_knob(3, probe)
            try:
                return (eng.count_triangle_pattern if directed else eng.count_triangles)(edges)
            except OutOfMemory:
                return None
    want = count(0)  # with room; loads the kernels too
    assert count(2) == want
    counted = []
    for free_mb in (700, 500, 350, 250, 180):
        gc.collect()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        full = torch.empty(free - (free_mb << 20), dtype=torch.uint8, device="cuda")
        try:
            probed, auto = count(2), count(0)
        finally:
            del full
            torch.cuda.empty_cache()
        assert probed in (None, want) and auto in (None, want)
        assert auto == want or probed is None, free_mb
        counted.append(auto)
    assert counted[0] == want
