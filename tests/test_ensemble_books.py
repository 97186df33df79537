"""The books of an FP32 ensemble's TMA step (ens_tma.cuh ens_tma_books) by a warp or by a thread block per
block: the stored heat is the sum over the cells, for largest blocks of one brick, on either side of the
line between the two, and of more partials than threads, and for counts about the warps of a thread block."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SUB = dict(density=1000.0, conductivity=100.0, specific_heat=1000.0, emissivity=0.0)


# a brick is 32 x 8 cells by 16 planes
@pytest.mark.parametrize("largest", [(32, 8, 16), (32, 8, 256), (32, 8, 257), (33, 40, 80), (5, 6, 7)])
@pytest.mark.parametrize("count", [1, 7, 8, 9, 17])
def test_stored_heat_is_the_sum_over_the_cells(largest, count):
    from pantometry_b200.domains import Ensemble

    r = np.random.RandomState(count)
    counts = [tuple(int(v) for v in r.randint(3, 20, 3)) for _ in range(count - 1)] + [largest]
    grids = [{"counts": c, "dx": 1e-3, "substance": SUB, "initial": 300.0, "convection": (0.0, math.inf)[q % 2]}
             for q, c in enumerate(counts)]
    for g, limit in zip(grids, Ensemble.max_stable_dt(grids)):
        g["dt"] = 0.9 * limit
    e = Ensemble(grids)
    e.upload(300.0 + 50.0 * r.rand(e.n))
    assert e.step(3) is None
    cells = e.download()
    for q, led in enumerate(e.ledgers()):
        dev = e.block(cells, q) - 300.0
        # FP64 sums of the same f32 deviations, which the download carries to 2^-44 of 350 K each
        cap = SUB["density"] * 1e-9 * SUB["specific_heat"]
        assert abs(led["parts"][0] - cap * dev.sum()) <= cap * dev.size * 350.0 * 2.0**-44, q
        assert led["steps"] == 3
