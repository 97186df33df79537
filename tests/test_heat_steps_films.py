"""Convective films in the many-step kernel (heat_plain_pair_steps): tiles of one plane form them in the march,
thicker ones ahead of it; plain f64 bit for bit with the oracle in tiles of 8 and 32 rows on either side."""
import numpy as np
import pytest

from helpers import heat_pair

pytestmark = pytest.mark.gpu

PLASTIC = dict(density=1240.0, conductivity=0.13, specific_heat=1800.0)
# planes a tile: 1, 1, 2, 2, 4, and 8 with the films' eight planes and a remainder
COUNTS = [(34, 33, 60), (66, 9, 40), (64, 34, 150), (30, 30, 200), (66, 65, 70), (66, 130, 69)]


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("faces", [(0, 1, 2, 3, 4, 5), (1, 2), (4, 5)])
def test_many_convective_steps_match_the_oracle(counts, faces):
    dx = 1e-3
    nx, ny, nz = counts
    areas = [ny * nz, ny * nz, nx * nz, nx * nz, nx * ny, nx * ny]
    films = [(f, 290.0 + 3.0 * f, 12.0 + f, areas[f] * dx * dx) for f in faces]
    cells = 300.0 + 40.0 * np.random.RandomState(nx).rand(nx * ny * nz)
    o, g = heat_pair(counts, dx, PLASTIC, 300.0, films=films, cells=cells)
    assert "pair_steps" in g.step_kernel(3)[0]
    dt = 0.8 * o.max_stable_dt()
    for _ in range(3):
        assert o.step(dt) is None
    assert g.step(dt, 3) is None
    assert np.array_equal(g.cells.view(np.uint64), o.cells.view(np.uint64))
    assert abs(g.ledger()["total"] - o.ledger()["total"]) <= 1e-12 * o.ledger()["scale"]
