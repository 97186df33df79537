"""Films with a finite conductance, formed ahead of the march for a tile's x and y face cells
(heat_kernels.cuh HeatFilmCells): plain f64 blocks at the edges of the tiles (32, 64 or 128 cells by 8
rows, films eight planes at a time), every subset of faces that splits the cells differently between
the slots and the march, bit for bit with the oracle, the state-dependent limit included. FP32 fields
on a radiating block (the one FP32 kernel that forms films ahead) within f32 rounding of the oracle."""
import numpy as np
import pytest

from helpers import heat_pair

pytestmark = pytest.mark.gpu

PLASTIC = dict(density=1240.0, conductivity=0.13, specific_heat=1800.0)
COUNTS = [(1, 1, 1), (1, 9, 8), (2, 8, 9), (3, 1, 17), (33, 9, 8), (34, 17, 7), (64, 8, 16), (65, 7, 9), (128, 9, 3), (132, 1, 2)]
FACES = [(0, 1, 2, 3, 4, 5), (0,), (1, 2), (3, 4), (5,)]


def _films(counts, dx, faces):
    nx, ny, nz = counts
    areas = [ny * nz, ny * nz, nx * nz, nx * nz, nx * ny, nx * ny]
    return [(f, 290.0 + 3.0 * f, 12.0 + f, areas[f] * dx * dx) for f in faces]


def _cells(counts, seed):
    r = np.random.RandomState(seed)
    return 300.0 + 40.0 * r.rand(int(np.prod(counts)))


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("emissivity", [0.0, 0.9])
def test_plain_films_match_the_oracle_bit_for_bit(counts, emissivity):
    dx = 1e-3
    for q, faces in enumerate(FACES):
        o, g = heat_pair(counts, dx, dict(PLASTIC, emissivity=emissivity), 300.0, films=_films(counts, dx, faces),
                         cells=_cells(counts, q))
        dt = 0.8 * o.max_stable_dt()
        assert g.max_stable_dt() == o.max_stable_dt()
        for n in (1, 4):  # one step, and the many-step path where the block takes it
            for _ in range(n):
                assert o.step(dt) is None
            assert g.step(dt, n) is None
            assert np.array_equal(g.cells.view(np.uint64), o.cells.view(np.uint64)), (counts, faces, n)
            assert g.max_stable_dt() == o.max_stable_dt(), (counts, faces, n)


@pytest.mark.parametrize("counts", COUNTS)
def test_radiating_f32_films_stay_within_rounding(counts):
    dx = 1e-3
    for q, faces in enumerate(FACES):
        o, g = heat_pair(counts, dx, dict(PLASTIC, emissivity=0.9), 300.0, films=_films(counts, dx, faces),
                         cells=_cells(counts, q), precision="f32")
        dt = 0.8 * o.max_stable_dt()
        for _ in range(5):
            assert o.step(dt) is None
        assert g.step(dt, 5) is None
        # deviations below 64 K, stored to half an ulp (2^-19 K) a step, five contracting steps
        assert np.abs(g.cells - o.cells).max() < 5 * 4 * 2.0 ** -19, (counts, faces)
