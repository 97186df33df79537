"""All magnetic and open walls in one launch (yee_walls), and obstacles zeroed by the step kernels where
they lie off those walls (Cavity::solid_after_walls): boxes down to one and two cells an axis, where
walls meet or stand an edge apart, mixed kinds in orders that make every wall the earlier and the later
of a pair, obstacles on, beside and off the walls. Plain f64 bit for bit with the oracle; FP32 bit for
bit between an obstacle's box stepped in one call and step by step (outside any graph).

A magnetic wall across a one-cell axis is left out: its mirror there is the opposite wall, whose
tangential E the step kernels hold at zero before the walls run, where the reference keeps the last
step's."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

WALLS = ("XLow", "XHigh", "YLow", "YHigh", "ZLow", "ZHigh")
COUNTS = [(1, 5, 4), (2, 2, 2), (3, 2, 7), (9, 8, 7), (33, 9, 5)]
KINDS = [(2, 2, 2, 2, 2, 2), (1, 2, 2, 1, 0, 2), (2, 1, 1, 0, 1, 2), (0, 2, 0, 1, 2, 1), (1, 1, 1, 1, 1, 1)]


def _solid(counts, where):
    nx, ny, nz = counts
    m = np.zeros((nz, ny, nx), dtype=np.uint8)
    if where == "wall":
        m[0, 0, 0] = m[-1, -1, -1] = 1
    elif where == "beside":
        m[min(1, nz - 1), min(1, ny - 1), min(1, nx - 1)] = 1
    elif where == "off" and min(counts) >= 5:
        m[2:nz - 2, 2:ny - 2, 2:nx - 2] = 1
    return m


def _fields(counts, seed):
    from pantometry_b200.domains import Cavity

    r = np.random.RandomState(seed)
    c = Cavity(counts, 1e-3)
    return {k: r.uniform(-1.0, 1.0, v) * (1.0 if k[0] == "e" else 1.0 / 377.0) for k, v in c.shapes().items()}


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("kinds", KINDS)
def test_plain_walls_and_obstacles_match_the_oracle(counts, kinds):
    from pantometry_b200.domains import Cavity

    if counts[0] == 1 and 1 in kinds[:2]:
        pytest.skip("a magnetic wall across a one-cell axis")
    for where in ("none", "wall", "beside", "off"):
        o, g = oracle.Yee(counts, 1e-3), Cavity(counts, 1e-3)
        for w, kind in enumerate(kinds):
            o.set_boundary(w, kind)
            g.set_boundary(w, kind)
        m = _solid(counts, where)
        f = _fields(counts, 7)
        o.set_fields(f, True)
        g.set_fields(f, True)
        if m.any():
            o.obstruct(m)
            g.obstruct(m)
        dt = 0.9 * g.courant_limit()
        for n in (1, 2, 5):
            assert o.step(dt, n) is None
            assert g.step(dt, n) is None
            a, b = g.fields(), o.fields()
            for k in a:
                assert np.array_equal(a[k].view(np.uint64), b[k].view(np.uint64)), (counts, kinds, where, n, k)


@pytest.mark.parametrize("where", ["wall", "off"])
def test_f32_obstacles_and_open_walls_agree_in_and_out_of_a_graph(where):
    from pantometry_b200.domains import Cavity

    counts = (40, 17, 12)
    pair = []
    for _ in range(2):
        c = Cavity(counts, 1e-3, precision="f32")
        for w in WALLS:
            c.set_boundary(w, "open")
        c.obstruct(_solid(counts, where))
        c.set_fields(_fields(counts, 11), True) if where == "off" else None
        c.set_source(20 + 41 * (8 + 18 * 6), np.sin(0.3 * np.arange(200)) * 1e6)
        pair.append(c)
    dt = 0.9 * pair[0].courant_limit()
    assert pair[0].step(dt, 150) is None
    for _ in range(150):
        assert pair[1].step(dt) is None
    a, b = pair[0].fields(), pair[1].fields()
    for k in a:
        assert np.array_equal(a[k], b[k]), (where, k)
