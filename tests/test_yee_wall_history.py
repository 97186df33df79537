"""A wall set open on a cavity that has already stepped, an obstacle beside it: the reference keeps E after
the walls and before the obstacles are zeroed as Mur's history (cavity.rs:1159-1163, 1497-1499) whichever
walls are open then, so the wall's first update reads what the obstacle's edges held."""
import numpy as np
import pytest

from helpers import assert_bitexact, cavity_pair

COUNTS = (12, 10, 9)


def _run(wall, depth):
    """The pair after ten steps with the wall across from `wall` open and twenty more with `wall` open too."""
    axis, high = wall // 2, wall % 2
    solid = np.zeros(COUNTS[::-1], dtype=np.uint8)
    at = [slice(3, 6)] * 3
    cell = COUNTS[axis] - 1 - depth if high else depth
    at[2 - axis] = slice(cell, cell + 1)
    solid[tuple(at)] = 1
    o, g = cavity_pair(COUNTS, 1e-3)
    o.set_boundary(wall ^ 1, 2)
    g.set_boundary(wall ^ 1, 2)
    r = np.random.RandomState(wall)
    fields = {k: r.uniform(-1.0, 1.0, v) * (1.0 if k[0] == "e" else 1.0 / 377.0) for k, v in g.shapes().items()}
    o.set_fields(fields, True)
    g.set_fields(fields, True)
    o.obstruct(solid.reshape(-1))
    g.obstruct(solid.reshape(-1))
    dt = 0.9 * o.courant_limit()
    assert o.step(dt, 10) is None and g.step(dt, 10) is None
    o.set_boundary(wall, 2)
    g.set_boundary(wall, 2)
    assert o.step(dt, 20) is None and g.step(dt, 20) is None
    return o.fields(), g.fields()


@pytest.mark.gpu
@pytest.mark.parametrize("depth", [0, 1, 2])  # the obstacle on the wall, beside it and off it
@pytest.mark.parametrize("wall", range(6))
def test_plain_form_is_bit_exact(wall, depth):
    want, got = _run(wall, depth)
    for k in want:
        assert_bitexact(k, got[k], want[k])


@pytest.mark.gpu
def test_a_kept_history_follows_the_fields_out_of_the_padded_lattice():
    """FP32: E rewritten between steps, so the history is kept aside, then media with conductivity, which only
    the reference layout steps. Open walls read that history in the next step."""
    o, g = cavity_pair(COUNTS, 1e-3, precision="f32")
    r = np.random.RandomState(3)
    size = {k: 1.0 if k[0] == "e" else 1.0 / 377.0 for k in g.shapes()}
    first = {k: r.uniform(-1.0, 1.0, v) * size[k] for k, v in g.shapes().items()}
    second = {k: r.uniform(-1.0, 1.0, v) * size[k] for k, v in g.shapes().items()}
    sigma = 0.01 * r.rand(int(np.prod(COUNTS)))
    dt = 0.9 * o.courant_limit()
    for c in (o, g):
        for w in range(6):
            c.set_boundary(w, 2)
        c.set_fields(first, True)
        assert c.step(dt, 5) is None
        c.set_fields(second, True)
        (c.set_cells if c is o else c.fill_cells)(sigma=sigma)
        assert c.step(dt, 1) is None
    want, got = o.fields(), g.fields()
    # six steps, each value formed from itself and four others by at most eight roundings of 2^-24
    for c in "eh":
        top = max(max(np.abs(want[k]).max() for k in want if k[0] == c), 1.0 if c == "e" else 1.0 / 377.0)
        for k in want:
            if k[0] == c:
                assert np.abs(got[k] - want[k]).max() < 6 * 8 * 5 * 2.0**-24 * top, k
