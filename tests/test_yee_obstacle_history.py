"""Mur's history after steps in a box of conducting walls with an obstacle beside one: what the reference kept
is E before the obstacle's edges were zeroed (cavity.rs:1159-1163, 1497-1499), and the wall set open next
reads it, whatever rewrote E or the media in between. Plain f64 bit for bit with the oracle, FP32 within
its rounding (media with conductivity take it from the padded lattice to the reference layout)."""
import numpy as np
import pytest

from helpers import assert_bitexact, cavity_pair

pytestmark = pytest.mark.gpu

COUNTS = (12, 10, 9)
N = int(np.prod(COUNTS))


def _solid(wall, depth):
    axis, high = wall // 2, wall % 2
    m = np.zeros(COUNTS[::-1], dtype=np.uint8)
    at = [slice(2, 6)] * 3
    cell = COUNTS[axis] - 1 - depth if high else depth
    at[2 - axis] = slice(cell, cell + 1)
    m[tuple(at)] = 1
    return m.reshape(-1)


def _between(what, dt, fields):
    """What happens to the pair between the steps and the wall's opening."""
    eps = np.where(np.arange(N) % 5 == 0, 2.0, 1.0)
    more = np.zeros(COUNTS[::-1], dtype=np.uint8)
    more[4, 5, 6] = 1
    return {
        "nothing": lambda c, o: None,
        "release": lambda c, o: c.release_mode((2, 1), 0.5, dt),
        "obstruct": lambda c, o: c.obstruct(more.reshape(-1)),
        "media": lambda c, o: (c.set_cells if o else c.fill_cells)(eps_r=eps),
        "lossy": lambda c, o: (c.set_cells if o else c.fill_cells)(sigma=0.02 * (eps - 1.0)),
        "upload": lambda c, o: c.set_fields(fields, True),
        "upload and a step": lambda c, o: (c.set_fields(fields, True), c.step(dt, 1)),
    }[what]


def _run(wall, depth, media, between, precision):
    o, g = cavity_pair(COUNTS, 1e-3, precision=precision)
    r = np.random.RandomState(wall)
    if media:
        eps, sigma = 1.0 + 3.0 * r.rand(N), 0.03 * r.rand(N)
        o.set_cells(eps_r=eps, sigma=sigma)
        g.fill_cells(eps_r=eps, sigma=sigma)
    f = {k: r.uniform(-1.0, 1.0, v) * (1.0 if k[0] == "e" else 1.0 / 377.0) for k, v in g.shapes().items()}
    dt = 0.9 * o.courant_limit()
    act = _between(between, dt, f)
    for c, oracle_side in ((o, True), (g, False)):
        c.set_fields(f, True)
        c.obstruct(_solid(wall, depth))
        assert c.step(dt, 9) is None
        act(c, oracle_side)
        c.set_boundary(wall, 2)
        assert c.step(dt, 1) is None
        c.set_boundary(wall ^ 1, 2)
        assert c.step(dt, 15) is None
    return o.fields(), g.fields()


@pytest.mark.parametrize("depth", [0, 1, 2])
@pytest.mark.parametrize("wall", range(6))
def test_a_wall_opened_after_conducting_steps(wall, depth):
    want, got = _run(wall, depth, False, "nothing", "f64")
    for k in want:
        assert_bitexact(k, got[k], want[k])


@pytest.mark.parametrize("between", ["nothing", "release", "obstruct", "media", "lossy", "upload", "upload and a step"])
@pytest.mark.parametrize("media", [False, True], ids=["vacuum", "lossy media"])
@pytest.mark.parametrize("wall", [1, 2])
def test_whatever_rewrote_the_state_between(wall, media, between):
    want, got = _run(wall, 1, media, between, "f64")
    for k in want:
        assert_bitexact(k, got[k], want[k])


@pytest.mark.parametrize("between", ["nothing", "release", "media", "lossy", "upload"])
def test_f32_stays_within_rounding(between):
    want, got = _run(1, 1, False, between, "f32")
    # 25 steps, each value formed from itself and four others by at most eight roundings of 2^-24
    for c in "eh":
        top = max(max(np.abs(want[k]).max() for k in want if k[0] == c), 1.0 if c == "e" else 1.0 / 377.0)
        for k in want:
            if k[0] == c:
                assert np.abs(got[k] - want[k]).max() < 25 * 8 * 5 * 2.0**-24 * top, k
