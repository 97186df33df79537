"""Magnetic walls across an axis of one cell: the mirror's inner edges lie on the opposite wall, whose
tangential E no update reaches (cavity.rs:1383-1452), so the walls read what the last step left there
(cavity.rs:1170-1236). Plain f64 bit for bit with the oracle, FP32 within its rounding."""
import numpy as np
import pytest

import oracle
from helpers import assert_bitexact

COUNTS = [(1, 5, 4), (5, 1, 4), (5, 4, 1), (1, 1, 6), (1, 33, 9), (1, 1, 1)]
KINDS = [(1, 1, 1, 1, 1, 1), (1, 0, 1, 0, 1, 0), (0, 1, 2, 1, 1, 2), (1, 2, 0, 1, 2, 1), (2, 1, 1, 2, 0, 0), (2, 2, 1, 1, 2, 2)]


def _run(counts, kinds, solid, precision):
    from pantometry_b200.domains import Cavity

    o, g = oracle.Yee(counts, 1e-3), Cavity(counts, 1e-3, precision=precision)
    for w, kind in enumerate(kinds):
        o.set_boundary(w, kind)
        g.set_boundary(w, kind)
    r = np.random.RandomState(7)
    f = {k: r.uniform(-1.0, 1.0, v) * (1.0 if k[0] == "e" else 1.0 / 377.0) for k, v in g.shapes().items()}
    o.set_fields(f, True)
    g.set_fields(f, True)
    if solid:
        m = np.zeros(int(np.prod(counts)), dtype=np.uint8)
        m[-1] = 1
        o.obstruct(m)
        g.obstruct(m)
    dt = 0.9 * g.courant_limit()
    for n in (1, 2, 5, 70):
        assert o.step(dt, n) is None and g.step(dt, n) is None
        yield o.fields(), g.fields()
        if n == 2:  # E rewritten between steps, the edges on the walls with it
            o.set_fields(f, True)
            g.set_fields(f, True)


@pytest.mark.gpu
@pytest.mark.parametrize("solid", [False, True], ids=["empty", "solid"])
@pytest.mark.parametrize("kinds", KINDS)
@pytest.mark.parametrize("counts", COUNTS)
def test_plain_form_is_bit_exact(counts, kinds, solid):
    for want, got in _run(counts, kinds, solid, "f64"):
        for k in want:
            assert_bitexact(f"{counts} {kinds} {k}", got[k], want[k])


@pytest.mark.gpu
@pytest.mark.parametrize("kinds", KINDS[:2])
@pytest.mark.parametrize("counts", COUNTS)
def test_f32_form_stays_within_rounding(counts, kinds):
    # one set of conducting or magnetic walls: a lossless box, whose fields keep their size over 78 steps
    # of at most eight roundings of 2^-24 each
    for want, got in _run(counts, kinds, False, "f32"):
        for c in "eh":
            top = max(max(np.abs(want[k]).max() for k in want if k[0] == c), 1.0 if c == "e" else 1.0 / 377.0)
            for k in want:
                if k[0] == c:
                    assert np.abs(got[k] - want[k]).max() < 78 * 8 * 2.0**-24 * top, (counts, kinds, k)
