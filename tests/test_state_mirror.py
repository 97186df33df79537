"""The host's mirror of a handle's state block (Handle::mirror): a handle that keeps it answers every call as
one whose mirror is dropped before the call (`set_stream` drops it and changes nothing else), through
violations, changed tolerances, heat handed in, rewritten states, checkpoints and changed domains."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SUB = dict(density=1240.0, conductivity=0.13, specific_heat=1800.0)


def _noise(n, seed, lo=-1.0, hi=1.0):
    return np.random.RandomState(seed).uniform(lo, hi, n)


def _heat(precision, emissivity, filled):
    from pantometry_b200.domains import Solid3D

    n = (9, 8, 7)
    b = Solid3D(n, 1e-3, **SUB, initial=300.0, emissivity=emissivity, precision=precision)
    cells = int(np.prod(n))
    if filled:
        m = np.zeros(cells, dtype=np.uint8)
        m[: cells // 2] = 1
        b.fill(m, 2500.0, 1.1, 800.0, emissivity)
    for f in range(6):
        b.losing_from(f, 290.0 + f, 20.0, 6e-5)
    b.cells = 300.0 + 20.0 * _noise(cells, 1)
    dt = 0.5 * b.max_stable_dt()
    chip = np.zeros(cells, dtype=np.uint8)
    chip[cells // 3] = 1
    extra = [lambda d: d.absorb(3.0), lambda d: setattr(d, "cells", 310.0 + 10.0 * _noise(cells, 2)),
             lambda d: d.losing_from(1, 280.0, math.inf, 6e-5) if not filled and emissivity == 0.0 else None,
             lambda d: d.max_stable_dt(), lambda d: d.sample((0, 0, 0), (9e-3, 8e-3, 7e-3), (3, 2, 2)).tolist()]
    if precision == "f64" or emissivity == 0.0:
        extra.append(lambda d: d.dissipating(2.0, chip))
    return b, dt, extra, lambda d: {"t": d.cells}


def _bar(precision):
    from pantometry_b200.domains import Bar

    b = Bar(40, 1e-3, 1e-4, **SUB, initial=300.0, precision=precision)
    b.cells = 300.0 + 20.0 * _noise(40, 1)
    extra = [lambda d: d.absorb(2.0), lambda d: d.deposit(1e-2 * _noise(40, 4, 0.0)),
             lambda d: setattr(d, "cells", 310.0 + _noise(40, 2)), lambda d: d.max_stable_dt(),
             lambda d: d.sample((0, 0, 0), (4e-2, 0, 0), (5, 1, 1)).tolist()]
    return b, 0.5 * b.max_stable_dt(), extra, lambda d: {"t": d.cells}


def _hall(precision):
    from pantometry_b200.domains import Hall

    h = Hall(0.55, 0.5, 0.45, 12, 343.0, 1.2, precision=precision)
    h.release(_noise(h.n, 1))
    wave = np.sin(0.3 * np.arange(40))
    extra = [lambda d: d.set_source(d.n // 2, wave), lambda d: d.release(_noise(d.n, 5)), lambda d: d.max_stable_dt(),
             lambda d: d.sample((0, 0, 0), (0.55, 0.5, 0.45), (3, 2, 2)).tolist()]
    return h, 0.5 * h.max_stable_dt(), extra, lambda d: d.fields()


def _room(precision):
    from pantometry_b200.domains import Room

    r = Room(1.0, 0.8, 21, precision=precision)
    r.release(_noise(r.n, 1))
    extra = [lambda d: d.release(_noise(d.n, 5)), lambda d: d.max_stable_dt(),
             lambda d: d.sample((0, 0, 0), (1.0, 0.8, 0), (3, 2, 1)).tolist()]
    return r, 0.5 * r.max_stable_dt(), extra, lambda d: d.fields()


def _tube(precision):
    from pantometry_b200.domains import Tube

    t = Tube(1.0, 50, precision=precision)
    t.release(_noise(50, 1))
    extra = [lambda d: d.release(_noise(50, 5)), lambda d: d.max_stable_dt()]
    return t, 0.5 * t.max_stable_dt(), extra, lambda d: d.fields()


def _cavity(precision):
    from pantometry_b200.domains import Cavity

    c = Cavity((12, 11, 10), 1e-3, precision=precision)
    dt = 0.8 * c.courant_limit()
    c.release_mode((1, 1), 1.0, dt)
    f = {k: _noise(v, 6) * (1.0 if k[0] == "e" else 1.0 / 377.0) for k, v in c.shapes().items()}
    solid = np.zeros(12 * 11 * 10, dtype=np.uint8)
    solid[500] = 1
    extra = [lambda d: d.set_source(6 + 13 * (5 + 12 * 5), 1e3 * np.sin(0.3 * np.arange(60))),
             lambda d: d.energies(), lambda d: d.obstruct(solid), lambda d: d.set_fields(f, True),
             lambda d: d.release_mode((2, 1), 0.5, dt), lambda d: d.set_boundary(1, 2), lambda d: d.courant_limit(),
             lambda d: d.sample((0, 0, 0), (12e-3, 11e-3, 10e-3), (3, 2, 2)).tolist(),
             lambda d: d.fill_cells(eps_r=np.where(np.arange(12 * 11 * 10) % 5 == 0, 2.0, 1.0))]
    return c, dt, extra, lambda d: d.fields()


KINDS = {
    "heat": lambda p: _heat(p, 0.0, False),
    "heat radiating": lambda p: _heat(p, 0.9, False),
    "heat filled": lambda p: _heat(p, 0.0, True),
    "bar": _bar,
    "hall": _hall,
    "room": _room,
    "tube": _tube,
    "cavity": _cavity,
}


def _calls(dt, extra):
    """Steps, ledgers, violations and checkpoints, then each of the domain's other calls between two steps."""
    step = lambda n, h=dt: (lambda d: d.step(h, n))  # noqa: E731
    out = [step(1), lambda d: d.ledger(), step(3), step(2), lambda d: d.ledger(),
           lambda d: d.set_tolerance(0.0), step(4), lambda d: d.ledger(), step(1), step(1),  # an audit that may fail
           lambda d: d.set_tolerance(1e-3), step(2), lambda d: d.ledger(), lambda d: d.set_tolerance(-1.0), step(2),
           step(1, 1e3 * dt), lambda d: d.ledger(), step(2),  # refused: past the stable step
           lambda d: d.checkpoint(), step(3), lambda d: d.ledger(), lambda d: d.restore(), lambda d: d.ledger(), step(3),
           lambda d: d.ledger()]
    for e in extra:
        out += [e, step(1), lambda d: d.ledger(), e, lambda d: d.ledger(), step(2), step(70), lambda d: d.ledger()]
    return out


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("kind", KINDS)
def test_a_kept_mirror_answers_as_a_dropped_one(kind, precision):
    a, dt, extra, fields = KINDS[kind](precision)
    b, _, _, _ = KINDS[kind](precision)
    for q, call in enumerate(_calls(dt, extra)):
        b.set_stream(None)
        ra, rb = call(a), call(b)
        if ra is not a:  # some setters answer with the domain itself
            assert ra == rb, (kind, q, ra, rb)
        fa, fb = fields(a), fields(b)
        for k in fa:
            assert np.array_equal(fa[k].view(np.uint64), fb[k].view(np.uint64)), (kind, q, k)
