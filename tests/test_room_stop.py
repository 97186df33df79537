"""Audits that fail inside a call of many room steps (room_kernels.cuh room_steps): the call ends with the
failing step's own state whichever slot of the pressure's ring, parity of the velocities and launch of the
call it falls in. The tolerances lie between the drifts that the same steps show one call at a time."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one block, fewer rows than blocks, a row or two a block, several nodes a thread
NODES = [(3, 3), (17, 17), (40, 33), (130, 66)]
STEPS = 400


def _room(nodes, precision):
    from pantometry_b200.domains import Room

    dx = 0.05
    r = Room((nodes[0] - 1) * dx, (nodes[1] - 1) * dx, nodes[0], precision=precision)
    assert r.cells == nodes
    r.release(np.random.RandomState(11).uniform(-1.0, 1.0, nodes[0] * nodes[1]))
    dt = 0.6 * r.max_stable_dt()
    assert r.step(dt, 2) is None  # past the leapfrog's first step, which sets the books' offset
    return r, dt


def _drifts(room, dt, n):
    """The books' relative change at each of `n` steps, as the audit takes it, one call a step."""
    out = []
    was = room.ledger()
    for _ in range(n):
        assert room.step(dt) is None
        now = room.ledger()
        out.append(abs(now["total"] - was["total"]) / max(abs(was["total"]), abs(now["total"]), was["scale"], now["scale"]))
        was = now
    return np.array(out)


def _same(a, b, what):
    fa, fb = a.fields(), b.fields()
    for k in fa:
        assert np.array_equal(fa[k].view(np.uint64), fb[k].view(np.uint64)), (what, k)


@pytest.mark.parametrize("nodes", NODES)
def test_the_failing_step_leaves_its_own_state(nodes):
    r, dt = _room(nodes, "f32")
    drift = _drifts(r, dt, STEPS)
    seen = set()
    for k in range(0, STEPS - 40, 29):  # calls that begin at step k: their first steps past a tolerance
        high = np.maximum.accumulate(drift[k:])
        # a step that drifts further than all before it in the call, by far more than the two forms' sums differ
        late = [m for m in range(2, high.size) if drift[k + m] > high[m - 1] + 1e-11]
        for m in late[:2]:
            seen.add((m % 2, m % 3))
            a, _ = _room(nodes, "f32")
            b, _ = _room(nodes, "f32")
            if k:
                assert a.step(dt, k) is None and b.step(dt, k) is None
            a.set_tolerance(0.5 * (high[m - 1] + drift[k + m]))
            v = a.step(dt, STEPS)
            assert v is not None and v["quantity"] == "energy" and v["step"] == m + 1
            for _ in range(m + 1):
                assert b.step(dt) is None
            _same(a, b, (k, m, "failed"))
            assert a.ledger()["steps"] == b.ledger()["steps"]
            a.set_tolerance(-1.0)
            assert a.step(dt, 3) is None
            for _ in range(3):
                assert b.step(dt) is None
            _same(a, b, (k, m, "after"))
    assert len(seen) >= 3  # slots of the ring and parities


def test_a_call_longer_than_one_launch():
    nodes = (5, 7)
    a, dt = _room(nodes, "f64")
    b, _ = _room(nodes, "f64")
    assert a.step(dt, 4096 + 3) is None
    for _ in range(4096 + 3):
        assert b.step(dt) is None
    _same(a, b, "long")
    assert a.ledger()["steps"] == b.ledger()["steps"]


def test_a_launch_after_a_failed_audit_changes_nothing():
    nodes = (17, 17)
    r, dt = _room(nodes, "f32")
    drift = _drifts(r, dt, 3)
    a, _ = _room(nodes, "f32")
    b, _ = _room(nodes, "f32")
    a.set_tolerance(0.5 * float(drift.max()))
    m = int(np.argmax(drift > 0.5 * drift.max()))
    v = a.step(dt, 3 * 4096 + 1)
    assert v is not None and v["step"] == m + 1
    for _ in range(m + 1):
        assert b.step(dt) is None
    _same(a, b, m)
