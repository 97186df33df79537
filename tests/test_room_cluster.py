"""Many steps of a room in one cluster's shared memory (room_kernels.cuh room_steps) against the same
steps one call at a time (room_step) and the oracle: sizes about the cluster's split of the rows, the
block's 512 threads and the largest room a cluster holds, an audit that fails inside the call."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

# nodes (nx, ny): fewer rows than blocks, a row a block, uneven splits, more nodes than threads, a room
# too large for a cluster's shared memory
NODES = [(3, 3), (5, 7), (4, 16), (17, 17), (101, 31), (130, 66), (513, 19), (700, 500)]


def _build(nodes, precision, **kw):
    from pantometry_b200.domains import Room

    nx, ny = nodes
    dx = 0.05
    r = Room((nx - 1) * dx, (ny - 1) * dx, nx, precision=precision, **kw)
    assert r.cells == nodes
    return r, dx


def _pressure(nodes, seed):
    return np.random.RandomState(seed).uniform(-1.0, 1.0, nodes[0] * nodes[1])


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("nodes", NODES)
def test_one_call_of_many_steps_is_many_calls_of_one(nodes, precision):
    a, _ = _build(nodes, precision)
    b, _ = _build(nodes, precision)
    dt = 0.6 * a.max_stable_dt()
    p = _pressure(nodes, 3)
    a.release(p)
    b.release(p)
    for n in (1, 2, 3, 8):
        assert a.step(dt, n) is None
        for _ in range(n):
            assert b.step(dt) is None
        fa, fb = a.fields(), b.fields()
        for k in fa:
            assert np.array_equal(fa[k].view(np.uint64), fb[k].view(np.uint64)), (nodes, n, k)
        la, lb = a.ledger(), b.ledger()
        assert la["steps"] == lb["steps"]
        assert abs(la["total"] - lb["total"]) <= 1e-12 * max(la["scale"], lb["scale"])


@pytest.mark.parametrize("nodes", [(5, 7), (101, 31)])
def test_plain_cluster_steps_match_the_oracle(nodes):
    g, dx = _build(nodes, "f64")
    nx, ny = nodes
    o = oracle.Room((nx - 1) * dx, (ny - 1) * dx, nx)
    p = _pressure(nodes, 5)
    g.release(p)
    o.release(p)
    dt = 0.7 * g.max_stable_dt()
    assert g.step(dt, 300) is None
    assert o.step(dt, 300) is None
    fg, fo = g.fields(), o.fields()
    for k in fg:
        assert np.array_equal(fg[k].view(np.uint64), fo[k].view(np.uint64)), k


@pytest.mark.parametrize("nodes", [(17, 17), (130, 66)])
def test_a_failed_audit_inside_the_call_leaves_that_steps_state(nodes):
    a, _ = _build(nodes, "f32")
    b, _ = _build(nodes, "f32")
    dt = 0.6 * a.max_stable_dt()
    p = _pressure(nodes, 9)
    for r in (a, b):
        r.release(p)
        assert r.step(dt, 6) is None
        r.set_tolerance(0.0)  # the first step whose FP64 sum moves at all
    v = a.step(dt, 50)
    assert v is not None and v["quantity"] == "energy" and 1 <= v["step"] < 50
    w = None
    for n in range(v["step"]):
        assert w is None
        w = b.step(dt)
    # the two reductions associate differently, so the exact step of a zero tolerance may differ: the
    # state is compared at the cluster's
    b.set_tolerance(-1.0)
    fa, fb = a.fields(), b.fields()
    assert a.ledger()["steps"] == 6 + v["step"]
    if b.ledger()["steps"] == a.ledger()["steps"]:
        for k in fa:
            assert np.array_equal(fa[k].view(np.uint64), fb[k].view(np.uint64)), k
    # and the run goes on from there
    a.set_tolerance(-1.0)
    assert a.step(dt, 5) is None
