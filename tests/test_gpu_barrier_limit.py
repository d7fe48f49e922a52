"""The resident step kernel's barriers give up after a set number of polls: the
blocks leave, every call that reads the run says so however many launches
followed, and the context is as good as new for drop-in calls and the next
run. (A limit of 0 gives up at the first barrier, larger ones somewhere in the
first steps or not at all.)"""
import numpy as np
import pytest

from crushrs_b200 import abi, scenarios as S
from crushrs_b200.engine import Context
from crushrs_b200.native import CrushError, check, lib

pytestmark = pytest.mark.gpu


def _crash():
    """Fronts of 16 x 16 faces (a dynamic grid each way) and a road."""
    a = S.vehicle(2000.0, (0.8, 1.6, 1.6), S.honeycomb(5e6, 120.0, 0.4e6, 0.2e6, densification=(0.8, 5e6)))
    b = S.vehicle(1400.0, (0.6, 1.6, 1.6), S.honeycomb(5e6, 90.0, 0.25e6, 0.2e6, densification=(0.8, 5e6)))
    return S.Model.build(S.scenario(a, b, 14.0, 12.0, offset=0.1, element_size=0.1, end_time=0.02))


def _outcome(r):
    return (r.time, r.steps, r.eroded_elements, r.dt_min, r.status, [list(r.vehicle[k].delta_v) for k in range(r.n_vehicles)])


def _limit(ctx, polls):
    check(lib().crush_set_barrier_polls(ctx.h, polls))


def _times_out(call, *args):
    with pytest.raises(CrushError) as e:
        call(*args)
    assert e.value.status == abi.CRUSH_ERR_TIMEOUT


@pytest.mark.parametrize("polls", [0, 1, 3, 10])
def test_gives_up_and_begins_anew(polls):
    model = _crash()
    fresh, ctx = Context(model.desc), Context(model.desc)
    want = _outcome(fresh.run())
    for c in (fresh, ctx):
        c.close()
    fresh, ctx = Context(model.desc), Context(model.desc)
    for c in (fresh, ctx):
        c.history_config(1, 100, [model.accelerometer(0)])
    _limit(ctx, polls)
    ctx.run_begin()
    check(lib().crush_run_issue(ctx.h, 2500))  # several launches, nothing read between them
    if polls == 0:
        for _ in range(2):
            _times_out(ctx.results)
            _times_out(ctx.state)
            _times_out(ctx.get_state)
            _times_out(ctx.history)
            _times_out(ctx.batch_done)
            _times_out(ctx.run_steps, 1)
    else:
        try:
            ctx.batch_done()
        except CrushError as e:
            assert e.status == abi.CRUSH_ERR_TIMEOUT
    # drop-in calls find the search's bookkeeping clear
    u = np.random.default_rng(0).normal(scale=0.01, size=3 * model.desc.n_nodes)
    masses, _ = ctx.masses()
    for c in range(model.desc.n_contacts):
        f, g = np.zeros_like(u), np.zeros_like(u)
        assert ctx.contact_apply(c, u, None, masses, 1e-4, f) == fresh.contact_apply(c, u, None, masses, 1e-4, g)
        assert np.array_equal(f, g)
    # so does the next run
    _limit(ctx, 1 << 22)
    assert _outcome(ctx.run()) == want
    assert _outcome(fresh.run()) == want
    for x, y in zip(ctx.state(), fresh.state()):
        assert np.array_equal(x, y)


def test_a_crash_joins_a_run_that_gave_up():
    model = _crash()
    ctx = Context(model.desc, room={"slots": 2, "contacts": 16, "nodes": 30000, "hexes": 20000, "faces": 20000, "primary_nodes": 20000})
    _limit(ctx, 0)
    ctx.run_begin()
    check(lib().crush_run_issue(ctx.h, 40))
    assert ctx.append([model.desc]) == 1
    check(lib().crush_run_issue(ctx.h, 40))
    _times_out(ctx.batch_done)
    _times_out(ctx.results, 1)
    _limit(ctx, 1 << 22)
    ctx.batch_run()
    alone = Context(model.desc)
    want = _outcome(alone.run())
    assert _outcome(ctx.results(0)) == want and _outcome(ctx.results(1)) == want


def test_refuses_a_negative_limit():
    model = _crash()
    ctx = Context(model.desc)
    assert lib().crush_set_barrier_polls(ctx.h, -1) == abi.CRUSH_ERR_INVALID
    assert lib().crush_set_barrier_polls(None, 1) == abi.CRUSH_ERR_INVALID
