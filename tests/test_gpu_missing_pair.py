"""Crashes whose gridded contacts keep no primary node (two vehicles that pass
each other): the resident step kernel leaves the grids' counts at zero for
whatever searches next — the same context's next run, a drop-in call, a
gridded crash that joins."""
import numpy as np
import pytest

from crushrs_b200 import scenarios as S
from crushrs_b200.engine import Context

pytestmark = pytest.mark.gpu


def _crash(offset, end_time=0.02):
    """Fronts of 16 x 16 faces: a grid each way."""
    a = S.vehicle(2000.0, (0.8, 1.6, 1.6), S.honeycomb(5e6, 120.0, 0.4e6, 0.2e6, densification=(0.8, 5e6)))
    b = S.vehicle(1400.0, (0.6, 1.6, 1.6), S.honeycomb(5e6, 90.0, 0.25e6, 0.2e6, densification=(0.8, 5e6)))
    return S.Model.build(S.scenario(a, b, 14.0, 12.0, offset=offset, element_size=0.1, end_time=end_time))


def _outcome(ctx, slot=0):
    r = ctx.results(slot)
    return (r.time, r.steps, r.eroded_elements, r.dt_min, r.status, [list(r.vehicle[k].delta_v) for k in range(r.n_vehicles)])


def _pair_contacts(model):
    """The contacts between the vehicles: every one with 256 faces."""
    return [k for k in range(model.desc.n_contacts) if model.desc.contacts[k].n_faces == 256]


def test_run_again_and_drop_in():
    model = _crash(4.0)
    ids = _pair_contacts(model)
    assert len(ids) == 2
    fresh, ctx = Context(model.desc), Context(model.desc)
    fresh.run()
    for _ in range(3):
        before = ctx.launches()
        ctx.run()
        assert ctx.launches() - before < 60  # the resident kernel ran
        assert _outcome(ctx) == _outcome(fresh)
        for x, y in zip(ctx.state(), fresh.state()):
            assert np.array_equal(x, y)
    u = np.random.default_rng(0).normal(scale=0.01, size=3 * model.desc.n_nodes)
    masses, _ = ctx.masses()
    other = Context(model.desc)
    for c in ids:
        f, g = np.zeros_like(u), np.zeros_like(u)
        assert ctx.contact_apply(c, u, None, masses, 1e-4, f) == other.contact_apply(c, u, None, masses, 1e-4, g)
        assert np.array_equal(f, g)


def test_gridded_crash_joins():
    miss, hit = _crash(4.0, end_time=0.03), _crash(0.1)
    assert len(_pair_contacts(hit)) == 2
    want, passing = Context(hit.desc), Context(miss.desc)
    want.run()
    passing.run()
    ctx = Context(miss.desc, room={"slots": 2, "contacts": 16, "nodes": 30000, "hexes": 20000, "faces": 20000, "primary_nodes": 20000})
    ctx.run_begin()
    ctx.run_steps(120)
    slot = ctx.append([hit.desc])
    done = False
    while not done:
        done = ctx.run_steps(40)
    assert _outcome(ctx, 0) == _outcome(passing) and _outcome(ctx, slot) == _outcome(want)
