"""A run that leaves the resident step kernel, or comes back to it, at any step:
the bits of a run that never changes over. The step graphs' kernels visit the
chunks of lists that a lone crash's resident steps do not read."""
import numpy as np
import pytest

from crushrs_b200 import scenarios as S
from crushrs_b200.engine import Context

pytestmark = pytest.mark.gpu


def _crash(size=0.2, n=4, **settings):
    a = S.vehicle(2000.0, (3 * n * size, n * size, n * size), S.honeycomb(5e6, 120.0, 0.4e6, 0.2e6, densification=(0.8, 5e6)))
    b = S.vehicle(1400.0, (3 * n * size, n * size, n * size), S.honeycomb(5e6, 90.0, 0.25e6, 0.2e6, densification=(0.8, 5e6)))
    return S.Model.build(S.scenario(a, b, 14.0, 12.0, element_size=size, **settings))


def _outcome(ctx, slot=0):
    r = ctx.results(slot)
    return (r.time, r.steps, r.eroded_elements, r.dt_min, r.status,
            [(list(r.vehicle[k].delta_v), r.vehicle[k].crush) for k in range(r.n_vehicles)])


def _phases(ctx, n):
    ctx.run_steps_timed(n, phases=True)


def _phases_and_back(ctx, n):
    ctx.run_steps_timed(n // 2, phases=True)
    ctx.run_steps_timed(n - n // 2)


def _tuning(ctx, n):
    ctx.set_tuning(32, 2)
    ctx.run_steps(n)


def _fusion(ctx, n):
    ctx.set_step_fusion(True)
    ctx.run_steps(n)


def _exhaustive_and_back(ctx, n):
    ctx.set_contact_search(1)
    ctx.run_steps(n // 2)
    ctx.set_contact_search(0)
    ctx.run_steps(n - n // 2)


@pytest.mark.parametrize("slots", [1, 3])
@pytest.mark.parametrize("first", [7, 20, 33])
@pytest.mark.parametrize("leave", [_phases, _phases_and_back, _tuning, _fusion, _exhaustive_and_back])
def test_leaves_at_any_step(leave, first, slots):
    models = [_crash(n=4 - k) for k in range(slots)]  # a description points into its model
    descs = [m.desc for m in models]
    want, ctx = Context(descs), Context(descs)
    want.run_begin()
    want.run_steps(first + 75)
    ctx.run_begin()
    ctx.run_steps(first)
    leave(ctx, 75)
    for k in range(slots):
        assert _outcome(ctx, k) == _outcome(want, k)
    for x, y in zip(ctx.state(), want.state()):
        assert np.array_equal(x, y)
    assert np.any(ctx.state()[0] != 0.0)


@pytest.mark.parametrize("graph", [False, True])
def test_joins_between_list_builds(graph):
    # a fixed step and a cadence without a step graph: slots may join at any step
    models = [_crash(n=n, time_step=2e-5, adaptive_check_steps=201, end_time=0.003) for n in (4, 3)]
    alone = []
    for m in models:
        alone.append(Context(m.desc))
        alone[-1].run()
    ctx = Context(models[0].desc, room={"slots": 2, "contacts": 16, "nodes": 6000, "hexes": 6000, "faces": 4000, "primary_nodes": 4000})
    if graph:
        ctx.set_tuning(32, 2)
    ctx.run_begin()
    ctx.run_steps(7)
    assert ctx.append([models[1].desc]) == 1
    done = False
    while not done:
        done = ctx.run_steps(31)
    for k in range(2):
        assert _outcome(ctx, k) == _outcome(alone[k])
