"""The resident step kernel with many crashes of which most are done: more
slots than threads in a block, chunk lists rebuilt as they stop, contexts
whose size alone would be the step graphs', room that is not used."""
import numpy as np
import pytest

from crushrs_b200 import scenarios as S
from crushrs_b200.engine import Context

pytestmark = pytest.mark.gpu


def _crash(size, n, end_time):
    a = S.vehicle(2000.0, (3 * n * size, n * size, n * size), S.honeycomb(5e6, 120.0, 0.4e6, 0.2e6, densification=(0.8, 5e6)))
    b = S.vehicle(1400.0, (3 * n * size, n * size, n * size), S.honeycomb(5e6, 90.0, 0.25e6, 0.2e6, densification=(0.8, 5e6)))
    return S.Model.build(S.scenario(a, b, 14.0, 12.0, element_size=size, end_time=end_time))


def _same(ctx, slot, want):
    got, ref = ctx.results(slot), want.results(0)
    assert (got.time, got.steps, got.eroded_elements, got.dt_min) == (ref.time, ref.steps, ref.eroded_elements, ref.dt_min)
    for k in range(ref.n_vehicles):
        assert list(got.vehicle[k].delta_v) == list(ref.vehicle[k].delta_v) and got.vehicle[k].crush == ref.vehicle[k].crush


def test_many_slots_stopping_apart():
    kinds = [_crash(0.3, 2, 0.004 + 0.004 * k) for k in range(6)]
    alone = []
    for m in kinds:
        ctx = Context(m.desc)
        ctx.run()
        alone.append(ctx)
    ctx = Context([kinds[k % 6].desc for k in range(600)])
    before = ctx.launches()
    ctx.batch_run()
    assert ctx.launches() - before < 60  # a few launches of many steps
    for k in range(600):
        _same(ctx, k, alone[k % 6])


def test_large_context_with_few_running():
    long, short = _crash(0.2, 4, 0.03), _crash(0.05, 19, 0.0008)  # 41,000 elements each, a few steps
    want = Context(long.desc)
    want.run()
    ctx = Context([long.desc] + [short.desc] * 5)  # step graphs, then the resident kernel for the one left
    ctx.batch_run()
    _same(ctx, 0, want)
    end = Context(short.desc)
    end.run()
    for k in range(1, 6):
        _same(ctx, k, end)


def test_room_left_over():
    m = _crash(0.2, 4, 0.01)
    want = Context(m.desc)
    want.run()
    ctx = Context([m.desc, m.desc], room={"slots": 8, "contacts": 64, "nodes": 400000, "hexes": 300000, "faces": 40000, "primary_nodes": 40000})
    ctx.run_begin()
    ctx.run_steps(40)
    first = ctx.append([m.desc, m.desc])
    done = False
    while not done:
        done = ctx.run_steps(40)
    for k in (0, 1, first, first + 1):
        _same(ctx, k, want)
    u, v = ctx.state()
    assert np.all(np.isfinite(u)) and np.all(np.isfinite(v))
