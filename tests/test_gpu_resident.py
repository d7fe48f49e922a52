"""The resident step kernel against the step graphs: the same bits, at the
sizes where its dealing of work can go wrong (less than a warp, more elements
than threads), with one crash and several, heavy contact nodes, a dynamic
contact grid, elastic elements, histories at every step, odd stable-dt
cadences, the separation stop rule and calls that split a run anywhere."""
import numpy as np
import pytest

from crushrs_b200 import abi, scenarios as S
from crushrs_b200.calibrate import HeadOn
from crushrs_b200.engine import Context
from crushrs_b200.model import single_hex

pytestmark = pytest.mark.gpu


def _pair(size, n, layout=abi.LAYOUT_HEADON, **settings):
    a = S.vehicle(2000.0, (3 * n * size, n * size, n * size), S.honeycomb(5e6, 120.0, 0.4e6, 0.2e6, densification=(0.8, 5e6)))
    b = S.vehicle(1400.0, (n * size, 3 * n * size, n * size) if layout == abi.LAYOUT_TBONE else (3 * n * size, n * size, n * size),
                  S.honeycomb(5e6, 90.0, 0.25e6, 0.2e6, densification=(0.8, 5e6)))
    return S.Model.build(S.scenario(a, b, 14.0, 0.0 if layout == abi.LAYOUT_TBONE else 12.0, element_size=size, layout=layout, **settings))


def _run(models, chunks, graph, history=None):
    ctx = Context([m.desc for m in models] if len(models) > 1 else models[0].desc)
    if graph:
        ctx.set_tuning(32, 2)  # a schedule fixed by the caller: the step graphs
    for slot, accel in enumerate(history or ()):
        ctx.history_config(1, 400, accel, slot=slot)
    ctx.run_begin()
    for n in chunks:
        ctx.run_steps(n)
    out = [ctx.results(k) for k in range(len(models))], ctx.state(), [ctx.history(k) for k in range(len(history or ()))], ctx.launches()
    ctx.close()
    return out


def _same(models, chunks, history=None):
    a, b = _run(models, chunks, False, history), _run(models, chunks, True, history)
    assert a[3] < b[3] // 4  # a handful of launches: the resident kernel ran
    for x, y in zip(a[0], b[0]):
        for f in ("time", "steps", "eroded_elements", "dt_min", "status"):
            assert getattr(x, f) == getattr(y, f), f
        assert abs(x.added_mass_max - y.added_mass_max) <= 1e-12 * abs(y.added_mass_max)  # a sum of atomics
        for k in range(x.n_vehicles):
            assert list(x.vehicle[k].delta_v) == list(y.vehicle[k].delta_v) and x.vehicle[k].crush == y.vehicle[k].crush
    for x, y in zip(a[1], b[1]):
        assert np.array_equal(x, y)
    for x, y in zip(a[2], b[2]):
        assert x["records"] == y["records"] > 0
        for k in ("time", "step", "parts", "nodes"):
            assert np.array_equal(x[k], y[k]), k


@pytest.mark.parametrize("size, n", [(0.3, 2), (0.2, 5), (0.1, 12), (0.05, 26)])  # 48 ... 105,000 elements and the road
def test_one_crash(size, n):
    _same([_pair(size, n)], [1, 7, 32, 160])


def test_single_element_without_contacts():
    m = single_hex(S.honeycomb(5e6, 100.0, 0.3e6, 0.2e6), side=0.3)
    m.initial_velocity[4:, 2] = -3.0
    _same([m], [20, 3, 57])


@pytest.mark.parametrize("settings", [dict(adaptive_check_steps=7), dict(time_step=2e-5), dict(stop_rule=abi.STOP_SEPARATION, max_steps=333),
                                      dict(end_time=0.004)])
def test_settings(settings):
    _same([_pair(0.2, 5, **settings)], [40, 400])


def test_dynamic_grid_and_heavy_nodes():
    # B's side has 20 x 60 faces (a grid); one stretched face list follows as elements crush
    _same([_pair(0.08, 20, layout=abi.LAYOUT_TBONE)], [100, 300])


def test_batch_with_stops():
    models = [_pair(0.3, 2), _pair(0.2, 4, end_time=0.01), _pair(0.15, 6, layout=abi.LAYOUT_TBONE), _pair(0.2, 5, max_steps=77)]
    _same(models, [20, 100, 300])


def test_elastic_and_history():
    models = [HeadOn(13.5, 13.0).build(S.lincoln_navigator_1999(), S.neon_1996_pulse()),
              S.Model.build(S.barrier(S.neon_1996_pulse(), 15.6))]
    _same(models, [33, 20, 147], [[m.accelerometer(0)] for m in models])
