"""Contexts on threads of their own, with slot counts whose launches differ in
shared memory, with and without elastic parts: each run is that of the context
alone, whatever the others launch meanwhile."""
import threading

import pytest

from crushrs_b200 import scenarios as S
from crushrs_b200.calibrate import HeadOn
from crushrs_b200.engine import Context
from crushrs_b200.native import check, lib

pytestmark = pytest.mark.gpu
STEPS = 400


def _crash(n, end_time):
    size = 0.2
    a = S.vehicle(2000.0, (3 * n * size, n * size, n * size), S.honeycomb(5e6, 120.0, 0.4e6, 0.2e6, densification=(0.8, 5e6)))
    b = S.vehicle(1400.0, (3 * n * size, n * size, n * size), S.honeycomb(5e6, 90.0, 0.25e6, 0.2e6, densification=(0.8, 5e6)))
    return S.Model.build(S.scenario(a, b, 14.0, 12.0, element_size=size, end_time=end_time))


def _outcomes(ctx):
    out = []
    for slot in range(ctx.n_slots):
        r = ctx.results(slot)
        out.append((r.time, r.steps, r.eroded_elements, r.dt_min, r.status,
                    [(list(r.vehicle[k].delta_v), r.vehicle[k].crush) for k in range(r.n_vehicles)]))
    return out


@pytest.mark.parametrize("kind, counts", [("honeycomb", [1, 200, 300, 450, 600]), ("elastic", [1, 2, 5, 9])])
def test_slot_counts_side_by_side(kind, counts):
    model = _crash(2, 0.1) if kind == "honeycomb" else HeadOn(13.5, 13.0).build(S.lincoln_navigator_1999(), S.neon_1996_pulse())
    ctxs = [Context([model.desc] * n) for n in counts]
    ctxs[0].run_begin()
    ctxs[0].run_steps(STEPS)
    want = _outcomes(ctxs[0])[0]
    assert want[1] == STEPS
    errors, launches = [], [c.launches() for c in ctxs]
    gate = threading.Barrier(len(ctxs))

    def work(ctx):
        try:
            gate.wait()
            ctx.run_begin()
            for _ in range(STEPS):
                check(lib().crush_run_issue(ctx.h, 1))  # a launch each, without a wait between them
            ctx.batch_done()
            assert _outcomes(ctx) == [want] * ctx.n_slots
        except Exception as e:  # noqa: BLE001 - reported by the test's thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(c,)) for c in ctxs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert all(c.launches() > n for c, n in zip(ctxs, launches))
