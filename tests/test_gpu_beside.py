"""A small context beside one that is too large for the resident step kernel:
it steps by graphs while the other is at work and by the resident kernel when it
is not, to the same bits."""
import threading
import time

import numpy as np
import pytest

from crushrs_b200 import scenarios as S
from crushrs_b200.engine import Context
from crushrs_b200.native import check, lib

pytestmark = pytest.mark.gpu


def _crash(size, n, **settings):
    a = S.vehicle(2000.0, (3 * n * size, n * size, n * size), S.honeycomb(5e6, 120.0, 0.4e6, 0.2e6, densification=(0.8, 5e6)))
    b = S.vehicle(1400.0, (3 * n * size, n * size, n * size), S.honeycomb(5e6, 90.0, 0.25e6, 0.2e6, densification=(0.8, 5e6)))
    return S.Model.build(S.scenario(a, b, 14.0, 12.0, element_size=size, **settings))


def _outcome(ctx):
    r = ctx.results()
    return (r.time, r.steps, r.eroded_elements, r.dt_min, r.status,
            [(list(r.vehicle[k].delta_v), r.vehicle[k].crush) for k in range(r.n_vehicles)])


def _launches(ctx, steps):
    before = ctx.launches()
    ctx.run_steps(steps)
    return ctx.launches() - before


def _graphs_beside(ctx, big, steps):
    """Whether ctx takes `steps` steps by graphs right behind an issue of the
    large context's (which counts as at work for 5 ms from then on, so a host
    that is slower in between tries again); the steps taken."""
    for k in range(1, 6):
        check(lib().crush_run_issue(big.h, 20))
        if _launches(ctx, steps) > 100:
            return k * steps
    raise AssertionError("stayed resident beside the large context")


def test_changes_over_and_back():
    small, large = _crash(0.2, 4), _crash(0.04, 28, max_steps=400)  # 384 and 131,712 elements
    alone, ctx, big = Context(small.desc), Context(small.desc), Context(large.desc)
    for c in (alone, ctx, big):
        c.run_begin()
    time.sleep(0.05)
    assert _launches(ctx, 40) < 10  # the large context is idle
    steps = 40 + _graphs_beside(ctx, big, 40)
    steps += _graphs_beside(ctx, big, 27)
    big.run_steps(0)
    time.sleep(0.05)
    assert _launches(ctx, 33) < 10
    check(lib().crush_run_issue(big.h, 100))
    big.close()
    assert _launches(ctx, 60) < 10
    alone.run_steps(steps + 93)
    assert _outcome(ctx) == _outcome(alone)
    for x, y in zip(ctx.state(), alone.state()):
        assert np.array_equal(x, y)


def test_threads():
    small, large = _crash(0.2, 4, end_time=0.03), _crash(0.04, 28, max_steps=400)
    want = []
    for m in (small, large):
        c = Context(m.desc)
        c.run()
        want.append(_outcome(c))
        c.close()
    ctxs = [Context(small.desc), Context(small.desc), Context(large.desc)]
    errors, stop = [], threading.Event()

    def work(ctx, expected, once):
        try:
            while True:
                ctx.run()
                assert _outcome(ctx) == expected
                if once or stop.is_set():
                    break
        except Exception as e:  # noqa: BLE001 - reported by the test's thread
            errors.append(e)
        finally:
            if once:
                stop.set()

    threads = [threading.Thread(target=work, args=(c, want[k == 2], k == 2)) for k, c in enumerate(ctxs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
