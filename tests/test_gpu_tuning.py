"""The launch schedule of a context that steps in the resident kernel: asked
for, it is measured and reported, the run goes on as if it had not been, and
fixing it takes the step graphs with it to the same bits."""
import numpy as np
import pytest

from crushrs_b200 import scenarios as S
from crushrs_b200.engine import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 20])  # exhaustive contacts, contacts with a dynamic grid
def test_reported_without_a_trace(n):
    size = 0.8 / n
    a = S.vehicle(2000.0, (1.6, 0.8, 0.8), S.honeycomb(5e6, 120.0, 0.4e6, 0.2e6, densification=(0.8, 5e6)))
    b = S.vehicle(1400.0, (1.2, 0.8, 0.8), S.honeycomb(5e6, 90.0, 0.25e6, 0.2e6, densification=(0.8, 5e6)))
    model = S.Model.build(S.scenario(a, b, 14.0, 12.0, element_size=size))
    want, ctx = Context(model.desc), Context(model.desc)
    assert ctx.tuning()[1] == [0.0] * 6  # no run yet: nothing measured
    for c in (want, ctx):
        c.run_begin()
    want.run_steps(140)
    ctx.run_steps(47)
    lanes, ms = ctx.tuning()
    assert lanes in (1, 2, 4, 8, 16, 32) and min(ms) > 0.0
    assert ctx.tuning() == (lanes, ms)  # measured once
    before = ctx.launches()
    ctx.run_steps(33)
    assert ctx.launches() - before < 10  # still resident
    ctx.fix_schedule()
    ctx.run_steps(60)
    assert ctx.launches() - before > 100  # the step graphs
    assert ctx.tuning() == (lanes, ms)
    for x, y in zip(ctx.state(), want.state()):
        assert np.array_equal(x, y)
    assert ctx.results().steps == want.results().steps == 140
