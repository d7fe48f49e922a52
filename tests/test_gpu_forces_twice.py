"""The element kernel of step sequences in its two forms (gradients and base
vectors held in registers, or read twice in large contexts): a crash's bits do
not depend on which one its context takes."""
import pytest

from crushrs_b200 import scenarios as S
from crushrs_b200.engine import Context

pytestmark = pytest.mark.gpu


def _crash(size, n, **settings):
    a = S.vehicle(2000.0, (3 * n * size, n * size, n * size), S.honeycomb(5e6, 120.0, 0.4e6, 0.2e6, densification=(0.8, 5e6)))
    b = S.vehicle(1400.0, (3 * n * size, n * size, n * size), S.honeycomb(5e6, 90.0, 0.25e6, 0.2e6, densification=(0.8, 5e6)))
    return S.Model.build(S.scenario(a, b, 14.0, 12.0, element_size=size, **settings))


def _outcome(ctx, slot=0):
    r = ctx.results(slot)
    return (r.time, r.steps, r.eroded_elements, r.dt_min, r.status,
            [(list(r.vehicle[k].delta_v), r.vehicle[k].crush) for k in range(r.n_vehicles)])


# fillers that put the context below the change of form, and above
@pytest.mark.parametrize("fillers", [4, 5])
def test_same_crash_in_either_form(fillers):
    small, large = _crash(0.2, 7), _crash(0.05, 25)  # 2058 and 93,750 elements
    assert 4 * 93750 + 4 * 2058 < 475000 <= 5 * 93750 + 4 * 2058
    alone = Context(small.desc)
    alone.set_tuning(32, 2)
    ctx = Context([small.desc] * 4 + [large.desc] * fillers)
    for c in (alone, ctx):
        c.run_begin()
        c.run_steps(200)
    for k in range(4):
        assert _outcome(ctx, k) == _outcome(alone)
    want = Context(large.desc)
    want.run_begin()
    want.run_steps(200)
    for k in range(fillers):
        assert _outcome(ctx, 4 + k) == _outcome(want)
