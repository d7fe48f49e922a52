"""The face pass of step sequences on one lane per face and on four: a crash's
bits do not depend on how many faces its context holds, nor on the exhaustive
search, which keeps four."""
import pytest

from crushrs_b200 import scenarios as S
from crushrs_b200.engine import Context

pytestmark = pytest.mark.gpu


def _crash(n):
    size = 0.25
    a = S.vehicle(2000.0, (3 * n * size, n * size, n * size), S.honeycomb(5e6, 120.0, 0.4e6, 0.2e6, densification=(0.8, 5e6)))
    b = S.vehicle(1400.0, (3 * n * size, n * size, n * size), S.honeycomb(5e6, 90.0, 0.25e6, 0.2e6, densification=(0.8, 5e6)))
    return S.Model.build(S.scenario(a, b, 14.0, 12.0, element_size=size))


def _outcome(ctx, slot=0):
    r = ctx.results(slot)
    return (r.time, r.steps, r.eroded_elements, r.dt_min, r.status,
            [(list(r.vehicle[k].delta_v), r.vehicle[k].crush) for k in range(r.n_vehicles)])


# 2 x 25 moving faces a crash: 3950, 4000 and 4050
@pytest.mark.parametrize("crashes", [79, 80, 81])
@pytest.mark.parametrize("exhaustive", [False, True])
def test_same_crash(crashes, exhaustive):
    model = _crash(5)
    contacts = [model.desc.contacts[k].n_faces for k in range(model.desc.n_contacts)]
    assert contacts.count(25) == 2
    ctxs = [Context(model.desc), Context([model.desc] * crashes)]
    for c in ctxs:
        c.set_tuning(32, 2)
        c.set_contact_search(exhaustive)
        c.run_begin()
        c.run_steps(130)
    want = _outcome(ctxs[0])
    for k in range(crashes):
        assert _outcome(ctxs[1], k) == want
