"""Part sums of the time histories at the chunk sizes their warps split: one
column of nodes per lane, eight columns per lane, several rounds of columns.
Each recorded mean against an fsum over the part's nodes, within the rounding
bound of any order of n additions."""
import math

import numpy as np
import pytest

from crushrs_b200 import scenarios as S
from crushrs_b200.engine import Context

pytestmark = pytest.mark.gpu


# nodes per chunk of the larger part: 32, 170, 690
@pytest.mark.parametrize("size", [0.3, 0.15, 0.09])
def test_part_means(size):
    a = S.vehicle(2622.0, (6.9, 1.8, 1.5), S.honeycomb(5e6, 140.0, 0.5e6, 0.2e6))
    b = S.vehicle(1354.0, (7.5, 1.8, 1.2), S.honeycomb(5e6, 84.0, 0.3e6, 0.2e6))
    m = S.Model.build(S.scenario(a, b, 13.0, 13.0, element_size=size))
    ctx = Context(m.desc)
    ctx.history_config(5, 4)
    ctx.run_begin()
    ctx.run_steps(5)
    u, v = (x.reshape(-1, 3) for x in ctx.state())
    mass, _ = ctx.masses()
    h = ctx.history()
    ctx.close()
    assert list(h["step"]) == [0, 5]
    for p in range(m.desc.n_parts):
        nodes = np.unique(m.hexes()[m.hex_part() == p])
        w = mass[nodes]
        total = math.fsum(w)
        eps = 4 * len(nodes) * 2.0 ** -53  # n products and n sums of either side, then the division
        rec = h["parts"][1, p]
        assert abs(rec[0] - total) <= eps * total
        for d in range(3):
            for k, x in ((1, v), (4, u)):
                scale = math.fsum(w * np.abs(x[nodes, d])) / total
                assert abs(rec[k + d] - math.fsum(w * x[nodes, d]) / total) <= eps * scale
        kinetic = math.fsum((0.5 * w[:, None] * v[nodes] ** 2).reshape(-1))
        assert abs(rec[10] - kinetic) <= 3 * eps * kinetic
