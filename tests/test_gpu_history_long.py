"""Part sums of the time histories where a context holds short part units (a
warp per chunk of nodes) and long ones (a block per chunk) together: the bits of
the one order of summation, recomputed here, in resident steps and step graphs."""
import numpy as np
import pytest

from crushrs_b200 import scenarios as S
from crushrs_b200.engine import Context

pytestmark = pytest.mark.gpu
CHUNKS, COLUMNS, LONG = 32, 256, 8192


def _sum(values):
    """Chunk by chunk: 256 columns of nodes, each added in order, then a tree (column c and c + 128 first)."""
    per = -(-len(values) // CHUNKS)
    total = np.float64(0.0)
    for b in range(CHUNKS):
        chunk = values[b * per : (b + 1) * per]
        columns = np.zeros(COLUMNS)
        for i in range(0, len(chunk), COLUMNS):
            row = chunk[i : i + COLUMNS]
            columns[: len(row)] += row
        while len(columns) > 1:
            half = len(columns) // 2
            columns = columns[:half] + columns[half:]
        total = total + columns[0]
    return total


def _kinetic(w, v):
    """The nodes' three terms go into the column one after the other."""
    per = -(-len(w) // CHUNKS)
    total = np.float64(0.0)
    for b in range(CHUNKS):
        cw, cv = w[b * per : (b + 1) * per], v[b * per : (b + 1) * per]
        columns = np.zeros(COLUMNS)
        for i in range(0, len(cw), COLUMNS):
            n = len(cw[i : i + COLUMNS])
            for d in range(3):
                x = cv[i : i + COLUMNS, d]
                columns[:n] += 0.5 * cw[i : i + COLUMNS] * x * x
        while len(columns) > 1:
            half = len(columns) // 2
            columns = columns[:half] + columns[half:]
        total = total + columns[0]
    return total


def _crash(size, n):
    a = S.vehicle(2000.0, (3 * n * size, n * size, n * size), S.honeycomb(5e6, 120.0, 0.4e6, 0.2e6, densification=(0.8, 5e6)))
    b = S.vehicle(1400.0, (2 * n * size, n * size, n * size), S.honeycomb(5e6, 90.0, 0.25e6, 0.2e6, densification=(0.8, 5e6)))
    return S.Model.build(S.scenario(a, b, 14.0, 12.0, element_size=size))


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("sizes", [[3, 5], [13, 4, 15], [14]])  # parts of 48 ... 11,776 nodes
def test_bits(sizes, graph):
    models = [_crash(1.2 / n, n) for n in sizes]
    ctx = Context([m.desc for m in models])
    if graph:
        ctx.set_tuning(32, 2)
    for k in range(len(models)):
        ctx.history_config(5, 4, slot=k)
    ctx.run_begin()
    ctx.run_steps(10)
    u, v = (x.reshape(-1, 3) for x in ctx.state())
    mass, _ = ctx.masses()
    node0, longest = 0, 0
    for k, m in enumerate(models):
        h = ctx.history(k)
        assert list(h["step"]) == [0, 5, 10]
        for p in range(m.desc.n_parts):
            nodes = node0 + np.unique(m.hexes()[m.hex_part() == p])
            longest = max(longest, len(nodes))
            w, rec = mass[nodes], h["parts"][2, p]
            total = _sum(w)
            inv = 1.0 / total
            assert rec[0] == total
            for d in range(3):
                assert rec[1 + d] == _sum(w * v[nodes, d]) * inv
                assert rec[4 + d] == _sum(w * u[nodes, d]) * inv
            assert rec[10] == _kinetic(w, v[nodes])
        node0 += m.desc.n_nodes
    assert (longest > LONG) == (max(sizes) >= 14)
    ctx.close()
