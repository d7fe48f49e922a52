"""Element forces of a call over a whole large mesh, which small blocks take:
the same rows of honeycomb cubes, repeated to just below, at and just above
one wave of them, give the bits of a row alone."""
import numpy as np
import pytest

from crushrs_b200 import scenarios as S
from crushrs_b200.engine import Context
from crushrs_b200.model import ArrayModel

pytestmark = pytest.mark.gpu
WAVE = 148 * 512


@pytest.mark.parametrize("copies", [WAVE // 64 - 1, WAVE // 64, WAVE // 64 + 1])
def test_same_forces(copies):
    n = 64
    g = np.stack(np.meshgrid(np.arange(n + 1) * 0.2, [0.0, 0.2], [0.0, 0.2], indexing="ij"), axis=-1).reshape(-1, 3)
    at = lambda i, j, k: (i * 2 + j) * 2 + k  # noqa: E731
    hexes = np.array([[at(i, 0, 0), at(i + 1, 0, 0), at(i + 1, 1, 0), at(i, 1, 0),
                       at(i, 0, 1), at(i + 1, 0, 1), at(i + 1, 1, 1), at(i, 1, 1)] for i in range(n)], dtype=np.uint32)
    rng = np.random.default_rng(n)
    g = g + rng.uniform(-0.02, 0.02, size=g.shape)
    model = ArrayModel(g, hexes, np.zeros(n, np.int32), [S.honeycomb(5e6, 100.0, 3e5, 2e5, densification=(0.8, 5e6))])
    alone, many = Context(model.desc), Context([model.desc] * copies)
    for u in (rng.normal(scale=0.01, size=g.shape), g * [-0.4, 0.05, 0.0], g * [-1.5, 0.0, 0.0]):
        u = u.reshape(-1)
        a, b = np.zeros(3 * model.n_nodes), np.zeros(3 * model.n_nodes * copies)
        na, nb = alone.compute_forces(u, a), many.compute_forces(np.tile(u, copies), b)
        assert nb == na * copies
        assert np.array_equal(b.reshape(copies, -1), np.broadcast_to(a, (copies, len(a))))
    assert na == n  # the last state eroded them all
    alone.close()
    many.close()
