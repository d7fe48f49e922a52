"""Force calls over whole meshes that one launch of small blocks takes, and over
the same meshes copied until their elastic elements are too many for it: the
same bits, at counts that fill no block."""
import numpy as np
import pytest

from crushrs_b200 import scenarios as S
from crushrs_b200.engine import Context
from crushrs_b200.model import ArrayModel

pytestmark = pytest.mark.gpu
LINE = 2368  # elastic elements


def _row(n):
    """A row of n cubes along x, corners moved at random, elastic and honeycomb by turns."""
    g = np.stack(np.meshgrid(np.arange(n + 1) * 0.2, [0.0, 0.2], [0.0, 0.2], indexing="ij"), axis=-1).reshape(-1, 3)
    at = lambda i, j, k: (i * 2 + j) * 2 + k  # noqa: E731
    hexes = np.array([[at(i, 0, 0), at(i + 1, 0, 0), at(i + 1, 1, 0), at(i, 1, 0),
                       at(i, 0, 1), at(i + 1, 0, 1), at(i + 1, 1, 1), at(i, 1, 1)] for i in range(n)], dtype=np.uint32)
    g = g + np.random.default_rng(n).uniform(-0.02, 0.02, size=g.shape)
    mats = [S.honeycomb(5e6, 100.0, 3e5, 2e5, densification=(0.8, 5e6)), S.elastic(2e8, 0.3, 1000.0)]
    return ArrayModel(g, hexes, (np.arange(n) % 2).astype(np.int32), mats)


@pytest.mark.parametrize("n", [1, 2, 37, 101, 131])
def test_same_forces(n):
    model = _row(n)
    per = n // 2
    below = LINE // per if per else 130
    rng = np.random.default_rng(n)
    states = [rng.normal(scale=0.01, size=model.positions.shape), model.positions * [-0.4, 0.05, 0.0], model.positions * [-1.5, 0.0, 0.0]]
    alone = Context(model.desc)
    want = []
    for u in states:
        f = np.zeros(3 * model.n_nodes)
        want.append((alone.compute_forces(u.reshape(-1), f), f))
    assert want[-1][0] == n  # the last state eroded them all
    for copies in (below, below + 1):
        many = Context([model.desc] * copies)
        for u, (eroded, f) in zip(states, want):
            g = np.zeros(3 * model.n_nodes * copies)
            assert many.compute_forces(np.tile(u.reshape(-1), copies), g) == eroded * copies
            assert np.array_equal(g.reshape(copies, -1), np.broadcast_to(f, (copies, len(f))))
        many.close()
