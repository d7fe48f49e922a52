"""Elastic elements on eight lanes (a small mesh, one launch) against a thread
per element (the same mesh copied until it is a large one): the same bits at
the states where the eigensolver branches (undeformed, diagonal, repeated
eigenvalues, general, inverted) and at counts that fill no warp."""
import numpy as np
import pytest

from crushrs_b200 import scenarios as S
from crushrs_b200.engine import Context
from crushrs_b200.model import ArrayModel

pytestmark = pytest.mark.gpu


def _row(n, distort):
    """A row of n elastic cubes along x, corners moved at random."""
    g = np.stack(np.meshgrid(np.arange(n + 1) * 0.2, [0.0, 0.2], [0.0, 0.2], indexing="ij"), axis=-1).reshape(-1, 3)
    at = lambda i, j, k: (i * 2 + j) * 2 + k  # noqa: E731
    hexes = np.array([[at(i, 0, 0), at(i + 1, 0, 0), at(i + 1, 1, 0), at(i, 1, 0),
                       at(i, 0, 1), at(i + 1, 0, 1), at(i + 1, 1, 1), at(i, 1, 1)] for i in range(n)], dtype=np.uint32)
    g = g + np.random.default_rng(n).uniform(-distort, distort, size=g.shape)
    return ArrayModel(g, hexes, np.zeros(n, np.int32), [S.elastic(2e8, 0.3, 1000.0)])


def _states(model):
    x = model.positions
    rng = np.random.default_rng(1)
    yield np.zeros_like(x)
    yield x * [0.1, 0.0, 0.0]                                   # diagonal
    yield x * [-0.2, 0.05, 0.05]                                # two equal eigenvalues
    yield x @ np.array([[0.0, 0.3, 0.0], [0.0, 0.0, 0.1], [0.0, 0.0, 0.0]])  # shear
    yield rng.normal(scale=0.02, size=x.shape)
    yield x * [-1.5, 0.0, 0.0]                                  # inverted: every element erodes


@pytest.mark.parametrize("n, distort", [(1, 0.0), (3, 0.02), (5, 0.0), (13, 0.02)])
def test_same_forces(n, distort):
    model = _row(n, distort)
    copies = 2400 // n + 1
    small, large = Context(model.desc), Context([model.desc] * copies)
    for u in _states(model):
        u = u.reshape(-1)
        a, b = np.zeros(3 * model.n_nodes), np.zeros(3 * model.n_nodes * copies)
        na, nb = small.compute_forces(u, a), large.compute_forces(np.tile(u, copies), b)
        assert nb == na * copies
        assert np.array_equal(b.reshape(copies, -1), np.broadcast_to(a, (copies, len(a))))
        assert np.all(np.isfinite(a))
    assert na == n  # the last state eroded them all
    small.close()
    large.close()
