"""The element kernel's shape table: forces equal to the f32 lane restatement
bit for bit whether an element's gradients and base vectors come from a table
entry it shares, from one of its own, or from its planes (more shapes than the
table has entries)."""
import numpy as np
import pytest

from crushrs_b200 import scenarios as S
from crushrs_b200.engine import Context
from crushrs_b200.model import ArrayModel
from tests import oracle_lib as O

pytestmark = pytest.mark.gpu


def _grid(nx, ny, nz, h):
    """Positions and C3D8 connectivity of a block of cubes."""
    g = np.stack(np.meshgrid(np.arange(nx + 1), np.arange(ny + 1), np.arange(nz + 1), indexing="ij"), axis=-1).reshape(-1, 3) * h
    idx = lambda i, j, k: (i * (ny + 1) + j) * (nz + 1) + k  # noqa: E731
    hexes = [[idx(i, j, k), idx(i + 1, j, k), idx(i + 1, j + 1, k), idx(i, j + 1, k),
              idx(i, j, k + 1), idx(i + 1, j, k + 1), idx(i + 1, j + 1, k + 1), idx(i, j + 1, k + 1)]
             for i in range(nx) for j in range(ny) for k in range(nz)]
    return g.astype(np.float64), np.array(hexes, dtype=np.uint32)


def _model(nx, distorted, seed):
    """A block whose first `distorted` layers of nodes along x are moved at random."""
    x, hexes = _grid(nx, 8, 16, 0.1)
    rng = np.random.default_rng(seed)
    move = x[:, 0] < (distorted - 0.5) * 0.1
    x[move] += rng.uniform(-0.01, 0.01, size=(int(move.sum()), 3))
    mat = S.honeycomb(5e6, 120.0, 0.3e6, 0.2e6, densification=(0.8, 5e6))
    return ArrayModel(x, hexes, np.zeros(len(hexes), np.int32), [mat])


# boxes only; one layer of single shapes; 1408 shapes of 1536 elements (more than the table's 1024 entries)
@pytest.mark.parametrize("nx, distorted", [(1, 0), (3, 1), (12, 11)])
def test_forces_equal_lane_kernel(nx, distorted):
    model = _model(nx, distorted, 3)
    ctx, sess = Context(model.desc), O.Session(model.desc, simd=True)
    sess.set_lane_geometry(*ctx.element_data())
    rng = np.random.default_rng(4)
    for k in range(3):
        u = rng.normal(scale=0.004 * (k + 1), size=3 * model.n_nodes)
        fd, fo = np.zeros(3 * model.n_nodes), np.zeros(3 * model.n_nodes)
        nd = ctx.compute_forces(u, fd)
        _, no = sess.forces(u, fo)
        assert nd == no
        assert np.array_equal(fd, fo)
    ctx.close()


def test_batch_equals_alone_with_a_full_table():
    models = [_model(12, 11, 5), _model(3, 1, 6), _model(2, 0, 7)]
    ctx = Context([m.desc for m in models])
    n = sum(m.n_nodes for m in models)
    u = np.random.default_rng(8).normal(scale=0.004, size=3 * n)
    f = np.zeros(3 * n)
    ctx.compute_forces(u, f)
    at = 0
    for m in models:
        alone, one = Context(m.desc), np.zeros(3 * m.n_nodes)
        alone.compute_forces(u[at:at + 3 * m.n_nodes], one)
        assert np.array_equal(f[at:at + 3 * m.n_nodes], one)
        at += 3 * m.n_nodes
        alone.close()
    ctx.close()
