"""crush_contact_apply_static at the edges of its passes' sizes (a face batch,
more face blocks than a warp combines at once, entries past a tile, none at
all) against crush_contact_apply, bit for bit. Sorts after the other GPU
tests, like the call's other test file."""
import numpy as np
import pytest

from crushrs_b200 import abi, scenarios as S
from crushrs_b200.engine import Context, contact_apply_static
from crushrs_b200.model import ArrayModel

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _plates(n, m):
    """Two layers of n x m elements, the upper one's bottom nodes 5 mm inside the lower one's top faces."""
    def grid(z0):
        g = np.stack(np.meshgrid(np.arange(n + 1) * 0.1, np.arange(m + 1) * 0.1, [z0, z0 + 0.1], indexing="ij"), axis=-1).reshape(-1, 3)
        at = lambda i, j, k: (i * (m + 1) + j) * 2 + k  # noqa: E731
        h = [[at(i, j, 0), at(i + 1, j, 0), at(i + 1, j + 1, 0), at(i, j + 1, 0),
              at(i, j, 1), at(i + 1, j, 1), at(i + 1, j + 1, 1), at(i, j + 1, 1)] for i in range(n) for j in range(m)]
        return g, np.array(h, dtype=np.uint32)

    (xa, ha), (xb, hb) = grid(0.0), grid(0.095)
    x = np.concatenate([xa, xb + [0.013, 0.027, 0.0]])
    hexes = np.concatenate([ha, hb + len(xa)])
    nodes = np.unique(hb[:, :4] + len(xa))
    mat = S.honeycomb(5e6, 100.0, 0.3e6, 0.2e6)
    contact = {"nodes": nodes, "faces": ha[:, 4:], "stiffness": 1e6, "max_distance": 0.03}
    return ArrayModel(x, hexes, np.zeros(len(hexes), np.int32), [mat], contacts=[contact])


def _dev(a, dtype):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dtype=dtype, device="cuda")


def _call(model, u, masses, nodes, faces, dt, f):
    stats = torch.zeros(3, dtype=torch.int64, device="cuda")
    args = (_dev(model.positions.reshape(-1), torch.float64), _dev(u, torch.float64), _dev(masses, torch.float64),
            _dev(nodes.view(np.int32), torch.int32), _dev(faces.reshape(-1).view(np.int32), torch.int32))
    contact_apply_static(model.n_nodes, args[0].data_ptr(), args[1].data_ptr(), args[2].data_ptr(), (args[3].data_ptr(), len(nodes)),
                         None, (args[4].data_ptr(), len(faces)), 1e6, 0.03, dt, f.data_ptr(), stats.data_ptr(),
                         torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return abi.ContactStats.from_buffer_copy(stats.cpu().numpy().tobytes())


@pytest.mark.parametrize("n, m", [(1, 1), (8, 16), (3, 43), (70, 70), (128, 128)])  # 1, 128, 129, 4900, 16384 faces
def test_sizes(n, m):
    model = _plates(n, m)
    nodes, faces = model._contacts[0][0][:abi.STATIC_MAX_NODES], model._contacts[0][1]
    ctx = Context(model.desc)
    masses, _ = ctx.masses()
    u = np.random.default_rng(n + m).normal(scale=0.003, size=3 * model.n_nodes)
    f = torch.zeros(3 * model.n_nodes, dtype=torch.float64, device="cuda")
    st = _call(model, u, masses, nodes, faces, 1e-4, f)
    if len(nodes) == len(model._contacts[0][0]):
        want = np.zeros(3 * model.n_nodes)
        count, deepest = ctx.contact_apply(0, u, None, masses, 1e-4, want)
        assert (st.status, st.penetration_count, st.max_penetration) == (abi.CRUSH_OK, count, deepest) and count > 0
        assert np.array_equal(f.cpu().numpy(), want)
    else:  # the call's limit on nodes is below the plate's: the forces balance
        got = f.cpu().numpy().reshape(-1, 3)
        assert st.penetration_count > 0 and np.all(np.abs(got.sum(axis=0)) <= 1e-9 * np.abs(got).sum(axis=0))
    ctx.close()


def test_nothing_to_do():
    model = _plates(2, 2)
    nodes, faces = model._contacts[0][:2]
    masses, u = np.ones(model.n_nodes), np.zeros(3 * model.n_nodes)
    f = torch.full((3 * model.n_nodes,), 2.5, dtype=torch.float64, device="cuda")
    for a, b in ((nodes[:0], faces), (nodes, faces[:0]), (nodes[:0], faces[:0])):
        st = _call(model, u, masses, a, b, 1e-4, f)
        assert (st.status, st.penetration_count, st.max_penetration) == (abi.CRUSH_OK, 0, 0.0)
        assert bool(torch.all(f == 2.5))
