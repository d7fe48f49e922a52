"""crush_contact_apply_static where few entries hit, anywhere among the rest
(the sums number the hits by groups of 128 entries, most of them empty),
against crush_contact_apply, bit for bit. Sorts after the other GPU tests, like
the call's other test files."""
import numpy as np
import pytest

from crushrs_b200 import abi
from crushrs_b200.engine import Context
from tests.test_zz_static_sizes import _call, _plates

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

PATTERNS = {
    "none": [],
    "first": [0],
    "last": [1680],
    "last over the plate": [1638],
    "across groups": [127, 128, 255, 256],
    "one group": list(range(384, 512)),
    "two tiles and one": list(range(640, 897)),
    "sparse": list(range(5, 1681, 131)),
    "every other": list(range(0, 1681, 2)),
    "all": list(range(1681)),
}


@pytest.mark.parametrize("pattern", PATTERNS)
def test_few_hits(pattern):
    model = _plates(40, 40)
    nodes, faces = model._contacts[0][:2]
    assert len(nodes) == 1681
    ctx = Context(model.desc)
    masses, _ = ctx.masses()
    u = np.random.default_rng(len(pattern)).normal(scale=0.0003, size=(model.n_nodes, 3))
    away = np.setdiff1d(np.arange(len(nodes)), PATTERNS[pattern])
    u[nodes[away], 2] += 0.05  # clear of the faces
    u = u.reshape(-1)
    f = torch.zeros(3 * model.n_nodes, dtype=torch.float64, device="cuda")
    st = _call(model, u, masses, nodes, faces, 1e-4, f)
    want = np.zeros(3 * model.n_nodes)
    count, deepest = ctx.contact_apply(0, u, None, masses, 1e-4, want)
    assert (st.status, st.penetration_count, st.max_penetration) == (abi.CRUSH_OK, count, deepest)
    # entry 41 i + j; the rows i = 40 and j = 40 hang over the lower plate's edge and miss
    assert count == sum(k // 41 < 40 and k % 41 < 40 for k in PATTERNS[pattern])
    assert np.array_equal(f.cpu().numpy(), want)
    ctx.close()
