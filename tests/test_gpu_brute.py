"""The exhaustive search at the edges of its lanes' masks (255 faces is the
most it takes) and of its lane choice (few contacts 16 lanes, many 4): forces
against the oracle, and a batch of 80 such contacts under the step graphs
against the same crash alone."""
import numpy as np
import pytest

from crushrs_b200 import abi, scenarios as S
from crushrs_b200.engine import Context
from crushrs_b200.model import ArrayModel
from tests import oracle_lib as O

pytestmark = pytest.mark.gpu


def _plates(n, m, speed):
    """Two layers of n x m elements, the upper one falling on the lower; contacts both ways."""
    def grid(z0):
        g = np.stack(np.meshgrid(np.arange(n + 1) * 0.1, np.arange(m + 1) * 0.1, [z0, z0 + 0.1], indexing="ij"), axis=-1).reshape(-1, 3)
        at = lambda i, j, k: (i * (m + 1) + j) * 2 + k  # noqa: E731
        return g, np.array([[at(i, j, 0), at(i + 1, j, 0), at(i + 1, j + 1, 0), at(i, j + 1, 0),
                             at(i, j, 1), at(i + 1, j, 1), at(i + 1, j + 1, 1), at(i, j + 1, 1)] for i in range(n) for j in range(m)], np.uint32)

    (xa, ha), (xb, hb) = grid(0.0), grid(0.1005)
    x = np.concatenate([xa, xb + [0.013, 0.027, 0.0]])
    hb = hb + len(xa)
    v = np.zeros_like(x)
    v[len(xa):, 2] = -speed
    mat = S.honeycomb(5e6, 100.0, 0.3e6, 0.2e6, densification=(0.8, 5e6))
    down = {"nodes": np.unique(hb[:, :4]), "faces": ha[:, 4:], "stiffness": 2e5, "max_distance": 0.05}
    up = {"nodes": np.unique(ha[:, 4:]), "faces": hb[:, [3, 2, 1, 0]], "stiffness": 2e5, "max_distance": 0.05}
    vehicles = [{"nodes": np.arange(len(xa)), "accel": 0, "front": [0]}, {"nodes": np.arange(len(xa), len(x)), "accel": len(xa), "front": [len(xa)]}]
    settings = abi.Settings(end_time=0.02, dt_scale=0.85, time_step=0.0, adaptive_check_steps=5, hourglass=0.1, velocity_damping=1.0,
                            mass_scaling=0.25, stop_rule=0, max_steps=0)
    return ArrayModel(x, np.concatenate([ha, hb]), np.zeros(2 * n * m, np.int32), [mat], initial_velocity=v, contacts=[down, up],
                      vehicles=vehicles, settings=settings)


@pytest.mark.parametrize("n, m", [(1, 1), (2, 8), (4, 16), (5, 13), (15, 17)])  # 1, 16, 64, 65, 255 faces
def test_forces_equal_oracle(n, m):
    model = _plates(n, m, 0.0)
    ctx, sess = Context(model.desc), O.Session(model.desc, simd=True)
    masses, _ = ctx.masses()
    u = np.random.default_rng(n * m).normal(scale=0.004, size=3 * model.n_nodes)
    hits = 0
    for c in range(2):
        f, want = np.zeros(3 * model.n_nodes), np.zeros(3 * model.n_nodes)
        count, deepest = ctx.contact_apply(c, u, None, masses, 1e-4, f)
        _, n_want, d_want = sess.contact_apply(c, u, None, masses, 1e-4, want)
        assert (count, deepest) == (n_want, d_want)
        assert np.array_equal(f, want)
        hits += count
    assert hits > 0
    ctx.close()


def test_many_contacts_equal_one():
    models = [_plates(15, 17, 3.0 + 0.05 * (k % 4)) for k in range(40)]  # 80 contacts: 4 lanes per node
    ctx = Context([m.desc for m in models])
    ctx.set_tuning(32, 2)
    ctx.run_begin()
    ctx.run_steps(120)
    u, v = (x.reshape(40, -1) for x in ctx.state())
    rs = [ctx.results(k) for k in range(40)]
    ctx.close()
    for k in range(4):
        alone = Context(models[k].desc)
        alone.run_begin()
        alone.run_steps(120)
        r = alone.results()
        ua, va = alone.state()
        alone.close()
        assert r.vehicle[0].velocity[2] < 0.0  # the upper plate pushed the lower one down
        for j in range(k, 40, 4):
            assert np.array_equal(u[j], ua) and np.array_equal(v[j], va)
            assert rs[j].steps == r.steps and list(rs[j].vehicle[1].delta_v) == list(r.vehicle[1].delta_v)
