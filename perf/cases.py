"""Performance cases of the crash engine: the calls its users make, over the
sizes they make them at.

Two kinds of user: a solver that keeps its own time loop and calls the
hot-path functions one at a time (element forces, one contact's penalty
forces, the stable step and the mass scaling), and programs that hand whole
crashes over (one crash, a batch, a calibration's round of barrier probes, a
stream of delta-v queries to the server). Every case builds its models with the
package's scenario builders from a seed and goes through the package's public
classes and functions.

Sizes: 300-20,000 hexahedra for a delta-v query, 300-6,000 for a crash of a
batch, 866-2,208 for the two-part vehicles of the calibrations, 278,640 for the
refined head-on.
"""
import math

import numpy as np
import torch

from crushrs_b200 import calibrate as K
from crushrs_b200 import scenarios as S
from crushrs_b200.engine import Context, contact_apply_static, solve_batch
from crushrs_b200.serve import Server

E_BLOCK = 5e6  # Pa, the synthetic blocks' modulus


def listed():
    return [
        # One element-force evaluation of the 1290-hexahedron head-on, device
        # buffers in and out: the smallest call of a solver that keeps its own
        # time loop on the GPU, where launches and latency count.
        {"name": "forces 1290", "call": "forces", "layout": "head-on", "elements": 1290, "size": 0.3},
        # The same call on the refined mesh (two blocks, 0.05 m, an 8-knot
        # yield curve): bound by memory traffic.
        {"name": "forces 278640", "call": "forces", "layout": "head-on", "elements": 278640, "size": 0.05},
        # One contact of a T-bone query through the call that allocates
        # nothing, device arrays: a solver with its own memory pool.
        {"name": "contact 6000", "call": "contact", "layout": "t-bone", "elements": 6000, "size": 0.15},
        # One stable-step check, one step's contacts and its element forces
        # through host arrays: a CPU solver that offloads its hot path.
        {"name": "drop-in 6000", "call": "drop-in", "layout": "head-on", "elements": 6000, "size": 0.15},
        # A whole small crash from the model to delta-v, final u and v: the
        # interactive use (about 650 steps).
        {"name": "run 1290", "call": "run", "layout": "head-on", "elements": 1290, "size": 0.3, "end_time": 0.1275, "max_steps": 0},
        # The largest delta-v query alone, a T-bone with an odd element size.
        {"name": "run 20000", "call": "run", "layout": "t-bone", "elements": 20000, "size": 0.1375, "end_time": 0.12, "max_steps": 0},
        # The refined head-on from the model through its first 1500 steps
        # (contact, crushing and the first eroded elements).
        {"name": "run 278640", "call": "run", "layout": "head-on", "elements": 278640, "size": 0.05, "end_time": 1.0, "max_steps": 1500},
        # A pulse-fitted two-part pair (crush zones, bumpers, elastic bodies,
        # rail boxes) head-on: elastic and honeycomb elements together, some
        # 4000 short steps; the first 50 of its 150 ms.
        {"name": "two-part 2208", "call": "two-part", "end_time": 0.05},
        # One round of the pulse calibration: 18 barrier probes of a table
        # vehicle as one batch, the accelerometer recorded at every step, the
        # CFC 60 pulses filtered on the host; the first 40 of 150 ms.
        {"name": "barrier probes 18", "call": "barrier", "probes": 18, "end_time": 0.04},
        # A parameter study in one call: seeded uneven crashes, set-up
        # pipelined with the run.
        {"name": "solve 512", "call": "solve", "crashes": 512, "lo": 300, "hi": 6000, "end_time": 0.12},
        # A small study in a context of its own.
        {"name": "batch 24", "call": "batch", "crashes": 24, "lo": 300, "hi": 6000, "end_time": 0.12},
        # A burst of mixed queries (head-on, T-bone, rear-end) to a running
        # server, until the last result.
        {"name": "serve 16", "call": "serve", "crashes": 16, "lo": 300, "hi": 20000, "end_time": 0.12},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    call = rng.choice(["forces", "forces", "contact", "drop-in", "run", "run", "refined", "two-part", "barrier", "solve", "batch", "serve"])
    layout = rng.choice(["head-on", "t-bone", "rear-end"])
    size = round(rng.uniform(0.1, 0.3), 4)
    if call == "forces":
        return {"call": call, "layout": layout, "elements": int(_log(rng, 300, 278640)), "size": size}
    if call in ("contact", "drop-in"):
        return {"call": call, "layout": layout, "elements": int(_log(rng, 300, 20000)), "size": size}
    if call == "run":
        return {"call": call, "layout": layout, "elements": int(_log(rng, 300, 20000)), "size": size,
                "end_time": round(rng.uniform(0.06, 0.12), 4), "max_steps": 0}
    if call == "refined":
        return {"call": "run", "layout": "head-on", "elements": int(_log(rng, 40000, 278640)), "size": round(rng.uniform(0.05, 0.08), 4),
                "end_time": 1.0, "max_steps": int(rng.uniform(300, 1400))}
    if call == "two-part":
        return {"call": call, "end_time": round(rng.uniform(0.015, 0.05), 4)}
    if call == "barrier":
        return {"call": call, "probes": rng.randint(4, 18), "end_time": round(rng.uniform(0.02, 0.04), 4)}
    if call == "solve":
        return {"call": call, "crashes": int(_log(rng, 40, 480)), "lo": 300, "hi": 6000, "end_time": round(rng.uniform(0.06, 0.12), 4)}
    if call == "batch":
        return {"call": call, "crashes": int(_log(rng, 2, 64)), "lo": 300, "hi": rng.choice([2000, 6000]),
                "end_time": round(rng.uniform(0.06, 0.12), 4)}
    return {"call": call, "crashes": int(_log(rng, 2, 16)), "lo": 300, "hi": rng.choice([6000, 20000]),
            "end_time": round(rng.uniform(0.06, 0.12), 4)}


# ---------------- models ----------------

def _block(elements, size, length=1.0):
    """A car-like block of about `elements` cubes: length 3.8 and width 1.2 times the height."""
    nz = max(2, round((elements / (3.8 * 1.2 * length)) ** (1.0 / 3.0)))
    ny = max(2, round(1.2 * nz))
    nx = max(2, round(elements / (ny * nz)))
    return nx * size, ny * size, nz * size


def _scenario(layout, elements, size, end_time, rng, max_steps=0):
    """Two blocks of `elements` hexahedra together; masses, yield stresses and
    speeds from `rng`, the offset from the size (the road's mesh follows it),
    within the ranges of the delta-v queries."""
    place = np.random.default_rng([elements, int(1e4 * size)])
    if elements == 278640:  # the refined head-on's blocks
        sa, sb = (138 * size, 36 * size, 30 * size), (150 * size, 36 * size, 24 * size)
        ma, mb = 2622.0, 1354.0
    elif elements == 1290:  # the plain head-on's blocks
        sa, sb = (23 * size, 6 * size, 5 * size), (25 * size, 6 * size, 4 * size)
        ma, mb = 2622.0, 1354.0
    else:
        sa, sb = _block(elements / 2, size, 0.9), _block(elements / 2, size, 1.1)
        ma, mb = rng.uniform(1400, 2600), rng.uniform(1400, 2600)
    curve = None
    if elements >= 40000:  # a tabulated curve with the lock-up knot's place taken by the eighth knot
        curve = [(k * 0.8 / 7.0, 0.3e6 + k * (0.9e6 / 7.0)) for k in range(8)]

    def material(mass, dims, sigma_y):
        rho = mass / (dims[0] * dims[1] * dims[2])
        if curve is not None:
            return S.honeycomb(E_BLOCK, rho, 0.3e6, 0.2e6, curve=curve)
        return S.honeycomb(E_BLOCK, rho, sigma_y, 0.2e6, densification=(0.8, E_BLOCK))

    a = S.vehicle(ma, sa, material(ma, sa, rng.uniform(0.3e6, 0.6e6)))
    mat_b = material(mb, sb, rng.uniform(0.2e6, 0.5e6))
    settings = {"max_steps": max_steps}
    if layout == "t-bone":  # B turned 90 degrees, its side facing A's front
        b = S.vehicle(mb, (sb[1], sb[0], sb[2]), mat_b)
        return S.scenario(a, b, rng.uniform(8, 20), 0.0, offset=place.uniform(0.0, 0.3) * sb[0], element_size=size,
                          layout=S.abi.LAYOUT_TBONE, end_time=end_time, **settings)
    b = S.vehicle(mb, sb, mat_b)
    if layout == "rear-end":
        va = rng.uniform(12, 25)
        return S.scenario(a, b, va, -va * rng.uniform(0.1, 0.6), offset=place.uniform(0.0, 0.5), element_size=size, end_time=end_time, **settings)
    return S.scenario(a, b, rng.uniform(10, 16), rng.uniform(10, 16), offset=place.uniform(0.0, 0.6), element_size=size, end_time=end_time,
                      **settings)


def _one(case, seed):
    rng = np.random.default_rng([seed, 1])
    return S.Model.build(_scenario(case["layout"], case["elements"], case["size"], case.get("end_time", 0.12), rng, case.get("max_steps", 0)))


def _many(case, seed):
    rng = np.random.default_rng([seed, 2])
    # the crashes' sizes do not depend on the seed, so that its passes cost the same
    sizes = np.random.default_rng([case["crashes"], case["lo"], case["hi"]])
    out = []
    for _ in range(case["crashes"]):
        n = int(math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"]))))
        size = float(sizes.choice([0.15, 0.1875, 0.2, 0.25, 0.3]))
        layout = ("head-on", "t-bone", "rear-end")[int(sizes.integers(3))] if case["call"] != "solve" else "head-on"
        out.append(S.Model.build(_scenario(layout, n, size, case["end_time"], rng)))
    return out


def _displacement(model, seed, size):
    """A crushed configuration: both blocks moved towards each other behind
    noses that overlap by a few centimetres and sink a little, with a few per
    cent of an element of node-to-node noise near the front."""
    rng = np.random.default_rng([seed, 3])
    x = model.positions()
    amp, nose = float(rng.uniform(0.15, 0.25)), float(rng.uniform(0.015, 0.03))
    near = np.exp(-np.abs(x[:, 0]) / 0.6)
    u = np.zeros_like(x)
    u[:, 0] = -np.sign(x[:, 0]) * (amp * (1.0 - near) + nose)
    u[:, 2] = -0.05 * near
    u += rng.normal(scale=0.03 * size, size=u.shape) * near[:, None]
    u[model.fixed_nodes()] = 0.0
    return np.ascontiguousarray(u.reshape(-1))


def _two_part(case, seed):
    rng = np.random.default_rng([seed, 4])
    va, vb = (S.MPH * float(x) for x in rng.uniform(28.0, 32.0, 2))
    return K.HeadOn(va, vb, end_time=case["end_time"]).build(S.lincoln_navigator_1999(), S.neon_1996_pulse())


def _probes(case, seed):
    """The up-and-down probes of a pattern search around the pulse-fitted Neon."""
    rng = np.random.default_rng([seed, 5])
    out = []
    for k in range(case["probes"]):
        v = S.neon_1996_pulse(table=True)
        f = math.exp((0.3 if k % 2 == 0 else -0.3) * float(rng.uniform(0.8, 1.0)))
        param = (k // 2) % 9
        if param < 7:
            t = [list(q) for q in v.table]
            t[param][1] *= f
            for i in range(2, len(t)):
                t[i][1] = max(t[i][1], t[i - 1][1])
            v.table = [tuple(q) for q in t]
        elif param == 7:
            v.modulus *= f
        else:
            v.body_modulus *= f
        out.append(v.spec())
    return out


def _device(a, dtype):
    return torch.from_numpy(np.ascontiguousarray(a)).to(device="cuda", dtype=dtype)


def prepare(case, seed):
    call = case["call"]
    if call in ("forces", "contact", "drop-in"):
        model = _one(case, seed)
        u = _displacement(model, seed, case["size"])
        if call == "forces":
            state = {"call": call, "model": model, "ctx": Context(model.desc), "u": _device(u, torch.float64),
                     "f": torch.zeros(3 * model.n_nodes, dtype=torch.float64, device="cuda")}
            torch.cuda.synchronize()
            return state
        ctx = Context(model.desc)
        masses, _ = ctx.masses()
        if call == "drop-in":
            return {"call": call, "model": model, "ctx": ctx, "u": u, "masses": masses}
        ctx.close()
        c = _front_contact(model)
        nodes, faces, scale, stiffness, max_distance = model.contact(c)
        state = {"call": call, "model": model, "stiffness": stiffness, "max_distance": max_distance,
                 "pos": _device(model.positions().reshape(-1), torch.float64), "u": _device(u, torch.float64),
                 "masses": _device(masses, torch.float64), "nodes": _device(nodes.view(np.int32), torch.int32),
                 "faces": _device(faces.reshape(-1).view(np.int32), torch.int32),
                 "scale": None if scale is None else _device(scale, torch.float64),
                 "f": torch.zeros(3 * model.n_nodes, dtype=torch.float64, device="cuda"),
                 "stats": torch.zeros(3, dtype=torch.int64, device="cuda")}
        torch.cuda.synchronize()
        return state
    if call == "run":
        return {"call": call, "model": _one(case, seed)}
    if call == "two-part":
        return {"call": call, "model": _two_part(case, seed)}
    if call == "barrier":
        rng = np.random.default_rng([seed, 6])
        return {"call": call, "vehicles": _probes(case, seed), "speed": S.MPH * float(rng.uniform(34.0, 36.0)), "end_time": case["end_time"]}
    models = _many(case, seed)
    if call == "serve":
        return {"call": call, "models": models, "server": Server()}
    return {"call": call, "models": models}


CONTACT_DT = 5e-5  # s, the step the drop-in calls limit the contact stiffness with


def _front_contact(model):
    """The vehicle-to-vehicle contact with the most nodes x faces (the road's faces are fixed nodes)."""
    fixed = np.zeros(model.n_nodes, bool)
    fixed[model.fixed_nodes()] = True
    best, most = 0, -1
    for c in range(model.desc.n_contacts):
        nodes, faces, _, _, _ = model.contact(c)
        if not fixed[faces].all() and len(nodes) * len(faces) > most:
            best, most = c, len(nodes) * len(faces)
    return best


def _results(rs):
    """The results of crashes as arrays."""
    out = {"time": [], "steps": [], "eroded": [], "dt_min": [], "added_mass_max": [], "status": []}
    veh = {"mass": [], "delta_v": [], "velocity": [], "crush": []}
    for r in rs:
        out["time"].append(r.time)
        out["steps"].append(r.steps)
        out["eroded"].append(r.eroded_elements)
        out["dt_min"].append(r.dt_min)
        out["added_mass_max"].append(r.added_mass_max)
        out["status"].append(r.status)
        for k in range(r.n_vehicles):
            v = r.vehicle[k]
            veh["mass"].append(v.mass)
            veh["delta_v"].append(list(v.delta_v))
            veh["velocity"].append(list(v.velocity))
            veh["crush"].append(v.crush)
    out.update(veh)
    return {k: np.array(v) for k, v in out.items()}


def run(state):
    call = state["call"]
    if call == "forces":
        state["ctx"].compute_forces_device(state["u"].data_ptr(), state["f"].data_ptr())
        return state["f"]
    if call == "contact":
        state["f"].zero_()
        scale = state["scale"]
        contact_apply_static(state["model"].n_nodes, state["pos"].data_ptr(), state["u"].data_ptr(), state["masses"].data_ptr(),
                             (state["nodes"].data_ptr(), state["nodes"].numel()), None if scale is None else scale.data_ptr(),
                             (state["faces"].data_ptr(), state["faces"].numel() // 4), state["stiffness"], state["max_distance"], CONTACT_DT,
                             state["f"].data_ptr(), state["stats"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"f": state["f"], "count": state["stats"][0], "max": state["stats"][1:2].view(torch.float64)}
    if call == "drop-in":
        ctx, model, u = state["ctx"], state["model"], state["u"]
        dt = ctx.stable_time_step(u)
        total, added = ctx.mass_scaling(u, 1.05 * dt)
        f_ext, f_int = np.zeros(3 * model.n_nodes), np.zeros(3 * model.n_nodes)
        hits, deepest = 0, 0.0
        for c in range(model.desc.n_contacts):
            n, d = ctx.contact_apply(c, u, None, state["masses"], CONTACT_DT, f_ext)
            hits, deepest = hits + n, max(deepest, d)
        eroded = ctx.compute_forces(u, f_int)
        return {"dt": dt, "total": total, "added": added, "f_ext": f_ext, "f_int": f_int, "hits": hits, "deepest": deepest, "eroded": eroded}
    if call in ("run", "two-part"):
        ctx = Context(state["model"].desc)
        r = ctx.run()
        u, v = ctx.state()
        ctx.close()
        return {**_results([r]), "u": u, "v": v}
    if call == "barrier":
        pulses = K.run_barrier_pulses(state["vehicles"], state["speed"], end_time=state["end_time"])
        return [p.accel for p in pulses]
    if call == "solve":
        return _results(solve_batch([m.desc for m in state["models"]]))
    if call == "batch":
        ctx = Context([m.desc for m in state["models"]])
        rs = ctx.batch_run()
        u, v = ctx.state()
        ctx.close()
        return {**_results(rs), "u": u, "v": v}
    server, got = state["server"], {}
    tickets = [server.submit(m.desc) for m in state["models"]]
    while len(got) < len(tickets):
        for r in server.poll(wait_ms=100):
            got[r.ticket] = r.results
    return _results([got[t] for t in tickets])


# ---------------- work ----------------
# Per honeycomb element and force evaluation: node ids 32 B, the material
# state (25 values and a flag) read and written 208 B, the symmetric 12 x 12
# hourglass stiffness 312 B; per node reference position and displacement in
# and the force out, 72 B. A time step also updates u and v and reads the mass:
# 56 B more per node. About 1500 operations per element (the deformation
# gradient, the rate-form update, the hourglass product), 20 per node.
# A run's steps are counted at the initial stable step of its mesh
# (0.85 size sqrt(density / modulus)), which crushing only shortens.
ELEM_BYTES, NODE_BYTES, STEP_NODE_BYTES = 552.0, 72.0, 56.0
ELEM_FLOPS, NODE_FLOPS = 1500.0, 20.0


def _steps(end_time, size, rho, max_steps=0):
    n = max(1.0, end_time / (0.85 * size * math.sqrt(rho / E_BLOCK)))
    return min(n, max_steps) if max_steps else n


def _step_work(elements, nodes, steps):
    return {"bytes": steps * (ELEM_BYTES * elements + (NODE_BYTES + STEP_NODE_BYTES) * nodes),
            "flops": steps * (ELEM_FLOPS * elements + NODE_FLOPS * nodes)}


def work(case):
    call = case["call"]
    if call == "two-part":  # 2208 hexahedra, 3330 nodes, 4251 steps to 150 ms
        return _step_work(2208, 3330, case["end_time"] / 0.15 * 4251)
    if call == "barrier":  # 866 hexahedra, 1386 nodes, about 4200 steps to 150 ms
        w = _step_work(866, 1386, case["end_time"] / 0.15 * 4200)
        return {k: case["probes"] * v for k, v in w.items()}
    if call in ("solve", "batch", "serve"):
        total = {"bytes": 0.0, "flops": 0.0}
        sizes = np.random.default_rng([case["crashes"], case["lo"], case["hi"]])
        for _ in range(case["crashes"]):
            n = int(math.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"]))))
            size = float(sizes.choice([0.15, 0.1875, 0.2, 0.25, 0.3]))
            sizes.integers(3)
            rho = 2000.0 / (0.5 * n * size ** 3)
            w = _step_work(n, 1.3 * n, _steps(case["end_time"], size, rho))
            total = {k: total[k] + w[k] for k in total}
        return total
    n, size = case["elements"], case["size"]
    nodes = 1.3 * n if n < 40000 else 1.1 * n
    if call == "forces":
        return {"bytes": ELEM_BYTES * n + NODE_BYTES * nodes, "flops": ELEM_FLOPS * n}
    m = _one(case, 1)
    if call == "contact":
        nodes, faces, _, _, _ = m.contact(_front_contact(m))
        pairs = len(nodes) * len(faces)
        # node and face ids, the positions and displacements of both sides' nodes, masses and scales, and the forces
        return {"bytes": 16.0 * len(faces) + 76.0 * len(nodes) + 48.0 * len(faces) + 24.0 * m.n_nodes, "flops": 6.0 * pairs}
    if call == "drop-in":
        pairs = sum(len(m.contact(c)[0]) * len(m.contact(c)[1]) for c in range(m.desc.n_contacts))
        per = 48.0 * m.n_nodes  # u in, forces (or the added masses and the contact masses) out
        return {"bytes": ELEM_BYTES * n + 32.0 * n + per * (m.desc.n_contacts + 3), "flops": (ELEM_FLOPS + 500.0) * n + 6.0 * pairs}
    rho = 2000.0 / (0.5 * n * size ** 3)
    return _step_work(m.n_hexes, m.n_nodes, _steps(case["end_time"], size, rho, case["max_steps"]))


# ---------------- the calls in 64 bits ----------------

_XI = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], dtype=np.float64)
_MODES = np.array([[1, 1, -1, -1, -1, -1, 1, 1], [1, -1, -1, 1, -1, 1, 1, -1], [1, -1, 1, -1, 1, -1, 1, -1],
                   [-1, 1, -1, 1, 1, -1, 1, -1]], dtype=np.float64)


def _dn(xi):
    """Shape-function derivatives (8, 3) of the 8-node hexahedron at a local point."""
    s = 1.0 + _XI * xi
    return 0.125 * _XI * np.stack([s[:, 1] * s[:, 2], s[:, 0] * s[:, 2], s[:, 0] * s[:, 1]], axis=1)


def _gradients(x, dn):
    """Reference gradients (E, 8, 3) and det J (E) for node positions x (E, 8, 3)."""
    j = dn.T @ x
    return dn @ np.linalg.inv(j).transpose(0, 2, 1), np.linalg.det(j)


def _honeycomb_forces(x, u, youngs, hourglass, sy, hard, trans):
    """Corner forces (E, 8, 3) of one-point honeycomb hexahedra deformed in
    one increment from the initial state: the rate-form law (midpoint
    deformation rate, Cayley rotation), its per-axis yield caps and the exact
    rank-12 hourglass stiffness."""
    grad, _ = _gradients(x, _dn(np.zeros(3)))
    gam = _MODES.T[None] - np.einsum("eic,eac->eia", grad, np.einsum("aj,ejc->eac", _MODES, x))
    n = len(x)
    gkg, volume = np.zeros((n, 12, 12)), np.zeros(n)
    mu = 0.5 * hourglass * youngs  # Poisson's ratio 0
    weight = np.array([2.0, 2.0, 2.0, 1.0, 1.0, 1.0])
    for p in _XI / math.sqrt(3.0):
        gq, detj = _gradients(x, _dn(p))
        pm = gam.transpose(0, 2, 1) @ (gq - grad)
        m = np.zeros((n, 6, 4, 3))  # strain rows xx yy zz xy yz xz
        for d in range(3):
            m[:, d, :, d] = pm[:, :, d]
        for row, (a, b) in ((3, (0, 1)), (4, (1, 2)), (5, (0, 2))):
            m[:, row, :, a] = pm[:, :, b]
            m[:, row, :, b] = pm[:, :, a]
        m = m.reshape(n, 6, 12)
        gkg += (m * (mu * detj)[:, None, None] * weight[:, None]).transpose(0, 2, 1) @ m
        volume += detj
    ainv = np.linalg.inv(gam.transpose(0, 2, 1) @ gam)
    h = (ainv @ gkg.reshape(n, 4, 36)).reshape(n, 4, 3, 4, 3).transpose(0, 3, 4, 1, 2)  # (b, f, a, d): the columns on the left for the other factor
    h = (ainv @ h.reshape(n, 4, 36)).reshape(n, 12, 12).transpose(0, 2, 1)

    eye = np.eye(3)
    f = (x + u).transpose(0, 2, 1) @ grad
    det = np.linalg.det(f)
    g = (f - eye) @ np.linalg.inv(0.5 * (f + eye))
    d, w = 0.5 * (g + g.transpose(0, 2, 1)), 0.5 * (g - g.transpose(0, 2, 1))
    om = w[:, 0, 1] ** 2 + w[:, 0, 2] ** 2 + w[:, 1, 2] ** 2
    r = eye + (w + 0.5 * w @ w) / (1.0 + 0.25 * om)[:, None, None]
    s = youngs[:, None, None] * (r.transpose(0, 2, 1) @ d @ r)
    dc = np.zeros(n)
    cap = np.stack([np.ones(n), trans, trans], axis=1)
    diag = np.stack([s[:, k, k] for k in range(3)], axis=1)
    for _ in range(3):
        over = -diag > cap * (sy + hard * dc)[:, None]
        total = np.where(over, -diag - cap * sy[:, None], 0.0).sum(axis=1)
        active = np.where(over, cap, 0.0).sum(axis=1)
        dc = np.where(active > 0.0, total / (youngs + active * hard), 0.0)
    sig = np.maximum(sy + hard * dc, 0.0)
    for k in range(3):
        s[:, k, k] = np.clip(diag[:, k], -cap[:, k] * sig, cap[:, k] * sig)
        for q in range(3):
            if q != k:
                s[:, k, q] = np.clip(s[:, k, q], -0.5 * sig, 0.5 * sig)
    tau = det[:, None, None] * (r @ s @ r.transpose(0, 2, 1))
    out = grad @ (tau @ np.linalg.inv(f).transpose(0, 2, 1)).transpose(0, 2, 1) * volume[:, None, None]
    q = (gam.transpose(0, 2, 1) @ u).reshape(n, 12, 1)
    out += gam @ (h @ q).reshape(n, 4, 3)
    out[det <= 0.0] = 0.0
    return out


def _exact_forces(model, u):
    """Nodal element forces; the road's elements carry none (their nodes do not move)."""
    x, hexes, part = model.positions(), model.hexes(), model.hex_part()
    u = u.reshape(-1, 3)
    f = np.zeros_like(x)
    for p in range(model.desc.n_parts):
        mat = model.material(p)
        if mat.model != S.abi.MAT_HONEYCOMB:
            continue
        sel = np.nonzero(part == p)[0]
        sy = mat.curve[0][1] if mat.n_curve else mat.yield_stress
        hard = (mat.curve[1][1] - mat.curve[0][1]) / (mat.curve[1][0] - mat.curve[0][0]) if mat.n_curve else mat.hardening
        for k in range(0, len(sel), 20000):
            hx = hexes[sel[k:k + 20000]]
            full = lambda v: np.full(len(hx), float(v))  # noqa: E731
            c = _honeycomb_forces(x[hx], u[hx], full(mat.youngs_modulus), model.settings.hourglass, full(sy), full(hard),
                                  full(mat.transverse_factor))
            for i in range(8):
                for d in range(3):
                    f[:, d] += np.bincount(hx[:, i], weights=c[:, i, d], minlength=len(f))
    return f.reshape(-1)


def _in_triangle(p, a, b, c):
    v0, v1, v2 = c - a, b - a, p - a
    dot = lambda s, t: (s * t).sum(axis=-1)  # noqa: E731
    d00, d01, d02, d11, d12 = dot(v0, v0), dot(v0, v1), dot(v0, v2), dot(v1, v1), dot(v1, v2)
    with np.errstate(divide="ignore", invalid="ignore"):
        inv = 1.0 / (d00 * d11 - d01 * d01)
        s, t = (d11 * d02 - d01 * d12) * inv, (d00 * d12 - d01 * d02) * inv
        return (s >= -0.1) & (t >= -0.1) & (s + t <= 1.1)


def _exact_contact(model, c, u, masses, f):
    """One contact's penalty forces added into f (N, 3): every node takes the
    first face that it lies behind; hits and the deepest one returned."""
    nodes, faces, scale, stiffness, md = model.contact(c)
    x0 = model.positions()
    lo, hi = x0[faces].min(axis=(0, 1)) - md, x0[faces].max(axis=(0, 1)) + md
    near = ((x0[nodes] >= lo) & (x0[nodes] <= hi)).all(axis=1)
    scale = np.ones(len(nodes)) if scale is None else np.asarray(scale)
    nodes, scale = nodes[near].astype(np.int64), scale[near]
    x = x0 + u.reshape(-1, 3)
    q = x[faces]
    nrm = np.cross(q[:, 1] - q[:, 0], q[:, 2] - q[:, 0])
    nrm /= np.linalg.norm(nrm, axis=1)[:, None]
    cen = q.mean(axis=1)
    blo, bhi = q.min(axis=1) - md, q.max(axis=1) + md
    hits, deepest = 0, 0.0
    for n, sc in zip(nodes, scale):
        p = x[n]
        sd = -((cen - p) * nrm).sum(axis=1)
        ok = (p >= blo).all(axis=1) & (p <= bhi).all(axis=1) & (sd <= 0.0) & (sd >= -md)
        k = np.nonzero(ok)[0]
        if not len(k):
            continue
        proj, t = p - nrm[k] * sd[k, None], q[k]
        inside = (_in_triangle(proj, t[:, 0], t[:, 1], t[:, 2]) | _in_triangle(proj, t[:, 0], t[:, 2], t[:, 3])
                  | _in_triangle(proj, t[:, 1], t[:, 2], t[:, 3]) | _in_triangle(proj, t[:, 1], t[:, 3], t[:, 0]))
        k = k[inside]
        if not len(k):
            continue
        k = k[0]
        m = masses[n]
        mag = min(min(stiffness * sc, 0.1 * m / CONTACT_DT ** 2) * min(-sd[k], 0.1 * md), m * 1e5)
        f[n] += mag * nrm[k]
        for j in range(4):
            f[faces[k, j]] -= 0.25 * mag * nrm[k]
        hits, deepest = hits + 1, max(deepest, -sd[k])
    return hits, deepest


_TETS = [(0, 1, 2, 6), (0, 2, 3, 6), (0, 3, 7, 6), (0, 7, 4, 6), (0, 4, 5, 6), (0, 5, 1, 6)]
_FACES = [(0, 1, 2, 3), (4, 5, 6, 7), (0, 1, 5, 4), (1, 2, 6, 5), (2, 3, 7, 6), (3, 0, 4, 7)]


def _exact_limits(model, u):
    """Every element's stable step (volume over its largest face, over the
    wave speed) and mass."""
    hexes, part = model.hexes(), model.hex_part()
    rest = model.positions()[hexes]
    p = rest + u.reshape(-1, 3)[hexes]

    def volume(q):
        return sum((np.cross(q[:, b] - q[:, a], q[:, c] - q[:, a]) * (q[:, d] - q[:, a])).sum(axis=1) / 6.0 for a, b, c, d in _TETS)

    area = np.max([0.5 * np.linalg.norm(np.cross(p[:, c] - p[:, a], p[:, d] - p[:, b]), axis=1) for a, b, c, d in _FACES], axis=0)
    vol = volume(p)
    mats = [model.material(k) for k in range(model.desc.n_parts)]
    factor = np.array([(1.0 - 0.36 * m.poisson_ratio) / math.sqrt(m.youngs_modulus * (1.0 - m.poisson_ratio) / (
        (1.0 + m.poisson_ratio) * (1.0 - 2.0 * m.poisson_ratio)) / m.density) for m in mats])
    rho = np.array([m.density for m in mats])
    with np.errstate(divide="ignore", invalid="ignore"):
        dt = np.where((vol > 0.0) & (area > 0.0), vol / area * factor[part], np.inf)
    return dt, volume(rest) * rho[part]


def _exact_masses(model):
    """Lumped nodal masses of box-shaped elements: an eighth of the element at every corner."""
    hexes = model.hexes()
    _, em = _exact_limits(model, np.zeros(3 * model.n_nodes))
    return np.bincount(hexes.reshape(-1), weights=np.repeat(em / 8.0, 8), minlength=model.n_nodes)


def exact(case, seed):
    call = case["call"]
    if call not in ("forces", "contact", "drop-in"):
        return None  # thousands of steps: no 64-bit run within seconds
    model = _one(case, seed)
    u = _displacement(model, seed, case["size"])
    if call == "forces":
        return _exact_forces(model, u)
    masses = _exact_masses(model)
    f = np.zeros((model.n_nodes, 3))
    if call == "contact":
        hits, deepest = _exact_contact(model, _front_contact(model), u, masses, f)
        return {"f": f.reshape(-1), "count": hits, "max": np.array([deepest])}
    hits, deepest = 0, 0.0
    for c in range(model.desc.n_contacts):
        n, d = _exact_contact(model, c, u, masses, f)
        hits, deepest = hits + n, max(deepest, d)
    dt, em = _exact_limits(model, u)
    step = float(dt.min())
    with np.errstate(divide="ignore"):
        extra = np.where(dt < 1.05 * step, (np.minimum((1.05 * step / dt) ** 2, 100.0) - 1.0) * em, 0.0)
    added = np.bincount(model.hexes().reshape(-1), weights=np.repeat(extra / 8.0, 8), minlength=model.n_nodes)
    return {"dt": step, "total": float(extra.sum()), "added": added, "f_ext": f.reshape(-1), "f_int": _exact_forces(model, u),
            "hits": hits, "deepest": deepest, "eroded": 0}
