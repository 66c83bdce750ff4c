"""The workloads that users of this framework wait for, as timed cases.

Each case is one call pattern of a program around `CudaPhysics` and
`CudaRenderer`: the control loop of a policy (on the GPU or on the host), a
rollout, a batch of objects in contact, randomisation at an episode's end, a
batch of images. `prepare` builds what such a program has in hand (the
handle, its states, controls, buffers), `run` makes one pass through the
public entry points.

States are drawn around the ones that a simulation meets, not simulated up
to: an Ant walking on the floor with joints at their limits, objects standing
on the table, hulls lying about on the floor, a few of them toppling. So a
state depends on the seed alone.
"""
from __future__ import annotations

import functools

import numpy as np
import torch

from pippin_b200 import CudaPhysics, Field, mjcf, scenes
from pippin_b200.physics import Param, Solver, WarmStart
from pippin_b200.render import CudaRenderer, RenderConfig, ViewSource

TOL, ITERS = 1e-10, 30  # the solver settings of the benchmark
N_CTRL = 8              # control sets a state cycles through, pass by pass

# FP64 operations per env and substep of the reference's algorithm (the CPU
# restatement's counters on states like these)
FLOPS = {"ant": 22e3, "cartpole": 2.6e3, "arm3hinge": 2.8e3, "arm3d": 6.2e3, "tabletop": 56e3, "hulls": 72e3}


def listed():
    return [
        # one evaluation or debugging loop on the host: a few envs, latency is all
        {"name": "ant_host_16", "kind": "step", "model": "ant", "api": "host", "n": 16, "nstep": 1, "warm": "prev"},
        # the asynchronous host loop of a mid-sized batch: controls in, a frame of
        # several substeps, observations out
        {"name": "ant_host_4096", "kind": "step", "model": "ant", "api": "host", "n": 4096, "nstep": 4, "warm": "prev"},
        # the benchmark's headline: one substep per call, controls already on the GPU
        {"name": "ant_device_16384", "kind": "step", "model": "ant", "api": "device", "n": 16384, "nstep": 1,
         "warm": "prev"},
        # the largest batches, where throughput is all; the cold start is the faster mode
        {"name": "ant_device_65536", "kind": "step", "model": "ant", "api": "device", "n": 65536, "nstep": 1,
         "warm": "cold"},
        # sampling-based planning: short rollouts with their own controls, states back
        {"name": "ant_rollout_1000x16", "kind": "rollout", "model": "ant", "n": 1000, "nstep": 16},
        # contact-free models (control tasks, arms): a frame of ten short substeps
        {"name": "cartpole_device_16384x10", "kind": "step", "model": "cartpole", "api": "device", "n": 16384,
         "nstep": 10, "warm": "prev"},
        # many small objects on a table: primitives and general convex pairs, islands
        {"name": "tabletop_4096", "kind": "step", "model": "tabletop", "api": "device", "n": 4096, "nstep": 1,
         "warm": "prev"},
        # hulls in contact, Newton and the other solver
        {"name": "hulls_4096", "kind": "step", "model": "hulls", "api": "device", "n": 4096, "nstep": 1, "warm": "prev"},
        {"name": "hulls_pgs_1001", "kind": "step", "model": "hulls", "api": "device", "n": 1001, "nstep": 1,
         "warm": "pgs"},
        # the end of an episode: new masses and friction per env, a part of the
        # envs reset, the poses handed to a renderer
        {"name": "ant_randomise_8192", "kind": "randomise", "model": "ant", "n": 8192},
        # image observations for a policy on the GPU
        {"name": "render_device_4096_64", "kind": "render", "api": "device", "n": 4096, "size": 64},
        # images for a host program (logging, data sets)
        {"name": "render_host_250_128", "kind": "render", "api": "host", "n": 250, "size": 128},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["ant", "ant", "ant", "rollout", "free", "free", "tabletop", "hulls", "randomise", "render",
                       "render"])
    if kind == "ant":
        return {"kind": "step", "model": "ant", "api": rng.choice(["device", "device", "host"]),
                "n": _log_int(rng, 8, 65536), "nstep": rng.choice([1, 1, 2, 4]), "warm": rng.choice(["prev", "cold"])}
    if kind == "rollout":
        return {"kind": "rollout", "model": "ant", "n": _log_int(rng, 16, 3000), "nstep": rng.randint(4, 20)}
    if kind == "free":
        return {"kind": "step", "model": rng.choice(["cartpole", "arm3hinge", "arm3d"]),
                "api": rng.choice(["device", "host"]), "n": _log_int(rng, 16, 20000), "nstep": rng.randint(1, 10),
                "warm": "prev"}
    if kind == "tabletop":
        return {"kind": "step", "model": "tabletop", "api": "device", "n": _log_int(rng, 60, 4096), "nstep": 1,
                "warm": rng.choice(["prev", "cold"])}
    if kind == "hulls":
        warm = rng.choice(["prev", "cold", "pgs"])
        return {"kind": "step", "model": "hulls", "api": "device",
                "n": _log_int(rng, 60, 1000 if warm == "pgs" else 4096), "nstep": 1, "warm": warm}
    if kind == "randomise":
        return {"kind": "randomise", "model": "ant", "n": _log_int(rng, 100, 16384)}
    api = rng.choice(["device", "host"])
    return {"kind": "render", "api": api, "n": _log_int(rng, 16, 2000 if api == "device" else 250),
            "size": rng.randint(32, 128)}


# ------------------------------------------------------------------ models
@functools.lru_cache(maxsize=None)
def _model(name):
    xml = {"ant": lambda: scenes.ant_xml(tolerance=TOL, iterations=ITERS), "cartpole": scenes.cartpole_xml,
           "arm3hinge": scenes.arm3hinge_xml, "arm3d": scenes.arm3d_xml, "hulls": scenes.hull_tumble_xml}[name]()
    m = mjcf.load_string(xml)
    return m, mjcf.to_blob(m)


@functools.lru_cache(maxsize=2)
def _tabletop(n):
    plan = scenes.tabletop(n, seed=5)
    m = mjcf.load_string(plan.xml)
    return plan, m, mjcf.to_blob(m)


def _unit(x):
    return x / np.linalg.norm(x, axis=-1, keepdims=True)


def _ant_state(m, n, rng):
    """A walking Ant: torso near its standing height, slightly tilted, hips and
    ankles over their whole range and a little past it."""
    q = np.tile(np.array(m.qpos0), (n, 1))
    q[:, 0:2] = rng.uniform(-3, 3, (n, 2))
    q[:, 2] = rng.uniform(0.5, 0.8, n)
    q[:, 3:7] = _unit(np.concatenate([np.ones((n, 1)), rng.normal(0, [0.12, 0.12, 0.4], (n, 3))], axis=1))
    q[:, 7::2] = rng.uniform(-0.56, 0.56, (n, 4))
    q[:, 8::2] = np.array([1, -1, -1, 1]) * rng.uniform(0.48, 1.26, (n, 4))
    v = rng.normal(0, [0.5] * 3 + [1.2] * 3 + [2.5] * 8, (n, m.nv))
    return q, v


def _free_state(m, n, rng):
    q = np.tile(np.array(m.qpos0), (n, 1))
    for j in range(m.njnt):
        a = m.jnt_qposadr[j]
        if m.jnt_type[j] == mjcf.JNT_HINGE:
            q[:, a] += rng.uniform(-np.pi, np.pi, n)
        elif m.jnt_type[j] == mjcf.JNT_SLIDE:
            q[:, a] += rng.uniform(-0.5, 0.5, n)
        else:  # ball
            q[:, a:a + 4] = _unit(rng.normal(size=(n, 4)))
    return q, rng.normal(0, 1, (n, m.nv))


def _table_state(plan, n, rng):
    """Objects at rest on the table (upright to a milliradian, their lowest
    points a fraction of a millimetre in it); one in twenty topples from a
    random pose."""
    q = plan.qpos0.copy()
    slots = plan.nq // 7
    on = {e: v for p, e, v in plan.params if p == int(Param.GEOM_CONTYPE)}
    size = {e: v for p, e, v in plan.params if p == int(Param.GEOM_SIZE)}
    v = rng.normal(0, 1e-3, (n, 6 * slots))
    for s in range(slots):
        g = 6 + 3 * s  # the slot's box, cylinder, sphere
        active = q[:, 7 * s] < 50.0  # the others are parked away from the table
        rest = (on[g][:, 0] * size[g][:, 2] + on[g + 1][:, 0] * size[g + 1][:, 1] + on[g + 2][:, 0] * size[g + 2][:, 0])
        yaw = rng.uniform(-np.pi, np.pi, n)
        up = _unit(np.stack([np.cos(yaw / 2), rng.normal(0, 5e-4, n), rng.normal(0, 5e-4, n), np.sin(yaw / 2)], axis=1))
        topple = rng.random(n) < 0.05
        quat = np.where(topple[:, None], _unit(rng.normal(size=(n, 4))), up)
        z = 0.4 + rest + np.where(topple, rng.uniform(0.005, 0.02, n), rng.uniform(-3e-4, -1e-4, n))
        q[active, 7 * s + 2] = z[active]
        q[active, 7 * s + 3:7 * s + 7] = quat[active]
        v[~active, 6 * s:6 * s + 6] = 0.0
    return q, v


@functools.lru_cache(maxsize=None)
def _rest_faces():
    """Of each hull of the tumble: the quaternions that turn a face it can
    rest on (the centre of mass over it) down, and its height above the floor."""
    m, _ = _model("hulls")
    out = []
    for b in range(m.nv // 6):
        vert, com = np.asarray(m.hull_vert[b]), np.asarray(m.body_ipos[b + 1])
        faces, _ = mjcf.hull_features(m.hull_vert[b], m.hull_tri[b])
        rows = []
        for nrm, d, loop in faces:
            nrm, p = np.asarray(nrm), vert[loop]
            over = np.einsum("ij,ij->i", np.cross(np.roll(p, -1, 0) - p, com - p), np.tile(nrm, (len(p), 1))) > 0
            if over.all():
                c, w = np.cross(nrm, [0, 0, -1.0]), 1.0 - nrm[2]
                rows.append(np.concatenate([_unit(np.array([w, *c])) if w > 1e-9 else [0.0, 1, 0, 0], [d]]))
        out.append(np.array(rows))
    return out


def _hull_state(m, n, rng):
    """Hulls lying on their faces, some against a neighbour; one in twenty topples."""
    q = np.tile(np.array(m.qpos0), (n, 1))
    v = rng.normal(0, 1e-3, (n, m.nv))
    for b, rest in enumerate(_rest_faces()):
        f = rest[rng.integers(len(rest), size=n)]
        yaw = rng.uniform(-np.pi, np.pi, n)
        cz, sz = np.cos(yaw / 2), np.sin(yaw / 2)
        w, x, y, z = f[:, 0], f[:, 1], f[:, 2], f[:, 3]
        down = np.stack([cz * w - sz * z, cz * x - sz * y, cz * y + sz * x, cz * z + sz * w], axis=1)
        topple = rng.random(n) < 0.05
        q[:, 7 * b:7 * b + 2] += rng.uniform(-0.03, 0.03, (n, 2))
        q[:, 7 * b + 2] = np.where(topple, 0.06, f[:, 4] - rng.uniform(1e-4, 3e-4, n))
        q[:, 7 * b + 3:7 * b + 7] = np.where(topple[:, None], _unit(rng.normal(size=(n, 4))), down)
    return q, v


# ------------------------------------------------------------------ prepare
def _physics(case, rng):
    n, name = case["n"], case["model"]
    envs = range(n)
    if name == "tabletop":
        plan, m, blob = _tabletop(n)
        p = CudaPhysics(blob, n)
        plan.apply(lambda pid, e, v: p.set_param(Param(pid), e, envs, v), lambda: p.reset(envs))
        q, v = _table_state(plan, n, rng)
    else:
        m, blob = _model(name)
        p = CudaPhysics(blob, n)
        q, v = {"ant": _ant_state, "hulls": _hull_state}.get(name, _free_state)(m, n, rng)
    warm = case.get("warm", "prev")
    p.set_solver(kind=int(Solver.PGS if warm == "pgs" else Solver.NEWTON), iterations=ITERS, tolerance=TOL,
                 warm=int(WarmStart.COLD if warm == "cold" else WarmStart.REF_PREV_QACC))
    p.set(Field.QPOS, envs, q)
    p.set(Field.QVEL, envs, v)
    return m, p


def _views(size):
    return RenderConfig(size, size, [ViewSource.look_at([1.5, -1.5, 1.2], [0.0, 0.0, 0.3], 45.0)], 0.01, 20.0)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    n = case["n"]
    st = {"case": case, "t": 0, "envs": range(n)}
    if case["kind"] == "render":
        m, p = _physics(dict(case, model="ant"), rng)
        q = p.get(Field.QPOS, range(n))
        q[:, 0:2] = rng.uniform(-0.3, 0.3, (n, 2))  # in the view
        p.set(Field.QPOS, range(n), q)
        scene = p.scene()
        r = CudaRenderer(scene, _views(case["size"]))
        st.update(renderer=r, n=n)
        if case["api"] == "host":
            st["geoms"], st["cams"] = p.poses(range(n))
        else:
            st["geoms"] = torch.empty((n, len(scene.geoms), 12), dtype=torch.float32, device="cuda")
            p.poses_device(range(n), st["geoms"].data_ptr())
            px = (n, 1, case["size"], case["size"])
            st["look"] = torch.from_numpy(np.tile(r.base_appearance, (n, 1, 1))).cuda()
            st["rgba"] = torch.zeros(px + (4,), dtype=torch.uint8, device="cuda")
            st["depth"] = torch.zeros(px, dtype=torch.float32, device="cuda")
            st["seg"] = torch.zeros(px, dtype=torch.int32, device="cuda")
        p.synchronize()
        p.close()
        return st
    m, p = _physics(case, rng)
    st["p"] = p
    if case["kind"] == "step":
        sets = rng.uniform(-1, 1, (N_CTRL, n, m.nu))
        if case["api"] == "device":
            st["ctrl"] = torch.from_numpy(sets).cuda()
            st["view"] = [p.device_view(f) for f in (Field.QPOS, Field.QVEL, Field.QACC)]
        else:
            st["ctrl"] = torch.from_numpy(sets).pin_memory().numpy()
            st["out"] = [torch.empty((n, w), dtype=torch.float64).pin_memory().numpy() for w in (m.nq, m.nv)]
    elif case["kind"] == "rollout":
        st["ctrl"] = rng.uniform(-1, 1, (N_CTRL, n, case["nstep"], m.nu))
    else:  # randomise
        k = N_CTRL
        st["mass"] = [np.asarray(m.body_mass[1]) * rng.uniform(0.7, 1.4, (n, 1)) for _ in range(k)]
        st["friction"] = [rng.uniform(0.5, 1.2, (n, 1)) for _ in range(k)]
        st["done"] = [np.sort(rng.choice(n, n // 4, replace=False)) for _ in range(k)]
        st["geoms"] = torch.zeros((n, p.dims().ngeom, 12), dtype=torch.float32, device="cuda")
        st["view"] = [p.device_view(f) for f in (Field.QPOS, Field.QVEL)]
    p.synchronize()
    return st


# ------------------------------------------------------------------ run
def run(st):
    case, envs = st["case"], st["envs"]
    k = st["t"] % N_CTRL
    st["t"] += 1
    if case["kind"] == "render":
        r = st["renderer"]
        if case["api"] == "host":
            f = r.render(0, st["n"], st["geoms"], st["cams"])
            return f.rgba, f.depth, f.segmentation
        r.render_device(st["n"], st["geoms"].data_ptr(), 0, st["look"].data_ptr(), st["rgba"].data_ptr(),
                        st["depth"].data_ptr(), st["seg"].data_ptr())
        return st["rgba"], st["depth"], st["seg"]
    p = st["p"]
    if case["kind"] == "step":
        if case["api"] == "device":
            p.step_device(envs, case["nstep"], st["ctrl"][k].data_ptr())
            return st["view"]
        p.set(Field.CTRL, envs, st["ctrl"][k])
        p.step(envs, case["nstep"])
        p.get(Field.QPOS, envs, out=st["out"][0])
        p.get(Field.QVEL, envs, out=st["out"][1])
        return st["out"]
    if case["kind"] == "rollout":
        return p.rollout(st["ctrl"][k])
    p.set_param(Param.BODY_MASS, 1, envs, st["mass"][k])
    p.set_param(Param.GEOM_FRICTION, 0, envs, st["friction"][k])
    p.reset(st["done"][k])
    p.poses_device(envs, st["geoms"].data_ptr())
    return st["geoms"], st["view"], p.get_param(Param.BODY_MASS, 1, envs)


def work(case):
    n = case["n"]
    if case["kind"] == "render":
        px = n * case["size"] ** 2
        return {"bytes": px * 12 + n * 14 * 48, "flops": px * 100 + n * 14978 * 60}
    if case["kind"] == "randomise":
        # new values in, state of the reset envs and all poses out, the set-up of M and its factor per env
        return {"bytes": n * (16 + 8 + 14 * 48) + n // 4 * 51 * 8, "flops": n * 12e3}
    nq, nv, nu = {"ant": (15, 14, 8), "cartpole": (3, 3, 2), "arm3hinge": (3, 3, 3), "arm3d": (9, 8, 4),
                  "tabletop": (42, 36, 0), "hulls": (56, 48, 0)}[case["model"]]
    state = 8 * (2 * nq + 2 * nv + 2 * nv)
    if case["kind"] == "rollout":
        return {"bytes": n * (state + case["nstep"] * 8 * (nu + nq)), "flops": n * case["nstep"] * FLOPS["ant"]}
    return {"bytes": n * (state + 8 * nu), "flops": n * case["nstep"] * FLOPS[case["model"]]}


def exact(case, seed):
    """No value but the library's own: a substep's contacts, active sets and
    line searches have no closed form in plain torch or numpy."""
    return None
