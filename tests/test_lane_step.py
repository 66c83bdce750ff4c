"""The substep with one lane or four lanes per env (pg_lane.cu, pg_quad.cu)
against the oracle, step by step from the same states: models without rows
(one lane; 4 and 8 dofs of register arrays), chains, two limbs, three and more
on a trunk (four lanes; 8, 12, 14 and 16), a second round of limbs, a tree
that neither takes, and batches around the sizes where warps and blocks fill.

Tolerance: the per-step bar of the other parity tests, 1e-10 of the largest
component (a step's rounding is below 1e-14 of it, the factorisations and the
Newton exit leave four digits more).
"""
import numpy as np
import pytest

from oracle.oracle import CTRL, QACC, QFRC_APPLIED, QPOS, QVEL, Oracle
from pippin_b200 import CudaPhysics, Field, Param, WarmStart, mjcf, scenes

pytestmark = pytest.mark.gpu
TOL = 1e-10

OPT = '<compiler angle="degree"/><option timestep="0.004" tolerance="1e-10" iterations="30"/>'
FLOOR = '<geom type="plane" size="5 5 .1" friction="0.8 0.1 0.1"/>'


def _limb(k, geom, free_end=True):
    """Two hinges, the first with a range, out along the k-th direction."""
    a = 2.0 * np.pi * k / 5.0
    x, y = 0.25 * np.cos(a), 0.25 * np.sin(a)
    g = {"capsule": f'<geom type="capsule" fromto="0 0 0 {x:.4f} {y:.4f} -0.1" size="0.05"/>',
         "sphere": f'<geom type="sphere" pos="{x:.4f} {y:.4f} -0.1" size="0.07"/>',
         "box": f'<geom type="box" pos="{x:.4f} {y:.4f} -0.1" size="0.06 0.05 0.04" euler="10 20 30"/>'}[geom]
    return (f'<body pos="{0.4 * x:.4f} {0.4 * y:.4f} 0" euler="0 0 {7 * k}">'
            f'<joint name="a{k}" axis="0 0 1" range="-20 20" limited="true" damping="0.3" armature="0.02"/>{g}'
            f'<body pos="{x:.4f} {y:.4f} -0.1"><joint name="b{k}" axis="{y:.4f} {-x:.4f} 0" pos="0.01 0 0.02" '
            f'stiffness="3" armature="0.01"/>{g}</body></body>')


def _star(limbs, root='<freejoint/>', geoms=("capsule", "sphere", "box"), extra=""):
    body = "".join(_limb(k, geoms[k % len(geoms)]) for k in range(limbs))
    motors = "".join(f'<motor joint="a{k}" gear="4"/><position joint="b{k}" kp="6" kv="0.3"/>' for k in range(limbs))
    return (f'<mujoco>{OPT}<worldbody>{FLOOR}{extra}<body pos="0 0 0.35">{root}'
            f'<geom type="sphere" size="0.1" density="400"/>{body}</body></worldbody><actuator>{motors}</actuator></mujoco>')


def _chain(n, ball=False):
    s, e = "", ""
    for k in range(n):
        ax = ["0 0 1", "0 1 0", "1 0 0"][k % 3]
        j = '<joint type="ball" damping="0.05"/>' if ball and k == n - 1 else (
            f'<joint name="j{k}" axis="{ax}" range="-40 40" limited="true" armature="0.02" damping="{0.1 * (k % 2)}"/>')
        s += (f'<body pos="0.12 0 0" euler="0 {5 * (k % 2)} 0">{j}'
              '<geom type="capsule" fromto="0 0 0 0.12 0 0" size="0.035"/>')
        e += "</body>"
    return (f'<mujoco>{OPT}<worldbody>{FLOOR}<body pos="0 0 0.1"><geom type="box" size="0.03 0.03 0.03"/>{s}{e}</body>'
            '</worldbody><actuator><motor joint="j0" gear="3"/></actuator></mujoco>')


MODELS = {
    "pendulum": scenes.pendulum_xml(),                     # one lane, 4
    "chain_7_ball": _chain(5, ball=True),                  # four lanes, 8: a trunk alone, a ball
    "chain_6": _chain(6),                                  # four lanes, 8: as deep as it goes
    "two_limbs": _star(2),                                 # four lanes, 12
    "arm3d": scenes.arm3d_xml(),                           # one lane, 8: ball, slide, offsets
    "hinge_3_limbs": _star(3, root='<joint axis="0 0 1" damping="0.2" armature="0.05"/>'),   # four lanes, 8
    "free_3_limbs": _star(3),                              # four lanes, 12
    "ant": scenes.ant_xml(timestep=0.004, tolerance=1e-10),                                 # four lanes, 14
    "free_5_limbs": _star(5),                              # four lanes, 16: two rounds of limbs
    # the phase kernels: a branching tree and a static body beside it
    "static_box": _star(4, geoms=("capsule",), extra='<body pos="0.3 0 0"><geom type="box" size="0.1 0.5 0.05"/></body>'),
}


LANES = {"pendulum": 1, "arm3d": 1, "static_box": 0}  # the others: 4


def _states(m, n, rng):
    q = np.tile(np.array(m.qpos0), (n, 1))
    for j in range(m.njnt):
        a, t = m.jnt_qposadr[j], m.jnt_type[j]
        if t == mjcf.JNT_FREE:
            q[:, a:a + 2] = rng.uniform(-0.2, 0.2, (n, 2))
            q[:, a + 2] = rng.uniform(0.1, 0.5, n)
            a += 3
        if t in (mjcf.JNT_FREE, mjcf.JNT_BALL):
            w = rng.normal(0, 1, (n, 4)) * 0.15 + np.array([1.0, 0, 0, 0])
            q[:, a:a + 4] = w / np.linalg.norm(w, axis=1, keepdims=True)
        elif t == mjcf.JNT_HINGE:
            q[:, a] += rng.uniform(-0.8, 0.8, n)
        else:
            q[:, a] += rng.uniform(-0.1, 0.1, n)
    return q, rng.normal(0, 1.0, (n, m.nv))


def _rel(a, b):
    return float(np.max(np.abs(a - b)) / max(float(np.max(np.abs(b))), 1.0))


@pytest.mark.parametrize("name", list(MODELS))
@pytest.mark.parametrize("n", [1, 8, 33, 700])
def test_step_matches_oracle(name, n):
    m = mjcf.load_string(MODELS[name])
    blob = mjcf.to_blob(m)
    g, o = CudaPhysics(blob, n), Oracle(blob, n, threads=8)
    assert g.step_lanes() == LANES.get(name, 4)
    o.set_solver(tolerance=1e-10, iterations=30)
    g.set_solver(tolerance=1e-10, iterations=30, warm=int(WarmStart.REF_PREV_QACC))
    rng = np.random.default_rng(n)
    q, v = _states(m, n, rng)
    g.set(Field.QPOS, range(n), q)
    g.set(Field.QVEL, range(n), v)
    rows = 0
    for t in range(6):
        if t == 3:  # per-env parameters: the kernels' own copy of them
            mass = np.asarray(m.body_mass[m.nbody - 1]) * rng.uniform(0.7, 1.5, (n, 1))
            fric = rng.uniform(0.4, 1.1, (n, 1))
            for pid, elem, val in ((5, m.nbody - 1, mass), (0, 0, fric), (6, m.nv - 1, fric)):
                g.set_param(Param(pid), elem, range(n), val)
                o.set_param(pid, elem, val, 0, n)
        if m.nu:
            g.set(Field.CTRL, range(n), rng.uniform(-1, 1, (n, m.nu)))
        for fg, fo in ((Field.QPOS, QPOS), (Field.QVEL, QVEL), (Field.QACC, QACC), (Field.CTRL, CTRL)):
            if g.dims().width(fg):
                o.set(fo, g.get(fg, range(n)))
        g.step(range(n), 1)
        o.step(0, n, 1)
        for fg, fo in ((Field.QACC, QACC), (Field.QVEL, QVEL), (Field.QPOS, QPOS)):
            assert _rel(g.get(fg, range(n)), o.get(fo)) < TOL, (t, fg)
        sg, so = g.stats(), o.stats()
        np.testing.assert_array_equal(sg["ncon"], so["ncon"])
        np.testing.assert_array_equal(sg["nrows"], so["nrows"])
        assert not sg["status"].any()
        rows += int(sg["nrows"].sum())
    assert rows > 0 or n < 33 or name in ("pendulum", "arm3d")  # (these two have no contacts and no limits)


def test_named_shape_runs_the_phase_kernels():
    """set_launch names a shape of the phase kernels: the step then takes
    them, and agrees with the default within the step tolerance."""
    n = 100
    m = mjcf.load_string(MODELS["ant"])
    blob = mjcf.to_blob(m)
    a, b = CudaPhysics(blob, n), CudaPhysics(blob, n)
    b.set_launch(16, 4)
    q, v = _states(m, n, np.random.default_rng(3))
    for p in (a, b):
        p.set(Field.QPOS, range(n), q)
        p.set(Field.QVEL, range(n), v)
        p.step(range(n), 2)
    assert _rel(a.get(Field.QACC, range(n)), b.get(Field.QACC, range(n))) < TOL


def test_masks_that_let_pairs_touch_leave_the_one_lane_step():
    """A model whose pairs are all masked out steps one lane an env; once
    set_param lets geoms touch, its contacts are found like the oracle's."""
    n = 40
    xml = _chain(5).replace("<geom ", '<geom contype="0" conaffinity="0" ').replace('limited="true"', 'limited="false"')
    m = mjcf.load_string(xml)
    blob = mjcf.to_blob(m)
    g, o = CudaPhysics(blob, n), Oracle(blob, n, threads=8)
    for sim in (g, o):
        sim.set_solver(tolerance=1e-10, iterations=30)
    q, v = _states(m, n, np.random.default_rng(4))
    g.set(Field.QPOS, range(n), q)
    g.set(Field.QVEL, range(n), v)
    assert g.step_lanes() == 1
    contacts = 0
    for t in range(6):
        if t == 2:
            for geom in range(len(m.geom_body)):
                for pid in (3, 4):
                    g.set_param(Param(pid), geom, range(n), np.ones((n, 1)))
                    o.set_param(pid, geom, np.ones((n, 1)), 0, n)
            assert g.step_lanes() == 0
        for fg, fo in ((Field.QPOS, QPOS), (Field.QVEL, QVEL), (Field.QACC, QACC), (Field.CTRL, CTRL)):
            o.set(fo, g.get(fg, range(n)))
        g.step(range(n), 1)
        o.step(0, n, 1)
        assert _rel(g.get(Field.QACC, range(n)), o.get(QACC)) < TOL, t
        np.testing.assert_array_equal(g.stats()["ncon"], o.stats()["ncon"])
        contacts += int(g.stats()["ncon"].sum())
    assert contacts > 0


def test_long_calls_and_cold_start():
    """A call longer than one launch takes, and the cold start, from one state
    give the bits of single steps."""
    n, t = 40, 130
    m = mjcf.load_string(MODELS["free_5_limbs"])
    blob = mjcf.to_blob(m)
    a, b = CudaPhysics(blob, n), CudaPhysics(blob, n)
    q, v = _states(m, n, np.random.default_rng(9))
    for p in (a, b):
        p.set_solver(warm=int(WarmStart.COLD))
        p.set(Field.QPOS, range(n), q)
        p.set(Field.QVEL, range(n), v)
    a.step(range(n), t)
    for _ in range(t):
        b.step(range(n), 1)
    for f in (Field.QPOS, Field.QVEL, Field.QACC):
        np.testing.assert_array_equal(a.get(f, range(n)), b.get(f, range(n)))


# light limbs on a heavy trunk, stiff contacts and limits, tangents far softer
# and far harder than the normals
HARD = {
    "light_limbs": dict(limb="2", trunk="40000"),
    "impratio_100": dict(opt='impratio="100"'),
    "impratio_0.01": dict(opt='impratio="0.01"'),
    "stiff": dict(opt='o_solref="0.009 1"', solimp=(0.95, 0.9999, 0.0005, 0.5, 2.0)),
    "light_and_stiff": dict(limb="2", trunk="40000", opt='impratio="100"', solimp=(0.95, 0.9999, 0.0005, 0.5, 2.0)),
}


@pytest.mark.parametrize("hard", list(HARD))
@pytest.mark.parametrize("name", ["free_3_limbs", "free_5_limbs"])
def test_hard_models_lose_no_more_than_in_the_phase_kernels(name, hard):
    """M and the Newton systems with condition numbers two to six decades
    above the other models': the four-lane step's qacc is as near to the
    oracle's as that of the phase kernels. Both factorisations are backward
    stable, so their errors differ by a small factor (8 is allowed, above a
    floor of 1e-13, some rounding of a well-conditioned step)."""
    n = 120
    opt = HARD[hard]
    xml = MODELS[name].replace('density="400"', f'density="{opt.get("trunk", 400)}"')
    if "limb" in opt:
        for geom in ('size="0.05"/>', 'size="0.07"/>', 'euler="10 20 30"/>'):
            xml = xml.replace(geom, f'{geom[:-2]} density="{opt["limb"]}"/>')
        xml = xml.replace('armature="0.02"', "").replace('armature="0.01"', "")
    xml = xml.replace('iterations="30"/>', f'iterations="30" {opt.get("opt", "")}/>')
    m = mjcf.load_string(xml)
    m.solimp = opt.get("solimp", m.solimp)
    blob = mjcf.to_blob(m)
    lanes, phases, o = CudaPhysics(blob, n), CudaPhysics(blob, n), Oracle(blob, n, threads=8)
    phases.set_launch(16, 4)
    assert (lanes.step_lanes(), phases.step_lanes()) == (4, 0)
    for sim in (lanes, phases, o):
        sim.set_solver(tolerance=1e-10, iterations=60)
    rng = np.random.default_rng(17)
    q, v = _states(m, n, rng)
    lanes.set(Field.QPOS, range(n), q)
    lanes.set(Field.QVEL, range(n), v)
    worst, rows = [0.0, 0.0], 0
    for _ in range(6):
        lanes.set(Field.CTRL, range(n), rng.uniform(-1, 1, (n, m.nu)))
        for fg, fo in ((Field.QPOS, QPOS), (Field.QVEL, QVEL), (Field.QACC, QACC), (Field.CTRL, CTRL)):
            s = lanes.get(fg, range(n))
            o.set(fo, s)
            phases.set(fg, range(n), s)
        for p in (lanes, phases):
            p.step(range(n), 1)
        o.step(0, n, 1)
        ref = o.get(QACC)
        scale = np.maximum(np.abs(ref).max(axis=1), 1.0)
        for k, p in enumerate((lanes, phases)):
            worst[k] = max(worst[k], float((np.abs(p.get(Field.QACC, range(n)) - ref).max(axis=1) / scale).max()))
        assert not lanes.stats()["status"].any()
        rows += int(lanes.stats()["nrows"].sum())
    assert rows > 0
    assert worst[0] <= 8 * max(worst[1], 1e-13), worst


def _oracle_step(g, o, n, tol):
    """One substep of both from g's states: the largest relative difference,
    which must be below tol."""
    for fg, fo in ((Field.QPOS, QPOS), (Field.QVEL, QVEL), (Field.QACC, QACC), (Field.CTRL, CTRL)):
        if g.dims().width(fg):
            o.set(fo, g.get(fg, range(n)))
    g.step(range(n), 1)
    o.step(0, n, 1)
    sg, so = g.stats(), o.stats()
    np.testing.assert_array_equal(sg["ncon"], so["ncon"])
    np.testing.assert_array_equal(sg["nrows"], so["nrows"])
    assert not sg["status"].any()
    for fg, fo in ((Field.QACC, QACC), (Field.QVEL, QVEL), (Field.QPOS, QPOS)):
        assert _rel(g.get(fg, range(n)), o.get(fo)) < tol, fg
    return so


@pytest.mark.parametrize("name", ["chain_6", "free_3_limbs", "pendulum_chain"])
def test_body_frames_turned_by_less_than_the_real_part_shows(name):
    """A body frame turned by 2e-8 has a quaternion whose real part rounds to
    one; the turn still tilts all that hangs on it."""
    n = 33
    xml = MODELS.get(name) or _chain(4).replace("<geom ", '<geom contype="0" conaffinity="0" ').replace(
        'limited="true"', 'limited="false"')
    xml = xml.replace('<body pos="0.12 0 0" euler="0 0 0">', '<body pos="0.12 0 0" quat="1 9e-9 -9e-9 9e-9">')
    xml = xml.replace('euler="0 0 0"', 'quat="1 9e-9 -9e-9 9e-9"')
    assert "9e-9" in xml
    m = mjcf.load_string(xml)
    blob = mjcf.to_blob(m)
    assert any(q[0] == 1.0 and q[1] != 0.0 for q in np.reshape(m.body_quat, (-1, 4)))
    g, o = CudaPhysics(blob, n), Oracle(blob, n, threads=4)
    assert g.step_lanes() == (1 if name == "pendulum_chain" else 4)
    for sim in (g, o):
        sim.set_solver(tolerance=1e-10, iterations=30)
    q, v = _states(m, n, np.random.default_rng(2))
    g.set(Field.QPOS, range(n), q)
    g.set(Field.QVEL, range(n), v)
    _oracle_step(g, o, n, TOL)


def _arms(arms, depth, fork=0, root=True):
    """Contact-free arms of `depth` hinges off one body, `fork` more bodies at
    the end of each."""
    g = '<geom type="capsule" fromto="0 0 0 0.12 0 0" size="0.035" contype="0" conaffinity="0"/>'

    def link(k, inner):
        axis = ["0 0 1", "0 1 0", "1 0 0"][k % 3]
        return (f'<body pos="0.12 0.02 0" euler="0 {5 * (k % 3)} {4 * k}"><joint axis="{axis}" armature="0.02" '
                f'damping="{0.1 * (k % 2)}"/>{g}{inner}</body>')

    def arm(a, k):
        return "".join(link(a + k + f, "") for f in range(fork)) if k == depth else link(a + k, arm(a, k + 1))

    body = "".join(arm(a, 0) for a in range(arms))
    joint = '<joint axis="0 0 1" armature="0.1"/>' if root else ""
    return f'<mujoco>{OPT}<worldbody><body pos="0 0 1">{joint}{g}{body}</body></worldbody></mujoco>'


FREE = {  # dofs, lanes
    "arm_of_7": (_arms(1, 7, root=False), 7, 1),
    "two_arms_and_root_9": (_arms(2, 4), 9, 4),
    "two_arms_15": (_arms(2, 7), 15, 4),
    "three_arms_16": (_arms(3, 5), 16, 4),
    "forks_7": (_arms(2, 1, fork=2), 7, 1),
    "forks_13": (_arms(4, 1, fork=2), 13, 0),
}


@pytest.mark.parametrize("name", list(FREE))
@pytest.mark.parametrize("n", [1, 33, 700, 5001])
def test_models_without_rows(name, n):
    """One lane up to 8 dofs, four lanes up to 16 where the branches are
    chains, the phase kernels beyond."""
    xml, dofs, lanes = FREE[name]
    m = mjcf.load_string(xml)
    assert m.nv == dofs
    blob = mjcf.to_blob(m)
    g, o = CudaPhysics(blob, n), Oracle(blob, n, threads=8)
    assert g.step_lanes() == lanes
    rng = np.random.default_rng(n)
    q, v = _states(m, n, rng)
    g.set(Field.QPOS, range(n), q)
    g.set(Field.QVEL, range(n), v)
    g.set(Field.QFRC_APPLIED, range(n), rng.normal(0, 1, (n, m.nv)))
    o.set(QFRC_APPLIED, g.get(Field.QFRC_APPLIED, range(n)))
    for _ in range(3):
        assert not _oracle_step(g, o, n, TOL)["nrows"].any()


@pytest.mark.parametrize("name", ["hinge_3_limbs", "free_3_limbs", "free_5_limbs"])
@pytest.mark.parametrize("n", [2501, 9001])
def test_full_warps_and_blocks(name, n):
    """Batches of four and eight envs a warp, the last warp ragged, up to
    eight warps a block, for each size of the matrix but Ant's."""
    m = mjcf.load_string(MODELS[name])
    blob = mjcf.to_blob(m)
    g, o = CudaPhysics(blob, n), Oracle(blob, n, threads=8)
    assert g.step_lanes() == 4
    for sim in (g, o):
        sim.set_solver(tolerance=1e-10, iterations=30)
    q, v = _states(m, n, np.random.default_rng(n))
    g.set(Field.QPOS, range(n), q)
    g.set(Field.QVEL, range(n), v)
    for _ in range(2):
        rows = _oracle_step(g, o, n, TOL)["nrows"]
    assert rows.any()


def test_more_than_128_candidate_pairs():
    """A second pass of the pair loop, whose pairs (limb against limb, after
    those of the floor and the trunk) touch while earlier ones do as well."""
    n = 60
    extra = "".join(f'<geom type="sphere" size="0.03" pos="{0.02 * k - 0.13:.2f} 0 0.08"/>' for k in range(14))
    xml = _star(5, geoms=("sphere",)).replace('density="400"/>', f'density="400"/>{extra}').replace('size="0.07"/>', 'size="0.22"/>')
    m = mjcf.load_string(xml)
    blob = mjcf.to_blob(m)
    ng = len(m.geom_type)
    assert ng <= 32
    g, o = CudaPhysics(blob, n), Oracle(blob, n, threads=8)
    assert g.step_lanes() == 4
    for sim in (g, o):
        sim.set_solver(tolerance=1e-10, iterations=30)
    q, v = _states(m, n, np.random.default_rng(6))
    g.set(Field.QPOS, range(n), q)
    g.set(Field.QVEL, range(n), v)
    early = late = 0
    for _ in range(3):
        for e in range(n):
            pairs = [(int(c[10]), int(c[11])) for c in g.debug_forward(e)["contacts"]]
            late += any(min(p) >= ng - 4 for p in pairs)  # between the last two limbs
            early += any(min(p) == 0 for p in pairs)      # with the floor
        _oracle_step(g, o, n, TOL)
    assert early and late
