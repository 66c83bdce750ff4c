"""What must hold whichever kernel a step runs in: a captured step replays with
the parameters of the time it is replayed at, calls that a caller's stream
capture cannot take are refused, and setting parameters costs no device memory.

Two handles start from the same states; one replays a captured step, the other
steps live after the same calls. They may run different kernels, so they agree
within the per-step bar of the other parity tests, 1e-10.
"""
import numpy as np
import pytest
import torch

from pippin_b200 import CudaPhysics, Field, Param, PhysicsError, _native, mjcf, scenes
from tests.test_lane_step import MODELS, TOL, _chain, _rel, _states

pytestmark = pytest.mark.gpu


class Capture:
    """What runs inside, recorded from the handle's stream."""

    def __init__(self, phys):
        self.stream = torch.cuda.ExternalStream(phys.stream())
        self.graph = torch.cuda.CUDAGraph()

    def __enter__(self):
        torch.cuda.synchronize()
        self.scope = torch.cuda.stream(self.stream)
        self.scope.__enter__()
        self.graph.capture_begin(capture_error_mode="thread_local")
        return self

    def __exit__(self, *exc):
        self.graph.capture_end()
        self.scope.__exit__(None, None, None)

    def replay(self):
        with torch.cuda.stream(self.stream):
            self.graph.replay()


def _pair(xml, n, seed):
    m = mjcf.load_string(xml)
    blob = mjcf.to_blob(m)
    a, b = CudaPhysics(blob, n), CudaPhysics(blob, n)
    q, v = _states(m, n, np.random.default_rng(seed))

    def start():
        for p in (a, b):
            p.set(Field.QPOS, range(n), q)
            p.set(Field.QVEL, range(n), v)
            p.set(Field.QACC, range(n), np.zeros((n, m.nv)))

    start()
    return m, a, b, start


def _static(p, n, nstep=1):
    assert _native.load().pg_step_static(p._h, 0, n, nstep) == 0, _native.last_error()


@pytest.mark.parametrize("name", ["ant", "pendulum", "chain_6", "static_box"])
def test_a_captured_step_takes_the_parameters_of_its_replay(name):
    n = 24
    m, a, b, start = _pair(MODELS[name], n, 21)
    for p in (a, b):
        _static(p, n)  # loads the library's device image
        p.synchronize()
    with Capture(a) as c:
        _static(a, n, 2)
    rng = np.random.default_rng(22)
    start()
    base = CudaPhysics(mjcf.to_blob(m), n)
    for f in (Field.QPOS, Field.QVEL):
        base.set(f, range(n), a.get(f, range(n)))
    body = m.nbody - 1
    mass = np.asarray(m.body_mass[body]) * rng.uniform(0.5, 2.0, (n, 1))
    damp = rng.uniform(0.1, 2.0, (n, 1))
    fric = rng.uniform(0.2, 1.5, (n, 1))
    for p in (a, b):
        for pid, elem, val in ((5, body, mass), (6, m.nv - 1, damp), (0, 0, fric)):
            p.set_param(Param(pid), elem, range(n), val)
    c.replay()
    a.synchronize()  # (the static scratch is shared: one handle at a time)
    for p in (b, base):
        _static(p, n, 2)
        p.synchronize()
    for f in (Field.QACC, Field.QVEL, Field.QPOS):
        assert _rel(a.get(f, range(n)), b.get(f, range(n))) < TOL, f
    assert _rel(a.get(Field.QACC, range(n)), base.get(Field.QACC, range(n))) > 1e-3  # the parameters matter


@pytest.mark.parametrize("solver", [0, 1], ids=["newton", "pgs"])
def test_set_param_takes_no_device_memory(solver):
    """(But for the values themselves: a copy of the parameter blocks of these
    envs would take 56 MB.)"""
    free = 0
    for n in (4, 16384):  # the small handle loads the kernels
        p = CudaPhysics(scenes.ant_xml(), n)
        p.set_solver(kind=solver)
        free = torch.cuda.mem_get_info()[0]
        p.set_param(Param.BODY_MASS, 1, range(n), np.full((n, 1), 2.0))
    assert free - torch.cuda.mem_get_info()[0] < 8 << 20


def test_a_captured_step_finds_the_contacts_that_new_masks_allow():
    n = 40
    xml = _chain(5).replace("<geom ", '<geom contype="0" conaffinity="0" ').replace('limited="true"', 'limited="false"')
    m, a, b, start = _pair(xml, n, 4)
    assert a.step_lanes() == 1
    for p in (a, b):
        _static(p, n)
        p.synchronize()
    with Capture(a) as c:
        _static(a, n)
    start()
    for p in (a, b):
        for geom in range(len(m.geom_body)):
            for pid in (3, 4):
                p.set_param(Param(pid), geom, range(n), np.ones((n, 1)))
    c.replay()
    a.synchronize()
    _static(b, n)
    b.synchronize()
    assert b.stats()["ncon"].sum() > 0
    np.testing.assert_array_equal(a.stats()["ncon"], b.stats()["ncon"])
    assert _rel(a.get(Field.QACC, range(n)), b.get(Field.QACC, range(n))) < TOL


@pytest.mark.parametrize("name", ["ant", "pendulum", "static_box"])
def test_steps_that_cannot_be_captured_are_refused(name):
    """pg_step and pg_step_device replay graphs of their own: under a caller's
    capture they return an error, whichever kernel the handle steps in, and
    the handle steps on afterwards."""
    n = 8
    m, a, b, _ = _pair(MODELS[name], n, 5)
    ctrl = torch.zeros(n, max(m.nu, 1), dtype=torch.float64, device="cuda")
    with Capture(a):
        with pytest.raises(PhysicsError, match="captur"):
            a.step(range(n), 1)
        with pytest.raises(PhysicsError, match="captur"):
            a.step_device(range(n), 1, ctrl.data_ptr())
    for p in (a, b):
        p.step(range(n), 1)
        p.synchronize()
    np.testing.assert_array_equal(a.get(Field.QACC, range(n)), b.get(Field.QACC, range(n)))


def test_static_steps_refuse_models_past_their_scratch():
    """Four links of 28 masked-out boxes each: 2352 candidate pairs, whose rows
    take 4 MB a tile, 17 a block. The step needs no tile while nothing can
    touch, but may need one for the next call; pg_step takes the model."""
    box = "".join(f'<geom type="box" size="0.01 0.01 0.01" pos="0 0 {0.03 * i:.2f}" contype="0" conaffinity="0"/>'
                  for i in range(28))
    link = f'<body pos="0.1 0 0"><joint axis="0 1 0"/>{box}'
    p = CudaPhysics(f'<mujoco><worldbody>{4 * link}{4 * "</body>"}</worldbody></mujoco>', 2)
    assert p.step_lanes() == 1
    assert _native.load().pg_step_static(p._h, 0, 2, 1) == 4  # PG_ERR_UNSUPPORTED
    assert "scratch" in _native.last_error()
    p.step(range(2), 1)
    p.synchronize()


def test_set_launch_and_autotune_leave_the_kernel_to_the_caller():
    n = 2048
    p = CudaPhysics(scenes.ant_xml(), n)
    assert p.step_lanes() == 4
    with pytest.raises(PhysicsError):
        p.set_launch(64, 4)  # refused: nothing changes
    assert p.step_lanes() == 4
    p.set_launch(32, 1)
    assert p.step_lanes() == 0
    p.set_launch()  # names no shape any more
    assert p.step_lanes() == 4
    shapes = p.phase_launch()
    assert all(s[:2] == (32, 1) for s in shapes.values())
    # the phase kernels' shapes are searched all the same: PGS, the learned
    # start and time_phases run in them
    rng = np.random.default_rng(0)
    p.set(Field.QVEL, range(n), rng.normal(0, 1, (n, 14)))
    p.step(range(n), 20)
    state = {f: p.get(f, range(n)) for f in Field}
    p.autotune()
    assert p.step_lanes() == 4
    assert any(s[:2] != (32, 1) for s in p.phase_launch().values())
    for f in Field:
        np.testing.assert_array_equal(p.get(f, range(n)), state[f])


@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 33])
def test_get_param_returns_what_set_param_wrote(count):
    n, s0 = 70, 30
    p = CudaPhysics(scenes.ant_xml(), n)
    rng = np.random.default_rng(count)
    for pid in Param:
        w = p.param_width(pid)
        if pid == Param.QPOS0:
            val = np.tile(p.get_param(pid, 0, range(1)), (count, 1)) + 0.01 * rng.random((count, 1))
            val[:, 3:7] = [1.0, 0.0, 0.0, 0.0]
        elif pid in (Param.GEOM_CONTYPE, Param.GEOM_CONAFFINITY):
            val = rng.integers(0, 8, (count, w)).astype(float)
        elif pid == Param.BODY_INERTIA:
            val = 1.0 + 0.1 * rng.random((count, w))
        else:  # (colours are kept in 32 bits)
            val = (0.5 + rng.random((count, w))).astype(np.float32).astype(float)
        before = p.get_param(pid, 0 if pid == Param.QPOS0 else 1, range(n))
        elem = 0 if pid == Param.QPOS0 else 1
        p.set_param(pid, elem, range(s0, s0 + count), val)
        np.testing.assert_array_equal(p.get_param(pid, elem, range(s0, s0 + count)), val)
        for e in (s0 - 1, s0 + count):  # the neighbours keep theirs
            np.testing.assert_array_equal(p.get_param(pid, elem, range(e, e + 1))[0], before[e])


def test_collision_lanes_by_pairs_and_batch():
    """Models of many pairs take 32 lanes an env in the collision phase while
    one wave holds the batch, 16 beyond; models of few pairs 16."""
    tabletop = scenes.tabletop(2).xml
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for xml, n, lanes in ((tabletop, 60, 32), (tabletop, 16 * sms, 32), (tabletop, 16 * sms + 1, 16),
                          (scenes.hull_tumble_xml(), 60, 16), (scenes.hull_tumble_xml(), 16 * sms + 1, 16)):
        with CudaPhysics(xml, n) as p:
            assert p.phase_launch()["collide"][0] == lanes, n


def test_solver_switch_keeps_shapes_and_matches_a_model_compiled_for_it():
    """PGS's kernel is prepared when a handle turns to it, at creation or by
    pg_set_solver, in the shapes of the handle."""
    n = 300
    a = CudaPhysics(scenes.ant_xml(solver="PGS"), n)
    b = CudaPhysics(scenes.ant_xml(), n)
    b.set_launch(16, 8)
    a.set_launch(16, 8)
    b.set_solver(kind=1)
    assert a.phase_launch() == b.phase_launch()
    v = np.random.default_rng(1).normal(0, 1, (n, 14))
    for p in (a, b):
        p.set(Field.QVEL, range(n), v)
        p.step(range(n), 40)
    assert a.stats()["nrows"].any()
    for f in Field:
        np.testing.assert_array_equal(a.get(f, range(n)), b.get(f, range(n)))
    b.set_solver(kind=0)
    b.set_launch()
    assert b.step_lanes() == 4


@pytest.mark.parametrize("n", [1, 31, 33, 100])
def test_one_lane_columns_follow_every_parameter(n):
    """The one-lane kernel reads per-env parameters from columns written with
    the blocks: each parameter it uses, for a part of the envs, against a
    handle on the phase kernels."""
    m = mjcf.load_string(scenes.arm3d_xml())
    blob = mjcf.to_blob(m)
    a, b = CudaPhysics(blob, n), CudaPhysics(blob, n)
    b.set_launch(16, 4)
    assert (a.step_lanes(), b.step_lanes()) == (1, 0)
    rng = np.random.default_rng(n)
    q, v = _states(m, n, rng)
    ctrl = rng.uniform(-1, 1, (n, m.nu))
    base = None
    for pid, elem in ((None, 0), (Param.BODY_MASS, 2), (Param.BODY_INERTIA, m.nbody - 1), (Param.BODY_IPOS, 3),
                      (Param.DOF_DAMPING, 4), (Param.ACTUATOR_GAIN, 1), (Param.ACTUATOR_BIAS, 2), (Param.GEOM_SIZE, 1),
                      (Param.GEOM_FRICTION, 1), (Param.BODY_MASS, 1)):
        s0 = n // 3
        if pid is not None:
            w = a.param_width(pid)
            val = a.get_param(pid, elem, range(s0, n)) + rng.uniform(0.1, 0.5, (n - s0, w)) * (
                0.01 if pid in (Param.BODY_INERTIA, Param.BODY_IPOS) else 1.0)
            for p in (a, b):
                p.set_param(pid, elem, range(s0, n), val)
        for p in (a, b):
            p.set(Field.QPOS, range(n), q)
            p.set(Field.QVEL, range(n), v)
            p.set(Field.CTRL, range(n), ctrl)
            p.step(range(n), 1)
        qa, qb = a.get(Field.QACC, range(n)), b.get(Field.QACC, range(n))
        assert _rel(qa, qb) < TOL, pid
        if pid is None:
            base = qa
        else:
            np.testing.assert_array_equal(qa[:s0], base[:s0])
        if pid == Param.BODY_MASS:
            assert _rel(qa[s0:], base[s0:]) > 1e-4
