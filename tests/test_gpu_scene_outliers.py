"""State checks in scenes whose obstacles are not all in one place (floors, walls, obstacles
parked far away, obstacles without a usable position): the verdicts are the oracle's, and no
scene makes a check cost more than testing every obstacle against one bounding sphere a link
and the spheres of what is near, twice."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from isaac_sim_ros2_humble_gb300 import _lib, api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

f = np.float32


def _sphere(e, p, r=0.1):
    return dataclasses.replace(e, sphere_pos=np.concatenate([e.sphere_pos, f([p])]),
                               sphere_r=np.concatenate([e.sphere_r, f([r])]))


def _box(e, p, half):
    return dataclasses.replace(e, box_pos=np.concatenate([e.box_pos, f([p])]),
                               box_rot=np.concatenate([e.box_rot, np.eye(3, dtype=f)[None]]),
                               box_min=np.concatenate([e.box_min, -f([half])]),
                               box_max=np.concatenate([e.box_max, f([half])]))


def _scene(which):
    e = W.random_env(102, 256, 64, 16, oriented=True)
    if which == "a floor":
        return _box(e, (0, 0, -0.75), (10, 10, 0.05))
    if which == "a room":
        for a in range(3):
            for s in (-1, 1):
                p, half = np.zeros(3), np.full(3, 3.0)
                p[a], half[a] = 2.2 * s, 0.05
                e = _box(e, p, half)
        return e
    if which == "two places":     # three obstacles in four here, one in four 8 m away
        far = np.arange(256) % 4 == 0
        return dataclasses.replace(e, sphere_pos=e.sphere_pos + f(8) * far[:, None].astype(f))
    if which in ("a pile 4 m away", "a pile 30 m away"):   # one obstacle in ten by the robot
        here = np.arange(256) % 10 == 0
        far = f(float(which.split()[2])) * (~here)[:, None].astype(f) * f([1, 0, 0])
        return dataclasses.replace(e, sphere_pos=e.sphere_pos + far).subset(256, 0, 0)
    return e if which == "one place" else _sphere(e, {"20 m": (20, 20, 0), "1e4 m": (1e4, 0, 0), "1e9 m": (1e9, 0, 0),
                                                     "1e25 m": (0, -1e25, 0), "infinity": (-np.inf, 0, 0),
                                                     "no number": (np.nan, 0, 0)}[which])


def _check(R, E, q, cb=False):
    v = torch.full((q.shape[0],), 9, dtype=torch.uint8, device="cuda")
    if cb:
        api.CheckBatch(max_requests=1).run([dict(robot=R, env=E, q=q, verdict=v)])
    else:
        api.check_states(R, E, q, v)
    torch.cuda.synchronize()
    return v.cpu().numpy()


@pytest.mark.parametrize("which", ["one place", "a floor", "a room", "two places",
                                   "a pile 4 m away", "a pile 30 m away", "20 m", "1e4 m", "1e9 m", "1e25 m",
                                   "infinity", "no number"])
def test_verdicts_and_work(which):
    robot = W.serial_arm(2, dof=8, n_spheres=110, prismatic_torso=True)
    env = _scene(which)
    R, E, m = api.Robot(robot), api.Env(env), O.OracleModel(robot, env)
    n = 6000
    q = robot.sample_full(np.random.default_rng(9), n)
    d = torch.from_numpy(q).cuda()
    v = _check(R, E, d)
    for k in (1, 40):
        np.testing.assert_array_equal(_check(R, E, d[:k]), v[:k])
    np.testing.assert_array_equal(_check(R, E, d, cb=True), v)
    cl = m.clearance(q[:2000])
    clear = np.abs(cl) > 1e-4
    assert 0.1 < (cl < 0).mean() < 0.9
    np.testing.assert_array_equal(v[:2000].astype(bool)[clear], (cl < 0)[clear])
    vc, total = torch.full((n,), 9, dtype=torch.uint8, device="cuda"), torch.zeros(n, device="cuda")
    api.check_states(R, E, d, vc, None, total, _lib.CHECK_COST)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(vc.cpu().numpy()[:2000].astype(bool)[clear], (cl < 0)[clear])
    np.testing.assert_allclose(total.cpu().numpy()[:500], m.check_states(q[:500])[1], rtol=1e-4, atol=2e-5)

    def work(E):
        _lib.work_counting(True)
        try:
            _check(R, E, d)
            flops, states = _lib.work_read()
        finally:
            _lib.work_counting(False)
        assert states == n
        return flops / n

    ns, nb, nc = env.counts
    links = len(np.unique(robot.sphere_link))
    all_obstacles = links * (9 * ns + 33 * nb + 34 * nc)     # flops of one test of each kind
    assert work(E) <= work(api.Env(W.Environment.empty())) + 2 * all_obstacles


@pytest.mark.parametrize("obstacle", ["sphere", "cylinder"])
@pytest.mark.parametrize("far", [0.0, 9e17])
def test_states_that_are_no_numbers_near_one_obstacle(obstacle, far):
    """A cell of a field with one obstacle names one; a state that is no number meets it, and
    collides just where it is a cylinder, whose clamps drop the NaN."""
    robot = W.serial_arm(79, dof=7, n_spheres=40)
    e = W.Environment.empty()
    if obstacle == "sphere":
        e.sphere_pos, e.sphere_r = f([[0.4 + far, 0.2, 0.5]]), f([0.1])
    else:
        e.cyl_pos, e.cyl_rot = f([[0.4 + far, 0.2, 0.5]]), np.eye(3, dtype=f)[None]
        e.cyl_radius, e.cyl_height = f([0.1]), f([0.4])
    R, E = api.Robot(robot), api.Env(e)
    q = torch.from_numpy(robot.sample_full(np.random.default_rng(2), 65)).cuda()
    q[::2, 1] = float("nan")
    v, total = torch.full((65,), 9, dtype=torch.uint8, device="cuda"), torch.zeros(65, device="cuda")
    api.check_states(R, E, q, v, None, total, _lib.CHECK_COST)
    torch.cuda.synchronize()
    assert (v[::2] == (obstacle == "cylinder")).all()
    np.testing.assert_array_equal(_check(R, E, q)[::2], v.cpu().numpy()[::2])
