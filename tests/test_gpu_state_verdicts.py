"""Verdicts of many states by one warp, against the oracle and against the same states one
call each: counts that fill the warps' share unevenly, robots and scenes at the limits of
the launch shapes, outputs at unaligned addresses."""
import numpy as np
import pytest

import oracle as O
from isaac_sim_ros2_humble_gb300 import _lib, api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _check(R, E, q, poses=None, centers=None):
    v = torch.full((q.shape[0],), 9, dtype=torch.uint8, device="cuda")
    api.check_states(R, E, q, v, poses=poses, centers=centers)
    torch.cuda.synchronize()
    return v.cpu().numpy()


def _parity(m, q, v):
    cl = m.clearance(q)
    clear = np.abs(cl) > 1e-4
    np.testing.assert_array_equal(v.astype(bool)[clear], (cl < 0)[clear])


@pytest.mark.parametrize("n", [1, 2, 151, 153, 1217, 3649, 7297, 30001])
def test_counts(n):
    robot = W.serial_arm(71, dof=7, n_spheres=61)
    env = W.random_env(72, 50, 9, 5, oriented=True)
    R, E = api.Robot(robot), api.Env(env)
    q = robot.sample_full(np.random.default_rng(n), n)
    d = torch.from_numpy(q).cuda()
    L, S = robot.num_links, robot.num_spheres
    buf = torch.full((n * L * 16 + 1,), 5.0, device="cuda")
    cen = torch.zeros((n, S, 3), device="cuda")
    v = _check(R, E, d, poses=buf[1:], centers=cen)      # 4 bytes off a 16-byte boundary
    pick = np.arange(n) if n < 4000 else np.random.default_rng(0).choice(n, 4000, replace=False)
    _parity(O.OracleModel(robot, env), q[pick], v[pick])
    np.testing.assert_array_equal(_check(R, E, d), v)
    ref_p, ref_c = torch.zeros((n, L, 16), device="cuda"), torch.zeros((n, S, 3), device="cuda")
    api.fk(R, d, ref_p, ref_c)
    torch.cuda.synchronize()
    assert torch.equal(buf[1:].view(n, L, 16), ref_p) and torch.equal(cen, ref_c) and buf[0].item() == 5.0
    few = d[: min(n, 40)]
    np.testing.assert_array_equal([_check(R, E, few[k: k + 1])[0] for k in range(len(few))], v[: len(few)])


@pytest.mark.parametrize("dof,n_spheres,obstacles", [(2, 1, 1), (40, 200, 60), (63, 250, 300), (8, 256, 4300)])
def test_robots_and_scenes_at_the_limits(dof, n_spheres, obstacles):
    """One sphere; more than 32 sphere groups; 64 links; a scene of 170 KB next to which
    only small launch shapes fit."""
    robot = W.serial_arm(73 + dof, dof=dof, n_spheres=n_spheres, offset_range=(0.02, 0.3 if dof < 20 else 0.06),
                         radius_range=(0.01, 0.03))
    env = W.random_env(74, obstacles, 0, 0, size=1.2 if obstacles < 1000 else 5.0,
                       sphere_r=(0.05, 0.15) if obstacles < 1000 else (0.02, 0.05))
    R, E = api.Robot(robot), api.Env(env)
    q = robot.sample_full(np.random.default_rng(1), 700)
    v = _check(R, E, torch.from_numpy(q).cuda())
    _parity(O.OracleModel(robot, env), q, v)


def test_a_scene_too_large_for_the_robot_is_refused():
    robot = W.serial_arm(75, dof=60, n_spheres=256)
    env = W.random_env(76, 5300, 0, 0, size=9.0)
    R, E = api.Robot(robot), api.Env(env)
    q = torch.from_numpy(robot.sample_full(np.random.default_rng(1), 4)).cuda()
    with pytest.raises(_lib.GbmpError) as e:
        _check(R, E, q)
    assert e.value.status == 5


@pytest.mark.parametrize("n", [1, 33, 700, 60000])
def test_costs(n):
    """Costs against the oracle (a sample), and the same to the bit whatever states go
    with a state: alone, in a batch request, or among many."""
    robot = W.serial_arm(77, dof=8, n_spheres=90, prismatic_torso=True)
    env = W.random_env(78, 150, 40, 12, oriented=True)
    R, E, m = api.Robot(robot), api.Env(env), O.OracleModel(robot, env)
    q = robot.sample_full(np.random.default_rng(n), n)
    d = torch.from_numpy(q).cuda()
    costs, total = torch.full((4, n), -1.0, device="cuda"), torch.full((n,), -1.0, device="cuda")
    v = torch.full((n,), 9, dtype=torch.uint8, device="cuda")
    api.check_states(R, E, d, v, costs, total, _lib.CHECK_COST)
    pick = np.arange(n) if n <= 700 else np.random.default_rng(0).choice(n, 700, replace=False)
    oc, ot = m.check_states(q[pick])
    c, tt, vv = costs.cpu().numpy(), total.cpu().numpy(), v.cpu().numpy()
    np.testing.assert_allclose(c[:, pick], oc, rtol=1e-4, atol=2e-5)
    np.testing.assert_allclose(tt[pick], ot, rtol=1e-4, atol=2e-5)
    np.testing.assert_array_equal(vv, tt != 0)
    if n >= 700:
        assert 0 < vv.sum() < n and all((c[k] > 0).any() for k in range(4))
    at = min(n - 1, 5)
    one, t1 = torch.zeros((4, 1), device="cuda"), torch.zeros(1, device="cuda")
    api.check_states(R, E, d[at: at + 1].contiguous(), None, one, t1, _lib.CHECK_COST)
    torch.cuda.synchronize()
    assert torch.equal(one[:, 0], costs[:, at]) and torch.equal(t1[0], total[at])
    cb = api.CheckBatch(max_requests=3)
    few = d[: min(n, 301)].contiguous()
    bc, bt = torch.zeros((4, len(few)), device="cuda"), torch.zeros(len(few), device="cuda")
    cb.run([dict(robot=R, env=E, q=d[:1].contiguous()), dict(robot=R, env=E, q=few, costs=bc, total=bt)], mode=_lib.CHECK_COST)
    torch.cuda.synchronize()
    assert torch.equal(bc, costs[:, : len(few)]) and torch.equal(bt, total[: len(few)])


@pytest.mark.parametrize("cylinders", [0, 3])
def test_states_that_are_no_numbers(cylinders):
    """A state with a joint that is not a number: every distance comparison is false but a
    cylinder's, whose clamps drop the NaN, so it collides just where there are cylinders."""
    robot = W.serial_arm(79, dof=7, n_spheres=40)
    R, E = api.Robot(robot), api.Env(W.random_env(80, 40, 8, cylinders, oriented=True))
    q = torch.from_numpy(robot.sample_full(np.random.default_rng(2), 65)).cuda()
    q[::2, 1] = float("nan")
    v, total = torch.full((65,), 9, dtype=torch.uint8, device="cuda"), torch.zeros(65, device="cuda")
    api.check_states(R, E, q, v, None, total, _lib.CHECK_COST)
    torch.cuda.synchronize()
    assert (v[::2] == (1 if cylinders else 0)).all()
    np.testing.assert_array_equal(_check(R, E, q)[::2], v.cpu().numpy()[::2])
