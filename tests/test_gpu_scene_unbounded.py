"""Obstacles that their bounding spheres do not bound: half-spaces (boxes with infinite
extents) and matrices that scale.  State checks and plans of one problem test them by the per-pair formulas."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from isaac_sim_ros2_humble_gb300 import _lib, api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _scene(which):
    f = np.float32
    e = W.random_env(81, 40, 6, 3, oriented=True)
    inf = np.inf
    if which == "half-space":            # a wall at y = 0.7, one of many boxes
        return dataclasses.replace(e, box_pos=np.concatenate([e.box_pos, f([[0, 0.7, 0]])]),
                                   box_rot=np.concatenate([e.box_rot, np.eye(3, dtype=f)[None]]),
                                   box_min=np.concatenate([e.box_min, f([[-inf, 0, -inf]])]),
                                   box_max=np.concatenate([e.box_max, f([[inf, inf, inf]])]))
    if which == "only a half-space":
        return dataclasses.replace(W.Environment.empty(), box_pos=f([[0, 0.7, 0]]), box_rot=np.eye(3, dtype=f)[None],
                                   box_min=f([[-inf, 0, -inf]]), box_max=f([[inf, inf, inf]]))
    if which == "scaled boxes":
        return dataclasses.replace(e, box_rot=f(0.4) * e.box_rot)
    if which == "scaled cylinders":
        return dataclasses.replace(e, cyl_rot=f(0.4) * e.cyl_rot)
    # nearly orthonormal: its spheres bound it to a fraction of a millimetre
    return dataclasses.replace(e, box_rot=f(1 - 2e-5) * e.box_rot, cyl_rot=f(1 + 2e-5) * e.cyl_rot)


@pytest.mark.parametrize("which", ["half-space", "only a half-space", "scaled boxes", "scaled cylinders", "nearly"])
def test_against_the_oracle(which):
    robot = W.serial_arm(82, dof=7, n_spheres=70)
    env = _scene(which)
    R, E, m = api.Robot(robot), api.Env(env), O.OracleModel(robot, env)
    n = 3000
    q = robot.sample_full(np.random.default_rng(7), n)
    d = torch.from_numpy(q).cuda()
    v, vc = (torch.full((n,), 9, dtype=torch.uint8, device="cuda") for _ in range(2))
    costs, total = torch.zeros((4, n), device="cuda"), torch.zeros(n, device="cuda")
    api.check_states(R, E, d, v)
    api.check_states(R, E, d, vc, costs, total, _lib.CHECK_COST)
    torch.cuda.synchronize()
    cl = m.clearance(q)
    clear = np.abs(cl) > 1e-4
    assert 0.1 < (cl < 0).mean() < 0.95
    for got in (v, vc):
        np.testing.assert_array_equal(got.cpu().numpy().astype(bool)[clear], (cl < 0)[clear])
    oc, ot = m.check_states(q)
    np.testing.assert_allclose(costs.cpu().numpy(), oc, rtol=1e-4, atol=2e-5)
    np.testing.assert_allclose(total.cpu().numpy(), ot, rtol=1e-4, atol=2e-5)


@pytest.mark.parametrize("which", ["half-space", "scaled boxes"])
def test_plans_against_the_oracle(which):
    robot = W.serial_arm(82, dof=7, n_spheres=70)
    env = _scene(which)
    R, E, m = api.Robot(robot), api.Env(env), O.OracleModel(robot, env)
    q = robot.sample_full(np.random.default_rng(8), 400)
    free = q[m.clearance(q) > 1e-3]
    planner = api.Planner(R, max_nodes=20000, path_cap=2048)
    solved = 0
    for k in range(12):
        res, path = planner.solve(E, free[2 * k], free[2 * k + 1], lanes=32, max_iters=400, range_=0.6, resolution=0.02,
                                  rule=_lib.STEP_LINF, seed=k)
        if not res["solved"]:
            continue
        solved += 1
        ok, fh, _, _ = m.check_motions(path[:-1], path[1:], 0.02, _lib.STEP_LINF)
        for i in np.nonzero(~ok)[0]:
            states = m.edge_states(path[i], path[i + 1], 0.02, _lib.STEP_LINF)
            assert np.abs(m.clearance(states[fh[i]: fh[i] + 1])).max() <= 1e-4
    assert solved >= 4


def _with_sphere(env, p):
    return dataclasses.replace(env, sphere_pos=np.concatenate([env.sphere_pos, np.float32([p])]),
                               sphere_r=np.concatenate([env.sphere_r, np.float32([0.1])]))


@pytest.mark.parametrize("form", [0, 1, 4])
@pytest.mark.parametrize("which", ["half-space", "scaled boxes", "scaled cylinders", "nearly", "-infinity", "-1e20 m"])
def test_edges_against_the_oracle(which, form):
    robot = W.serial_arm(82, dof=7, n_spheres=70)
    env = _scene(which)
    if which[0] == "-":
        env = _with_sphere(W.random_env(81, 90, 6, 3, oriented=True), (float(which.split()[0].replace("inity", "")), 0, 0))
    R, E, m = api.Robot(robot), api.Env(env), O.OracleModel(robot, env)
    n = 300
    q = robot.sample_full(np.random.default_rng(11), 2 * n)
    a, b = q[:n], (q[:n] + 0.3 * (q[n:] - q[:n])).astype(np.float32)
    ok, okv = (torch.full((n,), 9, dtype=torch.uint8, device="cuda") for _ in range(2))
    fh = torch.full((n,), -9, dtype=torch.int32, device="cuda")
    R.set_edge_form(form)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    api.check_edges(R, E, da, db, 0.05, _lib.STEP_LINF, ok, fh)
    api.check_edges(R, E, da, db, 0.05, _lib.STEP_LINF, okv)
    torch.cuda.synchronize()
    assert torch.equal(ok, okv)
    o_ok, o_fh, _, _ = m.check_motions(a, b, 0.05, _lib.STEP_LINF)
    assert 0.1 < o_ok.mean() < 0.9
    fh = fh.cpu().numpy()
    for k in np.nonzero(fh != o_fh)[0]:     # a state at the surface decided otherwise
        s = [x for x in (fh[k], o_fh[k]) if x >= 0]
        assert np.abs(m.clearance(m.edge_states(a[k], b[k], 0.05, _lib.STEP_LINF)[min(s): min(s) + 1]))[0] <= 1e-4
