"""Projection and constrained motions where the joints do not fit one lane each, or few do:
against the oracle (the stable states' bar of one iteration, bit-exact limit pulls), and the
recorded states of a motion checked in groups: motions of fewer states than a group, and
feasibility that fails at any place in one."""
import numpy as np
import pytest

import oracle as O
from isaac_sim_ros2_humble_gb300 import api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _gpu(R, q, **kw):
    d = torch.from_numpy(np.ascontiguousarray(q)).cuda()
    tc, bc = torch.zeros(len(q), device="cuda"), torch.zeros(len(q), device="cuda")
    api.project_states(R, d, task_cost=tc, bound_cost=bc, **kw)
    torch.cuda.synchronize()
    return d.cpu().numpy(), tc.cpu().numpy(), bc.cpu().numpy()


@pytest.mark.parametrize("dof", [1, 3, 4, 7, 30, 31, 32, 45, 63])
@pytest.mark.parametrize("link", ["tip", "middle"])
def test_one_iteration(dof, link):
    robot = W.serial_arm(80 + dof, dof=dof, n_spheres=dof, offset_range=(0.02, 0.3 if dof < 20 else 0.08))
    R, m = api.Robot(robot), O.OracleModel(robot)
    at = robot.num_links - 1 if link == "tip" else max(1, robot.num_links // 2)
    q0 = robot.sample_full(np.random.default_rng(dof), 1)
    T = W.fk_numpy(robot, q0)[0][at]
    off = np.eye(4, dtype=np.float32)
    off[:3, :3] = T[:3, :3].T
    kw = dict(task_link=at, offset=off, reference=[*map(float, T[:3, 3]), 0.0, 0.0, 0.0],
              tolerance=(1e-3,) * 3 + (1e-2,) * 3, iterations=1)
    rng = np.random.default_rng(4)
    q = (q0 + 0.1 * rng.standard_normal((300, robot.num_links)) * robot.active).astype(np.float32)
    qg, tg, bg = _gpu(R, q, **kw)
    qo, to, bo = m.project(q, O.projection(**kw))
    act = robot.active.astype(bool)
    q_ulp = q.copy()
    q_ulp[:, act] = np.nextafter(q[:, act], np.float32(np.inf))
    qu, _, _ = m.project(q_ulp, O.projection(**kw))
    stable = np.abs(qu - qo).max(axis=1) < 1e-5
    assert stable.sum() > 20
    assert np.abs(qg[stable] - qo[stable]).max() < 1e-4
    np.testing.assert_array_equal(qg[:, ~act], q[:, ~act])
    kw = dict(task_link=-1, use_boundary=True, iterations=1)
    q[:, act] += rng.uniform(-3.0, 3.0, size=(300, act.sum())).astype(np.float32)
    got, want = _gpu(R, q, **kw), m.project(q, O.projection(**kw))
    np.testing.assert_array_equal(got[0], want[0])
    np.testing.assert_array_equal(got[2], want[2])


def test_groups_of_recorded_states():
    """With no task region every motion is the straight one, so the oracle's edge states say
    which recorded state collides first; start and goal a few to some dozen steps apart."""
    robot = W.serial_arm(1, dof=7, n_spheres=59)
    env = W.random_env(7, 24, 6, 3, oriented=True)
    R, E, m = api.Robot(robot), api.Env(env), O.OracleModel(robot, env)
    rng = np.random.default_rng(3)
    a = robot.sample_full(rng, 400) * np.float32(0.9)
    b = (a + rng.normal(size=a.shape).astype(np.float32) * rng.uniform(0.005, 0.3, (400, 1)).astype(np.float32)
         * robot.active).astype(np.float32)
    res = 0.02
    kw = dict(task_link=-1, use_boundary=True)
    ok = torch.zeros(400, dtype=torch.uint8, device="cuda")
    cnt = torch.zeros(400, dtype=torch.int32, device="cuda")
    st = torch.zeros((400, 128, robot.num_links), device="cuda")
    api.constrained_motions(R, E, torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), resolution=res, ok=ok,
                            num_states=cnt, states=st, **kw)
    torch.cuda.synchronize()
    o_ok, _, o_cnt, o_st = m.constrained_motions(a, b, O.projection(iterations=2, **kw), res, cap=128)
    ok, cnt, st = ok.cpu().numpy().astype(bool), cnt.cpu().numpy(), st.cpu().numpy()
    np.testing.assert_array_equal(cnt, o_cnt)
    assert cnt.min() < 8 < cnt.max() and 40 < ok.sum() < 360
    for k in np.nonzero(ok != o_ok)[0]:   # only where a recorded state lies at the surface
        assert np.any(np.abs(m.clearance(st[k, : cnt[k]])) <= 1e-4), k
