"""Scenes in which some states touch and others do not, at what a distance field could get
wrong: obstacles far smaller than a cell, a grid one cell high, obstacles that reach out of the
region, cells that clamped queries read, a coarse grid.  Verdicts, first hits and costs equal those of the same
obstacles without a field, and they are not the empty scene's."""
import dataclasses

import numpy as np
import pytest

import oracle as O
from isaac_sim_ros2_humble_gb300 import api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

f = np.float32
ROBOT = dict(seed=62, dof=7, n_spheres=70)


def _robot():
    return W.serial_arm(**ROBOT)


def _scene(which):
    robot = _robot()
    c = W.sphere_centers_numpy(robot, robot.sample_full(np.random.default_rng(60), 400))   # [N, S, 3]
    none = W.Environment.empty()

    def rare(p):                        # of the points, those that the arm touches now and then
        d = np.linalg.norm(c[:, :, None] - p, axis=-1) - robot.sphere_r[None, :, None]
        share = (d.min(1) < 0.05).mean(0)
        return p[(share > 0.005) & (share < 0.06)].astype(f)

    at = rare(c[np.arange(60) * 6, 40 + np.arange(60) % 30])               # where a sphere of the arm has been
    assert len(at) >= 12
    at = at[:12]
    if which == "tiny spheres":
        return dataclasses.replace(none, sphere_pos=at, sphere_r=np.full(len(at), 1e-3, f))
    if which == "one tiny sphere":
        return dataclasses.replace(none, sphere_pos=at[:1], sphere_r=f([1e-3]))
    if which == "flat":                 # one cell high, at the height that the arm crosses most
        g = np.stack(np.meshgrid(np.linspace(-1, 1, 9), np.linspace(-1, 1, 9)), -1).reshape(-1, 2)
        p = rare(np.c_[g, np.full(len(g), np.median(c[:, 40:, 2]))])
        return dataclasses.replace(none, sphere_pos=p, sphere_r=np.full(len(p), 0.02, f))
    if which in ("a floor", "only a floor"):
        e = W.random_env(61, 12, 3, 2, oriented=True) if which == "a floor" else none
        top = np.quantile(c[:, :, 2].min(1), 0.3)                          # three states in ten reach below it
        return dataclasses.replace(e, box_pos=np.concatenate([e.box_pos, f([[0, 0, top - 5]])]),
                                   box_rot=np.concatenate([e.box_rot, np.eye(3, dtype=f)[None]]),
                                   box_min=np.concatenate([e.box_min, f([[-80, -80, -5]])]),
                                   box_max=np.concatenate([e.box_max, f([[80, 80, 5]])]))
    if which == "far cluster":          # the region is around it; what is near lies outside
        far = W.random_env(63, 60, 0, 0)
        return dataclasses.replace(none, sphere_pos=np.concatenate([far.sphere_pos + f(25), at[:4]]),
                                   sphere_r=np.concatenate([far.sphere_r, np.full(4, 0.03, f)]))
    if which == "coarse":               # six obstacles, 40 m apart: cells of more than a metre
        return dataclasses.replace(none, sphere_pos=np.concatenate([at[:3], f([[40, 0, 0], [0, 40, 0], [0, 0, 40]])]),
                                   sphere_r=np.full(6, 0.06, f))
    return W.random_env(61, 40, 10, 6, oriented=True)


def _without_field(env):
    """With an obstacle that touches nothing and leaves the scene without a field."""
    return dataclasses.replace(env, sphere_pos=np.concatenate([env.sphere_pos, np.full((1, 3), np.nan, f)]),
                               sphere_r=np.concatenate([env.sphere_r, f([0.1])]))


def _outputs(R, env, q):
    E = api.Env(env)
    n = q.shape[0]
    v, vc, ok = (torch.zeros(n, dtype=torch.uint8, device="cuda") for _ in range(3))
    total, costs = torch.zeros(n, device="cuda"), torch.zeros((4, n), device="cuda")
    fh = torch.zeros(n // 2, dtype=torch.int32, device="cuda")
    api.check_states(R, E, q, v)
    api.check_states(R, E, q, vc, costs, total, 1)
    api.check_edges(R, E, q[: n // 2].contiguous(), q[n // 2:].contiguous(), 0.05, 1, ok[: n // 2], fh)
    torch.cuda.synchronize()
    return [x.cpu().numpy() for x in (v, vc, costs, total, ok, fh)]


@pytest.mark.parametrize("which", ["mixed", "one tiny sphere", "tiny spheres", "flat", "a floor", "only a floor",
                                   "far cluster", "coarse"])
def test_contacts(which):
    robot, env = _robot(), _scene(which)
    R, m = api.Robot(robot), O.OracleModel(robot, env)
    q = robot.sample_full(np.random.default_rng(6), 4000)
    d = torch.from_numpy(q).cuda()
    got, want, empty = (_outputs(R, e, d) for e in (env, _without_field(env), W.Environment.empty()))
    for k in (0, 1, 4, 5):
        np.testing.assert_array_equal(got[k], want[k])
    for k in (2, 3):   # sums of the same terms, possibly in another order: a few roundings of the largest
        np.testing.assert_allclose(got[k], want[k], rtol=2e-5, atol=1e-6)
    cl = m.clearance(q[:1500])
    clear = np.abs(cl) > 1e-4
    np.testing.assert_array_equal(got[0][:1500].astype(bool)[clear], (cl < 0)[clear])
    scene = got[2][1:].sum(0)
    assert 0 < got[0].sum() < len(q) and (got[0] != empty[0]).any() and (got[5] != empty[5]).any()
    assert 5 <= (scene > 0).sum() < len(q) and (scene[empty[0] == 0] > 0).any()
