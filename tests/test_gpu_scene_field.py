"""The scene's distance field only spares tests: verdicts, first hits and costs equal those
of the same obstacles in a scene without a field (one that holds an obstacle at a position
that is not a number, which touches nothing), where the field is coarse, absent, or far
from the robot."""
import dataclasses

import numpy as np
import pytest

from isaac_sim_ros2_humble_gb300 import api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _without_field(env):
    nan = np.full((1, 3), np.nan, np.float32)
    return dataclasses.replace(env, sphere_pos=np.concatenate([env.sphere_pos, nan]),
                               sphere_r=np.concatenate([env.sphere_r, np.float32([0.1])]))


def _outputs(R, env, q):
    E = api.Env(env)
    n = q.shape[0]
    v, ok = (torch.zeros(n, dtype=torch.uint8, device="cuda") for _ in range(2))
    api.check_states(R, E, q, v)
    total = torch.zeros(n, device="cuda")
    costs = torch.zeros((4, n), device="cuda")
    vc = torch.zeros(n, dtype=torch.uint8, device="cuda")
    api.check_states(R, E, q, vc, costs, total, 1)
    fh = torch.zeros(n // 2, dtype=torch.int32, device="cuda")
    api.check_edges(R, E, q[: n // 2].contiguous(), q[n // 2:].contiguous(), 0.05, 1, ok[: n // 2], fh)
    torch.cuda.synchronize()
    return [x.cpu().numpy() for x in (v, vc, costs, total, ok, fh)]


def _scene(which):
    e = W.random_env(61, 40, 10, 6, oriented=True)
    f = np.float32
    if which == "one tiny sphere":
        return dataclasses.replace(W.Environment.empty(), sphere_pos=f([[0.5, 0.1, 0.6]]), sphere_r=f([1e-3]))
    if which == "a floor":          # far larger than the field's obstacles
        return dataclasses.replace(e, box_pos=np.concatenate([e.box_pos, f([[0, 0, -5.05]])]),
                                   box_rot=np.concatenate([e.box_rot, np.eye(3, dtype=f)[None]]),
                                   box_min=np.concatenate([e.box_min, f([[-80, -80, -5]])]),
                                   box_max=np.concatenate([e.box_max, f([[80, 80, 5]])]))
    if which == "only a floor":
        return dataclasses.replace(W.Environment.empty(), box_pos=f([[0, 0, -5.0]]), box_rot=np.eye(3, dtype=f)[None],
                                   box_min=f([[-80, -80, -5]]), box_max=f([[80, 80, 5]]))
    if which == "flat":             # one cell high
        return dataclasses.replace(e, sphere_pos=e.sphere_pos * f([4, 4, 1e-4]) + f([0, 0, 0.8]),
                                   sphere_r=e.sphere_r * f(0.2)).subset(40, 0, 0)
    if which == "far away":
        return dataclasses.replace(e, sphere_pos=e.sphere_pos + f(30)).subset(40, 0, 0)
    return e


@pytest.mark.parametrize("which", ["mixed", "one tiny sphere", "a floor", "only a floor", "flat", "far away"])
def test_field_changes_no_output(which):
    robot = W.serial_arm(62, dof=7, n_spheres=70)
    R = api.Robot(robot)
    q = torch.from_numpy(robot.sample_full(np.random.default_rng(6), 4000)).cuda()
    env = _scene(which)
    got, want = _outputs(R, env, q), _outputs(R, _without_field(env), q)
    for k in (0, 1, 4, 5):
        np.testing.assert_array_equal(got[k], want[k])
    # sums of the same terms, possibly in another order: a few roundings of the largest
    for k in (2, 3):
        np.testing.assert_allclose(got[k], want[k], rtol=2e-5, atol=1e-6)
    if which == "mixed":
        assert 0 < got[0].sum() < len(got[0])
