"""One-problem planning with the edge checks by chunks and, for robots of more than 32 sphere
groups and scenes next to which the chunk scratch does not fit, state by state."""
import numpy as np
import pytest

from isaac_sim_ros2_humble_gb300 import _lib, api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [1, 64])
@pytest.mark.parametrize("dof,n_spheres,obstacles,size", [(6, 40, 60, 2.5), (8, 120, 4600, 12.0), (38, 80, 40, 12.0)])
def test_paths(dof, n_spheres, obstacles, size, lanes):
    """A path's edges are free under the rule that made it, and one lane gives the same path
    each time."""
    m = W.serial_arm(93, dof=dof, n_spheres=n_spheres, offset_range=(0.02, 0.3 if dof < 20 else 0.06),
                     radius_range=(0.01, 0.03))
    R = api.Robot(m)
    E = api.Env(W.random_env(94, obstacles, 0, 0, size=size, sphere_r=(0.02, 0.06)))
    q = torch.from_numpy(m.sample_full(np.random.default_rng(5), 4000)).cuda()
    v = torch.zeros(4000, dtype=torch.uint8, device="cuda")
    api.check_states(R, E, q, v)
    free = q[v == 0].cpu().numpy()
    assert len(free) >= 6
    planner = api.Planner(R, max_nodes=20000, path_cap=2048)
    solved = 0
    for k in range(3):
        def plan():
            return planner.solve(E, free[2 * k], free[2 * k + 1], lanes=lanes, max_iters=400, range_=0.6,
                                 resolution=0.03, rule=_lib.STEP_LINF, seed=k)
        res, path = plan()
        if lanes == 1:
            again, path2 = plan()
            assert again["iterations"] == res["iterations"] and np.array_equal(path, path2)
        if not res["solved"]:
            continue
        solved += 1
        p = torch.from_numpy(np.ascontiguousarray(path)).cuda()
        ok = torch.zeros(len(path) - 1, dtype=torch.uint8, device="cuda")
        api.check_edges(R, E, p[:-1].contiguous(), p[1:].contiguous(), 0.03, _lib.STEP_LINF, ok)
        torch.cuda.synchronize()
        assert ok.all()
    if lanes > 1:
        assert solved
