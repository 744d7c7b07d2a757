"""Which form a one-problem plan takes: its edge checks by chunks of states where their scratch
fits next to the scene, else state by state; and that paths of both are free."""
import numpy as np
import pytest

import oracle as O
from isaac_sim_ros2_humble_gb300 import _lib, api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _kernels(call):
    """Names of the kernels a call launches (a process's first recording stays empty)."""
    from torch.profiler import ProfilerActivity, profile
    for _ in range(2):
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            call()
            torch.cuda.synchronize()
    return [e.key for e in p.key_averages()]


# Shared memory in bytes of 232,432: by chunks 207,136 and 210,944 (of 233,536 if a state's
# scratch stood beside a chunk's); 246,000 of which a state's form needs 220,336.
@pytest.mark.parametrize("dof,n_spheres,obstacles,chunks", [(8, 120, 5000, True), (8, 250, 5000, True),
                                                            (25, 60, 5300, False)])
@pytest.mark.parametrize("lanes", [1, 64])
def test_forms(dof, n_spheres, obstacles, chunks, lanes):
    m = W.serial_arm(93, dof=dof, n_spheres=n_spheres, offset_range=(0.02, 0.3 if dof < 20 else 0.06),
                     radius_range=(0.01, 0.03))
    env = W.random_env(94, obstacles, 0, 0, size=12.0 if dof < 20 else 16.0, sphere_r=(0.02, 0.06))
    R, E, om = api.Robot(m), api.Env(env), O.OracleModel(m, env)
    q = m.sample_full(np.random.default_rng(5), 600)
    free = q[om.clearance(q) > 1e-3]
    # to a state a quarter of the way to another: problems that one lane solves too
    goals = (free[:-1] + 0.25 * (free[1:] - free[:-1])).astype(np.float32)
    pairs = [(a, b) for a, b, c in zip(free, goals, om.clearance(goals)) if c > 1e-3][:10]
    planner = api.Planner(R, max_nodes=20000, path_cap=2048)

    def plan(k):
        return planner.solve(E, *pairs[k], lanes=lanes, max_iters=2000, range_=0.6, resolution=0.03, rule=_lib.STEP_LINF,
                             seed=k)

    names = _kernels(lambda: plan(0))
    assert any("k_rrtc" in n for n in names), names
    assert any("k_rrtc_chunk" in n for n in names) == chunks, names
    solved = 0
    for k in range(len(pairs)):
        res, path = plan(k)
        if not res["solved"]:
            continue
        solved += 1
        ok, fh, _, _ = om.check_motions(path[:-1], path[1:], 0.03, _lib.STEP_LINF)
        for i in np.nonzero(~ok)[0]:
            states = om.edge_states(path[i], path[i + 1], 0.03, _lib.STEP_LINF)
            assert np.abs(om.clearance(states[fh[i]: fh[i] + 1])).max() <= 1e-4
    assert solved


@pytest.mark.parametrize("lanes", [457, 700])
@pytest.mark.parametrize("max_iters", [60, 2048, 100000])
def test_lanes_that_join_late(lanes, max_iters):
    """More lanes than start at once: a path as soon as there is one, all lanes' iterations where
    there is none, and an end at the deadline."""
    m = W.serial_arm(1, dof=7, n_spheres=59)
    env = W.shelf_env(4)
    R, E, om = api.Robot(m), api.Env(env), O.OracleModel(m, env)
    q = m.sample_full(np.random.default_rng(5), 200)
    free = q[om.clearance(q) > 1e-3]
    planner = api.Planner(R, max_nodes=60000, path_cap=2048)
    kw = dict(lanes=lanes, max_iters=max_iters, range_=0.3, resolution=0.02, rule=_lib.STEP_LINF)
    for k in range(6):
        res, path = planner.solve(E, free[2 * k], free[2 * k + 1], seed=k, **kw)
        assert res["solved"]
        ok, fh, _, _ = om.check_motions(path[:-1], path[1:], 0.02, _lib.STEP_LINF)
        for i in np.nonzero(~ok)[0]:
            states = om.edge_states(path[i], path[i + 1], 0.02, _lib.STEP_LINF)
            assert np.abs(om.clearance(states[fh[i]: fh[i] + 1])).max() <= 1e-4
    # hardly a way out where a shell of obstacles surrounds the tip: a cap or the deadline may end it
    c = W.sphere_centers_numpy(m, free[:1])[0]
    pts = c[-1] + 0.25 * np.asarray([W._unit(np.random.default_rng(k)) for k in range(400)])
    pts = pts[(np.linalg.norm(pts[:, None] - c, axis=-1) - m.sphere_r > 0.045).all(1)].astype(np.float32)
    shell = W.Environment.empty()
    shell.sphere_pos, shell.sphere_r = pts, np.full(len(pts), 0.04, np.float32)
    res, _ = planner.solve(api.Env(shell), free[0], free[1], seed=1, time_limit_s=0.5, **kw)
    assert res["solved"] or res["status"] in (2, 3, 4)
    if res["status"] == 3:
        assert res["iterations"] == max_iters
