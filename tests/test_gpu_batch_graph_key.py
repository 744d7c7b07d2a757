"""A captured launch of the batched planner is replayed for the same settings only: solves of
one planner that differ in one setting each check their edges by their own."""
import numpy as np
import pytest

import oracle as O
from isaac_sim_ros2_humble_gb300 import _lib, api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

RES = 0.25


def _problems():
    m = W.serial_arm(51, dof=7, n_spheres=40, radius_range=(0.02, 0.03))
    env = W.random_env(52, 60, 10, 0, sphere_r=(0.02, 0.05), box_side=(0.02, 0.1), size=1.6)
    R, E, om = api.Robot(m), api.Env(env), O.OracleModel(m, env)
    q = m.sample_full(np.random.default_rng(3), 300)
    free = q[om.clearance(q) > 1e-3]
    return om, [(R, E, free[2 * k], free[2 * k + 1], k) for k in range(24)]


def _colliding_edges(om, out, rule, res):
    bad = solved = 0
    for r, path in out:
        if not r["solved"]:
            continue
        solved += 1
        ok, fh, _, _ = om.check_motions(path[:-1], path[1:], res, rule)
        for i in np.nonzero(~ok)[0]:
            states = om.edge_states(path[i], path[i + 1], res, rule)
            bad += bool(np.abs(om.clearance(states[fh[i]: fh[i] + 1])).max() > 1e-4)
    assert solved >= 12
    return bad


def test_step_rule_and_resolution():
    om, problems = _problems()
    bp = api.BatchPlanner(max_problems=32, max_nodes=8192, max_links=16, path_cap=2048)
    kw = dict(lanes_per_problem=8, range_=0.9, max_iters=3000)
    for rule, res in ((_lib.STEP_LINF, RES), (_lib.STEP_L2, RES), (_lib.STEP_LINF, RES / 8), (_lib.STEP_LINF, RES)):
        out = bp.solve(problems, use_graph=True, rule=rule, resolution=res, **kw)
        assert _colliding_edges(om, out, rule, res) == 0
    # what the L-infinity rule passes, the L2 rule does not: the solves above had to differ
    out = bp.solve(problems, use_graph=False, rule=_lib.STEP_LINF, resolution=RES, **kw)
    assert _colliding_edges(om, out, _lib.STEP_L2, RES) > 0
