"""Planners of several threads next to each other: small scenes and one that needs nearly all
shared memory, so that the threads want different limits of one kernel."""
import threading

import numpy as np
import pytest

import oracle as O
from isaac_sim_ros2_humble_gb300 import _lib, api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batched", [False, True])
def test_scenes_of_different_sizes(batched):
    m = W.serial_arm(1, dof=7, n_spheres=59)
    R = api.Robot(m)
    jobs = []
    for obstacles, size in ((20, 4.0), (1500, 14.0), (4500, 20.0)):
        env = W.random_env(5, obstacles, 0, 0, size=size, sphere_r=(0.02, 0.06))
        q = m.sample_full(np.random.default_rng(2), 200)
        free = q[O.OracleModel(m, env).clearance(q) > 1e-3]
        E = api.Env(env)
        if batched:
            planner = api.BatchPlanner(max_problems=4, max_nodes=4096, max_links=16, path_cap=512)
        else:
            planner = api.Planner(R, max_nodes=4096, path_cap=512)
        jobs.append((E, free, planner))
    failures, solved = [], [0] * len(jobs)

    def work(i):
        E, free, planner = jobs[i]
        stream = torch.cuda.Stream()
        kw = dict(range_=0.8, resolution=0.05, rule=_lib.STEP_LINF, max_iters=200, time_limit_s=1.0, stream=stream)
        for k in range(60):
            a, b = free[k % 20], free[k % 20 + 20]
            try:
                if batched:
                    out = planner.solve([(R, E, a, b, k), (R, E, b, a, k)], lanes_per_problem=4, use_graph=k % 2 == 0, **kw)
                    solved[i] += sum(r["solved"] for r, _ in out)
                else:
                    solved[i] += planner.solve(E, a, b, lanes=8, seed=k, **kw)[0]["solved"]
            except _lib.GbmpError as e:
                failures.append((i, k, str(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
    assert min(solved) >= 10
