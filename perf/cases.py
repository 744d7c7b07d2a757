"""Workloads of the motion-planning library, as a user's program runs them through the
Python handles: batched state checks, edge validation, forward kinematics, nearest
neighbours, projection onto a constraint, constrained motions, one round of a roadmap
planner and one reproducible plan.

Sizes are those of the benchmark configurations, of the tests and of the roadmap planner's
defaults, and what lies between them.  A case names its robot (`robot`, `dof`, `spheres`,
`robot_seed`) and its scene (`obstacles`, `scene_seed`); the joint values come from the seed
of prepare().  Plans of many lanes are left out: which lane connects first depends on timing,
so two runs on the same inputs return different paths.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from isaac_sim_ros2_humble_gb300 import _lib, api
from isaac_sim_ros2_humble_gb300 import workloads as W


def listed():
    bench_arm = dict(robot="arm", dof=8, spheres=110, robot_seed=2, scene="mixed", obstacles=336, scene_seed=102)
    small_arm = dict(robot="arm", dof=7, spheres=59, robot_seed=1)
    return [
        # One iteration of the roadmap planner with its defaults (30 samples): sample, nearest,
        # steer, check the states with costs, nearest vertices, validate the motions.  The
        # smallest calls: latency and launches.
        dict(name="rrg_round_30", kind="round", n=30, tree=3000, resolution=0.02, rule="l2", **small_arm,
             scene="shelf", obstacles=45, scene_seed=3),
        # A planner's handful of candidate motions, validated before anything else can go on.
        dict(name="edges_64", kind="edges", n=64, resolution=0.01, rule="linf", first_hit=False, **bench_arm),
        # The benchmark's batch of edges: verdict and length of each.
        dict(name="edges_65536", kind="edges", n=65536, resolution=0.01, rule="linf", first_hit=False, **bench_arm),
        # A mobile manipulator (30 links, most of them fixed, branching) under the reference's
        # step rule, with each edge's first colliding state: where a path has to be repaired.
        dict(name="edges_first_hit_mobile_3001", kind="edges", n=3001, resolution=0.02, rule="l2", first_hit=True,
             robot="mobile", dof=8, spheres=110, robot_seed=5, scene="mixed", obstacles=120, scene_seed=31),
        # Plain FK + collision: flags and link poses of 4,096 configurations.
        dict(name="states_plain_4096", kind="states", n=4096, mode="verdict", poses=True, **small_arm, scene="boxes",
             obstacles=40, scene_seed=101),
        # checkStates as the reference has it: the cost of every constraint.  An odd count.
        dict(name="states_cost_20011", kind="states", n=20011, mode="cost", poses=False, **bench_arm),
        # What a request server sends in one go: 256 uneven requests over 4 robots and 16 scenes.
        dict(name="check_batch_256", kind="batch", n=256, largest=65536, mix_seed=17),
        # Forward kinematics alone, poses and sphere centres: a data-set or a reachability map.
        dict(name="fk_1048576", kind="fk", n=1 << 20, centers=True, robot="arm", dof=8, spheres=110, robot_seed=2),
        # Nearest vertices of a batch of samples in a grown tree.
        dict(name="nearest_1000_in_100000", kind="nearest", n=1000, tree=100000, share=1.0, **small_arm),
        # Projection of states a step away from a task-space region back onto it, the
        # reference's 10 rounds.
        dict(name="project_4096", kind="project", n=4096, iterations=10, spread=0.02, **small_arm),
        # Motions that hold the tip at a height: the constrained form of edge validation.
        dict(name="constrained_200", kind="constrained", n=200, resolution=0.02, **small_arm, scene="mixed",
             obstacles=33, scene_seed=7),
        # A plan of one lane (the form whose result does not depend on timing) in the shelf.
        dict(name="plan_one_lane", kind="plan", resolution=0.02, **small_arm, scene="shelf", obstacles=45,
             scene_seed=3),
    ]


def draw(rng):
    kind = rng.choice(["round", "edges", "edges", "edges", "states", "states", "batch", "fk", "nearest", "project",
                       "constrained"])

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def arm():
        if kind in ("edges", "states", "fk") and rng.random() < 0.25:
            return dict(robot="mobile", dof=8, spheres=rng.randint(60, 120), robot_seed=rng.randint(1, 9))
        return dict(robot="arm", dof=rng.randint(6, 9), spheres=rng.randint(30, 120), robot_seed=rng.randint(1, 40))

    def scene():
        which = rng.choice(["mixed", "mixed", "boxes", "shelf"])
        return dict(scene=which, obstacles=45 if which == "shelf" else rng.randint(10, 336),
                    scene_seed=rng.randint(1, 200))

    step = dict(resolution=rng.choice([0.01, 0.02, 0.05]), rule=rng.choice(["l2", "linf"]))
    if kind == "round":
        return dict(kind=kind, n=size(10, 1000), tree=size(100, 30000), **step, **arm(), **scene())
    if kind == "edges":
        if step["rule"] == "l2":
            step["resolution"] = max(step["resolution"], 0.02)   # about as many states as 0.01 per joint
        return dict(kind=kind, n=size(16, 50000), first_hit=rng.random() < 0.3, **step, **arm(), **scene())
    if kind == "states":
        mode = rng.choice(["verdict", "verdict", "cost"])
        return dict(kind=kind, n=size(1, 100000 if mode == "verdict" else 20000), mode=mode,
                    poses=rng.random() < 0.3, **arm(), **scene())
    if kind == "batch":
        return dict(kind=kind, n=size(2, 256), largest=size(1000, 65536), mix_seed=rng.randint(1, 1000))
    if kind == "fk":
        return dict(kind=kind, n=size(100, 300000), centers=rng.random() < 0.7, **arm())
    if kind == "nearest":
        return dict(kind=kind, n=size(1, 4000), tree=size(300, 200000), share=rng.choice([1.0, 1.0, 0.4]), **arm())
    if kind == "project":
        return dict(kind=kind, n=size(30, 8192), iterations=rng.choice([2, 10]), spread=rng.choice([0.02, 0.02, 0.15]),
                    **arm())
    return dict(kind=kind, n=size(10, 300), resolution=rng.choice([0.02, 0.05]), **arm(), scene="mixed",
                obstacles=rng.randint(10, 40), scene_seed=rng.randint(1, 200))


# ---- robots and scenes (host tables; a program reads them from its files once) ----------

def _mobile(seed, n_spheres):
    """A mobile manipulator as robot descriptions have it: 30 links, a lift, a 7-joint arm,
    a pan / tilt head and a gripper that the planner leaves alone, and fixed frames."""
    rng = np.random.default_rng(seed)
    parent, types, active = [-1], [W.FIXED], [0]

    def link(par, ty, act=0):
        parent.append(par)
        types.append(ty)
        active.append(act)
        return len(parent) - 1

    for _ in range(3):
        link(0, W.FIXED)                                   # sensor frames of the base
    for _ in range(2):
        link(0, W.REVOLUTE)                                # wheels
    lift = link(0, W.PRISMATIC, 1)
    link(lift, W.FIXED)
    pan = link(lift, W.REVOLUTE)
    tilt = link(pan, W.REVOLUTE)
    for _ in range(6):
        link(tilt, W.FIXED)                                # camera frames
    arm, last = [], lift
    for _ in range(7):
        last = link(last, W.REVOLUTE, 1)
        arm.append(last)
    wrist = link(last, W.FIXED)
    fingers = [link(wrist, W.PRISMATIC) for _ in range(2)]
    while len(parent) < 30:
        link(wrist, W.FIXED)
    L = len(parent)
    poses = np.tile(np.eye(4), (L, 1, 1))
    axes = np.zeros((L, 3))
    axes[:, 2] = 1.0
    for i in range(1, L):
        length = rng.uniform(0.1, 0.3) if i in arm else rng.uniform(0.02, 0.12)
        poses[i, :3, 3] = W._unit(rng) * length
        if types[i] != W.FIXED and i != lift:
            poses[i, :3, :3] = W._random_rotation(rng)
    poses[lift, :3, 3] = (0.0, 0.0, 0.35)
    lower, upper = np.full(L, -2.8, np.float32), np.full(L, 2.8, np.float32)
    lower[lift], upper[lift] = 0.0, 0.4
    act = np.asarray(active, np.uint8)
    lower[act == 0] = upper[act == 0] = 0.0
    carriers = [0, lift, pan, tilt, wrist] + arm + fingers
    s_link = np.asarray([carriers[k % len(carriers)] for k in range(n_spheres)], np.int32)
    s_pos = rng.normal(scale=0.05, size=(n_spheres, 3))
    s_r = rng.uniform(0.03, 0.07, n_spheres)
    enables = np.ones((L, L), np.uint8)
    for i in range(L):
        enables[i, i] = 0
        if parent[i] >= 0:
            enables[i, parent[i]] = enables[parent[i], i] = 0
    m = W.RobotModel(name="mobile", joint_types=np.asarray(types, np.int32), joint_poses=poses.astype(np.float32),
                     joint_axes=axes.astype(np.float32), parent=np.asarray(parent, np.int32), sphere_link=s_link,
                     sphere_pos=s_pos.astype(np.float32), sphere_r=s_r.astype(np.float32), active=act, lower=lower,
                     upper=upper, default=np.zeros(L, np.float32), enables=enables,
                     link_names=["link_%d" % i for i in range(L)], resolution=0.02)
    W.disable_default_collisions(m, np.random.default_rng(seed + 7), samples=500)
    return m


@functools.lru_cache(maxsize=64)
def _robot(kind, dof, spheres, seed):
    if kind == "mobile":
        return _mobile(seed, spheres)
    return W.serial_arm(seed, dof=dof, n_spheres=spheres, prismatic_torso=dof >= 8, resolution=0.02)


@functools.lru_cache(maxsize=64)
def _scene(kind, obstacles, seed):
    if kind == "shelf":
        return W.shelf_env(seed, n_boxes=max(0, obstacles - 5))
    if kind == "boxes":                                    # spheres and axis-aligned boxes, 4 : 1
        nb = obstacles // 5
        return W.random_env(seed, obstacles - nb, nb, 0)
    nb, nc = int(round(obstacles * 64 / 336)), int(round(obstacles * 16 / 336))
    return W.random_env(seed, obstacles - nb - nc, nb, nc, oriented=True)


def _model(c):
    return _robot(c["robot"], c["dof"], c["spheres"], c["robot_seed"])


def _env(c):
    return _scene(c["scene"], c["obstacles"], c["scene_seed"])


def _zeros(*shape, dtype=torch.float32):
    return torch.zeros(shape, dtype=dtype, device="cuda")


def _states(m, rng, n):
    """n configurations uniform in the limits (made on the GPU: a million take a moment)."""
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 62)))
    u = torch.rand((n, m.num_links), generator=g, device="cuda")
    lo, up = torch.from_numpy(m.lower).cuda(), torch.from_numpy(m.upper).cuda()
    act = torch.from_numpy(m.active.astype(bool)).cuda()
    return torch.where(act, lo + u * (up - lo), torch.from_numpy(m.default).cuda()).contiguous()


RULE = {"l2": _lib.STEP_L2, "linf": _lib.STEP_LINF}


# ---- prepare / run -----------------------------------------------------------------------

def prepare(case, seed):
    return _PREPARE[case["kind"]](case, np.random.default_rng(seed))


def run(state):
    return state["run"](state)


def _prepare_edges(c, rng):
    m, n = _model(c), c["n"]
    s = dict(run=_run_edges, c=c, R=api.Robot(m), E=api.Env(_env(c)), a=_states(m, rng, n), b=_states(m, rng, n),
             ok=_zeros(n, dtype=torch.uint8), length=_zeros(n))
    if c["first_hit"]:
        s["hit"], s["steps"] = _zeros(n, dtype=torch.int32), _zeros(n, dtype=torch.int32)
    return s


def _run_edges(s):
    c = s["c"]
    api.check_edges(s["R"], s["E"], s["a"], s["b"], c["resolution"], RULE[c["rule"]], s["ok"], s.get("hit"),
                    s["length"], s.get("steps"))
    out = dict(ok=s["ok"], length=s["length"])
    if c["first_hit"]:
        out.update(hit=s["hit"], steps=s["steps"])
    return out


def _prepare_states(c, rng):
    m, n = _model(c), c["n"]
    s = dict(run=_run_states, c=c, R=api.Robot(m), E=api.Env(_env(c)), q=_states(m, rng, n),
             verdict=_zeros(n, dtype=torch.uint8))
    if c["mode"] == "cost":
        s.update(costs=_zeros(4, n), total=_zeros(n))
    if c["poses"]:
        s["poses"] = _zeros(n, m.num_links, 4, 4)
    return s


def _run_states(s):
    mode = _lib.CHECK_COST if s["c"]["mode"] == "cost" else _lib.CHECK_VERDICT
    api.check_states(s["R"], s["E"], s["q"], s["verdict"], s.get("costs"), s.get("total"), mode,
                     poses=s.get("poses"))
    return {k: s[k] for k in ("verdict", "costs", "total", "poses") if k in s}


def _mix(c):
    """The (robot, scene, size) of each request of a batch."""
    g = np.random.default_rng(c["mix_seed"])
    mix = []
    for _ in range(c["n"]):
        i, k = int(g.integers(4)), int(g.integers(16))
        mix.append((i, k, int(min(c["largest"], np.exp(g.uniform(0, np.log(c["largest"])))))))
    return mix


def _prepare_batch(c, rng):
    models = [_robot("arm", 6 + i, 40 + 25 * i, 80 + i) for i in range(4)]
    R = [api.Robot(m) for m in models]
    E = [api.Env(_scene("mixed", 50 + 30 * k, 90 + k)) for k in range(16)]
    reqs = [dict(robot=R[i], env=E[k], q=_states(models[i], rng, n), verdict=_zeros(n, dtype=torch.uint8))
            for i, k, n in _mix(c)]
    return dict(run=_run_batch, c=c, reqs=reqs, cb=api.CheckBatch(max_requests=len(reqs)),
                verdicts=[r["verdict"] for r in reqs])


def _run_batch(s):
    s["cb"].run(s["reqs"])
    return torch.cat(s["verdicts"])


def _prepare_fk(c, rng):
    m, n = _model(c), c["n"]
    s = dict(run=_run_fk, c=c, R=api.Robot(m), q=_states(m, rng, n), poses=_zeros(n, m.num_links, 4, 4))
    if c["centers"]:
        s["centers"] = _zeros(n, m.num_spheres, 3)
    return s


def _run_fk(s):
    api.fk(s["R"], s["q"], s["poses"], s.get("centers"))
    return {k: s[k] for k in ("poses", "centers") if k in s}


def _prepare_nearest(c, rng):
    m, n = _model(c), c["n"]
    s = dict(run=_run_nearest, c=c, R=api.Robot(m), tree=_states(m, rng, c["tree"]), q=_states(m, rng, n), cand=None,
             out=_zeros(n, dtype=torch.int32))
    if c["share"] < 1.0:   # one connected group of the graph
        pick = rng.permutation(c["tree"])[: max(1, int(c["share"] * c["tree"]))]
        s["cand"] = torch.from_numpy(np.sort(pick).astype(np.int32)).cuda()
    return s


def _run_nearest(s):
    api.nearest(s["R"], s["tree"], s["q"], s["out"], cand=s["cand"])
    return s["out"]


def _region(m, case, height_only):
    """A task-space region through one configuration of the arm: the tip's position, or its
    height alone."""
    q0 = m.sample_full(np.random.default_rng(case["robot_seed"] + 3), 1)
    tip = m.num_links - 1
    T = W.fk_numpy(m, q0)[0][tip]
    if height_only:
        return q0, dict(task_link=tip, reference=(0.0, 0.0, float(T[2, 3]), 0.0, 0.0, 0.0),
                        tolerance=(10.0, 10.0, 0.01, 10.0, 10.0, 10.0), use_boundary=True)
    off = np.eye(4, dtype=np.float32)
    off[:3, :3] = T[:3, :3].T
    return q0, dict(task_link=tip, offset=off, reference=(float(T[0, 3]), float(T[1, 3]), float(T[2, 3]), 0.0, 0.0, 0.0),
                    tolerance=(1e-3,) * 3 + (2 * math.pi,) * 3, use_boundary=True)


def _near(m, q0, rng, n, spread):
    """n configurations around q0, inside the limits."""
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 62)))
    d = spread * torch.randn((n, m.num_links), generator=g, device="cuda")
    q = torch.from_numpy(q0).cuda() + d * torch.from_numpy(m.active.astype(np.float32)).cuda()
    return torch.maximum(torch.minimum(q, torch.from_numpy(m.upper).cuda()), torch.from_numpy(m.lower).cuda())


def _prepare_project(c, rng):
    m, n = _model(c), c["n"]
    q0, region = _region(m, c, False)
    q = _near(m, q0, rng, n, c["spread"]).contiguous()
    return dict(run=_run_project, c=c, R=api.Robot(m), region=region, samples=q, q=torch.empty_like(q),
                task=_zeros(n), bound=_zeros(n))


def _run_project(s):
    s["q"].copy_(s["samples"])
    api.project_states(s["R"], s["q"], iterations=s["c"]["iterations"], task_cost=s["task"], bound_cost=s["bound"],
                       **s["region"])
    return dict(q=s["q"], task=s["task"], bound=s["bound"])


STATES_CAP = 512


def _prepare_constrained(c, rng):
    m, n = _model(c), c["n"]
    q0, region = _region(m, c, True)
    R, E = api.Robot(m), api.Env(_env(c))
    have = _zeros(0, m.num_links)
    for _ in range(8):   # states of the region within the limits, free of collision where there are such
        q = (torch.from_numpy(q0).cuda() + 0.6 * (_states(m, rng, 16 * n + 512) - torch.from_numpy(q0).cuda())).contiguous()
        k = q.shape[0]
        task, bound, v = _zeros(k), _zeros(k), _zeros(k, dtype=torch.uint8)
        api.project_states(R, q, iterations=10, task_cost=task, bound_cost=bound, **region)
        api.check_states(R, E, q, v)
        have = torch.cat([have, q[(task == 0) & (bound == 0) & (v == 0)]])
        if have.shape[0] >= 2 * n:
            break
    else:
        have = torch.cat([have, _states(m, rng, 2 * n)])
    return dict(run=_run_constrained, c=c, R=R, E=E, region=region, a=have[:n].contiguous(),
                b=have[n: 2 * n].contiguous(), ok=_zeros(n, dtype=torch.uint8), cost=_zeros(n),
                count=_zeros(n, dtype=torch.int32), states=_zeros(n, STATES_CAP, m.num_links))


def _run_constrained(s):
    api.constrained_motions(s["R"], s["E"], s["a"], s["b"], resolution=s["c"]["resolution"], ok=s["ok"],
                            cost=s["cost"], num_states=s["count"], states=s["states"], **s["region"])
    return dict(ok=s["ok"], cost=s["cost"], count=s["count"], states=s["states"])


def _prepare_round(c, rng):
    m, n = _model(c), c["n"]
    return dict(run=_run_round, c=c, R=api.Robot(m), E=api.Env(_env(c)), seed=int(rng.integers(1 << 31)),
                tree=_states(m, rng, c["tree"]), q=_zeros(n, m.num_links), near=_zeros(n, dtype=torch.int32),
                total=_zeros(n), to=_zeros(n, m.num_links), ok=_zeros(n, dtype=torch.uint8), length=_zeros(n),
                free=_zeros(n, dtype=torch.uint8))


def _run_round(s):
    c, R = s["c"], s["R"]
    api.sample(R, s["seed"], 0, s["q"])
    api.nearest(R, s["tree"], s["q"], s["near"])
    api.steer(R, s["tree"], s["q"], 1.0, idx=s["near"])
    api.check_states(R, s["E"], s["q"], s["free"], None, s["total"], _lib.CHECK_COST)
    api.nearest(R, s["tree"], s["q"], s["near"])
    api.gather_states(s["tree"], s["near"], s["to"])
    api.check_edges(R, s["E"], s["q"], s["to"], c["resolution"], RULE[c["rule"]], s["ok"], None, s["length"])
    return dict(q=s["q"], total=s["total"], collides=s["free"], near=s["near"], ok=s["ok"], length=s["length"])


PATH_CAP = 512


def _prepare_plan(c, rng):
    m = _model(c)
    R, E = api.Robot(m), api.Env(_env(c))

    def free(q):
        v = _zeros(q.shape[0], dtype=torch.uint8)
        api.check_states(R, E, q, v)
        return q[v == 0]

    def edge_free(a, b):
        ok = _zeros(a.shape[0], dtype=torch.uint8)
        api.check_edges(R, E, a, b, c["resolution"], _lib.STEP_LINF, ok)
        return ok != 0

    q = free(_states(m, rng, 4096))
    k = q.shape[0] // 2
    a, b = q[:k].contiguous(), q[k: 2 * k].contiguous()
    far = torch.nonzero(~edge_free(a, b)).reshape(-1)   # the straight edge collides
    i = int(far[0])
    return dict(run=_run_plan, c=c, R=R, E=E, planner=api.Planner(R, max_nodes=100000, path_cap=PATH_CAP),
                start=a[i].cpu().numpy(), goal=b[i].cpu().numpy(), seed=int(rng.integers(1 << 31)))


def _run_plan(s):
    res, path = s["planner"].solve(s["E"], s["start"], s["goal"], lanes=1, max_iters=2000, range_=0.5,
                                   resolution=s["c"]["resolution"], rule=_lib.STEP_LINF, seed=s["seed"],
                                   balance=_lib.BALANCE_SWAP)
    whole = np.zeros((PATH_CAP, path.shape[1]), np.float32)   # a path's length is another for each problem
    whole[: len(path)] = path
    return dict(solved=res["solved"], iterations=res["iterations"], cost=float(res["cost"]), path=whole)


_PREPARE = dict(edges=_prepare_edges, states=_prepare_states, batch=_prepare_batch, fk=_prepare_fk,
                nearest=_prepare_nearest, project=_prepare_project, constrained=_prepare_constrained,
                round=_prepare_round, plan=_prepare_plan)


# ---- work ---------------------------------------------------------------------------------

def _fk_flops(m):
    """FK of one state: 151 operations per revolute joint, 129 prismatic, 63 fixed."""
    t = m.joint_types[1:]
    return 151 * int((t == W.REVOLUTE).sum()) + 129 * int((t == W.PRISMATIC).sum()) + 63 * int((t == W.FIXED).sum())


def _edge_states(c, n):
    """About how many states have to be looked at: the longest joint moves 3.8 rad on average,
    the whole vector 1.6 times that; a colliding edge is done after its first contact, so a
    fifth of the states remain."""
    return n * 0.2 * 3.8 * (1.6 if c["rule"] == "l2" else 1.0) / c["resolution"]


def work(case):
    c, k = case, case["kind"]
    n = c.get("n", 1)
    if k == "batch":
        models = [_robot("arm", 6 + i, 40 + 25 * i, 80 + i) for i in range(4)]
        by, fl = 0, 0
        for i, _, cnt in _mix(c):
            by += cnt * (4 * models[i].num_links + 1)
            fl += cnt * (_fk_flops(models[i]) + 18 * models[i].num_spheres)
        return dict(bytes=by, flops=fl)
    m = _model(c)
    L, S, D = m.num_links, m.num_spheres, m.dim
    state = _fk_flops(m) + 18 * S   # FK and sphere centres
    if k == "edges":
        return dict(bytes=n * (8 * L + 5 + (8 if c["first_hit"] else 0)), flops=_edge_states(c, n) * state)
    if k == "states":
        out = 1 + (20 if c["mode"] == "cost" else 0) + (64 * L if c["poses"] else 0)
        return dict(bytes=n * (4 * L + out), flops=n * state)
    if k == "fk":
        return dict(bytes=n * (4 * L + 64 * L + (12 * S if c["centers"] else 0)), flops=n * state)
    if k == "nearest":
        t = max(1, int(c["share"] * c["tree"]))
        return dict(bytes=4 * L * (t + n) + 4 * n, flops=3.0 * D * t * n)
    if k == "project":
        one = _fk_flops(m) + 40 * L + 21 * 2 * D + 6 * 6 * 12 * 2 + 72 * D + 12 * D
        return dict(bytes=n * (8 * L + 8), flops=n * (c["iterations"] * one + _fk_flops(m)))
    if k == "constrained":
        one = 2 * (_fk_flops(m) + 40 * L + 21 * 2 * D + 6 * 6 * 12 * 2 + 84 * D) + state
        return dict(bytes=n * (8 * L + 9), flops=n * 3.0 / c["resolution"] * one)
    if k == "round":
        return dict(bytes=4 * L * (c["tree"] + 3 * n) + 14 * n,
                    flops=6.0 * D * c["tree"] * n + n * state * (1 + 0.5 / c["resolution"]))
    return dict(bytes=8 * L, flops=200 * 0.5 / c["resolution"] * state)   # plan: some hundred extensions


# ---- exact: the same in 64 bits, plain torch ------------------------------------------------

def _fk64(m, q):
    """Link poses [n, L, 4, 4] of q [n, L] in 64 bits."""
    q = q.double()
    n = q.shape[0]
    P = [torch.eye(4, dtype=torch.float64, device="cuda").expand(n, 4, 4)]
    for i in range(1, m.num_links):
        J = torch.from_numpy(m.joint_poses[i].astype(np.float64)).cuda()
        a = m.joint_axes[i].astype(np.float64)
        X = torch.eye(4, dtype=torch.float64, device="cuda").repeat(n, 1, 1)
        if m.joint_types[i] == W.REVOLUTE:
            a = a / np.linalg.norm(a)
            K = torch.tensor([[0, -a[2], a[1]], [a[2], 0, -a[0]], [-a[1], a[0], 0]], dtype=torch.float64, device="cuda")
            aa = torch.from_numpy(np.outer(a, a)).cuda()
            c, s = torch.cos(q[:, i])[:, None, None], torch.sin(q[:, i])[:, None, None]
            X[:, :3, :3] = c * torch.eye(3, dtype=torch.float64, device="cuda") + s * K + (1 - c) * aa
        elif m.joint_types[i] == W.PRISMATIC:
            X[:, :3, 3] = q[:, i, None] * torch.from_numpy(a).cuda()
        P.append(P[m.parent[i]] @ (J @ X))
    return torch.stack(P, 1)


def _centers64(m, P):
    T = P[:, torch.from_numpy(m.sphere_link.astype(np.int64)).cuda()]
    p = torch.from_numpy(m.sphere_pos.astype(np.float64)).cuda()
    return (T[..., :3, :3] @ p[..., None])[..., 0] + T[..., :3, 3]


def _costs64(m, e, q):
    """The four costs [4, n]: self, spheres, boxes, cylinders."""
    d = lambda a: torch.from_numpy(np.asarray(a, np.float64)).cuda()   # noqa: E731
    S = m.num_spheres
    i, j = np.triu_indices(S, 1)
    li, lj = m.sphere_link[i], m.sphere_link[j]
    on = (li != lj) & (m.enables[li, lj] != 0)
    i, j = torch.from_numpy(i[on]).cuda(), torch.from_numpy(j[on]).cuda()
    r = d(m.sphere_r)
    parts = []
    for at in range(0, q.shape[0], 1024):
        C = _centers64(m, _fk64(m, q[at: at + 1024]))
        pen = (r[i] + r[j]) - (C[:, i] - C[:, j]).norm(dim=-1)
        cost = [pen.clamp(min=0).sum(1)]
        pen = r[None, :, None] + d(e.sphere_r) - torch.cdist(C, d(e.sphere_pos)[None].expand(C.shape[0], -1, -1),
                                                               compute_mode="donot_use_mm_for_euclid_dist")
        cost.append(pen.clamp(min=0).sum((1, 2)))
        tot = torch.zeros(C.shape[0], dtype=torch.float64, device="cuda")
        for k in range(len(e.box_pos)):
            x = (C - d(e.box_pos[k])) @ d(e.box_rot[k])
            out = x - torch.maximum(torch.minimum(x, d(e.box_max[k])), d(e.box_min[k]))
            tot += (r - out.norm(dim=-1)).clamp(min=0).sum(1)
        cost.append(tot)
        tot = torch.zeros(C.shape[0], dtype=torch.float64, device="cuda")
        for k in range(len(e.cyl_radius)):
            x = (C - d(e.cyl_pos[k])) @ d(e.cyl_rot[k])
            a = x[..., :2].norm(dim=-1) - float(e.cyl_radius[k])
            h = x[..., 2].abs() - 0.5 * float(e.cyl_height[k])
            sd = torch.hypot(a.clamp(min=0), h.clamp(min=0)) + torch.maximum(a, h).clamp(max=0)
            tot += (r - sd).clamp(min=0).sum(1)
        cost.append(tot)
        parts.append(torch.stack(cost))
    return torch.cat(parts, 1)


def _project64(m, region, q, iterations):
    tip = region["task_link"]
    off = torch.from_numpy(np.asarray(region["offset"], np.float64)).cuda()
    d = lambda a: torch.tensor(np.asarray(a, np.float64), device="cuda")   # noqa: E731
    ref, tol = d(np.float32(region["reference"])), d(np.float32(region["tolerance"]))
    act = torch.from_numpy(m.active.astype(bool)).cuda()
    lo, up = d(m.lower), d(m.upper)
    q = q.double().clone()
    eye = torch.eye(6, dtype=torch.float64, device="cuda")
    for _ in range(iterations):
        P = _fk64(m, q)
        F = P[:, tip] @ off
        v = torch.stack([F[:, 0, 3], F[:, 1, 3], F[:, 2, 3], torch.atan2(F[:, 2, 1], F[:, 2, 2]),
                         torch.asin(-F[:, 2, 0]), torch.atan2(F[:, 1, 0], F[:, 0, 0])], 1)
        e = ref - v
        e = torch.sign(e) * (e.abs() - tol).clamp(min=0)
        e = torch.cat([e[:, 3:], e[:, :3]], 1)
        J = torch.zeros((q.shape[0], 6, m.num_links), dtype=torch.float64, device="cuda")
        for j in range(tip + 1):
            w = P[:, j, :3, :3] @ d(m.joint_axes[j])
            if m.joint_types[j] == W.REVOLUTE:
                J[:, :3, j] = w
                J[:, 3:, j] = torch.linalg.cross(w, v[:, :3] - P[:, j, :3, 3])
            elif m.joint_types[j] == W.PRISMATIC:
                J[:, 3:, j] = w
        J = J * act
        step = (J.transpose(1, 2) @ torch.linalg.solve(J @ J.transpose(1, 2) + 1e-4 * eye, e[..., None]))[..., 0]
        pull = torch.where(q < lo, lo - q, torch.where(q > up, up - q, torch.zeros_like(q)))
        q = q + torch.where(act, step + pull, torch.zeros_like(q))
    return q


def exact(case, seed):
    c, k = case, case["kind"]
    if k in ("nearest", "batch", "constrained", "plan"):
        return None   # indices and flags; motions and plans whose course depends on single comparisons
    s = prepare(c, seed)
    m = _model(c)
    if k == "edges":
        return dict(ok=None, length=(s["a"].double() - s["b"].double()).norm(dim=1))
    if k == "states":
        if c["mode"] == "verdict" and not c["poses"]:
            return None
        out = dict(verdict=None)
        if c["mode"] == "cost":
            out["costs"] = _costs64(m, _env(c), s["q"])
            out["total"] = out["costs"].sum(0)
        if c["poses"]:
            out["poses"] = _fk64(m, s["q"])
        return out
    if k == "fk":
        P = _fk64(m, s["q"])
        out = dict(poses=P)
        if c["centers"]:
            out["centers"] = torch.cat([_centers64(m, P[at: at + 65536]) for at in range(0, P.shape[0], 65536)])
        return out
    if k == "project":   # the costs drop to 0 below 1e-4: no value of their own near it
        if c["spread"] > 0.05:   # some states pass near a singular pose: no value that rounding leaves alone
            return None
        return dict(q=_project64(m, s["region"], s["samples"], c["iterations"]), task=None, bound=None)
    return None   # round: its parts stand above, each by itself
