"""The chunk kernel of edge validation (states of a chunk side by side in the lanes)
against the state-by-state kernel: identical verdicts and first hits, where the chunk's
items do not fill the lanes evenly or do not take the common path."""
import dataclasses

import numpy as np
import pytest

from isaac_sim_ros2_humble_gb300 import _lib, api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _run(R, E, a, b, res, first_hit):
    n = a.shape[0]
    ok = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
    fh = torch.full((n,), 99, dtype=torch.int32, device="cuda")
    api.check_edges(R, E, a, b, res, 1, ok, fh if first_hit else None)
    torch.cuda.synchronize()
    return ok.cpu().numpy(), fh.cpu().numpy()


def _forms_agree(robot, env, n, res, forms=(4, 10), seed=5):
    R, E = api.Robot(robot), api.Env(env)
    rng = np.random.default_rng(seed)
    a, b = (torch.from_numpy(robot.sample_full(rng, n)).cuda() for _ in range(2))
    R.set_edge_form(1)
    ok, fh = _run(R, E, a, b, res, True)
    np.testing.assert_array_equal(ok, fh == -1)
    for form in forms:
        R.set_edge_form(form)
        ok_f, fh_f = _run(R, E, a, b, res, True)
        np.testing.assert_array_equal(fh_f, fh)
        np.testing.assert_array_equal(ok_f, ok)
        np.testing.assert_array_equal(_run(R, E, a, b, res, False)[0], ok)
    return ok


@pytest.mark.parametrize("n_spheres", [1, 7, 33, 57, 200])
def test_odd_sphere_counts(n_spheres):
    robot = W.serial_arm(51, dof=7, n_spheres=n_spheres, radius_range=(0.02, 0.05))
    ok = _forms_agree(robot, W.random_env(52, 33, 5, 3, oriented=True), 513, 0.03)
    assert 0 < ok.sum() < len(ok)


def test_one_sided_link_mask_takes_the_pair_list():
    """A mask that enables (link of the lower sphere index, link of the higher) one way
    only, with the spheres in random order: the pairs of two groups are then not all
    (sphere of a, sphere of b) pairs, and the pair list decides."""
    base = W.serial_arm(53, dof=6, n_spheres=60, radius_range=(0.03, 0.06))
    order = np.random.default_rng(3).permutation(60)
    robot = dataclasses.replace(base, sphere_link=base.sphere_link[order], sphere_pos=base.sphere_pos[order],
                                sphere_r=base.sphere_r[order], enables=np.triu(base.enables, 1).astype(np.uint8))
    ok = _forms_agree(robot, W.Environment.empty(), 600, 0.03)
    assert 0 < ok.sum() < len(ok)


def test_branching_robot_with_many_links():
    """A robot of 20 links (4 states a chunk): parents that are not the previous link."""
    t = W.tree_robot(4, n_spheres=60)
    parent = np.concatenate([t.parent, [9, 10, 8, 12, 2, 14, 14, 5, 17, 1]]).astype(np.int32)
    L = len(parent)
    ext = lambda a, fill: np.concatenate([a, np.full((L - len(t.parent),) + a.shape[1:], fill, a.dtype)])   # noqa: E731
    poses = ext(t.joint_poses, 0)
    poses[len(t.parent):] = t.joint_poses[1]
    enables = np.zeros((L, L), np.uint8)
    enables[: len(t.parent), : len(t.parent)] = t.enables
    robot = dataclasses.replace(t, parent=parent, joint_types=ext(t.joint_types, W.REVOLUTE), joint_poses=poses,
                                joint_axes=ext(t.joint_axes, 1.0), active=ext(t.active, 1),
                                lower=ext(t.lower, -2.0), upper=ext(t.upper, 2.0), default=ext(t.default, 0.0),
                                enables=enables, link_names=["l%d" % i for i in range(L)])
    ok = _forms_agree(robot, W.random_env(54, 40, 8, 4, oriented=True), 400, 0.03, forms=(0, 4, 10))
    assert 0 < ok.sum() < len(ok)


@pytest.mark.parametrize("n", [1, 2, 31, 57, 300, 4000])
@pytest.mark.parametrize("res", [0.004, 0.02, 3.0])
def test_edges_cut_into_parts(n, res):
    """From a single edge (all of its chunks at once on different warps) to more edges than
    warps; long edges (up to 1,400 states, past the last length bucket), and edges of one
    or two states."""
    robot = W.serial_arm(55, dof=7, n_spheres=50)
    ok = _forms_agree(robot, W.random_env(56, 24, 6, 2, oriented=True), n, res, forms=(0,), seed=n)
    if n >= 300:
        assert 0 < ok.sum() < n


def test_outputs_of_long_and_free_edges_without_any_hit():
    """Edges too long to validate beside free ones: the outputs that no warp touches."""
    robot = W.serial_arm(57, dof=6, n_spheres=12, radius_range=(0.01, 0.02))
    robot.enables[:] = 0
    R, E = api.Robot(robot), api.Env(W.Environment.empty())
    a = torch.zeros((5, robot.num_links), device="cuda")
    b = a.clone()
    b[1, 2], b[3, 1] = 2.0, 1e-3
    ok, fh = _run(R, E, a, b, 2e-7, True)
    np.testing.assert_array_equal(ok, [1, 0, 1, 1, 1])
    np.testing.assert_array_equal(fh, [-1, -2, -1, -1, -1])
    np.testing.assert_array_equal(_run(R, E, a, b, 2e-7, False)[0], ok)


@pytest.mark.parametrize("n", [3, 160, 700, 5000])
def test_batches_whose_edges_are_settled_by_their_probes(n):
    """Every edge starts, or ends, in collision, or only some do: later parts are dropped."""
    robot = W.serial_arm(58, dof=7, n_spheres=50)
    env = W.random_env(59, 60, 10, 4, oriented=True)
    R, E = api.Robot(robot), api.Env(env)
    q = torch.from_numpy(robot.sample_full(np.random.default_rng(n), 30000)).cuda()
    v = torch.zeros(30000, dtype=torch.uint8, device="cuda")
    api.check_states(R, E, q, v)
    hit, free = q[v == 1], q[v == 0]
    for a, b in ((hit[:n], free[:n]), (free[:n], hit[:n]), (torch.cat([hit[: n // 2], free[: n - n // 2]]), free[n: 2 * n])):
        a, b = a.contiguous(), b.contiguous()
        R.set_edge_form(1)
        want = _run(R, E, a, b, 0.01, True)
        R.set_edge_form(0)
        for k in range(3):
            got = _run(R, E, a, b, 0.01, True)
            np.testing.assert_array_equal(got[0], want[0])
            np.testing.assert_array_equal(got[1], want[1])
            np.testing.assert_array_equal(_run(R, E, a, b, 0.01, False)[0], want[0])


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1024, 1025])
def test_few_edges_as_among_many(n, form):
    """Up to 1,024 edges are prepared by one block: every output as in a batch of 3,000."""
    robot = W.serial_arm(95, dof=7, n_spheres=50)
    R, E = api.Robot(robot), api.Env(W.random_env(96, 60, 8, 4, oriented=True))
    R.set_edge_form(form)
    g = np.random.default_rng(7)
    a, b = (torch.from_numpy(robot.sample_full(g, 3000)).cuda() for _ in range(2))
    b[::17] = a[::17]                      # edges of one state
    b[5, 2] = float("inf")                 # an edge too long to validate

    def check(k):
        ok, length = torch.full((k,), 7, dtype=torch.uint8, device="cuda"), torch.zeros(k, device="cuda")
        hit, steps = (torch.full((k,), 9, dtype=torch.int32, device="cuda") for _ in range(2))
        api.check_edges(R, E, a[:k].contiguous(), b[:k].contiguous(), 0.05, _lib.STEP_LINF, ok, hit, length, steps)
        torch.cuda.synchronize()
        return ok, hit, length, steps

    for few, many in zip(check(n), check(3000)):
        assert torch.equal(few, many[:n])
