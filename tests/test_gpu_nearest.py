"""Nearest neighbours at the edges of the kernel's tiles: bit-exact against the oracle,
the lowest candidate position on ties, whatever the number of queries, candidates and
active joints."""
import numpy as np
import pytest

import oracle as O
from isaac_sim_ros2_humble_gb300 import api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _nearest(robot, R, tree, q, cand=None):
    out = torch.full((len(q),), -7, dtype=torch.int32, device="cuda")
    api.nearest(R, torch.from_numpy(tree).cuda(), torch.from_numpy(q).cuda(), out,
                cand=None if cand is None else torch.from_numpy(cand).cuda())
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.fixture(scope="module")
def arm():
    robot = W.serial_arm(1, dof=7, n_spheres=20)
    return robot, api.Robot(robot)


@pytest.mark.parametrize("M", [1, 31, 128, 129, 1024, 1025, 8193, 20011])
@pytest.mark.parametrize("Q", [1, 19, 20, 77, 700])
def test_sizes_and_ties(arm, M, Q):
    robot, R = arm
    rng = np.random.default_rng(M + Q)
    tree, q = robot.sample_full(rng, M), robot.sample_full(rng, Q)
    tree[rng.integers(0, M, M // 3)] = tree[rng.integers(0, M, M // 3)]   # equal rows
    q[: Q // 2] = tree[rng.integers(0, M, Q // 2)]                         # distance 0
    np.testing.assert_array_equal(_nearest(robot, R, tree, q), O.nearest(tree, q, active=robot.active))
    cand = rng.permutation(M)[: max(1, M // 2)].astype(np.int32)           # any order
    np.testing.assert_array_equal(_nearest(robot, R, tree, q, cand), O.nearest(tree, q, active=robot.active, cand=cand))


@pytest.mark.parametrize("dof", [1, 2, 3, 8, 9, 15, 16, 17])
def test_active_joint_counts(dof):
    robot = W.serial_arm(60 + dof, dof=dof, n_spheres=dof)
    rng = np.random.default_rng(dof)
    tree, q = robot.sample_full(rng, 3000), robot.sample_full(rng, 50)
    np.testing.assert_array_equal(_nearest(robot, api.Robot(robot), tree, q), O.nearest(tree, q, active=robot.active))


def test_inactive_joints_and_rows_that_are_not_numbers():
    robot = W.tree_robot(3)                       # 10 links, 8 active joints in between fixed ones
    R = api.Robot(robot)
    rng = np.random.default_rng(1)
    tree, q = robot.sample_full(rng, 2000), robot.sample_full(rng, 40)
    want = O.nearest(tree, q, active=robot.active)
    tree[:, ~robot.active.astype(bool)] = np.nan  # not read
    np.testing.assert_array_equal(_nearest(robot, R, tree, q), want)
    lost = tree.copy()
    lost[want] = np.nan                           # a row that is not a number is never nearest
    rest = np.setdiff1d(np.arange(2000), want).astype(np.int32)
    np.testing.assert_array_equal(_nearest(robot, R, lost, q), O.nearest(np.nan_to_num(tree), q, active=robot.active, cand=rest))
    far = np.full((5, robot.num_links), np.inf, np.float32)
    np.testing.assert_array_equal(_nearest(robot, R, far, q), np.full(40, -1))
