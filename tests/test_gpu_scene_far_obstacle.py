"""A scene that holds an obstacle very far away: its distance field has cells of kilometres,
and a robot sphere that is a fraction of a millimetre inside an obstacle at hand still collides
with it."""
import numpy as np
import pytest

from isaac_sim_ros2_humble_gb300 import _lib, api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _point_robot(radius):
    """One sphere that three prismatic joints put anywhere."""
    L = 4
    f = np.float32
    enables = np.zeros((L, L), np.uint8)
    lim = np.full(L, 5.0, f)
    return W.RobotModel(name="point", joint_types=np.int32([W.FIXED] + [W.PRISMATIC] * 3),
                        joint_poses=np.tile(np.eye(4, dtype=f), (L, 1, 1)),
                        joint_axes=f([[0, 0, 1], [1, 0, 0], [0, 1, 0], [0, 0, 1]]),
                        parent=np.arange(-1, L - 1, dtype=np.int32), sphere_link=np.int32([L - 1]),
                        sphere_pos=np.zeros((1, 3), f), sphere_r=f([radius]),
                        active=np.uint8([0, 1, 1, 1]), lower=-lim, upper=lim, default=np.zeros(L, f),
                        enables=enables, link_names=["l%d" % i for i in range(L)], resolution=0.02)


@pytest.mark.parametrize("far,near", [
    ((1e4, 0, 0), (0.4, -0.39, -0.19)),
    ((1e5, 1e5, 0), (0.4, -0.39, -0.19)),
    ((-600943.1875, 600943.1875, -600943.1875), (-0.3606899380683899, -0.5153268575668335, -0.09450481086969376)),
    ((-966279.9375, 0, -966279.9375), (0.40003231167793274, -0.3934936821460724, -0.1876811981201172)),
    ((787103.6875, 0, 787103.6875), (-0.0006793711218051612, -0.5797777771949768, -0.5161899924278259)),
    ((1e6, 1e6, 1e6), (0.4, -0.39, -0.19)),
])
def test_contacts_at_hand(far, near):
    r, ro = np.float32(0.05), np.float32(0.1)
    R = api.Robot(_point_robot(r))
    e = W.Environment.empty()
    f = np.float32
    e.sphere_pos, e.sphere_r = f([near, far]), f([ro, ro])
    E = api.Env(e)
    rng = np.random.default_rng(5)
    n = 200000
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    # the first half touches by 0.1 to 1 mm, the others stay clear by as much
    gap = rng.uniform(1e-4, 1e-3, n) * np.where(np.arange(n) < n // 2, -1, 1)
    q = np.zeros((n, 4), f)
    q[:, 1:] = f(near).astype(np.float64) + u * (0.15 + gap)[:, None]
    d = torch.from_numpy(q).cuda()
    v, vc = (torch.full((n,), 9, dtype=torch.uint8, device="cuda") for _ in range(2))
    costs, total = torch.zeros((4, n), device="cuda"), torch.zeros(n, device="cuda")
    api.check_states(R, E, d, v)
    api.check_states(R, E, d, vc, costs, total, _lib.CHECK_COST)
    ok = torch.full((n,), 9, dtype=torch.uint8, device="cuda")
    api.check_edges(R, E, d, d, 0.02, _lib.STEP_LINF, ok)     # edges of one state
    torch.cuda.synchronize()
    hit = np.arange(n) < n // 2
    np.testing.assert_array_equal(v.cpu().numpy() != 0, hit)
    np.testing.assert_array_equal(vc.cpu().numpy() != 0, hit)
    np.testing.assert_array_equal(ok.cpu().numpy() == 0, hit)
    # the penetration: positions and radii are rounded at some 1e-8
    np.testing.assert_allclose(total.cpu().numpy(), np.where(hit, -gap, 0), atol=1e-6)
