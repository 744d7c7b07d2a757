"""FK of many states by one warp: link counts on both sides of the rules for the states of a
chunk, counts that leave a remainder."""
import numpy as np
import pytest

from isaac_sim_ros2_humble_gb300 import api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 6, 1003])
@pytest.mark.parametrize("dof", [1, 15, 16, 17, 31, 63])
def test_links(dof, n):
    m = W.serial_arm(91, dof=dof, n_spheres=2 * dof + 1, offset_range=(0.02, 0.06))
    q = m.sample_full(np.random.default_rng(n), n)
    L, S = m.num_links, m.num_spheres
    poses, centers = torch.zeros((n, L, 4, 4), device="cuda"), torch.zeros((n, S, 3), device="cuda")
    api.fk(api.Robot(m), torch.from_numpy(q).cuda(), poses, centers)
    torch.cuda.synchronize()
    want = W.fk_numpy(m, q)
    # single precision along at most 63 links of up to 0.1 m: 64 x 2^-23 x a few
    np.testing.assert_allclose(poses.cpu().numpy(), want, atol=5e-5)
    link = want[:, m.sphere_link]
    at = np.einsum("nsij,sj->nsi", link[..., :3, :3], m.sphere_pos) + link[..., :3, 3]
    np.testing.assert_allclose(centers.cpu().numpy(), at, atol=5e-5)
