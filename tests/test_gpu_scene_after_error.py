"""After a call that failed for want of memory, scenes can be made and calls launch."""
import pytest

from isaac_sim_ros2_humble_gb300 import _lib, api, workloads as W

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_scene_after_a_failed_allocation():
    with pytest.raises(_lib.GbmpError) as e:
        api.BatchPlanner(max_problems=4096, max_nodes=1 << 24, max_links=16)    # some 10 TB
    assert e.value.status == 2
    env = W.random_env(3, 20, 5, 2, oriented=True)
    api.Env(env)


def test_calls_after_a_failed_allocation():
    robot = W.serial_arm(4, dof=6, n_spheres=30)
    R, E = api.Robot(robot), api.Env(W.random_env(3, 20, 5, 2, oriented=True))
    q = torch.zeros((8, robot.num_links), device="cuda")
    v = torch.full((8,), 9, dtype=torch.uint8, device="cuda")
    api.check_states(R, E, q, v)     # the kernel is loaded
    v.fill_(9)
    with pytest.raises(_lib.GbmpError) as e:
        api.BatchPlanner(max_problems=4096, max_nodes=1 << 24, max_links=16)
    assert e.value.status == 2
    api.check_states(R, E, q, v)
    torch.cuda.synchronize()
    assert (v <= 1).all()
