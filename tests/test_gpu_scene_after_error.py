"""A scene can be made after a call that failed for want of memory."""
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
