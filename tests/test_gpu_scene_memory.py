"""The device's free memory around scenes that come and go."""
import pytest

import mesoengine_gb300 as meso

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

KEPT = 1 << 30  # of freed scenes' memory, by a context
SLACK = 256 << 20  # what a first launch or a cached temporary may take


def free():
    return torch.cuda.mem_get_info()[0]


def test_destroyed_scenes_give_their_memory_back():
    c = meso.Context(0)
    c.scene_from_terrain(meso.terrain_preset("small")).destroy()
    c.sync()
    before = free()
    big = c.scene_from_terrain(meso.terrain_preset("small"), spare_bricks=6 << 20)  # 6.5 GiB
    assert before - free() > 6 << 30
    big.destroy()
    assert before - free() < KEPT + SLACK
    c.close()
    assert before - free() < SLACK
