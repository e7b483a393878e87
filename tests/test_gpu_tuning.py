"""setTuning names the fields that it sets; the others stay the library's choice."""
import pytest

import __graft_entry__ as graft

pytestmark = pytest.mark.gpu


def test_one_knob_keeps_the_chosen_shape():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    pkg = graft.load_package()
    from habitat_sim_gb300 import procedural
    wl = procedural.config0(seed=5, envs=40, resolution=96, room_subdiv=10, boxes=4)
    a, b = (procedural.build_renderer(pkg, wl, mode=pkg.DrawMode.PerScene) for _ in range(2))
    a.setTuning(queue_fill_percent=50)
    b.draw()
    b.setTuning(queue_fill_percent=50)
    a.draw()
    assert a.tuning() == b.tuning() and a.tuning()["queue_fill_percent"] == 50
    assert a.tuning()["threads"] == 512 and a.tuning()["region_height"] == 64
    kept = a.tuning()
    with pytest.raises(pkg.GbrError):
        a.setTuning(threads=100)
    assert a.tuning() == kept
