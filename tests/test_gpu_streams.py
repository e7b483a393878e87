"""Draws of one renderer on alternating non-blocking streams, and while the legacy
default stream is busy: every image equals the one drawn alone."""
import numpy as np
import pytest

import __graft_entry__ as graft

pytestmark = pytest.mark.gpu


def _planes(pkg, r):
    return [r.sceneImage(p, s) for p in (pkg.Plane.Color, pkg.Plane.Depth, pkg.Plane.Semantic)
            for s in range(r.sceneCount())]


@pytest.mark.parametrize("mode", [0, 1], ids=["per_scene", "batched"])
def test_streams_in_turn(mode):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    pkg = graft.load_package()
    from habitat_sim_gb300 import procedural
    wl = procedural.config0(seed=17, envs=170, resolution=100, room_subdiv=10, boxes=4)
    a, b = (procedural.build_renderer(pkg, wl, mode=pkg.DrawMode(mode)) for _ in range(2))
    streams = [torch.cuda.Stream() for _ in range(2)]
    for step in range(6):
        poses = procedural.camera_poses(wl, step)
        for r in (a, b):
            procedural.set_cameras(r, wl, poses)
        if step % 3 == 0:
            torch.cuda._sleep(20_000_000)  # about 10 ms of work on the legacy stream
            for r in (a, b):  # the scene tables are built again
                r.setSemanticId(0, 0, 100 + step)
        if step == 3:
            a.addTexture(np.full((2, 2, 4), 7, np.uint8))
        # Two draws in flight at once, on different streams; the second one counts.
        a.draw(streams[step % 2], graph=bool(mode))
        a.draw(streams[1 - step % 2], graph=bool(mode))
        b.draw()
        torch.cuda.synchronize()
        for x, y in zip(_planes(pkg, a), _planes(pkg, b)):
            assert np.array_equal(x, y), step
