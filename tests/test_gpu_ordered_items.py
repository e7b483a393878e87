"""Steps of several waves, whose items the device orders (a third launch), are
bit-exact against the per-scene form: viewports of odd sizes, scenes switched
off and on under a captured graph, a scene of more regions than the
kernel counts in shared memory, and a step without occlusion culling."""
import numpy as np
import pytest

import __graft_entry__ as graft

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return graft.load_package()


def _pair(pkg, viewports, seed, **tuning):
    from habitat_sim_gb300 import procedural
    wl = procedural.config0(seed=seed, envs=len(viewports), room_subdiv=12, boxes=6)
    wl.viewports = viewports
    wl.uniform = len(set(viewports)) == 1
    a = procedural.build_renderer(pkg, wl, mode=pkg.DrawMode.Batched)
    b = procedural.build_renderer(pkg, wl, mode=pkg.DrawMode.PerScene)
    if tuning:
        a.setTuning(**tuning)
    return wl, a, b


def _launches(r):
    return r.lastDrawStats()["kernel_launches"]


def _same(pkg, a, b, scenes):
    for plane in (pkg.Plane.Color, pkg.Plane.Depth, pkg.Plane.LinearDepth, pkg.Plane.Semantic):
        for s in scenes:
            assert np.array_equal(a.sceneImage(plane, s), b.sceneImage(plane, s)), (plane, s)


@pytest.mark.parametrize("name,viewports,tuning", [
    ("odd", [(1 + 37 * s % 200, 1 + 53 * s % 150) for s in range(90)],
     dict(threads=512, ctas_per_sm=2, region_width=64, region_height=32)),
    ("whole", [(128, 128)] * 200, {}),
    ("regions of 64", [(130, 70)] * 96, dict(threads=512, ctas_per_sm=2, region_width=64, region_height=64)),
    ("many regions", [(64, 64)] * 20 + [(2112, 2112)],
     dict(threads=512, ctas_per_sm=2, region_width=64, region_height=64)),
    ("no culling", [(100, 100)] * 200, dict(occlusion_culling=0)),
], ids=lambda v: v if isinstance(v, str) else "")
def test_ordered_equals_per_scene(pkg, name, viewports, tuning):
    from habitat_sim_gb300 import procedural
    wl, a, b = _pair(pkg, viewports, 41, **tuning)
    for step in range(2):
        poses = procedural.camera_poses(wl, step)
        for r in (a, b):
            procedural.set_cameras(r, wl, poses)
            r.draw()
        assert _launches(a) == 3, name
        _same(pkg, a, b, range(len(viewports)))


def test_ordered_under_a_graph(pkg):
    """Scenes come and go: the list changes between ordered and not, and within
    the ordered form, under captured graphs."""
    from habitat_sim_gb300 import procedural
    n = 160
    wl, a, b = _pair(pkg, [(96, 80)] * n, 42)
    seen = set()
    for step, on in enumerate([n, n, 120, 3, 140, n, 20]):
        poses = procedural.camera_poses(wl, step)
        for r in (a, b):
            procedural.set_cameras(r, wl, poses)
            for s in range(n):
                r.setSceneEnabled(s, (s * 7) % n < on)
        a.draw(graph=True)
        b.draw()
        seen.add(_launches(a))
        _same(pkg, a, b, [s for s in range(n) if (s * 7) % n < on])
    assert seen == {2, 3}


def test_ordered_per_scene_form(pkg):
    """The per-scene form's launches of several waves are ordered as well, in
    the room of the batched form's list: both forms in turn on one renderer."""
    from habitat_sim_gb300 import procedural
    wl, a, b = _pair(pkg, [(1 + 37 * s % 200, 1 + 53 * s % 150) for s in range(90)], 43)
    tuned = dict(threads=512, ctas_per_sm=2, region_width=64, region_height=64, plain_region_width=64,
                 plain_region_height=32)
    b.setTuning(**tuned)
    for step in range(3):
        poses = procedural.camera_poses(wl, step)
        for r in (a, b):
            procedural.set_cameras(r, wl, poses)
        a.draw()
        b.draw()  # per scene
        assert _launches(b) == 3
        _same(pkg, a, b, range(90))
        b.draw(mode=pkg.DrawMode.Batched)
        _same(pkg, a, b, range(90))
