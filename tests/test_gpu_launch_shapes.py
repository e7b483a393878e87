"""The launch shapes chosen by the library (no tuning set), bit-exact against
the oracle or the other draw mode: regions split for a few views, the per-scene
form's one launch over many scenes, spill slots shared by a grid larger than
what is resident, and triangle ordinals that do not fit with their draw's
index."""
import numpy as np
import pytest

import __graft_entry__ as graft
import scenarios as S
from parity import assert_parity, compare_scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return graft.load_package()


@pytest.mark.parametrize("mode", [0, 1], ids=["per_scene", "batched"])
@pytest.mark.parametrize("envs,size", [(1, (1, 1)), (1, (33, 17)), (1, (300, 210)), (2, (130, 70)), (5, (64, 64)),
                                       (17, (48, 31))])
def test_few_views_match_oracle(pkg, mode, envs, size):
    from habitat_sim_gb300 import procedural
    from oracle.model import OracleRenderer
    wl = procedural.config0(seed=31, envs=envs, room_subdiv=12, boxes=6)
    wl.viewports = [size] * envs
    poses = procedural.camera_poses(wl, 3)
    gpu = procedural.build_renderer(pkg, wl, mode=pkg.DrawMode(mode))
    cpu = procedural.build_oracle(OracleRenderer, wl)
    for r in (gpu, cpu):
        procedural.set_cameras(r, wl, poses)
    gpu.draw(graph=bool(mode))
    cpu.draw()
    assert_parity([compare_scene(gpu, cpu, pkg, s) for s in range(envs)])


def test_modes_agree_when_views_come_and_go(pkg):
    """The item list, and with it the z-buffer a CTA is launched with, changes
    under a captured graph as scenes are disabled and enabled."""
    from habitat_sim_gb300 import procedural
    wl = procedural.config0(seed=32, envs=40, resolution=128, room_subdiv=10, boxes=4)
    a = procedural.build_renderer(pkg, wl, mode=pkg.DrawMode.Batched)
    b = procedural.build_renderer(pkg, wl, mode=pkg.DrawMode.PerScene)
    for step, on in enumerate([40, 1, 3, 40, 17, 2]):
        poses = procedural.camera_poses(wl, step)
        for r in (a, b):
            procedural.set_cameras(r, wl, poses)
            for s in range(40):
                r.setSceneEnabled(s, s < on)
        a.draw(graph=True)
        b.draw()
        for plane in (pkg.Plane.Color, pkg.Plane.Depth, pkg.Plane.LinearDepth, pkg.Plane.Semantic):
            for s in range(on):
                assert np.array_equal(a.sceneImage(plane, s), b.sceneImage(plane, s)), (step, plane, s)


def test_spill_slots_shared_by_a_large_grid(pkg):
    """1200 CTAs of which at most 608 are resident, each queueing more large
    triangles than its shared queue holds: the per-scene form equals the
    batched form, whose CTAs own their spill areas."""
    rng = np.random.default_rng(12)
    n = 1024
    z = rng.uniform(-3.0, -1.0, n).astype(np.float32)
    z[::5] = np.float32(-2.0)
    pos = np.zeros((3 * n, 3), np.float32)
    for k, (dx, dy) in enumerate([(-3.0, -3.0), (3.0, -3.0), (0.0, 3.0)]):
        pos[k::3, 0], pos[k::3, 1], pos[k::3, 2] = dx * -z, dy * -z, z
    col = rng.uniform(0, 1, (3 * n, 4)).astype(np.float32)
    out = []
    for mode in (pkg.DrawMode.PerScene, pkg.DrawMode.Batched):
        cfg = pkg.RendererConfiguration().setTileSizeCount((640, 480), (1, 1)).setDrawMode(mode)
        r = pkg.RendererStandalone(cfg)
        r.setTuning(threads=256, region_width=64, region_height=64, ctas_per_sm=4, plain_region_width=16,
                    plain_region_height=16)
        m = r.addMesh(pos, col, None, None, np.arange(3 * n, dtype=np.uint32))
        r.addNodeHierarchyTemplate("stack", [(m, 0, 3 * n, 0, None)])
        r.addNodeHierarchy(0, "stack")
        r.updateCamera(0, S.perspective(60.0, 640 / 480, 0.1, 10.0), S.translation(0.1, -0.2, 0.3))
        for _ in range(2):
            r.draw()
        out.append([r.colorImage(), r.depthImage(), r.semanticImage()])
    for p, b in zip(*out):
        assert np.array_equal(p, b)


@pytest.mark.parametrize("mode", [0, 1], ids=["per_scene", "batched"])
def test_ordinals_that_do_not_fit_with_the_draw_index(pkg, mode):
    """2100 draws beside one of 2^20 + 2 triangles: 12 + 21 bits, so pixels
    find their draw by search."""
    from oracle.model import OracleRenderer
    side = 725
    g = np.arange(side)
    x, y = np.meshgrid(np.linspace(-4, 4, side), np.linspace(-4, 4, side))
    pos = np.stack([x.ravel(), y.ravel(), np.full(side * side, -5.0)], 1).astype(np.float32)
    q = (g[:-1, None] * side + g[None, :-1]).ravel()
    tris = np.concatenate([np.stack([q, q + 1, q + side + 1], 1), np.stack([q, q + side + 1, q + side], 1)])
    tris = np.concatenate([tris, tris[:2]])[:(1 << 20) + 2].astype(np.uint32)
    quad = np.array([[-0.04, -0.04, 0], [0.04, -0.04, 0], [0, 0.04, 0]], np.float32)
    rng = np.random.default_rng(4)
    at = rng.uniform(-1.5, 1.5, (2100, 2))
    proj = S.perspective(70.0, 1.0, 0.1, 20.0)
    cfg = pkg.RendererConfiguration().setTileSizeCount((96, 96), (1, 1)).setDrawMode(pkg.DrawMode(mode))
    gpu, cpu = pkg.RendererStandalone(cfg), OracleRenderer((96, 96), (1, 1))
    for r in (gpu, cpu):
        big = r.addMesh(pos, rng.uniform(0, 1, (len(pos), 4)).astype(np.float32) * 0 + 0.5, None, None, tris.ravel())
        small = r.addMesh(quad, np.array([[1, 0, 0, 1], [0, 1, 0, 1], [0, 0, 1, 1]], np.float32), None, None,
                          np.arange(3, dtype=np.uint32))
        r.addNodeHierarchyTemplate("wall", [(big, 0, tris.size, 0, None)])
        r.addNodeHierarchyTemplate("quad", [(small, 0, 3, 0, None)])
        r.setSemanticId(0, r.addNodeHierarchy(0, "wall"), 7)
        for k, (u, v) in enumerate(at):
            m = np.eye(4, dtype=np.float32)
            m[3, :3] = (u, v, -2.0 - (k % 50) * 0.02)
            r.setSemanticId(0, r.addNodeHierarchy(0, "quad", m), 100 + k)
        r.updateCamera(0, proj, S.translation(0.0, 0.0, 0.0))
        r.draw()
    assert_parity([compare_scene(gpu, cpu, pkg, 0)])
    assert len(np.unique(gpu.semanticImage())) > 200
