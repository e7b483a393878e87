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


@pytest.mark.parametrize("threads", [256, 512, 1024])
def test_queue_sizes_draw_the_same(threads):
    """A stack of large triangles, more than queue and spill area hold at once."""
    import numpy as np
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    pkg = graft.load_package()
    import scenarios as S
    from oracle.model import OracleRenderer
    from parity import assert_parity, compare_scene
    rng = np.random.default_rng(12)
    n = 2500
    z = rng.uniform(-3.0, -1.0, n).astype(np.float32)
    pos = np.zeros((3 * n, 3), np.float32)
    for k, (dx, dy) in enumerate([(-3.0, -3.0), (3.0, -3.0), (0.0, 3.0)]):
        pos[k::3, 0], pos[k::3, 1], pos[k::3, 2] = dx * -z, dy * -z, z
    col = rng.uniform(0, 1, (3 * n, 4)).astype(np.float32)
    cpu = OracleRenderer((100, 70), (1, 1))
    cfg = pkg.RendererConfiguration().setTileSizeCount((100, 70), (1, 1)).setDrawMode(pkg.DrawMode.Batched)
    gpu = pkg.RendererStandalone(cfg)
    for r in (gpu, cpu):
        m = r.addMesh(pos, col, None, None, np.arange(3 * n, dtype=np.uint32))
        r.addNodeHierarchyTemplate("stack", [(m, 0, 3 * n, 0, None)])
        r.addNodeHierarchy(0, "stack")
        r.updateCamera(0, S.perspective(60.0, 100 / 70, 0.1, 10.0), S.translation(0.1, -0.2, 0.3))
    cpu.draw()
    for fill in (25, 68, 75, 76, 100):
        gpu.setTuning(threads=threads, queue_fill_percent=fill, occlusion_culling=0)
        gpu.draw()
        assert_parity([compare_scene(gpu, cpu, pkg, 0)])
