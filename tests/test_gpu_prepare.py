"""Scenes whose numbers of visible draws lie at the edges of the prepare
kernel's passes and sorts (blocks of 128 draws, ranks up to 512, a bitonic sort
up to 2048, draw order beyond; depths tie), bit-exact against the oracle."""
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


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 127, 128, 129, 511, 512, 513, 1000, 2048, 2049])
def test_number_of_visible_draws(pkg, n):
    from oracle.model import OracleRenderer
    rng = np.random.default_rng(n)
    quad = np.array([[-0.1, -0.1, 0], [0.1, -0.1, 0], [0, 0.1, 0]], np.float32)
    at = rng.uniform(-1.2, 1.2, (n, 2))
    z = rng.integers(3, 9, n) * -0.5 if n > 3 else rng.uniform(-4, -2, n)
    proj = S.perspective(70.0, 1.0, 0.1, 20.0)
    cfg = pkg.RendererConfiguration().setTileSizeCount((96, 96), (1, 1))
    gpu, cpu = pkg.RendererStandalone(cfg), OracleRenderer((96, 96), (1, 1))
    for r in (gpu, cpu):
        mesh = r.addMesh(quad, np.array([[1, 0, 0, 1], [0, 1, 0, 1], [0, 0, 1, 1]], np.float32), None, None,
                         np.arange(3, dtype=np.uint32))
        r.addNodeHierarchyTemplate("quad", [(mesh, 0, 3, 0, None)])
        for k in range(n):
            node = r.addNodeHierarchy(0, "quad")
            r.setSemanticId(0, node, k + 1)
            r.transformations(0)[node] = S.translation(at[k, 0], at[k, 1], z[k])
        r.updateCamera(0, proj, S.identity())
        r.draw()
    assert_parity([compare_scene(gpu, cpu, pkg, 0)])
