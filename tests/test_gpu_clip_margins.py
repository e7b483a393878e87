"""Chunks whose triangles the raster kernel takes for unclipped, at the edges of
that: boxes that touch the near plane to within the transform's rounding, far
from the origin, and triangles that leave the guard band of a wide or a
tall viewport.  Bit-exact against the oracle, which clips every triangle."""
import numpy as np
import pytest

import __graft_entry__ as graft
import scenarios as S
from parity import assert_parity, compare_scene

pytestmark = pytest.mark.gpu

f32 = np.float32
MODES = pytest.mark.parametrize("mode", [0, 1], ids=["per_scene", "batched"])


@pytest.fixture(scope="module")
def pkg():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return graft.load_package()


def _fma(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(f32)


def _row(m, r, v):
    """Row r of the vertex transform of points v [..., 3], in the kernel's order."""
    t = np.broadcast_to(m[..., 3, r], v.shape[:-1]).astype(f32)
    for k in range(3):
        t = _fma(np.broadcast_to(m[..., k, r], v.shape[:-1]).astype(f32), v[..., k], t)
    return t


def _grazing_triangle(rng, near, extent):
    """A camera and a triangle whose first vertex the vertex transform puts behind
    the near plane although the corner of its box, summed along the box's edges,
    lies before it.  (The sums differ by rounding; one try in a few hundred.)"""
    for _ in range(20000):
        eye = rng.uniform(-1.0, 1.0, 3) * extent
        fwd = rng.normal(size=3)
        fwd /= np.linalg.norm(fwd)
        right = np.cross(fwd, (0.0, 1.0, 0.0))
        right /= np.linalg.norm(right)
        up = np.cross(right, fwd)
        axes = np.stack([right, up, -fwd])
        view = np.eye(4)
        view[:3, :3], view[3, :3] = axes.T, -axes @ eye
        view = view.astype(f32)
        proj = S.perspective(0.25, 1.0, near, 10.0)
        pv = np.asarray(S.mul(proj, view), f32)
        # Step from the near plane along the box diagonal that leaves it fastest,
        # so that the nearest vertex is the nearest corner of the box.
        sign = np.where(fwd >= 0, 1.0, -1.0)
        a = (eye + fwd * near * (1.0 + rng.uniform(0.0, 1.2e-4))).astype(f32)
        size = 2.0 * near * np.tan(np.radians(0.25) / 2)
        b = (a + sign * np.abs(right) * size * rng.uniform(0.3, 1.0)).astype(f32)
        c = (a + sign * np.abs(up) * size * rng.uniform(0.3, 1.0)).astype(f32)
        v = np.stack([a, b, c])
        lo, hi = v.min(0), v.max(0)
        if not np.array_equal(np.where(fwd >= 0, lo, hi), a):
            continue
        z, w = _row(pv, 2, v), _row(pv, 3, v)
        if not (z[0] < -w[0] and (z[1:] > -w[1:]).all()):
            continue
        base = np.array([_row(pv, r, lo) for r in range(4)], f32)
        d = np.array([[pv[k, r] * (hi - lo)[k] for k in range(3)] for r in range(4)], f32)
        corners = []
        for k in range(8):
            q = base.copy()
            for bit, axis in ((4, 2), (2, 1), (1, 0)):
                if k & bit:
                    q = q + d[:, axis]
            corners.append(q)
        nz = np.array([q[2] / q[3] for q in corners], f32)
        if f32(0.5) * nz.min() + f32(0.5) > f32(1e-5):
            return proj, view, v
    raise AssertionError("no such triangle found")


@MODES
@pytest.mark.parametrize("extent", [10.0, 60.0])
def test_boxes_grazing_the_near_plane(pkg, mode, extent):
    from oracle.model import OracleRenderer
    rng = np.random.default_rng(int(extent))
    nx, ny = 8, 6
    cfg = pkg.RendererConfiguration().setTileSizeCount((32, 32), (nx, ny)).setDrawMode(pkg.DrawMode(mode))
    gpu, cpu = pkg.RendererStandalone(cfg), OracleRenderer((32, 32), (nx, ny))
    for s in range(nx * ny):
        proj, view, v = _grazing_triangle(rng, 0.01, extent)
        for r in (gpu, cpu):
            # Both windings: one of them faces the camera.
            m = r.addMesh(v, rng_colors(s), None, None, np.array([0, 1, 2, 0, 2, 1], np.uint32))
            r.addNodeHierarchyTemplate(f"t{s}", [(m, 0, 6, 0, None)])
            r.setSemanticId(s, r.addNodeHierarchy(s, f"t{s}"), 5)
            r.updateCamera(s, proj, view)
    gpu.draw()
    cpu.draw()
    assert_parity([compare_scene(gpu, cpu, pkg, s) for s in range(nx * ny)])


def rng_colors(seed):
    return np.random.default_rng(seed).uniform(0, 1, (3, 4)).astype(f32)


@MODES
@pytest.mark.parametrize("size", [(4096, 8), (8, 4096), (1600, 16), (16, 1600), (16384, 4)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
def test_triangles_beyond_the_guard_band(pkg, mode, size):
    """Triangles from 14400 to 16000 px left of or below the window's origin, some
    inside the band (which reaches 16384 px from the viewport's centre) and
    some not."""
    from oracle.model import OracleRenderer
    W, H = size
    rng = np.random.default_rng(W + H)
    n = 40
    proj = S.orthographic(2.0, 2.0, 0.1, 10.0)
    cfg = pkg.RendererConfiguration().setTileSizeCount(size, (1, 1)).setDrawMode(pkg.DrawMode(mode))
    gpu, cpu = pkg.RendererStandalone(cfg), OracleRenderer(size, (1, 1))
    across = 0 if W > H else 1
    px = np.zeros((n, 3, 2))
    lowest = max(W, H) / 2 - 16384.0
    px[:, 0, across] = rng.uniform(max(-15990.0, lowest - 1500.0), min(lowest + 500.0, -1.0), n)
    px[:, 0, 1 - across] = rng.uniform(-0.5, 1.5, n) * min(W, H)
    px[:, 1:, across] = rng.uniform(0.0, 1.0, (n, 2)) * max(W, H)
    px[:, 1:, 1 - across] = rng.uniform(-0.5, 1.5, (n, 2)) * min(W, H)
    pos = np.zeros((n, 3, 3), f32)
    pos[..., 0] = px[..., 0] / W * 2 - 1
    pos[..., 1] = px[..., 1] / H * 2 - 1
    pos[..., 2] = rng.uniform(-6.0, -2.0, (n, 3))
    colors = rng.uniform(0, 1, (3, 4)).astype(f32)
    for r in (gpu, cpu):
        for k in range(n):
            m = r.addMesh(pos[k], colors, None, None, np.array([0, 1, 2, 0, 2, 1], np.uint32))
            r.addNodeHierarchyTemplate(f"t{k}", [(m, 0, 6, 0, None)])
            r.setSemanticId(0, r.addNodeHierarchy(0, f"t{k}"), k + 1)
        r.updateCamera(0, proj, S.translation(0.0, 0.0, 0.0))
        r.draw()
    assert len(np.unique(cpu.semantic)) > 4  # the triangles are seen
    assert_parity([compare_scene(gpu, cpu, pkg, 0)])
