"""Ambient occlusion of one caller image at the edges of the kernels' tiles
(16 x 16 and 32 x 32, 3 pixels of halo) and on both sample paths (offsets
within and beyond the 32-bit texel arithmetic), bit-exact against the oracle."""
import numpy as np
import pytest

import __graft_entry__ as graft
import scenarios as S
from oracle import hbao as H

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return graft.load_package()


def check(pkg, h, w, pad=0, ortho=False, **kw):
    import torch
    rng = np.random.default_rng(h * 1000 + w)
    proj = S.perspective(75.0, w / h, 0.05, 20.0)
    y, x = np.mgrid[0:h, 0:w]
    depth = (1.2 + 0.02 * x + 0.6 * np.abs(np.sin(y / 7.0)) + 0.5 * (x > w // 2)).astype(np.float32)
    depth[rng.uniform(size=depth.shape) < 0.04] = 0.0
    color = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    cfg = pkg.HbaoConfiguration().setRadius(kw.get("radius", 0.9)).setIntensity(kw.get("intensity", 1.1))
    cfg.setBias(kw.get("bias", 0.05)).setBlurSharpness(kw.get("blur_sharpness", 10.0))
    cfg.setNoBlur(kw.get("no_blur", False)).setUseSpecialBlur(kw.get("special_blur", False))
    if kw.get("cache_aware"):
        cfg.setAlgorithm(pkg.HbaoType.CacheAware)
    want = dict(radius=0.9, intensity=1.1)
    want.update(kw)
    dt = torch.zeros(h, w + pad, device="cuda")
    ct = torch.zeros(h, w + pad, 4, dtype=torch.uint8, device="cuda")
    dt[:, :w] = torch.from_numpy(depth)
    ct[:, :w] = torch.from_numpy(color)
    pkg.hbaoApply(cfg, proj, dt[:, :w], ct[:, :w])
    got = ct.cpu().numpy()
    assert np.array_equal(got[:, :w], H.hbao(color, depth, proj, H.config(**want)))
    assert not got[:, w:].any()  # nothing beyond the image


@pytest.mark.parametrize("variant", [{}, {"special_blur": True}, {"no_blur": True}, {"cache_aware": True},
                                     {"cache_aware": True, "special_blur": True}],
                         ids=["classic", "special", "no_blur", "cache", "cache_special"])
@pytest.mark.parametrize("size", [(1, 1), (2, 5), (16, 16), (15, 33), (31, 32), (33, 65), (70, 17)])
def test_tile_edges(pkg, size, variant):
    check(pkg, *size, pad=3, **variant)


@pytest.mark.parametrize("cache_aware", [False, True])
@pytest.mark.parametrize("radius", [300.0, 3e5, 1e7])
def test_offsets_beyond_the_image_and_beyond_32_bits(pkg, radius, cache_aware):
    # 40 rows, 75 degrees: 26 pixels per metre of radius at 1 m; 3e5 m puts
    # some of a pixel's offsets beyond 2^21 and others below.
    check(pkg, 40, 52, radius=radius, cache_aware=cache_aware)


@pytest.mark.parametrize("kw", [dict(bias=0.0), dict(bias=0.00005), dict(bias=0.6), dict(intensity=0.0),
                                dict(intensity=60.0), dict(blur_sharpness=0.0), dict(blur_sharpness=400.0)])
def test_parameters(pkg, kw):
    check(pkg, 37, 45, **kw)


@pytest.mark.parametrize("variant", [{}, {"special_blur": True}, {"cache_aware": True, "special_blur": True}],
                         ids=["classic", "special", "cache_special"])
def test_camera_image(pkg, variant):
    """A whole 640 x 480 image: a single operation that rounds otherwise (a
    fused one, say) changes a handful of its 307,200 pixels."""
    check(pkg, 480, 640, **variant)
