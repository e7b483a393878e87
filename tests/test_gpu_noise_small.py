"""Depth noise on batches of small images and of images that end in a short chunk,
bit-exact against the oracle: several images to a block (up to half its threads),
counts that leave the last block part empty, chunk by chunk and image by image."""
import numpy as np
import pytest

import __graft_entry__ as graft
from oracle import noise as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,w,h,tiles_x", [
    (1, 1, 1, 1), (1000, 1, 1, 7), (513, 8, 8, 32), (37, 8, 16, 5), (37, 43, 3, 5), (37, 127, 1, 5), (6, 16, 16, 6),
    (5, 257, 1, 2),             # without tables
    (230, 80, 60, 13),          # tables: 4800 pixels in chunks of 1024
    (900, 80, 60, 30),          # and of 4096
    (900, 33, 36, 9), (2100, 512, 1, 3)])
def test_small_images_match_oracle(count, w, h, tiles_x):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    graft.load_package()
    from habitat_sim_gb300 import noise
    rng = np.random.default_rng(w * 7 + h)
    rows = -(-count // tiles_x)
    pitch = w * tiles_x + 1
    plane = rng.uniform(0.2, 10.2, (rows * h, pitch)).astype(np.float32)
    src = torch.from_numpy(plane).cuda()
    dst = torch.full_like(src, -7.0)
    model = noise.load_model()
    m = noise.RedwoodNoiseModelGPUImpl(model, 0, 1.0, seed=99)
    m.simulate_tiles(src.data_ptr(), dst.data_ptr(), pitch, w, h, tiles_x, count)
    torch.cuda.synchronize()
    got = dst.cpu().numpy()
    table = N.normal_table()
    want = np.full_like(plane, -7.0)
    for i in range(count):
        y, x = i // tiles_x * h, i % tiles_x * w
        want[y:y + h, x:x + w] = N.redwood_f32(plane[y:y + h, x:x + w], model, 1.0, 99, 0, image=i, table=table)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), int((got != want).sum())
    m.close()
