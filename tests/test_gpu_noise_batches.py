"""Depth noise on batches large enough for the shared-memory tables and on odd
tile grids, bit-exact against the oracle: sizes at the edges of a chunk, of a
block and of the cell table, one-pixel axes, multipliers that carry samples
across the image, depths at the model's limits."""
import numpy as np
import pytest

import __graft_entry__ as graft
from oracle import noise as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,w,h,tiles_x,mult", [
    (70, 128, 120, 9, 1.0),     # tables: 1.08 M pixels
    (257, 64, 65, 16, 2.5),     # chunks that end inside a block
    (1, 2300, 1900, 1, 1.0),    # one large image, beyond the cell table
    (260, 1, 4095, 26, 1.0),    # one column, rows at the cell table's limit
    (1, 4096, 1, 1, 1.0), (3, 33, 31, 2, 1.0), (5, 1, 1, 5, 1.0), (2, 1025, 3, 1, 40.0)])
def test_tiles_match_oracle(count, w, h, tiles_x, mult):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    graft.load_package()
    from habitat_sim_gb300 import noise
    rng = np.random.default_rng(w * 7 + h)
    rows = -(-count // tiles_x)
    pitch = w * tiles_x + 3
    plane = rng.uniform(0.05, 10.5, (rows * h, pitch)).astype(np.float32)
    special = [0.0, 1e-38, 1e-31, 1e-4, 0.02, 9.999999, 10.0, 1e30, np.inf, np.nan, -0.5, 3.0]
    at = rng.uniform(size=plane.shape) < 0.05
    plane[at] = rng.choice(np.array(special, np.float32), at.sum())
    src = torch.from_numpy(plane).cuda()
    dst = torch.full_like(src, -7.0)
    model = noise.load_model()
    m = noise.RedwoodNoiseModelGPUImpl(model, 0, mult, seed=0xabcdef0123)
    m.set_state(0xabcdef0123, 1 << 33)
    m.simulate_tiles(src.data_ptr(), dst.data_ptr(), pitch, w, h, tiles_x, count)
    torch.cuda.synchronize()
    got = dst.cpu().numpy()
    table = N.normal_table()
    want = np.full_like(plane, -7.0)
    for i in range(count):
        y, x = i // tiles_x * h, i % tiles_x * w
        with np.errstate(all="ignore"):
            want[y:y + h, x:x + w] = N.redwood_f32(plane[y:y + h, x:x + w], model, mult, 0xabcdef0123, 1 << 33,
                                                   image=i, table=table)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), int((got != want).sum())
    assert m.get_state() == (0xabcdef0123, (1 << 33) + 1)
    m.close()


@pytest.mark.parametrize("count", [3, 70])
def test_close_walls_match_oracle(count):
    """Depths whose quotients lie beyond the output table and around the end
    of the estimate's range (131072 / 281 per metre: 2 mm)."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    graft.load_package()
    from habitat_sim_gb300 import noise
    w, h = 128, 120
    rng = np.random.default_rng(count)
    plane = np.exp(rng.uniform(np.log(1e-4), np.log(0.4), (count * h, w))).astype(np.float32)
    src = torch.from_numpy(plane).cuda()
    dst = torch.empty_like(src)
    model = noise.load_model()
    m = noise.RedwoodNoiseModelGPUImpl(model, 0, 1.0, seed=7)
    m.set_state(7, 5)
    m.simulate_tiles(src.data_ptr(), dst.data_ptr(), w, w, h, 1, count)
    torch.cuda.synchronize()
    table = N.normal_table()
    want = np.concatenate([N.redwood_f32(plane[i * h:(i + 1) * h], model, 1.0, 7, 5, image=i, table=table)
                           for i in range(count)])
    assert np.array_equal(dst.cpu().numpy().view(np.uint32), want.view(np.uint32))
    m.close()
