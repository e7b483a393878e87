"""unprojectDepthDevice on dense, strided, misaligned and narrow images: equal
to the host form, elements between the rows untouched."""
import numpy as np
import pytest

import __graft_entry__ as graft

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,stride,offset", [
    (1, 1, 1, 0), (3, 4, 4, 0), (5, 7, 7, 0), (5, 7, 7, 1), (64, 1024, 1024, 0), (64, 1024, 1028, 0),
    (33, 4099, 4099, 0), (33, 4099, 4104, 0), (33, 4099, 4105, 2), (70000, 3, 5, 0), (70000, 2, 4, 0), (1, 5, 9, 3)])
def test_layouts(rows, cols, stride, offset):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    pkg = graft.load_package()
    rng = np.random.default_rng(rows + cols)
    flat = rng.uniform(0.0, 1.0, offset + rows * stride + 4).astype(np.float32)
    flat[rng.uniform(size=flat.shape) < 0.1] = 1.0
    flat[:2] = (np.nan, np.inf)
    u = np.array([-1.0010005, -0.010005], np.float32)
    dev = torch.from_numpy(flat.copy()).cuda()
    image = dev[offset:offset + rows * stride].view(rows, stride)[:, :cols]
    pkg.unprojectDepthDevice(u, image)
    host = np.lib.stride_tricks.as_strided(flat[offset:], (rows, cols), (4 * stride, 4))
    with np.errstate(all="ignore"):
        pkg.unprojectDepth(u, host)
    got = dev.cpu().numpy()
    assert np.array_equal(np.isnan(got), np.isnan(flat))  # (a NaN's payload is the machine's)
    fine = ~np.isnan(flat)
    assert np.array_equal(got[fine].view(np.uint32), flat[fine].view(np.uint32))
