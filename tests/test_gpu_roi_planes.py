"""ROI pooling with the planes of four channels in shared memory: channel counts that leave a part of a group, ROI counts around the
parts that a block takes, bins that are empty, tiny or the whole map, an image without ROIs, a map that does not fit."""
import numpy as np
import pytest

from conftest import bit_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["max", "avg"])
@pytest.mark.parametrize("h,w,c,n,k,sub", [
    (13, 9, 5, 3, 65, (7, 7)),        # one channel left over, one ROI more than a part
    (38, 50, 130, 2, 64, (6, 5)),     # two left over
    (7, 31, 3, 1, 1, (1, 1)),         # one ROI
    (5, 6, 512, 2, 9, (3, 16)),       # more bins than pixels
    (130, 120, 2, 2, 40, (2, 2)),     # a map too large for the planes
])
def test_roipool_planes(gpu, oracle, h, w, c, n, k, sub, method):
    nn, mat, _ = gpu
    rng = np.random.default_rng(h * 31 + k)
    x = np.asfortranarray(np.round(rng.standard_normal((h, w, c, n)) * 3).astype(np.float32) / 2)      # many ties
    u1, v1 = rng.uniform(0, w, k), rng.uniform(0, h, k)
    rois = np.asfortranarray(np.stack([np.where(np.arange(k) % 3 == 0, 1, n), u1, v1, u1 + rng.uniform(0, w, k) * (np.arange(k) % 4),
                                       v1 + rng.uniform(0, h, k) * (np.arange(k) % 2)]).astype(np.float32))
    y = oracle.roipool_forward(x, rois, sub, 1.0, method)
    dy = np.asfortranarray(rng.integers(-8, 9, y.shape).astype(np.float32))
    xd, rd, dyd = (mat.from_numpy(v) for v in (x, rois, dy))
    assert bit_equal(mat.to_numpy(nn.vl_nnroipool(xd, rd, subdivisions=sub, method=method)), y)
    dx = nn.vl_nnroipool(xd, rd, dyd, subdivisions=sub, method=method)
    want = oracle.roipool_backward(x, rois, dy, sub, 1.0, method)
    if h * w < 12000:
        assert bit_equal(mat.to_numpy(dx), want)
    else:
        assert np.allclose(mat.to_numpy(dx), want, rtol=1e-5, atol=1e-5)       # (may be an atomic scatter)
