"""Batch normalisation with one, two, four and eight blocks per channel, planes read in 16-byte and in 4-byte pieces, more and fewer
items than threads."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plane", [(4, 6), (5, 5), (56, 30), (1, 1)])
@pytest.mark.parametrize("c,n", [(450, 3), (230, 2), (120, 5), (3, 40)])
def test_bnorm_split(gpu, oracle, plane, c, n):
    nn, mat, _ = gpu
    rng = np.random.default_rng(c)
    x = np.asfortranarray(rng.standard_normal(plane + (c, n)).astype(np.float32) + 0.5)
    g, b = (np.asfortranarray(rng.standard_normal((c, 1)).astype(np.float32)) for _ in range(2))
    dy = np.asfortranarray(rng.standard_normal(x.shape).astype(np.float32))
    x64, g64, b64, dy64 = (v.astype(np.float64) for v in (x, g, b, dy))
    xd, gd, bd, dyd = (mat.from_numpy(v) for v in (x, g, b, dy))
    eps = 1e-2
    y, mom = nn.vl_nnbnorm(xd, gd, bd, epsilon=eps)
    ref = oracle.bnorm_forward(x64, g64, b64, eps)
    assert rel_l2(mat.to_numpy(y), ref[0]) < 1e-5 and rel_l2(mat.to_numpy(mom), ref[1]) < 1e-5
    got = nn.vl_nnbnorm(xd, gd, bd, dyd, epsilon=eps)
    want = oracle.bnorm_backward(x64, g64, b64, dy64, eps)
    scale = np.abs(dy).max() * np.abs(g).max() / np.sqrt(eps)
    assert np.abs(mat.to_numpy(got[0]) - want[0]).max() < 1e-5 * scale
    for i in (1, 2):
        assert np.abs(mat.to_numpy(got[i]).ravel() - want[i].ravel()).max() < 1e-4 * np.sqrt(plane[0] * plane[1] * n) * 4
    moments = nn.vl_nnbnorm(xd, gd, bd, dyd, epsilon=eps, moments=mom)
    assert np.abs(mat.to_numpy(moments[0]) - want[0]).max() < 1e-5 * scale
