"""The tiled pooling kernels and the register-window LRN kernels at the sizes where their tiling can go wrong: strips of a plane that does not
fit a tile, several planes per block with a ragged last block, windows further apart than they are wide, padding on every
side; LRN with the channels split over threads and every window depth."""
import numpy as np
import pytest

from conftest import bit_equal, rel_l2

pytestmark = pytest.mark.gpu

POOLS = [((75, 130, 2, 3), (3, 3), 2, 0),                      # strips: a plane of 39 KB
         ((76, 131, 3, 1), (3, 3), 2, (1, 2, 2, 1)),           # the same with padding on every side
         ((5, 6, 3, 700), (3, 3), 2, (2, 1, 1, 2)),            # tiny planes, many per block
         ((301, 67, 3, 1), (2, 5), (1, 3), (1, 0, 2, 4)),      # long columns, overlapping in one dimension
         ((13, 13, 37, 41), (3, 3), 2, (0, 1, 0, 1)),          # several planes per block, ragged last block
         ((9, 11, 5, 300), (2, 2), 4, 0),                      # elements that no window covers
         ((6, 5, 700, 2), (5, 4), 1, (4, 3, 3, 2)),            # windows larger than half the plane, stride 1
         ((4000, 3, 1, 2), (3, 2), (2, 1), (1, 1, 0, 0)),      # a strip of one or two columns
         ((12000, 2, 1, 1), (3, 2), (2, 1), 0)]                # too long for a tile: the generic kernels


@pytest.mark.parametrize("method", ["max", "avg"])
@pytest.mark.parametrize("case", range(len(POOLS)))
def test_pool_tiles_vs_oracle(gpu, oracle, case, method):
    nn, mat, ctx = gpu
    shape, pool, stride, pad = POOLS[case]
    two = lambda v: (v, v) if np.isscalar(v) else v      # noqa: E731
    four = lambda v: (v,) * 4 if np.isscalar(v) else v   # noqa: E731
    rng = np.random.default_rng(case)
    x = np.asfortranarray(np.round(rng.standard_normal(shape) * 4).astype(np.float32) / 4)       # many ties
    y = oracle.pool_forward(x, pool, two(stride), four(pad), method)
    dy = np.asfortranarray(rng.standard_normal(y.shape).astype(np.float32))
    dx = oracle.pool_backward(x, dy, pool, two(stride), four(pad), method)
    xd, dyd = mat.from_numpy(x), mat.from_numpy(dy)
    kw = dict(stride=stride, pad=pad, method=method)
    assert bit_equal(mat.to_numpy(nn.vl_nnpool(xd, pool, **kw)), y)
    assert bit_equal(mat.to_numpy(nn.vl_nnpool(xd, pool, dyd, **kw)), dx)
    assert bit_equal(mat.to_numpy(nn.vl_nnpool(xd, pool, dyd, through_relu=True, **kw)), np.where(x > 0, dx, np.float32(0)))


@pytest.mark.parametrize("prm", [[5, 1.0, 2e-5, 0.75], [3, 2.0, 0.1, 0.75], [7, 1.0, 0.05, 0.5], [9, 1.5, 1e-2, 0.75]])
@pytest.mark.parametrize("shape", [(55, 55, 96, 2), (3, 5, 130, 2), (1, 1, 7, 300), (13, 13, 4, 3)])
def test_lrn_windows_vs_oracle(gpu, oracle, shape, prm):
    nn, mat, ctx = gpu
    rng = np.random.default_rng(shape[2])
    x = np.asfortranarray(rng.standard_normal(shape).astype(np.float32) * 3)
    dy = np.asfortranarray(rng.standard_normal(shape).astype(np.float32))
    y = oracle.lrn_forward(x.astype(np.float64), prm)
    dx = oracle.lrn_backward(x.astype(np.float64), prm, dy.astype(np.float64))
    xd = mat.from_numpy(x)
    assert rel_l2(mat.to_numpy(nn.vl_nnnormalize(xd, prm)), y) < 1e-6
    got = mat.to_numpy(nn.vl_nnnormalize(xd, prm, mat.from_numpy(dy)))
    assert rel_l2(got, dx) < 1e-6
    assert bit_equal(mat.to_numpy(nn.vl_nnnormalize(xd, prm, mat.from_numpy(dy), through_relu=True)), np.where(x > 0, got, np.float32(0)))
