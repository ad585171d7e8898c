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


@pytest.mark.parametrize("shape", [(28, 28, 512, 64), (27, 27, 512, 48), (112, 112, 64, 32)])
def test_bnorm_sums_keep_their_digits_however_few_the_blocks(gpu, shape):
    """The sums of a channel in which one block has 35000 to 50000 terms, or eight have 400000, of inputs around zero, against 64 bits.  A sum of n terms in
    steps of sizes m_i errs by about 2^-24 / sqrt(3) of the partial sums' own spread per addition: 1.3e-7 of the result in the steps taken
    (four values, eight items, a thread's items, a warp, a block), and as measured; one running sum per thread errs by 2.2e-7 to 2.9e-7."""
    import torch
    nn, mat, _ = gpu
    c = shape[2]
    errors = {"mean": [], "dg": [], "dg_given": []}
    for seed in range(3):
        g = torch.Generator(device="cuda").manual_seed(seed)
        x, dy = (mat.empty(shape).normal_(generator=g) for _ in range(2))
        one = mat.zeros((c, 1)) + 1.0
        _, dg, _, mom = nn.vl_nnbnorm(x, one, one, dy, epsilon=1e-5)
        dg_given = nn.vl_nnbnorm(x, one, one, dy, epsilon=1e-5, moments=mom)[1]
        mean, var = x.double().mean(dim=(0, 1, 3)), (x.double() ** 2).mean(dim=(0, 1, 3))
        want = ((dy.double() * x.double()).sum(dim=(0, 1, 3)) - mean * dy.double().sum(dim=(0, 1, 3))) / (var - mean ** 2 + 1e-5).sqrt()
        for name, got, ref in (("mean", mom[:, 0], mean), ("dg", dg, want), ("dg_given", dg_given, want)):
            errors[name].append(float((got.double().reshape(-1) - ref).norm() / ref.norm()))
    for name, e in errors.items():
        assert np.mean(e) < 1.8e-7, (name, e)
