"""The general gather of the tensor-memory convolution kernel against the CPU checker: channel counts that are no multiple of
32 (every unit size), filter groups, and strided data gradients in both forms -- one problem per residue class of the input pixel, and
the shuffled form for few channels -- with dilation, uneven padding, classes that no filter tap reaches, and the ReLU mask."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# x, filters (FH, FW, C / groups, K), stride, pad (top bottom left right), dilate
CASES = {
    "unit1_c1": ((17, 15, 1, 3), (5, 4, 1, 20), (1, 1), (2, 1, 0, 2), (1, 1)),
    "unit3_rgb_11x11_s4": ((67, 59, 3, 3), (11, 11, 3, 24), (4, 4), (0, 0, 0, 0), (1, 1)),         # shuffled: 48 columns, ragged classes
    "unit4_c20": ((12, 12, 20, 7), (5, 5, 20, 50), (1, 1), (0, 0, 0, 0), (1, 1)),
    "unit16_c48": ((13, 9, 48, 5), (3, 3, 48, 70), (2, 1), (1, 1, 0, 1), (1, 1)),
    "unit32_tail_c90": ((29, 22, 90, 3), (3, 3, 90, 150), (2, 2), (1, 1, 1, 1), (1, 1)),           # classes of 4, 2, 2, 1 taps
    "one_by_one_s2": ((15, 16, 64, 4), (1, 1, 64, 96), (2, 2), (0, 0, 0, 0), (1, 1)),              # three classes without a tap
    "one_by_one_s2_narrow": ((14, 13, 8, 4), (1, 1, 8, 40), (2, 2), (0, 0, 0, 0), (1, 1)),         # the same, shuffled
    "s3_f2": ((16, 17, 32, 2), (2, 2, 32, 33), (3, 3), (0, 1, 1, 0), (1, 1)),                      # classes without a tap in each dimension
    "s2_dilate2": ((20, 18, 24, 2), (3, 3, 24, 40), (2, 2), (2, 2, 2, 2), (2, 2)),                 # taps reach even positions only
    "s3_dilate2_uneven": ((21, 23, 40, 2), (4, 3, 40, 36), (3, 2), (3, 0, 1, 4), (2, 3)),
    "pad_beyond_filter": ((9, 10, 33, 2), (2, 3, 33, 34), (2, 2), (4, 4, 5, 3), (1, 1)),
    "groups2": ((14, 13, 96, 3), (5, 5, 48, 128), (1, 1), (2, 2, 2, 2), (1, 1)),
    "groups2_wide_s2": ((15, 11, 80, 2), (3, 3, 40, 300), (2, 2), (1, 1, 1, 1), (1, 1)),           # several column tiles per group
    "groups4_narrow": ((12, 12, 24, 4), (3, 3, 6, 20), (1, 2), (1, 1, 1, 1), (1, 1)),
    "many_tiles_s2": ((96, 90, 40, 6), (3, 3, 40, 72), (2, 2), (1, 1, 1, 1), (1, 1)),              # more tiles than SMs: CTAs shared out
    "two_channels_5x3": ((71, 29, 2, 3), (5, 3, 2, 30), (1, 1), (4, 0, 1, 2), (1, 1)),             # tiled CUDA-core data gradient, ragged quads and chunks
    "four_channels_3x5": ((33, 66, 4, 2), (3, 5, 4, 9), (1, 1), (0, 2, 2, 2), (1, 1)),
    "s5_falls_back": ((23, 24, 8, 2), (3, 3, 8, 16), (5, 5), (1, 1, 1, 1), (2, 2)),                # 25 classes: more than one launch holds
}


@pytest.mark.parametrize("precision,tol", [(0, 1e-5), (1, 2e-3)])
@pytest.mark.parametrize("case", sorted(CASES))
def test_general_gather_vs_oracle(gpu, oracle, case, precision, tol):
    nn, mat, ctx = gpu
    xs, fs, stride, pad, dilate = CASES[case]
    kw = dict(stride=stride, pad=pad, dilate=dilate)
    rng = np.random.default_rng(sum(xs) + 7 * sum(fs))
    x = np.asfortranarray(np.maximum(rng.standard_normal(xs), -0.3).astype(np.float32))
    f = np.asfortranarray((rng.standard_normal(fs) * np.sqrt(2.0 / np.prod(fs[:3]))).astype(np.float32))
    b = (rng.standard_normal(fs[3]) * 0.1).astype(np.float32)
    x64, f64, b64 = (a.astype(np.float64) for a in (x, f, b))
    y_ref = oracle.conv_forward(x64, f64, b64, **kw)
    dy = np.asfortranarray(rng.standard_normal(y_ref.shape).astype(np.float32))
    dx_ref, df_ref, db_ref = oracle.conv_backward(x64, f64, dy.astype(np.float64), **kw)
    xd, fd, bd, dyd = (mat.from_numpy(a) for a in (x, f, b, dy))
    ctx.set_precision(precision)
    try:
        y = nn.vl_nnconv(xd, fd, bd, ctx=ctx, **kw)
        yr = nn.vl_nnconv(xd, fd, bd, relu=True, ctx=ctx, **kw)
        dx, df, db = nn.vl_nnconv(xd, fd, bd, dyd, ctx=ctx, **kw)
        dxm = nn.vl_nnconv(xd, fd, bd, dyd, through_relu=True, no_der_filters=True, no_der_biases=True, ctx=ctx, **kw)[0]
        assert ctx.device_status() == 0
        for got, want, name in ((y, y_ref, "y"), (dx, dx_ref, "dx"), (df, df_ref, "df"), (db, db_ref, "db")):
            assert rel_l2(mat.to_numpy(got).ravel(), np.asarray(want).ravel()) < tol, name
        assert np.array_equal(mat.to_numpy(yr), np.maximum(mat.to_numpy(y), 0))
        assert rel_l2(mat.to_numpy(dxm), np.where(x > 0, dx_ref, 0)) < tol
    finally:
        ctx.set_precision(0)


# the fully connected forward pass for few images, and reductions cut into ranges because the output tiles are few
FEW = {
    "fc_n1": ((7, 7, 64, 1), (7, 7, 64, 130), 0), "fc_n3_ragged": ((5, 3, 23, 3), (5, 3, 23, 1201), 0), "fc_n8": ((1, 1, 512, 8), (1, 1, 512, 67), 0),
    "few_tiles_plain": ((14, 14, 256, 1), (3, 3, 256, 160), 1), "few_tiles_windows": ((32, 16, 64, 1), (5, 5, 64, 48), 2),
    "few_tiles_general": ((8, 8, 50, 5), (5, 5, 50, 70), 0),
    "fc_n130_16_row_tiles": ((4, 4, 128, 130), (4, 4, 128, 4096), 0), "fc_below_the_line": ((4, 4, 128, 128), (4, 4, 128, 128), 0),
    "fc_dgrad_parts": ((1, 1, 300, 33), (1, 1, 300, 1000), 0),
}


@pytest.mark.parametrize("precision,tol", [(0, 1e-5), (1, 2e-3)])
@pytest.mark.parametrize("case", sorted(FEW))
def test_few_images_and_few_tiles_vs_oracle(gpu, oracle, case, precision, tol):
    nn, mat, ctx = gpu
    xs, fs, pad = FEW[case]
    rng = np.random.default_rng(len(case))
    x = np.asfortranarray(np.maximum(rng.standard_normal(xs), -0.3).astype(np.float32))
    f = np.asfortranarray((rng.standard_normal(fs) * np.sqrt(2.0 / np.prod(fs[:3]))).astype(np.float32))
    b = (rng.standard_normal(fs[3]) * 0.1).astype(np.float32)
    x64, f64, b64 = (a.astype(np.float64) for a in (x, f, b))
    kw = dict(pad=(pad,) * 4)
    y_ref = oracle.conv_forward(x64, f64, b64, **kw)
    dy = np.asfortranarray(rng.standard_normal(y_ref.shape).astype(np.float32))
    dx_ref, df_ref, db_ref = oracle.conv_backward(x64, f64, dy.astype(np.float64), **kw)
    xd, fd, bd, dyd = (mat.from_numpy(a) for a in (x, f, b, dy))
    ctx.set_precision(precision)
    try:
        y, yr = nn.vl_nnconv(xd, fd, bd, ctx=ctx, **kw), nn.vl_nnconv(xd, fd, bd, relu=True, ctx=ctx, **kw)
        dx, df, db = nn.vl_nnconv(xd, fd, bd, dyd, ctx=ctx, **kw)
        dxm = nn.vl_nnconv(xd, fd, bd, dyd, through_relu=True, ctx=ctx, **kw)[0]
        assert ctx.device_status() == 0
        for got, want, name in ((y, y_ref, "y"), (dx, dx_ref, "dx"), (df, df_ref, "df"), (db, db_ref, "db")):
            assert rel_l2(mat.to_numpy(got).ravel(), np.asarray(want).ravel()) < tol, name
        assert np.array_equal(mat.to_numpy(yr), np.maximum(mat.to_numpy(y), 0))
        assert rel_l2(mat.to_numpy(dxm), np.where(x > 0, dx_ref, 0)) < tol
    finally:
        ctx.set_precision(0)


@pytest.mark.parametrize("stride,k", [(2, 524321)])
def test_mask_and_bias_survive_a_refused_launch(gpu, stride, k):
    """A reduction of more than 65535 k-blocks (4 taps of k filters) is refused by the general gather and taken by the next kernel, which
    fuses neither the ReLU mask nor the bias of a transposed convolution: both are then applied by passes of their own, so the results
    equal the unfused ones bit for bit."""
    import torch
    nn, mat, ctx = gpu
    ctx.set_precision(0)
    g = torch.Generator(device="cuda").manual_seed(k)
    normal = lambda *s: mat.empty(s).normal_(generator=g)       # noqa: E731
    x, f = normal(4, 4, 8, 1), normal(3, 3, 8, k)
    side = 2 if stride == 2 else 4
    dy = normal(side, side, k, 1)
    kw = dict(stride=stride, pad=1, no_der_filters=True, no_der_biases=True, ctx=ctx)
    dx = nn.vl_nnconv(x, f, None, dy, **kw)[0]
    dxm = nn.vl_nnconv(x, f, None, dy, through_relu=True, **kw)[0]
    assert bool((dx != 0).all()) and torch.equal(dxm, torch.where(x > 0, dx, torch.zeros_like(dx)))
    b = normal(1, 8)
    crop = (1, 0, 1, 0) if stride == 2 else 1
    y = nn.vl_nnconvt(dy, f, None, upsample=stride, crop=crop, ctx=ctx)
    yb = nn.vl_nnconvt(dy, f, b, upsample=stride, crop=crop, ctx=ctx)
    assert torch.equal(yb, y + b.reshape(1, 1, 8, 1))
    assert ctx.device_status() == 0


def test_data_gradient_of_a_very_long_reduction(gpu):
    """65565 k-blocks in one output tile (9 taps of 233101 filters): longer than the bound of a single pipeline wait, which the warps without a
    share of the gather spend in one wait for the whole reduction.  Against 64-bit sums; the bound: the small terms of the split (2^-11 of the
    result) are added with truncation 2 * 4 * 65565 times, 2^-11 * 2^-24 * 524520 = 1.5e-5, the sums of chains far less."""
    import torch
    nn, mat, ctx = gpu
    ctx.set_precision(0)
    k = 233101
    g = torch.Generator(device="cuda").manual_seed(k)
    f = mat.empty((3, 3, 8, k)).normal_(generator=g)
    dy = mat.empty((4, 4, k, 1)).normal_(generator=g)
    x = mat.empty((4, 4, 8, 1)).normal_(generator=g)
    dx = nn.vl_nnconv(x, f, None, dy, pad=1, no_der_filters=True, no_der_biases=True, ctx=ctx)[0]
    dxm = nn.vl_nnconv(x, f, None, dy, pad=1, no_der_filters=True, no_der_biases=True, through_relu=True, ctx=ctx)[0]
    assert ctx.device_status() == 0
    want = torch.zeros(6, 6, 8, dtype=torch.float64, device="cuda")             # the padded plane
    f64, dy64 = f.double(), dy[..., 0].double()
    for a in range(3):
        for b in range(3):
            want[a:a + 4, b:b + 4] += dy64.reshape(16, k).matmul(f64[a, b].T).reshape(4, 4, 8)
    want = want[1:5, 1:5]
    assert float((dx[..., 0].double() - want).norm() / want.norm()) < 2e-5
    assert torch.equal(dxm, torch.where(x > 0, dx, torch.zeros_like(dx)))


# x, filters, stride, pad, groups, bounds of (y, dx, df), None: not this test's
NEAR = {
    "groups_short": ((30, 31, 48, 6), (3, 3, 12, 64), 1, 1, (1.6e-7, 1.6e-7, 2.4e-7)),           # 108 and 144 products
    "groups_512_products": ((9, 9, 96, 3), (1, 1, 48, 1024), 1, 0, (1.6e-7, 4.2e-7, None)),         # 48; 512: the first two-block chains
    "groups_511_products": ((9, 9, 14, 3), (1, 1, 7, 1022), 1, 0, (1.6e-7, 1.7e-7, None)),         # 7; 511: the last one-block chains
    "groups_small_batch": ((13, 13, 384, 1), (3, 3, 192, 384), 1, 1, (4.2e-7, 4.2e-7, 1.6e-7)),       # ranges of 85 pixels
    "groups_batch_8": ((13, 13, 384, 8), (3, 3, 192, 256), 1, 1, (4.2e-7, 4.2e-7, 3.6e-7)),       # of 451
    "strided": ((40, 41, 33, 5), (5, 5, 33, 70), 3, 2, (4.2e-7, 1.6e-7, None)),              # 280 and fewer products per class
    "fc_256_images": ((1, 1, 4096, 256), (1, 1, 4096, 4096), 1, 0, (4.3e-7, None, 4.2e-7)),        # the fine form of the tensor-memory kernel
    "fc_64_images": ((1, 1, 4096, 64), (1, 1, 4096, 4096), 1, 0, (None, None, 1.6e-7)),
}


@pytest.mark.parametrize("case", sorted(NEAR))
def test_default_arithmetic_is_as_near_as_the_kernels_before(gpu, case):
    """Strided and grouped layers came from the CUDA-core kernel (exact products, about 1.7e-8 * sqrt(products) off the exact sums), the fully connected ones from
    chains of large terms alone (6.4e-7): what took their place is no further off.  Chains of 1, 2 and 4 k-blocks measured 1.4e-7, 3.1 to 3.9e-7
    (gathered operand in tensor memory) or 2.0 and 3.2e-7 (both in shared memory); the bounds leave a tenth."""
    import torch
    import torch.nn.functional as F
    nn, mat, ctx = gpu
    ctx.set_precision(0)
    xs, fs, stride, pad, bounds = NEAR[case]
    g = torch.Generator(device="cuda").manual_seed(5)
    x, f = mat.empty(xs).normal_(generator=g), mat.empty(fs).normal_(0.0, float(np.sqrt(2.0 / np.prod(fs[:3]))), generator=g)
    X, W = (t.permute(3, 2, 1, 0).double().requires_grad_() for t in (x, f))
    Y = F.conv2d(X, W, stride=stride, padding=pad, groups=xs[2] // fs[2])
    y = nn.vl_nnconv(x, f, None, stride=stride, pad=pad, ctx=ctx)
    dy = mat.empty(tuple(y.shape)).normal_(generator=g)
    dx, df, _ = nn.vl_nnconv(x, f, None, dy, stride=stride, pad=pad, ctx=ctx)
    Y.backward(dy.permute(3, 2, 1, 0).double())
    for got, want, bound, name in zip((y, dx, df), (Y.detach(), X.grad, W.grad), bounds, ("y", "dx", "df")):
        if bound is not None:
            err = float((got.permute(3, 2, 1, 0).double() - want).norm() / want.norm())
            assert err < bound, (name, err)
    assert ctx.device_status() == 0
