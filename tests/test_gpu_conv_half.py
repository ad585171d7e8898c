"""Backward contractions on scaled half-precision operands (conv_half.cu): data gradients of split chunks, filter gradients with the images
along the reduction, both against float64, and what the powers of two have to keep: any magnitude, infinities in their own column or pixel.

Bound: an operand is off by 2^-22 of itself at most, a product by 2^-21, an fp32 sum of a k-block's 12 MMAs by about 2^-21 of itself; random signs leave
1.2e-7 to 6e-7 of the result's norm at every size measured, 1e-6 is asked for.  VLB_PRECISION_TF32 rounds the operands to 11 bits (2^-12 each on average
half of that): 2.4e-4, 5e-4 is asked for.  A filter gradient too small for these kernels comes from tc_gemm_kernel, whose plain TF32 operands are cut off
instead of rounded: each is 0 to 2^-10 of itself too small, 3.6e-4 on average (the mean of 2^-11 / mantissa), the product twice that, all in one direction; 1e-3
is asked for there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (H, W, C, N), (FH, FW, C/G, K), stride, pad, dilate
CASES = [((16, 16, 64, 8), (3, 3, 64, 64), 1, 1, 1),           # one block of 64 channels, 64 columns
         ((16, 16, 64, 8), (3, 3, 64, 16), 1, 1, 1),           # 16 filters: 16 of 64 places of a k-block
         ((9, 11, 65, 16), (3, 3, 65, 129), 1, 1, 1),          # one more than a block of channels, than a column tile
         ((8, 7, 128, 64), (3, 3, 128, 128), 1, 1, 1),         # whole tiles; 64 images: one pixel per k-block
         ((13, 13, 48, 70), (5, 5, 24, 96), 1, 2, 1),          # two filter groups, six images more than a group of 64
         ((14, 10, 96, 33), (3, 3, 96, 43), 2, 1, 1),          # stride 2; 43 channels filled up to 64
         ((12, 9, 32, 13), (3, 3, 32, 200), 1, 2, 2),          # dilation; 13 images: groups of eight
         ((7, 5, 70, 5), (1, 1, 70, 300), 1, 0, 1),            # 1x1, three column tiles
         ((6, 31, 40, 24), (3, 2, 40, 80), (1, 3), (0, 1, 1, 0), 1),
         ((4, 4, 512, 3), (3, 3, 512, 512), 1, 1, 1)]          # few tiles, long reduction: cut into ranges


def reference(x, f, dy, stride, pad, dilate):
    import torch
    import torch.nn.functional as F
    st = (stride, stride) if np.isscalar(stride) else stride
    p = (pad,) * 4 if np.isscalar(pad) else pad
    groups = x.shape[2] // f.shape[2]
    X, W = (t.permute(3, 2, 1, 0).double().requires_grad_() for t in (x, f))
    # (image, channel, column, row): torch's last dimension is the row here
    Y = F.conv2d(F.pad(X, p), W, stride=(st[1], st[0]), dilation=dilate, groups=groups)
    if dy is None:
        return tuple(Y.permute(3, 2, 1, 0).shape)
    Y.backward(dy.permute(3, 2, 1, 0).double())
    return X.grad.permute(3, 2, 1, 0), W.grad.permute(3, 2, 1, 0), dy.double().sum((0, 1, 3))


def inputs(mat, case):
    import torch
    xs, fs, stride, pad, dilate = CASES[case]
    g = torch.Generator(device="cuda").manual_seed(500 + case)
    x, f = mat.empty(xs).normal_(generator=g), mat.empty(fs).normal_(0.0, float((2.0 / np.prod(fs[:3])) ** 0.5), generator=g)
    dy = mat.empty(reference(x, f, None, stride, pad, dilate)).normal_(generator=g)
    return x, f, dy, dict(stride=stride, pad=pad, dilate=dilate)


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


@pytest.mark.parametrize("precision,bound", [(0, 1e-6), (1, 5e-4)])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_gradients_against_float64(gpu, case, precision, bound):
    import torch
    nn, mat, ctx = gpu
    x, f, dy, kw = inputs(mat, case)
    b = mat.zeros((1, f.shape[3]))
    dxr, dfr, dbr = reference(x, f, dy, **kw)
    ctx.set_precision(precision)
    lib = ctx.lib
    try:
        for switch in (0, 16):              # 16: the images along the reduction wherever they can be
            ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, switch))
            dx, df, db = nn.vl_nnconv(x, f, b, dy, ctx=ctx, **kw)
            again = nn.vl_nnconv(x, f, b, dy, ctx=ctx, **kw)
            assert ctx.device_status() == 0
            assert rel(dx, dxr) < bound and rel(db.reshape(-1), dbr) < 1e-6, switch
            assert rel(df, dfr) < (1e-3 if precision == 1 and switch == 0 else bound), switch
            assert all(torch.equal(a, c) for a, c in zip((dx, df, db), again))          # run to run identical
    finally:
        ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))
        ctx.set_precision(0)


@pytest.mark.parametrize("case", [0, 2, 3, 5])
@pytest.mark.parametrize("ex,ef,ed", [(40, -30, 20), (-60, 0, 50), (0, -20, -80), (70, 10, 30)])
def test_powers_of_two_change_nothing_but_the_scale(gpu, case, ex, ef, ed):
    """Operands times powers of two: the result times their product, bit for bit (as long as it has a normal exponent) -- also where the factor of a k-block has not."""
    import torch
    nn, mat, ctx = gpu
    x, f, dy, kw = inputs(mat, case)
    lib = ctx.lib
    try:
        for switch in (0, 16):
            ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, switch))
            dx, df, _ = nn.vl_nnconv(x, f, None, dy, ctx=ctx, **kw)
            dx2, df2, _ = nn.vl_nnconv(mat.as_mat(x * 2.0 ** ex), mat.as_mat(f * 2.0 ** ef), None, mat.as_mat(dy * 2.0 ** ed), ctx=ctx, **kw)
            small = 2.0 ** -10                # (what is left where a sum almost cancels may be subnormal on the way when scaled)
            for a, c, e in ((dx, dx2, ef + ed), (df, df2, ex + ed)):
                keep = a.abs() > small
                assert torch.equal((a.double() * 2.0 ** e)[keep], c.double()[keep]), (switch, e)
    finally:
        ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))


@pytest.mark.parametrize("case", [0, 3, 6])
def test_values_that_are_not_finite_stay_where_they_are(gpu, case):
    import torch
    nn, mat, ctx = gpu
    x, f, dy, kw = inputs(mat, case)
    lib = ctx.lib
    try:
        for switch in (0, 16):
            ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, switch))
            dx, df, _ = nn.vl_nnconv(x, f, None, dy, ctx=ctx, **kw)
            # a filter bank with an infinity in one channel: that channel's derivative only
            f2 = f.clone()
            f2[0, 0, 3, 1] = float("inf")
            dxf, _, _ = nn.vl_nnconv(x, mat.as_mat(f2), None, dy, no_der_filters=True, ctx=ctx, **kw)
            assert not torch.isfinite(dxf[:, :, 3]).all()
            other = [c for c in range(x.shape[2]) if c != 3]
            assert torch.equal(dxf[:, :, other], dx[:, :, other])
            # a derivative that is not a number: its filter's gradient only; the pixels it reaches only
            dy2 = dy.clone()
            dy2[2, 2, 5, 1] = float("nan")
            dxd, dfd, _ = nn.vl_nnconv(x, f, None, mat.as_mat(dy2), ctx=ctx, **kw)
            other = [k for k in range(f.shape[3]) if k != 5]
            assert torch.isnan(dfd[:, :, :, 5]).any() and torch.equal(dfd[:, :, :, other], df[:, :, :, other])
            assert torch.isnan(dxd[:, :, :, 1]).any() and torch.equal(dxd[:, :, :, 0], dx[:, :, :, 0])
            # an input that is infinite: its channel's rows only
            x2 = x.clone()
            x2[1, 1, 7, 0] = float("inf")
            _, dfx, _ = nn.vl_nnconv(mat.as_mat(x2), f, None, dy, no_der_data=True, ctx=ctx, **kw)
            other = [c for c in range(x.shape[2]) if c != 7]
            assert not torch.isfinite(dfx[:, :, 7]).all() and torch.equal(dfx[:, :, other], df[:, :, other])
    finally:
        ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("shape", [(10, 10), (14, 12), (8, 12)])
@pytest.mark.parametrize("images", [4, 8])
def test_a_filter_tap_knows_nothing_of_columns_that_it_does_not_read(gpu, images, shape, value):
    """The last column of a padded plane, which the first filter column never reads -- also where the plane's pixels are filled up to whole k-blocks."""
    import torch
    nn, mat, ctx = gpu
    g = torch.Generator(device="cuda").manual_seed(900 + images)
    x, f, dy = (mat.empty(s).normal_(generator=g) for s in (shape + (32, images), (3, 3, 32, 48), shape + (48, images)))
    x2 = x.clone()
    x2[5, shape[1] - 1, 7, images - 1] = value
    lib = ctx.lib
    try:
        for switch in (0, 16):
            ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, switch))
            _, df, _ = nn.vl_nnconv(x, f, None, dy, pad=1, no_der_data=True, ctx=ctx)
            _, df2, _ = nn.vl_nnconv(mat.as_mat(x2), f, None, dy, pad=1, no_der_data=True, ctx=ctx)
            assert torch.equal(df2[:, 0], df[:, 0]), switch
            assert not torch.isfinite(df2[:, 1:, 7]).any(), switch
    finally:
        ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))


@pytest.mark.parametrize("value", [float("inf"), float("nan"), 2.0 ** 60])
@pytest.mark.parametrize("images", [8, 16, 32, 64])
@pytest.mark.parametrize("stride", [1, 2])
def test_a_filter_tap_knows_nothing_of_rows_that_it_does_not_read(gpu, stride, images, value):
    """Stride 1: the last row of a padded plane, which the first filter row never reads.  Stride 2: an odd row, which the middle one never reads.  8, 16 and
    32 images: k-blocks of 8, 4 and 2 rows.  What a tap's sums are made of has not changed, so neither may one bit of them."""
    import torch
    nn, mat, ctx = gpu
    g = torch.Generator(device="cuda").manual_seed(600 + images)
    x, f = mat.empty((14, 12, 32, images)).normal_(generator=g), mat.empty((3, 3, 32, 48)).normal_(generator=g)
    kw = dict(stride=stride, pad=1)
    dy = mat.empty(reference(x, f, None, stride, 1, 1)).normal_(generator=g)
    row, tap = (13, 0) if stride == 1 else (5, 1)
    x2 = x.clone()
    x2[row, 4, 7, 2] = value
    lib = ctx.lib
    try:
        for switch in (0, 16):
            ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, switch))
            _, df, _ = nn.vl_nnconv(x, f, None, dy, no_der_data=True, ctx=ctx, **kw)
            _, df2, _ = nn.vl_nnconv(mat.as_mat(x2), f, None, dy, no_der_data=True, ctx=ctx, **kw)
            assert torch.equal(df2[tap], df[tap]), switch
            read = [t for t in range(3) if t != tap and (stride == 1 or t != 1)]
            assert not torch.equal(df2[read, :, 7], df[read, :, 7]), switch
            other = [c for c in range(32) if c != 7]
            assert torch.equal(df2[:, :, other], df[:, :, other]), switch
    finally:
        ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))


# input, filters, images whose tiles are 16, 32, 64 and two of 128 columns wide: K filters for the filter gradient, C channels for the data gradient
SMALL = [((8, 8, 64, 8), (3, 3, 64, 64)), ((8, 12, 32, 64), (3, 3, 32, 200)), ((14, 14, 16, 16), (1, 1, 16, 32)), ((10, 10, 200, 32), (3, 3, 200, 16)),
         ((9, 7, 40, 24), (3, 3, 40, 96)), ((8, 8, 128, 5), (3, 3, 128, 128))]


def columns_apart(got, want, axis, bound):
    got, want = (t.double().movedim(axis, 0).reshape(t.shape[axis], -1) for t in (got, want))
    off = (got - want).norm(dim=1) / want.norm(dim=1)
    assert float(off.max()) < bound, (int(off.argmax()), float(off.max()))


@pytest.mark.parametrize("precision,bound", [(0, 1e-6), (1, 5e-4)])
@pytest.mark.parametrize("e", [-15, -18, -30, -44, -70, -100])
@pytest.mark.parametrize("case", range(len(SMALL)))
def test_a_filter_or_channel_is_as_exact_beside_far_larger_ones(gpu, case, e, precision, bound):
    """Filters with small derivatives, channels with small weights, among ordinary ones: each one's gradient by itself against float64, within the bounds of
    ordinary ones.  At 2^-15 a column still has the tile's power of two, beyond 2^-16 its own."""
    nn, mat, ctx = gpu
    import torch
    xs, fs = SMALL[case]
    g = torch.Generator(device="cuda").manual_seed(700 + case)
    x, f = mat.empty(xs).normal_(generator=g), mat.empty(fs).normal_(generator=g)
    dy = mat.empty(reference(x, f, None, 1, 1, 1)).normal_(generator=g)
    dy[:, :, 1::3] *= 2.0 ** e
    f[:, :, 2::5] *= 2.0 ** e
    dxr, dfr, _ = reference(x, f, dy, 1, 1, 1)
    lib = ctx.lib
    ctx.set_precision(precision)
    try:
        for switch in (0, 16):
            ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, switch))
            dx, df, _ = nn.vl_nnconv(x, f, None, dy, pad=1, ctx=ctx)
            columns_apart(df, dfr, 3, 1e-3 if precision == 1 and switch == 0 else bound)
            # (16 filters fill too little of a block of 64: the gather that splits as it goes, whose plain TF32 filters are cut off)
            columns_apart(dx, dxr, 2, 1e-3 if precision == 1 and fs[3] == 16 else bound)
        assert ctx.device_status() == 0
    finally:
        ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))
        ctx.set_precision(0)


@pytest.mark.parametrize("precision,bound", [(0, 1e-6), (1, 5e-4)])
@pytest.mark.parametrize("e", [-15, -18, -30, -44, -70, -100])
@pytest.mark.parametrize("images", [32, 64, 160])
def test_an_image_is_as_exact_beside_far_larger_ones(gpu, images, e, precision, bound):
    """Fully connected: images, and filters, whose derivatives are small among ordinary ones."""
    nn, mat, ctx = gpu
    import torch
    g = torch.Generator(device="cuda").manual_seed(800 + images)
    x, f = mat.empty((4, 4, 512, images)).normal_(generator=g), mat.empty((4, 4, 512, 1024)).normal_(generator=g)
    dy = mat.empty((1, 1, 1024, images)).normal_(generator=g)
    X, F, D = x.double().reshape(-1, images), f.double().reshape(-1, 1024), dy.double().reshape(1024, images)
    small = torch.ones(images, device="cuda", dtype=torch.float64)
    small[1::3] = 2.0 ** e
    few = torch.ones(1024, device="cuda", dtype=torch.float64)
    few[::7] = 2.0 ** e
    ctx.set_precision(precision)
    try:
        dx, _, _ = nn.vl_nnconv(x, f, None, mat.as_mat(dy * small.float()), no_der_filters=True, ctx=ctx)
        columns_apart(dx.reshape(-1, images), F @ (D * small), 1, bound)
        _, df, _ = nn.vl_nnconv(x, f, None, mat.as_mat(dy * few.float()[:, None]), no_der_data=True, ctx=ctx)
        columns_apart(df.reshape(-1, 1024), X @ (D * few[:, None]).T, 1, bound)
        assert ctx.device_status() == 0
    finally:
        ctx.set_precision(0)


def test_more_groups_of_images_than_a_grid_is_high(gpu):
    """65537 groups of eight images: a launch takes 65535 along y, so the filter gradient has to come from a kernel that counts them otherwise."""
    import torch
    nn, mat, ctx = gpu
    g = torch.Generator(device="cuda").manual_seed(79)
    images = 8 * 65537
    x, f, dy = mat.empty((8, 1, 32, images)).normal_(generator=g), mat.empty((1, 1, 32, 16)).normal_(generator=g), mat.empty((8, 1, 16, images)).normal_(generator=g)
    want = torch.einsum("hwcn,hwkn->ck", x.double(), dy.double())
    lib = ctx.lib
    try:
        for switch in (0, 16):
            ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, switch))
            _, df, db = nn.vl_nnconv(x, f, mat.zeros((1, 16)), dy, no_der_data=True, ctx=ctx)
            assert rel(df[0, 0], want) < 1e-6 and rel(db.reshape(-1), dy.double().sum((0, 1, 3))) < 1e-5
    finally:
        ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))


def test_more_blocks_of_channels_than_a_grid_is_high(gpu):
    """The data gradient of 65537 blocks of 64 filters, two column tiles.  The reduction is cut into at least 74 ranges (two tiles on 148 SMs); the running sum
    of one has 886 k-blocks, whose rounding, 2^-24 each at random, comes to 1.8e-6 at most."""
    import torch
    nn, mat, ctx = gpu
    g = torch.Generator(device="cuda").manual_seed(80)
    k = 64 * 65537
    f, dy = mat.empty((1, 1, 130, k)).normal_(generator=g), mat.empty((2, 2, k, 1)).normal_(generator=g)
    dx, _, _ = nn.vl_nnconv(mat.zeros((2, 2, 130, 1)), f, None, dy, no_der_filters=True, ctx=ctx)
    assert rel(dx[..., 0], torch.einsum("ck,hwk->hwc", f[0, 0].double(), dy[..., 0].double())) < 2e-6
    ctx.check(ctx.lib.vlb_ctx_clear_workspace(ctx.handle))


def test_an_odd_number_of_run_buffers_keeps_the_groups_apart(gpu):
    """128-column tiles of the row mode (test switch bit 5 rules out the other form) have three run buffers for two groups of producers: a buffer's previous run
    belongs to the other group.  A group that did not wait for it to be let go of took a run of three k-blocks before for its own, once in some thousand launches."""
    import torch
    nn, mat, ctx = gpu
    g = torch.Generator(device="cuda").manual_seed(77)
    x, f, dy = mat.empty((28, 28, 512, 16)).normal_(generator=g), mat.empty((1, 1, 512, 128)).normal_(generator=g), mat.empty((28, 28, 128, 16)).normal_(generator=g)
    lib = ctx.lib
    ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 32))
    try:
        _, first, _ = nn.vl_nnconv(x, f, None, dy, no_der_data=True, ctx=ctx)
        wrong = torch.zeros((), device="cuda", dtype=torch.int64)
        for _ in range(20000):
            _, df, _ = nn.vl_nnconv(x, f, None, dy, no_der_data=True, ctx=ctx)
            wrong += (df != first).any()
        assert int(wrong) == 0
    finally:
        ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))
    assert ctx.device_status() == 0


def test_run_buffers_of_a_fully_connected_forward_pass(gpu):
    """128-column tiles with the sum in shared memory leave three run buffers to the two groups of producers there too; the sums are the same ones."""
    import torch
    nn, mat, ctx = gpu
    g = torch.Generator(device="cuda").manual_seed(78)
    x, f = mat.empty((4, 4, 512, 128)).normal_(generator=g), mat.empty((4, 4, 512, 256)).normal_(generator=g)
    y = nn.vl_nnconv(x, f, None, ctx=ctx)
    lib = ctx.lib
    ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 8))
    try:
        for _ in range(50):
            assert torch.equal(nn.vl_nnconv(x, f, None, ctx=ctx), y)
    finally:
        ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))
    assert ctx.device_status() == 0


# data, filters, stride: a data gradient in one piece, one by residue classes, one in filter groups; filter gradients of 64 images per k-block, of fewer, of planes
# that the row mode does not take
SCRATCH = [((28, 28, 64, 70), (3, 3, 64, 128), 1), ((14, 14, 64, 16), (3, 3, 64, 64), 2), ((13, 13, 128, 9), (3, 3, 64, 128), 1), ((7, 7, 512, 32), (3, 3, 512, 512), 1)]


@pytest.mark.parametrize("case", range(len(SCRATCH)))
def test_gradients_without_room_for_chunks(gpu, case):
    """Test switch bit 5: the kernels that need no copy of the data or of dY, in less scratch, as near to float64."""
    nn, mat, ctx = gpu
    import torch
    xs, fs, stride = SCRATCH[case]
    g = torch.Generator(device="cuda").manual_seed(1000 + case)
    x, f = mat.empty(xs).normal_(generator=g), mat.empty(fs).normal_(generator=g)
    dy = mat.empty(reference(x, f, None, stride, 1, 1)).normal_(generator=g)
    dxr, dfr, dbr = reference(x, f, dy, stride, 1, 1)
    lib = ctx.lib
    needs = {}
    try:
        for switch in (0, 16, 32, 48):
            ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, switch))
            needs[switch] = []
            for kw in (dict(no_der_filters=True, no_der_biases=True), dict(no_der_data=True)):
                ctx.check(lib.vlb_ctx_clear_workspace(ctx.handle))
                dx, df, db = nn.vl_nnconv(x, f, mat.zeros((1, fs[3])), dy, stride=stride, pad=1, ctx=ctx, **kw)
                needs[switch].append(lib.vlb_ctx_workspace_bytes(ctx.handle))
                if "no_der_data" in kw:
                    # (tc_gemm_kernel's chains: the bound of its own tests)
                    assert rel(df, dfr) < 1e-5 and rel(db.reshape(-1), dbr) < 1e-5, switch
                else:
                    assert rel(dx, dxr) < 1e-5, switch
        assert ctx.device_status() == 0
        assert needs[32] == needs[48] and needs[32][0] < needs[0][0] and needs[32][1] != needs[16][1]
    finally:
        ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))


@pytest.mark.parametrize("images", [256, 640])
def test_fully_connected_gradients_without_room_for_chunks(gpu, images):
    nn, mat, ctx = gpu
    import torch
    g = torch.Generator(device="cuda").manual_seed(1100 + images)
    x, f, dy = mat.empty((4, 4, 512, images)).normal_(generator=g), mat.empty((4, 4, 512, 512)).normal_(generator=g), mat.empty((1, 1, 512, images)).normal_(generator=g)
    X, F, D = x.double().reshape(-1, images), f.double().reshape(-1, 512), dy.double().reshape(512, images)
    lib = ctx.lib
    needs = {}
    try:
        for switch in (0, 32):
            ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, switch))
            ctx.check(lib.vlb_ctx_clear_workspace(ctx.handle))
            dx, df, _ = nn.vl_nnconv(x, f, None, dy, ctx=ctx)
            needs[switch] = lib.vlb_ctx_workspace_bytes(ctx.handle)
            assert rel(dx.reshape(-1, images), F @ D) < 1e-6 and rel(df.reshape(-1, 512), X @ D.T) < 1e-6, switch
        assert needs[32] < needs[0]
    finally:
        ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))


def test_a_device_without_room_for_chunks(gpu):
    """No switch: so little of the device's memory left that the 0.5 GB of dY's chunks, and 0.5 GB of the data's beside the tile images of dY, do not fit.  The
    same kernels as with the switch, so the same bits."""
    nn, mat, ctx = gpu
    import torch
    g = torch.Generator(device="cuda").manual_seed(1200)
    x, f, dy = mat.empty((56, 56, 64, 640)).normal_(generator=g), mat.empty((3, 3, 64, 64)).normal_(generator=g), mat.empty((56, 56, 64, 640)).normal_(generator=g)
    lib = ctx.lib
    taken = None
    try:
        for kw, which, left in ((dict(no_der_filters=True), 0, 256), (dict(no_der_data=True), 1, 768)):
            ctx.check(lib.vlb_ctx_clear_workspace(ctx.handle))
            ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 32))
            want = nn.vl_nnconv(x, f, None, dy, pad=1, ctx=ctx, **kw)[which]
            need = lib.vlb_ctx_workspace_bytes(ctx.handle)
            again = nn.vl_nnconv(x, f, None, dy, pad=1, ctx=ctx, **kw)[which]
            del again                                         # (torch keeps the room of a second output)
            ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))
            ctx.check(lib.vlb_ctx_clear_workspace(ctx.handle))
            torch.cuda.synchronize()
            taken = torch.empty(torch.cuda.mem_get_info()[0] - (left << 20), dtype=torch.uint8, device="cuda")
            for _ in range(2):
                got = nn.vl_nnconv(x, f, None, dy, pad=1, ctx=ctx, **kw)[which]
                assert torch.equal(got, want)
                del got
            assert lib.vlb_ctx_workspace_bytes(ctx.handle) == need
            del taken
            taken = None
            torch.cuda.empty_cache()
    finally:
        del taken
        torch.cuda.empty_cache()
        ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))
        ctx.check(lib.vlb_ctx_clear_workspace(ctx.handle))


def test_a_captured_call_makes_do_with_the_scratch_that_is_there(gpu):
    """A stream that is being captured can neither wait nor allocate."""
    nn, mat, ctx = gpu
    import torch
    g = torch.Generator(device="cuda").manual_seed(1300)
    x, f, dy = mat.empty((14, 14, 64, 64)).normal_(generator=g), mat.empty((3, 3, 64, 64)).normal_(generator=g), mat.empty((14, 14, 64, 64)).normal_(generator=g)
    lib = ctx.lib
    try:
        for kw, which in ((dict(no_der_filters=True), 0), (dict(no_der_data=True), 1)):
            ctx.check(lib.vlb_ctx_clear_workspace(ctx.handle))
            ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 32))
            want = nn.vl_nnconv(x, f, None, dy, pad=1, ctx=ctx, **kw)[which]
            need = lib.vlb_ctx_workspace_bytes(ctx.handle)
            ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                got = nn.vl_nnconv(x, f, None, dy, pad=1, ctx=ctx, **kw)[which]
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(got, want) and lib.vlb_ctx_workspace_bytes(ctx.handle) == need
            graph.reset()
    finally:
        ctx.check(lib.vlb_ctx_set_test_switch(ctx.handle, 0))
        nn.vl_nnrelu(x, ctx=ctx)            # (the context follows torch's current stream again)
        ctx.check(lib.vlb_ctx_clear_workspace(ctx.handle))
