"""Bilinear sampler with its planes in shared memory: bit for bit the oracle's result at the edges of the channel groups, of the
plane sizes and of the parts of a grid, both where images fill the chip and where they do not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,c,n,group,ho,wo", [
    (13, 11, 7, 80, 2, 35, 33),     # odd planes (copies of four bytes), three channels left over, two parts per grid, two grids per image
    (12, 16, 4, 150, 1, 12, 12),    # one whole channel group, copies of sixteen bytes
    (12, 12, 9, 160, 1, 32, 32),    # one channel left over, exactly one part; eight channels and one in the data gradient
    (20, 8, 3, 148, 1, 10, 8),      # fewer channels than a group, output half the input
    (16, 16, 13, 3, 2, 20, 20),     # few images: channels shared out among blocks
])
def test_sampler_planes(gpu, oracle, h, w, c, n, group, ho, wo):
    from matconvnet_b200 import mat, nn
    rng = np.random.default_rng(h * 100 + c)
    x = np.asfortranarray(rng.standard_normal((h, w, c, n)).astype(np.float32))
    yy, xx = np.meshgrid(np.linspace(-1.1, 1.1, ho), np.linspace(-1.1, 1.1, wo), indexing="ij")
    base = np.stack([yy, xx])[..., None] + 0.1 * rng.standard_normal((2, 1, 1, n * group))
    grid = np.asfortranarray(base.astype(np.float32))
    dy = np.asfortranarray(rng.standard_normal((ho, wo, c, n * group)).astype(np.float32))
    xd, gd, dyd = (mat.from_numpy(v) for v in (x, grid, dy))
    assert np.array_equal(mat.to_numpy(nn.vl_nnbilinearsampler(xd, gd)), oracle.sampler_forward(x, grid))
    dx, dgrid = nn.vl_nnbilinearsampler(xd, gd, dyd)
    dxr, dgr = oracle.sampler_backward(x, grid, dy)
    assert np.array_equal(mat.to_numpy(dx), dxr)
    assert np.array_equal(mat.to_numpy(dgrid), dgr)


def test_grid_derivative_of_the_largest_grid(gpu):
    """2^31 - 1 output pixels, more than the kernel with the planes in shared memory can count: the first and the last pixels equal those of a
    small call bit for bit (a pixel's derivative depends on no other pixel)."""
    import ctypes
    import torch
    nn, mat, ctx = gpu
    H = W = 8
    C, Q, few = 3, (1 << 31) - 1, 5000
    torch.cuda.empty_cache()
    g = torch.Generator(device="cuda").manual_seed(2)
    x = mat.empty((H, W, C, 1)).normal_(generator=g)
    ends = torch.rand(2 * few, 2, device="cuda", generator=g) * 2.4 - 1.2
    dends = torch.randn(C, 2 * few, device="cuda", generator=g)

    def run(grid, dy, q):
        out = torch.empty(q, 2, device="cuda")
        ctx.set_stream(torch.cuda.current_stream().cuda_stream)
        ctx.check(ctx.lib.vlb_sampler_backward(ctx.handle, None, *(ctypes.c_void_p(t.data_ptr()) for t in (out, x, grid, dy)), H, W, C, 1, 1, q, 1))
        return out

    want = run(ends, dends, 2 * few)
    grid, dy = torch.zeros(Q, 2, device="cuda"), torch.zeros(C, Q, device="cuda")
    for t, e in ((grid.T, ends.T), (dy, dends)):
        t[:, :few], t[:, Q - few:] = e[:, :few], e[:, few:]
    got = run(grid, dy, Q)
    assert torch.equal(got[:few], want[:few]) and torch.equal(got[Q - few:], want[few:])
    del grid, dy, got
    torch.cuda.empty_cache()
