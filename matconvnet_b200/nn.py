"""The reference's building blocks with their MATLAB call signatures, on device tensors.

Forward:  ``y = vl_nnX(x, params...)``;  backward: ``dx, dparams... = vl_nnX(x, params..., dzdy)``
-- the convention of every block of the reference (matlab/vl_nnconv.m, vl_nnbnorm.m,
vl_nnpool.m, vl_nnroipool.m, vl_nnbilinearsampler.m, vl_nnrelu.m, vl_nnsoftmaxloss.m).
Arguments are column-major CUDA float32 tensors (see ``mat``); each function validates
shapes as the corresponding MEX gateway does, allocates the outputs, and calls the C ABI -- all of it in one native call
per operator (csrc/hostpath.cpp).  Nothing here computes on the host.
"""
import ctypes as C

import numpy as np
import torch

from . import capi, mat

try:
    from . import _hostpath
except ImportError as e:
    raise ImportError("_hostpath.so is missing or does not load: build it with `python -m matconvnet_b200.build` "
                      "(this package has no other implementation): %s" % e) from e

_default_ctx = None


def default_context():
    """Process-wide context (the MEX-file-global `context` of the reference,
    matlab/src/vl_nnconv.cu:64)."""
    global _default_ctx
    if _default_ctx is None:
        _default_ctx = capi.Context()
    return _default_ctx


def _ctx(ctx):
    ctx = ctx or default_context()
    ctx.set_stream(torch.cuda.current_stream().cuda_stream)
    return ctx


def _need(t, name):
    if not (isinstance(t, torch.Tensor) and t.is_cuda and t.dtype == torch.float32):
        raise TypeError("%s must be a CUDA float32 tensor (this engine has no CPU path)" % name)
    return mat.as_mat(t)


def _pair(v, name):
    v = np.atleast_1d(np.asarray(v)).astype(int).ravel()
    if v.size == 1:
        return int(v[0]), int(v[0])
    if v.size == 2:
        return int(v[0]), int(v[1])
    raise ValueError("%s must have one or two elements" % name)


def _quad(v, name):
    v = np.atleast_1d(np.asarray(v)).astype(int).ravel()
    if v.size == 1:
        return (int(v[0]),) * 4
    if v.size == 4:
        return tuple(int(i) for i in v)
    raise ValueError("%s must have one or four elements" % name)


_hostpath.setup(_pair, _quad, capi.VlbError)


# --------------------------------------------------------------------- vl_nnconv
def vl_nnconv(x, f, b, dzdy=None, stride=1, pad=0, dilate=1, no_der_data=False, no_der_filters=False,
              no_der_biases=False, relu=False, through_relu=False, der_out=None, ctx=None):
    """Y = VL_NNCONV(X, F, B) / [DX, DF, DB] = VL_NNCONV(X, F, B, DZDY) (matlab/vl_nnconv.m;
    gateway matlab/src/vl_nnconv.cu:87-503).  B may be None.  Empty F (the subsampling mode of
    the reference) is not part of this engine.  relu=True (forward only) returns max(Y, 0) from the same kernels,
    bit-identical to vl_nnrelu(vl_nnconv(...)).  through_relu=True (backward only) is for an X that is the output of a
    ReLU: DX is then the derivative with respect to that ReLU's input, bit-identical to vl_nnrelu(X, DX).
    der_out=(DF, DB) (backward only; either may be None) makes the kernels write the parameter derivatives into tensors the
    caller owns -- views into a gradient-exchange bucket -- instead of new ones; they are returned as DF, DB."""
    if f is None or f.numel() == 0:
        raise capi.VlbError(1, "vl_nnconv with empty filters (subsampling) is not supported")
    return _hostpath.conv(ctx or default_context(), x, f, b, dzdy, stride, pad, dilate, no_der_data, no_der_filters,
                          no_der_biases, relu, through_relu, der_out)


# --------------------------------------------------------------------- vl_nnconvt
def vl_nnconvt(x, f, b, dzdy=None, upsample=1, crop=0, num_groups=1, no_der_data=False, no_der_filters=False,
               no_der_biases=False, ctx=None):
    """Y = VL_NNCONVT(X, F, B) / [DX, DF, DB] = VL_NNCONVT(X, F, B, DZDY) (matlab/vl_nnconvt.m; gateway
    matlab/src/vl_nnconvt.cu:87-417).  F is FH x FW x FD x C: FD output channels per filter group, its fourth dimension
    the depth of X.  B may be None."""
    return _hostpath.convt(ctx or default_context(), x, f, b, dzdy, upsample, crop, int(num_groups), no_der_data,
                           no_der_filters, no_der_biases)


# --------------------------------------------------------------------- vl_nnbnorm
def vl_nnbnorm(x, g, b, dzdy=None, epsilon=1e-4, moments=None, der_out=None, relu=False, ctx=None):
    """[Y, MOMENTS] = VL_NNBNORM(X, G, B) / [DX, DG, DB, MOMENTS] = VL_NNBNORM(X, G, B, DZDY)
    (matlab/vl_nnbnorm.m; gateway matlab/src/vl_nnbnorm.cu:73-302).  MOMENTS is C x 2:
    [mean, sigma] with sigma = sqrt(var + epsilon).  relu=True (forward, moments from the batch) returns max(Y, 0) from the
    same kernel, bit-identical to vl_nnrelu(vl_nnbnorm(...))."""
    return _hostpath.bnorm(ctx or default_context(), x, g, b, dzdy, epsilon, moments, der_out, relu)


# --------------------------------------------------------------------- vl_nnpool
def vl_nnpool(x, pool, dzdy=None, stride=1, pad=0, method="max", through_relu=False, ctx=None):
    """Y = VL_NNPOOL(X, POOL) / DX = VL_NNPOOL(X, POOL, DZDY) (matlab/vl_nnpool.m; gateway
    matlab/src/vl_nnpool.cu:72-315).  through_relu=True (backward only) is for an X that is the output of a ReLU: DX is
    then the derivative with respect to that ReLU's input, bit-identical to vl_nnrelu(X, DX)."""
    if method not in ("max", "avg"):
        raise ValueError("METHOD is not a supported method.")
    return _hostpath.pool(ctx or default_context(), x, pool, dzdy, stride, pad,
                          capi.POOL_MAX if method == "max" else capi.POOL_AVG, through_relu)


# --------------------------------------------------------------------- vl_nnroipool
def _transform(t):
    """2 x 3 affine transform as six doubles, column-major; a scalar scales and keeps pixel centres
    (matlab/src/vl_nnroipool.cu:150-155)."""
    if isinstance(t, (int, float)):
        t = float(t)
        return (t, 0.0, 0.0, t, 1.0 - t, 1.0 - t)
    t = np.asarray(t, dtype=np.float64).ravel(order="F")
    if t.size == 1:
        return _transform(float(t[0]))
    if t.size != 6:
        raise ValueError("TRANSFORM must be a scalar or a 2 x 3 matrix.")
    return tuple(float(v) for v in t)


def vl_nnroipool(x, rois, dzdy=None, subdivisions=(1, 1), transform=1.0, method="max", ctx=None):
    """Y = VL_NNROIPOOL(X, ROIS) / DX = VL_NNROIPOOL(X, ROIS, DZDY) (matlab/vl_nnroipool.m; gateway
    matlab/src/vl_nnroipool.cu:70-271).  ROIS is 5 x K: [image; u1; v1; u2; v2], 1-based."""
    return _hostpath.roipool(ctx or default_context(), x, rois, dzdy, subdivisions, _transform(transform),
                             capi.POOL_MAX if method == "max" else capi.POOL_AVG)


def roipool_bounds(rois, x_shape, subdivisions=(1, 1), transform=1.0, ctx=None):
    """Device bin geometry: (bounds int32 [4,S0,S1,K] = hstart,hend,wstart,wend; images int32 [K])."""
    ctx = _ctx(ctx)
    rois = _need(rois, "rois")
    H, W, _, N = x_shape
    K = rois.numel() // 5
    S0, S1 = _pair(subdivisions, "SUBDIVISIONS")
    bounds = mat.zeros((4, S0, S1, K), rois.device, torch.int32)
    images = torch.zeros(K, device=rois.device, dtype=torch.int32)
    ctx.check(ctx.lib.vlb_roipool_bounds(ctx.handle, mat.ptr(bounds), mat.ptr(images), mat.ptr(rois), H, W, N, K,
                                         S0, S1, (C.c_double * 6)(*_transform(transform))))
    return bounds, images


# --------------------------------------------------------------------- vl_nnbilinearsampler
def vl_nnbilinearsampler(x, grid, dzdy=None, ctx=None):
    """Y = VL_NNBILINEARSAMPLER(X, GRID) / [DX, DGRID] = VL_NNBILINEARSAMPLER(X, GRID, DZDY)
    (matlab/vl_nnbilinearsampler.m; gateway matlab/src/vl_nnbilinearsampler.cu:66-223)."""
    return _hostpath.sampler(ctx or default_context(), x, grid, dzdy)


# --------------------------------------------------------------------- gradient scaling
def scale_(t, alpha, ctx=None):
    """t *= alpha in place: the division by the number of workers of an all-reduced gradient
    (examples/cnn_train.m:482-483)."""
    ctx = _ctx(ctx)
    if not (t.is_cuda and t.dtype == torch.float32):
        raise TypeError("CUDA float32 tensor expected")
    ctx.check(ctx.lib.vlb_scale(ctx.handle, t.data_ptr(), float(alpha), t.numel()))
    return t


def vl_taccum(alpha, a, beta, b, out=None, ctx=None):
    """Y = VL_TACCUM(ALPHA, A, BETA, B) = ALPHA*A + BETA*B (matlab/vl_taccum.m); out=a updates A in place."""
    return _hostpath.taccum(ctx or default_context(), alpha, a, beta, b, out)


_NO_OPTS = (0.0, 0.0, 0.0, 0.0)


def sgd_update_(w, momentum_state, grad, grad_mult, decay, momentum, lr, nesterov=False, ctx=None):
    """The trainer's momentum-SGD step on one parameter tensor, in place on w and momentum_state
    (examples/cnn_train.m:478-499: four vl_taccum passes, here one kernel)."""
    sgd_update_many_([(w, momentum_state, grad, decay, lr)], grad_mult, momentum, nesterov, ctx)
    return w


def sgd_update_many_(updates, grad_mult, momentum, nesterov=False, ctx=None):
    """sgd_update_ on several parameter tensors in one launch; updates: [(w, momentum_state, grad, decay, lr)]."""
    _hostpath.update(ctx or default_context(), -1, [(w, m, None, g, decay, lr, 0) for w, m, g, decay, lr in updates], grad_mult,
                     momentum, nesterov, _NO_OPTS)


def solver_update_(solver, w, state, grad, grad_mult, decay, lr, opts=None, ctx=None):
    """One step of examples/+solver/<solver>.m on one parameter tensor, fused with the trainer's normalisation and weight
    decay pass (examples/cnn_train.m:481-507), in place on w and on the solver state.  state: {} before the first step;
    afterwards it holds the solver's tensors (g_sqr; g_sqr and delta_sqr; m, v and the step count t)."""
    solver_update_many_(solver, [(w, state, grad, decay, lr)], grad_mult, opts, ctx)
    return w


def solver_update_many_(solver, updates, grad_mult, opts=None, ctx=None):
    """solver_update_ on several parameter tensors in one launch; updates: [(w, state, grad, decay, lr)]."""
    if solver not in capi.SOLVERS:
        raise ValueError("unknown solver '%s'" % solver)
    o = dict(capi.SOLVER_DEFAULTS[solver])
    o.update(opts or {})
    two = solver in ("adadelta", "adam")
    for w, _, g, _, _ in updates:             # a refused list leaves every state and step count as it was
        if not all(isinstance(t, torch.Tensor) and t.is_cuda and t.dtype == torch.float32 for t in (w, g)):
            raise TypeError("w and grad must be CUDA float32 tensors")
        if w.numel() != g.numel():
            raise ValueError("parameter and gradient do not have the same number of elements.")
    items = []
    for w, state, g, decay, lr in updates:
        if "s1" not in state:
            state["s1"] = torch.zeros_like(w)
            if two:
                state["s2"] = torch.zeros_like(w)
            state["t"] = 0
        state["t"] += 1
        items.append((w, state["s1"], state["s2"] if two else None, g, decay, lr, state["t"]))
    _hostpath.update(ctx or default_context(), capi.SOLVERS[solver], items, grad_mult, 0.0, False,
                     (o.get("rho", 0.0), o["epsilon"], o.get("beta1", 0.0), o.get("beta2", 0.0)))


# --------------------------------------------------------------------- MATLAB-only blocks
def vl_nnrelu(x, dzdy=None, ctx=None):
    """matlab/vl_nnrelu.m:43-48 with LEAK = 0."""
    return _hostpath.relu(ctx or default_context(), x, dzdy)


def vl_nnnormalize(x, param, dzdy=None, ctx=None, through_relu=False):
    """Y = VL_NNNORMALIZE(X, PARAM) / DZDX = VL_NNNORMALIZE(X, PARAM, DZDY), PARAM = [N KAPPA ALPHA BETA]
    (matlab/vl_nnnormalize.m; gateway matlab/src/vl_nnnormalize.cu:117-162).  through_relu=True (backward only) is for an X that
    is the output of a ReLU: DZDX is then the derivative with respect to that ReLU's input."""
    if not (isinstance(param, (list, tuple)) and len(param) == 4):
        param = np.asarray(param, dtype=np.float64).ravel()
        if len(param) != 4:
            raise ValueError("PARAM is not a plain 4 vector.")
    depth = int(param[0])
    if depth < 1:
        raise ValueError("The normalization depth is smaller than 1.")
    return _hostpath.normalize(ctx or default_context(), x, dzdy, depth, float(param[1]), float(param[2]), float(param[3]), through_relu)


def vl_nnsoftmax(x, dzdy=None, ctx=None):
    """Y = VL_NNSOFTMAX(X) / DZDX = VL_NNSOFTMAX(X, DZDY): softmax over the channels (matlab/vl_nnsoftmax.m)."""
    return _hostpath.softmax(ctx or default_context(), x, dzdy)


def vl_nndropout(x, dzdy=None, rate=0.5, mask=None, seed=0, ctx=None):
    """[Y, MASK] = VL_NNDROPOUT(X, 'rate', R) / [DZDX, MASK] = VL_NNDROPOUT(X, DZDY, 'mask', MASK) (matlab/vl_nndropout.m).
    MASK is drawn when it is not given: 1/(1-rate) where a uniform number is at least the rate, else 0; `seed` selects the
    stream of the counter-based generator (the reference draws from MATLAB's global stream)."""
    return _hostpath.dropout(ctx or default_context(), x, dzdy, rate, mask, int(seed))


def vl_nnsoftmaxloss(x, c, dzdy=None, ctx=None):
    """matlab/vl_nnsoftmaxloss.m:56-84 with one class label (1-based) per image."""
    return _hostpath.softmaxloss(ctx or default_context(), x, c, dzdy)
