"""The work that users of this framework have it do, as measurable cases.

Seven kinds of work, each over its real range of sizes:

  net        a linear chain through ``simplenn.vl_simplenn``: the LeNet block, the CIFAR-10 network, an AlexNet-style network
             (strided and grouped convolutions, local response normalisation, dropout) and VGG-16; forward only
             ("infer"), forward + backward ("train") or a whole trainer step with the parameter update ("step")
  residual   a bottleneck block with batch normalisation and its shortcut, forward + backward
  frcnn      the Fast R-CNN head: ROI pooling and two fully connected layers, forward + backward
  sampler    the bilinear sampler of a spatial transformer, forward + backward
  conv       one convolution of any geometry, forward + backward
  convt      one convolution transpose (upsampling in segmentation networks), forward + backward
  update     the trainer's parameter update alone

A case is a dict of plain values; ``prepare`` makes what a program has in hand before the call (inputs, weights, solver
state), ``run`` is one pass, ``work`` what the pass cannot do without, ``tolerance`` how far another correct implementation
at the same precision may be.  Tensors are single precision in MATLAB order; "tf32" is the engine's fast arithmetic, which
rounds the operands of the contractions to TF32.
"""
import math

import torch

from matconvnet_b200 import capi, mat, nn, simplenn, train

_PRECISION = {"3xtf32": capi.PRECISION_3XTF32, "tf32": capi.PRECISION_TF32}
_contexts = {}


def _context(precision):
    """One context per arithmetic, kept by the program for its whole life; scratch grown once, up front."""
    if precision not in _contexts:
        ctx = nn.default_context() if precision == "3xtf32" else capi.Context(precision=_PRECISION[precision])
        ctx.reserve_workspace(3 << 30)
        _contexts[precision] = ctx
    return _contexts[precision]


# ------------------------------------------------------------------------------------------------ networks
def _chain(net, size, classes):
    """Layer specifications of a network for size x size inputs, and the input's depth."""
    conv = lambda fs, fc, k, stride=1, pad=0: dict(type="conv", fs=fs, fc=fc, k=k, stride=stride, pad=pad)     # noqa: E731
    pool = lambda method, p, stride, pad=(0, 0, 0, 0): dict(type="pool", method=method, p=p, stride=stride, pad=pad)  # noqa: E731
    relu = dict(type="relu")
    if net == "lenet":
        return [conv(5, 1, 20), pool("max", 2, 2), conv(5, 20, 50), pool("max", 2, 2)], 1
    if net == "cifar":
        odd = (0, 1, 0, 1)
        side = size
        for _ in range(3):
            side = (side + 1 - 3) // 2 + 1
        return [conv(5, 3, 32, pad=2), pool("max", 3, 2, odd), relu, conv(5, 32, 32, pad=2), relu, pool("avg", 3, 2, odd),
                conv(5, 32, 64, pad=2), relu, pool("avg", 3, 2, odd), conv(side, 64, 64), relu, conv(1, 64, classes),
                dict(type="softmaxloss")], 3
    if net == "alexnet":
        side = (size - 11) // 4 + 1
        for _ in range(3):
            side = (side - 3) // 2 + 1
        lrn, drop = dict(type="normalize", param=[5, 1.0, 1e-4 / 5, 0.75]), dict(type="dropout", rate=0.5, seed=1)
        return [conv(11, 3, 96, stride=4), relu, lrn, pool("max", 3, 2), conv(5, 48, 256, pad=2), relu, lrn, pool("max", 3, 2),
                conv(3, 256, 384, pad=1), relu, conv(3, 192, 384, pad=1), relu, conv(3, 192, 256, pad=1), relu,
                pool("max", 3, 2), conv(side, 256, 4096), relu, drop, conv(1, 4096, 4096), relu, drop,
                conv(1, 4096, classes), dict(type="softmaxloss")], 3
    if net == "vgg16":
        layers, cin, side = [], 3, size
        for cout, reps in ((64, 2), (128, 2), (256, 3), (512, 3), (512, 3)):
            for _ in range(reps):
                layers += [conv(3, cin, cout, pad=1), relu]
                cin = cout
            layers.append(pool("max", 2, 2))
            side //= 2
        return layers + [conv(side, 512, 4096), relu, conv(1, 4096, 4096), relu, conv(1, 4096, classes),
                         dict(type="softmaxloss")], 3
    raise ValueError("unknown network '%s'" % net)


def _walk(layers, h, w, c):
    """[(layer, input (h, w, c), output (h, w, c))] of a chain."""
    out = []
    for l in layers:
        src = (h, w, c)
        if l["type"] in ("conv", "pool"):
            f = l["fs"] if l["type"] == "conv" else l["p"]
            p = l["pad"] if isinstance(l["pad"], tuple) else (l["pad"],) * 4
            h, w = (h + p[0] + p[1] - f) // l["stride"] + 1, (w + p[2] + p[3] - f) // l["stride"] + 1
            c = l["k"] if l["type"] == "conv" else c
        elif l["type"] == "softmaxloss":
            h, w, c = 1, 1, 0
        out.append((l, src, (h, w, c)))
    return out


def _normal(gen, shape, std=1.0):
    return mat.empty(shape).normal_(0.0, std, generator=gen)


def _build(gen, layers, std=None, depth=None):
    """Layers as vl_simplenn takes them; He-normal filters unless a deviation is given, zero biases."""
    net = []
    for l in layers:
        if l["type"] == "conv":
            fan = l["fs"] * l["fs"] * l["fc"]
            net.append(dict(type="conv", weights=[_normal(gen, (l["fs"], l["fs"], l["fc"], l["k"]), std or math.sqrt(2.0 / fan)),
                                                  mat.zeros((1, l["k"])) if l.get("bias", True) else None],
                            stride=l["stride"], pad=list(l["pad"]) if isinstance(l["pad"], tuple) else l["pad"], dilate=1))
            depth = l["k"]
        elif l["type"] == "bnorm":
            net.append(dict(type="bnorm", weights=[mat.zeros((depth, 1)) + 1.0, mat.zeros((depth, 1))], epsilon=1e-5))
        elif l["type"] == "pool":
            net.append(dict(type="pool", method=l["method"], pool=[l["p"], l["p"]], stride=l["stride"], pad=list(l["pad"])))
        else:
            net.append(dict(l))
    return {"layers": net}


def _chain_work(walk, batch, mode, update=0):
    """Flops of the contractions; bytes of the input, the parameters, every activation vl_simplenn stores (once), and in
    training the derivatives of the input and of the parameters; `update`: tensors read and written per parameter besides."""
    flops = par = act = 0.0
    for l, (h, w, c), (ho, wo, co) in walk:
        act += ho * wo * co * batch
        if l["type"] == "conv":
            fan = l["fs"] * l["fs"] * l["fc"]
            flops += 2.0 * ho * wo * batch * l["k"] * fan
            par += l["k"] * (fan + (1 if l.get("bias", True) else 0))
    h, w, c = walk[0][1]
    x = h * w * c * batch
    if mode == "infer":
        return {"bytes": 4 * (x + par + act), "flops": flops}
    return {"bytes": 4 * (2 * x + act + (2 + update) * par), "flops": 3 * flops}


def _prepare_net(case, gen):
    layers, depth = _chain(case["net"], case["size"], case["classes"])
    if case["mode"] == "infer" and layers[-1]["type"] == "softmaxloss":
        layers = layers[:-1] + [dict(type="softmax")]
    if case["mode"] == "infer":
        layers = [l for l in layers if l["type"] != "dropout"]
    batch, size = case["batch"], case["size"]
    s = dict(net=_build(gen, layers, 0.01 if case["net"] in ("lenet", "cifar") else None),
             ctx=_context(case["precision"]), fuse=case["fuse"], mode=case["mode"])
    if case["net"] == "lenet":
        s["x"] = mat.empty((size, size, depth, batch)).uniform_(0.0, 1.0, generator=gen)
        s["dzdy"] = _normal(gen, _walk(layers, size, size, depth)[-1][2] + (batch,))
    else:
        s["x"] = _normal(gen, (size, size, depth, batch))
        s["dzdy"] = 1.0
        if case["mode"] != "infer":
            s["net"]["layers"][-1]["class"] = torch.randint(1, case["classes"] + 1, (batch,), device="cuda", generator=gen).float()
    if case["mode"] == "step":
        s["state"], s["params"] = {}, dict(train.default_params())
    return s


def _run_net(s):
    layers = s["net"]["layers"]
    if s["mode"] == "infer":
        # a program in test mode reads the class scores, and often the features of the pooling layers as well
        res = simplenn.vl_simplenn(s["net"], s["x"], ctx=s["ctx"], fuse_relu=s["fuse"])
        keep = [i + 1 for i, l in enumerate(layers) if l["type"] in ("pool", "softmax")] + [len(layers) - 1]
        return [res[i]["x"] for i in sorted(set(keep))]
    res = simplenn.vl_simplenn(s["net"], s["x"], s["dzdy"], ctx=s["ctx"], conserve_memory=True, fuse_relu=s["fuse"])
    out = {"y": res[-1]["x"], "dx": res[0]["dzdx"], "dw": [r["dzdw"] for r in res]}
    if s["mode"] == "step":
        train.accumulate_gradients(s["net"], res, s["state"], s["params"], ctx=s["ctx"])
        out["w"] = [l["weights"] for l in layers if "weights" in l]
        out["momentum"] = [s["state"][k] for k in sorted(s["state"])]
    return out


# ------------------------------------------------------------------------------------------------ residual block
def _residual_chain(case):
    wide, narrow, st = case["wide"], case["narrow"], case["stride"]
    cin = wide if st == 1 else wide // 2
    conv = lambda fs, fc, k, stride=1, pad=0: dict(type="conv", fs=fs, fc=fc, k=k, stride=stride, pad=pad, bias=False)   # noqa: E731
    bn, relu = dict(type="bnorm"), dict(type="relu")
    main = [conv(1, cin, narrow), bn, relu, conv(3, narrow, narrow, st, 1), bn, relu, conv(1, narrow, wide), bn]
    return main, ([conv(1, cin, wide, st), bn] if st > 1 else []), cin


def _prepare_residual(case, gen):
    main, short, cin = _residual_chain(case)
    size, batch = case["size"], case["batch"]
    ho, wo, co = _walk(main, size, size, cin)[-1][2]
    return dict(main=_build(gen, main), short=_build(gen, short) if short else None, ctx=_context(case["precision"]),
                fuse=case["fuse"], x=_normal(gen, (size, size, cin, batch)), dzdy=_normal(gen, (ho, wo, co, batch)))


def _run_residual(s):
    one = dict(ctx=s["ctx"], conserve_memory=True, fuse_relu=s["fuse"])
    res = simplenn.vl_simplenn(s["main"], s["x"], s["dzdy"], **one)
    dw = [r["dzdw"] for r in res]
    if s["short"] is None:
        y, dx = s["x"], s["dzdy"]
    else:
        cut = simplenn.vl_simplenn(s["short"], s["x"], s["dzdy"], **one)
        y, dx = cut[-1]["x"], cut[0]["dzdx"]
        dw += [r["dzdw"] for r in cut]
    return {"y": nn.vl_taccum(1.0, res[-1]["x"], 1.0, y, ctx=s["ctx"]),
            "dx": nn.vl_taccum(1.0, res[0]["dzdx"], 1.0, dx, ctx=s["ctx"]), "dw": dw}


# ------------------------------------------------------------------------------------------------ Fast R-CNN head
def _prepare_frcnn(case, gen):
    h, w, c, n, k, width = (case[q] for q in ("h", "w", "c", "n", "rois", "width"))
    rand = lambda: torch.rand(k, device="cuda", generator=gen)       # noqa: E731
    u1, v1 = rand() * (w - 3) + 1, rand() * (h - 3) + 1
    u2, v2 = (u1 + 2 + rand() * w).clamp(max=w), (v1 + 2 + rand() * h).clamp(max=h)
    rois = mat.as_mat(torch.stack([torch.arange(k, device="cuda") % n + 1.0, u1, v1, u2, v2]))
    return dict(x=_normal(gen, (h, w, c, n)), rois=rois, ctx=_context(case["precision"]),
                f6=_normal(gen, (7, 7, c, width), math.sqrt(2.0 / (49 * c))), b6=mat.zeros((1, width)),
                f7=_normal(gen, (1, 1, width, width), math.sqrt(2.0 / width)), b7=mat.zeros((1, width)),
                dzdy=_normal(gen, (1, 1, width, k)))


def _run_frcnn(s):
    ctx = s["ctx"]
    p = nn.vl_nnroipool(s["x"], s["rois"], subdivisions=(7, 7), ctx=ctx)
    h6 = nn.vl_nnconv(p, s["f6"], s["b6"], relu=True, ctx=ctx)
    y = nn.vl_nnconv(h6, s["f7"], s["b7"], ctx=ctx)
    d6, df7, db7 = nn.vl_nnconv(h6, s["f7"], s["b7"], s["dzdy"], through_relu=True, ctx=ctx)
    dp, df6, db6 = nn.vl_nnconv(p, s["f6"], s["b6"], d6, ctx=ctx)
    return [p, y, nn.vl_nnroipool(s["x"], s["rois"], dp, subdivisions=(7, 7), ctx=ctx), df6, db6, df7, db7]


# ------------------------------------------------------------------------------------------------ bilinear sampler
def _prepare_sampler(case, gen):
    h, w, c, n, ho, wo = (case[q] for q in ("h", "w", "c", "n", "ho", "wo"))
    # affine grids of small rotations, scales and shifts: grid = s * R * [y x] + t
    yy = torch.linspace(-1, 1, ho, device="cuda").view(ho, 1, 1)
    xx = torch.linspace(-1, 1, wo, device="cuda").view(1, wo, 1)
    rand = lambda *s: torch.rand(*s, device="cuda", generator=gen)    # noqa: E731
    th, sc, t = (rand(n) - 0.5) * 0.4, 0.8 + 0.4 * rand(n), (rand(2, n) - 0.5) * 0.2
    grid = torch.stack([sc * (torch.cos(th) * yy + torch.sin(th) * xx) + t[0],
                        sc * (torch.cos(th) * xx - torch.sin(th) * yy) + t[1]])
    return dict(x=_normal(gen, (h, w, c, n)), grid=mat.as_mat(grid), dzdy=_normal(gen, (ho, wo, c, n)))


def _run_sampler(s):
    y = nn.vl_nnbilinearsampler(s["x"], s["grid"])
    return [y, *nn.vl_nnbilinearsampler(s["x"], s["grid"], s["dzdy"])]


# ------------------------------------------------------------------------------------------------ single convolutions
def _conv_out(case):
    ext = (case["f"] - 1) * case["dilate"] + 1
    return tuple((case[q] + 2 * case["pad"] - ext) // case["stride"] + 1 for q in ("h", "w"))


def _prepare_conv(case, gen):
    f, fc = case["f"], case["c"] // case["groups"]
    return dict(x=_normal(gen, (case["h"], case["w"], case["c"], case["n"])),
                f=_normal(gen, (f, f, fc, case["k"]), math.sqrt(2.0 / (f * f * fc))), b=_normal(gen, (1, case["k"]), 0.1),
                dzdy=_normal(gen, _conv_out(case) + (case["k"], case["n"])),
                opts=dict(stride=case["stride"], pad=case["pad"], dilate=case["dilate"], ctx=_context(case["precision"])))


def _run_conv(s):
    y = nn.vl_nnconv(s["x"], s["f"], s["b"], **s["opts"])
    return [y, *nn.vl_nnconv(s["x"], s["f"], s["b"], s["dzdy"], **s["opts"])]


def _convt_out(case):
    return tuple((case[q] - 1) * case["up"] - 2 * case["crop"] + case["f"] for q in ("h", "w"))


def _prepare_convt(case, gen):
    f = case["f"]
    return dict(x=_normal(gen, (case["h"], case["w"], case["c"], case["n"])),
                f=_normal(gen, (f, f, case["k"], case["c"]), math.sqrt(2.0 / (f * f * case["c"]))),
                b=_normal(gen, (1, case["k"]), 0.1), dzdy=_normal(gen, _convt_out(case) + (case["k"], case["n"])),
                opts=dict(upsample=case["up"], crop=case["crop"], ctx=_context(case["precision"])))


def _run_convt(s):
    y = nn.vl_nnconvt(s["x"], s["f"], s["b"], **s["opts"])
    return [y, *nn.vl_nnconvt(s["x"], s["f"], s["b"], s["dzdy"], **s["opts"])]


# ------------------------------------------------------------------------------------------------ parameter update
def _update_sizes(case):
    """Filter shapes (fs, fc, k) of the network whose parameters are updated."""
    if case["net"] == "vgg16":
        return [(l["fs"], l["fc"], l["k"]) for l in _chain("vgg16", 224, 1000)[0] if l["type"] == "conv"]
    return [(3, case["width"], case["width"])] * case["layers"]


def _prepare_update(case, gen):
    layers, res = [], []
    for fs, fc, k in _update_sizes(case):
        layers.append(dict(type="conv", weights=[_normal(gen, (fs, fs, fc, k), 0.01), mat.zeros((1, k))]))
        res.append(dict(dzdw=[_normal(gen, (fs, fs, fc, k), 0.01), _normal(gen, (1, k), 0.01)]))
    params = dict(train.default_params(), nesterov_update=case["nesterov"])
    if case["solver"] != "sgd":
        params["solver"] = case["solver"]
    return dict(net={"layers": layers}, res=res, state={}, params=params, ctx=_context("3xtf32"))


def _run_update(s):
    train.accumulate_gradients(s["net"], s["res"], s["state"], s["params"], ctx=s["ctx"])
    state = [s["state"][k] for k in sorted(s["state"])]
    return {"w": [l["weights"] for l in s["net"]["layers"]],
            "state": [[v[q] for q in ("s1", "s2") if q in v] if isinstance(v, dict) else v for v in state]}


# ------------------------------------------------------------------------------------------------ the cases
_KINDS = {"net": (_prepare_net, _run_net), "residual": (_prepare_residual, _run_residual),
          "frcnn": (_prepare_frcnn, _run_frcnn), "sampler": (_prepare_sampler, _run_sampler),
          "conv": (_prepare_conv, _run_conv), "convt": (_prepare_convt, _run_convt),
          "update": (_prepare_update, _run_update)}


def _net(net, mode, batch, size, classes, precision="3xtf32", fuse=True):
    return dict(kind="net", net=net, mode=mode, batch=batch, size=size, classes=classes, precision=precision, fuse=fuse)


def listed():
    return [
        # the smallest network of the examples: a LeNet block on MNIST digits, the batch its trainer takes
        dict(_net("lenet", "train", 100, 28, 0, fuse=False), name="lenet_train_b100"),
        # a whole trainer step of the CIFAR-10 example: 13 small layers and the parameter update, called with the defaults
        dict(_net("cifar", "step", 100, 32, 10, fuse=False), name="cifar_step_b100"),
        # classifying one image at a time (serving): every launch and every pass over the weights counts
        dict(_net("vgg16", "infer", 1, 224, 1000), name="vgg16_infer_b1"),
        # the large-batch training step of the benchmark
        dict(_net("vgg16", "train", 64, 224, 1000), name="vgg16_train_b64"),
        # the other family of ImageNet models: strided first layer, filter groups, LRN, dropout, overlapping pooling
        dict(_net("alexnet", "train", 128, 227, 1000), name="alexnet_train_b128"),
        # residual networks: 1x1 and 3x3 convolutions with batch normalisation between them
        dict(kind="residual", size=28, wide=512, narrow=128, stride=1, batch=64, precision="3xtf32", fuse=True,
             name="bottleneck_28_b64"),
        # ... and the block that halves the map, with its strided shortcut, in the fast arithmetic
        dict(kind="residual", size=56, wide=512, narrow=128, stride=2, batch=32, precision="tf32", fuse=True,
             name="downsample_56_tf32_b32"),
        # detection: ROI pooling of a 38 x 50 map and two fully connected layers
        dict(kind="frcnn", h=38, w=50, c=512, n=2, rois=256, width=4096, precision="3xtf32", name="frcnn_head_256rois"),
        # spatial transformer
        dict(kind="sampler", h=64, w=64, c=32, n=256, ho=64, wo=64, name="sampler_64x64x32_b256"),
        # a ragged convolution: odd planes, channel counts that are no multiple of a tile, stride 2
        dict(kind="conv", h=57, w=43, c=90, n=13, f=3, k=150, stride=2, pad=1, dilate=1, groups=1, precision="3xtf32",
             name="conv_57x43x90_s2"),
        # segmentation: a score map of 21 classes upsampled by two with a bilinear-sized 4x4 filter bank
        dict(kind="convt", h=35, w=47, c=64, n=8, f=4, k=21, up=2, crop=1, precision="3xtf32", name="convt_35x47_up2"),
        # the trainer's update of all parameters of the benchmark network
        dict(kind="update", net="vgg16", layers=16, width=0, solver="sgd", nesterov=False, name="sgd_update_vgg16"),
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, even over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


_MOST_FLOPS = 4e11      # of a drawn case; the largest listed one has 6e12


def _fit(case, key):
    """Cuts the batch until the case costs no more than a drawn one may."""
    while case[key] > 1 and work(case)["flops"] > _MOST_FLOPS:
        case[key] = (case[key] + 1) // 2
    return case


def draw(rng):
    kind = rng.choice(["net", "net", "net", "residual", "frcnn", "sampler", "conv", "conv", "convt", "update"])
    precision = rng.choice(["3xtf32", "3xtf32", "3xtf32", "tf32"])
    fuse = rng.random() < 0.5
    if kind == "net":
        net = rng.choice(["lenet", "cifar", "alexnet", "vgg16"])
        mode = rng.choice(["train", "infer", "step"] if net == "cifar" else ["train", "infer"])
        size = {"lenet": 28, "cifar": 32, "alexnet": rng.randint(99, 227), "vgg16": rng.randint(64, 256)}[net]
        classes = {"lenet": 0, "cifar": 10}.get(net, rng.choice([20, 205, 1000]))
        batch = _log(rng, 1, {"lenet": 600, "cifar": 500, "alexnet": 128, "vgg16": 32}[net])
        return _fit(_net(net, mode, batch, size, classes, precision, fuse), "batch")
    if kind == "residual":
        narrow = rng.choice([16, 32, 48, 64, 96, 128, 256])
        return _fit(dict(kind=kind, size=rng.randint(7, 56), wide=4 * narrow, narrow=narrow, stride=rng.choice([1, 1, 2]),
                         batch=_log(rng, 1, 64), precision=precision, fuse=fuse), "batch")
    if kind == "frcnn":
        return dict(kind=kind, h=rng.randint(14, 60), w=rng.randint(14, 60), c=rng.choice([128, 256, 384, 512]), n=rng.randint(1, 4),
                    rois=_log(rng, 8, 300), width=rng.choice([1024, 2048, 4096]), precision=precision)
    if kind == "sampler":
        case = dict(kind=kind, h=_log(rng, 12, 100), w=_log(rng, 12, 100), c=_log(rng, 1, 64), n=_log(rng, 1, 256), ho=_log(rng, 12, 80),
                    wo=_log(rng, 12, 80))
        while case["n"] > 1 and work(case)["bytes"] > 1e9:
            case["n"] //= 2
        return case
    if kind == "conv":
        f, groups = rng.choice([1, 3, 3, 3, 5, 7]), rng.choice([1, 1, 1, 2, 4])
        stride, dilate = rng.choice([(1, 1), (1, 1), (1, 2), (2, 1), (2, 1), (3, 1)])
        pad = rng.choice([0, f // 2]) * dilate
        least = max(8, (f - 1) * dilate + 1 - 2 * pad)
        return _fit(dict(kind=kind, h=_log(rng, least, 112), w=_log(rng, least, 112), c=groups * _log(rng, 3, 512 // groups), n=_log(rng, 1, 64), f=f,
                         k=groups * _log(rng, 8, 512 // groups), stride=stride, pad=pad, dilate=dilate, groups=groups,
                         precision=precision), "n")
    if kind == "convt":
        up = rng.choice([2, 2, 3, 4])
        f = rng.choice([up, 2 * up])
        return _fit(dict(kind=kind, h=_log(rng, 5, 64), w=_log(rng, 5, 64), c=_log(rng, 8, 256), n=_log(rng, 1, 32), f=f, k=_log(rng, 8, 128),
                         up=up, crop=(f - up) // 2, precision=precision), "n")
    return dict(kind="update", net="plain", layers=rng.randint(1, 12), width=_log(rng, 16, 640),
                solver=rng.choice(["sgd", "adagrad", "adadelta", "adam", "rmsprop"]), nesterov=rng.random() < 0.5)


def prepare(case, seed):
    return dict(_KINDS[case["kind"]][0](case, torch.Generator(device="cuda").manual_seed(seed)), kind=case["kind"])


def run(state):
    return _KINDS[state["kind"]][1](state)


def work(case):
    kind = case["kind"]
    if kind == "net":
        layers, depth = _chain(case["net"], case["size"], case["classes"])
        if case["mode"] == "infer":
            layers = [l for l in layers if l["type"] != "dropout"]
        # a step reads and writes the parameters and the momentum besides the derivatives
        return _chain_work(_walk(layers, case["size"], case["size"], depth), case["batch"], case["mode"],
                           3 if case["mode"] == "step" else 0)
    if kind == "residual":
        main, short, cin = _residual_chain(case)
        both = [_chain_work(_walk(c, case["size"], case["size"], cin), case["batch"], "train") for c in (main, short) if c]
        ho, wo, co = _walk(main, case["size"], case["size"], cin)[-1][2]
        # x and dx count once, dzdy and the sum come on top
        return {"bytes": sum(b["bytes"] for b in both) - (len(both) - 1) * 8 * case["size"] ** 2 * cin * case["batch"]
                + 8 * ho * wo * co * case["batch"], "flops": sum(b["flops"] for b in both)}
    if kind == "frcnn":
        x, p = case["h"] * case["w"] * case["c"] * case["n"], 49 * case["c"] * case["rois"]
        par, hid = (49 * case["c"] + case["width"] + 2) * case["width"], case["width"] * case["rois"]
        return {"bytes": 4 * (2 * x + p + 2 * par + 3 * hid),
                "flops": 6.0 * case["rois"] * case["width"] * (49 * case["c"] + case["width"])}
    if kind == "sampler":
        x, y, g = (case["n"] * v for v in (case["h"] * case["w"] * case["c"], case["ho"] * case["wo"] * case["c"], 2 * case["ho"] * case["wo"]))
        return {"bytes": 4 * (2 * x + 2 * y + 2 * g), "flops": 40.0 * y}
    if kind in ("conv", "convt"):
        ho, wo = _conv_out(case) if kind == "conv" else _convt_out(case)
        x, y = case["h"] * case["w"] * case["c"] * case["n"], ho * wo * case["k"] * case["n"]
        fan = case["f"] ** 2 * case["c"] // case.get("groups", 1)
        pixels = ho * wo if kind == "conv" else case["h"] * case["w"]
        return {"bytes": 4 * (2 * x + 2 * y + 2 * fan * case["k"]), "flops": 6.0 * pixels * case["n"] * case["k"] * fan}
    par = sum(k * (fs * fs * fc + 1) for fs, fc, k in _update_sizes(case))
    state = 2 if case["solver"] in ("adadelta", "adam") else 1
    return {"bytes": 4 * par * (3 + 2 * state), "flops": 8.0 * par}


def tolerance(case):
    kind = case["kind"]
    fast = case.get("precision") == "tf32"
    if kind == "update":
        return {"rel": 1e-6}
    if kind == "sampler":
        return {"rel": 1e-5}
    if kind in ("conv", "convt"):
        # sums of products of single-precision values; operands rounded to TF32 (2^-11) in the fast arithmetic
        return {"rel": 2e-3 if fast else 1e-5}
    if kind == "net" and case["mode"] == "infer":
        return {"rel": 5e-3 if fast else 2e-5}
    # training through ReLU and max-pooling: an activation within rounding of a tie decides the other way, and the
    # derivatives below it change by whole elements
    return {"rel": 1e-2 if fast else 5e-3, "max": 0.9}
