"""Operator calls from several Python threads: the engine is called without the interpreter lock, and the calls of one context come one at a time."""
import threading
import time

import pytest

pytestmark = pytest.mark.gpu


def _inputs(mat, seed, c=32):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    normal = lambda *s: mat.empty(s).normal_(generator=g)       # noqa: E731
    return normal(14, 14, c, 4), normal(3, 3, c, 64), normal(1, 64), normal(14, 14, 64, 4)


def _calls(nn, ctx, x, f, b, dy):
    y = nn.vl_nnconv(x, f, b, pad=1, relu=True, ctx=ctx)
    out = [y, *nn.vl_nnconv(x, f, b, dy, pad=1, through_relu=True, ctx=ctx), *nn.vl_nnconv(x, f, b, dy, pad=1, ctx=ctx)]
    return out + [nn.vl_nnconvt(dy, f, None, crop=1, ctx=ctx), nn.vl_nnconv(x, f, b, pad=1, ctx=ctx)]


def test_other_threads_run_while_a_call_waits(gpu):
    """Scratch that grows waits for the stream; a thread that only sleeps and counts must go on meanwhile."""
    import torch
    from matconvnet_b200 import capi
    nn, mat, _ = gpu
    x, f, b, dy = _inputs(mat, 1, c=256)
    nn.vl_nnconv(x, f, b, pad=1)                           # kernels loaded, memory in torch's pool
    ctx = capi.Context()
    ctx.reserve_workspace(1 << 20)                          # the filter tile images need 1.2 MB
    ticks, stop = [], threading.Event()

    def count():
        while not stop.is_set():
            time.sleep(0.001)
            ticks.append(time.perf_counter())

    t = threading.Thread(target=count)
    t.start()
    try:
        torch.cuda.synchronize()
        torch.cuda._sleep(600_000_000)                      # about 0.3 s on the stream
        t0 = time.perf_counter()
        nn.vl_nnconv(x, f, b, pad=1, ctx=ctx)
        t1 = time.perf_counter()
    finally:
        stop.set()
        t.join()
    torch.cuda.synchronize()
    assert t1 - t0 > 0.1, "the call did not wait, so it shows nothing"
    assert sum(t0 < s < t1 for s in ticks) > (t1 - t0) / 0.02


@pytest.mark.parametrize("own", [True, False])
def test_threads_with_contexts_of_their_own_and_with_one_between_them(gpu, own):
    """own: a context and a stream per thread.  Not: all threads use the default context on the default stream; a call's flags (fused ReLU, mask,
    bias), scratch and launches must stay together."""
    import torch
    from matconvnet_b200 import capi
    nn, mat, shared = gpu
    data = [_inputs(mat, 10 + i, c=(32, 20, 64, 48)[i]) for i in range(4)]
    want = [_calls(nn, shared, *d) for d in data]
    torch.cuda.synchronize()
    failed = []

    def work(i):
        try:
            ctx = capi.Context() if own else shared
            with torch.cuda.stream(torch.cuda.Stream() if own else torch.cuda.default_stream()):
                for _ in range(40):
                    got = _calls(nn, ctx, *data[i])
                    torch.cuda.current_stream().synchronize()
                    if not all(torch.equal(p, q) for p, q in zip(got, want[i])):
                        failed.append(i)
                if own:
                    ctx.device_status()
        except Exception as e:       # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    assert shared.device_status() == 0


def test_errors_of_a_call_reach_its_own_thread(gpu):
    from matconvnet_b200 import capi
    nn, mat, ctx = gpu
    x, f, b, _ = _inputs(mat, 3)
    seen = {}

    def work(kw, text):
        for _ in range(50):
            try:
                nn.vl_nnconv(x, f, b, ctx=ctx, **kw)
            except capi.VlbError as e:
                seen.setdefault(text, set()).add(text in str(e) and e.code == 7)

    threads = [threading.Thread(target=work, args=a) for a in ((dict(stride=0), "STRIDE"), (dict(pad=-1), "PAD"), (dict(dilate=0), "DILATE"))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert seen == {"STRIDE": {True}, "PAD": {True}, "DILATE": {True}}
