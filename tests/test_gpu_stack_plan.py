"""EncoderStack's native call: replayed launches give, bit for bit, what issuing every layer gives, for
repeated and for new arguments, more argument sets than are recorded, weights rewritten in place, an
exchanged layer, inside a caller's own capture, and from two host threads in turn."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BATCH, SEQ, HIDDEN, NHEAD, FF = 2, 48, 256, 4, 512


def _layers(et, cuda, seed, n=3):
    return [et.EncoderLayer(et.synth.encoder_layer_weights(seed, l, HIDDEN, FF, std=0.05, fast=True), NHEAD,
                            et.ACT_GELU, device=cuda) for l in range(n)]


def _by_layer(et, layers, x, mask_kind=0, mask=None, vl=None):
    import torch
    ws = torch.empty(max(l.workspace_bytes(BATCH, SEQ) for l in layers), dtype=torch.uint8, device=x.device)
    for l in layers:
        out = torch.empty_like(x)
        l.forward(x, out, BATCH, SEQ, ws, mask_kind, mask, vl)
        x = out
    torch.cuda.synchronize()
    return x


def test_replayed_calls_equal_issued_calls(et, cuda):
    import torch
    layers = _layers(et, cuda, 91)
    stack = et.EncoderStack(layers, BATCH, SEQ, device=cuda)
    xs = [torch.randn((BATCH * SEQ, HIDDEN), device=cuda).half() for _ in range(12)]
    vl = torch.tensor([SEQ, 7], dtype=torch.int32, device=cuda)
    for _ in range(4):  # more inputs than recorded argument sets, two mask kinds each
        for x in xs:
            for kind, v in ((et.MASK_NONE, None), (et.MASK_PADDING, vl)):
                assert torch.equal(stack.forward(x, kind, None, v), _by_layer(et, layers, x, kind, None, v))
    # the contents behind the recorded addresses are read at every call
    xs[0].copy_(xs[1])
    vl.copy_(torch.tensor([3, SEQ], dtype=torch.int32))
    assert torch.equal(stack.forward(xs[0], et.MASK_PADDING, None, vl),
                       _by_layer(et, layers, xs[1], et.MASK_PADDING, None, vl))
    for t in layers[1]._keep:
        if t.dtype == torch.float16 and t.dim() == 2:
            t.mul_(1.5)
    torch.cuda.synchronize()
    assert torch.equal(stack.forward(xs[2]), _by_layer(et, layers, xs[2]))
    # another layer object, another description
    stack.layers[2] = _layers(et, cuda, 92, 1)[0]
    assert torch.equal(stack.forward(xs[2]), _by_layer(et, stack.layers, xs[2]))
    layers[0].desc.act = et.ACT_RELU
    for _ in range(3):
        assert torch.equal(stack.forward(xs[2]), _by_layer(et, stack.layers, xs[2]))
    assert et.device_error() == 0


def test_launch_count_and_capture(et, cuda):
    import torch
    layers = _layers(et, cuda, 93)
    stack = et.EncoderStack(layers, BATCH, SEQ, device=cuda)
    x = torch.randn((BATCH * SEQ, HIDDEN), device=cuda).half()
    counts = []
    for _ in range(4):
        n = et.lib().et_launch_count()
        y = stack.forward(x)
        counts.append(et.lib().et_launch_count() - n)
    assert len(set(counts)) == 1 and counts[0] >= 3 * len(layers)
    want = y.clone()
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        with torch.cuda.graph(g, stream=s):
            stack.forward(x)
    stack.buf[0].zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(stack.buf[0], want)


def test_two_threads_in_turn(et, cuda):
    import torch
    layers = _layers(et, cuda, 94)
    stack = et.EncoderStack(layers, BATCH, SEQ, device=cuda)
    xs = [torch.randn((BATCH * SEQ, HIDDEN), device=cuda).half() for _ in range(2)]
    want = [_by_layer(et, layers, x) for x in xs]
    lock, bad = threading.Lock(), []

    def work(i):
        torch.cuda.set_device(cuda)
        s = torch.cuda.Stream()
        for _ in range(20):
            with lock, torch.cuda.stream(s):
                y = stack.forward(xs[i])
                s.synchronize()
                if not torch.equal(y, want[i]):
                    bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad and et.device_error() == 0
    stack.close()
    stack.close()
    assert np.array_equal(stack.forward(xs[0]).cpu().numpy(), want[0].cpu().numpy())
