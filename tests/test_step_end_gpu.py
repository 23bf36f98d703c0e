"""The last layers of a step (softmax, loss, loss seed, softmax gradient): launched so that each kernel starts beside the one before
it, checked link by link in a chain that nothing synchronises, against float64, at the edges of their register passes, off the
16-byte boundaries, replayed from a graph and with results that are inputs of the next round."""
import numpy as np
import pytest
import torch

import vdnn_implementation_b200 as v

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -24


def softmax64(x):
    e = np.exp(x.astype(np.float64) - x.max(1, keepdims=True).astype(np.float64))
    return e / e.sum(1, keepdims=True)


def tensors(rows, cols, offset, count):
    out = []
    for _ in range(count):
        flat = torch.full((rows * cols + 4,), float("nan"), device="cuda")
        out.append(flat[offset:offset + rows * cols].view(rows, cols))
    return out


def chain(rows, cols, x, label, y, d, dx, out, stream=None):
    v.ops.softmax_fwd(rows, cols, x, y, stream=stream)
    v.ops.loss(rows, cols, y, label, out, stream=stream)
    v.ops.sub(rows * cols, y, label, d, stream=stream)
    v.ops.softmax_bwd(rows, cols, y, d, dx, stream=stream)


def check(x, label, y, d, dx, out):
    x, label, y, d, dx, out = (t.cpu().numpy() for t in (x, label, y, d, dx, out))
    rows = x.shape[0]
    want = softmax64(x)
    # expf within 2 ulp of an argument that was rounded once (|x - m| below 32: 2^-24 * 32 absolute), then the product's rounding
    assert np.abs(y - want).max() <= (32 + 6) * EPS
    assert np.array_equal(d, y - label)
    y64, d64 = y.astype(np.float64), d.astype(np.float64)
    grad = y64 * (d64 - (y64 * d64).sum(1, keepdims=True))
    assert np.all(np.abs(dx - grad) <= 2 * EPS * np.abs(grad) + 1e-14)      # sums in double, one rounding
    p = y64[np.arange(rows), label.argmax(1)]
    assert np.allclose(out, [0.5 * ((y64 - label) ** 2).sum() / rows,
                             -np.log(np.maximum(p, 1e-30)).mean()], rtol=1e-9, atol=1e-12)


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("rows,cols", [(1, 2), (5, 33), (7, 257), (8, 1000), (64, 1000), (3, 2049), (256, 4000)])
def test_chain(rows, cols, offset):
    gen = torch.Generator("cuda").manual_seed(rows * 4001 + cols)
    x, label, y, d, dx = tensors(rows, cols, offset, 5)
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    for _ in range(3):
        x.copy_(torch.randn(rows, cols, device="cuda", generator=gen).clamp_(-8, 8) * 2)
        label.zero_()
        label.scatter_(1, torch.randint(0, cols, (rows, 1), device="cuda", generator=gen), 1.0)
        chain(rows, cols, x, label, y, d, dx, out)
        torch.cuda.synchronize()
        check(x, label, y, d, dx, out)


def test_each_round_reads_the_last():
    """Forty rounds in a graph, x := x - 0.25 dx: a kernel that ran ahead of its predecessor would differ from the rounds run
    one at a time."""
    rows, cols = 64, 1000
    x, label, y, d, dx = tensors(rows, cols, 0, 5)
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    first = torch.randn(rows, cols, device="cuda", generator=torch.Generator("cuda").manual_seed(3)) * 3
    label.zero_()
    label[:, 7] = 1.0
    stream = torch.cuda.Stream()

    def rounds(synchronise):
        for _ in range(40):
            chain(rows, cols, x, label, y, d, dx, out, stream=stream.cuda_stream)
            v.ops.axpy(rows * cols, -0.25, dx, x, stream=stream.cuda_stream)
            if synchronise:
                torch.cuda.synchronize()

    x.copy_(first)
    torch.cuda.synchronize()
    rounds(True)
    want = [t.clone() for t in (x, y, d, dx, out)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        x.copy_(first)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            rounds(False)
        graph.replay()
    torch.cuda.synchronize()
    for got, ref in zip((x, y, d, dx, out), want):
        assert torch.equal(got, ref)
