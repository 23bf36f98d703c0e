"""Layers of at most four input channels, against the CPU oracle: every filter with a kernel instance of its own, ragged
images, fewer channels than the instance, more filters than one shared-memory load of weights holds."""
import numpy as np
import pytest
import torch

from helpers import rel_err

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


@pytest.mark.parametrize("n,c,h,w,k,r,pad,stride", [
    (2, 3, 31, 47, 20, 11, 0, 4), (1, 2, 40, 33, 5, 11, 3, 4), (1, 3, 23, 27, 150, 11, 2, 4), (2, 3, 17, 40, 12, 3, 1, 1), (1, 4, 9, 70, 8, 3, 0, 1),
    (3, 1, 20, 21, 6, 5, 2, 1), (2, 4, 11, 37, 7, 5, 1, 1), (2, 3, 33, 30, 9, 7, 3, 2), (1, 4, 19, 25, 5, 7, 0, 2), (1, 1, 8, 8, 3, 3, 2, 1)])
def test_first_layer(vdnn, oracle, n, c, h, w, k, r, pad, stride):
    ops, rng = vdnn.ops, np.random.default_rng(h * w + r)
    x = rng.standard_normal((n, c, h, w), dtype=np.float32)
    wt = rng.standard_normal((k, c, r, r), dtype=np.float32)
    d = ops.conv_desc(n, c, h, w, k, r, r, (pad, pad), (stride, stride))
    P, Q = ops.conv_out_dims(d)
    dy = rng.standard_normal((n, k, P, Q), dtype=np.float32)
    for algo in (0, 1):
        need = max(ops.conv_workspace_bytes(op, algo, d) for op in range(4))
        ws = torch.empty(max(need, 16), dtype=torch.uint8, device="cuda")
        how = {"algo_mode": algo, "workspace": ws, "workspace_bytes": need}
        y = torch.empty(n, k, P, Q, device="cuda")
        ops.conv_fwd(d, dev(x), dev(wt), y, **how)
        assert rel_err(y.cpu().numpy(), oracle.conv_fwd(x, wt, (pad, pad), (stride, stride))) < 1e-5
        dx0 = rng.standard_normal(x.shape, dtype=np.float32)
        for alpha, beta in ((1.0, 0.0), (0.5, 2.0)):
            dx = dev(dx0)
            ops.conv_bwd_data(d, dev(wt), dev(dy), dx, alpha=alpha, beta=beta, **how)
            want = alpha * oracle.conv_bwd_data(wt, dy, x.shape, (pad, pad), (stride, stride)) + beta * dx0
            assert rel_err(dx.cpu().numpy(), want) < 1e-5
        dw = torch.empty(wt.shape, device="cuda")
        ops.conv_bwd_filter(d, dev(x), dev(dy), dw, **how)
        assert rel_err(dw.cpu().numpy(), oracle.conv_bwd_filter(x, dy, wt.shape, (pad, pad), (stride, stride))) < 1e-5
    assert ops.engine_status() == 0


def _dgrad_error(vdnn, n, c, h, w, k, r, pad, stride, alpha=1.0, beta=0.0):
    """Relative error of a data gradient against float64 on the device."""
    ops = vdnn.ops
    d = ops.conv_desc(n, c, h, w, k, r, r, (pad, pad), (stride, stride))
    gen = torch.Generator(device="cuda").manual_seed(100 * r + stride)
    wt = torch.randn(k, c, r, r, device="cuda", generator=gen)
    dy = torch.randn((n, k) + tuple(ops.conv_out_dims(d)), device="cuda", generator=gen)
    dx = torch.randn(n, c, h, w, device="cuda", generator=gen)
    x = torch.zeros(dx.shape, dtype=torch.float64, device="cuda", requires_grad=True)
    y = torch.nn.functional.conv2d(x, wt.double(), padding=pad, stride=stride)
    want = alpha * torch.autograd.grad(y, x, dy.double())[0] + beta * dx.double()
    ops.conv_bwd_data(d, wt, dy, dx, alpha=alpha, beta=beta)
    return ((dx.double() - want).abs().max() / want.abs().max()).item()


# Every odd square filter up to 11 at every stride up to 4: on few positions (a row per thread, or the kernels beside it) and
# on enough of them for the rows of a thread to fill the GPU.  Sums of at most 6 * 121 products in fp32: 726 * 2^-24 = 4e-5 at
# the very worst, a few 1e-7 in practice.
@pytest.mark.parametrize("c", [2, 3, 4])
@pytest.mark.parametrize("r", [3, 5, 7, 9, 11])
@pytest.mark.parametrize("stride", [1, 2, 3, 4])
def test_first_layer_dgrad_every_filter(vdnn, c, r, stride):
    assert _dgrad_error(vdnn, 2, c, 29, 38, 6, r, r // 2, stride) < 1e-5
    n, h, w = {1: (16, 97, 101), 2: (32, 197, 203), 3: (16, 133, 147), 4: (16, 133, 147)}[stride]
    assert _dgrad_error(vdnn, n, c, h, w, 5, r, 0, stride, 0.5, 2.0) < 1e-5
    assert vdnn.ops.engine_status() == 0


# A few positions to either side of the lines: half a block of 256 for each of 148 SMs (5 x 5 / 1: eight rows a thread), a
# seventh of a block of 384 (11 x 11 / 4: two rows a thread).
@pytest.mark.parametrize("n,h,w,r,stride", [(73, 16, 124, 5, 1), (74, 16, 124, 5, 1), (75, 16, 124, 5, 1), (14, 64, 127, 11, 4), (15, 64, 131, 11, 4),
                                            (18, 64, 131, 11, 4)])
def test_first_layer_dgrad_around_the_lines(vdnn, n, h, w, r, stride):
    assert _dgrad_error(vdnn, n, 3, h, w, 4, r, r // 2, stride) < 1e-5
