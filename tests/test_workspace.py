"""Workspace figures follow the kernel that takes a shape: what runs without workspace reports none (a memory manager would
allocate it, trace it and count it into its peak), and the call runs in what is reported."""
import pytest
import torch

# n, c, h, w, k, r, pad, stride, operations (0 forward, 1 data gradient, 2 filter gradient) that use no workspace
NO_WORKSPACE = [
    (8, 3, 64, 64, 64, 3, 1, 1, (0, 1)),        # first layers: kernels of their own
    (3, 2, 30, 40, 132, 3, 1, 1, (0, 1)),
    (4, 3, 67, 67, 32, 11, 0, 4, (1,)),
    (4, 4, 33, 35, 16, 3, 1, 2, (1,)),          # ... a phase at a time
    (2, 2, 20, 24, 12, 6, 2, 1, (1,)),          # ... a thread for each pixel
    (64, 64, 6, 6, 256, 6, 0, 1, (0, 1, 2)),    # full extent: a dense product
    (200, 16, 5, 5, 132, 5, 0, 1, (0, 1, 2)),
]
# figures that must stay: the contraction reads packed weights and leaves parts
WITH_WORKSPACE = [
    (4, 48, 27, 31, 80, 3, 1, 1, (0, 1, 2)),
    (32, 120, 40, 38, 50, 3, 1, 1, (0, 1, 2)),
    (8, 64, 14, 14, 64, 3, 1, 2, (0, 1, 2)),
    (64, 15, 3, 3, 130, 3, 0, 1, (0,)),         # full extent, rows of 135 floats: no tensor copies
]


def _desc(ops, case):
    n, c, h, w, k, r, pad, st = case[:8]
    return ops.conv_desc(n, c, h, w, k, r, r, (pad, pad), (st, st))


@pytest.mark.parametrize("case", NO_WORKSPACE, ids=str)
def test_kernels_without_workspace_report_none(vdnn, case):
    ops = vdnn.ops
    d = _desc(ops, case)
    figures = [ops.conv_workspace_bytes(op, 1, d) for op in range(4)]
    assert [figures[op] for op in case[8]] == [0] * len(case[8]), figures
    assert figures[3] == max(figures[1], figures[2])


@pytest.mark.parametrize("case", WITH_WORKSPACE, ids=str)
def test_contractions_report_what_they_use(vdnn, case):
    d = _desc(vdnn.ops, case)
    assert all(vdnn.ops.conv_workspace_bytes(op, 1, d) > 0 for op in case[8])


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("case", NO_WORKSPACE + WITH_WORKSPACE, ids=str)
def test_each_operation_runs_in_the_bytes_it_reports(vdnn, case, offset):
    """Tensors on 16-byte boundaries and one float off them, each operation with its own figure, against float64."""
    ops = vdnn.ops
    n, c, h, w, k, r, pad, st = case[:8]
    d = _desc(ops, case)
    P, Q = ops.conv_out_dims(d)
    gen = torch.Generator(device="cuda").manual_seed(n + c + k)

    def tensor(*shape, scale=1.0):
        count = 1
        for extent in shape:
            count *= extent
        flat = torch.randn(count + 4, device="cuda", generator=gen) * scale
        return flat[offset:offset + count].view(shape)

    x, wt, dy = tensor(n, c, h, w), tensor(k, c, r, r, scale=0.1), tensor(n, k, P, Q)
    y, dx, dw = tensor(n, k, P, Q), tensor(n, c, h, w), tensor(k, c, r, r)
    calls = [lambda how: ops.conv_fwd(d, x, wt, y, **how), lambda how: ops.conv_bwd_data(d, wt, dy, dx, **how),
             lambda how: ops.conv_bwd_filter(d, x, dy, dw, **how)]
    for op, call in enumerate(calls):
        need = ops.conv_workspace_bytes(op, 1, d)
        work = torch.empty(need, dtype=torch.uint8, device="cuda") if need else None
        call({"algo_mode": 1, "workspace": work, "workspace_bytes": need})
    x64, w64, dy64 = (t.double().requires_grad_() for t in (x, wt, dy))
    y64 = torch.nn.functional.conv2d(x64, w64, padding=pad, stride=st)
    dx64, dw64 = torch.autograd.grad(y64, (x64, w64), dy64.detach())
    for got, want in ((y, y64), (dx, dx64), (dw, dw64)):
        # fp32 sums of at most 46,656 terms, each product exact to 2^-21 or better
        assert ((got.double() - want).norm() / want.norm()).item() < 1e-5
    assert ops.engine_status() == 0
