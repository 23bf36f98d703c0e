"""Data gradients of stride-1 layers without workspace on enough pixels for a kernel that never splits the reduction: boxes that
cross images, column tiles of 96 and 128 with columns to spare, filter counts that fill neither a chunk nor a 16-byte copy,
padding on one axis, maps wider than a box; and one size below the rule's limit."""
import numpy as np
import pytest
import torch

from helpers import rel_err

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


@pytest.mark.parametrize("n,c,h,w,k,r,s,pad", [
    (64, 70, 13, 17, 7, 5, 5, (2, 2)), (39, 230, 13, 17, 33, 3, 3, (1, 1)), (1, 96, 73, 250, 8, 3, 3, (0, 1)), (14, 190, 7, 128, 5, 7, 5, (3, 2)),
    (1400, 90, 4, 3, 1, 3, 3, (1, 1)), (10, 70, 13, 17, 7, 3, 3, (1, 1))])
def test_dgrad_unsplit(vdnn, oracle, n, c, h, w, k, r, s, pad):
    ops, rng = vdnn.ops, np.random.default_rng(h * w + r)
    d = ops.conv_desc(n, c, h, w, k, r, s, pad, (1, 1))
    P, Q = ops.conv_out_dims(d)
    wt = rng.standard_normal((k, c, r, s), dtype=np.float32)
    dy = rng.standard_normal((n, k, P, Q), dtype=np.float32)
    dx0 = rng.standard_normal((n, c, h, w), dtype=np.float32)
    plain = oracle.conv_bwd_data(wt, dy, dx0.shape, pad, (1, 1))
    for alpha, beta in ((1.0, 0.0), (0.5, 2.0)):
        dx = dev(dx0)
        ops.conv_bwd_data(d, dev(wt), dev(dy), dx, alpha=alpha, beta=beta)
        assert rel_err(dx.cpu().numpy(), alpha * plain + beta * dx0) < 1e-5
    assert ops.engine_status() == 0


@pytest.mark.parametrize("n,c,h,w,k,r", [(64, 70, 13, 17, 7, 5), (40, 230, 14, 17, 33, 3), (1, 96, 73, 250, 8, 3)])
def test_perf_opt_dgrad_off_blocks_of_32_runs_on_packed_weights(vdnn, oracle, n, c, h, w, k, r):
    """With workspace these run on the contraction that reads packed weights: right in the bytes that are reported, refused
    below them (too little workspace is an error, not a change of algorithm)."""
    ops, rng = vdnn.ops, np.random.default_rng(h * w + r)
    d = ops.conv_desc(n, c, h, w, k, r, r, (r // 2,) * 2, (1, 1))
    wt = rng.standard_normal((k, c, r, r), dtype=np.float32)
    dy = rng.standard_normal((n, k, h, w), dtype=np.float32)
    need = ops.conv_workspace_bytes(1, 1, d)
    assert need > 0
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    dx = torch.empty(n, c, h, w, device="cuda")
    ops.conv_bwd_data(d, dev(wt), dev(dy), dx, algo_mode=1, workspace=ws, workspace_bytes=need)
    assert rel_err(dx.cpu().numpy(), oracle.conv_bwd_data(wt, dy, (n, c, h, w), (r // 2,) * 2, (1, 1))) < 1e-5
    with pytest.raises(vdnn.VdnnError) as e:
        ops.conv_bwd_data(d, dev(wt), dev(dy), dx, algo_mode=1, workspace=ws, workspace_bytes=need - 4)
    assert e.value.status == -3
    assert ops.engine_status() == 0


# Both sides of the choice between the halo kernel and the gather without workspace: one wave of tiles and a little more than
# one, columns that fill the gather's tiles badly and well, rows wider than a box, boxes over many small images, few filters.
@pytest.mark.parametrize("n,c,h,w,k,r,s,pad", [
    (1, 300, 31, 250, 20, 3, 3, (1, 1)), (700, 300, 4, 3, 24, 3, 3, (1, 1)), (24, 300, 14, 17, 40, 3, 3, (0, 1)), (25, 300, 14, 17, 40, 3, 3, (1, 1)),
    (48, 256, 14, 14, 16, 3, 3, (1, 1)), (3, 96, 40, 250, 24, 3, 5, (1, 2)), (3, 130, 20, 21, 9, 5, 5, (2, 1)), (10, 70, 13, 17, 7, 3, 3, (1, 1))])
def test_dgrad_either_side_of_the_choice(vdnn, oracle, n, c, h, w, k, r, s, pad):
    test_dgrad_unsplit(vdnn, oracle, n, c, h, w, k, r, s, pad)
