"""Max-pool gradients of 2 x 2 and 3 x 3 windows at stride 2: planes that share a warp, rows and columns that no window reaches,
one window, bands of several window rows, many blocks; ties, whose first place counts."""
import numpy as np
import pytest
import torch

from helpers import rel_err

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


@pytest.mark.parametrize("n,c,h,w,win", [
    (1, 1, 3, 3, 3), (1, 1, 2, 2, 2), (3, 5, 4, 6, 3), (1, 31, 5, 4, 3), (2, 7, 13, 13, 3), (1, 3, 40, 61, 3), (1, 2, 41, 130, 3), (1, 5, 33, 34, 2),
    (2, 3, 7, 65, 2), (40, 60, 9, 27, 3)])
def test_maxpool_gradient(vdnn, oracle, n, c, h, w, win):
    ops, rng = vdnn.ops, np.random.default_rng(h * w + win)
    x = np.maximum(rng.standard_normal((n, c, h, w)), 0).astype(np.float32)
    P, Q = (h - win) // 2 + 1, (w - win) // 2 + 1
    dy = rng.standard_normal((n, c, P, Q)).astype(np.float32)
    y, dx = oracle.maxpool_fwd(x, (win, win), (2, 2)), torch.full((n, c, h, w), float("nan"), device="cuda")
    ops.maxpool_bwd(n, c, h, w, (win, win), (2, 2), dev(y), dev(dy), dev(x), dx)
    assert rel_err(dx.cpu().numpy(), oracle.maxpool_bwd(y, dy, x, (win, win), (2, 2))) < 1e-6
