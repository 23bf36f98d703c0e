"""Edges of the launch shapes of the bandwidth-bound kernels, against the CPU oracle."""
import numpy as np
import pytest
import torch

from helpers import rel_err

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


# planes of 1 .. 31 values are read along rows, larger ones by a cluster per channel; float4 or single values
@pytest.mark.parametrize("n,k,pq", [(1, 1, 1), (64, 40, 1), (300, 33, 1), (5, 7, 4), (40, 3, 25), (3, 35, 31), (3, 5, 32), (2, 96, 169), (70, 3, 3025),
                                    (9, 2, 20000)])
def test_bias(vdnn, oracle, n, k, pq):
    rng = np.random.default_rng(n + k + pq)
    dy = rng.standard_normal((n, k, 1, pq), dtype=np.float32)
    db0 = rng.standard_normal(k, dtype=np.float32)
    for alpha, beta in [(1.0, 0.0), (-0.1, 1.0), (0.5, 2.0)]:
        db = dev(db0)
        vdnn.ops.conv_bwd_bias(n, k, pq, dev(dy), db, alpha=alpha, beta=beta)
        assert rel_err(db.cpu().numpy(), oracle.conv_bwd_bias(dy, alpha=alpha, beta=beta, db=db0)) < 1e-5
    y = dev(dy)
    vdnn.ops.add_bias(n, k, pq, dev(db0), y)
    assert np.array_equal(y.cpu().numpy(), dy + db0.reshape(1, k, 1, 1))


@pytest.mark.parametrize("rows,cols", [(1, 1), (7, 33), (8, 128), (9, 129), (200, 1000), (3, 2048), (2, 2049), (1, 5000)])
def test_head(vdnn, oracle, rows, cols):
    ops, rng = vdnn.ops, np.random.default_rng(rows * cols)
    x = (4 * rng.standard_normal((rows, cols), dtype=np.float32)).astype(np.float32)
    label = np.eye(cols, dtype=np.float32)[rng.integers(cols, size=rows)]
    y, dx, loss = torch.empty(rows, cols, device="cuda"), torch.empty(rows, cols, device="cuda"), torch.empty(2, dtype=torch.float64, device="cuda")
    ops.softmax_fwd(rows, cols, dev(x), y)
    want = oracle.softmax_fwd(x)
    assert rel_err(y.cpu().numpy(), want) < 1e-6
    ops.loss(rows, cols, dev(want), dev(label), loss)
    assert np.allclose(loss.cpu().numpy(), oracle.loss(want, label), rtol=1e-12, atol=1e-15)
    ops.softmax_bwd(rows, cols, dev(want), dev(want - label), dx)
    assert rel_err(dx.cpu().numpy(), oracle.softmax_bwd(want, want - label)) < 1e-6


@pytest.mark.parametrize("beta", [0.75, 0.6])
@pytest.mark.parametrize("n,c,hw", [(1, 1, 1), (2, 15, 63), (1, 16, 64), (2, 17, 65), (1, 65, 130), (2, 130, 9)])
def test_lrn(vdnn, oracle, n, c, hw, beta):
    ops, rng = vdnn.ops, np.random.default_rng(c * hw)
    x = (3 * rng.standard_normal((n, c, hw, 1), dtype=np.float32)).astype(np.float32)
    dy = rng.standard_normal(x.shape, dtype=np.float32)
    y, dx = torch.empty(x.shape, device="cuda"), torch.empty(x.shape, device="cuda")
    how = {"alpha": 0.3, "beta": beta, "k": 2.0}
    ops.lrn_fwd(n, c, hw, dev(x), y, **how)
    want = oracle.lrn_fwd(x, **how)
    assert rel_err(y.cpu().numpy(), want) < 1e-6
    ops.lrn_bwd(n, c, hw, dev(x), dev(want), dev(dy), dx, **how)
    assert rel_err(dx.cpu().numpy(), oracle.lrn_bwd(x, want, dy, **how)) < 1e-5


# bands of rows: one band, several, a last one of one row; rows and columns below the last window; windows of any shape
@pytest.mark.parametrize("h,w,win,stride", [(55, 55, 3, 2), (56, 58, 3, 2), (3, 3, 3, 2), (129, 33, 3, 2), (14, 14, 2, 2), (15, 17, 2, 2), (31, 29, 5, 3),
                                            (12, 13, 4, 4), (9, 9, 3, 1), (90, 70, 2, 3)])
def test_maxpool(vdnn, oracle, h, w, win, stride):
    ops, rng, n, c = vdnn.ops, np.random.default_rng(h * w + win), 2, 3
    x = rng.integers(-3, 4, size=(n, c, h, w)).astype(np.float32)          # many ties
    P, Q = (h - win) // stride + 1, (w - win) // stride + 1
    y, dx = torch.empty(n, c, P, Q, device="cuda"), torch.full((n, c, h, w), 7.0, device="cuda")
    ops.maxpool_fwd(n, c, h, w, (win, win), (stride, stride), dev(x), y)
    want = oracle.maxpool_fwd(x, (win, win), (stride, stride))
    assert np.array_equal(y.cpu().numpy(), want)
    dy = rng.integers(-8, 9, size=want.shape).astype(np.float32)           # sums of up to nine of these are exact
    ops.maxpool_bwd(n, c, h, w, (win, win), (stride, stride), y, dev(dy), dev(x), dx)
    assert np.array_equal(dx.cpu().numpy(), oracle.maxpool_bwd(want, dy, x, (win, win), (stride, stride)))


def test_parameters_round_trip(vdnn):
    """Tensors above the direct-copy limit move in 2 MB chunks on several threads, whatever their size and host alignment."""
    sizes = [(63, 1), (65, 1024), (700, 1001), (1500, 1400)]
    specs, n = [], 2
    for k, cin in sizes:
        specs.append((vdnn.FC_GEMM, n, cin, 1, 1, 0, 0, 0, 0, k, 1, 1))
    for spec in specs:
        net = vdnn.Network("CUSTOM_CNN", "VDNN_NONE", "VDNN_MEMORY_OPT_ALGO", device=0, pool_bytes=1e9,
                           custom_layers=[spec, (vdnn.SOFTMAX, n, spec[9], 1, 1, 0, 0, 0, 0, 0, 0, 0)])
        try:
            count = net.tensor_size(0, vdnn.abi.TENSOR_WEIGHT)
            assert count == spec[2] * spec[9]
            values = np.random.default_rng(count).standard_normal(count, dtype=np.float32)
            net.write_tensor(0, vdnn.abi.TENSOR_WEIGHT, values)
            assert np.array_equal(net.weights(0), values)
        finally:
            net.close()
