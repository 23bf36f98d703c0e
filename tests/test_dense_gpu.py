"""SGEMM on operands that tensor copies can fetch (16-byte aligned columns), which run on the kernel with A in tensor memory:
all orientations at tile edges, against the CPU oracle."""
import numpy as np
import pytest
import torch

from helpers import rel_err

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


# m, n, k: one block; ragged in every dimension (column tiles of 32, 64 and 128); several tiles; a reduction long enough to split
SIZES = [(4, 4, 4), (128, 32, 32), (132, 36, 40), (260, 68, 100), (12, 132, 36), (384, 256, 64), (516, 20, 2052), (1000, 60, 4100)]


@pytest.mark.parametrize("algo", [0, 1])
@pytest.mark.parametrize("trans", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("size", SIZES)
def test_sgemm_aligned(vdnn, oracle, size, trans, algo):
    (m, n, k), (ta, tb), ops = size, trans, vdnn.ops
    rng = np.random.default_rng(m + 3 * n + 7 * k + 2 * ta + tb)
    lda, ldb = (k if ta else m) + 4, ((n if tb else k) + 3) // 4 * 4
    A = rng.standard_normal(lda * (m if ta else k), dtype=np.float32)
    B = rng.standard_normal(ldb * (k if tb else n), dtype=np.float32)
    for ldc, alpha, beta in [(m, 1.0, 0.0), (m, -0.5, 1.0), (m + 3, 0.5, 2.0)]:
        C0 = rng.standard_normal(ldc * n, dtype=np.float32)
        C = dev(C0)
        need = ops.sgemm_workspace_bytes(algo, m, n, k)
        ws = torch.empty(max(need, 4) // 4, device="cuda")
        ops.sgemm(ta, tb, m, n, k, alpha, dev(A), lda, dev(B), ldb, beta, C, ldc, algo_mode=algo, workspace=ws, workspace_bytes=need)
        want = oracle.sgemm(ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C0, ldc).reshape(n, ldc)
        got = C.cpu().numpy().reshape(n, ldc)
        assert rel_err(got[:, :m], want[:, :m]) < 1e-5
        assert np.array_equal(got[:, m:], C0.reshape(n, ldc)[:, m:])
    assert ops.engine_status() == 0


@pytest.mark.parametrize("n,k", [(320, 320), (320, 324), (321, 192), (321, 193), (324, 196), (64, 320), (32, 321), (1000, 256)])
def test_sgemm_around_the_short_reductions(vdnn, oracle, n, k):
    """Sizes at the lines between tiles whose C goes out through shared memory and the others."""
    test_sgemm_aligned(vdnn, oracle, (260, n, k), (0, 1), 0)
    test_sgemm_aligned(vdnn, oracle, (260, n, k), (1, 0), 0)


@pytest.mark.parametrize("rows", [148 * 128, 148 * 128 + 1000])
@pytest.mark.parametrize("n", [8, 64, 128])
def test_sgemm_long_reduction(vdnn, n, rows):
    """One row tile per SM and a reduction of many times the stage ring: the operand stages are reused over and over while
    the copies are what everything waits for.  With rows left over, their tiles are split in a second launch.  The sum of the
    parts has a fixed order: every run gives the same bits."""
    m, k, ops = rows, 4096, vdnn.ops
    gen = torch.Generator(device="cuda").manual_seed(n)
    A, B = torch.randn(m, k, device="cuda", generator=gen), torch.randn(n, k, device="cuda", generator=gen)
    C = torch.empty(n, m, device="cuda")
    want, first = B.double() @ A.double().t(), None
    for _ in range(3):
        ops.sgemm(1, 0, m, n, k, 1.0, A, k, B, k, 0.0, C, m)
        assert float((C.double() - want).abs().max() / want.abs().max()) < 1e-5
        first = C.clone() if first is None else first
        assert torch.equal(C, first)


def test_weight_step_in_place(vdnn):
    """C += alpha * A B^T with many tiles per CTA: old tiles are fetched one ahead through two buffers."""
    m, n, k, ops = 5000, 2000, 68, vdnn.ops
    gen = torch.Generator(device="cuda").manual_seed(1)
    A, B, C = (torch.randn(*s, device="cuda", generator=gen) for s in ((k, m), (k, n), (n, m)))
    want = C.double()
    for _ in range(3):
        want = want - 0.5 * (B.double().t() @ A.double())
        ops.sgemm(0, 1, m, n, k, -0.5, A, m, B, n, 1.0, C, m)
    assert float((C.double() - want).abs().max() / want.abs().max()) < 1e-5
