"""Convolutions on operands split into pairs of 16-bit floats, against float64.

An element is carried to 2^-22 of itself (down to 2^-28 of its tensor's largest), the product of two lower halves is left out
(2^-24), and a chain of at most 24 tensor-core additions truncates each to 24 bits: at worst 2^-21.4 + 24 * 2^-24 = 1.8e-6 of a
sum of terms of one sign.  With signs at random both average out; 2e-6 in the 2-norm leaves that bound in place."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BOUND = 2e-6


@pytest.fixture
def tensor_cores(vdnn):
    vdnn.ops.set_engine(vdnn.ENGINE_TCGEN05)       # small shapes too
    yield vdnn.ops
    vdnn.ops.set_engine(vdnn.ENGINE_AUTO)


def rel(got, want):
    return ((got.double() - want).norm() / want.norm().clamp_min(1e-300)).item()


def make(ops, n, c, h, w, k, r, s, pad, offset=0, seed=0, stride=1):
    gen = torch.Generator(device="cuda").manual_seed(seed + n + c + h + k)
    d = ops.conv_desc(n, c, h, w, k, r, s, pad, (stride, stride))
    P, Q = ops.conv_out_dims(d)

    def tensor(*shape):
        count = torch.Size(shape).numel()
        return torch.randn(count + 4, device="cuda", generator=gen)[offset:offset + count].view(shape)

    t = {"x": torch.relu(tensor(n, c, h, w)) if offset == 0 else tensor(n, c, h, w), "w": tensor(k, c, r, s) * 0.1 if offset == 0 else tensor(k, c, r, s),
         "dy": tensor(n, k, P, Q), "b": tensor(k)}
    for name, like in (("y", "dy"), ("dx", "x"), ("dw", "w"), ("db", "b")):
        t[name] = tensor(*t[like].shape)
    return d, t


def run(ops, d, t, **backward):
    for op, call in ((0, lambda **how: ops.conv_fwd(d, t["x"], t["w"], t["y"], bias=t["b"], **how)),
                     (3, lambda **how: ops.conv_bwd_data_filter_bias(d, t["w"], t["x"], t["dy"], t["dx"], t["dw"], t["db"], **backward, **how))):
        need = ops.conv_workspace_bytes(op, 1, d)
        work = torch.full((need,), 0xff, dtype=torch.uint8, device="cuda")      # NaN in every format: nothing is read before it is written
        call(algo_mode=1, workspace=work, workspace_bytes=need)
    assert ops.engine_status() == 0


def exact(t, pad, stride=1):
    x, w = t["x"].double().requires_grad_(), t["w"].double().requires_grad_()
    y = torch.nn.functional.conv2d(x, w, t["b"].double(), padding=pad, stride=stride)
    dx, dw = torch.autograd.grad(y, (x, w), t["dy"].double())
    return y.detach(), dx, dw, t["dy"].double().sum((0, 2, 3))


SHAPES = [  # n, c, h, w, k, r, s, pad
    (1, 32, 5, 7, 32, 3, 3, (1, 1)),          # less than a tile everywhere, half-empty channel blocks
    (3, 64, 17, 15, 64, 3, 3, (1, 1)),        # 64 columns; planes of odd size
    (2, 96, 16, 16, 128, 3, 3, (1, 1)),       # 128 columns on a pair; a block and a half of channels
    (5, 128, 12, 10, 160, 3, 3, (1, 1)),      # a ragged second column tile
    (2, 192, 9, 31, 256, 3, 3, (1, 1)),       # 256 columns; an odd number of channel blocks on pairs
    (1, 320, 8, 8, 288, 3, 3, (1, 1)),        # ... and a ragged second column tile
    (7, 64, 4, 3, 256, 1, 1, (0, 0)),         # 1 x 1; one channel block: the filter gradient on single CTAs
    (4, 160, 6, 5, 64, 1, 1, (0, 0)),
    (2, 64, 14, 13, 96, 5, 5, (2, 2)),        # 25 taps: several CTAs share the groups
    (2, 64, 13, 14, 64, 3, 5, (0, 2)),        # filter and padding differ by direction
    (2, 32, 21, 19, 64, 9, 9, (4, 4)),        # the widest strip
    (2, 64, 15, 24, 64, 3, 11, (1, 5)),       # wider: one strip per tap
    (2, 64, 15, 24, 300, 11, 11, (0, 0)),
    (3, 32, 6, 6, 64, 3, 3, (2, 2)),          # the output is larger than the image
    (2, 64, 5, 5, 64, 2, 2, (3, 3)),          # padding wider than the filter
    (1, 64, 130, 3, 64, 3, 3, (1, 1)),
    (2, 37, 9, 11, 50, 3, 3, (1, 1)),         # channels and filters off every block
    (3, 8, 14, 9, 130, 5, 5, (2, 2)),
    (1, 129, 7, 7, 257, 3, 3, (1, 1)),
]


STRIDED = [  # n, c, h, w, k, r, s, pad, stride: computed in folded form
    (3, 3, 39, 47, 96, 11, 11, (0, 0), 4),    # a first layer; pixels that no tap reaches
    (2, 3, 30, 31, 64, 7, 7, (3, 3), 2),
    (2, 1, 23, 24, 32, 5, 5, (2, 1), 3),
    (3, 32, 14, 15, 64, 3, 3, (1, 1), 2),
    (2, 50, 9, 20, 130, 3, 3, (1, 1), 2),     # channels off every block
    (4, 64, 13, 13, 256, 1, 1, (0, 0), 2),    # three pixels of four unused
    (2, 19, 17, 70, 40, 2, 5, (0, 2), 3),     # the filter smaller than the stride in one direction
    (1, 16, 150, 9, 64, 3, 3, (0, 0), 4),
]


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("case", [shape + (1,) for shape in SHAPES] + STRIDED, ids=str)
def test_against_float64(tensor_cores, case, offset):
    """offset 1: every tensor one float off the 16-byte boundaries."""
    n, c, h, w, k, r, s, pad, stride = case
    d, t = make(tensor_cores, n, c, h, w, k, r, s, pad, offset, stride=stride)
    run(tensor_cores, d, t)
    for got, want in zip((t["y"], t["dx"], t["dw"], t["db"]), exact(t, pad, stride)):
        assert rel(got, want) < BOUND


@pytest.mark.parametrize("stride", [1, 2])
def test_scaling_and_update_in_place(tensor_cores, stride):
    d, t = make(tensor_cores, 4, 64, 12, 12, 128, 3, 3, (1, 1), stride=stride)
    y, dx, dw, db = exact(t, (1, 1), stride)
    w0, b0, dx0 = t["w"].double(), t["b"].double(), t["dx"].double()
    want = w0 - 0.25 * dw, b0 - 0.5 * db, 2.0 * dx + 0.5 * dx0
    t["dw"], t["db"] = t["w"], t["b"]
    run(tensor_cores, d, t, alpha_dx=2.0, beta_dx=0.5, alpha_w=-0.25, beta_w=1.0, alpha_b=-0.5, beta_b=1.0)
    for got, ref in zip((t["w"], t["b"], t["dx"]), want):
        assert rel(got, ref) < BOUND


@pytest.mark.parametrize("sx, sw, sdy", [(1e30, 1e-30, 1e-20), (1e-30, 1e25, 1e5), (1e-37, 1.0, 1e37), (1.0, 1e-38, 1e36)])
def test_extreme_magnitudes(tensor_cores, sx, sw, sdy):
    d, t = make(tensor_cores, 3, 64, 9, 9, 64, 3, 3, (1, 1))
    for name, scale in (("x", sx), ("w", sw), ("dy", sdy)):
        t[name] *= scale
    t["b"].zero_()
    run(tensor_cores, d, t)
    for name, got, want in zip(("y", "dx", "dw"), (t["y"], t["dx"], t["dw"]), exact(t, (1, 1))):
        # operands near the end of the range of fp32 have lost bits themselves, and so has a result there
        tiny = want.abs().max().item() < 1e-36
        assert tiny or rel(got, want) < BOUND, name


@pytest.mark.parametrize("beta", [0.0, 1.0])
@pytest.mark.parametrize("case", [(6, 64, 10, 11, 64, 3, 3, (1, 1)), (6, 128, 8, 8, 256, 3, 3, (1, 1))], ids=str)
def test_operands_of_wide_range(tensor_cores, case, beta):
    """Images 2^-40 of the largest one: no scale holds both in 16 bits.  Every image keeps the precision of fp32."""
    n, c, h, w, k, r, s, pad = case
    d, t = make(tensor_cores, n, c, h, w, k, r, s, pad)
    t["x"][1::2] *= 2.0 ** -40
    t["dy"][0::2] *= 2.0 ** -40
    t["b"].zero_()
    y, dx, dw, db = exact(t, pad)
    dx0, dw0 = t["dx"].double(), t["dw"].double()
    dx0[0::2] = 0
    t["dx"][0::2] = 0
    run(tensor_cores, d, t, beta_dx=beta, beta_w=beta)
    for i in range(n):
        assert rel(t["y"][i], y[i]) < BOUND and rel(t["dx"][i], dx[i] + beta * dx0[i]) < BOUND
    assert rel(t["dw"], dw + beta * dw0) < BOUND and rel(t["db"], db) < BOUND


def test_zeros_infinities_and_nan(tensor_cores):
    d, t = make(tensor_cores, 3, 64, 20, 20, 64, 3, 3, (1, 1))
    x = t["x"].clone()
    y = exact(t, (1, 1))[0]
    t["x"][1, 5, 10, 10], t["x"][2, 7, 3, 4] = float("inf"), float("nan")
    run(tensor_cores, d, t)
    near = torch.zeros(3, 20, 20, dtype=torch.bool, device="cuda")
    near[1, 9:12, 9:12] = near[2, 2:5, 3:6] = True
    far = (~near)[:, None].expand_as(y)
    assert not torch.isfinite(t["y"].permute(0, 2, 3, 1)[near]).any()
    assert rel(t["y"][far], y[far]) < BOUND
    t["x"].zero_()
    run(tensor_cores, d, t)
    assert torch.equal(t["y"], t["b"].view(1, -1, 1, 1).expand_as(t["y"])) and not t["dw"].any()
    t["x"].copy_(x)
    t["dy"].zero_()
    run(tensor_cores, d, t)
    assert not t["dx"].any() and not t["dw"].any() and not t["db"].any()


def test_results_do_not_differ_from_run_to_run(vdnn):
    ops = vdnn.ops
    d, t = make(ops, 32, 64, 56, 56, 64, 3, 3, (1, 1))
    run(ops, d, t)
    first = [t[name].clone() for name in ("y", "dx", "dw")]
    run(ops, d, t)
    assert all(torch.equal(a, t[name]) for a, name in zip(first, ("y", "dx", "dw")))
