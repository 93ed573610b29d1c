"""Edges of the convolution's row tiling on the GPU against the float64 oracle
(oracle/conv_ref.py): planes short enough for one run of rows and planes that
need three bands, single-row planes, ragged widths around the 8-voxel groups and
the 4-group tiles, odd channel-group counts, split and padded output channels,
short and long K, and outputs that are only element-aligned.

Tolerances as FP32 accumulation of BF16 products gives them (at most 3456
terms): 1e-4 of the output's scale, plus BF16 rounding (2^-8) for the forward
pass."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPES = [  # (batch, d, h, w, cin, cout, taps)
    (1, 1, 1, 1, 8, 8, 27), (2, 3, 1, 9, 8, 24, 27),     # single-row planes, two taps per MMA not possible
    (1, 2, 17, 31, 16, 16, 27), (1, 2, 18, 33, 8, 40, 27),  # one run of rows / three bands; ragged x tiles
    (3, 3, 3, 8, 24, 128, 27), (1, 2, 2, 3, 120, 8, 27),  # odd channel groups, split N, long K
    (17, 2, 15, 65, 16, 16, 27),                          # wide tiles whose last x groups are empty
    (1, 1, 3, 5, 8, 16, 1), (2, 5, 7, 11, 72, 104, 1),    # pointwise: partial rows of 32 voxels
]


@pytest.fixture(scope="module")
def ops(wt_lib):
    from windtunnel.net import Ops
    return Ops()


def offset_tensor(shape, dtype, fill):
    """A tensor of this shape that starts one element past an aligned address, and its storage."""
    flat = torch.full((int(np.prod(shape)) + 1,), fill, dtype=dtype, device="cuda")
    return flat[1:].view(shape), flat


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("case", SHAPES)
def test_forward_and_data_gradient(ops, case, aligned):
    from oracle import conv_ref as ref
    b, d, h, w, cin, cout, taps = case
    rng = np.random.default_rng(sum(case))
    x = ref.bf16_round(rng.standard_normal((b, d, h, w, cin)))
    wt = ref.bf16_round(rng.standard_normal((cout, taps, cin)) / np.sqrt(taps * cin))
    dy = ref.bf16_round(rng.standard_normal((b, d, h, w, cout)))
    bias = rng.standard_normal(cout).astype(np.float32) * 0.1

    def dev(a):
        return torch.tensor(np.ascontiguousarray(a, np.float32), device="cuda").to(torch.bfloat16)

    if aligned:
        y = torch.empty((b, d, h, w, cout), dtype=torch.bfloat16, device="cuda")
        dx = torch.empty((b, d, h, w, cin), dtype=torch.float32, device="cuda")
    else:
        (y, yf), (dx, dxf) = offset_tensor((b, d, h, w, cout), torch.bfloat16, 7.0), offset_tensor((b, d, h, w, cin), torch.float32, 7.0)
    ops.conv_forward(dev(x), dev(wt), torch.tensor(bias, device="cuda"), y, True)
    ops.conv_backward_data(dev(dy), dev(np.transpose(wt, (2, 1, 0))), dx, cin, cout, taps)
    ops.check()
    want = ref.conv3d(x, wt, bias, True)
    got = y.float().cpu().numpy().astype(np.float64)
    assert np.all(np.abs(got - want) <= 2.0 ** -8 * np.abs(want) + 1e-4 * np.abs(want).max())
    want = ref.conv3d_backward_data(dy, wt)
    assert np.abs(dx.cpu().numpy() - want).max() <= 1e-4 * np.abs(want).max()
    if not aligned:
        assert float(yf[0]) == 7.0 and float(dxf[0]) == 7.0


WEIGHT_SHAPES = SHAPES + [
    (1, 17, 65, 66, 88, 8, 27),    # enough splits for all channels in a block: one MMA per dy (N = 96)
    (1, 8, 160, 161, 8, 16, 27),   # enough splits for the three dx in a block; ragged last x group
    (1, 8, 160, 160, 48, 72, 27),  # the same at the most accumulator columns (432), M = 128
    (2, 9, 31, 30, 40, 64, 27),    # channels in chunks, the last one short; M = 64
]


@pytest.mark.parametrize("case", WEIGHT_SHAPES)
def test_weight_gradient(ops, case):
    """FP32 sums of at most 9216 products per split: 1e-4 of the output's scale."""
    from oracle import conv_ref as ref
    b, d, h, w, cin, cout, taps = case
    rng = np.random.default_rng(sum(case))
    x = ref.bf16_round(rng.standard_normal((b, d, h, w, cin)))
    dy = ref.bf16_round(rng.standard_normal((b, d, h, w, cout)))
    xs, ds = (torch.tensor(np.ascontiguousarray(a, np.float32), device="cuda").to(torch.bfloat16) for a in (x, dy))
    ws = torch.empty(max(1, ops.workspace_bytes(xs.shape, cin, cout, taps) // 4), device="cuda")
    dw = torch.full((cout, taps, cin), 7.0, device="cuda")
    ops.conv_backward_weight(xs, ds, dw, ws, taps)
    ops.check()
    want = ref.conv3d_backward_weight(x, dy, taps)
    assert np.abs(dw.cpu().numpy() - want).max() <= 1e-4 * np.abs(want).max()


def test_weight_gradient_keeps_infinities_in_their_taps(ops):
    """An infinite input in the last column of a ragged row reaches the taps whose
    products contain it and no others (dx = -1 never reads that column)."""
    b, d, h, w, c = 1, 3, 5, 13, 16
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn((b, d, h, w, c), generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn((b, d, h, w, c), generator=g, device="cuda").to(torch.bfloat16)
    x[0, 1, 4, 12, 5] = float("inf")
    ws = torch.empty(max(1, ops.workspace_bytes(x.shape, c, c, 27) // 4), device="cuda")
    dw = torch.empty((c, 27, c), device="cuda")
    ops.conv_backward_weight(x, dy, dw, ws, 27)
    ops.check()
    finite = torch.isfinite(dw).all(dim=0).cpu().numpy()  # [tap, ci]
    for t in range(27):
        dyi, dxi = t // 3 % 3 - 1, t % 3 - 1
        hit = dxi >= 0 and dyi >= 0  # the voxel minus the tap's offset lies in the grid (it is in the last row and column)
        assert finite[t, 5] == (not hit) and finite[t, np.arange(c) != 5].all(), t
