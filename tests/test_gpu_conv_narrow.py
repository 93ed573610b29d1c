"""Convolutions of grids whose rows fill little of a tile of numbered rows, which are
gathered voxel by voxel: forward, data and weight gradient against 64-bit sums.

Tolerances as FP32 accumulation of BF16 products gives them (at most 4096 terms): 1e-4
of the output's scale, plus BF16 rounding (2^-8) for the forward pass."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ops(wt_lib):
    from windtunnel.net import Ops
    return Ops()


def conv(x, w):
    """[b, d, h, w, ci] by [co, 27, ci], zero padding."""
    _, d, h, ww, _ = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    return sum(p[:, t // 9:t // 9 + d, t // 3 % 3:t // 3 % 3 + h, t % 3:t % 3 + ww] @ w[:, t].T for t in range(27))


# voxels not a multiple of 128 or of 64 among them, channels that are no power of two, splits without voxels
@pytest.mark.parametrize("case", [
    (65537, 1, 1, 1, 8, 8), (21001, 1, 1, 3, 24, 40), (9001, 2, 2, 2, 16, 128), (4999, 4, 4, 1, 128, 8),
    (30011, 1, 2, 1, 72, 104), (263000, 1, 1, 1, 8, 24),
])
def test_narrow_grids(ops, case):
    b, d, h, w, cin, cout = case
    g = torch.Generator(device="cuda").manual_seed(b)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    x, dy = r(b, d, h, w, cin).to(torch.bfloat16), r(b, d, h, w, cout).to(torch.bfloat16)
    wt = (r(cout, 27, cin) / (27 * cin) ** 0.5).to(torch.bfloat16)
    bias = r(cout) * 0.1
    y = torch.full((b, d, h, w, cout), 7.0, dtype=torch.bfloat16, device="cuda")
    dx = torch.full((b, d, h, w, cin), 7.0, device="cuda")
    dw = torch.full((cout, 27, cin), 7.0, device="cuda")
    ws = torch.empty(ops.workspace_bytes(x.shape, cin, cout, 27) // 4, device="cuda")
    ops.conv_forward(x, wt, bias, y, True)
    ops.conv_backward_data(dy, wt.permute(2, 1, 0).contiguous(), dx, cin, cout, 27)
    ops.conv_backward_weight(x, dy, dw, ws, 27)
    ops.check()
    want = torch.relu(conv(x.double(), wt.double()) + bias.double())
    assert bool(((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-4 * want.abs().max()).all())
    want = conv(dy.double(), wt.double().flip(1).permute(2, 1, 0))
    assert float((dx - want).abs().max()) <= 1e-4 * float(want.abs().max())
    p = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1))
    dyf = dy.double().reshape(-1, cout).T
    want = torch.stack([dyf @ p[:, t // 9:t // 9 + d, t // 3 % 3:t // 3 % 3 + h, t % 3:t % 3 + w].reshape(-1, cin)
                        for t in range(27)], 1)
    assert float((dw - want).abs().max()) <= 1e-4 * float(want.abs().max())


def test_more_numbered_rows_than_31_bits(ops):
    """2^29 + 5 grids of one voxel (four numbered rows each).  Small whole numbers, so that every sum is exact."""
    n = 2 ** 29 + 5
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.empty((n, 1, 1, 1, 8), dtype=torch.bfloat16, device="cuda").random_(0, 2, generator=g)
    wt = torch.empty((8, 27, 8), dtype=torch.bfloat16, device="cuda").random_(0, 3, generator=g)
    y = torch.empty((n, 1, 1, 1, 8), dtype=torch.bfloat16, device="cuda")
    ops.conv_forward(x, wt, None, y, False)
    ops.check()
    flat_x, flat_y = x.view(n, 8), y.view(n, 8)
    for k in range(0, n, 2 ** 24):
        assert torch.equal(flat_y[k:k + 2 ** 24].float(), flat_x[k:k + 2 ** 24].float() @ wt[:, 13].float().T)
    y.random_(0, 2, generator=g)  # now the output's gradient
    dw = torch.empty((8, 27, 8), device="cuda")
    ws = torch.empty(ops.workspace_bytes(x.shape, 8, 8, 27) // 4, device="cuda")
    ops.conv_backward_weight(x, y, dw, ws, 27)
    ops.check()
    want = torch.zeros((8, 27, 8), dtype=torch.float64, device="cuda")
    for k in range(0, n, 2 ** 24):
        want[:, 13] += (flat_y[k:k + 2 ** 24].float().T @ flat_x[k:k + 2 ** 24].float()).double()
    assert torch.equal(dw, want.float())
