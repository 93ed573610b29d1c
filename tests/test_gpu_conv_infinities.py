"""Weight gradients with infinite inputs under positive output gradients: the taps whose
products contain one are infinite and all others finite, also where a tile's last K step
is half empty: rows of one group, rows whose tile has a group past the grid, three dx to
a block, one MMA per dy, and a tile that takes fewer rows."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("case", [
    (1, 3, 3, 8, 16, 16), (5, 3, 3, 5, 128, 128), (1, 3, 7, 24, 16, 16), (1, 5, 5, 20, 24, 8), (1, 3, 3, 44, 16, 72),
    (1, 3, 5, 40, 8, 16), (3, 7, 3, 56, 40, 64),
    (1, 91, 97, 24, 16, 8), (1, 163, 161, 8, 48, 72),                     # three dx
    (1, 31, 97, 24, 128, 64), (1, 31, 101, 23, 88, 8), (1, 97, 97, 8, 96, 40),  # one MMA per dy
    (1, 31, 65, 33, 120, 128),                                            # fewer rows
])
def test_infinities_stay_in_their_taps(wt_lib, case):
    from windtunnel.net import Ops
    ops = Ops()
    b, d, h, w, cin, cout = case
    g = torch.Generator(device="cuda").manual_seed(w)
    x = torch.randn((b, d, h, w, cin), generator=g, device="cuda").to(torch.bfloat16)
    dy = (torch.rand((b, d, h, w, cout), generator=g, device="cuda") + 0.5).to(torch.bfloat16)
    inf = float("inf")
    for ci, sign, at in ((3, 1, (b - 1, d - 1, h - 1, w - 1)), (5, -1, (0, 0, 0, 0)), (7, 1, (b - 1, d - 1, h - 1, w // 2)),
                         (6, -1, (0, d // 2, h - 1, w - 1))):
        x[(*at, ci)] = sign * inf
    ws = torch.empty(ops.workspace_bytes(x.shape, cin, cout, 27) // 4, device="cuda")
    dw = torch.empty((cout, 27, cin), device="cuda")
    ops.conv_backward_weight(x, dy, dw, ws, 27)
    ops.check()
    p = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1))
    for t in range(27):
        s = p[:, t // 9:t // 9 + d, t // 3 % 3:t // 3 % 3 + h, t % 3:t % 3 + w].reshape(-1, cin)
        want = s.sum(0).expand(cout, cin)  # the gradients are positive: an infinity where this sum has one
        assert torch.equal(torch.isposinf(dw[:, t]), torch.isposinf(want)), t
        assert torch.equal(torch.isneginf(dw[:, t]), torch.isneginf(want)), t
        assert not bool(torch.isnan(dw[:, t]).any()), t
