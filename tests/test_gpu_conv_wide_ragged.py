"""Weight gradients with 112 to 128 channels on both sides, more splits than fill the
device with one block each and rows that are not walked whole: the tile of 16 rows is
over a block's shared memory there, and takes fewer rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("case", [(2, 32, 32, 33, 128, 128), (3, 24, 24, 40, 128, 112), (1, 97, 97, 7, 128, 120)])
def test_weight_gradient(wt_lib, case):
    """FP32 sums of at most 4224 products per split: 1e-4 of the output's scale."""
    from windtunnel.net import Ops
    ops = Ops()
    b, d, h, w, cin, cout = case
    g = torch.Generator(device="cuda").manual_seed(sum(case))
    x = torch.randn((b, d, h, w, cin), generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn((b, d, h, w, cout), generator=g, device="cuda").to(torch.bfloat16)
    ws = torch.empty(ops.workspace_bytes(x.shape, cin, cout, 27) // 4, device="cuda")
    assert ws.numel() >= 17 * 27 * cin * cout
    dw = torch.full((cout, 27, cin), 7.0, device="cuda")
    ops.conv_backward_weight(x, dy, dw, ws, 27)
    ops.check()
    p = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1))
    dyf = dy.double().reshape(-1, cout).T
    want = torch.stack([dyf @ p[:, t // 9:t // 9 + d, t // 3 % 3:t // 3 % 3 + h, t % 3:t % 3 + w].reshape(-1, cin)
                        for t in range(27)], 1)
    assert float((dw - want).abs().max()) <= 1e-4 * float(want.abs().max())
