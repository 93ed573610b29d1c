"""Weight gradients of grids whose rows are walked whole (8 groups of voxels, and one
group with the odd row of a tile left to the next), against the float64 oracle: tiles of
8 and of 4 rows, splits that begin inside a plane, planes with an odd number of rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("case", [
    (1, 3, 5, 64, 8, 16), (2, 24, 24, 64, 16, 16), (2, 13, 11, 64, 64, 32), (3, 7, 5, 64, 32, 16),
    (5, 3, 3, 8, 128, 128), (7, 5, 7, 8, 16, 64), (31, 3, 17, 8, 32, 8),
])
def test_weight_gradient(wt_lib, case):
    """FP32 sums of at most 4608 products per split: 1e-4 of the output's scale."""
    from oracle import conv_ref as ref
    from windtunnel.net import Ops
    ops = Ops()
    b, d, h, w, cin, cout = case
    rng = np.random.default_rng(sum(case))
    x = ref.bf16_round(rng.standard_normal((b, d, h, w, cin)))
    dy = ref.bf16_round(rng.standard_normal((b, d, h, w, cout)))
    xs, ds = (torch.tensor(np.ascontiguousarray(a, np.float32), device="cuda").to(torch.bfloat16) for a in (x, dy))
    ws = torch.empty(ops.workspace_bytes(xs.shape, cin, cout, 27) // 4, device="cuda")
    dw = torch.full((cout, 27, cin), 7.0, device="cuda")
    ops.conv_backward_weight(xs, ds, dw, ws, 27)
    ops.check()
    want = ref.conv3d_backward_weight(x, dy, 27)
    assert np.abs(dw.cpu().numpy() - want).max() <= 1e-4 * np.abs(want).max()
