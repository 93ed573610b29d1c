"""The weight gradient's bounded stage waits made to run out (a poll budget of 0): its
blocks leave the loop at their first tile instead of running to its end, write nothing
to the workspace and raise the flag that wt_net_check reports.  The next launch with the
normal budget is right."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


# one dx a block and one MMA a K step; one MMA per dy; three dx a block; pointwise; gathered voxels
@pytest.mark.parametrize("case", [
    (1, 6, 6, 8, 16, 32, 27), (8, 24, 24, 64, 128, 128, 27), (16, 24, 24, 64, 32, 16, 27), (4, 24, 24, 64, 128, 64, 1),
    (65536, 1, 1, 1, 16, 16, 27),
])
def test_expired_stage_wait(wt_lib, case):
    from windtunnel import WindTunnelError
    from windtunnel.net import Ops
    ops = Ops()
    b, d, h, w, cin, cout, taps = case
    g = torch.Generator(device="cuda").manual_seed(cin)
    x = torch.randn((b, d, h, w, cin), generator=g, device="cuda").to(torch.bfloat16)
    dy = torch.randn((b, d, h, w, cout), generator=g, device="cuda").to(torch.bfloat16)
    ws = torch.empty(ops.workspace_bytes(x.shape, cin, cout, taps) // 4, device="cuda")
    dw = torch.empty((cout, taps, cin), device="cuda")

    def timed():
        a, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        ops.conv_backward_weight(x, dy, dw, ws, taps)
        e.record()
        torch.cuda.synchronize()
        return a.elapsed_time(e)

    timed()
    ops.check()
    full = min(timed() for _ in range(3))
    want = dw.clone()
    ws.fill_(7.0)
    prev = ops.lib.wt_net_set_stage_wait_limit(0)
    try:
        expired = timed()
        with pytest.raises(WindTunnelError, match="wait expired"):
            ops.check()
    finally:
        ops.lib.wt_net_set_stage_wait_limit(prev)
    assert bool((ws == 7.0).all())
    if full > 0.3:  # long enough that leaving the loop shows in the time
        assert expired < 0.5 * full, (expired, full)
    timed()
    ops.check()
    assert torch.equal(dw, want)
