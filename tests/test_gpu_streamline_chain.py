"""The streamline pass against the same chain of RK2 steps driven point by point
through wt_sample_flow in float32 numpy (both round every operation alike), bit for
bit: line lengths around the pass's chunks of 128 steps, every colour mode, seeds on
both sides of the symmetry plane, inside the body and past the domain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


@pytest.fixture(scope="module")
def flow(wt_lib):
    import windtunnel as wt
    e = wt.AeroEngine(dims=(88, 33, 27), origin=(wt.ORIGIN_X, 0.0, 0.0), h=0.13)
    e.set_shape_raw(wt.config_f1_shape(3))
    e.frame(40)
    yield e
    e.close()


def length(u):
    x, y, z = u[:, 0], u[:, 1], u[:, 2]
    return np.sqrt((x * x + y * y) + z * z)


def chain(e, seeds, steps, view, step_len):
    p = seeds.astype(F)
    alive = np.ones(len(p), bool)
    nx, ny, nz = e.dims
    h = F(e.h)
    hi = [F(F(e.origin[a]) + F(F(n) * h)) for a, n in enumerate((nx, ny, nz))]
    out = np.zeros((len(p), steps, 4), F)
    speed = np.zeros((len(p), steps), F)
    for k in range(steps):
        s1 = e.sample_flow(p)
        l1 = length(s1[:, :3])
        alive &= ~((s1[:, 5] < F(0.3)) | (l1 < F(view.u_in) * F(0.03)))
        out[:, k, :3] = p
        out[:, k, 3] = np.where(alive, 0, -1)
        speed[:, k] = np.minimum(np.maximum(l1 / (F(view.u_in) * F(view.speed_max)), F(0)), F(1))
        with np.errstate(all="ignore"):
            mid = p + ((s1[:, :3] / l1[:, None]) * F(step_len)) * F(0.5)
            s2 = e.sample_flow(np.where(alive[:, None], mid, p))
            d = np.where((s2[:, 5] > F(0.3))[:, None], s2[:, :3], s1[:, :3])
            new = p + (d / length(d)[:, None]) * F(step_len)
        p = np.where(alive[:, None], new, p).astype(F)
        alive &= ~((p[:, 0] > F(hi[0] - h * F(3))) | (p[:, 1] < F(0.01)) | (p[:, 1] > hi[1]) | (np.abs(p[:, 2]) > hi[2]))
    return out, speed


@pytest.mark.parametrize("steps", [1, 127, 128, 129, 300])
def test_lines_follow_the_sampled_flow(flow, steps):
    from windtunnel import _abi
    e = flow
    view = _abi.View()
    view.u_in, view.v_real, view.cp_min, view.cp_max = e.sim.u_in, 69.0, -1.1, 0.7
    view.t_min, view.t_max, view.speed_max, view.vort_max = 0.0, 220.0, 1.5, 0.6
    s = _abi.StreamParams()
    s.rows, s.cols, s.lines, s.per_emitter, s.emitters, s.step_len, s.steps = 9, 5, 45, 1, 1, 0.04, steps
    s.seed_min[:] = (-1.5, 0.03, -0.9)
    s.seed_max[:] = (0.0, 1.6, 0.9)
    rows, cols = np.divmod(np.arange(45), 5)
    fy, fz = (rows.astype(F) + F(0.5)) / F(9), (cols.astype(F) + F(0.5)) / F(5)

    def mix(a, b, t):
        return F(a) * (F(1) - t) + F(b) * t

    for x0 in (-1.5, 0.4, 2.2, 8.8):  # upstream, at the front wing, in the body, near the outlet
        s.seed_min[0] = x0
        seeds = np.stack([np.full(45, x0, F), mix(0.03, 1.6, fy), mix(-0.9, 0.9, fz)], 1).astype(F)
        want, speed = chain(e, seeds, steps, view, 0.04)
        got = {}
        for mode in range(5):
            s.color_mode = mode
            got[mode] = e.streamlines(s, view)
            assert np.array_equal(got[mode][..., :3], want[..., :3]), (x0, mode)
            assert np.array_equal(got[mode][..., 3] == -1, want[..., 3] == -1)
        live = want[..., 3] == 0
        assert np.array_equal(got[0][..., 3][live], speed[live])
        _, vort = e.sample_flow(want[..., :3].reshape(-1, 3), vorticity=True)
        v = np.clip(vort / (F(view.u_in) * F(view.vort_max)), F(0), F(1)).reshape(live.shape)
        assert np.array_equal(got[3][..., 3][live], v[live])
