"""Force readbacks that take their pending steps with them: the sums against the
per-step history, for step counts around the reduction's split over the steps and the
number of steps a reduction covers, with records on one block and on many."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(9, 5, 4), (150, 40, 30)])
def test_readback_equals_history(wt_lib, dims):
    import windtunnel as wt
    rng = np.random.default_rng(dims[0])
    nx, ny, nz = dims
    solid = np.where(rng.random((nz, ny, nx)) < 0.1, rng.integers(1, 4, (nz, ny, nx)), 0).astype(np.uint32)
    solid[:, :, 0] = solid[:, :, -1] = 0
    e = wt.AeroEngine(dims=dims, origin=(0.0, 0.0, 0.0), h=0.05, sim=wt.make_sim(u_in=0.05, tau0=0.7, smag=0.1))
    e.set_solid(solid, np.zeros(solid.shape, np.float32))
    e.step(4, 0, 1.0)
    e.read_forces_raw()
    for n in (2, 8, 14, 16, 18, 62, 64, 66, 130):
        e.step(n, 0, 1.0)
        t = e.read_forces_async(reset=False)
        kept, f = e.collect_forces(t), e.read_forces_raw()
        h = e.force_history(n)
        # 64-bit sums in another order: n + 8 roundings of at most the sum of the magnitudes
        np.testing.assert_allclose(f.sum[:], h.sum(0), rtol=0, atol=(n + 8) * 2.0**-52 * np.abs(h).sum(0).max())
        assert list(kept.sum[:]) == list(f.sum[:]) and list(kept.raw) == list(f.raw) and kept.steps == f.steps == n
        raw = np.array(f.raw[:9], np.float64).reshape(3, 3)[:, :2]
        scaled = h.sum(0).reshape(3, 3)[:, :2] * 10_000
        assert np.all(np.abs(raw - scaled) <= n * np.prod(dims))  # each cell and step rounds once
        again = e.read_forces_raw()
        assert list(again.sum[:]) == [0.0] * 9 and list(again.raw) == [0] * len(again.raw) and again.steps == 0
        assert again.mass == f.mass
    e.close()
