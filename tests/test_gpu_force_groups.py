"""Forces and boundary rows of lattices with random solid groups and duct cells,
solids on every face but x = 0 and x = nx - 1 included, bit for bit against the
oracle: cells whose links meet one group and cells whose links meet several, links
through the symmetry plane, warps with no, one and three groups, and the boundary
precedence at every edge (the moving floor's corners among them)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,frac,block", [
    ((9, 3, 3), 0.3, None), ((34, 5, 4), 0.15, (32, 2)), ((70, 12, 9), 0.02, (64, 4)), ((131, 7, 6), 0.3, None),
    ((64, 2, 2), 0.1, None),
])
def test_forces_bitexact(wt_lib, oracle_mod, monkeypatch, dims, frac, block):
    import windtunnel as wt
    if block:
        monkeypatch.setenv("WT_STEP_BX", str(block[0]))
        monkeypatch.setenv("WT_STEP_BY", str(block[1]))
    rng = np.random.default_rng(dims[0])
    nx, ny, nz = dims
    solid = np.where(rng.random((nz, ny, nx)) < frac, rng.integers(1, 4, (nz, ny, nx)), 0).astype(np.uint32)
    solid[:, :, 0] = solid[:, :, -1] = 0
    emit = np.where((solid == 0) & (rng.random(solid.shape) < 0.1), -1.0, 0.0).astype(np.float32)
    sim = wt.make_sim(u_in=0.06, tau0=0.7, smag=0.1)
    e = wt.AeroEngine(dims=dims, origin=(0.0, 0.0, 0.0), h=0.05, sim=sim)
    o = oracle_mod.Oracle(dims, (0.0, 0.0, 0.0), 0.05, sim)
    e.set_solid(solid, emit)
    o.set_solid(solid.reshape(-1), emit.reshape(-1))
    o.reset()
    for _ in range(3):
        e.step(4, 2, 2.0)
        o.frame(4)
        f, d, od = e.read_forces_raw(), e.debug_read(links=True), o.read(reset_forces=True)
        assert np.array_equal(d["links"], o.link_mask())
        assert np.array_equal(d["fields"], od["fields"]) and np.array_equal(e.read_populations(), od["f"])
        assert list(f.raw) == od["forces"].tolist()
        np.testing.assert_allclose(f.sum[:], od["forces64"], rtol=1e-9, atol=1e-9)
    e.close()
