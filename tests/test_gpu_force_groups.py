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


def test_large_forces_take_the_fp64_sums(wt_lib, oracle_mod):
    """Populations of 1.15 along x by a wall give forces above 2 per cell (the exact integer sums hold below
    that) in some warps and small ones in others, in one block."""
    import windtunnel as wt
    dims = (130, 6, 5)
    n = int(np.prod(dims))
    sim = wt.make_sim(u_in=0.02, tau0=0.9, smag=0.0)
    solid = np.zeros((5, 6, 130), np.uint32)
    solid[2, 3, 20], solid[2, 3, 90], solid[1, 2, 50] = 1, 1, 2
    f = np.tile(np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12, np.float32)[:, None], (1, n))
    cell = lambda x, y, z: x + 130 * (y + 6 * z)  # noqa: E731
    # after streaming, cell (19, 3, 2) holds these along +x (from its neighbour) and -x (bounced off (20, 3, 2))
    f[1, cell(18, 3, 2)] = f[1, cell(19, 3, 2)] = 1.15
    f[0, cell(19, 3, 2)] = 0.05
    e = wt.AeroEngine(dims=dims, origin=(0.0, 0.0, 0.0), h=0.05, sim=sim)
    o = oracle_mod.Oracle(dims, (0.0, 0.0, 0.0), 0.05, sim)
    emit = np.zeros(n, np.float32)
    e.set_solid(solid, emit)
    o.set_solid(solid.reshape(-1), emit)
    o.reset()
    e.write_state(f=f)
    o.write_state(f=f)
    e.step(2)
    o.steps(2)
    h, od = e.force_history(2), o.read(reset_forces=True)
    assert np.abs(h).max() > 2.0
    fr = e.read_forces_raw()
    assert list(fr.raw) == od["forces"].tolist() and fr.guarded == o.guarded()
    np.testing.assert_allclose(fr.sum[:], od["forces64"], rtol=1e-9, atol=1e-9)
    e.close()
