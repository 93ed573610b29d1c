"""The slots of force-carrying blocks and the cell counts formed on the device:
counts against the flags given, the number of blocks with a force link against the
link masks, over empty, tiny, ragged and larger lattices and more blocks than the
scan has threads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [  # dims, fraction of random solid cells
    ((8, 3, 3), 0.0), ((8, 3, 3), 0.3), ((33, 5, 4), 0.1), ((130, 17, 9), 0.02), ((64, 64, 33), 0.001), ((40, 70, 61), 0.5),
]


@pytest.mark.parametrize("dims,frac", CASES)
def test_counts_and_slots(wt_lib, dims, frac):
    import windtunnel as wt
    rng = np.random.default_rng(int(frac * 1000) + dims[0])
    nx, ny, nz = dims
    n = nx * ny * nz
    solid = np.where(rng.random(n) < frac, rng.integers(1, 4, n), 0).astype(np.uint32)
    emit = np.where((solid == 0) & (rng.random(n) < 0.05), -1.0, 0.0).astype(np.float32)  # some duct cells: no force
    with wt.AeroEngine(dims=dims, origin=(0.0, 0.0, 0.0), h=0.05, sim=wt.make_sim(tau0=0.6)) as e:
        e.set_solid(solid, emit)
        info = e.info()
        assert info.fluid_cells == int((solid == 0).sum())
        assert list(info.solid_cells) == [int((solid == k).sum()) for k in (1, 2, 3)]
        d = e.debug_read(links=True)
        links = (d["links"] & 0x7FFFE).reshape(nz, ny, nx)
        # a link to the mirror image (z = 0, c_z > 0) carries no force; the others do, outside ducts
        up = sum(1 << i for i in (5, 11, 14, 15, 18))
        force = links != 0
        force[0] = (links[0] & ~np.uint32(up)) != 0
        force &= ~((emit < 0) & (solid == 0)).reshape(nz, ny, nx)
        f = np.zeros((nz, ny, -(-nx // 128) * 128), bool)
        f[..., :nx] = force
        assert info.boundary_blocks == int(f.reshape(nz, ny, -1, 128).any(-1).sum())
        e.step(16)
        a = e.force_history(16)
        assert frac == 0.0 or np.abs(a).sum() > 0


def test_blocks_beyond_one_scan_run(wt_lib):
    """18,960 blocks for the scan's 1024 threads: the FP64 sums over the blocks' records agree with the i32
    sums of the same per-cell forces, each rounded to 1e-4 (half a unit per cell and step)."""
    import windtunnel as wt
    dims = (256, 79, 120)
    with wt.AeroEngine(dims=dims, origin=(wt.ORIGIN_X, 0.0, 0.0), h=0.045) as e:
        e.set_shape_raw(wt.config_f1_shape(1))
        e.step(32)
        f = e.read_forces_raw()
        solid = e.debug_read()["solid"]
        info = e.info()
        assert info.fluid_cells == int((solid == 0).sum()) and 0 < info.boundary_blocks < 18960
        whole = np.array(f.sum[:])
        raw = np.array([f.raw[i] for i in (0, 1, 3, 4, 6, 7)])
    assert np.abs(whole[[0, 1, 3, 4, 6, 7]] * 1e4 - raw).max() <= 0.5 * 32 * info.boundary_blocks * 128
