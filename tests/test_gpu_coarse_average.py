"""The coarse box average against 64-bit means of the same fluid cells: one cell to a
box, ragged boxes, boxes above the size that is summed in integers, and a coarse grid
whose last block is not full; boxes without a fluid cell give (0, 0, 0, 1)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,coarse", [
    ((9, 5, 4), (9, 5, 4)), ((61, 23, 17), (8, 5, 3)), ((61, 23, 17), (1, 1, 1)), ((70, 40, 30), (2, 3, 1)),
    ((64, 24, 20), (13, 7, 20)), ((40, 12, 9), (40, 1, 9)),
])
def test_means(wt_lib, dims, coarse):
    import windtunnel as wt
    rng = np.random.default_rng(sum(dims))
    nx, ny, nz = dims
    solid = (rng.random((nz, ny, nx)) < 0.05).astype(np.uint32)
    solid[1:nz // 2 + 1, 0:ny // 2, 1:nx // 2] = 1
    solid[:, :, 0] = solid[:, :, -1] = 0
    e = wt.AeroEngine(dims=dims, origin=(0.0, 0.0, 0.0), h=0.05, sim=wt.make_sim(u_in=0.05, tau0=0.7, smag=0.1))
    e.set_solid(solid, np.zeros(solid.shape, np.float32))
    e.step(20, 0, 1.0)
    f = e.debug_read()["fields"].reshape(nz, ny, nx, 4).astype(np.float64)
    got = e.read_coarse(*coarse)
    e.close()
    cut = [[k * d // c for k in range(c + 1)] for d, c in zip(dims, coarse)]
    for c in range(coarse[2]):
        for b in range(coarse[1]):
            for a in range(coarse[0]):
                box = np.s_[cut[2][c]:cut[2][c + 1], cut[1][b]:cut[1][b + 1], cut[0][a]:cut[0][a + 1]]
                v = f[box][solid[box] == 0]
                if len(v) == 0:
                    assert got[c, b, a].tolist() == [0.0, 0.0, 0.0, 1.0]
                    continue
                ref, top = v.mean(0), np.abs(v).max(0)
                # one rounding to 32 bits, and sums good to 2^-48 of the largest term
                assert np.all(np.abs(got[c, b, a] - ref) <= 2.0**-24 * np.abs(ref) + 2.0**-48 * top + 2.0**-149)
