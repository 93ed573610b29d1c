"""The coarse box average at the edges of its integer sums, against exact means: boxes of
2048, 4095, 4096 and more cells (the largest that are summed in integers, and the first in
FP64) and of fewer than ten (a thread to each), values over 60 binades of both signs, and infinities and NaN, whose boxes are
summed in FP64 beside boxes of the same warp that are not."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def boxes(dims, coarse):
    cut = [[k * d // c for k in range(c + 1)] for d, c in zip(dims, coarse)]
    for c in range(coarse[2]):
        for b in range(coarse[1]):
            for a in range(coarse[0]):
                yield (c, b, a), np.s_[cut[2][c]:cut[2][c + 1], cut[1][b]:cut[1][b + 1], cut[0][a]:cut[0][a + 1]]


def averages(dims, coarse, fields, solid):
    import windtunnel as wt
    e = wt.AeroEngine(dims=dims, origin=(0.0, 0.0, 0.0), h=0.05, sim=wt.make_sim(u_in=0.05, tau0=0.7, smag=0.1))
    e.set_solid(solid, np.zeros(solid.shape, np.float32))
    e.write_state(fields=fields.reshape(-1, 4))
    got = e.read_coarse(*coarse)
    e.close()
    return got


@pytest.mark.parametrize("dims,coarse", [
    ((32, 8, 8), (1, 1, 1)), ((65, 9, 7), (1, 1, 1)), ((32, 16, 8), (1, 1, 1)), ((683, 3, 2), (1, 1, 1)),
    ((96, 32, 8), (3, 2, 1)), ((40, 12, 9), (10, 4, 3)), ((40, 12, 9), (20, 6, 9)), ((41, 13, 9), (41, 7, 3)),
])
@pytest.mark.parametrize("spread", [0, 60])
def test_means(wt_lib, dims, coarse, spread):
    rng = np.random.default_rng(sum(dims) + spread)
    nx, ny, nz = dims
    v = rng.uniform(0.5, 1.0, (nz, ny, nx, 4)) * 2.0 ** rng.uniform(-spread, 0, (nz, ny, nx, 4)) * rng.choice([-1, 1], (nz, ny, nx, 4))
    v = v.astype(np.float32)
    solid = np.zeros((nz, ny, nx), np.uint32)
    got = averages(dims, coarse, v, solid)
    for at, box in boxes(dims, coarse):
        cells = v[box].reshape(-1, 4).astype(np.float64)
        for k in range(4):
            ref, top = math.fsum(cells[:, k]) / len(cells), np.abs(cells[:, k]).max()
            # one rounding to 32 bits, and sums good to 2^-48 of the largest term (FP64 sums: n 2^-53)
            assert abs(got[at][k] - ref) <= 2.0 ** -24 * abs(ref) + max(2.0 ** -48, len(cells) * 2.0 ** -53) * top


@pytest.mark.parametrize("dims,coarse", [((40, 12, 9), (10, 4, 3)), ((96, 32, 24), (3, 2, 3)), ((40, 12, 9), (10, 12, 9))])
def test_infinities_and_nan(wt_lib, dims, coarse):
    """Eight and 32 lanes to a box, and one; some boxes of every warp hold a special value."""
    rng = np.random.default_rng(3)
    nx, ny, nz = dims
    v = rng.normal(size=(nz, ny, nx, 4)).astype(np.float32)
    solid = np.zeros((nz, ny, nx), np.uint32)
    special = {}
    for n, (at, box) in enumerate(boxes(dims, coarse)):
        k, kind = n % 4, n % 5
        cells = v[box][..., k]  # a view
        if kind == 0:
            cells[0, 0, 0], special[at, k] = np.inf, np.inf
        elif kind == 1:
            cells[-1, -1, -1], special[at, k] = -np.inf, -np.inf
        elif kind == 2:
            cells[0, 0, 0], cells[-1, -1, -1], special[at, k] = np.inf, -np.inf, np.nan
        elif kind == 3:
            cells[0, -1, 0], special[at, k] = np.nan, np.nan
    got = averages(dims, coarse, v, solid)
    for at, box in boxes(dims, coarse):
        cells = v[box].reshape(-1, 4).astype(np.float64)
        for k in range(4):
            if (at, k) in special:
                np.testing.assert_equal(float(got[at][k]), special[at, k])
            else:
                ref, top = math.fsum(cells[:, k]) / len(cells), np.abs(cells[:, k]).max()
                assert abs(got[at][k] - ref) <= 2.0 ** -24 * abs(ref) + max(2.0 ** -48, len(cells) * 2.0 ** -53) * top
