"""Force sums of a bf16 lattice near rest, whose populations' deviations have any
exponent: every term counts with all its bits, however small.  The state is put in
through a checkpoint file (the format keeps the populations' own bits); the first step
after a load bounces the stored values, so its forces follow from them.

Tolerance: FP64 sums of at most 2000 terms, 2000 x 2^-53 of the sum of magnitudes."""
import math
import struct

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C = np.array([[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1], [1, 1, 0], [-1, -1, 0],
              [1, -1, 0], [-1, 1, 0], [1, 0, 1], [-1, 0, -1], [1, 0, -1], [-1, 0, 1], [0, 1, 1], [0, -1, -1],
              [0, 1, -1], [0, -1, 1]])


def fnv1a(data):
    h = 1469598103934665603
    for b in data:
        h = ((h ^ b) * 1099511628211) & 0xFFFFFFFFFFFFFFFF
    return h


@pytest.mark.parametrize("low,high", [(-70, -50), (-60, -20), (-120, -90)])
def test_terms_of_any_size(wt_lib, tmp_path, low, high):
    import windtunnel as wt
    from windtunnel import _abi
    import ctypes
    dims = nx, ny, nz = (37, 8, 7)
    n = nx * ny * nz
    rng = np.random.default_rng(-low)
    solid = np.where(rng.random((nz, ny, nx)) < 0.15, rng.integers(1, 4, (nz, ny, nx)), 0).astype(np.uint32)
    solid[:, :, 0] = solid[:, :, -1] = 0
    e = wt.AeroEngine(dims=dims, origin=(0.0, 0.0, 0.0), h=0.05, sim=wt.make_sim(storage="bf16", u_in=0.0, tau0=0.7, smag=0.0))
    e.set_solid(solid, np.zeros(n, np.float32))
    path = str(tmp_path / "state")
    e.save(path)
    data = bytearray(open(path, "rb").read())
    # bf16 bits: any sign and significand, exponents in [low, high)
    bits = (rng.integers(0, 2, (19, n)) << 15 | (rng.integers(low, high, (19, n)) + 127) << 7 | rng.integers(0, 128, (19, n))).astype(np.uint16)
    bits[:, solid.reshape(-1) != 0] = 0
    at = 8 + 7 * 4 + ctypes.sizeof(_abi.Sim) + ctypes.sizeof(_abi.Shape) + 2 * 8
    assert len(data) > at + bits.nbytes
    data[at:at + bits.nbytes] = bits.tobytes()
    data[-8:] = struct.pack("<Q", fnv1a(data[:-8]))
    open(path, "wb").write(data)
    e.load(path)
    links = e.debug_read(links=True)["links"].reshape(nz, ny, nx)
    e.step(2)
    got = e.force_history(2)[0]
    e.close()
    f = (bits.astype(np.uint32) << 16).view(np.float32).reshape(19, nz, ny, nx)
    cell = np.zeros((9, nz, ny, nx), np.float32)
    for i in range(1, 19):
        for z, y, x in np.argwhere((links >> i) & 1):
            cx, cy, cz = (int(v) for v in C[i])
            if z - cz < 0:
                continue  # through the symmetry plane: no force
            g = int(solid[z - cz, y - cy, x - cx]) - 1
            t = np.float32(2) * f[i, z, y, x]
            for a, c in enumerate((cx, cy, cz)):
                if c:
                    k = 3 * g + a
                    cell[k, z, y, x] = cell[k, z, y, x] - t if c > 0 else cell[k, z, y, x] + t
    for k in range(9):
        terms = cell[k].astype(np.float64).ravel().tolist()
        assert abs(got[k] - math.fsum(terms)) <= 2000 * 2.0 ** -53 * math.fsum(map(abs, terms)), k
        assert got[k] != 0.0
