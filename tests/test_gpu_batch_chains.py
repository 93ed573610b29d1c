"""Batches whose lattices step as chains side by side: every lattice bit for bit as a
single lattice of its own (populations, temperatures, per-step forces, mass), with
one, several and the most chains, uneven sizes, direct, captured and replayed calls,
calls across the reduction's 64 steps and calls too long to capture, and a
re-voxelization in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths,storage,calls", [
    ((256, 232), "f32", (2, 70, 70, 70)),               # two chains
    ((128, 144, 176, 104, 160), "f16", (64, 64, 64)),   # several
    ((100,) * 9 + (64,), "bf16", (4, 1000, 6, 6, 6)),   # eight chains of lattices; 10 x 1000 steps run directly
    ((512, 40), "f16", (2, 2)),                          # one large lattice and one small
])
def test_chains_match_single_lattices(wt_lib, widths, storage, calls):
    import windtunnel as wt
    sim = wt.make_sim(u_in=0.08, tau0=0.55, smag=0.1, storage=storage)
    grids = [((nx, max(24, nx * 3 // 8), max(20, nx * 5 // 16)), (wt.ORIGIN_X, 0.0, 0.0), 11.52 / nx) for nx in widths]
    cells = [int(np.prod(g[0])) for g in grids]
    assert np.mean(cells) >= 65536
    b = wt.AeroBatch(grids, sim)
    singles = [wt.AeroEngine(dims=d, origin=o, h=h, sim=sim) for d, o, h in grids]
    try:
        for k, (x, y) in enumerate(zip(b.lattices, singles)):
            for e in (x, y):
                e.set_shape_raw(wt.config_f1_shape(k))
        for i, n in enumerate(calls):
            heat = 2 * (i % 2)
            b.step(n, heat)
            for k, (x, y) in enumerate(zip(b.lattices, singles)):
                y.step(n, heat)
                assert np.array_equal(x.force_history(n), y.force_history(n)), (i, k)
            if i == 1:
                for e in (b.lattices[1], singles[1]):
                    e.set_shape_raw(wt.config_f1_shape(99))
        for x, y in zip(b.lattices, singles):
            assert np.array_equal(x.read_populations(), y.read_populations())
            dx, dy = x.debug_read(), y.debug_read()
            assert np.array_equal(dx["fields"], dy["fields"]) and np.array_equal(dx["temps"], dy["temps"])
            fx, fy = x.read_forces_raw(), y.read_forces_raw()
            assert list(fx.raw) == list(fy.raw) and fx.mass == fy.mass and fx.steps == fy.steps
    finally:
        for e in singles:
            e.close()
        b.close()
