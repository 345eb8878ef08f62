"""Block tiles (tile.cuh, step_tile.cu): small grids on their default plan run several steps per
launch on tiles held in registers.  Results must be bitwise those of the strip march (an
explicit variant), for both layouts, at the tiles' edges: grids smaller than a tile, one node
over and under a whole number of tiles, step counts that do not fill the last launch.  The
bounds-checked build must refuse no access."""
import numpy as np
import pytest

from le2d_b200 import capi
from oracle.oracle import ST_AOS, ST_SOA

pytestmark = pytest.mark.gpu

# Chosen so that every tile shape is planned for some grid (asserted below).
SIZES = ((3, 3), (4, 7), (5, 300), (61, 5), (52, 9), (53, 8), (100, 67), (255, 257), (300, 256), (501, 333), (511, 513), (640, 480), (1001, 640))


def _run(lib, nx, ny, stype, g0, steps, variant=None, calls=False):
    mat = lib.le_init_material(2.0, 1.1, 1.3)
    t = lib.le_init_task(0.2, (1.0, 0.9), mat, (nx, ny), stype)
    try:
        if variant is not None:
            assert lib.set_variant(t, variant, 0) == 0
        tiles = lib.block_tiles(t)
        assert lib.upload(t, g0) == 0
        if calls:
            for _ in range(steps):
                (lib.le_step if stype == ST_AOS else lib.le_step_soa)(t)
        else:
            assert lib.step_n(t, steps) == 0
        out = np.zeros_like(g0)
        assert lib.download(t, out) == 0 and lib.last_error(t) == 0
        assert lib.sim_time(t)[2] == steps
        return out, tiles
    finally:
        lib.le_free_task(t)


@pytest.mark.parametrize("prec", ["f", "d"])
def test_block_tiles_equal_strips(prec):
    lib, chk = capi.Lib(prec), capi.Lib(prec, checked=True)
    rng = np.random.default_rng(31)
    shapes = set()
    for nx, ny in SIZES:
        # a zero background with steps and noise in it, as solves have
        g0 = (rng.standard_normal(5 * nx * ny) * rng.choice([0.0, 0.0, 1e-3, 1.0], 5 * nx * ny)).astype(lib.dtype)
        for stype in (ST_AOS, ST_SOA):
            for steps in (1, 13):
                want, none = _run(lib, nx, ny, stype, g0, steps, variant=2)
                assert none["depth"] == 0
                got, tiles = _run(lib, nx, ny, stype, g0, steps)
                if tiles["depth"]:
                    shapes.add((tiles["cols"], tiles["rows"]))
                assert got.tobytes() == want.tobytes(), (nx, ny, stype, steps, tiles)
                if steps > 1:
                    assert _run(lib, nx, ny, stype, g0, steps, calls=True)[0].tobytes() == want.tobytes(), (nx, ny, stype)
                    assert _run(chk, nx, ny, stype, g0, steps)[0].tobytes() == want.tobytes(), (nx, ny, stype)
        assert chk.check_violations() == (True, 0), (nx, ny)
    assert len(shapes) >= (4 if prec == "f" else 3), shapes
