"""Block tiles at the grid's ends with values near the type's range (tile.cuh,
sweep_x_lane_packed<V, true>): the face of an edge column and its clamped copy has no difference,
however large the column's values are, as on the strip march."""
import numpy as np
import pytest

from le2d_b200 import capi
from oracle.oracle import ST_AOS, ST_SOA

pytestmark = pytest.mark.gpu


def _run(lib, nx, ny, stype, g0, variant):
    # rho c1 = 2e-3: a stress of 1e36 is 5e38 as a velocity, past the range of FP32
    t = lib.le_init_task(0.2, (1.0, 0.9), lib.le_init_material(2.0, 1.0, 1e-3), (nx, ny), stype)
    try:
        if variant is not None:
            assert lib.set_variant(t, variant, 0) == 0
        depth = lib.block_tiles(t)["depth"]
        assert (depth > 0) == (variant is None)
        assert lib.upload(t, g0) == 0 and lib.step_n(t, 9) == 0
        out = np.zeros_like(g0)
        assert lib.download(t, out) == 0 and lib.last_error(t) == 0
        return out
    finally:
        lib.le_free_task(t)


@pytest.mark.parametrize("prec", ["f", "d"])
@pytest.mark.parametrize("nx,ny", [(3, 3), (61, 5), (64, 41), (100, 67), (131, 130)])
def test_uniform_stress_beyond_the_range_of_its_velocity(prec, nx, ny):
    lib = capi.Lib(prec)
    # FP64 forms the invariants themselves, as the reference does: they have to be finite there
    big = 1e36 if prec == "f" else 1e300
    for stype in (ST_AOS, ST_SOA):
        f = np.zeros((ny, nx, 5), lib.dtype)
        f[..., 2] = f[..., 4] = big  # a hydrostatic state: nothing moves
        f[..., 0] = np.random.default_rng(nx).uniform(-1, 1, size=(ny, 1))  # vx by row: only the y-sweep works
        g0 = np.ascontiguousarray(f if stype == ST_AOS else np.moveaxis(f, -1, 0)).reshape(-1)
        want = _run(lib, nx, ny, stype, g0, 2)
        assert np.all(np.isfinite(want))
        assert _run(lib, nx, ny, stype, g0, None).tobytes() == want.tobytes(), (nx, ny, stype)
