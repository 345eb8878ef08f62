"""Two steps per launch on le_step_soa's far end (march_pair.cuh): the rows the second step reads
past the last one are the first step's rows ny-5 and ny-4, marched again by the last tile of a
strip.  Grids and segments that put the end everywhere a tile can meet it, whole launches, launches
in halves and batched instances: bitwise single steps, and no access refused in the
bounds-checked build."""
import numpy as np
import pytest

from le2d_b200 import capi, workloads
from oracle.oracle import ST_SOA

pytestmark = pytest.mark.gpu

PAIR_VARIANTS = (9, 10, 11, 12, 13)


def _run(lib, nx, ny, g0, steps, variant, seg, calls=False):
    t = lib.le_init_task(0.2, (1.0, 0.9), lib.le_init_material(2.0, 1.1, 1.3), (nx, ny), ST_SOA)
    try:
        assert lib.set_variant(t, variant, seg) == 0
        assert lib.upload(t, g0) == 0
        if calls:
            for _ in range(steps):
                lib.le_step_soa(t)
        else:
            assert lib.step_n(t, steps) == 0
        out = np.zeros_like(g0)
        assert lib.download(t, out) == 0 and lib.last_error(t) == 0
        return out.tobytes()
    finally:
        lib.le_free_task(t)


@pytest.mark.parametrize("prec", ["f", "d"])
@pytest.mark.parametrize("nx,ny", [(3, 3), (5, 4), (9, 5), (57, 6), (111, 7), (113, 9), (225, 17), (130, 33)])
def test_soa_two_steps_edges(prec, nx, ny):
    lib, chk = capi.Lib(prec), capi.Lib(prec, checked=True)
    g0 = np.random.default_rng(nx * 100 + ny).uniform(-1, 1, 5 * nx * ny).astype(lib.dtype)
    want = _run(lib, nx, ny, g0, 7, 2, 0)
    for var in PAIR_VARIANTS:
        for seg in (0, 1, 2, 3, 5, 8):
            assert _run(lib, nx, ny, g0, 7, var, seg) == want, (var, seg)
    for seg in (1, 3, 8):
        assert _run(chk, nx, ny, g0, 7, 13, seg) == want, seg
    assert chk.check_violations() == (True, 0)


@pytest.mark.parametrize("prec", ["f", "d"])
def test_soa_two_steps_halves_and_batch(prec):
    lib = capi.Lib(prec)
    for nx, ny, steps in ((130, 300, 31), (513, 257, 12)):
        g0 = np.random.default_rng(ny).uniform(-1, 1, 5 * nx * ny).astype(lib.dtype)
        want = _run(lib, nx, ny, g0, steps, 13, 0, calls=True)  # whole launches
        assert _run(lib, nx, ny, g0, steps, 13, 0) == want      # halves
        assert _run(lib, nx, ny, g0, steps, 2, 0) == want       # single steps
    for ny in (8, 9, 17, 64, 201):  # the last tile of one row, of a whole height, of part of one
        p = workloads.Problem(150, ny, 1.0, 0.9, 2.0, 1.1, 1.3, 0.2, 21, [])
        g0 = np.random.default_rng(ny).uniform(-1, 1, 5 * 150 * ny).astype(lib.dtype)
        with capi.Batch(lib, 1 << 26) as b:
            i = b.add(b.problem(p, ST_SOA), init=g0)
            assert b.run(window_steps=8)[0] == 0
            assert b.fields(i).tobytes() == _run(lib, 150, ny, g0, 21, 2, 0), ny
