"""Batched windows with the path they take stated: strips of 8 rows whose last tile has one row, part
of a tile or all of it (le_step_soa's far end of two-step items reaches into the tile above it), and
block tiles for the small instances that test_batch_tiles_gpu.py solves on them."""
import numpy as np
import pytest

from le2d_b200 import capi
from oracle.oracle import ST_AOS, ST_SOA

from test_batch_tiles_gpu import SIZES, _alone, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f", "d"])
@pytest.mark.parametrize("rows", [8, 9, 16])
def test_short_strips(prec, rows):
    lib, chk = capi.Lib(prec), capi.Lib(prec, checked=True)
    todo = []
    for k, ny in enumerate((3, 7, 8, 9, 12, 17, 18, 64, 65, 201)):
        nx = (150, 113, 57, 225)[k % 4]
        for stype in (ST_SOA, ST_AOS):
            p = _problem(nx, ny, k)
            g0 = np.random.default_rng(ny).uniform(-1, 1, 5 * nx * ny).astype(lib.dtype)
            row = (ny - 1, 0, ny // 2)[k % 3]
            todo.append((p, stype, g0, row, _alone(lib, p, stype, g0, row, 3)))
    for L in (lib, chk):
        for window in (8, 5):
            with capi.Batch(L, 1 << 28) as b:
                assert b.set_strips(7) == capi.LE2D_EINVAL and b.set_strips(rows) == 0
                ids = [b.add(b.problem(p, st, receiver_row=row, receiver_every=3), init=g0)
                       for p, st, g0, row, _ in todo]
                assert b.next_cut(window)["tile_depth"] == 0
                assert b.run(window_steps=window)[0] == 0
                for i, (p, st, _, _, (want, samples)) in zip(ids, todo):
                    assert b.fields(i).tobytes() == want.tobytes(), (p.nx, p.ny, st, window)
                    assert b.receivers(i).tobytes() == samples.tobytes(), (p.nx, p.ny, st, window)
    assert chk.check_violations() == (True, 0)


@pytest.mark.parametrize("prec", ["f", "d"])
def test_small_instances_take_block_tiles(prec):
    """The windows of test_batch_windows_on_tiles_and_strips and of the stalled block tile are on tiles."""
    lib = capi.Lib(prec)
    lib.batch_autotune_reset()
    with capi.Batch(lib, 1 << 28) as b:
        for k, (nx, ny) in enumerate(SIZES):
            b.add(b.problem(_problem(nx, ny, k), ST_SOA if k % 2 else ST_AOS), disks=[(1.0, 1.0, 1.0, 1.0)])
        for window in (7, 10, 256):
            assert b.next_cut(window)["tile_depth"] > 0, window
        assert b.run(7)[0] == 0
        with pytest.raises(RuntimeError):
            b.next_cut(7)  # no steps left


@pytest.mark.parametrize("prec", ["f", "d"])
def test_tuned_class_keeps_block_tiles(prec):
    """A tuned height is one for strips: it does not keep a window of small instances, tuned or not, off
    block tiles."""
    lib = capi.Lib(prec)
    lib.batch_autotune_reset()
    try:
        lib.batch_autotune(100, 70)
        todo = []
        for k, (nx, ny) in enumerate(((100, 70), (90, 120), (200, 150), (65, 128), (128, 65), (40, 30))):
            p = _problem(nx, ny, k)
            g0 = np.random.default_rng(k).uniform(-1, 1, 5 * nx * ny).astype(lib.dtype)
            todo.append((p, g0, _alone(lib, p, ST_AOS, g0, 0, 1000)[0]))
        for strips in (0, 16):
            with capi.Batch(lib, 1 << 28) as b:
                if strips:
                    assert b.set_strips(strips) == 0
                ids = [b.add(b.problem(p), init=g0) for p, g0, _ in todo]
                assert (b.next_cut(64)["tile_depth"] > 0) == (strips == 0)
                assert b.run(64)[0] == 0
                for i, (p, _, want) in zip(ids, todo):
                    assert b.fields(i).tobytes() == want.tobytes(), (p.nx, p.ny, strips)
    finally:
        lib.batch_autotune_reset()
