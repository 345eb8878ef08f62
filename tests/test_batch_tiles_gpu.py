"""Batched windows on block tiles (batch.cu, batch_tile_kernel) and on strips: the same instances,
small enough for the first, and again with their size classes in the batched autotuner's table,
which keeps them on strips.  Sizes at the tiles' edges, both layouts, receiver lines sampled
inside an item, odd windows; fields and samples bitwise those of the instances solved alone."""
import numpy as np
import pytest

from le2d_b200 import capi, workloads
from oracle.oracle import ST_AOS, ST_SOA

pytestmark = pytest.mark.gpu

SIZES = ((3, 3), (40, 24), (41, 25), (52, 36), (53, 37), (57, 13), (64, 48), (105, 73), (130, 5), (9, 101))


def _problem(nx, ny, k):
    return workloads.Problem(nx, ny, 1.0, 0.9, 2.0, 1.1, 1.3, 0.2, 17 + k, [])


def _alone(lib, p, stype, g0, row, every):
    t = lib.le_init_task(p.dt, (p.hx, p.hy), lib.le_init_material(p.c1, p.c2, p.rho), (p.nx, p.ny), stype)
    samples = []
    try:
        assert lib.set_variant(t, 2, 0) == 0
        assert lib.upload(t, g0) == 0
        out = np.zeros_like(g0)
        for s in range(p.steps):
            assert lib.step_n(t, 1) == 0
            if (s + 1) % every == 0:
                assert lib.download(t, out) == 0
                f = out.reshape(p.ny, p.nx, 5) if stype == ST_AOS else np.moveaxis(out.reshape(5, p.ny, p.nx), 0, -1)
                samples.append(np.stack([f[row, :, 0], f[row, :, 1]]))
        assert lib.download(t, out) == 0
        return out, np.array(samples)
    finally:
        lib.le_free_task(t)


@pytest.mark.parametrize("prec", ["f", "d"])
def test_batch_windows_on_tiles_and_strips(prec):
    lib, chk = capi.Lib(prec), capi.Lib(prec, checked=True)
    lib.batch_autotune_reset()
    rng = np.random.default_rng(12)
    todo = []
    for k, (nx, ny) in enumerate(SIZES):
        stype, p = (ST_SOA if k % 2 else ST_AOS), _problem(nx, ny, k)
        g0 = rng.uniform(-1, 1, 5 * nx * ny).astype(lib.dtype)
        row = (0, ny - 1, ny // 2)[k % 3]
        todo.append((p, stype, g0, row, _alone(lib, p, stype, g0, row, 4)))

    def run(L, window):
        with capi.Batch(L, 1 << 28) as b:
            ids = [b.add(b.problem(p, st, receiver_row=row, receiver_every=4), init=g0) for p, st, g0, row, _ in todo]
            assert b.run(window_steps=window)[0] == 0
            for i, (p, st, _, _, (want, samples)) in zip(ids, todo):
                assert b.fields(i).tobytes() == want.tobytes(), (p.nx, p.ny, st, window)
                assert b.receivers(i).tobytes() == samples.tobytes(), (p.nx, p.ny, st, window)

    for window in (7, 10, 256):
        run(lib, window)
    run(chk, 7)
    assert chk.check_violations() == (True, 0)
    try:
        for nx, ny in SIZES:
            lib.batch_autotune(nx, ny)  # instances of a tuned class keep its strips
        run(lib, 7)
    finally:
        lib.batch_autotune_reset()


@pytest.mark.parametrize("prec", ["f", "d"])
def test_block_tile_wait_gives_up(prec, monkeypatch):
    """A block tile that never publishes its first item (test hook): the waits that depend on it run
    out, its instance fails alone and the others' results hold."""
    lib = capi.Lib(prec)
    victim = workloads.Problem(200, 150, 1.0, 0.9, 2.0, 1.1, 1.3, 0.2, 40, [(100.0, 70.0, 30.0, 1.0)])
    other = workloads.Problem(90, 60, 1.0, 0.9, 2.0, 1.1, 1.3, 0.2, 11, [])
    g0 = np.random.default_rng(4).uniform(-1, 1, 5 * 90 * 60).astype(lib.dtype)
    monkeypatch.setenv("LE2D_TEST_STALL_BLOCK", "0")  # tile 0: the instance of most items
    with capi.Batch(lib, 1 << 28) as b:
        assert b.set_wait_limit(50_000_000) == 0  # 50 ms
        iv = b.add(b.problem(victim), disks=victim.disks)
        io = b.add(b.problem(other), init=g0)
        assert b.run(window_steps=64)[0] == capi.LE2D_ETIMEOUT
        out = np.zeros(5 * 200 * 150, lib.dtype)
        assert lib.lib.le2d_batch_fields(b.h, iv, out.ctypes.data) == capi.LE2D_ETIMEOUT
        assert b.fields(io).tobytes() == _alone(lib, other, ST_AOS, g0, 0, 100)[0].tobytes()
    monkeypatch.delenv("LE2D_TEST_STALL_BLOCK")
    with capi.Batch(lib, 1 << 28) as b:  # a normal run afterwards
        io = b.add(b.problem(other), init=g0)
        assert b.run()[0] == 0
        assert b.fields(io).tobytes() == _alone(lib, other, ST_AOS, g0, 0, 100)[0].tobytes()
