"""Results of a server in the pool's pieces (result_pool.h): bursts on one server, so that the first
results are malloc'd and later ones page-locked; sizes under, at and over a piece, receivers,
zero steps, results kept while later bursts run and read from several threads."""
import threading

import numpy as np
import pytest

from le2d_b200 import capi, workloads
from oracle.oracle import ST_AOS, ST_SOA

pytestmark = pytest.mark.gpu

# 5 x 160 x 163 floats are just under a piece of 512 KiB, 5 x 256 x 512 doubles ten of them
SIZES = ((9, 7, 3), (160, 163, 5), (164, 160, 0), (256, 512, 4), (301, 177, 6), (700, 401, 2))


def _alone(lib, nx, ny, steps, stype, g0):
    t = lib.le_init_task(0.2, (1.0, 0.9), lib.le_init_material(2.0, 1.1, 1.3), (nx, ny), stype)
    try:
        out = np.zeros_like(g0)
        assert lib.upload(t, g0) == 0 and lib.step_n(t, steps) == 0 and lib.download(t, out) == 0
        return out
    finally:
        lib.le_free_task(t)


@pytest.mark.parametrize("prec", ["f", "d"])
def test_bursts_of_results(prec):
    lib = capi.Lib(prec)
    todo = []
    for k, (nx, ny, steps) in enumerate(SIZES):
        stype = ST_SOA if k % 2 else ST_AOS
        g0 = np.random.default_rng(k).uniform(-1, 1, 5 * nx * ny).astype(lib.dtype)
        p = workloads.Problem(nx, ny, 1.0, 0.9, 2.0, 1.1, 1.3, 0.2, steps, [])
        todo.append((p, stype, g0, _alone(lib, nx, ny, steps, stype, g0)))
    with capi.Server(lib, 1 << 28, window_steps=3) as srv:
        kept, bad = [], []

        def submit(p, stype, g0, want=capi.LE2D_WANT_FIELDS):
            prob = lib.le2d_problem(p.nx, p.ny, p.hx, p.hy, p.dt, p.c1, p.c2, p.rho, p.steps, stype,
                                    p.ny // 2 if want == capi.LE2D_WANT_RECEIVERS else -1, 1)
            return srv.submit(prob, init=g0, want=want)

        for burst in range(5):
            tickets = [(submit(p, st, g0), want) for p, st, g0, want in todo]
            lines = [(submit(p, st, g0, capi.LE2D_WANT_RECEIVERS), p, st, want) for p, st, g0, want in todo[:2]]

            def read(part):
                for t, want in part:
                    if srv.wait(t, 60.0) != 0 or srv.result(t).tobytes() != want.tobytes():
                        bad.append(t)

            threads = [threading.Thread(target=read, args=(tickets[k::3],)) for k in range(3)]
            for x in threads:
                x.start()
            for x in threads:
                x.join()
            assert not bad, (burst, bad)
            for t, p, st, want in lines:
                assert srv.wait(t, 60.0) == 0
                s = srv.result(t)
                f = want.reshape(p.ny, p.nx, 5) if st == ST_AOS else np.moveaxis(want.reshape(5, p.ny, p.nx), 0, -1)
                assert s[-1].tobytes() == np.stack([f[p.ny // 2, :, 0], f[p.ny // 2, :, 1]]).tobytes()
                assert srv.release(t) == 0
            for k, (t, want) in enumerate(tickets):
                if k == burst:
                    kept.append((t, want))  # read again after the bursts that follow
                else:
                    assert srv.release(t) == 0
        for t, want in kept:
            assert srv.result(t).tobytes() == want.tobytes()
