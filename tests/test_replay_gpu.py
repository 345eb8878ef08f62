"""Runs of many steps replay captured CUDA graphs (le2d_api.cu, run_steps)."""
import numpy as np
import pytest

from le2d_b200 import capi
from oracle.oracle import ST_AOS, ST_SOA

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f", "d"])
def test_replayed_steps_equal_single_steps(prec):
    """Runs long enough to replay captured graphs, from either buffer (an odd number of launches
    between replays) and after a changed dt, are bitwise the same steps taken in short calls."""
    lib = capi.Lib(prec)
    nx, ny = 130, 300
    rng = np.random.default_rng(17)
    for stype in (ST_AOS, ST_SOA):
        g0 = rng.uniform(-1, 1, size=5 * nx * ny).astype(lib.dtype)

        def run(calls):
            t = lib.le_init_task(0.2, (1.0, 0.9), lib.le_init_material(2.0, 1.1, 1.3), (nx, ny), stype)
            try:
                assert lib.set_variant(t, 13, 0) == 0
                assert lib.upload(t, g0.copy()) == 0
                for dt, steps in calls:
                    t.dt = dt
                    assert lib.step_n(t, steps) == 0
                out = np.zeros_like(g0)
                assert lib.download(t, out) == 0 and lib.last_error(t) == 0
                return out
            finally:
                lib.le_free_task(t)

        long = [(0.2, 700), (0.2, 65), (0.2, 131), (0.1, 640)]
        short = []
        for dt, steps in long:
            short += [(dt, 20)] * (steps // 20) + [(dt, steps % 20)]
        assert run(long).tobytes() == run(short).tobytes(), stype


@pytest.mark.parametrize("prec,variant", [("f", 13), ("f", 2), ("d", 15), ("d", 13)])
def test_call_loops_in_halves(prec, variant):
    """Loops of le_step / le_step_soa calls leave their sequence of launches in halves open between
    calls; anything else that uses the state joins it first.  Bitwise the same steps in one call."""
    lib = capi.Lib(prec)
    nx, ny = 140, 290
    for stype in (ST_AOS, ST_SOA):
        g0 = np.random.default_rng(3).uniform(-1, 1, size=5 * nx * ny).astype(lib.dtype)
        step = lib.le_step if stype == ST_AOS else lib.le_step_soa

        def run(calls):
            t = lib.le_init_task(0.2, (1.0, 0.9), lib.le_init_material(2.0, 1.1, 1.3), (nx, ny), stype)
            seen = []
            try:
                assert lib.set_variant(t, variant, 0) == 0 and lib.launch_parts(t) == 3
                assert lib.upload(t, g0) == 0
                for n in (5, 1, 4):
                    if calls:
                        for _ in range(n):
                            step(t)
                    else:
                        assert lib.step_n(t, n) == 0
                    lib.le_set_ball(t, (70.0, 140.0 + n), 9.0, 0.25)
                    out = np.zeros_like(g0)
                    assert lib.download(t, out) == 0
                    seen.append(out.tobytes())
                for _ in range(3):
                    step(t)
                t.dt = 0.15  # other constants: no shared launch
                for _ in range(3):
                    step(t)
                assert lib.step_n(t, 6) == 0
                step(t)
                assert lib.wait(t) == 0
                out = np.zeros_like(g0)
                assert lib.download(t, out) == 0 and lib.last_error(t) == 0
                seen.append(out.tobytes())
                step(t)
                return seen
            finally:
                lib.le_free_task(t)  # with a call queued or held back

        assert run(True) == run(False), stype
