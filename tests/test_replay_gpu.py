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
