"""A replayed graph of warp-pair launches whose wait gave up is reported like launches queued one by
one (le2d_api.cu, run_steps, check_pairs)."""
import numpy as np
import pytest

from le2d_b200 import capi
from oracle.oracle import ST_AOS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["f", "d"])
def test_replayed_pair_timeout_is_reported(prec, monkeypatch):
    """A producer warp that hands nothing over (test hook) in every launch of a run: 512 steps queued
    one by one, 64 captured and replayed, and 64 that only replay, each after a synchronisation."""
    lib = capi.Lib(prec)
    monkeypatch.setenv("LE2D_TEST_STALL_PAIR", "0")
    t = lib.le_init_task(0.2, (1.0, 0.9), lib.le_init_material(2.0, 1.1, 1.3), (120, 60), ST_AOS)
    try:
        assert lib.set_variant(t, 9, 0) == 0 and lib.get_plan(t)["warps_per_task"] == 2
        assert lib.upload(t, np.zeros(5 * 120 * 60, lib.dtype)) == 0
        for steps in (512, 64, 64):
            assert lib.step_n(t, steps) == 0
            assert lib.wait(t) == capi.LE2D_ETIMEOUT, steps
            assert lib.wait(t) == 0  # reported once
    finally:
        lib.le_free_task(t)
