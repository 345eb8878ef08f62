"""Strip launches whole (LE2D_HALVES=0) against the same launches in halves (LE2D_HALVES=1): grids small
enough for block tiles and taller ones, both layouts, one call and loops of calls.  Either setting
means the strip plan, and the launches are checked to be what is compared."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r"""
import hashlib, json, sys
import numpy as np
from le2d_b200 import capi
parts, out = int(sys.argv[1]), {}
for prec in ("f", "d"):
    lib = capi.Lib(prec)
    for nx, ny, steps in ((64, 37, 5), (130, 300, 31), (513, 257, 12), (97, 1000, 7), (300, 16, 9)):
        for stype in (capi.ST_AOS, capi.ST_SOA):
            g = np.random.default_rng(nx * 7 + ny).uniform(-1, 1, 5 * nx * ny).astype(lib.dtype)
            for calls in (False, True):
                t = lib.le_init_task(0.2, (1.0, 0.9), lib.le_init_material(2.1, 1.1, 1.3), (nx, ny), stype)
                try:
                    assert lib.block_tiles(t)["depth"] == 0 and lib.launch_parts(t) == parts
                    assert (lib.get_plan(t)["depth"] == 2) == (prec == "f")
                    assert lib.upload(t, g) == 0
                    if calls:
                        for _ in range(steps):
                            (lib.le_step if stype == capi.ST_AOS else lib.le_step_soa)(t)
                    else:
                        assert lib.step_n(t, steps) == 0
                    got = np.zeros_like(g)
                    assert lib.download(t, got) == 0 and lib.last_error(t) == 0
                    assert got.tobytes() != g.tobytes()
                finally:
                    lib.le_free_task(t)
                out[f"{prec} {nx}x{ny} {stype} {calls}"] = hashlib.sha256(got.tobytes()).hexdigest()
print(json.dumps(out))
"""


def _run(halves: str, parts: int) -> dict:
    env = dict(os.environ, LE2D_HALVES=halves, PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(parts)], env=env, cwd=ROOT, capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_whole_launches_equal_halves():
    whole, halves = _run("0", 1), _run("1", 3)
    assert whole == halves
    for key, digest in whole.items():  # loops of calls as one call
        assert whole[key.replace("True", "False")] == digest, key
