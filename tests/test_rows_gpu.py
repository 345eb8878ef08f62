"""le2d_rows_out / le2d_rows_in (layout.cu, copy_rows_kernel) and the diagnostics kernel (diag.cu) at
the widths and alignments their vector accesses can meet."""
import numpy as np
import pytest

from le2d_b200 import capi
from oracle.oracle import ST_AOS, ST_SOA

pytestmark = pytest.mark.gpu


def _task(lib, nx, ny, stype, g):
    t = lib.le_init_task(0.2, (1.0, 0.9), lib.le_init_material(2.0, 1.1, 1.3), (nx, ny), stype)
    assert lib.upload(t, g) == 0
    return t


@pytest.mark.parametrize("prec", ["f", "d"])
@pytest.mark.parametrize("nx,ny", [(3, 3), (4, 5), (127, 9), (128, 6), (129, 4), (512, 3), (516, 7), (1030, 5)])
def test_rows_out_and_in(prec, nx, ny):
    import torch

    lib = capi.Lib(prec)
    dt = torch.float32 if prec == "f" else torch.float64
    rng = np.random.default_rng(nx)
    g = rng.standard_normal((5, ny, nx)).astype(lib.dtype)
    t = _task(lib, nx, ny, ST_SOA, np.ascontiguousarray(g.reshape(-1)))
    try:
        for row0, rows in ((0, ny), (1, ny - 2), (ny - 1, 1)):
            for shift in (0, 1):  # a buffer 16-byte aligned, and one element past it
                flat = torch.full((5 * rows * nx + 8,), -7.0, dtype=dt, device="cuda")
                at = flat[shift:].data_ptr()
                assert lib.rows_out(t, row0, rows, at, torch.cuda.current_stream().cuda_stream) == 0
                got = flat.cpu().numpy()
                assert np.array_equal(got[shift:shift + 5 * rows * nx].reshape(5, rows, nx), g[:, row0:row0 + rows])
                assert np.all(got[shift + 5 * rows * nx:] == -7.0) and np.all(got[:shift] == -7.0)
                new = rng.standard_normal((5, rows, nx)).astype(lib.dtype)
                flat[shift:shift + new.size] = torch.from_numpy(new.reshape(-1)).cuda()
                assert lib.rows_in(t, row0, rows, at, torch.cuda.current_stream().cuda_stream) == 0
                g[:, row0:row0 + rows] = new
        pinned = torch.zeros(5 * ny * nx, dtype=dt, pin_memory=True)  # not device memory: a copy call
        assert lib.rows_out(t, 0, ny, pinned.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert np.array_equal(pinned.numpy().reshape(5, ny, nx), g)
        out = np.zeros(5 * ny * nx, lib.dtype)
        assert lib.download(t, out) == 0
        assert np.array_equal(out.reshape(5, ny, nx), g)
    finally:
        lib.le_free_task(t)


@pytest.mark.parametrize("prec", ["f", "d"])
@pytest.mark.parametrize("nx,ny", [(3, 4), (63, 5), (64, 7), (127, 3), (128, 9), (130, 33), (700, 41)])
def test_diagnostics_widths(prec, nx, ny):
    lib = capi.Lib(prec)
    g = np.random.default_rng(ny).standard_normal((ny, nx, 5)).astype(lib.dtype)
    t = _task(lib, nx, ny, ST_AOS, np.ascontiguousarray(g.reshape(-1)))
    try:
        assert lib.step_n(t, 3) == 0  # the rows' padding then holds values too
        out = np.zeros(5 * nx * ny, lib.dtype)
        assert lib.download(t, out) == 0
        f = out.reshape(ny, nx, 5).astype(np.float64)
        rc, d = lib.diagnostics(t)
        assert rc == 0
        rho, c1, c2 = (float(lib.dtype(v)) for v in (1.3, 2.0, 1.1))
        mu, la = rho * c2 * c2, rho * c1 * c1 - 2 * rho * c2 * c2
        vx, vy, sxx, sxy, syy = (f[..., k] for k in range(5))
        e = 0.5 * rho * (vx**2 + vy**2) + (la + 2 * mu) / (8 * mu * (la + mu)) * (sxx**2 + syy**2)
        e = e - 2 * la / (8 * mu * (la + mu)) * sxx * syy + sxy**2 / (2 * mu)
        want = e.sum() * 1.0 * float(lib.dtype(0.9))
        assert abs(d["energy"] - want) <= 1e-12 * abs(want)  # FP64 sums of at most 28700 terms in any order
        for k in range(5):
            assert abs(d["sumsq"][k] - (f[..., k] ** 2).sum()) <= 1e-12 * (f[..., k] ** 2).sum()
            assert d["maxabs"][k] == np.abs(f[..., k]).max()
    finally:
        lib.le_free_task(t)
