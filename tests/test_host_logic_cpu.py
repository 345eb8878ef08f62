"""Host logic that stands in headers without CUDA calls, compiled and run here by the host compiler."""
import os
import subprocess
import tempfile

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "le2d_b200", "csrc")


def _run(source: str) -> list[str]:
    with tempfile.TemporaryDirectory() as td:
        src, exe = os.path.join(td, "p.cpp"), os.path.join(td, "p")
        open(src, "w").write(source)
        subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I", CSRC, src, "-o", exe], check=True)
        return subprocess.run([exe], check=True, capture_output=True, text=True, timeout=60).stdout.split()


def test_rows_copied_by_kernel_only_on_one_device():
    """le2d_rows_out / le2d_rows_in: one kernel only if the state, the buffer and the current device
    agree, the buffer is aligned to an element and the copy lies within its allocation."""
    cases = [  # device memory, its device, address, base, extent, bytes, element, task's and current device -> kernel
        (1, 0, 4096, 4096, 400, 400, 4, 0, 0, 1),
        (1, 2, 4100, 4096, 404, 400, 4, 2, 2, 1),
        (1, 1, 4096, 4096, 400, 400, 4, 0, 1, 0),  # the state on another device than the buffer
        (1, 0, 4096, 4096, 400, 400, 4, 0, 1, 0),  # both on another device than the current one
        (1, 1, 4096, 4096, 400, 400, 4, 0, 0, 0),
        (0, 0, 4096, 4096, 400, 400, 4, 0, 0, 0),  # not plain device memory
        (1, 0, 4098, 4096, 800, 400, 4, 0, 0, 0),  # not aligned to an element
        (1, 0, 4100, 4096, 800, 400, 8, 0, 0, 0),
        (1, 0, 4096, 4096, 399, 400, 4, 0, 0, 0),  # past the end of the allocation
        (1, 0, 4100, 4096, 400, 400, 4, 0, 0, 0),
        (1, 0, 4096, 4100, 800, 400, 4, 0, 0, 0),  # not in the allocation found
        (1, 0, 8192, 4096, 400, 400, 4, 0, 0, 0),
    ]
    body = "".join(
        f"  {{ le2d::RowsBuffer b; b.device_memory = {c[0]}; b.device = {c[1]}; b.at = {c[2]}; b.base = {c[3]}; "
        f"b.extent = {c[4]}; std::printf(\"%d \", (int)le2d::rows_by_kernel(b, {c[5]}, {c[6]}, {c[7]}, {c[8]})); }}\n"
        for c in cases)
    out = _run('#include <cstdio>\n#include "rows_copy.h"\nint main() {\n' + body + "}\n")
    assert [int(x) for x in out] == [c[-1] for c in cases]
