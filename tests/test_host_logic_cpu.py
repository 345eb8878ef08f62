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


POOL = r"""
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <thread>
#include "result_pool.h"
static std::atomic<int> locks{0}, unlocks{0};
static bool none = false;
struct Fake {
  static void* lock(size_t n) { if (none) return nullptr; ++locks; return malloc(n); }
  static void unlock(void* p) { ++unlocks; free(p); }
};
using Pool = le2d::ResultPool<Fake>;
using Result = le2d::PooledResult<Fake>;
constexpr size_t P = Pool::kPiece;
static std::unique_ptr<Result> get(const std::shared_ptr<Pool>& p, size_t bytes, bool contiguous = false) {
  auto r = std::make_unique<Result>();
  if (!r->make(p, bytes, contiguous) || r->bytes() != bytes) { std::printf("no-memory "); return nullptr; }
  unsigned char v = 0;
  for (auto& q : r->parts()) for (size_t i = 0; i < q.second; i += 4096) q.first[i] = (char)++v;
  std::vector<char> out(bytes + 1, 77);
  r->copy_to(out.data());
  if (out[bytes] != 77) std::printf("past-the-end ");
  size_t at = 0; v = 0;
  for (auto& q : r->parts()) { for (size_t i = 0; i < q.second; i += 4096) if (out[at + i] != (char)++v) std::printf("wrong "); at += q.second; }
  if (at != bytes) std::printf("size ");
  return r;
}
static void burst(const std::shared_ptr<Pool>& p, std::vector<size_t> sizes) {
  std::vector<std::unique_ptr<Result>> held;
  for (size_t n : sizes) held.push_back(get(p, n));
  p->idle();
}
static int grow_all(const std::shared_ptr<Pool>& p) { int n = 0; while (p->wants_more()) { p->grow(); ++n; } return n; }
int main() {
  {
    auto p = std::make_shared<Pool>();
    const std::vector<size_t> mixed{0, 1, P - 1, P, P + 1, 5 * P + 3, 17 * P};  // 1+1+1+1+2+6+17 = 29 pieces
    p->idle();
    burst(p, mixed);
    std::printf("%d ", grow_all(p));               // one busy period alone: nothing
    burst(p, mixed);
    const int before = locks;                      // nothing locked while results come and go
    std::printf("%d %d ", before, grow_all(p));    // then ceil(29 / 8) slabs
    burst(p, mixed); burst(p, {40 * P, 3 * P, 9 * P});  // other sizes: no unlocking, no locking
    std::printf("%d %d ", (int)locks, (int)unlocks);
    { auto a = get(p, 29 * P); auto b = get(p, 4 * P); auto c = get(p, 2 * P, true); }  // malloc where the pool is short
    burst(p, {Pool::kHeld + 1}); burst(p, {Pool::kHeld + 1});  // never fits: not asked for
    std::printf("%d ", grow_all(p));               // 33 at once just now, 52 before: a fifth slab
    std::vector<size_t> many(3000, P);             // more than the pool may hold
    burst(p, many); burst(p, many);
    std::printf("%d %d ", grow_all(p), (int)(locks * Pool::kSlabPieces * P <= Pool::kHeld));
    none = true; many.assign(8, P);
    auto held = get(p, P); p.reset();              // a result outlives the server's handle on the pool
    held.reset();
    std::printf("%d ", (int)(locks == unlocks));
  }
  {
    auto p = std::make_shared<Pool>();             // page-locking fails: malloc, and no endless tries
    burst(p, {P}); burst(p, {P});
    std::printf("%d ", grow_all(p));
    auto r = get(p, 3 * P);
  }
  none = false;
  {
    auto p = std::make_shared<Pool>();
    burst(p, std::vector<size_t>(64, P)); burst(p, std::vector<size_t>(64, P));
    std::vector<std::thread> th;
    for (int k = 0; k < 6; ++k) th.emplace_back([&, k] { for (int i = 0; i < 300; ++i) auto r = get(p, (i * 7 + k) % 9 * P / 2); });
    std::thread worker([&] { for (int i = 0; i < 200; ++i) { p->idle(); if (p->wants_more()) p->grow(); } });
    for (auto& t : th) t.join();
    worker.join();
    grow_all(p);
    std::printf("%d", (int)(p->take(64).size() == 64));  // every piece came back
  }
}
"""


def test_result_pool():
    """A server's page-locked results (result_pool.h): nothing is locked or unlocked between results,
    mixed sizes share the pieces, growth waits for two busy periods and ends at the bound."""
    out = _run(POOL)
    assert out == ["0", "0", "4", "4", "0", "1", "59", "1", "1", "1", "1"], out


# FP64 default (148 SMs x 12 warps, 60 columns a strip), whole launches: us a step by segment length.
WHOLE_F64 = {
    (1000, 1000): {16: 30.8, 24: 41.3, 32: 38.9, 40: 47.1, 48: 55.3, 64: 71.0, 96: 102.4, 128: 133.2},
    (1500, 1500): {16: 62.6, 24: 55.5, 32: 53.1, 40: 63.6, 48: 74.1, 64: 94.2, 96: 102.8, 128: 135.3},
    (1800, 1800): {16: 74.6, 24: 90.1, 32: 74.0, 40: 88.5, 48: 76.3, 64: 98.0, 96: 104.5, 128: 135.3},
    (2048, 2048): {16: 95.3, 24: 105.6, 32: 114.5, 40: 112.8, 48: 104.1, 64: 97.7, 96: 140.6, 128: 135.6},
    (3000, 3000): {16: 187.1, 24: 188.0, 32: 182.9, 40: 182.2, 48: 202.6, 64: 221.7, 96: 196.9, 128: 248.4},
    (4096, 4096): {16: 336.4, 24: 326.1, 32: 319.6, 40: 322.4, 48: 323.0, 64: 317.0, 96: 347.1, 128: 398.7},
    (6000, 6000): {16: 729.5, 24: 720.4, 32: 693.1, 40: 691.4, 48: 686.8, 64: 662.8, 96: 676.2, 128: 659.7},
    (8192, 2048): {16: 333.0, 24: 316.0, 32: 309.3, 40: 307.8, 48: 305.8, 64: 316.6, 96: 314.6, 128: 386.5},
    (16384, 128): {16: 61.7, 24: 55.1, 32: 53.2, 40: 63.8, 48: 74.6, 64: 71.7, 96: 102.7, 128: 135.2},
}


def test_segment_model_of_whole_fp64_launches():
    """The segment length picked for the FP64 default is within 5 % of the fastest one measured."""
    calls = "".join(f'  std::printf("%d ", le2d::model_segment(le2d::kDefaultModelF64, {ny}, {(nx + 59) // 60}, '
                    f'148 * 12, 16));\n' for nx, ny in WHOLE_F64)
    out = _run('#include <cstdio>\n#include "segment_model.h"\nint main() {\n' + calls + "}\n")
    for (size, times), seg in zip(WHOLE_F64.items(), map(int, out)):
        assert times[seg] <= 1.05 * min(times.values()), (size, seg)
