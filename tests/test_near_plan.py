"""How the symmetric near field cuts its work (csrc/near_plan.hpp), at sizes of parts that no test could run: the scratch
stays within its bound, the slots fit an int, and no size is refused."""
import ctypes as C
import os
import subprocess

import pytest

from conftest import ROOT

SHIM = r"""
#include "near_plan.hpp"
extern "C" int part_length(long long n) { return fb::equal_part_length(n); }
extern "C" double part_scratch(long long n) { return fb::equal_part_scratch(n); }
// part a is near the parts up to `reach` away
extern "C" void plan(int n, const int *count, int slotBytes, double direct, int reach, long long *out) {
  const std::vector<int> c(count, count + n);
  const fb::NearPlan p = fb::plan_near_tasks(c, slotBytes, direct, [&](auto f) {
    for (int a = 0; a < n; a++)
      for (int b = a + 1; b < n && b - a <= reach; b++) f(a, b, true);
  });
  out[0] = p.tasks; out[1] = p.chunk; out[2] = p.slots; out[3] = p.count;
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "cuda-fabipb_b200", "csrc"),
                    str(d / "plan.cpp"), "-o", str(d / "plan.so")], check=True)
    so = C.CDLL(str(d / "plan.so"))
    so.part_length.argtypes = [C.c_longlong]
    so.part_scratch.argtypes, so.part_scratch.restype = [C.c_longlong], C.c_double
    return so


def plan(so, count, slot_bytes, direct, reach):
    """direct: the direct context's limit in bytes, 0 for an FMM context"""
    out = (C.c_longlong * 4)()
    so.plan(len(count), (C.c_int * len(count))(*count), slot_bytes, C.c_double(direct), reach, out)
    tasks, chunk, slots, n = out
    # the slots and tasks by the tasks' own arithmetic
    want = number = 0
    for a in range(len(count)):
        for b in range(a + 1, min(len(count), a + reach + 1)):
            r, t = max(count[a], count[b]), min(count[a], count[b])
            k = -(-r // chunk)
            want, number = want + r + k * t, number + k
    assert (slots, n) == (want, number)
    return bool(tasks), chunk, slots, n


@pytest.mark.parametrize("panels", [2, 129, 320, 12797, 32768, 32769, 65537, 100352, 204800, 800000, 2097152, 8388608])
def test_direct_fp64_context(shim, panels):
    """Runs of panels: at most 256 of them, their scratch within 4 KiB a panel."""
    size = shim.part_length(panels)
    count = [size] * (panels // size) + ([panels % size] if panels % size else [])
    assert len(count) <= 256
    on, chunk, slots, n = plan(shim, count, 16, shim.part_scratch(panels), len(count))
    assert on == (len(count) > 1) and 16 * slots <= 4096 * panels
    assert panels < 100000 or n > 14000   # tasks for the whole chip


@pytest.mark.parametrize("leaves,size,tasks", [(70, 290, True), (100, 2000, True), (56, 37500, False), (8, 2 ** 18, False), (4000, 500, False)])
def test_direct_mixed_context(shim, leaves, size, tasks):
    """The leaves: within 512 MiB and with work for half the chip, or no tasks."""
    on, chunk, slots, n = plan(shim, [size] * leaves, 8, 1.02 * 512 * 1024 ** 2, leaves)
    assert on == tasks
    assert not on or (8 * slots <= 1.02 * 512 * 1024 ** 2 and (chunk <= 256 or 2 * n >= 2368))


@pytest.mark.parametrize("leaves,size,reach,tasks,chunk", [
    (70, 290, 70, True, 256),            # a small surface in large leaves: the chunks cost little
    (7930, 264, 21, True, 256),          # the two-shell surface's leaves
    (7930, 264, 5, True, 256),
    (56, 37500, 56, True, 16384),        # a shallow tree on 2,100,000 panels: chunks grow until they cost a copy of T or so
    (8, 2 ** 18, 8, True, 2 ** 15),
    (3, 5 * 10 ** 8, 3, False, None),    # above 2^31 slots however it is cut: the finishing kernel
])
def test_fmm_context(shim, leaves, size, reach, tasks, chunk):
    for slot_bytes in (8, 16):
        on, got, slots, _ = plan(shim, [size] * leaves, slot_bytes, 0.0, reach)
        assert on == tasks
        if tasks:
            whole = sum(2 * size * min(reach, leaves - 1 - a) for a in range(leaves))
            assert slots < 2 ** 31 and slots * slot_bytes <= max(512 * 1024 ** 2, 2 * whole * slot_bytes)
        if chunk and slot_bytes == 8:
            assert got == chunk
