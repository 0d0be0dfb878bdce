"""How a batched launch shares its lanes out (the host functions that size the
grid and the rule the kernels apply to it, compiled for the host): a limit on
the blocks keeps every launch to one thread per line, whatever its size and
that of the batch's other store types; without one the shape the kernel forms
fits the grid."""
import ctypes
import subprocess

import pytest

from fastqsl_gb300 import _build, api

SOURCE = r"""
#include "qsl_internal.h"
#include "qsl_batch.cuh"
using namespace qsl;
extern "C" void shape(long long n, int resident, int max_blocks, long long out[3]) {
    const int grid = batch_grid(n, resident, max_blocks);
    const LaunchShape s = batch_shape(n, (long long)grid * (kTraceThreads / 32), max_blocks <= 0);
    out[0] = grid; out[1] = s.split; out[2] = s.spread;
}
"""
RESIDENT = 152 * 6  # blocks of the batched kernels at their default budget


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    d = tmp_path_factory.mktemp("shape_probe")
    src, lib = d / "probe.cu", d / "probe.so"
    src.write_text(SOURCE)
    subprocess.run([_build.NVCC, *_build.COMMON, *_build.ARCH, "-shared", "-cudart", "static", str(src), "-o",
                    str(lib)], check=True, capture_output=True)
    f = ctypes.CDLL(str(lib)).shape

    def call(n, max_blocks=0):
        out = (ctypes.c_longlong * 3)()
        f(ctypes.c_longlong(n), RESIDENT, max_blocks, out)
        return tuple(out)
    return call


LINES = [1, 31, 32, 33, 64, 96, 128, 1000, 4096, 14592, 14593, 29184, 29185, 58368, 58369, 58400, 10 ** 6]


@pytest.mark.parametrize("n", LINES)
def test_a_limit_keeps_one_thread_per_line(shape, n):
    for limit in (1, 2, 100, (n + 127) // 128, 4 * ((n + 127) // 128), 1 << 30):
        grid, split, spread = shape(n, limit)
        assert (split, spread) == (0, 1)
        assert grid == min(limit, (n + 127) // 128)


@pytest.mark.parametrize("n", LINES)
def test_without_a_limit_one_turn_of_the_grid_holds_the_lines(shape, n):
    grid, split, spread = shape(n)
    assert spread in (1, 2, 4) and (split or spread == 1)
    lines = grid * 4 // 2 * (32 // spread) if split else grid * 128
    assert lines >= n
    if n <= 14000:
        assert split and spread == 4 and grid <= RESIDENT
    if n > 60000:
        assert not split


def test_a_shared_launch_is_limited_without_being_cut(monkeypatch):
    calls = []

    class Lib:
        def __getattr__(self, name):
            return lambda *a: calls.append((name, a)) or 0

    monkeypatch.setattr(api._lib, "load", Lib)
    b = object.__new__(api.PlaneQBatch)
    b.handle, b.occupancy, b.Q = None, 0, []
    for blocks, share, limit in ((0, False, 0), (0, True, 1 << 30), (300, True, 300), (300, False, 300)):
        b.max_blocks = blocks
        calls.clear()
        b.run_main(stream=0, share=share)
        b.run_post(stream=0, share=share)
        assert [a[3 if n.endswith("main") else 1] for n, a in calls if "run_" in n] == [limit, limit]
