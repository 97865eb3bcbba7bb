"""Shared-memory limits of the ring kernels (s2let_gb300/csrc/smemlimit.h): one
kernel serves several sizes from several host threads, so a limit, once raised for
a launch, stays."""
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "s2let_gb300", "csrc")

HARNESS = r"""
#include "smemlimit.h"
int main() {
  s2g::SharedMemoryLimits limits;
  int kernel = 0, sets = 0, carve = 0;
  size_t limit = 48 * 1024;  // the attribute as the driver holds it
  const auto prepare = [&](size_t b, int c) {
    limits.prepare(&kernel, b, c, [&](size_t v) { limit = v; ++sets; }, [&](int v) { carve = v; });
  };
  prepare(64 << 10, 86);
  if (limit < (64 << 10) || carve != 86) return 1;
  prepare(128 << 10, 100);  // one thread prepares a large launch,
  prepare(64 << 10, 86);    // another a small one,
  if (limit < (128 << 10) || carve != 86) return 2;  // and the large one follows
  prepare(32 << 10, 50);
  prepare(128 << 10, 100);
  return limit >= (128 << 10) && carve == 100 && sets == 2 ? 0 : 3;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_limits_are_only_raised(tmp_path):
    (tmp_path / "h.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{CSRC}", str(tmp_path / "h.cpp"), "-o", str(tmp_path / "h")],
                   check=True)
    assert subprocess.run([str(tmp_path / "h")]).returncode == 0


@pytest.mark.gpu
def test_threads_with_rings_of_two_sizes(gpu):
    """64 KB and 128 KB launches of one kernel from four threads."""
    lib = gpu.lib
    rng = np.random.default_rng(5)
    f = {L: rng.normal(size=L * (2 * L - 1)) for L in (600, 1100)}
    try:
        assert lib.s2let_gpu_set_table_mode(2) == 0
        ref = {L: gpu.sht(0, f[L], L, 0, True) for L in f}
        bad = []

        def run(L):
            lib.s2let_gpu_set_table_mode(2)
            for _ in range(6):
                got = gpu.sht(0, f[L], L, 0, True)
                if lib.s2let_gpu_last_error() != 0 or not np.array_equal(got, ref[L]):
                    bad.append(L)

        threads = [threading.Thread(target=run, args=(L,)) for L in (600, 1100, 600, 1100)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not bad
    finally:
        lib.s2let_gpu_set_table_mode(0)
        lib.s2let_gpu_release_plans()
