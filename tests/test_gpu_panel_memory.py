"""Device memory and the optional digit panels of the FP64 contractions
(csrc/mixed.cu): refused, asked for again, and given back to calls that need the
room.  Whatever the route, results agree within twice the FP64 path's tolerance
(1e-12 normwise)."""
import ctypes as C
import os
import time

import numpy as np
import pytest

from conftest import rel_err
from s2let_gb300.capi import make_parameters

TOL = 2e-12


@pytest.fixture
def lib(gpu):
    lib = gpu.lib
    lib.s2let_gpu_release_plans()
    yield lib
    os.environ.pop("S2LET_GPU_PANEL_RESERVE_GB", None)
    lib.s2let_gpu_set_split_tables(1)
    lib.s2let_gpu_release_plans()


def _slicings(lib, fn):
    """(result, digit-slicing launches of fn)"""
    lib.s2let_gpu_timing_enable(1)
    out = fn()
    rep = (C.c_double * 36)()
    lib.s2let_gpu_timing_report(rep, 9)
    lib.s2let_gpu_timing_enable(0)
    return out, int(rep[4 * 8])


class Pool:
    """The device's default memory pool, through the driver."""

    def __init__(self):
        self.cu = C.CDLL("libcuda.so.1")
        self.pool = C.c_void_p()
        assert self.cu.cuDeviceGetDefaultMemPool(C.byref(self.pool), 0) == 0

    def reserved(self):
        v = C.c_uint64()
        assert self.cu.cuMemPoolGetAttribute(self.pool, 5, C.byref(v)) == 0  # RESERVED_MEM_CURRENT
        return v.value

    def trim(self):
        assert self.cu.cuMemPoolTrimTo(self.pool, C.c_size_t(0)) == 0

    def leave_idle(self, nbytes):
        p = C.c_uint64()
        assert self.cu.cuMemAllocAsync(C.byref(p), C.c_size_t(nbytes), None) == 0
        assert self.cu.cuMemFreeAsync(p, None) == 0


@pytest.mark.gpu
def test_refused_and_asked_again(gpu, lib):
    p = make_parameters(130, 2.0, 6, 2, 0, 0)
    f = np.random.default_rng(2).normal(size=gpu.sizes(p)["n_px"])
    lib.s2let_gpu_set_split_tables(0)
    (w0, s0), n = _slicings(lib, lambda: gpu.px2wav(f, p, real=True))
    assert n == 0 and lib.s2let_gpu_refused_tables() == 0
    lib.s2let_gpu_set_split_tables(1)
    os.environ["S2LET_GPU_PANEL_RESERVE_GB"] = "1e6"
    (w1, s1), n = _slicings(lib, lambda: gpu.px2wav(f, p, real=True))
    assert n == 0 and lib.s2let_gpu_refused_tables() > 0
    assert np.array_equal(w1, w0) and np.array_equal(s1, s0)
    del os.environ["S2LET_GPU_PANEL_RESERVE_GB"]
    time.sleep(0.7)
    (w2, s2), n = _slicings(lib, lambda: gpu.px2wav(f, p, real=True))
    assert n > 0 and lib.s2let_gpu_refused_tables() == 0
    assert rel_err(w2, w0) < TOL and rel_err(s2, s0) < TOL


@pytest.mark.gpu
def test_idle_pool_memory_counts_as_free(gpu, lib):
    torch = pytest.importorskip("torch")
    p = make_parameters(130, 2.0, 6, 2, 0, 0)
    f = np.random.default_rng(3).normal(size=gpu.sizes(p)["n_px"])
    lib.s2let_gpu_set_split_tables(0)
    gpu.px2wav(f, p, real=True)
    lib.s2let_gpu_set_split_tables(1)
    pool = Pool()
    pool.leave_idle(8 << 30)
    torch.cuda.synchronize()
    assert pool.reserved() >= 8 << 30
    free = torch.cuda.mem_get_info()[0]
    # panels (well below 8 GB) and the memory free now would not fit beside each other
    os.environ["S2LET_GPU_PANEL_RESERVE_GB"] = repr(free / 2.0 ** 30)
    _, n = _slicings(lib, lambda: gpu.px2wav(f, p, real=True))
    assert n > 0 and lib.s2let_gpu_refused_tables() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("part", [0.2, 0.5, 0.8])
def test_panels_make_way(gpu, lib, part):
    """With all other memory taken, a batch that fits without the panels runs."""
    torch = pytest.importorskip("torch")
    from s2let_gb300 import torch_ops as T

    p = make_parameters(256, 2.0, 6, 4, 0, 0)
    f = torch.randn(64, gpu.sizes(p)["n_px"], dtype=torch.float64, device="cuda",
                    generator=torch.Generator(device="cuda").manual_seed(1))
    lib.s2let_gpu_set_split_tables(0)
    w0, s0 = T.px2wav(f, p)
    torch.cuda.synchronize()
    before = lib.s2let_gpu_plan_bytes()
    lib.s2let_gpu_set_split_tables(1)
    pool = Pool()
    torch.cuda.synchronize()
    pool.trim()
    w, s = T.px2wav(f, p)
    torch.cuda.synchronize()
    panels, scratch = lib.s2let_gpu_plan_bytes() - before, pool.reserved()
    assert panels > 200 << 20 and lib.s2let_gpu_refused_tables() == 0
    pool.trim()
    free = torch.cuda.mem_get_info()[0]
    block = torch.empty(int(free - scratch + part * panels), dtype=torch.uint8, device="cuda")
    w.zero_()
    s.zero_()
    lib_px2wav = lib.s2let_gpu_analysis_px2wav_real_batch
    rc = lib_px2wav(C.c_void_p(w.data_ptr()), C.c_void_p(s.data_ptr()), C.c_void_p(f.data_ptr()), 64, C.byref(p),
                    C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == 0
    assert rel_err(w.cpu(), w0.cpu()) < TOL and rel_err(s.cpu(), s0.cpu()) < TOL
    given = lib.s2let_gpu_refused_tables()
    del block
    torch.cuda.empty_cache()
    time.sleep(0.7)
    w.zero_()
    T.px2wav(f, p)
    if given:  # not built again behind the caller's back
        assert lib.s2let_gpu_refused_tables() >= given
    lib.s2let_gpu_release_plans()
    assert lib.s2let_gpu_refused_tables() == 0


@pytest.mark.gpu
def test_first_met_inside_a_capture(gpu, lib):
    """A capture cannot build panels: it records the FP64 kernels; panels that it
    does record stay at their addresses."""
    torch = pytest.importorskip("torch")
    from s2let_gb300 import torch_ops as T

    p = make_parameters(130, 2.0, 6, 2, 0, 0)
    f = torch.randn(3, gpu.sizes(p)["n_px"], dtype=torch.float64, device="cuda")
    lib.s2let_gpu_set_split_tables(0)
    w0, s0 = T.px2wav(f, p)
    lib.s2let_gpu_set_split_tables(1)

    def captured():
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            w, s = T.px2wav(f, p)
        w.zero_()
        g.replay()
        torch.cuda.synchronize()
        return g, w, s

    g1, w1, s1 = captured()
    assert torch.equal(w1, w0) and torch.equal(s1, s0)
    w2, s2 = T.px2wav(f, p)  # builds the panels
    assert not torch.equal(w2, w0) and rel_err(w2.cpu(), w0.cpu()) < TOL
    g3, w3, s3 = captured()
    assert torch.equal(w3, w2) and torch.equal(s3, s2)


@pytest.mark.gpu
@pytest.mark.parametrize("L,ss,tensor", [(1364, 1, True), (1365, 0, True), (1365, 1, False), (1366, 0, False)])
def test_longest_reduction_in_eight_slices(gpu, lib, L, ss, tensor):
    """Sums over at most 1365 rings or degrees, so that the leading digit classes
    stay exact; longer ones on the FP64 pipe."""
    rng = np.random.default_rng(L)
    npx = (L + 1) * 2 * L if ss else L * (2 * L - 1)
    flm = gpu.sht(0, rng.normal(size=npx), L, 0, True, ss)  # coefficients of a real map
    (f, back), n = _slicings(lib, lambda: (lambda f: (f, gpu.sht(0, f, L, 0, True, ss)))(gpu.sht(1, flm, L, 0, True, ss)))
    assert (n > 0) == tensor
    assert rel_err(back, flm) < 1e-12


@pytest.mark.gpu
def test_switched_off_after_they_were_built(gpu, lib):
    """s2let_gpu_set_split_tables(0) means the FP64 tables from the next call on."""
    p = make_parameters(130, 2.0, 6, 2, 0, 0)
    f = np.random.default_rng(4).normal(size=gpu.sizes(p)["n_px"])
    (w1, s1), n = _slicings(lib, lambda: gpu.px2wav(f, p, real=True))
    assert n > 0
    lib.s2let_gpu_set_split_tables(0)
    (w0, s0), n = _slicings(lib, lambda: gpu.px2wav(f, p, real=True))
    assert n == 0 and rel_err(w0, w1) < TOL
    lib.s2let_gpu_set_split_tables(1)
    (w2, s2), n = _slicings(lib, lambda: gpu.px2wav(f, p, real=True))
    assert n > 0 and np.array_equal(w2, w1) and np.array_equal(s2, s1)


@pytest.mark.gpu
def test_given_back_beside_other_threads(gpu, lib):
    """Calls refused for want of memory take panels back while three threads build and
    use them; panels in use stay, the others' contractions go to the FP64 kernels."""
    import threading

    torch = pytest.importorskip("torch")
    sizes = [64, 70, 80, 90, 100, 110, 120, 128, 130, 140]
    maps, ref = {}, {}
    for L in sizes:
        p = make_parameters(L, 2.0, 4, 2, 0, 0)
        maps[L] = (p, np.random.default_rng(L).normal(size=gpu.sizes(p)["n_px"]))
        ref[L] = gpu.px2wav(maps[L][1], p, real=True)[0]
    lib.s2let_gpu_release_plans()
    bad, done = [], threading.Event()

    def transform(order):
        for L in order * 3:
            p, f = maps[L]
            w, _ = gpu.px2wav(f, p, real=True)
            if lib.s2let_gpu_last_error() != 0 or rel_err(w, ref[L]) > TOL:
                bad.append(L)

    p = make_parameters(48, 2.0, 2, 3, 0, 0)
    sz = gpu.sizes(p)
    f, w, s = (torch.zeros(sz[k], dtype=torch.float64, device="cuda") for k in ("n_px", "n_wav", "n_scal"))
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def exhaust():
        while not done.is_set():
            rc = lib.s2let_gpu_analysis_px2wav_real_batch(C.c_void_p(w.data_ptr()), C.c_void_p(s.data_ptr()),
                                                          C.c_void_p(f.data_ptr()), 20_000_000, C.byref(p), st)
            if rc != 4:
                bad.append(rc)
            time.sleep(0.01)

    lib.s2let_gpu_last_error()
    threads = [threading.Thread(target=transform, args=(sizes[k:] + sizes[:k],)) for k in (0, 3, 6)]
    other = threading.Thread(target=exhaust)
    other.start()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    done.set()
    other.join()
    assert not bad
    assert lib.s2let_gpu_refused_tables() > 0
