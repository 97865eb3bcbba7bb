"""Accuracy of the FP64 transforms on recomputed tables (csrc/recompute.cu), against
the stored tables, whose own errors (5e-16 inverse, 1e-15 forward) are far below.
Bounds: the errors of an unscaled FP64 recursion with an FP64 quadrature on the same
maps (rms), which a faster form has no business exceeding.  One map's error scatters by
a third, so the small band-limits go together (geometric mean)."""
import numpy as np
import pytest

from conftest import random_flm


def errors(gpu, L, spin):
    """rms errors (inverse, forward) over two white maps"""
    lib = gpu.lib
    rng = np.random.default_rng(L)
    real = spin == 0 and L < 300
    if L < 300:
        flms = [random_flm(rng, L, spin, real=real) for _ in range(2)]
    else:
        flms = []
        for _ in range(2):
            flms.append(rng.normal(size=L * L) + 1j * rng.normal(size=L * L))
            flms[-1][:spin * spin] = 0
    try:
        lib.s2let_gpu_release_plans()
        assert lib.s2let_gpu_set_table_mode(1) == 0
        ref = [gpu.sht(1, x, L, spin, real) for x in flms]
        lib.s2let_gpu_release_plans()
        assert lib.s2let_gpu_set_table_mode(2) == 0
        inv = [np.linalg.norm(gpu.sht(1, x, L, spin, real) - f) / np.linalg.norm(f) for x, f in zip(flms, ref)]
        fwd = [np.linalg.norm(gpu.sht(0, f, L, spin, real) - x) / np.linalg.norm(x) for x, f in zip(flms, ref)]
    finally:
        lib.s2let_gpu_set_table_mode(0)
        lib.s2let_gpu_release_plans()
    return np.sqrt(np.mean(np.square(inv))), np.sqrt(np.mean(np.square(fwd)))


@pytest.mark.gpu
@pytest.mark.parametrize("spin,inv,fwd", [(0, 4.50e-15, 2.41e-15), (2, 4.80e-15, 2.49e-15)])
def test_small_band_limits(gpu, spin, inv, fwd):
    e = np.array([errors(gpu, L, spin) for L in (64, 65, 70, 80, 96, 100, 128, 150, 181, 200, 256)])
    assert (np.exp(np.log(e).mean(axis=0)) <= [inv, fwd]).all()


@pytest.mark.gpu
@pytest.mark.parametrize("L,spin,inv,fwd", [(512, 0, 6.24e-15, 3.63e-15), (700, 0, 6.83e-15, 3.94e-15),
                                            (512, 2, 6.50e-15, 3.85e-15), (700, 2, 6.87e-15, 4.14e-15)])
def test_large_band_limits(gpu, L, spin, inv, fwd):
    e = errors(gpu, L, spin)
    assert e[0] <= inv
    assert e[1] <= fwd


@pytest.mark.gpu
def test_split_precision(gpu):
    """The double-float sums: white maps, and a constant map, whose sums have one sign.
    Bounds: the errors with sums renormalised after every term (geometric mean over the
    band-limits, rings and recursion of the time included)."""
    lib = gpu.lib
    e = []
    for L in (64, 70, 96, 100, 128, 150, 181, 200, 256, 300, 384, 512):
        rng = np.random.default_rng(L)
        flm = rng.normal(size=L * L) + 1j * rng.normal(size=L * L)
        f00 = 0.7 * np.sqrt(4 * np.pi)
        try:
            lib.s2let_gpu_release_plans()
            assert lib.s2let_gpu_set_table_mode(1) == 0
            f = gpu.sht(1, flm, L, 0, False)
            lib.s2let_gpu_release_plans()
            assert lib.s2let_gpu_set_table_mode(2) == 0 and lib.s2let_gpu_set_precision(1) == 0
            inv, fwd = gpu.sht(1, flm, L, 0, False), gpu.sht(0, f, L, 0, False)
            const = gpu.sht(0, np.full(L * (2 * L - 1), 0.7), L, 0, True)
        finally:
            lib.s2let_gpu_set_precision(0)
            lib.s2let_gpu_set_table_mode(0)
            lib.s2let_gpu_release_plans()
        const[0] -= f00
        e.append([np.linalg.norm(inv - f) / np.linalg.norm(f), np.linalg.norm(fwd - flm) / np.linalg.norm(flm),
                  np.linalg.norm(const) / f00])
    assert (np.exp(np.log(e).mean(axis=0)) <= [2.37e-14, 1.94e-14, 1.66e-14]).all()
