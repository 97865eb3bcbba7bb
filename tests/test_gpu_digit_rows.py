"""Table rows far below the largest: near the poles the Wigner functions of high
orders are tiny over every degree, down to the smallest normal numbers.  A row has
an exponent of its own in the digit slices (csrc/mixed.cu), so coefficients at the
row's largest degree come out of the tensor cores with the relative accuracy of the
FP64 kernels, ring by ring."""
import ctypes as C

import numpy as np
import pytest


@pytest.fixture
def lib(gpu):
    gpu.lib.s2let_gpu_release_plans()
    yield gpu.lib
    gpu.lib.s2let_gpu_set_split_tables(1)
    gpu.lib.s2let_gpu_release_plans()


@pytest.mark.gpu
@pytest.mark.parametrize("L,m,ss", [(256, 100, 0), (256, -200, 1), (512, 300, 0)])
def test_rings_near_the_poles(gpu, lib, L, m, ss):
    flm = np.zeros(L * L, np.complex128)
    l = L - 1
    flm[l * l + l + m] = 1.0 - 0.5j
    K = 2 * L if ss else 2 * L - 1

    def level():
        f = gpu.sht(1, flm, L, 0, False, ss).reshape(-1, K)
        return np.abs(f).max(axis=1)

    lib.s2let_gpu_timing_enable(1)
    got = level()
    rep = (C.c_double * 36)()
    lib.s2let_gpu_timing_report(rep, 9)
    lib.s2let_gpu_timing_enable(0)
    assert rep[4 * 8] > 0  # digit slicing ran
    lib.s2let_gpu_release_plans()
    lib.s2let_gpu_set_split_tables(0)
    ref = level()
    # rings out of the order's reach (sin theta < |m| / l), where the functions grow with
    # the degree and the row's largest value is the last; elsewhere they oscillate, and a
    # degree near a zero has a value far below its row's largest
    t = np.arange(ref.size)
    theta = np.pi * t / L if ss else np.pi * (2 * t + 1) / (2 * L - 1)
    seen = (ref > 1e-290) & (np.sin(theta) < 0.9 * abs(m) / l)
    assert (ref[seen] < 2.0 ** -130).sum() >= 4  # rings that a row exponent of 8 bits cannot hold
    # 55 bits for the row's largest entry; ring transforms 4e-16 each
    assert np.abs(got[seen] / ref[seen] - 1).max() < 2e-15
