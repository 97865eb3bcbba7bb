"""Ring DFTs at the padded lengths 2048, 4096 and 8192 through the plain inverse
transform, seen apart from the contraction: coefficients at a few orders m leave
every ring with those orders only, so each ring must equal the sum of its own
projections on them.  Bound 1e-15 of the ring's level: FP64 rounding of the
samples (1.1e-16), and the 4e-16 that an FP64 transform of the ring is off."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("ms", [[1 / 5], [-0.8, -0.3, 0.0, 0.3, 0.999]], ids=["one", "five"])
@pytest.mark.parametrize("L,ss", [(512, 0), (512, 1), (1024, 0), (1024, 1), (2048, 0)])
def test_rings_of_few_orders(gpu, L, ss, ms):
    ms = sorted({int(round(x * (L - 1))) for x in ms})
    flm = np.zeros(L * L, np.complex128)
    rng = np.random.default_rng(L)
    for m in ms:
        l = min(L - 1, abs(m) + 3)
        flm[l * l + l + m] = complex(*rng.normal(size=2))
    lib = gpu.lib
    try:
        assert lib.s2let_gpu_set_table_mode(2) == 0  # small tables
        f = gpu.sht(1, flm, L, 0, False, ss)
    finally:
        lib.s2let_gpu_set_table_mode(0)
        lib.s2let_gpu_release_plans()
    K = 2 * L if ss else 2 * L - 1
    rows = f.reshape(-1, K)
    rows = rows[np.unique(np.linspace(0, rows.shape[0] - 1, 48).astype(int))].astype(np.clongdouble)
    root = np.exp(2j * np.pi * np.arange(K).astype(np.longdouble) / K)
    basis = np.stack([root[(m * np.arange(K)) % K] for m in ms])
    proj = rows @ basis.conj().T / K
    err = np.sqrt((np.abs(rows - proj @ basis) ** 2).sum(1))
    level = np.sqrt((np.abs(rows) ** 2).sum(1))
    seen = level > 1e-200  # near the poles high orders underflow
    assert seen.sum() > 10
    assert (err[seen] / level[seen]).max() < 1e-15


@pytest.mark.gpu
@pytest.mark.parametrize("table_mode", [1, 2])
@pytest.mark.parametrize("L", [128, 512, 1024])
def test_monopole_of_white_maps(gpu, L, table_mode):
    """Rounding errors of one sign in every ring would add up in the monopole.  Bound
    1e-14 of a coefficient's level: the worst degree of an FP64 transform of such
    maps is 4e-15 off at L = 1024."""
    rng = np.random.default_rng(L)
    l = np.repeat(np.arange(L), 2 * np.arange(L) + 1)
    m = np.arange(L * L) - l * l - l
    flm = (rng.normal(size=L * L) + 1j * rng.normal(size=L * L)) / np.sqrt(2)
    neg, mir = m < 0, l * l + l - m
    flm[m == 0] = flm[m == 0].real * np.sqrt(2)
    flm[neg] = (-1.0) ** m[neg] * np.conj(flm[mir[neg]])
    flm[0] = 0.0
    lib = gpu.lib
    lib.s2let_gpu_release_plans()
    try:
        assert lib.s2let_gpu_set_table_mode(table_mode) == 0
        back = gpu.sht(0, gpu.sht(1, flm, L, 0, True), L, 0, True)
    finally:
        lib.s2let_gpu_set_table_mode(0)
        lib.s2let_gpu_release_plans()
    assert abs(back[0]) < 1e-14
