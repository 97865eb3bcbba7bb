"""Ring DFTs in block fixed point (csrc/ring.cu), through the plain spherical-
harmonic transforms and the directional ones.

The sizes are the edges of the padded transform length P (powers of two from 8;
K <= P/2 samples) and of its stage split (log2 P odd and even), on both
samplings.  Against the oracle the tolerance is the one of the FP64 path
(1e-12 normwise): a ring transform at P <= 512 contributes below 1e-14."""
import numpy as np
import pytest

from conftest import oracle_sht, random_flm, rel_err
from s2let_gb300.capi import make_parameters

TOL = 1e-12
SIZES = [1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129]


@pytest.mark.gpu
@pytest.mark.parametrize("ss", [0, 1])
@pytest.mark.parametrize("L", SIZES)
def test_sht_at_transform_length_edges(gpu, oracle_port, L, ss):
    rng = np.random.default_rng(7 * L + ss)
    npx = (L + 1) * 2 * L if ss else L * (2 * L - 1)
    for real, spin in ((True, 0), (False, 0), (False, min(2, L - 1))):
        f = rng.normal(size=npx) if real else rng.normal(size=npx) + 1j * rng.normal(size=npx)
        flm = random_flm(rng, L, spin, real=real)
        for direction, x in ((0, f), (1, flm), (2, flm), (3, f)):
            ref = oracle_sht(oracle_port, direction, x, L, spin, real, ss)
            for precision in (0, 1):
                assert gpu.lib.s2let_gpu_set_precision(precision) == 0
                try:
                    got = gpu.sht(direction, x, L, spin, real, ss)
                finally:
                    gpu.lib.s2let_gpu_set_precision(0)
                tol = TOL if precision == 0 or L < 128 else 1e-10  # tensor-core contraction from 128
                assert rel_err(got, ref) < tol, (direction, real, spin, precision)


@pytest.mark.gpu
@pytest.mark.parametrize("case", [(24, 3, 0), (24, 4, 0), (20, 3, 2)], ids=str)
def test_scaling_by_powers_of_two_is_exact(gpu, case):
    """Every ring carries its own power-of-two scale and the contractions are
    plain sums, so scaled inputs give scaled outputs bit for bit while nothing
    leaves the normal range."""
    L, N, spin = case
    p = make_parameters(L, 2.0, 1, N, spin, 0)
    rng = np.random.default_rng(L + N)
    n = gpu.sizes(p)["n_px"]
    f = rng.normal(size=n) if spin == 0 else rng.normal(size=n) + 1j * rng.normal(size=n)
    w, s = gpu.px2wav(f, p, real=spin == 0)
    r = gpu.wav2px(w, s, p, real=spin == 0)
    for k in (-900, 900):
        wk, sk = gpu.px2wav(f * 2.0 ** k, p, real=spin == 0)
        assert np.array_equal(wk, w * 2.0 ** k) and np.array_equal(sk, s * 2.0 ** k)
        assert np.array_equal(gpu.wav2px(wk, sk, p, real=spin == 0), r * 2.0 ** k)


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf], ids=str)
def test_non_finite_samples_come_out_as_nan(gpu, bad):
    L = 20
    p = make_parameters(L, 2.0, 1, 3, 0, 0)
    f = np.random.default_rng(1).normal(size=gpu.sizes(p)["n_px"])
    w, s = gpu.px2wav(f, p, real=True)
    f[77] = bad
    wb, sb = gpu.px2wav(f, p, real=True)
    assert not np.isfinite(wb).any() and not np.isfinite(sb).any()
    w[5] = bad  # one sample of the first scale
    assert not np.isfinite(gpu.wav2px(w, s, p, real=True)).any()


@pytest.mark.gpu
def test_zero_and_subnormal_rings(gpu, oracle_port):
    L = 16
    p = make_parameters(L, 2.0, 1, 3, 0, 0)
    n = gpu.sizes(p)["n_px"]
    w, s = gpu.px2wav(np.zeros(n), p, real=True)
    assert not w.any() and not s.any()
    f = np.random.default_rng(2).normal(size=n)
    tiny = f * 2.0 ** -1060  # subnormal samples: 14 bits and less
    got = gpu.sht(0, tiny, L, 0, True)
    ref = oracle_sht(oracle_port, 0, tiny, L, 0, True)
    # both sum subnormal terms: a few units of 2^-1074 each
    assert np.abs(got - ref).max() <= 64 * 2.0 ** -1074
