"""FP64 results from the tensor cores: contractions in eight digit slices
(csrc/mixed.cu), the FP64 mode's forward contractions and both modes' adjoints
from band-limit 128.

The band-limits are the edges of the kernel's 128-row tiles and 64-wide
K-chunks.  Against the oracle the tolerance is the FP64 path's (1e-12
normwise); the FP64 kernels, reached by switching table copies off, must agree
within twice that."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_err
from s2let_gb300.capi import make_parameters

TOL = 1e-12
# L, N, spin, real, sampling: L = 64 (the smallest), 128 (+-1: one row tile and K-chunk edge), 192, 193 (K = 3 x 64 and past it), 257
CASES = [(64, 3, 0, True, 0), (65, 2, 1, False, 1), (100, 4, 0, True, 0), (128, 3, 0, True, 0), (129, 2, 1, False, 0), (128, 2, 0, True, 1), (192, 1, 0, False, 0),
         (193, 4, 0, True, 0), (160, 3, 2, False, 1), (257, 2, 0, True, 0)]


def _signal(rng, n, real):
    return rng.normal(size=n) if real else rng.normal(size=n) + 1j * rng.normal(size=n)


def _all_ops(g, f, w, s, p, real):
    return [*g.px2wav(f, p, real=real), g.wav2px(w, s, p, real=real), g.analysis_adjoint_wav2px(w, s, p, real=real),
            *g.synthesis_adjoint_px2wav(f, p, real=real)]


@pytest.fixture
def fresh_plans(gpu):
    gpu.lib.s2let_gpu_release_plans()
    yield gpu.lib
    gpu.lib.s2let_gpu_set_split_tables(1)
    gpu.lib.s2let_gpu_set_precision(0)
    gpu.lib.s2let_gpu_release_plans()


def _slicings(lib, fn):
    """(result, digit-slicing launches of fn)"""
    lib.s2let_gpu_timing_enable(1)
    out = fn()
    rep = (C.c_double * 36)()
    lib.s2let_gpu_timing_report(rep, 9)
    lib.s2let_gpu_timing_enable(0)
    return out, int(rep[4 * 8])


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=str)
def test_against_oracle_and_fp64_kernels(gpu, oracle_port, fresh_plans, case):
    L, N, spin, real, ss = case
    lib = fresh_plans
    p = make_parameters(L, 2.0, 5, N, spin, 0, sampling_scheme=ss)
    rng = np.random.default_rng(31 * L + N)
    sz = gpu.sizes(p)
    f, w, s = (_signal(rng, sz[k], real) for k in ("n_px", "n_wav", "n_scal"))
    ref = _all_ops(oracle_port, f, w, s, p, real)
    got, sliced = _slicings(lib, lambda: _all_ops(gpu, f, w, s, p, real))
    assert sliced > 0
    for a, b in zip(got, ref):
        assert rel_err(a, b) < TOL
    # the adjoints at split precision take the same eight slices (one-map calls contract in double-float)
    lib.s2let_gpu_set_precision(1)
    old = lib.s2let_gpu_get_df_max_maps()
    lib.s2let_gpu_set_df_max_maps(0)
    try:
        adj = gpu.analysis_adjoint_wav2px(w, s, p, real=real)
    finally:
        lib.s2let_gpu_set_df_max_maps(old)
        lib.s2let_gpu_set_precision(0)
    assert rel_err(adj, ref[3]) < 10 * TOL
    lib.s2let_gpu_release_plans()
    lib.s2let_gpu_set_split_tables(0)
    fp64, sliced = _slicings(lib, lambda: _all_ops(gpu, f, w, s, p, real))
    assert sliced == 0
    for a, b in zip(got, fp64):
        assert rel_err(a, b) < 2 * TOL


@pytest.mark.gpu
@pytest.mark.parametrize("nb", [2, 5, 9, 17, 33])
def test_batches_give_the_bits_of_single_maps(gpu, fresh_plans, nb):
    """Every column is sliced and summed by itself, whatever the columns per
    pass (16, 32, 64) and the map groups per launch."""
    import torch

    from s2let_gb300 import torch_ops as T

    p = make_parameters(130, 2.0, 6, 2, 0, 0)
    f = torch.randn(nb, gpu.sizes(p)["n_px"], dtype=torch.float64, device="cuda",
                    generator=torch.Generator(device="cuda").manual_seed(nb))
    w, s = T.px2wav(f, p)
    r = T.wav2px(w, s, p)
    for b in (0, nb // 2, nb - 1):
        w1, s1 = T.px2wav(f[b:b + 1], p)
        assert torch.equal(w1[0], w[b]) and torch.equal(s1[0], s[b])
        assert torch.equal(T.wav2px(w1, s1, p)[0], r[b])


@pytest.mark.gpu
def test_scales_and_non_finite_values(gpu, fresh_plans):
    p = make_parameters(130, 2.0, 6, 3, 0, 0)
    sz = gpu.sizes(p)
    rng = np.random.default_rng(3)
    f = rng.normal(size=sz["n_px"])
    w, s = gpu.px2wav(f, p, real=True)
    r = gpu.wav2px(w, s, p, real=True)
    for k in (-900, 900):
        wk, sk = gpu.px2wav(f * 2.0 ** k, p, real=True)
        assert np.array_equal(wk, w * 2.0 ** k) and np.array_equal(sk, s * 2.0 ** k)
        assert np.array_equal(gpu.wav2px(wk, sk, p, real=True), r * 2.0 ** k)
    z, zs = gpu.px2wav(np.zeros_like(f), p, real=True)
    assert not z.any() and not zs.any()
    # an infinity reaches the outputs that it reaches through the FP64 kernels (a
    # scale without a degree below L stays zero)
    f[1000] = np.inf
    wb, sb = gpu.px2wav(f, p, real=True)
    lib = fresh_plans
    lib.s2let_gpu_release_plans()
    lib.s2let_gpu_set_split_tables(0)
    w64, s64 = gpu.px2wav(f, p, real=True)
    assert np.array_equal(np.isfinite(wb), np.isfinite(w64)) and np.array_equal(np.isfinite(sb), np.isfinite(s64))
    assert not np.isfinite(sb).any() and not np.isfinite(wb).all()
