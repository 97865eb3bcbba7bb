"""Recomputed tables shared by several problems (csrc/recompute.cu): the scales of
one band-limit and the directions n and -n on one regenerated row, and the
quadrature of up to eight problems per launch.  The sizes cross the kernels'
segments (64 degrees) and ring tiles (128); real and complex signals with n = 0
(both signs of m on one row), +-n, 1 to 5 parts, batches of 1 to 9.  Against the
stored tables the tolerance is the one recomputed tables have had (1e-12
normwise; 1e-11 at split precision)."""
import numpy as np
import pytest

from conftest import rel_err
from s2let_gb300.capi import make_parameters

CASES = [
    # L, N, J_min, spin, upsample, sampling, batch
    (64, 2, 5, 1, 0, 0, 3),    # +-1; one segment at m = 0
    (65, 3, 5, 0, 0, 0, 1),    # n = 0, 2 of a real map, a segment of one degree
    (129, 5, 6, 2, 0, 0, 2),   # n = 0 both ways, +-2, +-4; a ring tile of one ring
    (130, 4, 6, 0, 1, 0, 9),   # real, several scales of one band-limit
    (100, 3, 4, 1, 1, 1, 4),   # complex, MWSS, 4 scales x 2 parts
]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", CASES, ids=str)
def test_parts_against_stored_tables(gpu, case, precision):
    import torch

    from s2let_gb300 import torch_ops as T

    L, N, J_min, spin, up, ss, nb = case
    p = make_parameters(L, 2.0, J_min, N, spin, up, sampling_scheme=ss)
    sz = gpu.sizes(p)
    dt = torch.float64 if spin == 0 else torch.complex128
    gen = torch.Generator(device="cuda").manual_seed(L + N)
    f, w, s = (torch.randn(nb, sz[k], dtype=dt, device="cuda", generator=gen).requires_grad_(True)
               for k in ("n_px", "n_wav", "n_scal"))
    out = {}
    for mode in (1, 2):
        gpu.lib.s2let_gpu_set_table_mode(mode)
        try:
            prec = "mixed" if precision and mode == 2 else "fp64"
            for x in (f, w, s):
                x.grad = None
            gw, gs = T.px2wav(f, p, precision=prec)
            gf = T.wav2px(w, s, p, precision=prec)
            # the backward passes run on autograd's threads, in the automatic table mode
            out[mode] = [gw.detach(), gs.detach(), gf.detach()]
        finally:
            gpu.lib.s2let_gpu_set_table_mode(0)
    for a, b in zip(out[2], out[1]):
        assert rel_err(a.cpu(), b.cpu()) < (1e-11 if precision else 1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
def test_adjoints_against_stored_tables(gpu, precision):
    p = make_parameters(129, 2.0, 6, 5, 2, 0)
    sz = gpu.sizes(p)
    rng = np.random.default_rng(5)
    f, w, s = (rng.normal(size=sz[k]) + 1j * rng.normal(size=sz[k]) for k in ("n_px", "n_wav", "n_scal"))
    out = {}
    for mode in (1, 2):
        gpu.lib.s2let_gpu_set_table_mode(mode)
        gpu.lib.s2let_gpu_set_precision(precision if mode == 2 else 0)
        try:
            out[mode] = [gpu.analysis_adjoint_wav2px(w, s, p), *gpu.synthesis_adjoint_px2wav(f, p)]
        finally:
            gpu.lib.s2let_gpu_set_precision(0)
            gpu.lib.s2let_gpu_set_table_mode(0)
    for a, b in zip(out[2], out[1]):
        assert rel_err(a, b) < (1e-11 if precision else 1e-12)
