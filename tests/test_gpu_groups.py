"""Launches shared by several scales (csrc/exec.cu, kernels.cu, ring.cu): the
contractions and ring DFTs of the small band-limits in one launch each, up to
eight scales of one band-limit in one table pass, and ring DFTs that read the
spectra of a one-slice scale directly.  Every map of a batch against the oracle
(1e-12 normwise, the FP64 path's tolerance; 1e-10 at split precision)."""
import numpy as np
import pytest

from conftest import rel_err
from s2let_gb300.capi import make_parameters

CASES = [
    # L, N, J_min, spin, real, upsample, batch
    (70, 3, 1, 0, True, 1, 1),    # 7 scales of one band-limit: one pass of 7 parts
    (70, 2, 0, 0, True, 1, 3),    # 8 parts; one component per ring and scale (no cluster)
    (66, 1, 1, 1, False, 1, 5),   # one slice per scale, 6 parts per pass
    (64, 3, 1, 0, True, 1, 12),   # 2 parts per pass, an odd number of scales
    (40, 5, 2, 2, False, 0, 4),   # every scale small, 5 components
    (40, 1, 0, 0, True, 0, 3),    # one slice per scale, small
    (130, 4, 1, 0, True, 0, 3),   # small scales beside large ones
    (33, 9, 3, 0, False, 0, 2),   # 9 components: ring and gamma DFTs apart
]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", CASES, ids=str)
def test_shared_launches(gpu, oracle_port, case, precision):
    import torch

    from s2let_gb300 import torch_ops as T

    L, N, J_min, spin, real, up, nb = case
    p = make_parameters(L, 2.0, J_min, N, spin, up)
    sz = gpu.sizes(p)
    rng = np.random.default_rng(10 * L + N)
    draw = lambda n: rng.normal(size=(nb, n)) + (0 if real else 1j * rng.normal(size=(nb, n)))
    f, w, s = draw(sz["n_px"]), draw(sz["n_wav"]), draw(sz["n_scal"])
    dev = lambda a: torch.from_numpy(a).cuda().requires_grad_(True)
    prec = "mixed" if precision else "fp64"
    tol = 1e-10 if precision else 1e-12
    fd, wd, sd = dev(f), dev(w), dev(s)
    gw, gs = T.px2wav(fd, p, precision=prec)
    gf = T.wav2px(wd, sd, p, precision=prec)
    torch.autograd.backward([gw, gs], [wd.detach(), sd.detach()])
    gf.backward(fd.detach())
    # rows past the used length (N_j may fall short of N) are not written by the transforms
    for b in range(nb):
        ow, os_ = oracle_port.px2wav(f[b], p, real=real)
        nz = np.flatnonzero(ow)[-1] + 1
        assert rel_err(gw[b, :nz].detach().cpu(), ow[:nz]) < tol
        assert rel_err(gs[b].detach().cpu(), os_) < tol
        assert rel_err(gf[b].detach().cpu(), oracle_port.wav2px(w[b], s[b], p, real=real)) < tol
        assert rel_err(fd.grad[b].cpu(), oracle_port.analysis_adjoint_wav2px(w[b], s[b], p, real=real)) < tol
        aw, as_ = oracle_port.synthesis_adjoint_px2wav(f[b], p, real=real)
        nz = np.flatnonzero(aw)[-1] + 1
        assert rel_err(wd.grad[b, :nz].cpu(), aw[:nz]) < tol
        assert rel_err(sd.grad[b].cpu(), as_) < tol


@pytest.mark.gpu
@pytest.mark.parametrize("N", [1, 3])
def test_host_batches_with_small_scales(gpu, oracle_port, N):
    """The copy pipeline takes the large scales first and the shared launches of
    the small ones last."""
    from s2let_gb300.capi import ptr
    import ctypes as C

    p = make_parameters(72, 2.0, 1, N, 0, 0)
    sz = gpu.sizes(p)
    nb = 9
    rng = np.random.default_rng(N)
    f = rng.normal(size=(nb, sz["n_px"]))
    w, s, r = np.zeros((nb, sz["n_wav"])), np.zeros((nb, sz["n_scal"])), np.zeros_like(f)
    assert gpu.lib.s2let_gpu_analysis_px2wav_real_host_batch(ptr(w), ptr(s), ptr(f), nb, C.byref(p)) == 0
    assert gpu.lib.s2let_gpu_synthesis_wav2px_real_host_batch(ptr(r), ptr(w), ptr(s), nb, C.byref(p)) == 0
    for b in range(nb):
        ow, os_ = oracle_port.px2wav(f[b], p, real=True)
        assert rel_err(w[b], ow) < 1e-12 and rel_err(s[b], os_) < 1e-12
        assert rel_err(r[b], oracle_port.wav2px(ow, os_, p, real=True)) < 1e-12
