"""FP32 pixels read and written by the ring kernels (csrc/ring.cu: widen, narrow).

Widening is exact and the outputs are rounded to nearest from the FP64 results,
so every output must equal, bit by bit, the FP64-storage result on the widened
inputs rounded to single precision: for ordinary values, for inputs that are
subnormal as floats, for results that are subnormal or overflow as floats, and
for maps that hold an infinity or a NaN.  N = 12 has more directions than the
fused ring launch takes and goes through widened copies."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")

# L, N, J_min, spin, sampling: every ring route (one slice, slices, fused with the gamma
# DFT, separate), odd and even ring counts, P = 8 up to several butterflies per thread
CASES = [(4, 1, 0, 0, 0), (33, 1, 1, 0, 0), (40, 2, 1, 0, 1), (64, 4, 2, 0, 0), (65, 3, 1, 2, 0), (48, 5, 2, 1, 1), (33, 12, 1, 0, 0),
         (300, 3, 3, 0, 0)]


@pytest.fixture
def ops(gpu):
    from s2let_gb300 import torch_ops

    yield torch_ops
    gpu.lib.s2let_gpu_release_plans()


def _used(gpu, f, p, n):
    """length of the written part of an f_wav row (scales with fewer directions
    than N leave a tail)"""
    w = torch.full((f.shape[0], n["n_wav"]), 7.0, dtype=f.dtype, device="cuda")
    s = torch.empty((f.shape[0], n["n_scal"]), dtype=f.dtype, device="cuda")
    call = getattr(gpu.lib, "s2let_gpu_analysis_px2wav%s_batch" % ("" if f.is_complex() else "_real"))
    vp = lambda t: C.c_void_p(t.data_ptr())
    assert call(vp(w), vp(s), vp(f), f.shape[0], C.byref(p), C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    return int((w != 7.0).any(dim=0).nonzero().max()) + 1


def _same(a32, a64):
    assert a32.dtype in (torch.float32, torch.complex64)
    b = a64.to(a32.dtype)
    x, y = (torch.view_as_real(t.contiguous()) if t.is_complex() else t for t in (a32, b))
    assert torch.equal(torch.isnan(x), torch.isnan(y))
    ok = ~torch.isnan(x)
    assert torch.equal(x[ok], y[ok])


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1.0, 2.0**-138, 2.0**126], ids=["ordinary", "subnormal", "overflow"])
@pytest.mark.parametrize("case", CASES, ids=str)
def test_equals_fp64_storage_rounded(gpu, ops, case, scale):
    L, N, J_min, spin, ss = case
    p = ops.make_parameters(L, 2.0, J_min, N, spin, 0, sampling_scheme=ss)
    g = torch.Generator(device="cuda").manual_seed(L + N)
    n, nb = ops.sizes(p), 3
    d32, d64 = (torch.complex64, torch.complex128) if spin else (torch.float32, torch.float64)
    draw = lambda k: (torch.randn(nb, n[k], dtype=d64, device="cuda", generator=g) * scale).to(d32)
    f, w, s = draw("n_px"), draw("n_wav"), draw("n_scal")
    used = _used(gpu, f.to(d64), p, n)
    f[:, ::5] = 0.0
    if scale == 1.0:
        f[1, 3], f[2, 7] = float("inf"), float("nan")
    for prec in ("fp64", "mixed"):
        out32, out64 = ops.px2wav(f, p, precision=prec), ops.px2wav(f.to(d64), p, precision=prec)
        _same(out32[0][:, :used], out64[0][:, :used])
        _same(out32[1], out64[1])
        _same(ops.wav2px(w, s, p, precision=prec), ops.wav2px(w.to(d64), s.to(d64), p, precision=prec))


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES[1:6], ids=str)
def test_gradients_equal_fp64_storage_rounded(ops, case):
    L, N, J_min, spin, ss = case
    p = ops.make_parameters(L, 2.0, J_min, N, spin, 0, sampling_scheme=ss)
    g = torch.Generator(device="cuda").manual_seed(L)
    n = ops.sizes(p)
    d32, d64 = (torch.complex64, torch.complex128) if spin else (torch.float32, torch.float64)
    f, cw, cs = (torch.randn(2, n[k], dtype=d64, device="cuda", generator=g).to(d32) for k in ("n_px", "n_wav", "n_scal"))
    grads = []
    for d in (d32, d64):
        x = f.to(d).detach().clone().requires_grad_(True)
        w, s = ops.px2wav(x, p)
        torch.autograd.backward([w, s], [cw.to(d), cs.to(d)])
        a, b = (c.to(d).detach().clone().requires_grad_(True) for c in (cw, cs))
        ops.wav2px(a, b, p).backward(f.to(d))
        grads.append((x.grad, b.grad))
    for u, v in zip(*grads):
        _same(u, v)
