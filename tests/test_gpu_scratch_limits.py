"""Shared launches hold the spectra of several scales at once; where those do not
fit in device memory a call takes them two at a time, as it always could."""
import ctypes as C

import pytest

from conftest import rel_err
from s2let_gb300.capi import make_parameters
from test_gpu_panel_memory import Pool

TOL = 2e-12  # twice the FP64 path's tolerance


@pytest.mark.gpu
@pytest.mark.parametrize("L,nb,J_min", [(48, 3000, 2), (1000, 4, 6)], ids=["small scales", "parts of a pass"])
def test_fewer_spectra_at_once(gpu, L, nb, J_min):
    torch = pytest.importorskip("torch")
    from s2let_gb300 import torch_ops as T

    lib = gpu.lib
    lib.s2let_gpu_release_plans()
    lib.s2let_gpu_set_split_tables(0)  # nothing else to give back
    p = make_parameters(L, 2.0, J_min, 3, 0, 1)  # full resolution
    f = torch.randn(nb, gpu.sizes(p)["n_px"], dtype=torch.float64, device="cuda")
    pool = Pool()
    try:
        w0, s0 = T.px2wav(f, p)
        r0 = T.wav2px(w0, s0, p)
        nt, scales = L, int(round(gpu.sizes(p)["n_wav"] / (5 * L * (2 * L - 1))))
        one = nb * 2 * nt * (2 * L - 1) * 16  # spectra of a scale: two directions
        assert scales >= 4
        w, s, r = torch.empty_like(w0), torch.empty_like(s0), torch.empty_like(r0)
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)

        def analysis():
            return lib.s2let_gpu_analysis_px2wav_real_batch(C.c_void_p(w.data_ptr()), C.c_void_p(s.data_ptr()),
                                                            C.c_void_p(f.data_ptr()), nb, C.byref(p), st)

        def synthesis():
            return lib.s2let_gpu_synthesis_wav2px_real_batch(C.c_void_p(r.data_ptr()), C.c_void_p(w0.data_ptr()),
                                                             C.c_void_p(s0.data_ptr()), nb, C.byref(p), st)

        for call in (analysis, synthesis):
            torch.cuda.synchronize()
            pool.trim()
            assert call() == 0
            torch.cuda.synchronize()
            scratch = pool.reserved()
            pool.trim()
            torch.cuda.empty_cache()
            free = torch.cuda.mem_get_info()[0]
            block = torch.empty(int(free - scratch + one), dtype=torch.uint8, device="cuda")
            w.zero_(), s.zero_(), r.zero_()
            rc = call()
            torch.cuda.synchronize()
            del block
            torch.cuda.empty_cache()
            assert rc == 0
            if call is analysis:
                assert rel_err(w.cpu(), w0.cpu()) < TOL and rel_err(s.cpu(), s0.cpu()) < TOL
            else:
                assert rel_err(r.cpu(), r0.cpu()) < TOL
    finally:
        lib.s2let_gpu_set_split_tables(1)
        lib.s2let_gpu_release_plans()


@pytest.mark.gpu
def test_a_call_after_one_out_of_memory(gpu):
    """A batch whose first scratch buffer exceeds the device is refused before any
    launch, and leaves nothing behind for the next call or the caller."""
    torch = pytest.importorskip("torch")
    from s2let_gb300 import torch_ops as T

    lib = gpu.lib
    p = make_parameters(48, 2.0, 2, 3, 0, 0)
    f = torch.randn(2, gpu.sizes(p)["n_px"], dtype=torch.float64, device="cuda")
    w0, s0 = T.px2wav(f, p)
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def analysis(nb, w, s):
        return lib.s2let_gpu_analysis_px2wav_real_batch(C.c_void_p(w.data_ptr()), C.c_void_p(s.data_ptr()),
                                                        C.c_void_p(f.data_ptr()), nb, C.byref(p), st)

    w, s = torch.zeros_like(w0), torch.zeros_like(s0)
    assert analysis(20_000_000, w, s) == 4  # 737 GB of coefficients
    torch.cuda.synchronize()
    assert analysis(2, w, s) == 0
    torch.cuda.synchronize()
    assert torch.equal(w, w0) and torch.equal(s, s0)
