"""The process-wide switch between double-float and tensor-core contractions,
turned by one thread while others transform: which scales share launches, and so
which spectra are allocated, is settled once per call."""
import threading

import numpy as np
import pytest

from conftest import rel_err
from s2let_gb300.capi import make_parameters


@pytest.mark.gpu
def test_switch_turned_during_calls(gpu):
    p = make_parameters(128, 2.0, 2, 3, 0, 0)  # scales on both sides of every limit: 8 to 128
    lib = gpu.lib
    f = np.random.default_rng(1).normal(size=gpu.sizes(p)["n_px"])
    w, s = gpu.px2wav(f, p, real=True)
    r = gpu.wav2px(w, s, p, real=True)
    old = lib.s2let_gpu_get_df_max_maps()
    stop, bad = threading.Event(), []

    def turn():
        k = 0
        while not stop.is_set():
            lib.s2let_gpu_set_df_max_maps(k & 1)
            k += 1

    def transform():
        lib.s2let_gpu_set_precision(1)
        for _ in range(150):
            w1, s1 = gpu.px2wav(f, p, real=True)
            r1 = gpu.wav2px(w, s, p, real=True)
            if max(rel_err(w1, w), rel_err(s1, s), rel_err(r1, r)) > 1e-10:  # the bound of both routes
                bad.append(1)

    threads = [threading.Thread(target=transform) for _ in range(3)]
    turner = threading.Thread(target=turn)
    turner.start()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    stop.set()
    turner.join()
    lib.s2let_gpu_set_df_max_maps(old)
    assert not bad
