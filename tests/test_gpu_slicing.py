"""Coefficient slicing of the tensor-core contractions (csrc/mixed.cu,
k_slice_x): partly filled column sets and the ends of the number range.

The digits, their products and the class sums of a column do not depend on the
other columns, so a map's result is the same in a batch of any size, bit by bit.
(Real rings are transformed in pairs, which straddle maps when a map has an odd
number of rings, as at L = 193: the batches compared start at an even map, so that
every ring keeps its partner.)  Everything else scales by powers of two: a map
times 2^k gives the result times 2^k as long as nothing leaves the normal range.
Near the bottom of it each of the at most L^2 N values that a result sums
is rounded to a multiple of 2^-1074 instead; with maps of order 2^-1000 that is
below 2^-74 L^2 N < 2^-55 of the result's level, against a tolerance of 1e-13."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")


@pytest.fixture
def ops(gpu):
    from s2let_gb300 import torch_ops

    gpu.lib.s2let_gpu_release_plans()
    yield torch_ops
    gpu.lib.s2let_gpu_release_plans()


def _maps(T, p, nb, spin, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = torch.complex128 if spin else torch.float64
    return torch.randn(nb, T.sizes(p)["n_px"], dtype=dt, device="cuda", generator=g)


# band-limits at the edges of the 64-wide K chunks and 128-row tiles; batches that
# leave columns of the 16, 32 and 64 wide shapes without a map
@pytest.mark.gpu
@pytest.mark.parametrize("L,N,spin,precision", [(128, 2, 0, "fp64"), (129, 3, 1, "fp64"), (193, 2, 0, "mixed"), (128, 3, 2, "mixed")])
@pytest.mark.parametrize("nb", [3, 9, 17])
def test_batch_size_does_not_change_a_map(ops, L, N, spin, precision, nb):
    p = ops.make_parameters(L, 2.0, 5, N, spin, 0)
    f = _maps(ops, p, nb, spin, L + nb)
    w, s = ops.px2wav(f, p, precision=precision)
    r = ops.wav2px(w, s, p, precision=precision)
    for lo, hi, b in ((0, 2, 0), (nb - 3, nb, nb - 1)):
        w2, s2 = ops.px2wav(f[lo:hi], p, precision=precision)
        r2 = ops.wav2px(w2, s2, p, precision=precision)
        i = b - lo
        assert torch.equal(w2[i], w[b]) and torch.equal(s2[i], s[b]) and torch.equal(r2[i], r[b])


@pytest.mark.gpu
@pytest.mark.parametrize("L,N,spin", [(128, 2, 0), (150, 3, 2)])
@pytest.mark.parametrize("k", [-1000, -600, 600, 900])
def test_powers_of_two(ops, L, N, spin, k):
    p = ops.make_parameters(L, 2.0, 5, N, spin, 0)
    f = _maps(ops, p, 2, spin, L)
    f[:, ::7] = 0.0  # zeros take the weight product's other branch
    w, s = ops.px2wav(f, p)
    wk, sk = ops.px2wav(f * 2.0**k, p)
    for x, xk in ((w, wk), (s, sk)):
        y = xk * 2.0**-(k // 2) * 2.0**-(k - k // 2)  # in two steps: 2^1000 alone times a subnormal stays exact
        if k == -1000:
            assert torch.isfinite(torch.view_as_real(y) if y.is_complex() else y).all()
            assert float((y - x).abs().max()) <= 1e-13 * float(x.abs().max())
        else:
            assert torch.equal(y, x)
