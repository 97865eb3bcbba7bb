"""The work that users of this framework have it do, as timed cases.

Every case goes through a public entry point: the PyTorch operators on batches
in device memory, the drop-in host calls on NumPy arrays, and the multi-map
call with one parameter set per map.  ``prepare`` makes the inputs from the
seed, ``run`` is one pass, ``exact`` is the same pass in plain torch in 64 bits
(half-angle Wigner recursion, FFTs and the sampling's exact quadrature).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from s2let_gb300 import _lib
from s2let_gb300 import api as numpy_api
from s2let_gb300 import torch_ops as T
from s2let_gb300.capi import S2letParameters, make_parameters

LAMBDA = 0.05  # sparsity weight of the differentiable loss
THRESHOLD = 0.02  # soft threshold of its wavelet coefficients


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(kind, L, N, J_min, spin=0, upsample=0, mwss=0, batch=1, mixed=0, single=0):
    return dict(kind=kind, L=L, N=N, J_min=J_min, spin=spin, upsample=upsample, mwss=mwss, batch=batch,
                mixed=mixed, single=single)


def listed():
    return [
        # a drop-in call on a small map: latency and launches are all there is
        dict(name="host_small", **_case("host", 32, 3, 1)),
        # the axisymmetric transform of one scalar map, full resolution, host buffers
        dict(name="host_axisym", **_case("axisym", 128, 1, 0, upsample=1)),
        # upsampled wavelets (every scale at L) of a few maps on the device
        dict(name="upsampled", **_case("device", 96, 3, 2, upsample=1, batch=4)),
        # complex spin-1 maps on the symmetric sampling at an odd band-limit
        dict(name="mwss_odd", **_case("device", 181, 2, 1, spin=1, mwss=1, batch=3, mixed=1)),
        # a batch of polarisation maps in FP64, the default precision
        dict(name="spin2_fp64", **_case("device", 256, 3, 2, spin=2, batch=8)),
        # one map at a time in FP64, analysis and synthesis
        dict(name="map_fp64", **_case("device", 512, 4, 2, batch=1)),
        # harmonic input and output through the drop-in calls, split precision
        dict(name="host_harmonic", **_case("harmonic", 384, 4, 2, mixed=1)),
        # training step of a wavelet-sparsity loss: forward and backward, FP32 storage
        dict(name="sparsity_step", **_case("loss", 256, 4, 2, batch=32, mixed=1, single=1)),
        # maps that all have their own band-limit, N and spin, in one graph-replayed call
        dict(name="uneven_maps", **_case("uneven", 320, 5, 1, batch=32, mixed=1, single=1)),
        # polarisation maps with five directions, split precision
        dict(name="spin2_mixed", **_case("device", 512, 5, 3, spin=2, batch=4, mixed=1)),
        # full-resolution sky maps in FP64
        dict(name="large_fp64", **_case("device", 1024, 4, 2, batch=2)),
        # a serving batch of full-resolution sky maps, split precision
        dict(name="large_batch", **_case("device", 1024, 4, 2, batch=32, mixed=1)),
    ]


def _log_int(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["host", "axisym", "device", "device", "device", "device", "harmonic", "loss", "uneven"])
    mixed = rng.randint(0, 1)
    J_min = rng.randint(1, 3)
    N = rng.randint(1, min(5, 2 ** J_min + 1))
    if kind == "host":
        return _case(kind, _log_int(rng, 16, 160), N, J_min, mwss=rng.randint(0, 1), mixed=mixed)
    if kind == "axisym":
        return _case(kind, _log_int(rng, 32, 320), 1, rng.randint(0, 2), upsample=rng.randint(0, 1), mixed=mixed)
    if kind == "harmonic":
        return _case(kind, _log_int(rng, 48, 512), N, J_min, mixed=mixed)
    if kind == "loss":
        L = _log_int(rng, 48, 320)
        return _case(kind, L, N, J_min, batch=_log_int(rng, 1, 32), mixed=mixed, single=rng.randint(0, 1))
    if kind == "uneven":
        return _case(kind, _log_int(rng, 96, 320), 5, 1, batch=_log_int(rng, 6, 32), mixed=mixed, single=1)
    L = _log_int(rng, 48, 768)
    most = max(1, min(32, int(32 * (400.0 / L) ** 2)))  # keeps a pass below the largest listed one's
    return _case(kind, L, N, J_min, spin=rng.choice([0, 0, 1, 2]), upsample=int(L <= 128 and rng.random() < 0.3),
                 mwss=int(rng.random() < 0.25), batch=_log_int(rng, 1, most), mixed=mixed,
                 single=int(rng.random() < 0.25))


def _parameters(c):
    return make_parameters(c["L"], 2.0, c["J_min"], c["N"], c["spin"], c["upsample"],
                           sampling_scheme=c["mwss"])


def _uneven(c):
    """(L, N, spin) of the maps of an uneven case: L log-uniform on [64, c.L]
    and even, N in {1, 3, 5}, spin in {0, 2}.  The sizes belong to the case,
    the maps to the seed."""
    rng = np.random.default_rng(1000 * c["L"] + c["batch"])
    out = []
    for _ in range(c["batch"]):
        L = int(2 * round(math.exp(rng.uniform(math.log(64), math.log(c["L"]))) / 2))
        out.append((L, int(rng.choice([1, 3, 5])), int(rng.choice([0, 2]))))
    return out


# ---------------------------------------------------------------------------
# geometry of the reference's layouts
# ---------------------------------------------------------------------------
def _rings(bl, ss):
    return bl + 1 if ss else bl


def _ring_len(bl, ss):
    return 2 * bl if ss else 2 * bl - 1


def _n_px(L, ss):
    return _rings(L, ss) * _ring_len(L, ss)


def _j_max(L):
    return int(math.ceil(math.log(L) / math.log(2.0)))


def _scales(c):
    """[(j, band-limit, N_j)] of the wavelet scales and the scaling band-limit."""
    L, N = c["L"], c["N"]
    out = []
    for j in range(c["J_min"], _j_max(L) + 1):
        bl, nj = L, N
        if not c["upsample"]:
            bl = min(2 ** (j + 1), L)
            nj = min(N, bl)
            nj += (nj + N) % 2
        out.append((j, bl, nj))
    return out, (L if c["upsample"] else min(2 ** c["J_min"], L))


def work(c):
    """Inputs read and outputs written once; 4 flops per complex-by-real
    multiply-add of the transforms' Legendre sums, the fewest a separable
    transform on these grids does per pass."""
    if c["kind"] == "uneven":
        total = {"bytes": 0.0, "flops": 0.0}
        for L, N, spin in _uneven(c):
            one = work(_case("device", L, N, c["J_min"], spin=spin, single=c["single"]))
            total = {k: total[k] + one[k] for k in total}
        return total
    scales, bs = _scales(c)
    ss, L = c["mwss"], c["L"]
    real = c["spin"] == 0

    def sht(bl, n, both):
        ms = range(-(bl - 1), bl) if both else range(0, bl)
        return 4.0 * _rings(bl, ss) * sum(max(0, bl - max(abs(m), n)) for m in ms)

    flops = sht(bs, 0, not real) + (sht(L, abs(c["spin"]), not real) if c["kind"] != "harmonic" else 0.0)
    wav = 0
    for _, bl, nj in scales:
        wav += (2 * nj - 1) * _n_px(bl, ss)
        for n in range(-nj + 1, nj, 2):
            if not real or n >= 0:
                flops += sht(bl, abs(n), not real or n != 0)
    esz = (8 if real else 16) // (2 if c["single"] else 1)
    px, coef = esz * _n_px(L, ss), esz * (wav + _n_px(bs, ss))
    if c["kind"] == "loss":  # two transforms forward and their two adjoints; maps, targets and gradients
        return {"bytes": float(c["batch"] * 3 * px), "flops": 4.0 * c["batch"] * flops}
    ends = 2 * 16 * L * L if c["kind"] == "harmonic" else 2 * px
    return {"bytes": float(c["batch"] * (ends + coef)), "flops": 2.0 * c["batch"] * flops}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _maps(gen, L, ss, spin, batch, dev):
    """Smooth random maps with white noise: 16 plane waves per map with wave
    numbers log-uniform up to L/2 and amplitudes falling with them, sampled on
    the sphere, plus Gaussian noise of a tenth of their size."""
    nt, K = _rings(L, ss), _ring_len(L, ss)
    t = torch.arange(nt, dtype=torch.float64, device=dev)
    theta = math.pi * t / L if ss else math.pi * (2 * t + 1) / K
    phi = 2 * math.pi * torch.arange(K, dtype=torch.float64, device=dev) / K
    x = torch.outer(torch.sin(theta), torch.cos(phi)).reshape(-1)
    y = torch.outer(torch.sin(theta), torch.sin(phi)).reshape(-1)
    z = torch.cos(theta)[:, None].expand(nt, K).reshape(-1)
    xyz = torch.stack([x, y, z])
    out = torch.empty(batch, nt * K, dtype=torch.float64 if spin == 0 else torch.complex128, device=dev)
    for b in range(batch):
        parts = []
        for _ in range(1 if spin == 0 else 2):
            u = torch.rand(16, generator=gen, dtype=torch.float64, device=dev)
            q = torch.randn(16, 3, generator=gen, dtype=torch.float64, device=dev)
            ph = 2 * math.pi * torch.rand(16, generator=gen, dtype=torch.float64, device=dev)
            k = torch.exp(u * math.log(max(L / 2.0, 2.0)))
            q = q / q.norm(dim=1, keepdim=True) * k[:, None]
            f = torch.zeros(nt * K, dtype=torch.float64, device=dev)
            for w in range(16):  # one wave at a time: no (waves x pixels) array
                f += torch.cos(torch.mv(xyz.T, q[w]) + ph[w]) / torch.sqrt(k[w])
            f += 0.1 * torch.randn(nt * K, generator=gen, dtype=torch.float64, device=dev)
            parts.append(f)
        out[b] = parts[0] if spin == 0 else torch.complex(parts[0], parts[1])
    return out


def _real_flm(rng, L):
    """Gaussian flm of a real map with C_l = (l+1)^-2 and f_00 = 0."""
    l = np.repeat(np.arange(L), 2 * np.arange(L) + 1)
    m = np.arange(L * L) - l * l - l
    f = (rng.normal(size=L * L) + 1j * rng.normal(size=L * L)) / (l + 1.0) / np.sqrt(2.0)
    f[m == 0] = f[m == 0].real * np.sqrt(2.0)
    neg = m < 0
    f[neg] = np.where(m[neg] % 2 == 0, 1.0, -1.0) * np.conj(f[(l * l + l - m)[neg]])
    f[0] = 0.0
    return f


def _inputs(c, seed):
    """What the user holds, by name, made from the seed alone."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    single = torch.float32 if c["spin"] == 0 else torch.complex64
    if c["kind"] == "harmonic":
        return {"flm": _real_flm(np.random.default_rng(int(seed)), c["L"])}
    if c["kind"] == "uneven":
        return {"maps": [_maps(gen, L, 0, s, 1, dev)[0].to(torch.float32 if s == 0 else torch.complex64)
                         for L, _, s in _uneven(c)]}
    f = _maps(gen, c["L"], c["mwss"], c["spin"], c["batch"], dev)
    if c["kind"] == "loss":
        x = f + 0.1 * torch.randn(f.shape, generator=gen, dtype=torch.float64, device=dev)
        return {"x": x.to(single) if c["single"] else x, "y": f.to(single) if c["single"] else f}
    if c["kind"] in ("host", "axisym"):
        return {"f": f[0].cpu().numpy()}
    return {"f": f.to(single) if c["single"] else f}


_plans_of = [None]


def prepare(c, seed):
    lib = _lib.load()
    if _plans_of[0] not in (None, c):  # another program's plans do not stay beside this one's
        lib.s2let_gpu_release_plans()
    _plans_of[0] = dict(c)
    state = dict(c=c, lib=lib, precision="mixed" if c["mixed"] else "fp64")
    given = _inputs(c, seed)
    if c["kind"] != "uneven":
        state["p"] = _parameters(c)
        state.update(given)
        return state
    maps, n = given["maps"], c["batch"]
    params, real = (S2letParameters * n)(), (C.c_int * n)()
    wav, scal = [], []
    for k, (L, N, spin) in enumerate(_uneven(c)):
        params[k] = make_parameters(L, 2.0, c["J_min"], N, spin, 0)
        real[k] = int(spin == 0)
        one = _case("device", L, N, c["J_min"], spin=spin)
        scales, bs = _scales(one)
        wav.append(sum((2 * nj - 1) * _n_px(bl, 0) for _, bl, nj in scales))
        scal.append(_n_px(bs, 0))
    width = [1 if r else 2 for r in real]
    dev = maps[0].device

    def buffers(sizes):
        flat = torch.zeros(sum(w * s for w, s in zip(width, sizes)), dtype=torch.float32, device=dev)
        at, ptrs = 0, (C.c_void_p * n)()
        for k in range(n):
            ptrs[k] = flat.data_ptr() + 4 * at
            at += width[k] * sizes[k]
        return flat, ptrs

    state.update(n=n, params=params, real=real, maps=maps, stream=torch.cuda.Stream(dev),
                 px=(C.c_void_p * n)(*[f.data_ptr() for f in maps]))
    state["wav"], state["wav_ptr"] = buffers(wav)
    state["scal"], state["scal_ptr"] = buffers(scal)
    state["rec"], state["rec_ptr"] = buffers([f.numel() for f in maps])
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    c = state["c"]
    return globals()["_run_" + c["kind"]](state)


def _run_device(s):
    w, sc = T.px2wav(s["f"], s["p"], precision=s["precision"])
    return w, sc, T.wav2px(w, sc, s["p"], precision=s["precision"])


def _run_loss(s):
    x = s["x"].detach().requires_grad_(True)
    w, sc = T.px2wav(x, s["p"], precision=s["precision"])
    kept = torch.sign(w) * torch.clamp(w.abs() - THRESHOLD, min=0)
    r = T.wav2px(kept, sc, s["p"], precision=s["precision"]) - s["y"]
    loss = 0.5 * r.square().sum() + LAMBDA * w.abs().sum()
    loss.backward()
    return loss.detach(), x.grad


def _host_mode(s):
    s["lib"].s2let_gpu_set_precision(s["c"]["mixed"])
    return numpy_api()


def _run_host(s):
    a = _host_mode(s)
    w, sc = a.px2wav(s["f"], s["p"], real=True)
    return w, sc, a.wav2px(w, sc, s["p"], real=True)


def _run_axisym(s):
    a = _host_mode(s)
    multires = not s["c"]["upsample"]
    w, sc = a.axisym("analysis", [s["f"]], s["p"], multires=multires, real=True)
    return w, sc, a.axisym("synthesis", [w, sc], s["p"], multires=multires, real=True)


def _run_harmonic(s):
    a = _host_mode(s)
    w, sc = a.lm2wav(s["flm"], s["p"], real=True)
    return w, sc, a.wav2lm(w, sc, s["p"], real=True)


def _run_uneven(s):
    lib, st = s["lib"], C.c_void_p(s["stream"].cuda_stream)
    s["stream"].wait_stream(torch.cuda.current_stream())
    lib.s2let_gpu_set_precision(s["c"]["mixed"])
    lib.s2let_gpu_set_table_mode(2)  # no stored tables: every map has its own
    rc = lib.s2let_gpu_px2wav_multi_f32(s["wav_ptr"], s["scal_ptr"], s["px"], s["params"], s["real"], s["n"], 1, st)
    rc |= lib.s2let_gpu_wav2px_multi_f32(s["rec_ptr"], s["wav_ptr"], s["scal_ptr"], s["params"], s["real"], s["n"],
                                         1, st)
    lib.s2let_gpu_set_table_mode(0)
    torch.cuda.current_stream().wait_stream(s["stream"])
    if rc:
        raise RuntimeError(lib.s2let_gpu_last_error_string().decode())
    return s["wav"], s["scal"], s["rec"]


# ---------------------------------------------------------------------------
# the same in plain torch, in 64 bits
# ---------------------------------------------------------------------------
def _quarter_turns(L, dev):
    """Delta^l = d^l(pi/2), l = 0 .. L-1, as (2l+1, 2l+1) tensors indexed
    (m' + l, m + l): d^j built from d^{j-1/2} and a spin one half (Risbo 1996)."""
    h = math.sqrt(0.5)
    d = torch.ones(1, 1, dtype=torch.float64, device=dev)
    yield d
    for l in range(1, L):
        for twoj in (2 * l - 1, 2 * l):
            up = torch.sqrt(torch.arange(1, twoj + 1, dtype=torch.float64, device=dev))
            dn = torch.flip(up, [0])
            e = d * (h / twoj)
            d = torch.zeros(twoj + 1, twoj + 1, dtype=torch.float64, device=dev)
            d[1:, 1:] += up[:, None] * up[None, :] * e
            d[1:, :-1] -= up[:, None] * dn[None, :] * e
            d[:-1, 1:] += dn[:, None] * up[None, :] * e
            d[:-1, :-1] += dn[:, None] * dn[None, :] * e
        yield d


class _Grid:
    """theta rings of one band-limit: cos / sin of m theta, and the quadrature."""

    def __init__(self, bl, ss, dev):
        self.bl, self.ss, self.nt, self.K = bl, ss, _rings(bl, ss), _ring_len(bl, ss)
        t = torch.arange(self.nt, dtype=torch.int64, device=dev)
        m = torch.arange(bl, dtype=torch.int64, device=dev)
        half = bl if ss else self.K  # theta = pi * a / half
        a = t if ss else 2 * t + 1
        ang = (torch.outer(a, m) % (2 * half)).double() * (math.pi / half)
        two = torch.where(m > 0, 2.0, 1.0).double()
        self.cos, self.sin = torch.cos(ang) * two, torch.sin(ang) * two
        self._w, self._a, self._half, self._dev = {}, a, half, dev

    def quadrature(self, eps):
        """W[t][t']: extension of a ring function to the full circle with
        parity eps, Fourier transform, convolution with the transform of
        sin(theta) on [0, pi], and folding back."""
        if eps not in self._w:
            bl, dev = self.bl, self._dev
            m = torch.arange(-(bl - 1), bl, dtype=torch.int64, device=dev)
            ang = (torch.outer(m, self._a) % (2 * self._half)).double() * (math.pi / self._half)
            e = torch.complex(torch.cos(ang), -torch.sin(ang))
            t = torch.arange(self.nt, device=dev)
            mirrored = ((t >= 1) & (t <= bl - 1)) if self.ss else (t < bl - 1)
            A = e + eps * e.conj() * mirrored.double()
            p = m[:, None] + m[None, :]
            pd = p.double()
            even = torch.where(p % 2 == 0, 2.0 / (1.0 - pd * pd), torch.zeros_like(pd))
            odd = ((p == 1).double() - (p == -1).double()) * (0.5 * math.pi)
            kt = float(2 * bl if self.ss else self.K)
            self._w[eps] = (A.T @ (torch.complex(even, odd) @ A)).real / kt ** 2
        return self._w[eps]

    def weigh(self, spec, n, transpose=False):
        """The quadrature on ring spectra (batch, t, m), parity (-1)^(m+n)."""
        out = torch.empty_like(spec)
        for eps in (1, -1):
            W = self.quadrature(eps)
            W = W.T if transpose else W
            m0 = (self.bl - 1 + n + (0 if eps == 1 else 1)) % 2  # column of m = -(bl-1): parity bl-1
            part = spec[:, :, m0::2]
            out[:, :, m0::2] = torch.complex(W @ part.real.contiguous(), W @ part.imag.contiguous())
        return out


def _wigner(delta, l, n, g):
    """d^l_{m,n}(theta_t), n >= 0, m = -l..l, as (t, m): i^(m-n) sum_k Delta_km Delta_kn e^(-ik theta)."""
    prod = delta[l:] * delta[l:, l + n][:, None]  # k = 0..l
    d = torch.empty(g.nt, 2 * l + 1, dtype=torch.float64, device=delta.device)
    for r in range(4):
        at = (n + r + l) % 4  # columns with m - n = r (mod 4)
        if at < 2 * l + 1:
            table = g.cos if r % 2 == 0 else g.sin
            part = table[:, :l + 1] @ prod[:, at::4].contiguous()
            d[:, at::4] = part if r < 2 else -part
    return d


class _Plan:
    """One tiling on one sampling: the operators of the transforms and their adjoints."""

    def __init__(self, c, dev):
        self.c, self.dev, self.L, self.ss, self.s = c, dev, c["L"], c["mwss"], c["spin"]
        self.real = c["spin"] == 0
        self.axisym = c["kind"] == "axisym"
        self.scales, self.bs = _scales(c)
        self.grids = {}
        kappa, kappa0 = self._profiles()
        l = np.arange(self.L)
        low = l >= abs(self.s)
        self.phi = np.sqrt((2 * l + 1) / (4 * np.pi)) * kappa0 * low
        self.cl = (-1.0) ** self.s * np.sqrt((2 * l + 1) / (4 * np.pi)) * low
        self.bands = []  # per scale: (bl, ng, {n: weight over l})
        for j, bl, nj in self.scales:
            if self.axisym:
                self.bands.append((bl, 1, {0: (np.sqrt((2 * l + 1) / (4 * np.pi)) * kappa[j]).astype(complex)}))
                continue
            w = {n: np.sqrt((2 * l + 1) / (8 * np.pi ** 2)) * kappa[j] * low * self._direction(n)
                 for n in range(-nj + 1, nj, 2)}
            self.bands.append((bl, 2 * nj - 1, w))

    def _profiles(self):
        """Scale-discretised wavelet generating functions (B = 2): 300-panel
        trapezoid rule, as the transform is defined."""
        B, L, J = 2.0, self.L, _j_max(self.L)

        def f(k):
            t = (k - (1 / B)) * (2.0 * B / (B - 1)) - 1
            d = 1.0 - t * t
            if d == 0.0:
                return 0.0
            return math.exp(-2.0 / d) / k if d > 0 else math.inf

        def integral(a):
            # summed in the order of the definition: the finest scales' profiles
            # are differences of nearly equal values
            if a == 1.0:
                return 0.0
            h, total, f1 = (1.0 - a) / 300, 0.0, f(a)
            for i in range(300):
                f2 = f(a + (i + 1) * h)
                if math.isfinite(f1) and math.isfinite(f2):
                    total += ((f1 + f2) * h) / 2
                f1 = f2
            return total

        norm = integral(1 / B)
        phi2 = np.zeros((J + 2, L))
        for j in range(J + 2):
            for l in range(L):
                phi2[j, l] = 1.0 if l < B ** (j - 1) else 0.0 if l > B ** j else integral(l / B ** j) / norm
        kappa = {}
        for j in range(self.c["J_min"], J + 1):
            with np.errstate(invalid="ignore"):
                t = np.sqrt(phi2[j + 1] - phi2[j])
            # where rounding makes a difference negative, the value before it stands
            k = np.where(np.isfinite(t), t, np.concatenate([[0.0], t[:-1]]))
            for l in range(1, L):
                if not np.isfinite(k[l]):
                    k[l] = k[l - 1]
            kappa[j] = k
        return kappa, np.sqrt(phi2[self.c["J_min"]])

    def _direction(self, n):
        N, out = self.c["N"], np.zeros(self.L, complex)
        for l in range(1, self.L):
            if abs(n) > l or abs(n) >= N or (N + n) % 2 == 0:
                continue
            g = min(N - 1, l) if (N + l) % 2 else min(N - 1, l - 1)
            k = (g - n) // 2
            if 0 <= k <= g:
                out[l] = (1.0 if N % 2 else 1j) * math.sqrt(math.comb(g, k) / 2.0 ** g)
        return out

    def grid(self, bl):
        if bl not in self.grids:
            self.grids[bl] = _Grid(bl, self.ss, self.dev)
        return self.grids[bl]

    # sums over l, and over theta ----------------------------------------------------------
    def _to_rings(self, tasks, flm):
        """[(bl, n, weight)] -> ring spectra (batch, t, m) of sum_l w(l) d^l_mn flm."""
        out = []
        for bl, n, w in tasks:
            g = self.grid(bl)
            out.append(torch.zeros(flm.shape[0], g.nt, 2 * bl - 1, dtype=torch.complex128, device=self.dev))
        for l, delta in enumerate(_quarter_turns(self.L, self.dev)):
            known = {}
            for k, (bl, n, w) in enumerate(tasks):
                if l >= bl or abs(n) > l or w[l] == 0:
                    continue
                if (bl, abs(n)) not in known:
                    known[bl, abs(n)] = _wigner(delta, l, abs(n), self.grid(bl))
                d = known[bl, abs(n)]
                x = flm[:, l * l:(l + 1) ** 2] * complex(w[l])
                if n < 0:  # d_{m,-n} = (-1)^(m+n) d_{-m,n}
                    m = torch.arange(-l, l + 1, device=self.dev)
                    d = torch.flip(d, [1])
                    x = x * torch.where((m + n) % 2 == 0, 1.0, -1.0)
                out[k][:, :, bl - 1 - l:bl + l] += x[:, None, :] * d[None]
        return out

    def _to_lm(self, tasks, rings, nb):
        """[(bl, n, weight)] and their ring spectra -> sum of w(l) sum_t d^l_mn spec."""
        flm = torch.zeros(nb, self.L * self.L, dtype=torch.complex128, device=self.dev)
        for l, delta in enumerate(_quarter_turns(self.L, self.dev)):
            known = {}
            for (bl, n, w), spec in zip(tasks, rings):
                if l >= bl or abs(n) > l or w[l] == 0:
                    continue
                if (bl, abs(n)) not in known:
                    known[bl, abs(n)] = _wigner(delta, l, abs(n), self.grid(bl))
                d = known[bl, abs(n)]
                if n < 0:
                    m = torch.arange(-l, l + 1, device=self.dev)
                    d = torch.flip(d, [1]) * torch.where((m + n) % 2 == 0, 1.0, -1.0)
                y = (spec[:, :, bl - 1 - l:bl + l] * d[None]).sum(1)
                flm[:, l * l:(l + 1) ** 2] += complex(w[l]) * y
        return flm

    # rings ----------------------------------------------------------------------------------
    def _spectra(self, f, bl):
        """(..., t, p) -> (..., t, m), m = -(bl-1)..bl-1."""
        s = torch.fft.fft(f.to(torch.complex128), dim=-1)
        return torch.cat([s[..., s.shape[-1] - (bl - 1):], s[..., :bl]], -1)

    def _pixels(self, spec, bl):
        K = _ring_len(bl, self.ss)
        s = torch.zeros(*spec.shape[:-1], K, dtype=torch.complex128, device=self.dev)
        s[..., :bl] = spec[..., bl - 1:]
        if bl > 1:
            s[..., K - (bl - 1):] = spec[..., :bl - 1]
        f = torch.fft.ifft(s, dim=-1) * K
        return f.real if self.real else f

    # spherical-harmonic transform at L --------------------------------------------------------
    def sht(self, f, adjoint_of_inverse=False):
        g = self.grid(self.L)
        spec = self._spectra(f.reshape(f.shape[0], g.nt, g.K), self.L)
        c = self.cl.astype(complex)
        if not adjoint_of_inverse:
            spec, c = g.weigh(spec, self.s), c * (2 * math.pi / g.K)
        return self._to_lm([(self.L, -self.s, c)], [spec], f.shape[0])

    def isht(self, flm, adjoint_of_forward=False):
        g = self.grid(self.L)
        c = self.cl * (2 * math.pi / g.K if adjoint_of_forward else 1.0)
        spec = self._to_rings([(self.L, -self.s, c.astype(complex))], flm)[0]
        if adjoint_of_forward:
            spec = g.weigh(spec, self.s, transpose=True)
        return self._pixels(spec, self.L).reshape(flm.shape[0], -1)

    # harmonic <-> wavelet -----------------------------------------------------------------------
    def split(self, flm, adjoint_of_merge=False):
        adj = adjoint_of_merge
        c = 2 * math.pi / _ring_len(self.bs, self.ss) if adj else 1.0
        tasks = [(self.bs, 0, (self.phi * c).astype(complex))]
        for bl, ng, w in self.bands:
            K = _ring_len(bl, self.ss)
            if self.axisym:
                c = 2 * math.pi / K * math.sqrt(2 * math.pi) if adj else 1 / math.sqrt(2 * math.pi)
            else:
                c = 4 * math.pi ** 2 / K / ng if adj else 1.0
            tasks += [(bl, n, np.conj(w[n]) * c) for n in w]
        rings = self._to_rings(tasks, flm)
        if adj:
            rings = [self.grid(bl).weigh(r, n, transpose=True) for (bl, n, _), r in zip(tasks, rings)]
        nb = flm.shape[0]
        scal = self._pixels(rings.pop(0), self.bs).reshape(nb, -1)
        wav = []
        for bl, ng, w in self.bands:
            G = [rings.pop(0) for _ in w]
            for k in range(ng):
                e = [complex(np.exp(2j * np.pi * ((n * k) % ng) / ng)) for n in w]
                wav.append(self._pixels(sum(a * b for a, b in zip(e, G)), bl).reshape(nb, -1))
        return torch.cat(wav, 1), scal

    def merge(self, wav, scal, adjoint_of_split=False):
        adj, nb = adjoint_of_split, wav.shape[0]
        g = self.grid(self.bs)
        spec = self._spectra(scal.reshape(nb, g.nt, g.K), self.bs)
        tasks = [(self.bs, 0, (self.phi * (1.0 if adj else 2 * math.pi / g.K)).astype(complex))]
        rings, at = [spec if adj else g.weigh(spec, 0)], 0
        for bl, ng, w in self.bands:
            g = self.grid(bl)
            size = ng * g.nt * g.K
            f = self._spectra(wav[:, at:at + size].reshape(nb, ng, g.nt, g.K), bl)
            at += size
            if self.axisym:
                c = 1 / math.sqrt(2 * math.pi) if adj else 2 * math.pi / g.K * math.sqrt(2 * math.pi)
            else:
                c = 1.0 if adj else 4 * math.pi ** 2 / g.K / ng
            for n in w:
                G = sum(complex(np.exp(-2j * np.pi * ((n * k) % ng) / ng)) * f[:, k] for k in range(ng))
                rings.append(G if adj else g.weigh(G, n))
                tasks.append((bl, n, w[n] * c))
        return self._to_lm(tasks, rings, nb)


def _exact_uneven(c, maps, dev):
    wav, scal, rec = [], [], []
    for f, (L, N, spin) in zip(maps, _uneven(c)):
        one = _case("device", L, N, c["J_min"], spin=spin)
        P = _Plan(one, dev)
        w, s = P.split(P.sht(f[None].to(torch.float64 if P.real else torch.complex128)))
        # the transforms go on from the rounded coefficients
        half = torch.float32 if P.real else torch.complex64
        r = P.isht(P.merge(w.to(half).to(w.dtype), s.to(half).to(s.dtype)))
        for to, v in ((wav, w), (scal, s), (rec, r)):
            to.append((v if P.real else torch.view_as_real(v.contiguous())).reshape(-1))
    return torch.cat(wav), torch.cat(scal), torch.cat(rec)


def exact(c, seed):
    if c["L"] >= 1024 and c["batch"] > 4:
        return None  # minutes of work
    dev = _device()
    with torch.no_grad():
        given = _inputs(c, seed)
        if c["kind"] == "uneven":
            return _exact_uneven(c, given["maps"], dev)
        P = _Plan(c, dev)
        wide = torch.float64 if P.real else torch.complex128
        if c["kind"] == "harmonic":
            w, s = P.split(torch.from_numpy(given["flm"]).to(dev)[None])
            return w[0], s[0], P.merge(w, s)[0].cpu().numpy()
        if c["kind"] == "loss":
            x, y = given["x"].to(wide), given["y"].to(wide)
            w, s = P.split(P.sht(x))
            if c["single"]:
                w, s = w.float().double(), s.float().double()
            kept = torch.sign(w) * torch.clamp(w.abs() - THRESHOLD, min=0)
            r = P.isht(P.merge(kept, s)) - y
            loss = 0.5 * r.square().sum() + LAMBDA * w.abs().sum()
            gw, gs = P.split(P.sht(r, adjoint_of_inverse=True), adjoint_of_merge=True)
            gw = gw * (w.abs() > THRESHOLD) + LAMBDA * torch.sign(w)
            return loss, P.isht(P.merge(gw, gs, adjoint_of_split=True), adjoint_of_forward=True)
        f = torch.as_tensor(given["f"]).to(dev).to(wide)
        f = f[None] if f.dim() == 1 else f
        w, s = P.split(P.sht(f))
        if c["single"]:
            half = torch.float32 if P.real else torch.complex64
            w, s = w.to(half).to(wide), s.to(half).to(wide)
        out = (w, s, P.isht(P.merge(w, s)))
        return tuple(v[0] for v in out) if c["kind"] in ("host", "axisym") else out
