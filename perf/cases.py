"""Performance cases of the GPU NFFT: the calls a program makes in earnest,
from single small 2-D transforms to the 256^3 radial set, with the plans that
such a program keeps between calls.

A case is a dict of plain values.  ``kind`` says what one pass is:

  pair      mul!(fHat, p, f) and mul!(f, adjoint(p), fHat) into the caller's
            arrays, as one iteration of an iterative reconstruction does
  forward   p * f
  adjoint   adjoint(p) * fHat
  train     nfft_nodes(k, f, p) and its backward pass: one step of learning a
            trajectory (new nodes every step, gradients of the nodes and image)
  batch     a forward and an adjoint call of an NFFTBatch
  slices    a forward and an adjoint call of a directional plan (2-D NFFTs of
            the slices of a stack)
  toeplitz  the Gram operator A^H A by its Toeplitz kernel
  sdc       sampling density compensation weights, 20 iterations

``m`` = 0 asks for the plan's default accuracy (reltol 1e-9: m = 5, sigma = 2)
and ``pre`` = "" for its default window evaluation (POLYNOMIAL).
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nfft.jl_gb300"))

import nfftgb300 as nf  # noqa: E402
from nfftgb300 import autodiff, tools  # noqa: E402

DEV = "cuda"
GOLDEN = math.pi * (3.0 - math.sqrt(5.0))


def _case(name, kind, N, M, nodes, **kw):
    c = {"kind": kind, "D": len(N), "M": M, "nodes": nodes, "prec": 32, "m": 0, "sigma": 2.0, "pre": "",
         "compensated": False}
    if name:
        c["name"] = name
    for d, n in enumerate(N):
        c["N%d" % d] = n
    c.update(kw)
    return c


def listed():
    return [
        # one small double-precision image: latency and launches are what counts
        _case("small 2-D f64", "pair", (128, 128), 16384, "uniform", prec=64, m=4, pre="TENSOR"),
        # one slice with default parameters and an image size that is no power of two
        _case("ragged 2-D default", "pair", (300, 210), 98304, "radial"),
        # trajectory learning on a 256^2 spiral: nodes!, forward, both gradients
        _case("spiral training step", "train", (256, 256), 65536, "spiral", m=4),
        # density compensation of the same spiral before a reconstruction
        _case("spiral sdc", "sdc", (256, 256), 65536, "spiral", m=4, pre="TENSOR"),
        # one iteration of a 256^3 radial reconstruction: the largest case
        _case("radial 256^3 pair", "pair", (256, 256, 256), 8192 * 512, "radial", m=4, pre="TENSOR"),
        # simulation of a 3-D acquisition with default parameters, ordinary size
        _case("3-D default forward", "forward", (120, 108, 90), 600000, "radial"),
        # its gridding direction on an odd image
        _case("odd 3-D default adjoint", "adjoint", (101, 87, 75), 300001, "uniform"),
        # double precision with default parameters: what NumPy nodes give
        _case("3-D f64 default pair", "pair", (64, 64, 64), 262144, "uniform", prec=64),
        # the longest transform: a 1-D line with compensated sums
        _case("1-D line compensated", "pair", (1 << 22,), 1 << 24, "uniform", m=5, pre="TENSOR", compensated=True),
        # many independent 2-D problems of mixed sizes at once
        _case("32 batched 2-D plans", "batch", (64, 512), 10000, "uniform", m=4, pre="TENSOR", Mmax=1000000,
              plans=32),
        # a stack of slices that share one radial trajectory
        _case("64 slices", "slices", (256, 256), 131072, "radial", m=4, columns=64, columns_first=False),
        # one Gram product of the radial reconstruction by its Toeplitz kernel
        _case("Toeplitz 256^3", "toeplitz", (256, 256, 256), 8192 * 512, "radial", m=4, pre="TENSOR"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pair"] * 5 + ["forward"] * 2 + ["adjoint"] * 2 + ["train", "batch", "slices", "toeplitz",
                                                                         "sdc"])
    if kind == "batch":
        return _case("", kind, (rng.randint(24, 80), _log(rng, 96, 512)), _log(rng, 2000, 20000), "uniform", m=4,
                     pre=rng.choice(["", "TENSOR"]), Mmax=_log(rng, 30000, 1000000), plans=rng.randint(3, 32))
    if kind == "slices":
        n = _log(rng, 48, 256)
        return _case("", kind, (n, rng.randint(3 * n // 4, n)), _log(rng, 3000, 131072),
                     rng.choice(["radial", "uniform"]), m=rng.choice([3, 4, 4, 5]), columns=rng.randint(2, 64),
                     columns_first=rng.random() < 0.5)
    if kind == "sdc":
        n = _log(rng, 48, 320)
        return _case("", kind, (n, n), _log(rng, 8000, 200000), rng.choice(["radial", "spiral"]), m=4, pre="TENSOR")
    if kind == "train":
        n = _log(rng, 48, 400)
        return _case("", kind, (n, rng.randint(3 * n // 4, n)), _log(rng, 5000, 200000),
                     rng.choice(["radial", "spiral"]), m=rng.choice([0, 3, 4]))
    if kind == "toeplitz":
        if rng.random() < 0.5:
            n = _log(rng, 64, 384)
            return _case("", kind, (n, rng.randint(3 * n // 4, n)), _log(rng, 10000, 200000), "radial", m=4,
                         pre="TENSOR")
        n = rng.choice([32, 48, 64, 96, 128])
        return _case("", kind, (n, n, n), _log(rng, 50000, 500000), "radial", m=4, pre="TENSOR")
    D = rng.choice([1, 2, 2, 2, 3, 3, 3, 3])
    prec = 64 if rng.random() < 0.25 else 32
    if D == 1:
        N = (_log(rng, 1000, 1 << (18 if prec == 64 else 21)),)
    elif D == 2:
        n = _log(rng, 48, 512 if prec == 64 else 1000)
        N = (n, rng.randint(max(2, n // 2), n))
    else:
        n = _log(rng, 24, 90 if prec == 64 else 180)
        N = (n, rng.randint(2 * n // 3, n), rng.randint(n // 2, n))
    if rng.random() < 0.35:  # the sizes people pick for FFTs
        N = tuple(1 << max(4, round(math.log2(n))) for n in N)
    m = rng.choice([0, 0, 3, 4, 4, 5, 6])
    sigma = rng.choice([2.0, 2.0, 2.0, 1.5]) if m else 2.0
    taps = (2 * (m or 5)) ** D
    most = min(3000000 if D < 3 else 2000000, (1.0e8 if prec == 64 else 1.2e9) / taps)
    compensated = D == 1 and rng.random() < 0.3
    nodes = rng.choice(["uniform", "radial"]) if D > 1 else "uniform"
    pre = rng.choice(["", "", "TENSOR", "LINEAR"] if m and m <= 4 else ["", "", "TENSOR"])
    return _case("", kind, N, _log(rng, 3000, most), nodes, prec=prec, m=m, sigma=sigma, pre=pre,
                 compensated=compensated)


# ------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _shape(c):
    return tuple(c["N%d" % d] for d in range(c["D"]))


def _rdt(c):
    return torch.float32 if c["prec"] == 32 else torch.float64


def _cdt(c):
    return torch.complex64 if c["prec"] == 32 else torch.complex128


def _uniform(g, D, M):
    return torch.rand((D, M), generator=g, device=DEV, dtype=torch.float64) - 0.5


def _nodes(c, g, M=None):
    """(D, M) nodes in [-1/2, 1/2), made in FP64 and rounded to the plan's type."""
    D, M = c["D"], M or c["M"]
    if c["nodes"] == "uniform":
        k = _uniform(g, D, M)
    else:
        turn = 2 * math.pi * float(torch.rand(1, generator=g, device=DEV))
        if c["nodes"] == "spiral":  # 32 interleaved Archimedean spirals
            q = torch.arange(M, device=DEV, dtype=torch.float64)
            per = -(-M // 32)
            t, arm = (q % per) / per, torch.div(q, per, rounding_mode="floor")
            th = 8 * math.pi * t + 2 * math.pi * arm / 32 + turn
            k = torch.stack([0.5 * t * torch.cos(th), 0.5 * t * torch.sin(th)])
        else:  # golden-angle spokes through the centre of k-space
            samples = 512 if M >= 65536 else 128
            spokes = -(-M // samples)
            i = torch.arange(spokes, device=DEV, dtype=torch.float64)
            r = -0.5 + torch.arange(samples, device=DEV, dtype=torch.float64) / samples
            ph = i * GOLDEN + turn
            if D == 2:
                u = torch.stack([torch.cos(ph), torch.sin(ph)])
            else:
                z = (i + 0.5) / spokes
                s = torch.sqrt(1 - z * z)
                u = torch.stack([s * torch.cos(ph), s * torch.sin(ph), z])
            k = (u[:, :, None] * r[None, None, :]).reshape(D, -1)[:, :M]
    return k.clamp(-0.5, 0.4999999).to(_rdt(c)).contiguous()


def _image(c, g, N):
    """A column-major complex image with unit-variance noise on a smooth object."""
    x = nf.empty_image(N, _cdt(c), DEV)
    flat = torch.randn(N[::-1], generator=g, device=DEV, dtype=torch.complex128)
    for d, n in enumerate(N):
        t = torch.linspace(-1, 1, n, device=DEV, dtype=torch.float64)
        flat += torch.exp(-4 * t * t).reshape([n if e == len(N) - 1 - d else 1 for e in range(len(N))])
    x.copy_(flat.permute(*reversed(range(len(N)))))
    return x


def _values(c, g, n):
    return torch.randn(n, generator=g, device=DEV, dtype=torch.complex128).to(_cdt(c))


def _plan_kw(c):
    kw = {}
    if c["m"]:
        kw.update(m=c["m"], sigma=c["sigma"])
    if c["pre"]:
        kw["precompute"] = getattr(nf, c["pre"])
    if c["compensated"]:
        kw["compensated"] = True
    return kw


def _batch_sizes(c):
    """The image sizes and node counts of a batch (a function of the case alone)."""
    r = random.Random(c["plans"] * 1000003 + c["M"])
    out = []
    for _ in range(c["plans"]):
        n = _log(r, c["N0"], c["N1"])
        if r.random() < 0.7:
            n = 32 * max(2, round(n / 32))
        out.append(((n, n), _log(r, c["M"], c["Mmax"])))
    return out


def _inputs(c, seed):
    """The arrays of one pass: nodes, images and node values."""
    g = _gen(seed)
    if c["kind"] == "batch":
        return [(_nodes(c, g, M), _image(c, g, N), _values(c, g, M)) for N, M in _batch_sizes(c)]
    N = _shape(c)
    k = _nodes(c, g)
    if c["kind"] == "slices":
        C = c["columns"]
        full = (C,) + N if c["columns_first"] else N + (C,)
        f = _image(c, g, full)
        nout = (C, c["M"]) if c["columns_first"] else (c["M"], C)
        v = nf.empty_image(nout, _cdt(c), DEV)
        v.copy_(_values(c, g, c["M"] * C).reshape(nout))
        return k, f, v
    f = None if c["kind"] in ("sdc", "adjoint") else _image(c, g, N)
    v = None if c["kind"] in ("sdc", "forward", "toeplitz") else _values(c, g, c["M"])
    return k, f, v


def prepare(case, seed):
    c = case
    s = {"case": c}
    if c["kind"] == "batch":
        data = _inputs(c, seed)
        s["plans"] = [nf.plan_nfft(k, tuple(f.shape), **_plan_kw(c)) for k, f, _ in data]
        s["batch"] = nf.NFFTBatch(s["plans"])
        s["f"] = [f for _, f, _ in data]
        s["v"] = [v for _, _, v in data]
        s["y"] = [torch.empty_like(v) for v in s["v"]]
        s["x"] = [nf.empty_image(f.shape, f.dtype, DEV) for f in s["f"]]
        return s
    k, f, v = _inputs(c, seed)
    N = _shape(c)
    s.update(k=k, f=f, v=v)
    if c["kind"] == "slices":
        s["plan"] = nf.plan_nfft(k, tuple(f.shape), dims=(2, 3) if c["columns_first"] else (1, 2), m=c["m"],
                                 sigma=c["sigma"])
        s["y"] = nf.empty_image(v.shape, v.dtype, DEV)
        s["x"] = nf.empty_image(f.shape, f.dtype, DEV)
    elif c["kind"] == "toeplitz":
        s["tz"] = tools.Toeplitz(N, _cdt(c), DEV)
        s["lam"] = tools.calculate_toeplitz_kernel(N, k, m=c["m"], sigma=c["sigma"], toeplitz=s["tz"],
                                                   precompute=getattr(nf, c["pre"]))
        s["x"] = nf.empty_image(N, _cdt(c), DEV)
    else:
        s["plan"] = nf.plan_nfft(k, N, **_plan_kw(c))
        if c["kind"] == "pair":
            s["y"] = torch.empty_like(v)
            s["x"] = nf.empty_image(N, f.dtype, DEV)
        elif c["kind"] == "train":
            s["k"] = k.clone().requires_grad_(True)
            s["f"] = f.requires_grad_(True)
    return s


def run(state):
    s = state
    kind = s["case"]["kind"]
    if kind == "pair" or kind == "slices":
        nf.mul_(s["y"], s["plan"], s["f"])
        nf.mul_(s["x"], nf.adjoint(s["plan"]), s["v"])
        return [s["y"], s["x"]]
    if kind == "forward":
        return s["plan"] * s["f"]
    if kind == "adjoint":
        return nf.adjoint(s["plan"]) * s["v"]
    if kind == "train":
        y = autodiff.nfft_nodes(s["k"], s["f"], s["plan"])
        gk, gf = torch.autograd.grad(y, (s["k"], s["f"]), s["v"])
        return [y.detach(), gk, gf]
    if kind == "batch":
        s["batch"].forward_(s["y"], s["f"])
        s["batch"].adjoint_(s["x"], s["v"])
        return [s["y"], s["x"]]
    if kind == "toeplitz":
        s["x"].copy_(s["f"])
        return s["tz"].convolve_(s["x"], s["lam"])
    return tools.sdc(s["plan"], iters=20)


# --------------------------------------------------------------------- work
def _taps(c):
    return (2 * (c["m"] or 5)) ** c["D"]


def _grid(c, N):
    return float(np.prod([2 * (math.ceil(c["sigma"] * n) // 2) for n in N]))


def work(case):
    c = case
    sr = c["prec"] // 8
    sc = 2 * sr

    def transform(N, M, cols=1):
        g = _grid(c, N)
        n = float(np.prod(N))
        return (cols * (n + M) * sc + M * c["D"] * sr, cols * (4.0 * M * _taps(c) + 5.0 * g * math.log2(g)))

    if c["kind"] == "batch":
        both = [transform(N, M) for N, M in _batch_sizes(c)]
        return {"bytes": 2 * sum(b for b, _ in both), "flops": 2 * sum(f for _, f in both)}
    N = _shape(c)
    n = float(np.prod(N))
    b, f = transform(N, c["M"], c.get("columns", 1))
    if c["kind"] in ("pair", "slices"):
        return {"bytes": 2 * b, "flops": 2 * f}
    if c["kind"] == "train":  # forward, adjoint and node gradient, one set of nodes in and one gradient out
        return {"bytes": 2 * b, "flops": 3 * f}
    if c["kind"] == "toeplitz":
        g = n * 2 ** c["D"]
        return {"bytes": (2 * n + g) * sc, "flops": 2 * 5.0 * g * math.log2(g)}
    if c["kind"] == "sdc":  # 20 real spreading and gathering sums, one weight per node out
        return {"bytes": float(c["M"] * (c["D"] + 1) * sr), "flops": 40 * 2.0 * c["M"] * _taps(c)}
    return {"bytes": b, "flops": f}


# -------------------------------------------------------------------- exact
# the direct sums in FP64: node x frequency products that fit the time allowed
_MOST_TERMS = 1.3e12


def _phases(k, N, sign, deriv=False):
    """exp(sign 2 pi i k n), n = -N/2 .. (one row per node); the derivative with respect to k for deriv."""
    n = torch.arange(N, device=DEV, dtype=torch.float64) - N // 2
    e = torch.polar(torch.ones((), device=DEV, dtype=torch.float64), sign * 2 * math.pi * k[:, None] * n[None, :])
    return e * (sign * 2j * math.pi * n)[None, :] if deriv else e


def _ndft1(k, f, N, sign, adj):
    """1-D direct sums: forward values at the nodes, or the adjoint image."""
    A = max(1, math.isqrt(N))
    B = -(-N // A)
    step = max(1, int(2e7 // max(A, B)))
    a = torch.arange(A, device=DEV, dtype=torch.float64)
    b = torch.arange(B, device=DEV, dtype=torch.float64) * A - N // 2
    out = []
    if not adj:
        F = torch.zeros(A * B, dtype=torch.complex128, device=DEV)
        F[:N] = f
        F = F.reshape(B, A)
    else:
        acc = torch.zeros((B, A), dtype=torch.complex128, device=DEV)
    one = torch.ones((), device=DEV, dtype=torch.float64)
    for lo in range(0, k.shape[1], step):
        kc = k[0, lo:lo + step]
        ea = torch.polar(one, sign * 2 * math.pi * kc[:, None] * a)
        eb = torch.polar(one, sign * 2 * math.pi * kc[:, None] * b)
        if not adj:
            out.append(((eb @ F) * ea).sum(1))
        else:
            acc += (eb * f[lo:lo + step, None]).transpose(0, 1) @ ea
    return torch.cat(out) if not adj else acc.reshape(-1)[:N]


def _forward(k, f, deriv=-1):
    """f^(k_j) = sum_n f[n] exp(-2 pi i k_j n); with deriv = d its derivative with respect to k_d."""
    D, N = k.shape[0], f.shape
    if D == 1:
        return _ndft1(k, f.reshape(-1), N[0], -1.0, False)
    step = max(1, int(1.5e8 // (f.numel() // N[0])))
    F = f.reshape(N[0], -1)
    out = []
    for lo in range(0, k.shape[1], step):
        e = [_phases(k[d, lo:lo + step], N[d], -1.0, d == deriv) for d in range(D)]
        t = e[0] @ F
        for d in range(1, D):
            t = t.reshape(t.shape[0], N[d], -1)
            t = torch.einsum("jn,jnr->jr", e[d], t) if t.shape[2] > 1 else (e[d] * t[:, :, 0]).sum(1, keepdim=True)
        out.append(t[:, 0])
    return torch.cat(out)


def _adjoint(k, v, N):
    """f[n] = sum_j v_j exp(+2 pi i k_j n)."""
    D = k.shape[0]
    if D == 1:
        return _ndft1(k, v, N[0], 1.0, True)
    rest = int(np.prod(N[1:]))
    step = max(1, int(1.0e8 // rest))
    acc = torch.zeros((N[0], rest), dtype=torch.complex128, device=DEV)
    for lo in range(0, k.shape[1], step):
        e = [_phases(k[d, lo:lo + step], N[d], 1.0) for d in range(D)]
        t = e[1] * v[lo:lo + step, None]
        if D == 3:
            t = (t[:, :, None] * e[2][:, None, :]).reshape(t.shape[0], -1)
        acc += e[0].transpose(0, 1) @ t
    return acc.reshape(N)


def exact(case, seed):
    c = case
    if c["kind"] == "sdc":
        return None
    data = _inputs(c, seed)
    if c["kind"] == "batch":
        if 2 * sum(float(M) * N[0] * N[1] for N, M in _batch_sizes(c)) > _MOST_TERMS:
            return None
        data = [(k.double(), f.to(torch.complex128), v.to(torch.complex128)) for k, f, v in data]
        return [[_forward(k, f) for k, f, _ in data], [_adjoint(k, v, tuple(f.shape)) for k, f, v in data]]
    N = _shape(c)
    passes = {"pair": 2, "slices": 2, "train": 4, "toeplitz": 2}.get(c["kind"], 1)
    if passes * float(c["M"]) * float(np.prod(N)) * c.get("columns", 1) > _MOST_TERMS:
        return None
    k, f, v = data
    k = k.double()
    f = None if f is None else f.to(torch.complex128)
    v = None if v is None else v.to(torch.complex128)
    if c["kind"] == "slices":
        col = range(c["columns"])
        if c["columns_first"]:
            return [torch.stack([_forward(k, f[i].contiguous()) for i in col]),
                    torch.stack([_adjoint(k, v[i], N) for i in col])]
        return [torch.stack([_forward(k, f[..., i].contiguous()) for i in col], -1),
                torch.stack([_adjoint(k, v[:, i], N) for i in col], -1)]
    if c["kind"] == "forward":
        return _forward(k, f)
    if c["kind"] == "adjoint":
        return _adjoint(k, v, N)
    if c["kind"] == "toeplitz":
        return _adjoint(k, _forward(k, f), N)
    y = _forward(k, f)
    x = _adjoint(k, v, N)
    if c["kind"] == "train":
        gk = torch.stack([(v.conj() * _forward(k, f, d)).real for d in range(c["D"])])
        return [y, gk, x]
    return [y, x]
