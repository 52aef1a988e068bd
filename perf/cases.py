"""The calls this library is used for, with their inputs, for timing.

listed() names the cases, draw() gives another of the same ranges, prepare()
makes a case's inputs on the GPU (or on the host, for the calls that take
numpy arrays), run() makes one call through the public entry points, work()
says what a call cannot do without, and exact() gives its values from plain
torch arithmetic in 64 bits.

The spectra are what the library is for: Marchenko-Pastur bulks with a few
spikes above them, at the imaginary offsets eta = s / sqrt(p) that the
estimators use.  Families:

  deconvolve   deconvolve_spiked on a host spectrum: a small, latency-bound
               call of an interactive session
  host         stieltjes_transform on a host spectrum with its default method
               (exact sums), as the numpy caller of the reference does
  exact        stieltjes_m on a CUDA tensor, exact sums, no gradient
  train        stieltjes_m and its backward pass: one step of fitting a
               spectrum, returning the transform and the gradient
  treecode     stieltjes_m with a ChebCode preset: the large-p transform
  grid         the FFT grid methods (nufft, fft5) through the C ABI's
               device-pointer form
  batch        many spectra of uneven size in one device-pointer call
  matrix       cleaning a sample covariance, or estimating its precision
               matrix, from a device matrix
"""
from __future__ import annotations

import ctypes as C
import math

import torch

import shrinkers_b200 as rk
from shrinkers_b200 import _native
from shrinkers_b200.autograd import stieltjes_m

_PREC = {"f64": 0, "mixed": 1}
#: floating-point operations of one ordered pair: a difference, its square
#: plus eta^2 (2), a quotient, and two multiply-adds
_PAIR = 8.0
#: exact() is given where the pair sums it needs stay under this
_MOST_PAIRS = 2.5e11


# ---------------------------------------------------------------- cases --
def listed():
    return [
        # an interactive deconvolution of a small spectrum: launches and copies
        {"name": "deconvolve 1000", "kind": "deconvolve", "p": 1000, "c": 0.25, "points": 200},
        # the reference README's middle size, numpy in and out, defaults
        {"name": "host 4096", "kind": "host", "p": 4096, "eta": 0.1, "order": "ascending"},
        # the README's large size on the device, full precision
        {"name": "exact f64 50000", "kind": "exact", "p": 50000, "eta": 1.0, "precision": "f64",
         "order": "ascending"},
        # the benchmark's headline: every pair of a million eigenvalues
        {"name": "exact mixed 1000000", "kind": "exact", "p": 1000000, "eta": 1.0,
         "precision": "mixed", "order": "ascending"},
        # one optimisation step through the exact transform and its adjoint
        {"name": "train exact 20000", "kind": "train", "p": 20000, "eta": 1.0, "method": "exact",
         "precision": "f64"},
        # the same for a spectrum too large for the pair sums
        {"name": "train treecode 200003", "kind": "train", "p": 200003, "eta": 1.0,
         "method": "chebcode_xtreme", "precision": "f64"},
        # the treecode at the benchmark's size, its middle preset
        {"name": "chebcode 1000000", "kind": "treecode", "p": 1000000, "eta": 1.0,
         "method": "chebcode"},
        # the fastest transform of a large spectrum
        {"name": "nufft 1000000", "kind": "grid", "p": 1000000, "eta": 1.0, "method": "nufft"},
        # the fine-grid transform at an odd size
        {"name": "fft5 200003", "kind": "grid", "p": 200003, "eta": 1.0, "method": "fft5"},
        # rolling-window spectra, all sizes in one call
        {"name": "batch mixed 1024", "kind": "batch", "spectra": 1024, "largest": 16384,
         "precision": "mixed"},
        # a daily covariance of a few hundred assets, inverted
        {"name": "precision 501", "kind": "matrix", "p": 501, "ratio": 4.0, "output": "precision"},
        # cleaning the covariance of a large universe
        {"name": "clean 2048", "kind": "matrix", "p": 2048, "ratio": 4.0, "output": "clean"},
    ]


def _size(rng, lo, hi):
    """A whole number spread over [lo, hi] by its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["deconvolve", "host", "exact", "train", "treecode", "grid", "batch",
                       "matrix"])
    eta = rng.choice([0.1, 0.4, 1.0])  # the defaults of the transforms, the shrinkage, the adjoint
    order = rng.choice(["ascending", "ascending", "descending"])  # from eigh, or from an SVD
    if kind == "deconvolve":
        return {"kind": kind, "p": _size(rng, 100, 50000), "c": round(rng.uniform(0.05, 0.9), 3),
                "points": rng.choice([100, 200, 500])}
    if kind == "host":
        return {"kind": kind, "p": _size(rng, 100, 30000), "eta": eta, "order": order}
    if kind == "exact":
        return {"kind": kind, "p": _size(rng, 1000, 400000), "eta": eta,
                "precision": rng.choice(["f64", "mixed"]), "order": order}
    if kind == "train":
        method = rng.choice(["exact", "exact", "chebcode", "chebcode_xtreme"])
        return {"kind": kind, "p": _size(rng, 1000, 60000 if method == "exact" else 400000),
                "eta": 1.0, "method": method, "precision": rng.choice(["f64", "mixed"])}
    if kind == "treecode":
        return {"kind": kind, "p": _size(rng, 20000, 1000000), "eta": eta,
                "method": rng.choice(["chebcode_fast", "chebcode", "chebcode_balanced",
                                      "chebcode_xtreme"])}
    if kind == "grid":
        return {"kind": kind, "p": _size(rng, 20000, 1000000), "eta": eta,
                "method": rng.choice(["nufft", "fft5"])}
    if kind == "batch":
        return {"kind": kind, "spectra": _size(rng, 64, 2048),
                "largest": rng.choice([2048, 4096, 16384]),
                "precision": rng.choice(["f64", "mixed"])}
    return {"kind": kind, "p": _size(rng, 64, 2048), "ratio": round(rng.uniform(1.5, 8.0), 2),
            "output": rng.choice(["clean", "precision"])}


# --------------------------------------------------------------- inputs --
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(gen, n, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)


def _bulk(gen, p, c, sigma2=1.0):
    """p eigenvalues of a Marchenko-Pastur bulk, ascending: one in each of p
    slices of equal mass, by the inverse distribution function (a sample
    covariance's eigenvalues repel, so they spread as evenly as this)."""
    a, b = sigma2 * (1.0 - math.sqrt(c)) ** 2, sigma2 * (1.0 + math.sqrt(c)) ** 2
    n = 1 << 18 if p > 30000 else 1 << 12
    x = torch.linspace(a, b, n, dtype=torch.float64)
    f = torch.sqrt(torch.clamp((b - x) * (x - a), min=0.0)) / x
    cdf = torch.cumsum(0.5 * (f[1:] + f[:-1]), 0)  # on the host: the same sums every time
    cdf = torch.cat([cdf.new_zeros(1), cdf / cdf[-1]])
    x, cdf = x.cuda(), cdf.cuda()
    u = (torch.arange(p, device="cuda", dtype=torch.float64) + _uniform(gen, p)) / p
    k = torch.searchsorted(cdf, u, right=True).clamp(1, n - 1)
    w = (u - cdf[k - 1]) / (cdf[k] - cdf[k - 1]).clamp(min=1e-300)
    return x[k - 1] + w * (x[k] - x[k - 1])


def _spectrum(gen, p, c=0.3, spikes=5, order="ascending", top=20.0):
    """A bulk with its `spikes` largest values moved above it, in order."""
    ev = _bulk(gen, p, c)
    spikes = min(spikes, p // 20)
    if spikes:
        ev[-spikes:] = _uniform(gen, spikes, 1.7 * (1.0 + math.sqrt(c)) ** 2, top)
    return torch.sort(ev, descending=order == "descending").values.contiguous()


def _eta(case):
    return case["eta"] / math.sqrt(case["p"])


def _factor_covariance(gen, p, ratio):
    """Sample covariance of p variables with three common factors, ratio*p samples."""
    n = int(round(ratio * p))
    load = torch.randn(p, 3, generator=gen, device="cuda", dtype=torch.float64)
    load *= torch.tensor([6.0, 4.0, 3.0], device="cuda", dtype=torch.float64)
    f = torch.randn(n, 3, generator=gen, device="cuda", dtype=torch.float64)
    x = torch.randn(n, p, generator=gen, device="cuda", dtype=torch.float64)
    x = x + f @ load.T
    x -= x.mean(0)
    s = x.T @ x / (n - 1)
    return (0.5 * (s + s.T)).contiguous(), p / n


def _make(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "deconvolve":
        ev = _spectrum(gen, case["p"], case["c"], 3)
        return {"ev": ev.cpu().numpy()}
    if kind == "host":
        return {"ev": _spectrum(gen, case["p"], 0.25, 3, case["order"]).cpu().numpy()}
    if kind == "exact":
        return {"ev": _spectrum(gen, case["p"], 0.5, 0, case["order"])}
    if kind == "train":
        ev = _spectrum(gen, case["p"])
        g = torch.randn(2, case["p"], generator=gen, device="cuda", dtype=torch.float64)
        return {"ev": ev, "g": torch.complex(g[0], g[1]) / case["p"]}
    if kind in ("treecode", "grid"):
        # the nufft and fft5 grids span the spectrum: spikes stretch them
        return {"ev": _spectrum(gen, case["p"], 0.1, 20, top=50.0)}
    if kind == "batch":
        n = case["spectra"]
        # the sizes belong to the case, the values to the seed
        u = torch.rand(n, 4, generator=torch.Generator().manual_seed(n), dtype=torch.float64)
        p = torch.exp(math.log(256.0) + u[:, 0] * math.log(case["largest"] / 256.0)).round().long()
        parts = []
        for s in range(n):
            c, s2 = 0.05 + 0.85 * float(u[s, 1]), math.exp((2 * float(u[s, 2]) - 1) * math.log(2.0))
            ev = _bulk(gen, int(p[s]), c, s2)
            k = int(6 * float(u[s, 3]))
            if k:
                ev[-k:] = _uniform(gen, k, (1.0 + math.sqrt(c)) ** 2 * s2 * 1.5, 30.0)
            parts.append(torch.sort(ev).values)
        offsets = torch.zeros(n + 1, dtype=torch.int64)
        offsets[1:] = torch.cumsum(p, 0)
        return {"ev": torch.cat(parts), "offsets": offsets.cuda(),
                "eta": (1.0 / torch.sqrt(p.double())).cuda()}
    cov, c = _factor_covariance(gen, case["p"], case["ratio"])
    return {"cov": cov, "c": c}


def prepare(case, seed):
    state = dict(case)
    state.update(_make(case, seed))
    if case["kind"] in ("grid", "batch"):
        state["re"], state["im"] = (torch.empty_like(state["ev"]) for _ in range(2))
        state["method_id"] = rk.parse_method(case["method"]) if case["kind"] == "grid" else 0
    if case["kind"] == "matrix":
        state["out"] = torch.empty_like(state["cov"])
        state["v1"], state["v2"] = (state["cov"].new_empty(case["p"]) for _ in range(2))
    if case["kind"] == "train":
        state["ev"].requires_grad_(True)
    return state


# ----------------------------------------------------------------- calls --
def run(state):
    kind = state["kind"]
    if kind == "deconvolve":
        return rk.deconvolve_spiked(state["ev"], state["c"], n_points=state["points"], margin=1.2)
    if kind == "host":
        return rk.stieltjes_transform(state["ev"], eta=_eta(state))
    if kind == "exact":
        return stieltjes_m(state["ev"], _eta(state), state["precision"])
    if kind == "treecode":
        return stieltjes_m(state["ev"], _eta(state), method=state["method"])
    if kind == "train":
        m = stieltjes_m(state["ev"], _eta(state), state["precision"], state["method"])
        (grad,) = torch.autograd.grad(m, state["ev"], state["g"])
        return {"m": m.detach(), "grad": grad}
    L = _native.load()
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "grid":
        _native.check(L.shrk_stieltjes_all_dev(
            state["ev"].data_ptr(), state["p"], _eta(state), state["method_id"], 0, float("nan"), 0,
            state["re"].data_ptr(), state["im"].data_ptr(), stream))
        return {"real": state["re"], "imag": state["im"]}
    if kind == "batch":
        _native.check(L.shrk_stieltjes_batched_dev(
            state["ev"].data_ptr(), state["offsets"].data_ptr(), state["spectra"],
            state["eta"].data_ptr(), _PREC[state["precision"]], state["re"].data_ptr(),
            state["im"].data_ptr(), stream))
        return {"real": state["re"], "imag": state["im"]}
    scalar = C.c_double()
    if state["output"] == "clean":
        _native.check(L.shrk_clean_covariance_matrix_dev(
            state["cov"].data_ptr(), state["p"], state["c"], 0, state["out"].data_ptr(), None,
            state["v1"].data_ptr(), state["v2"].data_ptr(), C.byref(scalar), stream))
    else:
        _native.check(L.shrk_estimate_precision_matrix_dev(
            state["cov"].data_ptr(), state["p"], state["c"], 0, state["out"].data_ptr(), None,
            state["v1"].data_ptr(), state["v2"].data_ptr(), C.byref(scalar), stream))
    return {"matrix": state["out"], "first": state["v1"], "second": state["v2"],
            "scalar": scalar.value}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        # sizes are log-uniform in [256, largest]: the means of p and of p^2
        r = math.log(case["largest"] / 256.0)
        p = (case["largest"] - 256.0) / r
        p2 = (case["largest"] ** 2 - 256.0 ** 2) / (2.0 * r)
        return {"bytes": 24.0 * p * case["spectra"], "flops": _PAIR * p2 * case["spectra"]}
    p = float(case["p"])
    if kind == "deconvolve":
        # a tree over p sources, then a few leaves of 32 and a node or two a level per point
        return {"bytes": 8.0 * p + 56.0 * case["points"],
                "flops": _PAIR * 11.0 * (2.0 * p + 20.0 * case["points"])}
    if kind in ("host", "exact"):
        return {"bytes": 24.0 * p, "flops": _PAIR * p * p}
    if kind == "train":
        if case["method"] == "exact":
            return {"bytes": 56.0 * p, "flops": 2.5 * _PAIR * p * p}
        return {"bytes": 56.0 * p, "flops": 2.5 * _PAIR * p * 300.0}
    if kind == "treecode":
        return {"bytes": 24.0 * p, "flops": _PAIR * p * 200.0}
    if kind == "grid":
        m = 2.0 ** 16 if case["method"] == "nufft" else 2.0 ** 20
        return {"bytes": 24.0 * p, "flops": 10.0 * m * math.log2(m) + 50.0 * p}
    # reduction to tridiagonal form, back-transform, reconstruction
    return {"bytes": 16.0 * p * p, "flops": (4.0 / 3.0 + 2.0 + 1.0) * p ** 3}


# ----------------------------------------------------------------- exact --
def _rows(p):
    return max(1, (1 << 26) // p)


def _sums(ev, eta, per_point=None):
    """Raw sums of 1/((x - ev_j) - i eta) at every x = ev_i."""
    re, im = torch.empty_like(ev), torch.empty_like(ev)
    for a in range(0, ev.numel(), _rows(ev.numel())):
        x = ev[a:a + _rows(ev.numel()), None]
        e = eta if per_point is None else per_point[a:a + _rows(ev.numel()), None]
        d = x - ev[None, :]
        q = 1.0 / (d * d + e * e)
        re[a:a + x.shape[0]] = (d * q).sum(1)
        im[a:a + x.shape[0]] = (q * e).sum(1)
    return re, im


def _gradient(ev, eta, g):
    """dL/dev of L = sum_j Re(conj(g_j) m_j), m_j = mean_i 1/(ev_i - ev_j - i eta)."""
    p = ev.numel()
    grad = torch.empty_like(ev)
    w, v = g.real.contiguous(), g.imag.contiguous()
    for a in range(0, p, _rows(p) // 2 + 1):
        b = min(p, a + _rows(p) // 2 + 1)
        d = ev[a:b, None] - ev[None, :]
        q = 1.0 / (d * d + eta * eta)
        # t = 1/(d - i eta)^2 = (d + i eta)^2 q^2, as source k = row of target j = column
        t_re, t_im = (d * d - eta * eta) * q * q, (2.0 * eta) * d * q * q
        # as a source: -Re(conj(g_j) t); as a target, the same with d reversed, plus
        grad[a:b] = (t_re * (w[a:b, None] - w[None, :])
                     - t_im * (v[a:b, None] + v[None, :])).sum(1) / p
    return grad


def exact(case, seed):
    kind = case["kind"]
    if kind == "deconvolve":
        return None
    if kind not in ("batch", "matrix") and float(case["p"]) ** 2 > _MOST_PAIRS:
        return None
    s = _make(case, seed)
    if kind == "host":
        re, im = _sums(torch.from_numpy(s["ev"]).cuda(), _eta(case))
        return {"real": (re / case["p"]).cpu().numpy(), "imag": (im / case["p"]).cpu().numpy()}
    if kind in ("exact", "treecode"):
        re, im = _sums(s["ev"], _eta(case))
        return torch.complex(-re, im) / case["p"]
    if kind == "train":
        re, im = _sums(s["ev"], _eta(case))
        return {"m": torch.complex(-re, im) / case["p"],
                "grad": _gradient(s["ev"], _eta(case), s["g"])}
    if kind == "grid":
        re, im = _sums(s["ev"], _eta(case))
        return {"real": re / case["p"], "imag": im / case["p"]}
    if kind == "batch":
        off = s["offsets"].tolist()
        re, im = torch.empty_like(s["ev"]), torch.empty_like(s["ev"])
        for a, b in zip(off[:-1], off[1:]):
            r, i = _sums(s["ev"][a:b], 1.0 / math.sqrt(b - a))
            re[a:b], im[a:b] = r / (b - a), i / (b - a)
        return {"real": re, "imag": im}
    lam, vec = torch.linalg.eigh(s["cov"])
    lam, vec, c, p = lam.flip(0), vec.flip(1), s["c"], case["p"]
    if case["output"] == "clean":
        # Ledoit-Wolf eigenvalues at eta = 0.4/sqrt(p), rescaled to the trace
        re, im = _sums(lam, 0.4 / math.sqrt(p))
        # m = -conj(S)/p at lam + i eta; |1 - c - c lam m|^2 in the denominator
        d_re, d_im = 1.0 - c + c * lam * re / p, c * lam * im / p
        xi = lam / (d_re * d_re + d_im * d_im)
        xi = xi * (lam.sum() / xi.sum())
        med = lam[p // 2] if p % 2 else 0.5 * (lam[p // 2 - 1] + lam[p // 2])
        g = min(max(c, 0.0), 1.0)
        s2 = med / (0.999995823 - 0.333211332 * g - 0.0106766617 * g * g - 0.000758816762 * g ** 3
                    - 0.00256753402 * g ** 4)
        diff = xi - s2
        num, den = 1.0 - c * s2 * s2 / (diff * diff), 1.0 + c * s2 / diff
        a2 = torch.where((diff > 1e-12) & (num > 0.0), torch.clamp(num / den, max=1.0 - 1e-15),
                         torch.zeros_like(xi))
        idle = a2 == 0.0
        level = xi[idle].mean() if bool(idle.any()) else xi.min()
        cov = (vec * (a2 * (xi - level))) @ vec.T
        cov.diagonal().add_(level)
        return {"matrix": cov, "first": xi, "second": a2, "scalar": float(s2)}
    # quadratic inverse shrinkage at z_i = lam_i (1 + i h)
    h = min(c * c, 1.0 / (c * c)) ** 0.35 / p ** 0.35
    re, im = _sums(lam, None, h * lam)
    theta, htheta = lam * re / p, lam * im / p
    x, o = 1.0 / lam, 1.0 - c
    delta = 1.0 / (o * o * x + 2.0 * c * o * x * theta
                   + c * c * x * (theta * theta + htheta * htheta))
    delta = delta * (lam.sum() / delta.sum())
    return {"matrix": (vec / delta) @ vec.T, "first": 1.0 / delta, "second": delta, "scalar": h}
