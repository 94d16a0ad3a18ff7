"""The measured workloads of the normal-mode library.

Each case is one call sequence that a program of this library makes through
its public Python binding (a thin view of the C ABI): a Modess run, a ModBB
dispersion or propagation run, an azimuth sweep, a batch of served requests,
a receiver-array sum.  `listed()` names the fixed cases, `draw()` gives
further ones of the same ranges.  Atmospheres are those of the served request
stream (`workloads.perturbed_profile`): jets and temperature noise drawn from
the seed, so another seed is another atmosphere.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "ncpaprop-release_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import ncpa_gpu  # noqa: E402
import workloads  # noqa: E402

PI = 3.141592653589793
COARSE = 128  # the mode values' sign: positive at the largest of every 128th grid row


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _modess(freq, nz, n_ranges, dr, n_az=1, wkb=True, group=False, lossless=False, z_src=0.0, z_rcv=0.0):
    return {"kind": "modess", "freq": freq, "nz": nz, "n_ranges": n_ranges, "dr": dr, "n_az": n_az, "wkb": wkb,
            "group": group, "lossless": lossless, "z_src": z_src, "z_rcv": z_rcv}


def _modess2d(freq, nz, n_ranges, dr):
    return {"kind": "modess2d", "freq": freq, "nz": nz, "n_ranges": n_ranges, "dr": dr}


def _modbb(n_freq, f_max, nz, n_ranges, method="ess", n_wave=0):
    return {"kind": "modbb", "n_freq": n_freq, "f_max": f_max, "nz": nz, "n_ranges": n_ranges, "method": method,
            "n_wave": n_wave}


def _sweep(n_az, n_freq, f_lo, f_hi, ppw, n_ranges):
    return {"kind": "sweep", "n_az": n_az, "n_freq": n_freq, "f_lo": f_lo, "f_hi": f_hi, "ppw": ppw,
            "n_ranges": n_ranges}


def _requests(n_req, nz, n_ranges):
    return {"kind": "requests", "n_req": n_req, "nz": nz, "n_ranges": n_ranges}


def _receivers(freq, nz, n_rcv, n_ranges, dr):
    return {"kind": "receivers", "freq": freq, "nz": nz, "n_rcv": n_rcv, "n_ranges": n_ranges, "dr": dr}


def _propagation(n_freq, f_max, n_ranges, nfft, n_wave):
    return {"kind": "propagation", "n_freq": n_freq, "f_max": f_max, "n_ranges": n_ranges, "nfft": nfft,
            "n_wave": n_wave}


def listed():
    named = [
        # the smallest Modess call: low frequency, coarse grid, a short range table (latency)
        ("modess_low", _modess(0.05, 5000, 200, 1000.0)),
        # Modess with its default options: 0.1 Hz, Nz_grid 20000, 1000 ranges
        ("modess_default", _modess(0.1, 20000, 1000, 1000.0)),
        # one high frequency with group speeds (speeds.nm): many modes of one problem
        ("modess_2hz", _modess(2.0, 20000, 2000, 500.0, wkb=False, group=True)),
        # Modess --multiprop: every 10 degrees of azimuth
        ("modess_nx2d", _modess(0.5, 20000, 1000, 1000.0, n_az=36)),
        # Modess --write_2d_tloss: full eigenvectors and the range-height field
        ("modess_2d", _modess2d(0.3, 20000, 1000, 1000.0)),
        # ModBB --dispersion with 1-D TL and pulses at 11 ranges, the broadband benchmark's grid
        ("modbb_256", _modbb(256, 0.5, 20000, 1000, n_wave=11)),
        # a small broadband job on an odd grid
        ("modbb_33", _modbb(33, 0.25, 7013, 333, n_wave=3)),
        # ModBB --dispersion --method wmod
        ("modbb_wmod_64", _modbb(64, 0.5, 20000, 500, method="wmod")),
        # azimuth sweep whose grid follows the wavelength (mixed grids, 5000 to 60000 rows)
        ("sweep_45az", _sweep(45, 8, 0.1, 2.0, 60, 2000)),
        # requests of a server merged in one batch, each with its own atmosphere, frequency and azimuth
        ("requests_32", _requests(32, 20000, 1000)),
        # the field at a vertical array of receivers, in 64 bits as the 2-D TL (the tensor-core sums round in 32
        # bits, where a last place of the modes shows)
        ("receivers_64", _receivers(2.0, 20000, 64, 20000, 100.0)),
        # ModBB --propagation from a dispersion file, the manual's transform length
        ("propagation_256", _propagation(256, 0.5, 11, 16384, 4096)),
    ]
    return [dict(case, name=name) for name, case in named]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the listed ones' ranges; a kind is as likely as it is listed."""
    kind = rng.choice(["modess"] * 4 + ["modess2d"] + ["modbb"] * 3 + ["sweep", "requests", "receivers",
                                                                      "propagation"])
    if kind == "modess":
        n_az = rng.choice([1, 1, 1, rng.randint(2, 36)])
        freq = _log(rng, 0.05, 2.0 if n_az == 1 else 0.5)
        wkb = rng.random() < 0.5
        z = 0.0 if wkb else rng.choice([0.0, round(rng.uniform(0.5, 30.0), 2)])
        return _modess(round(freq, 4), int(_log(rng, 5000, 20000)), int(_log(rng, 100, 2000)),
                       round(rng.uniform(300.0, 1000.0), 1), n_az=n_az, wkb=wkb, group=rng.random() < 0.3,
                       lossless=rng.random() < 0.2, z_src=z, z_rcv=0.0 if z == 0.0 else round(z / 3, 2))
    if kind == "modess2d":
        return _modess2d(round(_log(rng, 0.05, 0.3), 4), int(_log(rng, 5000, 20000)), int(_log(rng, 100, 1000)),
                         round(rng.uniform(300.0, 1000.0), 1))
    if kind == "modbb":
        method = rng.choice(["ess", "ess", "wmod"])
        n = int(_log(rng, 32, 256 if method == "ess" else 64))
        return _modbb(n, round(rng.uniform(0.2, 0.5), 3), int(_log(rng, 5000, 20000)), int(_log(rng, 100, 1000)),
                      method=method, n_wave=rng.randint(1, 11) if method == "ess" else 0)
    if kind == "sweep":
        return _sweep(rng.randint(4, 45), rng.randint(2, 8), round(rng.uniform(0.05, 0.2), 3),
                      round(rng.uniform(0.5, 2.0), 3), rng.randint(30, 60), int(_log(rng, 200, 2000)))
    if kind == "requests":
        return _requests(rng.randint(2, 32), int(_log(rng, 5000, 20000)), int(_log(rng, 200, 1000)))
    if kind == "receivers":
        return _receivers(round(rng.uniform(0.5, 2.0), 3), int(_log(rng, 10000, 20000)), rng.randint(5, 64),
                          int(_log(rng, 500, 20000)), round(rng.uniform(100.0, 500.0), 1))
    n = int(_log(rng, 32, 256))
    nfft = rng.choice([4 * (n + 1), 2048, 4096, 16384])
    return _propagation(n, round(rng.uniform(0.2, 0.5), 3), rng.randint(1, 11), nfft, rng.randint(nfft // 8, nfft // 4))


def _n_modes(freq):
    return 2.0 + 560.0 * freq  # about, on these atmospheres


def work(case):
    """Inputs and outputs once; for the eigen-solves one evaluation of the characteristic polynomial (3
    operations a row) and one pass over the vector with its two integrals (7) for each mode."""
    knots = 6 * 1501 * 8.0
    kind = case["kind"]
    if kind in ("modess", "modess2d"):
        m = _n_modes(case["freq"]) * case.get("n_az", 1)
        b = knots + 40 * m + 24.0 * case["n_ranges"] * case.get("n_az", 1)
        f = m * (10.0 * case["nz"] + 12.0 * case["n_ranges"])
        if kind == "modess2d":
            heights = -(-case["nz"] // max(1, case["nz"] // 500))
            b += 16.0 * heights * case["n_ranges"]
            f += 4.0 * m * heights * case["n_ranges"]
        return {"bytes": b, "flops": f}
    if kind == "modbb":
        m = sum(_n_modes(case["f_max"] * (i + 1) / case["n_freq"]) for i in range(case["n_freq"]))
        nfft = _nfft(case["n_freq"] + 1, 256)
        return {"bytes": knots + 40 * m + 24.0 * case["n_ranges"] * case["n_freq"] + 8.0 * case["n_wave"] * nfft,
                "flops": m * (10.0 * case["nz"] + 12.0 * case["n_ranges"] + 12.0 * case["n_wave"]) +
                case["n_wave"] * 5.0 * nfft * math.log2(nfft)}
    if kind == "sweep":
        fr = workloads.sweep_freqs(case["n_freq"], case["f_lo"], case["f_hi"])
        ms = [_n_modes(f) * case["n_az"] for f in fr]
        nzs = [workloads.sweep_nz(f, points_per_wavelength=case["ppw"]) for f in fr]
        return {"bytes": knots + 40 * sum(ms) + 24.0 * case["n_ranges"] * len(fr) * case["n_az"],
                "flops": sum(m * (10.0 * nz + 12.0 * case["n_ranges"]) for m, nz in zip(ms, nzs))}
    if kind == "requests":
        m = case["n_req"] * _n_modes(0.53)
        return {"bytes": case["n_req"] * knots + 40 * m + 24.0 * case["n_ranges"] * case["n_req"],
                "flops": m * (10.0 * case["nz"] + 12.0 * case["n_ranges"])}
    if kind == "receivers":
        m = _n_modes(case["freq"])
        return {"bytes": 8.0 * m * (case["n_rcv"] + 4) + 16.0 * case["n_rcv"] * case["n_ranges"],
                "flops": 8.0 * m * case["n_rcv"] * case["n_ranges"]}
    m = sum(_n_modes(case["f_max"] * (i + 1) / case["n_freq"]) for i in range(case["n_freq"]))
    return {"bytes": 32 * m + 8.0 * case["n_ranges"] * case["nfft"] + 8.0 * case["n_wave"],
            "flops": 12.0 * m * case["n_ranges"] + case["n_ranges"] * 5.0 * case["nfft"] * math.log2(case["nfft"])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _nfft(nfreq_with_dc, n_wave):
    n = 4 * nfreq_with_dc
    while n_wave > n:
        n *= 2
    return n


_CTX = []


def _context():
    if not _CTX:
        _CTX.append(ncpa_gpu.Context(0))
    return _CTX[0]


class State(dict):
    """What a program keeps between calls: the context, its profiles, the case's inputs."""

    def __del__(self):
        for k in ("modes", "profile"):
            if self.get(k) is not None:
                self[k].close()
        for p in self.get("profiles", ()):
            p.close()


def _inputs(case, seed):
    """Host inputs of a case, from the seed alone."""
    rng = np.random.default_rng([int(seed), 977])
    kind = case["kind"]
    out = {}
    if kind == "requests":
        out["profiles"] = [workloads.perturbed_profile(rng) for _ in range(case["n_req"])]
        out["freqs"] = np.exp(rng.uniform(math.log(0.05), math.log(2.0), case["n_req"]))
        out["az"] = rng.uniform(0.0, 360.0, case["n_req"])
        return out
    if kind == "propagation":
        return _dispersion(case, rng)
    out["profile"] = workloads.perturbed_profile(rng)
    az0 = rng.uniform(0.0, 360.0)
    n_az = case.get("n_az", 1)
    out["az"] = (az0 + np.arange(n_az) * (360.0 / n_az)) % 360.0
    if kind == "receivers":
        out["heights"] = np.sort(rng.uniform(0.0, 100e3, case["n_rcv"]))
    if kind == "modbb":
        t, x = workloads.ricker_waveform()
        out["wave"] = x * rng.uniform(0.5, 2.0)
        out["wave_dt"] = t[1] - t[0]
    return out


def _dispersion(case, rng):
    """A dispersion set as ModBB reads it: phase speeds of a stratified atmosphere, weak attenuation growing with
    frequency and phase speed, mode values of the size a 150 km column gives."""
    n = case["n_freq"]
    f = np.concatenate([[0.0], case["f_max"] / n * np.arange(1, n + 1)])
    counts = np.concatenate([[0], np.maximum(2, np.rint([_n_modes(x) for x in f[1:]])).astype(int)])
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    total = int(off[-1])
    fm = np.repeat(f, counts)
    c = rng.uniform(320.0, 480.0, total)
    order = np.lexsort((-c, fm))
    c = c[order]
    re_k = 2 * PI * fm / c
    im_k = 10.0 ** rng.uniform(-9.0, -5.0, total) * np.maximum(fm, 0.01) * (c / 340.0) ** 4
    v = lambda: rng.standard_normal(total) * 10.0 ** rng.uniform(-5.0, -2.0, total)  # noqa: E731
    dt = 1.0 / (case["nfft"] * (f[2] - f[1]))
    t = np.arange(case["n_wave"]) * dt
    x = np.exp(-0.5 * ((t - t.mean()) / (t[-1] / 8.0)) ** 2) * np.cos(0.4 * PI * case["f_max"] * t +
                                                                     rng.uniform(0.0, 2 * PI))
    return {"f": f, "off": off, "re_k": re_k, "im_k": im_k, "vs": v(), "vr": v(), "rho_src": 1.2,
            "rho_rcv": float(rng.uniform(0.8, 1.2)), "ranges": np.sort(rng.uniform(100e3, 600e3, case["n_ranges"])),
            "max_cel": 340.0, "wave": x, "wave_dt": dt}


def prepare(case, seed):
    ctx = _context()
    s = State(_inputs(case, seed))
    kind = case["kind"]
    s["case"], s["ctx"] = case, ctx
    if kind == "requests":
        s["profiles"] = [ctx.profile_from_arrays(*p) for p in s["profiles"]]
        s["params"] = ncpa_gpu.default_params(nz_grid=case["nz"])
    elif kind != "propagation":
        s["profile"] = ctx.profile_from_arrays(*s["profile"])
    if kind == "modess":
        s["params"] = ncpa_gpu.default_params(nz_grid=case["nz"], turnoff_wkb=0 if case["wkb"] else 1,
                                              want_group_speed=int(case["group"]), sourceheight_km=case["z_src"],
                                              receiverheight_km=case["z_rcv"])
    elif kind == "modess2d":
        s["params"] = ncpa_gpu.default_params(nz_grid=case["nz"], turnoff_wkb=1, want_vectors=1)
    elif kind == "modbb":
        method = ncpa_gpu.METHOD_WMOD if case["method"] == "wmod" else ncpa_gpu.METHOD_ESS
        s["params"] = ncpa_gpu.default_params(nz_grid=case["nz"], turnoff_wkb=1, method=method)
        s["freqs"] = workloads.broadband_freqs(case["n_freq"], case["f_max"])
        s["ranges"] = np.linspace(200e3, 300e3, max(1, case["n_wave"]))
    elif kind == "sweep":
        s["params"] = ncpa_gpu.default_params()
        s["jobs"] = [(s["profile"], [f], s["az"], workloads.sweep_nz(f, points_per_wavelength=case["ppw"]))
                     for f in workloads.sweep_freqs(case["n_freq"], case["f_lo"], case["f_hi"])]
    elif kind == "receivers":
        prm = ncpa_gpu.default_params(nz_grid=case["nz"], turnoff_wkb=1, want_vectors=1, keep_on_device=1)
        s["modes"] = ctx.solve(s["profile"], prm, [case["freq"]], s["az"])
    if kind in ("modess", "modess2d"):
        s["bufs"] = _mode_buffers([case["freq"]], len(s["az"]))
    elif kind == "modbb":
        s["bufs"] = _mode_buffers(s["freqs"], 1)
    elif kind == "requests":
        s["bufs"] = _mode_buffers([2.0], case["n_req"])  # any request may be at the highest frequency
    elif kind == "sweep":
        s["bufs"] = _mode_buffers([j[1][0] for j in s["jobs"]], len(s["az"]))
    return s


def _mode_buffers(freqs, per_freq):
    """Host buffers that a program keeps for the modes of its batch (CSR order, zeros after the last mode)."""
    n = int(sum(40 + 1000.0 * f for f in freqs) * per_freq)
    return [np.zeros(n) for _ in range(5)]


def _modes_out(s, m, group=False):
    off = m.all_modes(out=s["bufs"])[0]
    out = dict(zip(("kr", "ki", "vs", "vr", "vg"), s["bufs"]), off=off)
    if not group:
        del out["vg"]
    return out


def _tl_out(out, tl):
    out["tl_re"], out["tl_im"], out["tl_inc"] = tl
    return out


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "modess":
        m = ctx.solve(s["profile"], s["params"], [case["freq"]], s["az"])
        out = _modes_out(s, m, case["group"])
        _tl_out(out, m.tl1d(case["n_ranges"], case["dr"], lossless=case["lossless"]))
        m.close()
        return out
    if kind == "modess2d":
        m = ctx.solve(s["profile"], s["params"], [case["freq"]], s["az"])
        out = _modes_out(s, m)
        _tl_out(out, m.tl1d(case["n_ranges"], case["dr"]))
        out["z"], out["field_re"], out["field_im"] = m.tl2d(0, case["n_ranges"], case["dr"])
        m.close()
        return out
    if kind == "modbb":
        m = ctx.solve(s["profile"], s["params"], s["freqs"], s["az"])
        out = _modes_out(s, m)
        _tl_out(out, m.tl1d(case["n_ranges"], 1000.0))
        if case["n_wave"]:
            nf = case["n_freq"] + 1
            nfft = _nfft(nf, len(s["wave"]))
            sre, sim = ctx.source_spectrum_waveform(s["wave"], s["wave_dt"], nfft, nf)
            out["wave"] = m.bb_synthesize(s["ranges"], 340.0, nfft, sre, sim)
        m.close()
        return out
    if kind == "sweep":
        m = ctx.solve_jobs(s["jobs"], s["params"])
        out = _tl_out(_modes_out(s, m), m.tl1d(case["n_ranges"], 500.0))
        m.close()
        return out
    if kind == "requests":
        jobs = [(p, [f], a) for p, f, a in zip(s["profiles"], s["freqs"], s["az"])]
        m = ctx.solve_jobs(jobs, s["params"])
        out = _tl_out(_modes_out(s, m), m.tl1d(case["n_ranges"], 500.0))
        m.close()
        return out
    if kind == "receivers":
        return s["modes"].tl_multi(0, s["heights"], case["n_ranges"], case["dr"], method=ncpa_gpu.Modes.SUM_FP64)
    nf = case["n_freq"] + 1
    sre, sim = ctx.source_spectrum_waveform(s["wave"], s["wave_dt"], case["nfft"], nf)
    w = ctx.bb_synthesize(s["f"], s["off"], s["re_k"], s["im_k"], s["vs"], s["vr"], s["rho_src"], s["rho_rcv"],
                          s["ranges"], s["max_cel"], case["nfft"], sre, sim)
    return {"src_re": sre, "src_im": sim, "wave": w}


# ---------------------------------------------------------------------------
# the same in plain numpy, in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "propagation":
        return _exact_propagation(case, _inputs(case, seed))
    # one problem of a few hundred modes at most: about ten seconds of row-by-row numpy
    if kind == "modess" and case["n_az"] == 1 and case["nz"] * case["freq"] <= 8000.0:
        return _exact_modess(case, _inputs(case, seed))
    return None


def _exact_propagation(case, s):
    n, nfft = case["n_freq"] + 1, case["nfft"]
    t = np.arange(len(s["wave"]))
    e = np.exp(2j * PI * ((np.arange(n)[:, None] * t) % nfft) / nfft)
    src = s["wave_dt"] * (e @ s["wave"])
    f, off = s["f"], s["off"]
    k = s["re_k"] + 1j * s["im_k"]
    amp = s["vs"] * s["vr"] / np.sqrt(k)
    which = np.repeat(np.arange(n), np.diff(off))
    smooth = int(math.floor(0.1 * n))
    taper = np.ones(n)
    if smooth > 0:
        b, last = n - smooth, n - 1
        taper[b:] = 1.0 if last == b else 0.5 * (np.cos(PI * (np.arange(b, n) - b) / (last - b)) + 1.0)
    out = np.empty((case["n_ranges"], nfft))
    for i, r in enumerate(s["ranges"]):
        terms = amp * np.exp(1j * k * r)
        h = np.bincount(which, terms.real, n) + 1j * np.bincount(which, terms.imag, n)
        h = h * taper * (1j * np.exp(-0.25j * PI) / np.sqrt(8 * PI * r) * np.sqrt(s["rho_rcv"] / s["rho_src"]))
        a = np.exp(-2j * PI * f * (r / s["max_cel"])) * src * h
        out[i] = 2.0 * (f[2] - f[1]) * np.fft.fft(a, nfft).real
    return {"src_re": src.real, "src_im": src.imag, "wave": out}


def _steffen(x, y):
    """Steffen's monotone cubic: (values at x) -> function."""
    h = np.diff(x)
    s = np.diff(y) / h
    p = (s[:-1] * h[1:] + s[1:] * h[:-1]) / (h[:-1] + h[1:])
    lim = np.minimum(np.minimum(np.abs(s[:-1]), np.abs(s[1:])), 0.5 * np.abs(p))
    sgn = lambda v: np.where(v < 0, -1.0, 1.0)  # noqa: E731
    d = np.concatenate([[s[0]], (sgn(s[:-1]) + sgn(s[1:])) * lim, [s[-1]]])
    a, b = (d[:-1] + d[1:] - 2 * s) / h / h, (3 * s - 2 * d[:-1] - d[1:]) / h

    def at(q):
        i = np.clip(np.searchsorted(x, q, side="right") - 1, 0, len(x) - 2)
        t = q - x[i]
        v = y[i] + t * (d[i] + t * (b[i] + t * a[i]))
        return np.where(q > x[-1], y[-1], np.where(q < x[0], y[0], v))

    return at


def _absorption(z, t, p, rho, f):
    """Sutherland and Bass's atmospheric absorption [Np/m]; z in km."""
    def ten(*c):  # each fit is used below or above its height, where its exponent is small
        return 10.0 ** np.minimum(sum(ck * z ** i for i, ck in enumerate(c)), 300.0)

    x = [np.where(z > 90, ten(49.296, -1.5524, 1.8714e-2, -1.1069e-4, 3.199e-7, -3.6211e-10), 10 ** -0.67887),
         np.where(z > 76, ten(1.3972e-1, -5.6269e-3, 3.9407e-5, -1.0737e-7), 10 ** -0.10744),
         10 ** -3.3979,
         np.where(z > 80, ten(-4.234, -3.0975e-2),
                  ten(-19.027, 1.3093, -4.6496e-2, 7.8543e-4, -6.5169e-6, 2.1343e-8)),
         np.where(z > 95, ten(-3.2456, 4.6642e-2, -2.6894e-4, 5.264e-7),
                  ten(-11.195, 1.5408e-1, -1.4348e-3, 1.0166e-5)),
         ten(-53.746, 1.5439, -1.8824e-2, 1.1587e-4, -3.5399e-7, 4.2609e-10),
         np.where(z > 30, ten(-4.2563, 7.6245e-2, -2.1824e-3, -2.3010e-6, 2.4265e-7, -1.25e-9),
                  ten(-1.7491, 4.4986e-2, -6.8549e-2, 5.4639e-3, -1.5539e-4, 1.5063e-6))]
    c = np.sqrt(1.4 * p / rho)
    mu_o = 18.192e-6
    mu = mu_o * np.sqrt(t / 293.15) * ((1 + 117.0 / 293.15) / (1 + 117.0 / t))
    nu = 8 * PI * mu * f / (3 * p)
    zr = 1.0 / (x[1] / (63.3 * np.exp(-16.7 * t ** (-1 / 3))) + x[0] / (54.1 * np.exp(-17.3 * t ** (-1 / 3))))
    sigma = 5.0 / math.sqrt(21.0)
    chi = 3.0 * ((4.0 / 5.0) * math.sqrt(3.0 / 7.0) * zr) * nu / 4.0
    cc = 2.36 * chi
    root = np.sqrt(1 + nu ** 2)
    kf = 2 * PI * f / c
    a_cl = kf * np.sqrt(0.5 * (root - 1) * (1 + cc ** 2) / ((1 + nu ** 2) * (1 + (sigma * cc) ** 2)))
    a_rot = kf * ((x[0] + x[1]) / 0.9903) * ((sigma ** 2 - 1) * chi / (2 * sigma)) * \
        np.sqrt(0.5 * (root + 1) / ((1 + nu ** 2) * (1 + cc ** 2)))
    tr = (t / 293.15) ** (-1 / 3) - 1.0
    hu = 100.0 * (x[3] + x[6])
    pf = (p / 101325.0) * (mu_o / mu)
    relax = [pf * ((x[0] + x[1]) * 24.0 * np.exp(-9.16 * tr) + (x[4] + x[5]) * 2400.0 +
                   40400.0 * np.exp(10.0 * tr) * hu * (0.02 * np.exp(-11.2 * tr) + hu) *
                   (0.391 * np.exp(8.41 * tr) + hu)),
             pf * (9.0 * np.exp(-19.9 * tr) + 60000.0 * x[3] + 28000.0 * np.exp(-4.17 * tr) * x[6]),
             pf * (22000.0 * np.exp(-7.68 * tr) * x[2] + 15100.0 * np.exp(-10.4 * tr) * (x[0] + 0.5 * x[4]) +
                   11500.0 * np.exp(-9.17 * tr) * (x[1] + 0.5 * x[5]) +
                   8.48e8 * np.exp(9.17 * tr) * (x[6] + x[3])),
             pf * 1.2e5 * np.exp(-7.72 * tr)]
    a = a_cl + a_rot + 0.003 * a_cl
    for xm, fv, th, cp, cv in zip(x, relax, (2239.1, 3352.0, 915.0, 1037.0), (3.5, 3.5, 4.0, 4.0),
                                  (2.5, 2.5, 3.0, 3.0)):
        et = np.exp(-th / t)
        cr = (th / t) ** 2 * et / (1 - et) ** 2
        a = a + xm * (PI / 2) * cr / (cp * (cv + cr)) / c * (2 * f * f / fv) / (1 + (f / fv) ** 2)
    return a


def _sturm(s, x):
    """Eigenvalues of diag(s) + unit off-diagonals below each x."""
    d = np.full(len(x), np.inf)
    n = np.zeros(len(x), dtype=np.int64)
    tiny = np.finfo(float).tiny ** 0.5
    for si in s:
        d = (si - x) - 1.0 / d
        d[d == 0.0] = tiny
        n += d < 0
    return n


def _eigen(s, lo, hi):
    """Eigenvalues in [lo, hi) by counting, and for each the vector of the twisted factorisation."""
    c_lo, c_hi = _sturm(s, np.array([lo, hi]))
    m = int(c_hi - c_lo)
    j = c_lo + np.arange(m)
    a, b = np.full(m, lo), np.full(m, hi)
    pieces = np.arange(1, 16) / 16.0
    while np.max(b - a) > 4e-18 + 1e-15 * hi:
        x = a[:, None] + (b - a)[:, None] * pieces
        below = (_sturm(s, x.ravel()).reshape(x.shape) <= j[:, None]).sum(axis=1)
        edges = np.concatenate([a[:, None], x, b[:, None]], axis=1)
        a, b = edges[np.arange(m), below], edges[np.arange(m), below + 1]
    x = 0.5 * (a + b)
    n = len(s)
    with np.errstate(divide="ignore", over="ignore", under="ignore"):
        for last in (False, True):
            up, dn = np.empty((n, m)), np.empty((n, m))
            d = np.full(m, np.inf)
            for i in range(n):
                d = (s[i] - x) - 1.0 / d
                up[i] = d
            d = np.full(m, np.inf)
            for i in range(n - 1, -1, -1):
                d = (s[i] - x) - 1.0 / d
                dn[i] = d
            gam = up + dn - (s[:, None] - x)
            r = np.argmin(np.abs(gam), axis=0)
            z = np.zeros((n, m))
            z[r, np.arange(m)] = 1.0
            for i in range(n - 2, -1, -1):
                z[i] = np.where(i < r, -z[i + 1] / up[i], z[i])
            for i in range(1, n):
                z[i] = np.where(i > r, -z[i - 1] / dn[i], z[i])
            if not last:  # Rayleigh quotient
                x = x + gam[r, np.arange(m)] / (z * z).sum(axis=0)
    rows = np.arange(0, n, COARSE)
    at = rows[np.argmax(np.abs(z[rows]), axis=0)]
    return x, z * np.sign(z[at, np.arange(m)])


def _exact_modess(case, s):
    zk, u, v, t, p, rho = s["profile"]
    nz, f = case["nz"], case["freq"]
    w = 2 * PI * f
    top = min(150e3, zk[-1] - 1e-6)
    dz = top / (nz - 1)
    z = np.arange(nz) * dz
    c0 = np.sqrt(1.4 * p / rho)
    wd = (PI / 2 - np.arctan2(v, u)) * 180.0 / PI
    c = _steffen(zk, np.hypot(u, v) * np.cos(wd * PI / 180.0 - s["az"][0] * PI / 180.0) + c0)(z)
    kk = (w / c) ** 2
    d = kk.copy()
    d[0] += 1.0 / dz ** 2
    d[-1] = kk[-2]
    diag = d * dz ** 2 - 2.0
    k_min, k_full = w / c[nz - nz // 10 + 1], w / c.min()
    k_max = k_full
    if case["wkb"]:
        k2, step = kk[0], (k_full ** 2 - kk[0]) / 100.0
        if step > 1e-10:
            while k2 < k_full ** 2:
                term = np.abs(k2 - kk)
                stop = np.flatnonzero(term <= step)
                n = stop[0] + 1 if len(stop) else nz
                if np.cumsum(dz * np.sqrt(term[:n]))[-1] >= 10.0:
                    break
                k2 = k2 + step
        k_max = math.sqrt(k2) if math.sqrt(k2) >= k_min else k_full
    x, vec = _eigen(diag, k_min ** 2 * dz ** 2, k_max ** 2 * dz ** 2)
    nrm = (vec ** 2).sum(axis=0)
    ct = np.sqrt(1.4 * _steffen(zk, p)(z) / _steffen(zk, rho)(z))
    wt = w / ct * _steffen(zk, _absorption(zk * 0.001, t, p, rho, f))(z) * 2
    k = np.sqrt(x / dz ** 2 + 1j * ((vec ** 2 * wt[:, None]).sum(axis=0) / nrm))
    vec = vec / np.sqrt(nrm * dz)
    i_s, i_r = (int(math.ceil(case[q] * 1000.0 / dz)) for q in ("z_src", "z_rcv"))
    out = {"kr": k.real, "ki": k.imag, "vs": vec[i_s], "vr": vec[i_r]}
    if case["group"]:
        out["vg"] = k.real / (w * (vec ** 2 / c[:, None] ** 2).sum(axis=0) * dz)
    size = len(_mode_buffers([f], 1)[0])
    out = {q: np.concatenate([a, np.zeros(size - len(a))]) for q, a in out.items()}
    out["off"] = None
    r = (np.arange(case["n_ranges"]) + 1) * case["dr"]
    kt = k.real + 0j if case["lossless"] else k
    e = np.exp(1j * kt * r[:, None])
    vv = vec[i_s] * vec[i_r]
    tl = 1000.0 * 4 * PI * 1j * np.exp(-0.25j * PI) / np.sqrt(8 * PI * r) * (e @ (vv / np.sqrt(kt)))
    inc = 1000.0 * 4 * PI * np.sqrt((np.abs(e) ** 2) @ (vv ** 2 / np.abs(kt))) / np.sqrt(8 * PI * r)
    out["tl_re"], out["tl_im"], out["tl_inc"] = tl.real[None], tl.imag[None], inc[None]
    return out
