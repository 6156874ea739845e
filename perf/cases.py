"""Performance cases: the work that movie registration has the library do.

``listed()`` names the workloads that the configurations, tests and benchmark of
this repository run: a 40-frame K2 counting movie (3838 x 3710 uint8, padded to
4096, cropped to 2048, maxShift 100), 20 frames of 1024 x 1024 float32, K3
super-resolution frames binned 2x, and the small movies of the tests.  Two of
them are whole registrations through ``ImageRegistrator.alignImageStack``; the
others are its stages through the C ABI, with the inputs a registration gives
them.  ``draw(rng)`` gives more of the same stages over the sizes, pixel types
and options that the entry points take.

Every case has a ``stage``; ``prepare``, ``run``, ``exact`` and ``work`` look up
the functions of that stage.
"""
import ctypes
import math

import numpy as np
import torch

from zorro_gb300 import _lib
from zorro_gb300 import hostmath
from zorro_gb300.registrator import ImageRegistrator

DEV = "cuda"
TYPES = {"f32": (torch.float32, _lib.ZR_F32, 4), "u8": (torch.uint8, _lib.ZR_U8, 1),
         "f16": (torch.float16, _lib.ZR_F16, 2)}
PADDED = (64, 128, 256, 512, 1024, 1536, 2048, 3072, 4096, 6144)
CROPS = (64, 128, 256, 384, 512, 768, 1024, 1536, 2048, 3072, 4096)
DOSE = [1.2 * 1.05 ** 2, 0.24499, -1.6649, 2.8141, 32, 0]


def listed():
    return [
        # a small movie from host arrays to host results: launches and host steps count
        {"name": "align small", "stage": "align", "N": 20, "H": 200, "W": 180, "P": 256, "C": 128, "mS": 20,
         "type": "f32", "hot": False, "device": False, "dose": 4.0},
        # the movie a K2 camera delivers, raw counts on the GPU, with the hot-pixel and dose filters
        {"name": "align k2", "stage": "align", "N": 40, "H": 3838, "W": 3710, "P": 4096, "C": 2048, "mS": 100,
         "type": "u8", "hot": True, "device": True, "dose": 0.8},
        # gain correction, unaligned sum, its histogram and the hot-pixel maps of that movie
        {"name": "hotpix k2", "stage": "hotpix", "N": 40, "H": 3838, "W": 3710, "type": "u8", "gain": True},
        # forward spectra of one chunk of its frames
        {"name": "spectra k2", "stage": "spectra", "N": 8, "H": 3838, "W": 3710, "P0": 4096, "P1": 4096, "C0": 2048,
         "C1": 2048, "type": "u8", "gain": True, "hot": True},
        # spectra, frame terms and all pair windows of 20 float32 frames of 1024 x 1024
        {"name": "correlate 1024", "stage": "correlate", "N": 20, "H": 1024, "W": 1024, "P": 1024, "C": 1024, "mS": 40,
         "type": "f32"},
        # frame terms and the 190 pair windows of a 20-frame half set of the K2 movie
        {"name": "pairs k2", "stage": "pairs", "N": 20, "H": 3838, "W": 3710, "P": 4096, "C": 2048, "mS": 100},
        # the peak search on those windows
        {"name": "peaks k2", "stage": "peaks", "M": 190, "mS": 100, "bmode": 1},
        # the peak search on the single window of a pair of half sums
        {"name": "peaks one", "stage": "peaks", "M": 1, "mS": 100, "bmode": 1},
        # rolled, Lanczos-shifted frames of the K2 movie and their sum
        {"name": "shift k2", "stage": "shift", "N": 40, "H": 3838, "W": 3710, "type": "u8", "gain": True, "hot": True,
         "halves": False, "aligned": True, "drift": 12.0},
        # dose-weighted sum of the K2 movie's aligned frames
        {"name": "dose k2", "stage": "dose", "N": 40, "H": 3838, "W": 3710, "P": 4096, "norm": False},
        # tiled Fourier ring correlation of the K2 movie's half sums
        {"name": "frc k2", "stage": "frc", "H": 3838, "W": 3710},
        # Fourier binning of K3 super-resolution frames
        {"name": "binning k3", "stage": "bin", "N": 2, "H": 8184, "W": 11520, "Hb": 4092, "Wb": 5760, "type": "u8"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    stage = rng.choice(["align", "hotpix", "spectra", "correlate", "pairs", "peaks", "peaks", "shift", "dose", "frc",
                        "bin"])
    kind = rng.choice(["u8", "f32", "f16"])
    H, W = _log(rng, 64, 4096), _log(rng, 64, 4096)
    if stage == "align":
        P = rng.choice([256, 512, 1024])
        return {"stage": stage, "N": rng.randint(16, 28), "H": _log(rng, 0.6 * P, P), "W": _log(rng, 0.6 * P, P),
                "P": P, "C": P // 2, "mS": rng.randint(16, 32), "type": "f32", "hot": False,
                "device": rng.random() < 0.5, "dose": 4.0}
    if stage == "hotpix":
        return {"stage": stage, "N": _log(rng, 2, 40), "H": max(H, 128), "W": max(W, 128), "type": kind,
                "gain": rng.random() < 0.7}
    if stage == "spectra":
        P0, P1 = (min(p for p in PADDED if p >= v) for v in (H, W))
        C0, C1 = (rng.choice([c for c in CROPS if p // 4 <= c <= p and c >= 64]) for p in (P0, P1))
        return {"stage": stage, "N": _log(rng, 1, 8), "H": H, "W": W, "P0": P0, "P1": P1, "C0": C0, "C1": C1,
                "type": kind, "gain": kind != "f32" and rng.random() < 0.7, "hot": rng.random() < 0.5}
    if stage in ("correlate", "pairs"):
        C = rng.choice(CROPS[:9])
        P = min(p for p in PADDED if p >= C and p >= rng.choice([C, 2 * C]))
        N = _log(rng, 2, 20)
        case = {"stage": stage, "N": N, "H": _log(rng, 0.7 * P, P), "W": _log(rng, 0.7 * P, P), "P": P, "C": C,
                "mS": rng.randint(8, max(8, min(100, C // 4)))}
        return dict(case, type=kind) if stage == "correlate" else case
    if stage == "peaks":
        return {"stage": stage, "M": _log(rng, 1, 190), "mS": _log(rng, 8, 112), "bmode": rng.choice([1, 1, 1, 2])}
    if stage == "shift":
        return {"stage": stage, "N": _log(rng, 2, 40), "H": H, "W": W, "type": kind,
                "gain": kind != "f32" and rng.random() < 0.7, "hot": rng.random() < 0.5,
                "halves": rng.random() < 0.4, "aligned": rng.random() < 0.6, "drift": rng.uniform(0.5, 20.0)}
    if stage == "dose":
        P = rng.choice([256, 512, 1024, 1536, 2048, 3072, 4096])
        return {"stage": stage, "N": _log(rng, 2, 40), "H": _log(rng, 0.6 * P, P), "W": _log(rng, 0.6 * P, P), "P": P,
                "norm": rng.random() < 0.3}
    if stage == "frc":
        return {"stage": stage, "H": _log(rng, 1100, 4096), "W": _log(rng, 1100, 4096)}
    H, W = _log(rng, 1100, 8192), _log(rng, 1100, 8192)
    s = rng.uniform(1.3, 2.0)
    return {"stage": stage, "N": rng.randint(1, 2), "H": H, "W": W, "Hb": 2 * int(H / s / 2), "Wb": 2 * int(W / s / 2),
            "type": kind}


def prepare(case, seed):
    lib = _lib.load()
    _lib.call("zr_init", torch.cuda.current_device())
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    state = {"case": case, "lib": lib, "stage": case["stage"]}
    STAGES[case["stage"]][0](case, g, state)
    return state


def run(state):
    return STAGES[state["stage"]][1](state)


def exact(case, seed):
    make = STAGES[case["stage"]][2]
    return None if make is None else make(case, prepare(case, seed))


def work(case):
    return STAGES[case["stage"]][3](case)


# ------------------------------------------------------------------ inputs

def _drift(N, sigma, g):
    """A random walk with jitter, centred (y, x per frame)."""
    step = torch.randn(N, 2, generator=g, device=DEV, dtype=torch.float64) * sigma
    d = torch.cumsum(step, 0) + 0.1 * torch.randn(N, 2, generator=g, device=DEV, dtype=torch.float64)
    return (d - d.mean(0)).cpu().numpy()


def _movie(N, H, W, kind, g, dose=0.8, sigma=1.0, gain=None, hot=0.0):
    """Poisson counts of a drifting band-limited specimen (the recipe of
    zorro_gb300.synthetic on the GPU), with a fraction of hot pixels."""
    drift = _drift(N, sigma, g)
    pad = int(np.ceil(np.abs(drift).max())) + 4
    cy, cx = H + 2 * pad, W + 2 * pad
    fy = torch.fft.fftfreq(cy, device=DEV)[:, None]
    fx = torch.fft.rfftfreq(cx, device=DEV)[None, :]
    S = torch.fft.rfft2(torch.randn(cy, cx, generator=g, device=DEV)) * torch.exp(-(fy * fy + fx * fx) / (2 * 0.0625 ** 2))
    field = torch.fft.irfft2(S, s=(cy, cx))
    S = torch.fft.rfft2(1.0 + 0.1 * field / field.std())
    out = torch.empty((N, H, W), dtype=TYPES[kind][0], device=DEV)
    for n in range(N):
        ph = -2.0 * math.pi * (fy * float(drift[n, 0]) + fx * float(drift[n, 1]))
        lam = dose * torch.fft.irfft2(S * torch.polar(torch.ones_like(ph), ph), s=(cy, cx))[pad:pad + H, pad:pad + W]
        lam = lam.clamp_(min=0.0) if gain is None else lam.clamp_(min=0.0) / gain
        c = torch.poisson(lam, generator=g)
        out[n] = c.clamp_(max=255.0) if kind == "u8" else c
    if hot:
        where = torch.randint(0, H * W, (max(1, int(hot * H * W)),), generator=g, device=DEV)
        out.view(N, -1)[:, where] = round(50 * dose)
    return out


def _gain(H, W, g):
    return 0.9 + 0.2 * torch.rand(H, W, generator=g, device=DEV)


def _hot_maps(H, W, mean, g):
    """Maps a, b of the outlier filter: nearly 1 and 0, a few pixels replaced."""
    a = 1.0 - 1e-3 * torch.rand(H, W, generator=g, device=DEV)
    where = torch.randint(0, H * W, (max(1, H * W // 10000),), generator=g, device=DEV)
    a.view(-1)[where] = 1e-3 * torch.rand(where.numel(), generator=g, device=DEV)
    return a, (1.0 - a) * mean


def _frames(raw, kind, gain=None, ha=None, hb=None):
    N, H, W = raw.shape
    return _lib.Frames(raw.data_ptr(), TYPES[kind][1], *(None if t is None else t.data_ptr() for t in (gain, ha, hb)),
                       0.0, N, H, W, 0)


def _counts(case, g, state):
    """Raw frames with the maps that the case asks for."""
    H, W = case["H"], case["W"]
    gain = _gain(H, W, g) if case.get("gain") else None
    raw = _movie(case["N"], H, W, case["type"], g, gain=gain, hot=1e-4 if case["stage"] == "hotpix" else 0.0)
    ha, hb = _hot_maps(H, W, 0.8, g) if case.get("hot") else (None, None)
    state.update(raw=raw, gain=gain, ha=ha, hb=hb, frames=_frames(raw, case["type"], gain, ha, hb))


def _corrected64(state, n):
    v = state["raw"][n].double()
    if state.get("gain") is not None:
        v = v * state["gain"].double()
    if state.get("ha") is not None:
        v = v * state["ha"].double() + state["hb"].double()
    return v


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _bytes(n):
    return torch.empty(max(int(n), 16), dtype=torch.uint8, device=DEV)


def _map_bytes(case):
    return case["H"] * case["W"] * (4 * bool(case.get("gain")) + 8 * bool(case.get("hot")))


def _fft_flops(n, length):
    return 5.0 * n * length * math.log2(length)


# ------------------------------------------------------------------ whole registrations

def _align_prepare(case, g, state):
    gain = _gain(case["H"], case["W"], g) if case["hot"] else None
    raw = _movie(case["N"], case["H"], case["W"], case["type"], g, dose=case["dose"], gain=gain,
                 hot=1e-4 if case["hot"] else 0.0)
    if not case["device"]:
        raw, gain = raw.cpu().numpy(), None if gain is None else gain.cpu().numpy()
    state.update(raw=raw, gain=gain)


def _align_run(state):
    case = state["case"]
    reg = ImageRegistrator()
    reg.images, reg.gainRef = state["raw"], state["gain"]
    reg.triMode, reg.shapePadded, reg.fouCrop = "tri", [case["P"], case["P"]], [case["C"], case["C"]]
    reg.maxShift, reg.pixelsize = case["mS"], 0.105
    reg.filterMode, reg.doseFiltParam = "hot,dose" if case["hot"] else "dose", list(DOSE)
    reg.returnDeviceArrays = case["device"]
    reg.keepAlignedImages = not case["device"]
    reg.alignImageStack()
    out = {"translations": reg.translations, "imageSum": reg.imageSum, "filtSum": reg.filtSum}
    if reg.FRC is not None and min(case["H"], case["W"]) > 1100:
        out.update(FRC=reg.FRC, FRC2D=reg.FRC2D)
    if reg.keepAlignedImages:
        out["images"] = reg.images
    return out


def _align_work(case):
    N, HW, C, P = case["N"], case["H"] * case["W"], case["C"], case["P"]
    M = N * (N - 1) // 2
    flops = N * 2 * (_fft_flops(P, P) + _fft_flops(C // 2, P)) + M * _fft_flops(C // 2 + case["mS"], C)
    return {"bytes": HW * (N * TYPES[case["type"]][2] + 8), "flops": flops + N * 0.5 * (_fft_flops(P, P) * 2)}


# ------------------------------------------------------------------ hot pixels

def _hotpix_prepare(case, g, state):
    _counts(case, g, state)
    N, H, W = case["N"], case["H"], case["W"]
    mean = sum(float(_corrected64(state, n).mean()) for n in range(N))
    _, std, edges = hostmath.hotpix_bins(mean, 8.0)
    p = _lib.HotpixParams()
    p.mu, p.sigma, p.cutoff_lower, p.cutoff_upper = mean, float(std), -4.0, 3.25
    p.logistic_k, p.relax, p.neighbour_thres, p.best_mean = 6.0, 0.925, 0.01, mean / N
    for i, v in enumerate(hostmath.psf_kernel("K2").ravel()):
        p.psf[i] = float(v)
    wb = state["lib"].zr_hotpix_work_bytes(H, W)
    state.update(params=p, edges=edges, sum=torch.empty(H, W, device=DEV), a=torch.empty(H, W, device=DEV),
                 b=torch.empty(H, W, device=DEV), work=_bytes(wb), wb=wb,
                 total=torch.zeros(1, dtype=torch.float64, device=DEV),
                 hist=torch.zeros(len(edges) - 1, dtype=torch.int32, device=DEV),
                 counts=torch.zeros(4, dtype=torch.int32, device=DEV))


def _hotpix_run(s):
    H, W, st = s["case"]["H"], s["case"]["W"], _stream()
    s["total"].zero_()
    s["hist"].zero_()
    s["counts"].zero_()
    _lib.call("zr_gain_sum", ctypes.byref(s["frames"]), s["sum"].data_ptr(), s["total"].data_ptr(), st)
    _lib.call("zr_histogram", s["sum"].data_ptr(), H * W, float(s["edges"][0]), len(s["edges"]) - 1,
              s["hist"].data_ptr(), st)
    _lib.call("zr_hotpix_maps", s["sum"].data_ptr(), H, W, s["case"]["N"], ctypes.byref(s["params"]),
              s["a"].data_ptr(), s["b"].data_ptr(), s["counts"].data_ptr(), s["work"].data_ptr(), s["wb"], st)
    return {"sum": s["sum"], "total": s["total"], "hist": s["hist"], "a": s["a"], "b": s["b"], "counts": s["counts"][:3]}


def _hotpix_exact(case, s):
    total = sum(_corrected64(s, n) for n in range(case["N"]))
    p = s["params"]
    sg = (total - p.mu) / p.sigma
    e1 = torch.exp(p.logistic_k * (sg - p.cutoff_lower * p.relax))
    e2 = torch.exp(p.logistic_k * (sg - p.cutoff_upper * p.relax))
    a = (1.0 - 1.0 / (1.0 + e1)) / (1.0 + e2)
    # the map b and the counts hang on thresholds
    return {"sum": total, "total": total.sum().reshape(1), "hist": None, "a": a, "b": None, "counts": None}


def _hotpix_work(case):
    HW = case["H"] * case["W"]
    return {"bytes": HW * (case["N"] * TYPES[case["type"]][2] + 4 * bool(case["gain"]) + 12),
            "flops": HW * (2.0 * case["N"] + 60)}


# ------------------------------------------------------------------ spectra

def _spectra_prepare(case, g, state):
    _counts(case, g, state)
    lib = state["lib"]
    C0, C1, N = case["C0"], case["C1"], case["N"]
    K4 = lib.zr_spectrum_pitch(C1)
    wb = lib.zr_spectra_work_bytes(case["H"], N, C1)
    mean = torch.stack([_corrected64(state, n).sum() for n in range(N)])
    state.update(mean=mean, G=torch.empty(N, K4, C0 + 4, 2, device=DEV), S=torch.empty(N, K4, C0 + 4, 2, device=DEV),
                 work=_bytes(wb), wb=wb)


def _spectra_run(s):
    c = s["case"]
    _lib.call("zr_spectra", ctypes.byref(s["frames"]), None, s["mean"].data_ptr(), 0, c["N"], 0, c["P0"], c["P1"],
              c["C0"], c["C1"], s["G"].data_ptr(), s["S"].data_ptr(), s["work"].data_ptr(), s["wb"], _stream())
    return {"G": s["G"], "S": s["S"]}


def _layout(F, P0, C0, C1, K4):
    """The library's spectrum layout [K4][C0 + 4] of a P0 x (P1/2 + 1) half spectrum."""
    rows = [r if r < C0 // 2 else P0 - C0 + r for r in range(C0)] + [C0 // 2]
    out = torch.zeros(K4, C0 + 4, dtype=torch.complex128, device=DEV)
    out[:C1 // 2 + 1, :C0 + 1] = F[torch.tensor(rows, device=DEV)][:, :C1 // 2 + 1].T
    return out


def _half_spectra64(v, mu, P0, P1, C0, C1, K4):
    """Layouts of the transforms of (v - mu) and (v - mu)^2 inside the frame."""
    u = torch.zeros(P0, P1, dtype=torch.float64, device=DEV)
    u[:v.shape[0], :v.shape[1]] = v - mu
    return _layout(torch.fft.rfft2(u), P0, C0, C1, K4), _layout(torch.fft.rfft2(u * u), P0, C0, C1, K4)


def _spectra_exact(case, s):
    K4 = s["G"].shape[1]
    out = torch.empty(2, case["N"], K4, case["C0"] + 4, 2, dtype=torch.float64, device=DEV)
    for n in range(case["N"]):
        mu = float(np.float32(float(s["mean"][n]) / (case["H"] * case["W"])))
        gs = _half_spectra64(_corrected64(s, n), mu, case["P0"], case["P1"], case["C0"], case["C1"], K4)
        for i in (0, 1):
            out[i, n] = torch.view_as_real(gs[i])
    return {"G": out[0], "S": out[1]}


def _spectra_work(case):
    N, H, C0, C1 = case["N"], case["H"], case["C0"], case["C1"]
    b = N * H * case["W"] * TYPES[case["type"]][2] + _map_bytes(case) + 2 * N * C0 * (C1 // 2 + 1) * 8
    return {"bytes": b, "flops": N * (_fft_flops(H, case["P1"]) + 2 * _fft_flops(C1 // 2 + 1, case["P0"]))}


# ------------------------------------------------------------------ pair correlation windows

def _pairs_buffers(case, state):
    lib = state["lib"]
    N, C, w = case["N"], case["C"], 2 * case["mS"]
    pairs = np.array([(i, j) for i in range(N) for j in range(i + 1, N)], dtype=np.int32)
    xw = min(1536 << 20, lib.zr_xcorr_work_bytes(len(pairs) + 2 * N + 1, C, case["mS"]))
    state.update(pairs=torch.from_numpy(pairs.reshape(-1)).to(DEV), M=len(pairs), xw=xw, xwork=_bytes(xw),
                 terms=torch.empty(4 * N + 1, w, w, device=DEV), windows=torch.empty(len(pairs), w, w, device=DEV))


def _pairs_calls(s):
    c = s["case"]
    st = _stream()
    size = (c["N"], c["C"], c["C"], c["mS"])
    _lib.call("zr_xcorr_terms", s["G"].data_ptr(), s["S"].data_ptr(), s["GM"].data_ptr(), *size,
              s["terms"].data_ptr(), s["xwork"].data_ptr(), s["xw"], st)
    _lib.call("zr_xcorr_pairs", s["G"].data_ptr(), s["terms"].data_ptr(), s["pairs"].data_ptr(), s["M"], *size,
              s["windows"].data_ptr(), s["xwork"].data_ptr(), s["xw"], st)


def _pairs_prepare(case, g, state):
    N, H, W, P, C = case["N"], case["H"], case["W"], case["P"], case["C"]
    raw = _movie(N, H, W, "f32", g)
    K4 = state["lib"].zr_spectrum_pitch(C)
    GS = torch.empty(2, N, K4, C + 4, 2, device=DEV)
    for n in range(N):
        v = raw[n].double()
        for i, F in enumerate(_half_spectra64(v, v.mean(), P, P, C, C, K4)):
            GS[i, n] = torch.view_as_real(F).float()
    ones = torch.ones(H, W, dtype=torch.float64, device=DEV)
    GM = torch.view_as_real(_half_spectra64(ones, 0.0, P, P, C, C, K4)[0]).float()
    state.update(G=GS[0], S=GS[1], GM=GM)
    _pairs_buffers(case, state)


def _pairs_run(s):
    _pairs_calls(s)
    return {"terms": s["terms"], "windows": s["windows"]}


def _full64(layout, C):
    """The C x C cropped spectrum of one layout [K4][C + 4] (complex)."""
    half = C // 2
    A = torch.empty(C, C, dtype=torch.complex128, device=DEV)
    A[:, :half] = layout[:half, :C].T
    mirror = torch.tensor([0] + [C if r == half else C - r for r in range(1, C)], device=DEV)
    A[:, half:] = layout[1:half + 1].flip(0)[:, mirror].T.conj()  # columns -C/2 .. -1
    return A


def _windows64(G, S, GM, case, pairs):
    """mnxc2's terms and windows from complex layouts."""
    C, N, mS = case["C"], case["N"], case["mS"]
    w = 2 * mS
    scale = 1.0 / float(C) ** 4
    idx = torch.arange(-mS, mS, device=DEV)

    def window(p, sign=1):
        return p[(sign * idx) % C][:, (sign * idx) % C]

    def plane(a, b):
        return torch.fft.ifft2(a * b.conj(), norm="forward").real * scale
    M = _full64(GM, C)
    F = [_full64(G[n], C) for n in range(N)]
    terms = torch.empty(4 * N + 1, w, w, dtype=torch.float64, device=DEV)
    for n in range(N):
        a, d = plane(F[n], M), plane(_full64(S[n], C), M)
        terms[n], terms[N + n], terms[2 * N + n], terms[3 * N + n] = window(a, -1), window(a), window(d, -1), window(d)
    mp = terms[4 * N] = window(plane(M, M))
    out = torch.empty(len(pairs), w, w, dtype=torch.float64, device=DEV)
    for k, (i, j) in enumerate(pairs):
        tm, bm = terms[i], terms[N + j]
        den = torch.sqrt((terms[3 * N + j] - bm * bm / mp) * (terms[2 * N + i] - tm * tm / mp))
        out[k] = (window(plane(F[j], F[i])) - tm * bm / mp) / den.clamp(min=1.0)
    return terms, out


def _pairs_exact(case, s):
    G, S, GM = (torch.view_as_complex(s[k].double()) for k in ("G", "S", "GM"))
    terms, windows = _windows64(G, S, GM, case, s["pairs"].cpu().numpy().reshape(-1, 2))
    return {"terms": terms, "windows": windows}


def _pairs_work(case):
    N, C, w = case["N"], case["C"], 2 * case["mS"]
    M = N * (N - 1) // 2
    spec = C * (C // 2 + 1) * 8
    return {"bytes": 2 * N * spec + (4 * N + M) * w * w * 4, "flops": (M + 2 * N) * _fft_flops(C // 2 + w // 2, C)}


def _correlate_prepare(case, g, state):
    _counts(case, g, state)
    lib = state["lib"]
    N, C = case["N"], case["C"]
    K4 = lib.zr_spectrum_pitch(C)
    wb = lib.zr_spectra_work_bytes(case["H"], N, C)
    state.update(mean=torch.empty(N, dtype=torch.float64, device=DEV), work=_bytes(wb), wb=wb,
                 G=torch.empty(N, K4, C + 4, 2, device=DEV), S=torch.empty(N, K4, C + 4, 2, device=DEV),
                 GM=torch.empty(K4, C + 4, 2, device=DEV))
    _pairs_buffers(case, state)


def _correlate_run(s):
    c = s["case"]
    st = _stream()
    fr = ctypes.byref(s["frames"])
    size = (c["P"], c["P"], c["C"], c["C"])
    s["mean"].zero_()
    _lib.call("zr_frame_sums", fr, s["mean"].data_ptr(), st)
    _lib.call("zr_spectra", fr, None, None, 0, 1, 1, *size, s["GM"].data_ptr(), None, s["work"].data_ptr(), s["wb"], st)
    _lib.call("zr_spectra", fr, None, s["mean"].data_ptr(), 0, c["N"], 0, *size, s["G"].data_ptr(), s["S"].data_ptr(),
              s["work"].data_ptr(), s["wb"], st)
    _pairs_calls(s)
    return {"G": s["G"], "S": s["S"], "GM": s["GM"], "terms": s["terms"], "windows": s["windows"]}


def _correlate_exact(case, s):
    N, P, C = case["N"], case["P"], case["C"]
    K4 = s["GM"].shape[0]
    GS = []
    for n in range(N):
        v = _corrected64(s, n)
        GS.append(_half_spectra64(v, float(np.float32(float(v.mean()))), P, P, C, C, K4))
    G, S = (torch.stack([x[i] for x in GS]) for i in (0, 1))
    GM = _half_spectra64(torch.ones(case["H"], case["W"], dtype=torch.float64, device=DEV), 0.0, P, P, C, C, K4)[0]
    terms, windows = _windows64(G, S, GM, case, s["pairs"].cpu().numpy().reshape(-1, 2))
    return {"G": torch.view_as_real(G), "S": torch.view_as_real(S), "GM": torch.view_as_real(GM), "terms": terms,
            "windows": windows}


def _correlate_work(case):
    a = _spectra_work(dict(case, P0=case["P"], P1=case["P"], C0=case["C"], C1=case["C"]))
    b = _pairs_work(case)
    return {k: a[k] + b[k] for k in a}


# ------------------------------------------------------------------ peak search

_RECORD = np.dtype([("shift_y", "f8"), ("shift_x", "f8"), ("sigma", "f8"), ("corr", "f4"), ("peaksig", "f4"),
                    ("origin", "f4"), ("cy", "i4"), ("cx", "i4"), ("flags", "i4"), ("nfev", "i4")], align=True)


def _peaks_prepare(case, g, state):
    """Windows as mnxc2 leaves them: correlated noise, a broad peak at the
    pair's shift and a spike of fixed-pattern noise at the origin."""
    M, mS = case["M"], case["mS"]
    w = 2 * mS
    y = torch.arange(w, device=DEV, dtype=torch.float32) - mS
    f = torch.fft.fftfreq(w, device=DEV)[:, None] ** 2 + torch.fft.rfftfreq(w, device=DEV)[None, :] ** 2
    noise = torch.randn(M, w, w, generator=g, device=DEV)
    noise = noise + 2.0 * torch.fft.irfft2(torch.fft.rfft2(noise) * torch.exp(-f / 0.02), s=(w, w))
    at = (torch.rand(M, 2, generator=g, device=DEV) - 0.5) * 0.6 * mS
    amp = 4.0 + 8.0 * torch.rand(M, 1, 1, generator=g, device=DEV)
    r2 = (y[None, :, None] - at[:, 0, None, None]) ** 2 + (y[None, None, :] - at[:, 1, None, None]) ** 2
    win = 5e-4 * (noise + amp * torch.exp(-r2 / (2 * 3.0 ** 2)))
    win[:, mS, mS] += 0.01
    pp = _lib.PeakParams(16, case["bmode"], 1, 1, 1.3, 1.3, 0.0, 7.0, 0.01, 15)
    state.update(windows=win.contiguous(), params=pp, out=torch.empty(M, _RECORD.itemsize, dtype=torch.uint8, device=DEV))


def _peaks_run(s):
    _lib.call("zr_locate_peaks", s["windows"].data_ptr(), s["case"]["M"], s["case"]["mS"], ctypes.byref(s["params"]),
              s["out"].data_ptr(), _stream())
    r = s["out"]
    return {"shifts": r[:, :16].view(torch.float64), "sigma": r[:, 16:24].view(torch.float64),
            "corr, peaksig, origin": r[:, 24:36].view(torch.float32),
            "position, flags, evaluations": r[:, 36:52].view(torch.int32)}


def _peaks_work(case):
    px = 4 * case["mS"] ** 2
    # about 11 separable Gaussian filters of 2 x 25 taps
    return {"bytes": case["M"] * (px * 4 + 56), "flops": case["M"] * px * (11 * 100.0 if case["bmode"] == 1 else 44.0)}


# ------------------------------------------------------------------ shifted sums

def _shift_prepare(case, g, state):
    _counts(case, g, state)
    N, H, W = case["N"], case["H"], case["W"]
    t = np.round(16 * _drift(N, case["drift"] / math.sqrt(N), g)) / 16
    t = np.clip(t, -min(H, W) / 3.0, min(H, W) / 3.0)
    table = hostmath.shift_table(t - t.mean(0), H, W)
    state.update(table=table, shifts=torch.from_numpy(table.view(np.uint8)).to(DEV), sum=torch.empty(H, W, device=DEV),
                 even=torch.empty(H, W, device=DEV) if case["halves"] else None,
                 odd=torch.empty(H, W, device=DEV) if case["halves"] else None,
                 aligned=torch.empty(N, H, W, device=DEV) if case["aligned"] else None)


def _shift_run(s):
    _lib.call("zr_shift_sum", ctypes.byref(s["frames"]), s["shifts"].data_ptr(),
              *(None if s[k] is None else s[k].data_ptr() for k in ("sum", "even", "odd", "aligned")), _stream())
    return {k: s[k] for k in ("sum", "even", "odd", "aligned") if s[k] is not None}


def _shift_exact(case, s):
    N, H, W = case["N"], case["H"], case["W"]
    sums = torch.zeros(3, H, W, dtype=torch.float64, device=DEV)
    small = case["aligned"] and N * H * W <= 1 << 28
    frames = []
    for n in range(N):
        t = s["table"][n]
        v = torch.roll(_corrected64(s, n), (int(t["roll_y"]), int(t["roll_x"])), (0, 1))
        if t["apply"]:
            for axis, k in ((0, t["ky"]), (1, t["kx"])):
                first, last = (v.narrow(axis, i, 1) for i in (0, v.shape[axis] - 1))
                e = torch.cat([first, v, last], axis)
                v = sum(float(k[i]) * e.narrow(axis, 2 - i, v.shape[axis]) for i in range(3))
        sums[0] += v
        sums[1 + n % 2] += v
        if small:
            frames.append(v)
    out = {"sum": sums[0]}
    if case["halves"]:
        out.update(even=sums[1], odd=sums[2])
    if case["aligned"]:
        out["aligned"] = torch.stack(frames) if small else None
    return out


def _shift_work(case):
    N, HW = case["N"], case["H"] * case["W"]
    b = HW * (N * (TYPES[case["type"]][2] + 4 * case["aligned"]) + 4 + 8 * case["halves"]) + _map_bytes(case)
    return {"bytes": b, "flops": N * HW * 14.0}


# ------------------------------------------------------------------ dose filter

def _dose_prepare(case, g, state):
    N, H, W, P = case["N"], case["H"], case["W"], case["P"]
    img = torch.empty(N, H, W, device=DEV)
    for n in range(N):
        img[n] = torch.poisson(torch.full((H, W), 0.8, device=DEV), generator=g)
        img[n] += 0.05 * torch.randn(H, W, generator=g, device=DEV)
    dc = hostmath.dose_constants(N, [P, P], 0.105, 300.0, DOSE)
    prm = _lib.DoseParams(dc["A"], dc["B"], dc["C"], dc["order"], dc["vs"], dc["invPSx"], dc["invPSy"], int(case["norm"]))
    lib = state["lib"]
    fixed = lib.zr_dose_work_bytes(P, P, 0)
    per = lib.zr_dose_work_bytes(P, P, 1) - fixed
    wb = fixed + per * max(2, min(N + (N & 1), ((1536 << 20) - fixed) // per))
    state.update(img=img, dc=dc, prm=prm, wb=wb, work=_bytes(wb), out=torch.empty(H, W, device=DEV),
                 tq=torch.from_numpy(dc["thresQ"].astype(np.float32)).to(DEV),
                 de=torch.from_numpy(dc["dose_end"].astype(np.float32)).to(DEV))


def _dose_run(s):
    c = s["case"]
    _lib.call("zr_dose_filter", s["img"].data_ptr(), c["N"], c["H"], c["W"], ctypes.byref(s["prm"]),
              s["tq"].data_ptr(), s["de"].data_ptr(), c["P"], c["P"], s["out"].data_ptr(), s["work"].data_ptr(),
              s["wb"], _stream())
    return s["out"]


def _dose_exact(case, s):
    N, H, W, P = case["N"], case["H"], case["W"], case["P"]
    dc = s["dc"]

    def sym(n):
        i = torch.arange(P, device=DEV) % (2 * n)
        return torch.where(i < n, i, 2 * n - 1 - i)
    iy, ix = sym(H), sym(W)
    fy = torch.fft.fftfreq(P, 1.0 / P, device=DEV, dtype=torch.float64)[:, None]
    fx = torch.arange(P // 2 + 1, device=DEV, dtype=torch.float64)[None, :]
    q = torch.sqrt((fx * dc["invPSx"]) ** 2 + (fy * dc["invPSy"]) ** 2)
    crit = dc["vs"] * (dc["A"] * q ** dc["B"] + dc["C"])
    crit[P // 2, P // 2] = crit[P // 2, P // 2 - 1] ** 2
    acc, total = torch.zeros_like(q) + 0j, torch.zeros_like(q)
    for n in range(N):
        f = torch.exp(-0.5 * dc["dose_end"][n] / crit) * torch.exp(-(q / dc["thresQ"][n]) ** dc["order"])
        acc += torch.fft.rfft2(s["img"][n].double()[iy][:, ix]) * f
        total += f
    if case["norm"]:
        acc /= total + 1.0
    return torch.fft.irfft2(acc, s=(P, P), norm="forward")[:H, :W].abs()


def _dose_work(case):
    N, HW, P = case["N"], case["H"] * case["W"], case["P"]
    return {"bytes": HW * 4 * (N + 1), "flops": (N + 1) * (_fft_flops(P // 2, P) + _fft_flops(P // 2 + 1, P))}


# ------------------------------------------------------------------ Fourier ring correlation

def _frc_prepare(case, g, state):
    H, W = case["H"], case["W"]
    raw = _movie(2, H, W, "f32", g, dose=16.0, sigma=0.0)
    offs, _ = hostmath.frc_tiles((H, W), None)
    wb = state["lib"].zr_frc_work_bytes(len(offs), 512)
    state.update(even=raw[0].contiguous(), odd=raw[1].contiguous(), offs=torch.from_numpy(offs.reshape(-1)).to(DEV),
                 n=len(offs), wb=wb, work=_bytes(wb), frc2d=torch.empty(512, 512, device=DEV),
                 frc=torch.empty(256, dtype=torch.float64, device=DEV))


def _frc_run(s):
    _lib.call("zr_tiled_frc", s["even"].data_ptr(), s["odd"].data_ptr(), s["case"]["H"], s["case"]["W"], 512,
              s["offs"].data_ptr(), s["n"], s["frc2d"].data_ptr(), s["frc"].data_ptr(), 256, s["work"].data_ptr(),
              s["wb"], _stream())
    return {"frc2d": s["frc2d"], "frc": s["frc"]}


def _frc_exact(case, s):
    B = 512
    x = (torch.arange(B, device=DEV, dtype=torch.float64) - B // 2) / (B // 2)
    r = torch.sqrt(x[:, None] ** 2 + x[None, :] ** 2)
    hann = torch.where(r <= 1.0, 0.5 * (1.0 + torch.cos(math.pi * r)), torch.zeros_like(r))
    acc = torch.zeros(B, B, dtype=torch.float64, device=DEV)
    for oy, ox in s["offs"].cpu().numpy().reshape(-1, 2):
        E, O = (torch.fft.fft2(hann * s[k][oy:oy + B, ox:ox + B].double()) for k in ("even", "odd"))
        acc += (E * O.conj()).real / (E.abs() * O.abs())
    acc = torch.fft.fftshift(acc / acc[0, 0])
    r = (B // 2) * r
    b0, rem = torch.floor(r).long(), r - torch.floor(r)
    num = torch.bincount(b0.view(-1), (acc * (1 - rem)).view(-1), minlength=400)
    num[1:] += torch.bincount(b0.view(-1), (acc * rem).view(-1), minlength=400)[:-1]
    den = torch.bincount(b0.view(-1), (1 - rem).view(-1), minlength=400)
    den[1:] += torch.bincount(b0.view(-1), rem.view(-1), minlength=400)[:-1]
    return {"frc2d": acc, "frc": (num / den)[:256]}


def _frc_work(case):
    n = len(hostmath.frc_tiles((case["H"], case["W"]), None)[0])
    return {"bytes": case["H"] * case["W"] * 8, "flops": n * (_fft_flops(512, 512) + 2 * _fft_flops(257, 512))}


# ------------------------------------------------------------------ Fourier binning

def _bin_prepare(case, g, state):
    N, H, W = case["N"], case["H"], case["W"]
    raw = torch.empty(N, H, W, dtype=TYPES[case["type"]][0], device=DEV)
    for n in range(N):
        raw[n] = torch.poisson(torch.full((H, W), 0.25, device=DEV), generator=g)
    wb = state["lib"].zr_bin_work_bytes(H, W, case["Hb"], case["Wb"])
    state.update(raw=raw, frames=_frames(raw, case["type"]), wb=wb, work=_bytes(wb),
                 out=torch.empty(N, case["Hb"], case["Wb"], device=DEV))


def _bin_run(s):
    _lib.call("zr_bin_fourier", ctypes.byref(s["frames"]), s["case"]["Hb"], s["case"]["Wb"], s["out"].data_ptr(),
              s["work"].data_ptr(), s["wb"], _stream())
    return s["out"]


def _bin_exact(case, s):
    N, H, W, Hb, Wb = (case[k] for k in ("N", "H", "W", "Hb", "Wb"))
    out = torch.empty(N, Hb, Wb, dtype=torch.float64, device=DEV)
    for n in range(N):
        F = torch.fft.fft2(s["raw"][n].double())
        F = torch.cat([F[:Hb // 2], F[H - Hb // 2:]], 0)
        F = torch.cat([F[:, :Wb // 2], F[:, W - Wb // 2:]], 1)
        out[n] = torch.fft.ifft2(F).real
    return out


def _bin_work(case):
    N, H, W, Hb, Wb = (case[k] for k in ("N", "H", "W", "Hb", "Wb"))
    flops = _fft_flops(H / 2, W) + _fft_flops(Wb / 2, H) + _fft_flops(Wb / 2, Hb) + _fft_flops(Hb / 2, Wb)
    return {"bytes": N * (H * W * TYPES[case["type"]][2] + Hb * Wb * 4), "flops": N * flops}


STAGES = {
    "align": (_align_prepare, _align_run, None, _align_work),
    "hotpix": (_hotpix_prepare, _hotpix_run, _hotpix_exact, _hotpix_work),
    "spectra": (_spectra_prepare, _spectra_run, _spectra_exact, _spectra_work),
    "correlate": (_correlate_prepare, _correlate_run, _correlate_exact, _correlate_work),
    "pairs": (_pairs_prepare, _pairs_run, _pairs_exact, _pairs_work),
    "peaks": (_peaks_prepare, _peaks_run, None, _peaks_work),
    "shift": (_shift_prepare, _shift_run, _shift_exact, _shift_work),
    "dose": (_dose_prepare, _dose_run, _dose_exact, _dose_work),
    "frc": (_frc_prepare, _frc_run, _frc_exact, _frc_work),
    "bin": (_bin_prepare, _bin_run, _bin_exact, _bin_work),
}
