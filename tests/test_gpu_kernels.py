"""Kernels at the sizes where they can go wrong: every transform length with
ragged frames, the window sizes around the pruned last pass, windows searched
by one CTA or a cluster, tile edges of the shifted sums and the hot-pixel
maps, direct and chirp sides of the binning, FRC boxes.

Tolerances are derived beforehand: a float32 transform of n points made of a
few passes is off by at most about log2(n) roundings of 2^-24 relative to the
result's norm, so errors are held to 6e-8 log2(n) in the 2-norm; what is only
copied, rolled or counted is equal; a k-tap float32 sum of a few roundings is
held to 2e-6 of the largest value."""
import ctypes as C

import numpy as np
import pytest

from oracle import zorro_oracle as zo
from tests import gpu_helpers as gh
from zorro_gb300 import _lib
from zorro_gb300 import hostmath as hm

pytestmark = pytest.mark.gpu

TYPES = {"f32": (np.float32, _lib.ZR_F32), "u8": (np.uint8, _lib.ZR_U8), "u16": (np.uint16, _lib.ZR_U16),
         "f16": (np.float16, _lib.ZR_F16)}


def _init():
    torch = gh.torch_mod()
    _lib.call("zr_init", torch.cuda.current_device())
    return torch, _lib.load()


def _movie(rng, kind, N, H, W, maps=False):
    """Raw counts on the device, their maps and the corrected float64 frames."""
    torch = gh.torch_mod()
    raw = rng.poisson(3.0, (N, H, W)).astype(TYPES[kind][0])
    dev = torch.from_numpy(raw.view(np.int16) if kind == "u16" else raw).cuda()
    v = raw.astype(np.float64)
    gain = ha = hb = None
    if maps:
        gain = rng.uniform(0.9, 1.1, (H, W)).astype(np.float32)
        ha = rng.uniform(0.95, 1.0, (H, W)).astype(np.float32)
        hb = rng.uniform(0.0, 0.2, (H, W)).astype(np.float32)
        v = v * gain * ha + hb
    dm = [None if m is None else torch.from_numpy(m).cuda() for m in (gain, ha, hb)]
    fr = _lib.Frames(dev.data_ptr(), TYPES[kind][1], *(None if m is None else m.data_ptr() for m in dm), 0.0, N, H, W, 0)
    return fr, v, (dev, dm)


def _rel(got, want):
    return float(np.linalg.norm(np.asarray(got, np.complex128) - want) / np.linalg.norm(want))


def _spectra(fr, mean, H, P, C_, N):
    torch, lib = _init()
    K4 = lib.zr_spectrum_pitch(C_[1])
    G = torch.full((N, K4, C_[0] + 4, 2), 1e30, device="cuda")
    S = torch.full((N, K4, C_[0] + 4, 2), 1e30, device="cuda")
    wb = lib.zr_spectra_work_bytes(H, N, C_[1])
    work = torch.empty(wb, dtype=torch.uint8, device="cuda")
    msub = torch.from_numpy(mean).cuda()
    _lib.call("zr_spectra", C.byref(fr), None, msub.data_ptr(), 0, N, 0, *P, *C_, G.data_ptr(), S.data_ptr(),
              work.data_ptr(), wb, gh.stream())
    torch.cuda.synchronize()
    return [torch.view_as_complex(t).cpu().numpy() for t in (G, S)]


@pytest.mark.parametrize("kind,maps,N,H,W,P,C_", [
    ("f32", False, 2, 64, 64, (64, 64), (64, 64)), ("u8", True, 3, 117, 121, (128, 128), (64, 128)),
    ("f16", False, 1, 255, 201, (256, 256), (256, 128)), ("u16", True, 3, 510, 449, (512, 512), (384, 256)),
    ("u8", True, 5, 1001, 1023, (1024, 1024), (512, 1024)), ("f32", True, 2, 1333, 1537, (1536, 3072), (768, 768)),
    ("u8", True, 3, 1795, 2045, (2048, 2048), (2048, 1024)), ("u8", True, 4, 3073, 4095, (4096, 4096), (1536, 2048)),
    ("f32", False, 1, 4093, 5761, (4096, 6144), (2048, 3072)), ("f16", True, 2, 6143, 130, (6144, 256), (4096, 64))])
def test_spectra_every_length(kind, maps, N, H, W, P, C_):
    rng = np.random.default_rng(H + W)
    fr, v, keep = _movie(rng, kind, N, H, W, maps)
    mean = v.sum(axis=(1, 2))
    got = _spectra(fr, mean, H, P, C_, N)
    rows = np.array([r if r < C_[0] // 2 else P[0] - C_[0] + r for r in range(C_[0])] + [C_[0] // 2])
    tol = 6e-8 * np.log2(P[0] * P[1])
    for n in range(N):
        u = np.zeros(P)
        u[:H, :W] = v[n] - np.float32(mean[n] / (H * W))
        for t, img in zip(got, (u, u * u)):
            F = np.fft.rfft2(img)[rows][:, :C_[1] // 2 + 1].T
            assert _rel(t[n, :C_[1] // 2 + 1, :C_[0] + 1], F) <= tol
            assert np.all(t[n, :, C_[0] + 1:] == 0) and np.all(t[n, C_[1] // 2 + 1:] == 0)


@pytest.mark.parametrize("C_,mS", [((128, 128), 8), ((256, 256), 7), ((256, 256), 8), ((512, 384), 64), ((512, 512), 63),
                                   ((512, 512), 128), ((1024, 1024), 64), ((1024, 512), 65), ((2048, 1024), 64)])
def test_windows_around_the_pruned_last_pass(C_, mS):
    """mnxc2's windows with at most, exactly and more rows than the last pass
    has butterflies, whole planes among them."""
    rng = np.random.default_rng(mS)
    N = 3
    H, W = C_[0] - 9, C_[1] - 20
    imgs = rng.poisson(2.0, (N, H, W)).astype(np.float32)
    P = (C_[0], {384: 512}.get(C_[1], C_[1]))  # 384 is a crop's side, not a frame's
    _, _, _, _, dev = gh.spectra(imgs, P, C_)
    pairs = [(0, 1), (0, 2), (1, 2)]
    _, cw, _ = gh.windows(dev, N, C_, mS, pairs)
    dt = zo.Dtypes(True)
    padded, mask = zo.pad_stack(imgs, P)
    GM, MP = zo.mask_spectrum(mask, np.array(C_), dt)
    spec = [zo.frame_spectra(padded[n], mask, np.array(C_), dt) for n in range(N)]
    for k, (I, J) in enumerate(pairs):
        ref, _ = zo.mnxc2(*spec[I], *spec[J], GM, MP, zo.norm_const2(np.array(C_)), mS, suppressOrigin=False, dt=dt)
        assert np.abs(cw[k] - ref).max() <= 2e-5 * np.abs(ref).max()


@pytest.mark.parametrize("mS", [8, 9, 20, 33, 50, 52, 100, 101, 104, 108])
def test_peaks_do_not_depend_on_the_split(mS):
    """The same windows searched one, 20, 40 and 160 at a launch (clusters of
    8, 4, 2 CTAs, one CTA each): the same records, bit for bit."""
    torch, _ = _init()
    rng = np.random.default_rng(mS)
    w = 2 * mS
    y = np.arange(w) - mS
    wins = np.empty((160, w, w), np.float32)
    for k in range(160):
        cy, cx = rng.uniform(-0.6 * mS, 0.6 * mS, 2)
        wins[k] = 5e-4 * (rng.standard_normal((w, w)) + rng.uniform(4, 12)
                          * np.exp(-((y[:, None] - cy) ** 2 + (y[None] - cx) ** 2) / 18))
    wins[3] = 0.0
    wins[:, mS, mS] += 0.01
    dev = gh.dev_tensor(wins)
    for bmode in (1, 0):
        whole = gh.peaks(dev, mS, bmode=bmode)
        for a, b in ((0, 1), (3, 4), (10, 30), (40, 80)):
            assert gh.peaks(dev[a:b], mS, bmode=bmode).tobytes() == whole[a:b].tobytes(), (bmode, a, b)


@pytest.mark.parametrize("scale", [1.0, 1e-18, 1e14])
@pytest.mark.parametrize("sp", [2, 4, 8, 16, 32])
def test_subpixel_maximum(sp, scale):
    """The sub-pixel point holds the largest value of the upsampled patch: a
    value summed in float32 is off by less than 64 roundings of sum |F|, so
    the point found lies within twice that of the float64 maximum.  Peaks,
    noise, a flat window (every point within rounding) and values whose squares leave the
    range of the quick search."""
    torch, _ = _init()
    rng = np.random.default_rng(sp)
    mS, M, L = 14, 12, 16 * sp
    y = np.arange(2 * mS) - mS
    wins = np.empty((M, 2 * mS, 2 * mS), np.float32)
    for k in range(M):
        cy, cx = rng.uniform(-4, 4, 2)
        wins[k] = scale * (0.1 * rng.standard_normal((2 * mS, 2 * mS))
                           + (k % 4 > 0) * np.exp(-((y[:, None] - cy) ** 2 + (y[None] - cx) ** 2) / rng.uniform(2, 30)))
    wins[1] = scale
    wins[1, mS, mS] = np.nextafter(np.float32(scale), np.float32(np.inf))
    f = np.concatenate([np.arange(8), np.arange(-8, 0)])
    E = np.exp(2j * np.pi * np.outer(np.arange(L), f) / L)
    inside = 0
    for k, r in enumerate(gh.peaks(gh.dev_tensor(wins), mS, subPixReg=sp, bmode=0, suppress=False)):
        cy, cx = int(r["cy"]), int(r["cx"])
        if not (8 <= cy <= 2 * mS - 8 and 8 <= cx <= 2 * mS - 8):
            continue
        inside += 1
        F = np.fft.fft2(wins[k, cy - 8:cy + 8, cx - 8:cx + 8].astype(np.float64))
        V = np.abs(E @ F @ E.T)
        tol = 64 * 2.0 ** -24 * np.abs(F).sum()
        sy, sx = (int(round((r[n] - (c - mS)) * sp + L / 2 - np.sign(c - mS)))
                  for n, c in (("sy", cy), ("sx", cx)))
        assert V[sy, sx] >= V.max() - 2 * tol
        assert abs(256 * float(r["corr"]) - V[sy, sx]) <= tol
    assert inside >= 6


@pytest.mark.parametrize("kind,maps,H,W,halves", [
    ("f32", False, 2, 2, True), ("u8", True, 17, 127, False), ("u8", True, 16, 128, True), ("u16", True, 33, 129, False),
    ("f16", False, 40, 257, True), ("u8", False, 15, 1030, False), ("f32", True, 700, 1023, True),
    ("u8", True, 640, 2050, False)])
def test_shift_sum_tile_edges(kind, maps, H, W, halves):
    """Rolled, Lanczos-filtered frames and their sums against the same steps
    in float64, at the edges of tiles, chunks and vector accesses; rolls that
    wrap inside a tile, and frames that are only rolled."""
    torch, _ = _init()
    rng = np.random.default_rng(H + W)
    N = 5
    fr, v, keep = _movie(rng, kind, N, H, W, maps)
    t = rng.uniform(-0.4, 0.4, (N, 2)) * [H, W]
    t[1] = np.round(t[1])
    tab = hm.shift_table(t, H, W)
    out = {k: torch.zeros((H, W), device="cuda") for k in ("sum", "even", "odd")}
    aligned = torch.zeros((N, H, W), device="cuda")
    sh = torch.from_numpy(tab.view(np.uint8)).cuda()
    _lib.call("zr_shift_sum", C.byref(fr), sh.data_ptr(), out["sum"].data_ptr(),
              out["even"].data_ptr() if halves else None, out["odd"].data_ptr() if halves else None, aligned.data_ptr(),
              gh.stream())
    want = np.empty((N, H, W))
    for n in range(N):
        a = np.roll(v[n], (int(tab["roll_y"][n]), int(tab["roll_x"][n])), (0, 1))
        if tab["apply"][n]:
            for ax, k in ((0, tab["ky"][n]), (1, tab["kx"][n])):
                e = np.concatenate([a.take([0], ax), a, a.take([-1], ax)], ax)
                m = a.shape[ax]
                a = sum(float(k[i]) * e.take(range(2 - i, 2 - i + m), ax) for i in range(3))
        want[n] = a
    tol = 2e-6 * np.abs(want).max()
    np.testing.assert_allclose(aligned.cpu().numpy(), want, rtol=0, atol=tol)
    np.testing.assert_allclose(out["sum"].cpu().numpy(), want.sum(0), rtol=0, atol=N * tol)
    if halves:
        np.testing.assert_allclose(out["even"].cpu().numpy(), want[0::2].sum(0), rtol=0, atol=N * tol)
        np.testing.assert_allclose(out["odd"].cpu().numpy(), want[1::2].sum(0), rtol=0, atol=N * tol)


@pytest.mark.parametrize("H,W", [(4, 4), (31, 63), (32, 64), (33, 65), (64, 130), (97, 191)])
@pytest.mark.parametrize("sigma", [3.0, 1e-30, 0.0])
def test_hotpix_map_tiles(H, W, sigma):
    """The mask against its float64 formula and the counts against the float64
    quotient at tile edges; infinite, NaN and huge sums, and a fit width so
    small (or zero) that the exponents leave the float pairs' range."""
    torch, lib = _init()
    rng = np.random.default_rng(H)
    s = rng.normal(20, 3, (H, W)).astype(np.float32)
    s.flat[:4] = [np.inf, -np.inf, 3e38, 0.0]
    p = _lib.HotpixParams()
    p.mu, p.sigma, p.cutoff_lower, p.cutoff_upper = 20.0, sigma, -2.0, 2.0
    p.logistic_k, p.relax, p.neighbour_thres, p.best_mean = 6.0, 0.925, 0.01, 2.0
    for i, k in enumerate(hm.psf_kernel("K2").ravel()):
        p.psf[i] = float(k)
    ds = gh.dev_tensor(s)
    a, b = (torch.full((H, W), 7.0, device="cuda") for _ in range(2))
    cnt = torch.zeros(4, dtype=torch.int32, device="cuda")
    wb = lib.zr_hotpix_work_bytes(H, W)
    work = torch.empty(wb, dtype=torch.uint8, device="cuda")
    _lib.call("zr_hotpix_maps", ds.data_ptr(), H, W, 10, C.byref(p), a.data_ptr(), b.data_ptr(), cnt.data_ptr(),
              work.data_ptr(), wb, gh.stream())
    with np.errstate(all="ignore"):
        q = (s.astype(np.float64) - 20.0) / sigma
        assert cnt[0].item() == np.sum(q < -2.0) and cnt[1].item() == np.sum(q > 2.0)
        if sigma > 0:
            lo, hi = (np.float64(np.float32(c) * np.float32(0.925)) for c in (-2.0, 2.0))
            e1, e2 = np.exp(6.0 * (q - lo)), np.exp(6.0 * (q - hi))
            want = (1.0 - 1.0 / (1.0 + e1)) / (1.0 + e2)
            # exponents are rounded to float32: up to 2^-24 of the largest that matters (88)
            np.testing.assert_allclose(a.cpu().numpy(), want, rtol=0, atol=88 * 2.0 ** -24 / 4 + 5e-7)


@pytest.mark.parametrize("H,W,Hb,Wb", [
    (3000, 4096, 2048, 3072), (8192, 600, 5760, 514), (700, 9216, 514, 5120),
    (7681, 1025, 6144, 1024), (16384, 530, 2050, 514), (515, 16384, 514, 12288), (521, 15360, 516, 10240)])
def test_binning_sides(H, W, Hb, Wb):
    """Direct and chirp sides, odd frames, crops that keep all or few
    frequencies, against numpy's float64 transforms."""
    torch, lib = _init()
    rng = np.random.default_rng(H)
    raw = rng.poisson(1.0, (1, H, W)).astype(np.uint8)
    dev = torch.from_numpy(raw).cuda()
    fr = _lib.Frames(dev.data_ptr(), _lib.ZR_U8, None, None, None, 0.0, 1, H, W, 0)
    out = torch.zeros((Hb, Wb), device="cuda")
    wb = lib.zr_bin_work_bytes(H, W, Hb, Wb)
    work = torch.full((wb,), 255, dtype=torch.uint8, device="cuda")
    _lib.call("zr_bin_fourier", C.byref(fr), Hb, Wb, out.data_ptr(), work.data_ptr(), wb, gh.stream())
    F = np.fft.fft2(raw[0].astype(np.float64))
    F = np.concatenate([F[:Hb // 2], F[H - Hb // 2:]], 0)
    F = np.concatenate([F[:, :Wb // 2], F[:, W - Wb // 2:]], 1)
    want = np.fft.ifft2(F).real
    # a chirp transform is two transforms of up to 16384 points a side
    assert _rel(out.cpu().numpy(), want) <= 6e-8 * 4 * 14


@pytest.mark.parametrize("box,H,W", [(128, 300, 290), (256, 530, 700), (512, 1200, 1111), (1024, 1100, 1400)])
def test_frc_boxes(box, H, W):
    """FRC plane and rings of every box against float64."""
    torch, lib = _init()
    rng = np.random.default_rng(box)
    base = rng.normal(10, 3, (H, W))
    ev, od = ((base + rng.normal(0, 2, (H, W))).astype(np.float32) for _ in range(2))
    offs = np.array([[y, x] for y in range(3, H - box, box // 2) for x in range(1, W - box, box // 2)], np.int32)
    nr = int(np.ceil(np.sqrt(2.0 * (box // 2) ** 2))) + 1
    wb = lib.zr_frc_work_bytes(len(offs), box)
    work = torch.full((wb,), 255, dtype=torch.uint8, device="cuda")
    de, do, dof = gh.dev_tensor(ev), gh.dev_tensor(od), gh.dev_tensor(offs.reshape(-1))
    f2 = torch.zeros((box, box), device="cuda")
    fr = torch.zeros(nr, dtype=torch.float64, device="cuda")
    _lib.call("zr_tiled_frc", de.data_ptr(), do.data_ptr(), H, W, box, dof.data_ptr(), len(offs), f2.data_ptr(),
              fr.data_ptr(), nr, work.data_ptr(), wb, gh.stream())
    x = (np.arange(box) - box // 2) / (box // 2)
    r = np.hypot(x[:, None], x[None])
    hann = np.where(r <= 1, 0.5 * (1 + np.cos(np.pi * r)), 0.0)
    acc = np.zeros((box, box))
    for oy, ox in offs:
        E, O = (np.fft.fft2(hann * t[oy:oy + box, ox:ox + box].astype(np.float64)) for t in (ev, od))
        acc += (E * O.conj()).real / (np.abs(E) * np.abs(O))
    acc = np.fft.fftshift(acc / acc[0, 0])
    rad = r * (box // 2)
    b0 = np.floor(rad).astype(int)
    rem = rad - b0
    num, den = np.zeros(nr + 2), np.zeros(nr + 2)
    for b, wt in ((b0, 1 - rem), (b0 + 1, rem)):
        np.add.at(num, b, acc * wt)
        np.add.at(den, b, wt)
    # frequencies where E or O nearly vanishes amplify the transforms' error
    assert _rel(f2.cpu().numpy(), acc) <= 1e-4
    np.testing.assert_allclose(fr.cpu().numpy(), num[:nr] / den[:nr], rtol=0, atol=1e-4)
