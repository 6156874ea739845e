"""Calls at the edges of what the entry points take: buffers aligned to no
more than an element, bounds in either order, every sub-pixel factor, the
planner's choices, windows without a finite value, wide-ranging sums.

What an input's alignment or the split between CTAs cannot change is held to
equality; the other tolerances are derived at their tests."""
import ctypes as C

import numpy as np
import pytest

from tests import gpu_helpers as gh
from zorro_gb300 import _lib
from zorro_gb300 import hostmath as hm

pytestmark = pytest.mark.gpu


def _init():
    torch = gh.torch_mod()
    _lib.call("zr_init", torch.cuda.current_device())
    return torch, _lib.load()


def _frames(raw, kind, maps=(None, None, None)):
    N, H, W = raw.shape
    return _lib.Frames(raw.data_ptr(), kind, *(None if m is None else m.data_ptr() for m in maps), 0.0, N, H, W, 0)


@pytest.mark.parametrize("H,W", [(40, 130), (33, 258), (2600, 300), (50, 127)])
@pytest.mark.parametrize("halves", [False, True])
def test_shift_sum_aligned_frames_at_any_float(H, W, halves):
    """The aligned frames go to any float-aligned buffer: one float past a
    256-byte boundary they hold the same bits as on it (even widths, whose
    rows are stored in pairs there, tiles of 8 and of 16 rows, and an odd
    width)."""
    torch, _ = _init()
    rng = np.random.default_rng(H * W)
    N = 3
    raw = torch.from_numpy(rng.poisson(4.0, (N, H, W)).astype(np.uint8)).cuda()
    fr = _frames(raw, _lib.ZR_U8)
    t = np.round(16 * rng.uniform(-5, 5, (N, 2))) / 16
    sh = torch.from_numpy(hm.shift_table(t, H, W).view(np.uint8)).cuda()
    got = []
    for skip in (0, 1):
        arena = torch.full((N * H * W + 64,), 7.0, device="cuda")
        assert arena.data_ptr() % 256 == 0
        out = torch.empty(3, H, W, device="cuda")
        even, odd = (out[1].data_ptr(), out[2].data_ptr()) if halves else (None, None)
        _lib.call("zr_shift_sum", C.byref(fr), sh.data_ptr(), out[0].data_ptr(), even, odd,
                  arena.data_ptr() + 4 * skip, gh.stream())
        torch.cuda.synchronize()
        rest = torch.cat([arena[:skip], arena[skip + N * H * W:]])
        assert bool((rest == 7.0).all())
        got.append((arena[skip:skip + N * H * W].clone(), out[:3 if halves else 1].clone()))
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("H,W,Hb,Wb", [(601, 640, 560, 562), (1100, 1024, 1026, 514), (2048, 3072, 1024, 1536)])
def test_binning_work_at_any_element(H, W, Hb, Wb):
    """``work`` holds complex floats and needs their alignment only: eight
    bytes past a 256-byte boundary the binned frames are the same bits (odd
    and even heights, chirp and direct sides), and nothing is written past
    zr_bin_work_bytes."""
    torch, lib = _init()
    rng = np.random.default_rng(H)
    raw = torch.from_numpy(rng.poisson(2.0, (2, H, W)).astype(np.uint8)).cuda()
    fr = _frames(raw, _lib.ZR_U8)
    wb = lib.zr_bin_work_bytes(H, W, Hb, Wb)
    got = []
    for skip in (0, 8):
        arena = torch.full((wb + 256,), 165, dtype=torch.uint8, device="cuda")
        assert arena.data_ptr() % 256 == 0
        out = torch.empty(2, Hb, Wb, device="cuda")
        _lib.call("zr_bin_fourier", C.byref(fr), Hb, Wb, out.data_ptr(), arena.data_ptr() + skip, wb, gh.stream())
        torch.cuda.synchronize()
        assert bool((arena[:skip] == 165).all()) and bool((arena[skip + wb:] == 165).all())
        got.append(out)
    assert torch.equal(*got)


def _windows(rng, M, mS):
    """Noise with a broad peak off the centre."""
    y = np.arange(2 * mS) - mS
    at = rng.uniform(-0.3, 0.3, (M, 2)) * mS
    r2 = (y[None, :, None] - at[:, 0, None, None]) ** 2 + (y[None, None, :] - at[:, 1, None, None]) ** 2
    win = rng.normal(0, 1, (M, 2 * mS, 2 * mS)) + 8.0 * np.exp(-r2 / 18.0)
    return (1e-3 * win).astype(np.float32)


def _locate(win, mS, **kw):
    torch, _ = _init()
    p = dict(sub_pix_reg=16, bmode=1, suppress_origin=1, use_mask=1, conv_sigma_y=0.0, conv_sigma_x=0.0, opti_lo=0.0,
             opti_hi=7.0, opti_xatol=0.01, opti_maxiter=15)
    p.update(kw)
    pp = _lib.PeakParams(**p)
    dev = torch.from_numpy(np.ascontiguousarray(win, dtype=np.float32)).cuda()
    out = torch.zeros((len(win), C.sizeof(_lib.PeakResult)), dtype=torch.uint8, device="cuda")
    _lib.call("zr_locate_peaks", dev.data_ptr(), len(win), mS, C.byref(pp), out.data_ptr(), gh.stream())
    torch.cuda.synchronize()
    return np.frombuffer(out.cpu().numpy().tobytes(), dtype=gh.PEAK_DTYPE)


@pytest.mark.parametrize("lo,hi", [(7.0, 0.0), (20.0, 1.0), (15.9, 15.8)])
@pytest.mark.parametrize("mS,M", [(20, 3), (25, 3), (50, 20), (111, 2), (33, 160)])
def test_opti_bounds_in_either_order(mS, M, lo, hi):
    """With opti_lo > opti_hi the bounded search ends at its first abscissa
    (FMM FMIN's test holds there), which may lie far above opti_hi: the records
    are those of that sigma given to bmode 2."""
    win = _windows(np.random.default_rng(mS), M, mS)
    got = _locate(win, mS, opti_lo=lo, opti_hi=hi)
    sigma = got["sigma"][0]
    assert np.all(got["nfev"] == 1) and np.all(got["sigma"] == sigma)
    assert abs(sigma - (lo + 0.5 * (3.0 - 5.0 ** 0.5) * (hi - lo))) < 1e-12
    want = _locate(win, mS, bmode=2, conv_sigma_y=sigma, conv_sigma_x=sigma)
    for k in ("sy", "sx", "corr", "peaksig", "origin", "cy", "cx", "flags"):
        assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("sp", [3, 5, 6, 9, 12, 15, 20, 24, 30])
@pytest.mark.parametrize("flat", [False, True])
def test_subpixel_factors_that_are_no_power_of_two(sp, flat):
    """Every sub-pixel factor that is taken finds the largest value of the
    upsampled patch, by the quick search and term by term (a flat window):
    within the 64 roundings of sum |F| that test_subpixel_maximum derives."""
    rng = np.random.default_rng(sp)
    mS, M, L = 14, 6, 16 * sp
    win = _windows(rng, M, mS)
    if flat:
        win[:] = 1.0
        win[:, mS, mS] = np.nextafter(np.float32(1.0), np.float32(2.0))
    f = np.concatenate([np.arange(8), np.arange(-8, 0)])
    E = np.exp(2j * np.pi * np.outer(np.arange(L), f) / L)
    inside = 0
    for k, r in enumerate(_locate(win, mS, sub_pix_reg=sp, bmode=0, suppress_origin=0)):
        cy, cx = int(r["cy"]), int(r["cx"])
        if not (8 <= cy <= 2 * mS - 8 and 8 <= cx <= 2 * mS - 8):
            continue
        inside += 1
        F = np.fft.fft2(win[k, cy - 8:cy + 8, cx - 8:cx + 8].astype(np.float64))
        V = np.abs(E @ F @ E.T)
        tol = 64 * 2.0 ** -24 * np.abs(F).sum()
        at = [(r[n] - (c - mS)) * sp + L / 2 - np.sign(c - mS) for n, c in (("sy", cy), ("sx", cx))]
        sy, sx = (int(round(v)) for v in at)
        assert np.allclose(at, (sy, sx), atol=1e-9) and 0 <= sy < L and 0 <= sx < L
        assert V[sy, sx] >= V.max() - 2 * tol
        assert abs(256 * float(r["corr"]) - V[sy, sx]) <= tol
    assert inside >= 4


@pytest.mark.parametrize("mS,M", [(20, 1), (20, 160), (25, 3)])
@pytest.mark.parametrize("spike", [2.4e19, 1e20])
def test_opti_search_avoids_infinite_statistics(mS, M, spike):
    """Where the filtered window's sum of squares passes float32's range (the
    sums are float32 within a warp of statistics threads, float64 across the
    warps) its contrast is infinite and the search turns away from it: the
    sigma found is that of the search over the float64 statistics with infinity
    in those places.  (Both stop at the edge of that range; the abscissas there
    lie within the search's xatol of 0.01 of one another, held to twice that.)"""
    import scipy.ndimage
    rng = np.random.default_rng(mS)
    w = 2 * mS
    win = 1e16 * rng.standard_normal((w, w))
    win[mS + 1, mS - 2] = spike
    win = win.astype(np.float32)
    # the statistics thread of each pixel: rows 2 ty, 2 ty + 1 and columns 4 tx
    # .. 4 tx + 3, or rows y mod 16 = ty and columns tx mod 64
    y, x = np.mgrid[:w, :w]
    warp = ((y // 2 % (4096 // w) * (w // 4) + x // 4) if w % 4 == 0 else (y % 16 * 64 + x % 64)) // 32
    search = hm.brent_bounded(0.0, 7.0, 0.01, 15)
    seen = []
    s = next(search)
    try:
        while True:
            F = scipy.ndimage.gaussian_filter(win.astype(np.float64), s)
            d = F - win.mean(dtype=np.float64)
            most = np.bincount(warp.ravel(), (d * d).ravel()).max()
            f = np.sqrt(d.var()) / (F.max() - F.mean()) if most < 3.4028235e38 else np.inf
            seen.append(f)
            s = search.send(f)
    except StopIteration as e:
        sigma = e.value[0]
    assert np.inf in seen
    got = _locate(np.repeat(win[None], M, 0), mS, suppress_origin=0)
    assert np.all(np.abs(got["sigma"] - sigma) <= 0.02), (got["sigma"][0], sigma)
    assert np.all((got["cy"] == mS + 1) & (got["cx"] == mS - 2))


@pytest.mark.parametrize("mS,M", [(20, 1), (20, 160), (25, 3), (100, 9)])
@pytest.mark.parametrize("bmode,use_mask", [(0, 0), (0, 1), (1, 0), (2, 0)])
def test_windows_of_nan(mS, M, bmode, use_mask):
    """A window without a number in it has its peak at np.argmax's index 0,
    the window's corner, where there is no sub-pixel step; a patch with a NaN
    has its sub-pixel maximum at index 0 too.  Windows beside them keep their
    records."""
    win = _windows(np.random.default_rng(mS), M, mS)
    kw = dict(bmode=bmode, use_mask=use_mask, conv_sigma_y=1.3, conv_sigma_x=1.3, suppress_origin=0)
    clean = _locate(win, mS, **kw)
    win[0] = np.nan
    got = _locate(win, mS, **kw)
    assert (got["cy"][0], got["cx"][0], got["flags"][0]) == (0, 0, 1)
    assert (got["sy"][0], got["sx"][0]) == (-mS, -mS)
    assert np.isnan(got["corr"][0]) and np.isnan(got["peaksig"][0]) and np.isnan(got["origin"][0])
    assert got[1:].tobytes() == clean[1:].tobytes()
    if bmode == 0:
        win[0] = 0.0
        win[0, mS, mS + 1], win[0, mS + 3, mS + 3] = 1.0, np.nan
        got = _locate(win, mS, **kw)[0]
        assert (got["cy"], got["cx"], got["flags"]) == (mS, mS + 1, 0) and np.isnan(got["corr"])
        assert (got["sy"], got["sx"]) == (-8.0, 1.0 + (1.0 - 128.0) / 16)


def test_whole_planes_of_nan():
    """The same for a plane that lies inside the search disc as a whole."""
    torch, lib = _init()
    n, Cc = 2, 32
    P = torch.full((n, Cc, Cc), float("nan"), device="cuda")
    P[1] = 0.0
    P[1, 20, 12] = 1.0
    wb = lib.zr_full_work_bytes(n, Cc)
    work = torch.empty(wb, dtype=torch.uint8, device="cuda")
    sel = torch.arange(n, dtype=torch.int32, device="cuda")
    rolls = torch.zeros(n, 2, dtype=torch.int32, device="cuda")
    mean, origin = torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    sigma, nfev = torch.ones(n, dtype=torch.float64, device="cuda"), torch.ones(n, dtype=torch.int32, device="cuda")
    out = torch.zeros((n, C.sizeof(_lib.PeakResult)), dtype=torch.uint8, device="cuda")
    _lib.call("zr_full_peaks", P.data_ptr(), P.data_ptr(), n, Cc, sel.data_ptr(), n, 64, rolls.data_ptr(),
              mean.data_ptr(), origin.data_ptr(), sigma.data_ptr(), nfev.data_ptr(), 16, out.data_ptr(),
              work.data_ptr(), wb, gh.stream())
    torch.cuda.synchronize()
    r = np.frombuffer(out.cpu().numpy().tobytes(), dtype=gh.PEAK_DTYPE)
    assert (r["cy"].tolist(), r["cx"].tolist(), r["flags"].tolist()) == ([0, 20], [0, 12], [1, 0])
    assert np.isnan(r["corr"][0]) and abs(r["corr"][1] - 1.0) < 1e-5


@pytest.mark.parametrize("mS", [8, 9, 20, 33, 47, 48, 51, 100, 112])
@pytest.mark.parametrize("use_mask", [0, 1])
@pytest.mark.parametrize("M", [1, 20, 60, 160])
def test_unfiltered_windows(mS, use_mask, M):
    """Without a filter the peak is the first largest value of the window or its
    disc (zeros outside compete) and its significance (max - mean) / std.  The
    statistics are float32 sums of at most 49 pixels a thread and 5 levels of a
    warp, float64 above: std is within 28 roundings, mean within 56 of std."""
    w = 2 * mS
    win = _windows(np.random.default_rng(mS), M, mS)
    win[1::2] = np.round(win[1::2] * np.float32(2000.0))  # ties
    y, x = np.mgrid[:w, :w] - mS
    disc = (y * y + x * x < mS * mS) if use_mask else np.ones((w, w), bool)
    got = _locate(win, mS, bmode=0, use_mask=use_mask, sub_pix_reg=1, suppress_origin=0)
    for k in range(M):
        at = int(np.argmax(np.where(disc, win[k], np.float32(0.0))))
        r, v = got[k], win[k].astype(np.float64)
        assert (r["cy"], r["cx"], r["corr"]) == (at // w, at % w, win[k].flat[at])
        assert (r["sy"], r["sx"]) == (at // w - mS, at % w - mS)
        sig = (np.where(disc, v, 0.0).max() - v[disc].mean()) / v[disc].std()
        assert abs(r["peaksig"] - sig) <= 2.0 ** -24 * (30 * sig + 60), (k, r["peaksig"], sig)


@pytest.mark.parametrize("mS", [8, 9, 25, 47, 48])
def test_one_windows_record_at_any_number(mS):
    """Around a wave of 152 windows, and on both sides of the size from which
    windows are split over CTAs, a window's record is the one it has alone."""
    win = _windows(np.random.default_rng(mS), 154, mS)
    whole = _locate(win, mS)
    for k in (0, 1, 152, 153):
        assert _locate(win[k:k + 1], mS).tobytes() == whole[k:k + 1].tobytes(), k
    assert _locate(win[:153], mS).tobytes() == whole[:153].tobytes()


class _KernelNode(C.Structure):
    """CUDA_KERNEL_NODE_PARAMS of the driver API."""
    _fields_ = [("func", C.c_void_p), ("grid", C.c_uint * 3), ("block", C.c_uint * 3), ("smem", C.c_uint),
                ("params", C.c_void_p), ("extra", C.c_void_p), ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def _grids(calls):
    """The grids of the two kernels that ``calls(stream)`` launches, in order,
    from a captured graph (nothing runs)."""
    torch = gh.torch_mod()
    cu = C.CDLL("libcuda.so.1")
    st = torch.cuda.Stream()
    s = C.c_void_p(st.cuda_stream)
    graph, n = C.c_void_p(), C.c_size_t(2)
    assert cu.cuStreamBeginCapture_v2(s, 2) == 0
    try:
        calls(st.cuda_stream)
    finally:
        assert cu.cuStreamEndCapture(s, C.byref(graph)) == 0
    nodes, root, one = (C.c_void_p * 2)(), (C.c_void_p * 1)(), C.c_size_t(1)
    assert cu.cuGraphGetNodes(graph, nodes, C.byref(n)) == 0 and n.value == 2
    assert cu.cuGraphGetRootNodes(graph, root, C.byref(one)) == 0 and one.value == 1
    got = []
    for node in [root[0]] + [v for v in nodes if v != root[0]]:
        p = _KernelNode()
        assert cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)) == 0
        got.append(tuple(p.grid))
    assert cu.cuGraphDestroy(graph) == 0
    return got


@pytest.mark.parametrize("P", [64, 128, 256, 512, 1024, 1536, 2048, 3072, 4096, 6144])
def test_spectra_run_the_planned_sequences_per_cta(P):
    """A choice of 1, 2 or 4 sequences per CTA is what runs, for every length
    (a choice of 2 ran four rows below 2048 points, one of 4 two at 6144)."""
    torch, lib = _init()
    Cc, N, H = min(P, 1024), 3, P - 3
    raw = torch.zeros(N, H, P, dtype=torch.uint8, device="cuda")
    fr = _frames(raw, _lib.ZR_U8)
    K4 = lib.zr_spectrum_pitch(Cc)
    G = torch.empty(2, N, K4, Cc + 4, 2, device="cuda")
    wb = lib.zr_spectra_work_bytes(H, N, Cc)
    work = torch.empty(wb, dtype=torch.uint8, device="cuda")
    shape = _lib.PlanShape(P, P, Cc, Cc, 8, 2)
    try:
        for rows in (1, 2, 4):
            cols = {1: 2, 2: 4, 4: 1}[rows]
            _lib.call("zr_plan_set", C.byref(shape), C.byref(_lib.PlanChoice(rows, cols, 0, 0)))
            a, b = _grids(lambda st: _lib.call("zr_spectra", C.byref(fr), None, None, 0, N, 0, P, P, Cc, Cc,
                                               G[0].data_ptr(), G[1].data_ptr(), work.data_ptr(), wb, st))
            assert a == (N, -(-H // rows), 1) and b == (K4 // cols, N, 2)
    finally:
        _lib.call("zr_plan_set", C.byref(shape), C.byref(_lib.PlanChoice(0, 0, 0, 0)))


@pytest.mark.parametrize("Cc", [64, 128, 256, 384, 512, 768, 1024, 1536, 2048, 3072, 4096])
@pytest.mark.parametrize("half", [False, True])
def test_windows_run_the_planned_sequences_per_cta(Cc, half):
    """The same for the correlation windows, narrow ones and whole planes, from
    float32 and from half-precision spectra."""
    torch, lib = _init()
    N, M = 2, 1
    K4 = lib.zr_spectrum_pitch(Cc)
    G = torch.empty(N, K4, Cc + 4, 2, dtype=torch.float16 if half else torch.float32, device="cuda")
    sc = torch.ones(2 * N + 1, device="cuda")
    pairs = torch.tensor([0, 1], dtype=torch.int32, device="cuda")
    try:
        for mS in (8, Cc // 2):
            w = 2 * mS
            terms, win = torch.empty(4 * N + 1, w, w, device="cuda"), torch.empty(M, w, w, device="cuda")
            wb = lib.zr_xcorr_work_bytes(M, Cc, mS)
            work = torch.empty(wb, dtype=torch.uint8, device="cuda")
            shape = _lib.PlanShape(Cc, Cc, Cc, Cc, mS, 2)
            for cols in (1, 2, 4):
                rows = {1: 2, 2: 4, 4: 1}[cols]
                _lib.call("zr_plan_set", C.byref(shape), C.byref(_lib.PlanChoice(0, 0, cols, rows)))
                head = [G.data_ptr()] + ([sc.data_ptr()] if half else [])
                a, b = _grids(lambda st: _lib.call("zr_xcorr_pairs_half" if half else "zr_xcorr_pairs", *head,
                                                   terms.data_ptr(), pairs.data_ptr(), M, N, Cc, Cc, mS,
                                                   win.data_ptr(), work.data_ptr(), wb, st))
                assert a == (M, K4 // cols, 1) and b == (-(-w // (2 * rows)), M, 1)
    finally:
        _lib.call("zr_plan_set", C.byref(shape), C.byref(_lib.PlanChoice(0, 0, 0, 0)))


def test_gain_sum_total_keeps_float64():
    """A thread's share of the total keeps every bit that a float64 sum of its
    pixels keeps: 16 shares of 1 + 2^-25 (1 + 2^-23) + 2^-26 (1 + 2^-23), whose
    sum needs 50 bits, add up exactly, on the vector and on the pixel path."""
    torch, _ = _init()
    share = [1.0, 2.0 ** -25 * (1 + 2.0 ** -23), 2.0 ** -26 * (1 + 2.0 ** -23), 0.0]
    img = np.tile(np.array(share, np.float32), 16).reshape(1, 8, 8)
    want = 16 * (share[0] + share[1] + share[2])
    assert (share[0] + share[1]) - share[0] == share[1]  # float64 holds it
    for off in (0, 1):  # one float past the vector boundary: pixel by pixel
        arena = torch.zeros(65, device="cuda")
        arena[off:off + 64] = torch.from_numpy(img.ravel()).cuda()
        fr = _lib.Frames(arena.data_ptr() + 4 * off, _lib.ZR_F32, None, None, None, 0.0, 1, 8, 8, 0)
        out = torch.empty(64, device="cuda")
        total = torch.zeros(1, dtype=torch.float64, device="cuda")
        _lib.call("zr_gain_sum", C.byref(fr), out.data_ptr(), total.data_ptr(), gh.stream())
        assert total.item() == want, (off, total.item() - want)
        assert np.array_equal(out.cpu().numpy().reshape(8, 8), img[0])


@pytest.mark.parametrize("H,W", [(5, 7), (64, 64), (201, 181), (700, 1000)])
@pytest.mark.parametrize("nbins", [1, 48, 103, 767, 769, 1600, 12289, 20000, 32768])
def test_histogram_of_any_number_of_bins(H, W, nbins):
    """Counts equal np.histogram's whatever the number of bins, hence of copies
    a CTA counts in, over values on and around the edges and outside them."""
    torch, _ = _init()
    rng = np.random.default_rng(nbins)
    v = (rng.normal(nbins / 2, nbins / 3, (H, W))).astype(np.float32)
    v.flat[::3] = np.round(v.flat[::3] * 2) / 2
    v.flat[:4] = [-0.5, nbins - 0.5, np.nextafter(np.float32(nbins - 0.5), np.float32(1e9)), np.inf]
    want = np.histogram(v[np.isfinite(v)].astype(np.float64), np.arange(nbins + 1) - 0.5)[0]
    dev = torch.from_numpy(v).cuda()
    counts = torch.zeros(nbins + 8, dtype=torch.int32, device="cuda")
    _lib.call("zr_histogram", dev.data_ptr(), H * W, -0.5, nbins, counts.data_ptr(), gh.stream())
    got = counts.cpu().numpy()
    assert np.array_equal(got[:nbins], want) and not got[nbins:].any()


@pytest.mark.parametrize("mu", [16000000.0 + 37 * i for i in range(12)])
def test_hot_maps_of_a_narrow_fit_far_from_zero(mu):
    """The logistic masks of sums whose mean is 1.2e9 fitted sigmas from zero:
    the exponents K (s - mu) / sigma - K c are differences of 7e10, which float64
    holds to 3 x 2^-53 of that, 2.4e-5; a mask moves by at most half of its
    exponents' error, and 2e-5 holds that and the float32 roundings."""
    torch, lib = _init()
    H, W, sigma, K = 8, 12, 0.0137, float(np.float32(59.3))
    p = _lib.HotpixParams()
    p.mu, p.sigma, p.cutoff_lower, p.cutoff_upper = mu, sigma, -0.01, 0.02
    p.logistic_k, p.relax, p.neighbour_thres, p.best_mean = K, 1.0, 0.01, mu / 10
    for i, v in enumerate(hm.psf_kernel("K2").ravel()):
        p.psf[i] = float(v)
    s = np.full((H, W), mu, np.float32)
    s[3, 4], s[5, 7] = mu + 1, mu - 1
    assert float(s[0, 0]) == mu
    dev = torch.from_numpy(s).cuda()
    a, b = torch.empty(H, W, device="cuda"), torch.empty(H, W, device="cuda")
    counts = torch.zeros(4, dtype=torch.int32, device="cuda")
    wb = lib.zr_hotpix_work_bytes(H, W)
    work = torch.empty(wb, dtype=torch.uint8, device="cuda")
    _lib.call("zr_hotpix_maps", dev.data_ptr(), H, W, 10, C.byref(p), a.data_ptr(), b.data_ptr(), counts.data_ptr(),
              work.data_ptr(), wb, gh.stream())
    sg = (s.astype(np.float64) - mu) / sigma
    with np.errstate(over="ignore"):
        e1, e2 = np.exp(K * (sg - float(np.float32(-0.01)))), np.exp(K * (sg - float(np.float32(0.02))))
        want = (1.0 - 1.0 / (1.0 + e1)) / (1.0 + e2)
    assert np.abs(a.cpu().numpy() - want).max() <= 2e-5
    assert counts.cpu().tolist()[:2] == [1, 1]


@pytest.mark.parametrize("box", [128, 256, 512, 1024])
def test_rings_are_float64_means_of_the_plane(box):
    """The FRC of one tile is exactly 1 at zero frequency, so frc2d holds the
    plane that the rings average without a rounding: they are its rotational
    mean (bilinear split, in extended precision here) within 4e-14: weights off
    by 2^-47, twice a ring's weight of them in the sum and in its divisor, and
    30 roundings of 2^-53."""
    torch, lib = _init()
    rng = np.random.default_rng(box)
    base = rng.poisson(300.0, (box, box))
    e, o = (torch.from_numpy((base + rng.poisson(60.0, (box, box))).astype(np.float32)).cuda() for _ in range(2))
    offs = torch.zeros(2, dtype=torch.int32, device="cuda")
    nr = int(np.ceil(np.sqrt(2.0) * (box // 2))) + 1
    wb = lib.zr_frc_work_bytes(1, box)
    work = torch.empty(wb, dtype=torch.uint8, device="cuda")
    frc2d, frc = torch.empty(box, box, device="cuda"), torch.empty(nr, dtype=torch.float64, device="cuda")
    _lib.call("zr_tiled_frc", e.data_ptr(), o.data_ptr(), box, box, box, offs.data_ptr(), 1, frc2d.data_ptr(),
              frc.data_ptr(), nr, work.data_ptr(), wb, gh.stream())
    v = frc2d.cpu().numpy().astype(np.longdouble)
    assert v[box // 2, box // 2] == 1.0
    x = np.arange(box) - box // 2
    rho = np.sqrt((x[:, None] ** 2 + x[None, :] ** 2).astype(np.longdouble))
    b0 = np.floor(rho).astype(int)
    num, den = np.zeros(nr + 1, np.longdouble), np.zeros(nr + 1, np.longdouble)
    for k, w in ((b0, 1 - (rho - b0)), (b0 + 1, rho - b0)):
        np.add.at(num, k, v * w)
        np.add.at(den, k, w)
    live = den[:nr] > 0
    assert np.abs(frc.cpu().numpy()[live] - (num[:nr] / den[:nr])[live]).max() <= 4e-14


def _hot_maps(s, sigma, n=10, mu=20.0):
    torch, lib = _init()
    H, W = s.shape
    p = _lib.HotpixParams()
    p.mu, p.sigma, p.cutoff_lower, p.cutoff_upper = mu, sigma, -4.0, 3.25
    p.logistic_k, p.relax, p.neighbour_thres, p.best_mean = 6.0, 0.925, 0.01, mu / n
    for i, k in enumerate(hm.psf_kernel("K2").ravel()):
        p.psf[i] = float(k)
    ds = torch.from_numpy(s).cuda()
    a, b = (torch.full((H, W), 7.0, device="cuda") for _ in range(2))
    cnt = torch.zeros(4, dtype=torch.int32, device="cuda")
    wb = lib.zr_hotpix_work_bytes(H, W)
    work = torch.empty(wb, dtype=torch.uint8, device="cuda")
    _lib.call("zr_hotpix_maps", ds.data_ptr(), H, W, n, C.byref(p), a.data_ptr(), b.data_ptr(), cnt.data_ptr(),
              work.data_ptr(), wb, gh.stream())
    return p, a.cpu().numpy(), b.cpu().numpy(), cnt.cpu().tolist()


@pytest.mark.parametrize("H,W", [(4, 4), (7, 63), (8, 64), (9, 65), (33, 130), (385, 833)])
def test_hot_fill_and_counts_at_tile_edges(H, W):
    """Both maps and all three counts against a float64 restatement (scipy's
    reflected convolution, the neighbour mean with the reference's slices), with
    single outliers, pairs and blocks of them on the rows and columns where
    tiles of 8 and of 32 rows meet and on the image's border, and a NaN.  Masks:
    exponents rounded to float32, as test_hotpix_map_tiles has it.  Fill: nine-tap
    float32 sums and the masks' error, 2e-6 and 2e-5 of the largest value a
    pixel's neighbourhood holds.  Pixels whose mask product lies within rounding
    of its threshold are left out, and what a NaN reaches."""
    import scipy.ndimage
    rng = np.random.default_rng(H * W)
    n, mu, sigma = 10, 20.0, 3.0
    s = rng.normal(mu, sigma, (H, W)).clip(mu - 2 * sigma, mu + 1.5 * sigma).astype(np.float32)
    ys = [y for y in (0, 1, 6, 7, 8, 9, 30, 31, 32, 33, 63, 64, 383, H - 1) if y < H]
    xs = [x for x in (0, 1, 62, 63, 64, 65, 127, 128, 767, 768, W - 1) if x < W]
    for y in ys:
        for x in xs:
            if rng.random() < 0.6:
                s[y, x] = rng.choice([0.0, 55.0, 90.0])
    if H > 32:
        s[20:24, 40:44] = 80.0
        s[12, 100] = np.nan
    p, a, b, counts = _hot_maps(s, sigma)
    v = s.astype(np.float64)
    with np.errstate(all="ignore"):
        q = (v - mu) / sigma
        lo, up = (np.float64(np.float32(c) * np.float32(0.925)) for c in (-4.0, 3.25))
        lm = (1.0 - 1.0 / (1.0 + np.exp(6.0 * (q - lo)))) / (1.0 + np.exp(6.0 * (q - up)))
        psf = hm.psf_kernel("K2").astype(np.float64).reshape(3, 3)
        conv, mean = 1.0 - lm, v / n
        nom = conv * scipy.ndimage.convolve(conv, psf, mode="reflect")
        mask = nom > p.neighbour_thres
        fill = conv * ~mask * scipy.ndimage.convolve(mean, psf, mode="reflect")
        for y, x in zip(*np.where(mask)):
            hood = mask[y - 1:y + 2, x - 1:x + 2]  # empty where it would start at -1
            ratio = hood.sum() / hood.size if hood.size else np.nan
            if ratio > 0.66 or ratio <= 0.001 or np.isnan(ratio):
                fill[y, x] += mu / n
            else:
                fill[y, x] += conv[y, x] * mean[y - 1:y + 2, x - 1:x + 2][~hood].mean()
    assert counts[:2] == [np.sum(q < -4.0), np.sum(q > 3.25)]
    np.testing.assert_allclose(a, lm, rtol=0, atol=88 * 2.0 ** -24 / 4 + 5e-7)
    close = np.abs(nom - p.neighbour_thres) < 1e-5
    assert abs(counts[2] - mask.sum()) <= close.sum()
    out = scipy.ndimage.maximum_filter((close | np.isnan(v)).astype(np.uint8), 5) > 0
    big = scipy.ndimage.maximum_filter(np.nan_to_num(mean), 5)
    assert np.isnan(b[np.isnan(v)]).all() and np.isfinite(b[~out]).all() and out.mean() < 0.5
    assert np.all(np.abs(b - fill)[~out] <= (2e-5 * big)[~out])
    assert H < 9 or counts[2] > 0


def test_hot_maps_of_a_fit_without_width():
    """sigma_fit 0: every sum but the mean itself is masked out, and that one is
    0 times infinity, as the step by step formula has it."""
    s = np.full((40, 70), 20.0, np.float32)
    s[::3, ::2] = np.linspace(-5.0, 60.0, s[::3, ::2].size).reshape(s[::3, ::2].shape)
    _, a, _, counts = _hot_maps(s, 0.0)
    assert np.array_equal(np.isnan(a), s == 20.0) and np.all(a[s != 20.0] == 0.0)
    assert counts[:2] == [np.sum(s < 20.0), np.sum(s > 20.0)]


@pytest.mark.parametrize("kind", ["u8", "u16", "f16", "f32"])
@pytest.mark.parametrize("gain,hot", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("H,W", [(301, 303), (501, 703), (701, 703), (905, 1003), (1501, 1003)])
def test_shift_sum_paths_agree(kind, gain, hot, H, W):
    """Frames that lie one after the other with an odd number of pixels are read
    pixel by pixel, a frame ahead or not by the number of tiles and by their
    maps; the same frames a multiple of four elements apart in chunks of four
    pixels.  Sums, half sums and aligned frames are the same bits, for rolls
    that wrap in both directions and a frame that is not filtered."""
    torch, _ = _init()
    rng = np.random.default_rng(H + W)
    N = 4
    np_t, z = {"u8": (np.uint8, _lib.ZR_U8), "u16": (np.uint16, _lib.ZR_U16), "f16": (np.float16, _lib.ZR_F16),
               "f32": (np.float32, _lib.ZR_F32)}[kind]
    raw = rng.poisson(4.0, (N, H * W)).astype(np_t)
    stride = (H * W + 3) // 4 * 4
    spread = np.zeros((N, stride), np_t)
    spread[:, :H * W] = raw
    dev = [torch.from_numpy(v.view(np.int16) if kind == "u16" else v).cuda() for v in (raw, spread)]
    maps = [torch.from_numpy(rng.uniform(0.9, 1.1, (H, W)).astype(np.float32)).cuda() for _ in range(3)]
    ptr = [m.data_ptr() if on else None for m, on in zip(maps, (gain, hot, hot))]
    t = np.array([[0.0, 0.0], [3.25, -7.5], [-11.0625, 4.75], [0.5, 250.125]])
    sh = torch.from_numpy(hm.shift_table(t, H, W).view(np.uint8)).cuda()
    got = []
    for v, gap in zip(dev, (0, stride)):
        fr = _lib.Frames(v.data_ptr(), z, *ptr, 0.0, N, H, W, gap)
        for halves in (False, True):
            out, ali = torch.zeros(3, H, W, device="cuda"), torch.zeros(N, H, W, device="cuda")
            h = [out[i].data_ptr() if halves else None for i in (1, 2)]
            _lib.call("zr_shift_sum", C.byref(fr), sh.data_ptr(), out[0].data_ptr(), *h, ali.data_ptr(), gh.stream())
            got.append((out, ali))
    for out, ali in got[1:]:
        assert torch.equal(ali, got[0][1]) and torch.equal(out[0], got[0][0][0])
    assert torch.equal(got[1][0], got[3][0])
    assert torch.equal(got[1][0][1], got[0][1][0] + got[0][1][2])


@pytest.mark.parametrize("kind,maps,H,W,P,Cc", [
    ("u8", True, 57, 61, 64, 64), ("f32", False, 100, 128, 128, 64), ("f16", True, 200, 233, 256, 128),
    ("u16", False, 301, 499, 512, 256), ("f32", True, 997, 1001, 1024, 512), ("u8", False, 1500, 1533, 1536, 768),
    ("u8", True, 2040, 1999, 2048, 1024), ("f32", False, 3000, 3071, 3072, 1536)])
def test_spectra_of_masked_frames_and_of_masks(kind, maps, H, W, P, Cc):
    """G and S of frames under a mask of any values, the mask's own spectrum and
    that of the default mask, against float64 transforms: 6e-8 log2 of the
    transform's length in the 2-norm, twice that for the squares."""
    torch, lib = _init()
    rng = np.random.default_rng(P)
    N = 2
    np_t, z = {"u8": (np.uint8, _lib.ZR_U8), "u16": (np.uint16, _lib.ZR_U16), "f16": (np.float16, _lib.ZR_F16),
               "f32": (np.float32, _lib.ZR_F32)}[kind]
    raw = rng.poisson(5.0, (N, H, W)).astype(np_t)
    dev = torch.from_numpy(raw.view(np.int16) if kind == "u16" else raw).cuda()
    mask = rng.uniform(0.0, 1.0, (P, P)).astype(np.float32) * (rng.random((P, P)) > 0.1)
    host = [rng.uniform(0.9, 1.1, (H, W)).astype(np.float32) for _ in range(3)] if maps else []
    dm = [torch.from_numpy(m).cuda() for m in host]
    fr = _lib.Frames(dev.data_ptr(), z, *([m.data_ptr() for m in dm] if maps else [None] * 3), 0.0, N, H, W, 0)
    v = raw.astype(np.float64)
    if maps:
        v = v * host[0] * host[1] + host[2]
    K4 = lib.zr_spectrum_pitch(Cc)
    G, S = (torch.empty(N, K4, Cc + 4, 2, device="cuda") for _ in range(2))
    sums = torch.from_numpy(v.reshape(N, -1).sum(1)).cuda()
    wb = lib.zr_spectra_work_bytes(P, N, Cc)
    work = torch.empty(wb, dtype=torch.uint8, device="cuda")
    dmask = torch.from_numpy(mask).cuda()

    def layout(u):
        F = np.fft.rfft2(u)
        rows = [r if r < Cc // 2 else P - Cc + r for r in range(Cc)] + [Cc // 2]
        return F[rows][:, :Cc // 2 + 1].T

    def check(t, u, tol):
        got = t.cpu().numpy().astype(np.float64)
        got = (got[..., 0] + 1j * got[..., 1])[:Cc // 2 + 1, :Cc + 1]
        want = layout(u)
        assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)

    tol = 6e-8 * 2 * np.log2(P)
    _lib.call("zr_spectra", C.byref(fr), dmask.data_ptr(), sums.data_ptr(), 0, N, 0, P, P, Cc, Cc, G.data_ptr(),
              S.data_ptr(), work.data_ptr(), wb, gh.stream())
    for n in range(N):
        mu = float(np.float32(sums[n].item() / (H * W)))
        u = np.zeros((P, P))
        u[:H, :W] = mask[:H, :W].astype(np.float64) * (v[n] - mu)
        check(G[n], u, tol)
        check(S[n], u * u, 2 * tol)
    for m, u in ((dmask.data_ptr(), mask.astype(np.float64)), (None, np.pad(np.ones((H, W)), ((0, P - H), (0, P - W))))):
        _lib.call("zr_spectra", C.byref(fr), m, None, 0, 1, 1, P, P, Cc, Cc, G.data_ptr(), None, work.data_ptr(), wb,
                  gh.stream())
        check(G[0], u, tol)
