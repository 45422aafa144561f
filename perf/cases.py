"""What the performance of this library is measured on.

Each case is one call (or the fixed sequence of calls) that a program using the library makes
through its public entry points: correlation maps of given spectra, one rank's part of a
sharded search, whole searches of one or several micrographs in the forms people run, and score
gradients of picks.  Micrographs are seeded noise with a few planted, CTF-modulated particles,
templates are projections of a blob map; both are made on the GPU.  Thresholds lie above the
noise so that the number of picks stays at the tens a search of a few particles gives; picks
land in a buffer of fixed size that the program keeps, as the C interface has it.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gisspa_v2.0_b200"))
import gisspa  # noqa: E402

PI = 3.1415926535  # the reference's own constant (utils/constants.h)


def listed():
    return [
        # correlation maps of one window with a handful of templates: the smallest call, an
        # interactive check of one particle's surroundings
        dict(name="maps_512_small", kind="maps", window=512, windows=1, templates=8, spec="fp32", noalloc=False),
        # the same through the entry point for callers that own the device memory, half-precision spectra
        dict(name="maps_256_noalloc_fp16", kind="maps", window=256, windows=3, templates=20, spec="fp16", noalloc=True),
        # maps of large windows, enough pairs to fill the GPU
        dict(name="maps_1024", kind="maps", window=1024, windows=4, templates=24, spec="fp32", noalloc=False),
        # the flagship search: a 4096^2 micrograph, 512 windows with 192 px overlap, 5 degree
        # steps, reference picks; 40 templates keep a pass below half a second
        dict(name="search_4096_w512", kind="search", nx=4096, ny=4096, window=512, overlap=192, templates=40,
             tsize=180, step=5.0, spec="fp32", pick="chunk", particles=20, signal=0.3, threshold=7.5),
        # one rank's part of a sharded one-sweep search with half-precision spectra: the merged
        # per-pixel sums and the picks
        dict(name="shard_2048_w512_fp16", kind="shard", nx=2048, ny=2048, window=512, overlap=192, templates=50,
             tsize=180, step=10.0, spec="fp16", pick="topk", particles=10, signal=0.6, threshold=6.5),
        # the same at the reference's default window size, FP32 spectra, an uneven micrograph
        dict(name="shard_1855_w320", kind="shard", nx=1855, ny=1919, window=320, overlap=120, templates=37,
             tsize=128, step=15.0, spec="fp32", pick="topk", particles=10, signal=0.8, threshold=6.0),
        # large windows (big particles): 3838 x 3710, a size that is no product of small primes
        dict(name="search_3710_w1024", kind="search", nx=3838, ny=3710, window=1024, overlap=256, templates=24,
             tsize=256, step=10.0, spec="fp32", pick="chunk", particles=8, signal=0.4, threshold=8.0),
        # a small search: a cropped micrograph, few small templates (a quick look, a test run)
        dict(name="search_768_w256", kind="search", nx=768, ny=768, window=256, overlap=64, templates=8, tsize=64,
             step=10.0, spec="fp32", pick="topk", particles=4, signal=1.2, threshold=4.6),
        # a window size without hand-tuned kernels
        dict(name="search_1500_w336", kind="search", nx=1500, ny=1401, window=336, overlap=100, templates=20,
             tsize=120, step=12.0, spec="fp32", pick="topk", particles=6, signal=0.8, threshold=5.7),
        # norm_type=0, the reference's tiled search: 1024^2 in 720^2 tiles, 8 templates, 10 degree steps
        dict(name="tiled_1024_w512", kind="tiled", nx=1024, ny=1024, window=512, overlap=128, templates=8, tsize=128,
             step=10.0, spec="fp32", pick="chunk", particles=4, signal=0.8, threshold=18.0),
        # several micrographs of uneven size in one call
        dict(name="batch_3_w512", kind="batch", nx=2048, ny=2048, window=512, overlap=200, templates=24, tsize=200,
             step=12.0, spec="fp32", pick="topk", particles=8, signal=0.6, threshold=6.0),
        # scores and gradients of picks (refinement's inner call) after a search
        dict(name="grad_2000", kind="grad", nx=2048, ny=2048, window=512, overlap=192, templates=12, tsize=180,
             step=30.0, spec="fp32", pick="topk", particles=10, signal=0.6, threshold=6.0, picks=2000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: other sizes (odd ones among them), windows, types."""
    kind = rng.choice(["maps", "maps", "search", "search", "search", "shard", "shard", "tiled", "batch", "grad"])
    spec = rng.choice(["fp32", "fp32", "fp16", "bf16"])
    if kind == "maps":
        w = rng.choice([256, 320, 512, 1024])
        noalloc = w != 320 and rng.random() < 0.4
        if noalloc:
            windows = rng.choice([1, 2])
            templates = rng.randint(1, max(1, (16 << 20) // (4 * w * w) // windows))
        else:
            windows, templates = rng.randint(1, 4), _log(rng, 1, 24 if w == 1024 else 64)
        return dict(kind="maps", window=w, windows=windows, templates=templates, spec=spec, noalloc=noalloc)
    if kind == "tiled":
        t = rng.randint(80, 140)
        return dict(kind="tiled", nx=rng.randint(960, 1300), ny=rng.randint(960, 1300), window=rng.choice([256, 512]),
                    overlap=128, templates=rng.randint(3, 10), tsize=t, step=rng.choice([10.0, 15.0, 20.0]),
                    spec="fp32", pick="chunk", particles=3, signal=0.8, threshold=18.0)
    w = rng.choice([256, 320, 320, 512, 512, 512, 1024, 336, 400])
    if kind == "grad":
        w = rng.choice([256, 512, 1024])
    t = {256: 96, 320: 128, 336: 120, 400: 150, 512: 180, 1024: 256}[w] - rng.randint(0, 20)
    side = 2600 if w in (512, 1024) else 1700
    big = spec == "fp32" and rng.random() < 0.5 and kind in ("search", "shard") and w not in (336, 400)
    nx, ny = _log(rng, w + 200, side), _log(rng, w + 200, side)
    nt = _log(rng, 10, 40 if big else 24)
    step = rng.choice([10.0, 12.0, 15.0])
    c = dict(kind=kind, nx=nx, ny=ny, window=w, overlap=rng.choice([w // 4, w // 3, 3 * w // 8]), templates=nt,
             tsize=t, step=step, spec=spec, pick="topk", particles=max(2, (nx - 2 * t) * (ny - 2 * t) // 400000),
             signal=round(100.0 / t, 2), threshold=4.9 if w == 256 else 5.3)
    if kind == "search" and w not in (336, 400) and rng.random() < 0.5:
        c.update(pick="chunk", threshold=5.0 if w == 256 else 6.0)
    if kind == "grad":
        c.update(step=30.0, templates=rng.randint(4, 16), picks=_log(rng, 50, 2000))
    return c


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _render(px, py, sig, amp, w, h):
    """[n][h][w] sums of 2D Gaussians amp exp(-r^2 / 2 sig^2) at (px, py), one set of blobs per image."""
    xs = torch.arange(w, device="cuda", dtype=torch.float64)
    ys = torch.arange(h, device="cuda", dtype=torch.float64)
    gx = torch.exp(-((xs - px[..., None]) ** 2) / (2 * sig[:, None] ** 2))
    gy = torch.exp(-((ys - py[..., None]) ** 2) / (2 * sig[:, None] ** 2)) * amp[:, None]
    return gy.transpose(1, 2) @ gx


def _blobs(g, n, tsize):
    """Blob map and its projections' 2D centres at n random orientations: (x, y) [n][blobs], sigma, amplitude."""
    nb = 60
    d = torch.randn((nb, 3), generator=g, device="cuda", dtype=torch.float64)
    c = d / d.norm(dim=1, keepdim=True) * 0.3 * tsize * _uniform(g, 0, 1, nb, 1) ** (1 / 3)
    sig = _uniform(g, 2.0, 4.0, nb)
    amp = _uniform(g, 0.5, 1.0, nb)
    alt = torch.arccos(_uniform(g, -1, 1, n))
    az = _uniform(g, 0, 2 * math.pi, n)
    ca, sa, cz, sz = torch.cos(alt), torch.sin(alt), torch.cos(az), torch.sin(az)
    x = cz[:, None] * c[:, 0] - sz[:, None] * c[:, 1]
    y = ca[:, None] * (sz[:, None] * c[:, 0] + cz[:, None] * c[:, 1]) - sa[:, None] * c[:, 2]
    return x, y, sig, amp


def _ctf_plain(ny, nx, ctf):
    """Signed CTF of the simulated microscope on the rfft2 grid."""
    lam = 12.2639 / math.sqrt(300.0 * 1000.0 + 0.97845 * 300.0 * 300.0)
    fy = torch.fft.fftfreq(ny, device="cuda", dtype=torch.float64)[:, None]
    fx = torch.fft.rfftfreq(nx, device="cuda", dtype=torch.float64)[None, :]
    s2 = fx * fx + fy * fy
    df = (ctf.defocus + ctf.dfdiff * torch.cos(2 * (math.radians(ctf.dfang) - torch.atan2(fy, fx)))) * 1e4
    gamma = math.pi * lam * df * s2 - 0.5 * math.pi * 2.7e7 * lam ** 3 * s2 * s2
    return math.sqrt(1 - 0.07 ** 2) * torch.sin(gamma) + 0.07 * torch.cos(gamma)


def _diameter(case):
    return 0.75 * case["tsize"]


def _micrograph(g, case, x, y, sig, amp, ctf, nx, ny):
    """Noise with `particles` copies of random templates at random in-plane angles, apart from one another."""
    t, p = case["tsize"], case["particles"]
    margin = int(_diameter(case)) + t // 2
    cx = max(1, (nx - 2 * margin) // (t + t // 4))
    cy = max(1, (ny - 2 * margin) // (t + t // 4))
    p = min(p, cx * cy)
    clean = torch.zeros((ny, nx), device="cuda", dtype=torch.float64)
    cells = torch.randperm(cx * cy, generator=g, device="cuda")[:p].tolist()
    which = torch.randint(0, case["templates"], (p,), generator=g, device="cuda")
    psi = _uniform(g, 0, 2 * math.pi, p)
    sub = _uniform(g, 0, 1, p, 2)
    c, s = torch.cos(psi)[:, None], torch.sin(psi)[:, None]
    rx = c * x[which] - s * y[which] + sub[:, :1] + t / 2
    ry = s * x[which] + c * y[which] + sub[:, 1:] + t / 2
    patch = _render(rx, ry, sig, amp * sig, t, t)
    for k, cell in enumerate(cells):
        x0 = margin - t // 2 + (cell % cx) * (t + t // 4)
        y0 = margin - t // 2 + (cell // cx) * (t + t // 4)
        h, w = min(t, ny - y0), min(t, nx - x0)
        if h > 0 and w > 0 and x0 >= 0 and y0 >= 0:
            clean[y0:y0 + h, x0:x0 + w] += patch[k, :h, :w]
    f = torch.fft.rfft2(clean) * _ctf_plain(ny, nx, ctf)
    clean = torch.fft.irfft2(f, s=(ny, nx))
    rms = patch.square().mean().sqrt()
    noise = torch.randn((ny, nx), generator=g, device="cuda")
    # zero mean, unit noise: a motion-corrected, normalised micrograph
    return (noise + clean.float() * (case["signal"] / rms.float())).cpu().numpy()


_SPEC = {"fp32": gisspa.SPEC_FP32, "fp16": gisspa.SPEC_FP16, "bf16": gisspa.SPEC_BF16}
_TORCH = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}


def _config(case):
    return gisspa.Config.default(
        angpix=1.0, phistep=case["step"], kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=200.0,
        diameter=_diameter(case), threshold=case["threshold"], window_size=case["window"], overlap=case["overlap"],
        norm_type=0 if case["kind"] == "tiled" else 1, spectrum_precision=_SPEC[case["spec"]],
        pick_mode=gisspa.PICK_TOPK if case["pick"] == "topk" else gisspa.PICK_CHUNK,
        topk=100, exclusion_radius=64.0,
        # statistics over the real templates only, also where windows outnumber them
        quirks=gisspa.QUIRK_OUTLIER_FP32_SERIAL | gisspa.QUIRK_NEULER_TRUNC,
        phase_flip=1 if case["kind"] == "tiled" else 0)


def _search_inputs(case, seed):
    g = _gen(seed)
    x, y, sig, amp = _blobs(g, case["templates"], case["tsize"])
    half = case["tsize"] / 2
    stack = _render(x + half, y + half, sig, amp * sig, case["tsize"], case["tsize"]).float().cpu().numpy()
    u = _uniform(g, 0, 1, 3).tolist()
    ctf = gisspa.Ctf(1.2 + 0.8 * u[0], 0.15 * u[1], 180.0 * u[2])
    sizes = [(case["nx"], case["ny"])]
    if case["kind"] == "batch":
        sizes += [(case["nx"] * 7 // 8 + 5, case["ny"]), (case["nx"] * 3 // 4, case["ny"] * 3 // 4 + 2)]
    images = [_micrograph(g, case, x, y, sig, amp, ctf, nx, ny) for nx, ny in sizes]
    return stack, images, ctf


def _map_inputs(case, seed):
    """Window and template half spectra, kx-major, of noise windows and of smooth templates."""
    g = _gen(seed)
    l, w, t = case["window"], case["windows"], case["templates"]
    win = torch.fft.rfft2(torch.randn((w, l, l), generator=g, device="cuda")) / l
    x, y, sig, amp = _blobs(g, t, l // 3)
    tm = _render(x + l / 2, y + l / 2, sig, amp, l, l).float()
    tm = (tm - tm.mean(dim=(1, 2), keepdim=True)) / tm.std(dim=(1, 2), keepdim=True)
    tm = torch.fft.rfft2(tm) / l

    def kx_major(s):
        return torch.view_as_real(s.transpose(1, 2).contiguous())

    return kx_major(win).contiguous(), kx_major(tm).to(_TORCH[case["spec"]]).contiguous()


PICKS = 4096  # the caller's pick buffer, per micrograph


class State:
    pass


def _ok(status):
    if status != gisspa.OK:
        raise RuntimeError(f"status {status}")


def prepare(case, seed):
    s = State()
    s.case = case
    s.lib = gisspa.load()
    if case["kind"] == "maps":
        s.win, s.tmpl = _map_inputs(case, seed)
        l = case["window"]
        s.out = torch.empty((case["windows"], case["templates"], l, l), device="cuda")
        if not case["noalloc"]:
            s.searcher = gisspa.Searcher(gisspa.Config.default(
                angpix=1.0, phistep=10.0, kk=3.0, energy=300.0, cs=2.7, highres=8.0, lowres=200.0, diameter=100.0,
                window_size=l, norm_type=1))
        torch.cuda.synchronize()
        return s
    stack, s.images, s.ctf = _search_inputs(case, seed)
    s.searcher = gisspa.Searcher(_config(case))
    s.searcher.set_templates(stack)
    if case["kind"] == "shard":
        nwin = _windows_along(case["nx"], case) * _windows_along(case["ny"], case)
        n = nwin * case["window"] ** 2
        s.sum = torch.empty(n, device="cuda", dtype=torch.float64)
        s.sum_sq = torch.empty(n, device="cuda", dtype=torch.float64)
        s.key = torch.empty(n, device="cuda", dtype=torch.int64)
    n = len(s.images) * PICKS
    s.picks = np.zeros(n, dtype=gisspa.PICK_DTYPE)
    if case["kind"] == "grad":
        # a search, then sub-pixel offsets around positions in its windows
        s.searcher.search(s.images[0], s.ctf, PICKS)
        s.picks, s.params = _grad_picks(case, seed)
    torch.cuda.synchronize()
    return s


def _windows_along(n, case):
    l, ov = case["window"], case["overlap"]
    return 1 if n <= l else 1 + -(-(n - l) // (l - ov))


def _grad_picks(case, seed):
    """Positions, templates and angles to evaluate: anywhere in the windows of the micrograph."""
    r = np.random.default_rng(seed)
    n, l, ov = case["picks"], case["window"], case["overlap"]
    bx, by = _windows_along(case["nx"], case), _windows_along(case["ny"], case)
    picks = np.zeros(n, dtype=gisspa.PICK_DTYPE)
    picks["window"] = r.integers(0, bx * by, n)
    picks["template_id"] = r.integers(0, case["templates"], n)
    picks["theta"] = r.uniform(0, 360, n)
    ox = np.minimum((picks["window"] % bx) * (l - ov), max(case["nx"] - l, 0))
    oy = np.minimum((picks["window"] // bx) * (l - ov), max(case["ny"] - l, 0))
    picks["x"] = ox + r.integers(l // 4, 3 * l // 4, n)
    picks["y"] = oy + r.integers(l // 4, 3 * l // 4, n)
    params = np.stack([r.uniform(-0.5, 0.5, n), r.uniform(-0.5, 0.5, n), picks["theta"]], 1).astype(np.float32)
    return picks, params


def _pick_arrays(p):
    return {k: np.ascontiguousarray(p[k]) for k in ("score", "x", "y", "angle", "template_id", "window", "tile",
                                                    "angle_index", "chunk")}


def run(s):
    case = s.case
    if case["kind"] == "maps":
        spec = _SPEC[case["spec"]]
        if case["noalloc"]:
            st = s.lib.gisspa_cc_maps_noalloc(s.win.data_ptr(), case["windows"], s.tmpl.data_ptr(), case["templates"],
                                              case["window"], spec, s.out.data_ptr(),
                                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        else:
            st = s.lib.gisspa_cc_maps(s.searcher.h, s.win.data_ptr(), case["windows"], s.tmpl.data_ptr(),
                                      case["templates"], spec, s.out.data_ptr())
        _ok(st)
        return s.out
    if case["kind"] == "shard":
        info = s.searcher.shard_begin(s.images[0], s.ctf)
        s.searcher.shard_sweep(1, 0, info.n_angles)
        s.searcher.shard_export(s.sum.data_ptr(), s.sum_sq.data_ptr(), s.key.data_ptr())
        s.searcher.shard_import(s.sum.data_ptr(), s.sum_sq.data_ptr(), s.key.data_ptr())
        count = ctypes.c_size_t(0)
        _ok(s.lib.gisspa_shard_picks(s.searcher.h, s.picks.ctypes.data, PICKS, ctypes.byref(count)))
        # the sums hold FP32 correlations: FP32 is what they are good for
        return {"sum": s.sum.float(), "sum_sq": s.sum_sq.float(), "picks": _pick_arrays(s.picks),
                "count": count.value}
    if case["kind"] == "grad":
        r = s.searcher.score_grad(s.picks, s.params)
        return {k: np.ascontiguousarray(r[k]) for k in r.dtype.names}
    if case["kind"] == "batch":
        n = len(s.images)
        ptrs = (ctypes.c_void_p * n)(*[i.ctypes.data for i in s.images])
        nxs = (ctypes.c_int * n)(*[i.shape[1] for i in s.images])
        nys = (ctypes.c_int * n)(*[i.shape[0] for i in s.images])
        offsets = (ctypes.c_size_t * (n + 1))()
        _ok(s.lib.gisspa_search_batch(s.searcher.h, n, ptrs, nxs, nys, (gisspa.Ctf * n)(*[s.ctf] * n),
                                      s.picks.ctypes.data, len(s.picks), offsets))
        return {"picks": _pick_arrays(s.picks), "offsets": list(offsets)}
    count = ctypes.c_size_t(0)
    image = s.images[0]
    _ok(s.lib.gisspa_search(s.searcher.h, image.ctypes.data, image.shape[1], image.shape[0], ctypes.byref(s.ctf),
                            s.picks.ctypes.data, PICKS, ctypes.byref(count)))
    return {"picks": _pick_arrays(s.picks), "count": count.value}


# ---------------------------------------------------------------- work
def work(case):
    b = {"fp32": 8, "fp16": 4, "bf16": 4}[case.get("spec", "fp32")]
    l = case["window"]
    fft2 = 2.5 * l * l * math.log2(l * l)  # one real 2D transform
    if case["kind"] == "maps":
        pairs = case["windows"] * case["templates"]
        h = (l // 2 + 1) * l
        return {"bytes": case["windows"] * h * 8 + case["templates"] * h * b + pairs * l * l * 4,
                "flops": pairs * (fft2 + 6 * h)}
    nt, t = case["templates"], case["tsize"]
    if case["kind"] == "grad":
        # per pick: the mask's area in the template, its three derivatives and the window; FP64 sums
        area = math.pi * (0.75 * _diameter(case) + 8) ** 2
        return {"bytes": case["picks"] * area * 4 * 5 + nt * t * t * 4, "flops": case["picks"] * area * 150}
    angles = math.ceil(360.0 / case["step"])
    sizes = [(case["nx"], case["ny"])]
    if case["kind"] == "batch":
        sizes += [(case["nx"] * 7 // 8 + 5, case["ny"]), (case["nx"] * 3 // 4, case["ny"] * 3 // 4 + 2)]
    flops = byts = 0.0
    for nx, ny in sizes:
        if case["kind"] == "tiled":
            per = 1 if 720 <= l else 1 + -(-(720 - l) // (l - case["overlap"]))
            w = math.ceil(nx / 720) * math.ceil(ny / 720) * per * per
        else:
            w = _windows_along(nx, case) * _windows_along(ny, case)
        flops += w * nt * angles * (fft2 + 3 * l * l)
        byts += nx * ny * 4 + nt * t * t * 4
        if case["kind"] == "shard":
            byts += w * l * l * 24
    return {"bytes": byts, "flops": flops}


# ---------------------------------------------------------------- 64-bit values
def _exact_maps(case, seed):
    win, tm = _map_inputs(case, seed)
    win = torch.view_as_complex(win.double())  # [n][kx][ky]
    tm = torch.view_as_complex(tm.double().contiguous())
    l = case["window"]
    out = torch.empty((case["windows"], case["templates"], l, l), device="cuda", dtype=torch.float64)
    for i in range(case["windows"]):
        for j in range(case["templates"]):
            z = (win[i] * tm[j].conj()).transpose(0, 1)  # [ky][kx]
            # as the two passes define it: along ky, then the real transform along kx, which takes
            # the real parts of columns 0 and l/2
            c = torch.fft.irfft(torch.fft.ifft(z, dim=0), n=l, dim=1)
            out[i, j] = torch.roll(c, (l // 2, l // 2), (0, 1))
    return out


def _grid(nx, ny):
    y = torch.arange(ny, device="cuda")[:, None]
    x = torch.arange(nx, device="cuda")[None, :]
    return x, y


def _shell(x, y, nx, ny):
    dy, dx = torch.minimum(y, ny - y), torch.minimum(x, nx - x)
    return torch.floor(torch.sqrt((dx * dx + dy * dy).double()) + 0.5).long() - 1


def _ctf_ast(x, y, nx, ny, ctf, apix=1.0):
    lam = 12.2639 / math.sqrt(300.0 * 1000.0 + 0.97845 * 300.0 * 300.0)
    amp = float(np.float32(0.07))
    cs = float(np.float32(2.7))
    y1 = torch.where(x > nx // 2, ny - y, y).double()
    x1 = torch.minimum(x, nx - x).double()
    dy = y1 - ny // 2
    ss = (x1 * x1 / (nx * nx) + dy * dy / (ny * ny)) / apix ** 2
    ag = torch.atan2(dy, x1)
    dfu, dfv = -ctf.defocus + ctf.dfdiff, -ctf.defocus - ctf.dfdiff
    df = 0.5 * (dfu + dfv + 2.0 * ctf.dfdiff * torch.cos(2.0 * (ctf.dfang * PI / 180.0 - ag)))
    gamma = -2.0 * PI * (cs * 2.5e6 * lam ** 3 * ss * ss + df * 5000.0 * lam * ss)
    return math.sqrt(1.0 - amp * amp) * torch.sin(gamma) + amp * torch.cos(gamma)


def _band(r, hi, lo):
    r = r.double()
    w = torch.zeros_like(r)
    w = torch.where((r >= lo - 8) & (r < lo) & (r >= 0), 0.5 * torch.cos(PI * (lo - r) / 16.0) + 0.5, w)
    w = torch.where((r >= hi) & (r < hi + 8), 0.5 * torch.cos(PI * (r - hi) / 16.0) + 0.5, w)
    return torch.where((r < hi) & (r >= 0), torch.ones_like(w), w)


def _f32(v):
    return float(np.float32(v))


def _noise_curves(ss):
    signal = torch.exp(_f32(-18.17) * ss * ss + _f32(-15.22) * ss + _f32(1.72))
    noise = torch.exp(_f32(-10.81) * ss * ss + 1.0 * ss + _f32(0.32))
    return signal, noise


def _radial(f, nx, ny, r, nb):
    """Mean power of each shell over the half plane x <= nx/2 (per image), on the full grid's shells."""
    half = (slice(None),) * (f.dim() - 1) + (slice(0, nx // 2 + 1),)
    rh = r[..., : nx // 2 + 1].reshape(-1)
    ok = (rh >= 0) & (rh < nb)
    p = f[half].abs().square().reshape(-1, rh.numel())
    s = torch.zeros((p.shape[0], nb), device="cuda", dtype=torch.float64).index_add_(1, rh[ok], p[:, ok])
    n = torch.zeros(nb, device="cuda", dtype=torch.float64).index_add_(0, rh[ok], torch.ones_like(rh[ok]).double())
    return s / n


def _rms(f, l, r):
    rh = r[:, : l // 2 + 1]
    ok = (rh >= 0) & (rh < l // 2)
    s = (f[:, :, : l // 2 + 1].abs().square() * ok).sum(dim=(1, 2))
    m = torch.sqrt(s) / ok.sum()
    return f / m[:, None, None]


def _exact_sums(case, seed):
    """S1 and S2 of every window pixel over templates and angles, in 64 bits."""
    stack, images, ctf = _search_inputs(case, seed)
    l, nx, ny, nt, t = case["window"], case["nx"], case["ny"], case["templates"], case["tsize"]
    dm, ehw, kk, hires, lores = 1.5 * _f32(_diameter(case)), 4.0, 3.0, 8.0, 200.0
    x, y = _grid(l, l)
    r = _shell(x, y, l, l)
    # templates: padding, edge mean, variance, whitening, weighting, RMS
    tb = torch.zeros((nt, l, l), device="cuda", dtype=torch.float64)
    o = (l - t) // 2
    tb[:, o:o + t, o:o + t] = torch.from_numpy(stack).cuda().double()
    rr = ((x - l // 2) ** 2 + (y - l // 2) ** 2).double()
    rf = l / 2 - 2
    ring = (rr >= (rf - 1) ** 2) & (rr <= (rf + 1) ** 2)
    em = (tb * ring).sum(dim=(1, 2)) / ring.sum()
    sd = tb.var(dim=(1, 2), unbiased=False).sqrt()
    f = torch.fft.fft2((tb - em[:, None, None]) / sd[:, None, None]) / (l * l)
    ok = (r >= 0) & (r < l // 2)
    rad = _radial(f, l, l, r, l // 2)
    f = torch.where(ok, f / rad[:, r.clamp(0, l // 2 - 1)].sqrt(), f)
    ss = torch.sqrt((torch.minimum(x, l - x) ** 2 + torch.minimum(y, l - y) ** 2).double()) / l
    v = _ctf_ast(x, (y + l // 2) % l, l, l, ctf).abs()
    signal, noise = _noise_curves(ss)
    noise = noise / (signal / (kk + 1))
    w = _band(r, l / hires, l / lores)
    w = torch.where(ok, w * v * torch.sqrt(1.0 / (noise + kk * v * v)), w)
    prep = torch.fft.ifft2(_rms(f * w, l, r)).real * (l * l)
    # micrograph: the reference's serial FP32 statistics, outliers, phase flip, whitening, weighting
    img = images[0].reshape(-1)
    f32 = np.float32
    terms = (img / f32(nx)) / f32(ny)
    avg = np.add.accumulate(terms, dtype=np.float32)[-1]
    sq = np.add.accumulate(((img * img) / f32(nx)) / f32(ny), dtype=np.float32)[-1]
    var = np.sqrt(sq - avg * avg)
    up, lo = f32(int(avg + f32(6) * var)), f32(int(avg - f32(6) * var))
    img = np.where((img > up) | (img < lo), avg, img) if sq > avg * avg else img
    g = torch.fft.fft2(torch.from_numpy(img.reshape(ny, nx)).cuda().double()) / (nx * ny)
    xi, yi = _grid(nx, ny)
    ri = _shell(xi, yi, nx, ny)
    c = _ctf_ast(xi, (yi + ny // 2) % ny, nx, ny, ctf)
    g = g * torch.where(c > 0, 1.0, -1.0)
    big, nb = max(nx, ny), max(nx, ny) // 2
    rad = _radial(g[None], nx, ny, ri, nb)[0]
    dx, dy = torch.minimum(xi, nx - xi).double(), torch.minimum(yi, ny - yi).double()
    ss = torch.sqrt(dx * dx / (nx * nx) + dy * dy / (ny * ny))
    ok = (ri >= 0) & (ri < big // 2)
    v = c.abs()
    signal, noise = _noise_curves(ss)
    fac = torch.sqrt((signal * v * v + noise) / signal) / rad[ri.clamp(0, nb - 1)].sqrt()
    fac = torch.where(ri > big / 6, fac * torch.exp(-100 * ss * ss), fac)
    fac = torch.where(ok, fac, torch.ones_like(fac)) * _band(ri, big / hires, big / lores)
    noise = noise / (signal / (kk + 1))
    fac = torch.where(ok, fac * torch.sqrt(1.0 / (noise + kk * v * v)), fac)
    fac[0, 0] = 0.0
    img = torch.fft.ifft2(g * fac).real * (nx * ny)
    del g, fac, v, signal, noise, ss, dx, dy, rad, c
    # windows
    def offsets(n):
        off, q = [0], 0
        while q + l < n:
            q += l - case["overlap"]
            if q + l >= n:
                q = n - l
            off.append(q)
        return off

    wins = torch.stack([img[b:b + l, a:a + l] for b in offsets(ny) for a in offsets(nx)])
    spec = _rms(torch.fft.fft2(wins) / (l * l), l, r)[:, :, : l // 2 + 1].contiguous()
    # sweep
    s1 = torch.zeros((len(wins), l, l), device="cuda", dtype=torch.float64)
    s2 = torch.zeros_like(s1)
    xc, yc = (x - l // 2).double(), (y - l // 2).double()
    rad = torch.sqrt(rr)
    mask = torch.where(rad >= dm / 2, 0.5 * torch.cos(PI * (rad - dm / 2) / (2.0 * ehw)) + 0.5, 1.0)
    mask = torch.where(rad > dm / 2 + 2 * ehw, 0.0, mask)
    theta = np.float32(0.0)
    while theta < 360.0:
        a = float(theta) * PI / 180.0
        ca, sa = _f32(math.cos(a)), _f32(math.sin(a))
        x2, y2 = ca * xc + sa * yc + l // 2, -sa * xc + ca * yc + l // 2
        inside = (x2 >= 0) & (x2 <= l - 1) & (y2 >= 0) & (y2 <= l - 1)
        ii, jj = torch.floor(x2).long().clamp(0, l - 1), torch.floor(y2).long().clamp(0, l - 1)
        i1, j1 = (ii + 1).clamp(max=l - 1), (jj + 1).clamp(max=l - 1)
        tt, uu = x2 - ii, y2 - jj
        rot = (prep[:, jj, ii] * ((1 - tt) * (1 - uu)) + prep[:, jj, i1] * (tt * (1 - uu)) +
               prep[:, j1, i1] * (tt * uu) + prep[:, j1, ii] * ((1 - tt) * uu))
        rot = rot * (inside * mask)
        rot = (rot - rot.mean(dim=(1, 2), keepdim=True)) / rot.var(dim=(1, 2), unbiased=False, keepdim=True).sqrt()
        ts = torch.fft.rfft2(rot) / (l * l)
        for n in range(nt):
            cc = torch.fft.irfft2(spec * ts[n].conj(), s=(l, l))
            s1 += cc
            s2 += cc * cc
        theta = np.float32(theta + np.float32(case["step"]))
    return {"sum": torch.roll(s1, (l // 2, l // 2), (1, 2)).reshape(-1),
            "sum_sq": torch.roll(s2, (l // 2, l // 2), (1, 2)).reshape(-1), "picks": None, "count": None}


def exact(case, seed):
    """Maps and per-pixel sums in 64 bits.  Whole searches give picks, choices among the
    correlations that the other cases check, and score gradients depend on a search's
    statistics: they have no value here."""
    if case["kind"] == "maps":
        return _exact_maps(case, seed)
    if case["kind"] == "shard":
        return _exact_sums(case, seed)
    return None
