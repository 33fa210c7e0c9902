"""What this library's speed is measured on: its public calls over the sizes,
methods and options that CTF estimation meets.

A case is a dict of plain values; `kind` names the call:

  spectrum    Context.setup + gen_half_spectrum: the averaged amplitude
              spectrum of one device image, background-removed and lowpassed,
              read back with its radial average
  noalloc     gcf_avg_spectrum_noalloc: the raw averaged spectrum into a
              device buffer, for callers that own every allocation
  micrograph  setup + gen_half_spectrum + set_phase + do2d: one micrograph in
              the CFindCtf2D call shape, with or without an extra-phase search
  series      Context.run_series: the package policy over a tilt series or a
              folder of equal frames
  batch       Context.run_batch: independent micrographs of uneven size in one
              call, by search method and rescale implementation
  train       Context.nn_train: Adam steps of the learned initialiser

Images are Poisson counts of a white object seen through a CTF, with a smooth
background (gctffind_b200.synth); defocus, astigmatism and dose are drawn from
the seed over the ranges of the uneven batch, sizes and pixel sizes belong to
the case.
"""
import math
import random

import numpy as np
import torch

import gctffind_b200 as G
from gctffind_b200 import synth

FIELDS = ("df_min", "df_max", "azimuth", "ext_phase", "score", "ctf_res", "df_1d", "phase_1d", "score_1d")
PLAIN, BF16, LEARNED = G.GCF_SEARCH_PLAIN, G.GCF_SEARCH_BF16, G.GCF_SEARCH_LEARNED
CUFFT, LINES, GEMM = G.GCF_RESCALE_CUFFT, G.GCF_RESCALE_LINES, G.GCF_RESCALE_GEMM


def listed():
    return [
        # the smallest call: a binned preview frame, where launches count
        {"name": "spectrum_1024", "kind": "spectrum", "w": 1024, "h": 1024, "px": 1.5, "tile": 512, "log": 0},
        # an ordinary ragged frame
        {"name": "spectrum_3838x3710", "kind": "spectrum", "w": 3838, "h": 3710, "px": 1.3, "tile": 512, "log": 0},
        # the largest frame: a super-resolution camera
        {"name": "spectrum_11520x8184", "kind": "spectrum", "w": 11520, "h": 8184, "px": 1.2, "tile": 512, "log": 0},
        # the command line's -TileSize and -LogSpect
        {"name": "spectrum_tile1024_log", "kind": "spectrum", "w": 4096, "h": 4096, "px": 1.35, "tile": 1024,
         "log": 1},
        # an acquisition loop that must not allocate
        {"name": "noalloc_5760x4092", "kind": "noalloc", "w": 5760, "h": 4092},
        # one small micrograph from image to result: latency
        {"name": "micrograph_2048", "kind": "micrograph", "w": 2048, "h": 2048, "px": 1.35, "phase": 0.0,
         "range": 0.0},
        # one phase-plate micrograph
        {"name": "micrograph_4096_phase", "kind": "micrograph", "w": 4096, "h": 4096, "px": 1.35, "phase": 60.0,
         "range": 90.0},
        # a tilt series, -60 to +60 degrees in 3 degree steps
        {"name": "series_41x4096", "kind": "series", "n": 41, "w": 4096, "h": 4096, "px": 1.35, "tomo": 1, "full": 0},
        # a folder of equal frames that are rescaled, with the diagnostic spectra the command line writes
        {"name": "series_folder_6", "kind": "series", "n": 6, "w": 5760, "h": 4092, "px": 0.83, "tomo": 0, "full": 1},
        # uneven micrographs by the reference's method and rescale
        {"name": "batch_plain_12", "kind": "batch", "n": 12, "px_lo": 0.8, "px_hi": 1.5, "mode": PLAIN,
         "rescale": CUFFT, "host": 0},
        # uneven micrographs by the fast method: learned window, tensor-core contraction and rescale
        {"name": "batch_learned_64", "kind": "batch", "n": 64, "px_lo": 0.8, "px_hi": 1.5, "mode": LEARNED,
         "rescale": GEMM, "host": 0},
        # training of the learned initialiser
        {"name": "train_4x256", "kind": "train", "steps": 4, "batch": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["spectrum", "spectrum", "noalloc", "micrograph", "micrograph", "series", "batch", "batch",
                       "batch", "train"])
    if kind == "spectrum":
        tile = rng.choice([512, 512, 512, 512, 256, 1024])
        return {"kind": kind, "w": _log_int(rng, max(600, tile), 11520), "h": _log_int(rng, max(600, tile), 8184),
                "px": round(rng.uniform(1.2, 1.6), 3), "tile": tile, "log": int(rng.random() < 0.2)}
    if kind == "noalloc":
        return {"kind": kind, "w": _log_int(rng, 512, 11520), "h": _log_int(rng, 512, 8184)}
    if kind == "micrograph":
        phase = rng.random() < 0.4
        return {"kind": kind, "w": _log_int(rng, 1024, 5760), "h": _log_int(rng, 1024, 5760),
                "px": round(rng.uniform(1.2, 1.6), 3), "phase": round(rng.uniform(0.0, 80.0), 1) if phase else 0.0,
                "range": round(rng.uniform(20.0, 120.0), 1) if phase else 0.0}
    if kind == "series":
        return {"kind": kind, "n": rng.randint(3, 24), "w": _log_int(rng, 1500, 4096), "h": _log_int(rng, 1500, 4096),
                "px": round(rng.uniform(0.9, 1.6), 3), "tomo": int(rng.random() < 0.6),
                "full": int(rng.random() < 0.5)}
    if kind == "batch":
        lo = round(rng.uniform(0.8, 1.3), 3)
        return {"kind": kind, "n": _log_int(rng, 1, 40), "px_lo": lo, "px_hi": round(lo + rng.uniform(0.0, 0.3), 3),
                "mode": rng.choice([PLAIN, BF16, LEARNED, LEARNED]), "rescale": rng.choice([CUFFT, LINES, GEMM, GEMM]),
                "host": int(rng.random() < 0.2)}
    return {"kind": kind, "steps": rng.randint(2, 5), "batch": rng.choice([64, 100, 192, 256])}


def _spec(g, w, h, px, seed, tilt=0.0, phase=0.0, df=None, ast=None, az=None):
    u = lambda lo, hi: g.uniform(lo, hi)  # noqa: E731
    mean = u(6000.0, 38000.0) if df is None else df
    ast = u(0.0, 1000.0) if ast is None else ast
    az = u(-90.0, 90.0) if az is None else az
    return synth.MicrographSpec(width=w, height=h, pixel_size=px, df_min=mean - 0.5 * ast, df_max=mean + 0.5 * ast,
                                azimuth_deg=az, dose=u(0.5, 3.0), ext_phase_deg=phase, tilt_deg=tilt, seed=seed)


def _image(spec):
    return synth.make_micrograph(spec, device="cuda")


def _batch_frames(case):
    """Size and pixel size of each micrograph: the three frame sizes in turn,
    pixel sizes spread evenly over the range in a shuffled order."""
    out = []
    for k in range(case["n"]):
        w, h = synth.UNEVEN_SIZES[k % len(synth.UNEVEN_SIZES)]
        f = (0.5 + 0.6180339887498949 * k) % 1.0
        out.append((w, h, case["px_lo"] + f * (case["px_hi"] - case["px_lo"])))
    return out


def prepare(case, seed):
    g = random.Random(seed)
    base = (seed * 7919) % (1 << 30)
    kind = case["kind"]
    s = {"case": case}
    if kind in ("spectrum", "noalloc", "micrograph"):
        s["img"] = _image(_spec(g, case["w"], case["h"], case.get("px", 1.35), base,
                                phase=case.get("phase", 0.0) + (0.2 * case["range"] if case.get("range") else 0.0)))
    if kind == "noalloc":
        s["out"] = torch.empty((512, 257), dtype=torch.float32, device="cuda")
        s["lib"] = G.load_library()
        torch.cuda.synchronize()
        return s
    s["ctx"] = G.Context(0, case.get("tile", 512), case.get("log", 0))
    s["optics"] = G.make_optics(pixel_size=case.get("px", 1.0))
    if kind == "series":
        n, tomo = case["n"], case["tomo"]
        tilts = [(i - (n - 1) // 2) * 3.0 for i in range(n)] if tomo else [0.0] * n
        df, ast, az = g.uniform(12000.0, 32000.0), g.uniform(0.0, 800.0), g.uniform(-90.0, 90.0)
        s["imgs"] = [_image(_spec(g, case["w"], case["h"], case["px"], base + i, tilt=t, df=df, ast=ast, az=az))
                     for i, t in enumerate(tilts)]
        s["order"] = G.series_order(tilts).order if tomo else list(range(n))
    elif kind == "batch":
        frames = _batch_frames(case)
        s["imgs"] = [_image(_spec(g, w, h, px, base + i)) for i, (w, h, px) in enumerate(frames)]
        if case["host"]:
            s["imgs"] = [a.cpu().pin_memory() for a in s["imgs"]]
        s["pxs"] = [px for _, _, px in frames]
        s["ctx"].set_rescale_impl(case["rescale"])
        if case["mode"] == LEARNED:
            G.load_learned(s["ctx"])
    elif kind == "train":
        s["ctx"].nn_init(seed)
        s["params"] = s["ctx"].nn_params()
        s["seed"] = base
    torch.cuda.synchronize()
    return s


def _table(results):
    out = {f: np.array([getattr(r, f) for r in results], np.float32) for f in FIELDS}
    out["lowpassed"] = np.array([r.lowpassed for r in results], np.int64)
    return out


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "noalloc":
        img, out = s["img"], s["out"]
        st = s["lib"].gcf_avg_spectrum_noalloc(img.data_ptr(), case["w"], case["h"], case["w"], out.data_ptr(),
                                               torch.cuda.current_stream().cuda_stream)
        if st != 0:
            raise RuntimeError("gcf_avg_spectrum_noalloc: status %d" % st)
        return out
    ctx = s["ctx"]
    if kind == "spectrum":
        ctx.setup(s["optics"], case["w"], case["h"])
        ctx.gen_half_spectrum(s["img"])
        return {"ctf": ctx.half_spectrum(False), "radial": ctx.radial_average()}
    if kind == "micrograph":
        ctx.setup(s["optics"], case["w"], case["h"])
        ctx.gen_half_spectrum(s["img"])
        ctx.set_phase(case["phase"], case["range"])
        return _table([ctx.do2d()])
    if kind == "series":
        r = ctx.run_series(s["imgs"], s["optics"], s["order"], is_tomo=bool(case["tomo"]),
                           want_full=bool(case["full"]))
        if case["full"]:
            return {"results": _table(r[0]), "full": r[1]}
        return _table(r)
    if kind == "batch":
        return _table(ctx.run_batch(s["imgs"], s["pxs"], s["optics"], mode=case["mode"]))
    ctx.nn_set_params(s["params"])
    losses = ctx.nn_train(s["optics"], case["steps"], case["batch"], s["seed"])
    return {"losses": losses, "params": ctx.nn_params()}


# Multiply-adds of one training sample: the four convolutions and the MLP.
_NET_MACS = 4096 * 16 * 16 + 1024 * 32 * 144 + 256 * 32 * 288 + 64 * 32 * 288 + 256 * 2304 + 128 * 256 + 3 * 128
_NET_PARAMS = 16 * 17 + 32 * 145 + 2 * 32 * 289 + 256 * 2305 + 128 * 257 + 3 * 129


def _fft2_flops(w, h):
    return 2.5 * w * h * math.log2(w * h)


def _tiles(w, h, tile):
    return ((w - tile // 2) // (tile // 2)) * ((h - tile // 2) // (tile // 2))


def _frame_work(w, h, px, tile, rescaled):
    """Bytes and flops of one frame: read once; the Fourier-crop rescale where
    it applies, the tiles' real 2D transforms."""
    nw, nh = w, h
    flops = 0.0
    if rescaled and px < 1.2:
        nw, nh, _ = G.rescale_dims(w, h, px)
        flops += _fft2_flops(w, h) + _fft2_flops(nw, nh)
    return 4.0 * w * h, flops + _tiles(nw, nh, tile) * (_fft2_flops(tile, tile) + 6.0 * tile * tile)


# Band pixels of a 512 tile near 1.2-1.5 A/px, and the 2D candidates of a full
# search (grid and line steps) and of a refinement; 2 flops a pair.
_BAND, _FULL, _REFINE = 6.0e4, 4550, 570


def work(case):
    kind = case["kind"]
    half = 4.0 * 257 * 512
    if kind in ("spectrum", "noalloc", "micrograph"):
        tile = case.get("tile", 512)
        b, f = _frame_work(case["w"], case["h"], 2.0, tile, False)
        if kind == "spectrum":
            b += 4.0 * tile * (tile // 2 + 1)
        elif kind == "noalloc":
            b += half
        else:
            b += 40.0
            f += 2.0 * _BAND * _FULL
        return {"bytes": b, "flops": f}
    if kind == "series":
        b, f = _frame_work(case["w"], case["h"], case["px"], 512, True)
        n = case["n"]
        search = 2.0 * _BAND * (_FULL + (n - 1) * (_REFINE if case["tomo"] else _REFINE + 2601))
        return {"bytes": n * (b + 40.0 + (4.0 * 512 * 512 if case["full"] else 0.0)), "flops": n * f + search}
    if kind == "batch":
        b = f = 0.0
        for w, h, px in _batch_frames(case):
            x, y = _frame_work(w, h, px, 512, True)
            b += x + 40.0
            f += y + 2.0 * _BAND * (_FULL if case["mode"] == PLAIN else 112)
        return {"bytes": b, "flops": f}
    n = case["steps"] * case["batch"]
    return {"bytes": 8.0 * _NET_PARAMS, "flops": 6.0 * n * _NET_MACS}


# ---------------------------------------------------------------------------
# The same spectra in 64 bits with torch: tile layout, taper, transforms,
# background and lowpass as the reference defines them.
def _raw64(img, tile):
    h, w = img.shape
    ov = tile // 2 // 2 * 2
    st = tile - ov
    ntx, nty = (w - ov) // st, (h - ov) // st
    ox, oy = (w - ntx * tile + (ntx - 1) * ov) // 2, (h - nty * tile + (nty - 1) * ov) // 2
    c = (torch.arange(tile, dtype=torch.float64, device=img.device) - 0.5 * tile).abs() * 2.0 / tile
    r = torch.sqrt(c[:, None] ** 2 + c[None, :] ** 2)
    q = 0.5 * (1.0 - torch.cos(math.pi * r))
    taper = torch.where(r < 1.0, 1.0 - q ** 3, torch.zeros_like(r))
    acc = torch.zeros((tile, tile // 2 + 1), dtype=torch.float64, device=img.device)
    for ty in range(nty):
        y = oy + ty * st
        rows = img[y:y + tile].double()
        t = torch.stack([rows[:, ox + tx * st:ox + tx * st + tile] for tx in range(ntx)])
        t = (t - t.mean(dim=(1, 2), keepdim=True)) * taper
        acc += torch.fft.rfft2(t).abs().sum(dim=0)
    return torch.roll(acc / (ntx * nty), tile // 2, dims=0)


def _ctf64(raw, log):
    tile = raw.shape[0]
    cx, half = tile // 2 + 1, tile // 2
    dev = raw.device
    box = min(int(np.float32(1.0) / np.float32(15.0) * np.float32(tile)), int(np.float32(0.3) * np.float32(tile)))
    box = max(box // 2 * 2 + 1, 7)
    hb = box // 2
    v = raw if log else torch.sqrt(raw)
    xx = torch.arange(-hb, cx + hb, device=dev)
    yy = torch.arange(-half - hb, half + hb, device=dev)
    xx = torch.where(xx >= half, xx - 2 * half, xx)
    ix = xx.abs()[None, :].expand(len(yy), len(xx))
    iy = torch.where(xx[None, :] >= 0, half + yy[:, None], half - yy[:, None])
    ext = v[iy % tile, ix]
    bg = torch.nn.functional.avg_pool2d(ext[None, None], box, stride=1)[0, 0]
    if not log:
        bg = bg * bg
    fx = np.arange(cx, dtype=np.float32) * np.float32(0.5) / np.float32(cx - 1)
    yr = np.arange(tile, dtype=np.int64) - half
    fy2 = (yr * yr).astype(np.float32) / np.float32(tile * tile)
    fr = np.sqrt((fx * fx)[None, :] + fy2[:, None]).astype(np.float32)
    keep = torch.from_numpy(fr.astype(np.float64) >= 0.04).to(dev)
    ctf = torch.where(keep, raw - bg, torch.zeros_like(raw))
    if float((ctf * ctf).mean() - ctf.mean() ** 2) < 1.0:
        return ctf
    y = torch.arange(tile, device=dev)
    mirror = ctf[(tile - y) % tile][:, 1:].flip(1)
    full = torch.cat([mirror, ctf[:, :half]], dim=1)
    k = torch.fft.fftfreq(tile, d=1.0 / tile, device=dev, dtype=torch.float64)
    gk = torch.exp(-10.0 / (2.0 * tile * tile) * k * k)
    full = torch.fft.ifft2(torch.fft.fft2(full) * gk[:, None] * gk[None, :]).real
    return torch.cat([full[:, half:], full[:, :1]], dim=1)


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("spectrum", "noalloc"):
        return None   # discrete searches over grids, stochastic training
    g = random.Random(seed)
    img = _image(_spec(g, case["w"], case["h"], case.get("px", 1.35), (seed * 7919) % (1 << 30)))
    raw = _raw64(img, case.get("tile", 512))
    if kind == "noalloc":
        return raw
    return {"ctf": _ctf64(raw, case["log"]), "radial": None}
