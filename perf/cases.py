"""Performance cases: the work that users of this package have it do, through its public entry points.

Frame pairs are synthetic, in the manner of the package's own workloads: a smooth gradient with Gaussian
texture as the reference picture; the other picture is it with every 16x16 block shifted, a global
colour offset and noise added. Frames are on the GPU as decoders leave them there, except in the case
that stands for frames read from files into pinned host memory.

A case is a dict:
    call        "pair"    one frame pair through Calc.compute
                "batch"   many frame pairs through Batch.compute
                "masked"  one frame pair and its mask through Calc.compute_masked
                "masked_batch"  many through Batch.compute_masked
    width, height, bitdepth, chroma, search_range, erp, metrics, pairs
    mixed       batch: the pairs' shapes, depths and search ranges are drawn from the mixed set
    host        frames in pinned host memory
    ssim_mode, ssim_stride   structural similarity options (default: averaged 8x8 blocks at stride 4)
"""
import math
import random

import numpy as np
import torch

import qmiv_b200 as qm

MIXED_SHAPES = [(1280, 720), (1920, 1080), (2048, 2048), (4096, 2048)]

DEFAULTS = dict(call="pair", width=1920, height=1080, bitdepth=10, chroma=420, search_range=2, erp=False,
                metrics="IVPSNR", pairs=1, mixed=False, host=False, ssim_mode=qm.SSM_BLOCK_AVERAGED, ssim_stride=4)


def _case(name=None, **kw):
    case = dict(DEFAULTS, **kw)
    if name is not None:
        case["name"] = name
    return case


def listed():
    return [
        # a preview-sized proxy scored frame by frame while an encoder is tuned: launches and latency
        _case("preview_320x180_10b", width=320, height=180, metrics="PSNR,IVPSNR"),
        # the plain CPU-sized job of the command line: one full-HD 8-bit pair, IV-PSNR
        _case("hd_1920x1080_8b", bitdepth=8),
        # a DCI flat 12-bit master with every metric switched on (ragged width and height)
        _case("cinema_1998x1080_12b_all", width=1998, height=1080, bitdepth=12,
              metrics="PSNR,WSPSNR,IVPSNR,SSIM,MSSSIM,IVSSIM,IVMSSSIM"),
        # screen content or rendered RGB kept at 4:4:4
        _case("screen_1920x1080_8b_444", bitdepth=8, chroma=444, metrics="PSNR,IVPSNR,SSIM"),
        # one 360-degree frame at a time, as frames come out of a decoder
        _case("erp_4096x2048_10b", width=4096, height=2048, erp=True, metrics="WSPSNR,IVPSNR,IVSSIM"),
        # the headline job: a 360-degree sequence in batches of eight frames
        _case("erp_batch8_4096x2048_10b", call="batch", width=4096, height=2048, erp=True, pairs=8,
              metrics="WSPSNR,IVPSNR,IVSSIM"),
        # a scoring service: sixteen pairs of uneven size, depth and search range in one call
        _case("service_mixed16", call="batch", pairs=16, mixed=True, metrics="PSNR,IVPSNR,IVSSIM"),
        # multi-scale metrics over a batch of square projections
        _case("msssim_batch8_2048x2048_10b", call="batch", width=2048, height=2048, pairs=8, metrics="MSSSIM,IVMSSSIM"),
        # frames read from files into pinned host memory, uploaded by the call itself
        _case("host_batch4_3840x2160_10b", call="batch", width=3840, height=2160, pairs=4, host=True, metrics="PSNR,IVPSNR"),
        # mask mode: only the visible part of a rendered view is scored
        _case("masked_4096x2048_10b", call="masked", width=4096, height=2048, erp=True, metrics="PSNR,WSPSNR,IVPSNR"),
        _case("masked_batch8_1920x1080_8b", call="masked_batch", bitdepth=8, pairs=8, metrics="PSNR,IVPSNR"),
        # the original paper's SSIM: an 11x11 Gaussian window at every sample
        _case("gaussian_1920x1080_8b", bitdepth=8, metrics="SSIM,IVSSIM", ssim_mode=qm.SSM_REGULAR_GAUSSIAN_FLT, ssim_stride=1),
    ]


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    def size(lo, hi, step):
        return max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step)

    kind = rng.choice(["pair", "pair", "pair", "batch", "batch", "mixed", "ms", "host", "masked", "masked_batch", "gaussian"])
    bitdepth = rng.choice([8, 8, 10, 10, 10, 12])
    search_range = rng.choice([1, 2, 2, 2, 2, 3, 4])
    erp = rng.random() < 0.5
    w, h = size(192, 4096, 2), size(128, 2048, 2)
    if w * h >= 1 << 21:
        search_range = min(search_range, 2)
    if kind == "pair":
        chroma = rng.choice([420, 420, 420, 422, 444])
        metrics = rng.choice(["IVPSNR", "PSNR,IVPSNR", "WSPSNR,IVPSNR,IVSSIM", "PSNR,SSIM", "PSNR,WSPSNR,IVPSNR,SSIM,MSSSIM,IVSSIM,IVMSSSIM"])
        return _case(width=w, height=h, bitdepth=bitdepth, chroma=chroma, search_range=search_range, erp=erp, metrics=metrics)
    if kind == "batch":
        return _case(call="batch", width=w, height=h, bitdepth=bitdepth, search_range=search_range,
                     erp=erp, pairs=rng.randint(2, 8), metrics=rng.choice(["IVPSNR", "PSNR,IVPSNR", "WSPSNR,IVPSNR,IVSSIM"]))
    if kind == "mixed":
        return _case(call="batch", pairs=rng.randint(4, 12), mixed=True, metrics=rng.choice(["PSNR,IVPSNR", "PSNR,IVPSNR,IVSSIM"]))
    if kind == "ms":
        n = size(256, 2048, 2)
        return _case(call="batch", width=n, height=n, bitdepth=rng.choice([8, 10]), pairs=rng.randint(2, 8),
                     metrics=rng.choice(["MSSSIM", "MSSSIM,IVMSSSIM"]))
    if kind == "host":
        return _case(call="batch", width=size(640, 3840, 2), height=size(360, 2160, 2), bitdepth=rng.choice([8, 10]),
                     pairs=rng.randint(1, 4), host=True, metrics="PSNR,IVPSNR")
    if kind in ("masked", "masked_batch"):
        many = kind == "masked_batch"
        return _case(call=kind, width=w, height=h, bitdepth=rng.choice([8, 10, 10]), search_range=min(search_range, 3),
                     erp=erp, pairs=rng.randint(2, 6) if many else 1, metrics=rng.choice(["PSNR,IVPSNR", "PSNR,WSPSNR,IVPSNR"]))
    return _case(width=size(192, 1920, 2), height=size(128, 1080, 2), bitdepth=rng.choice([8, 10]), metrics=rng.choice(["SSIM", "SSIM,IVSSIM"]),
                 ssim_mode=qm.SSM_REGULAR_GAUSSIAN_FLT, ssim_stride=rng.choice([1, 1, 2]))


# ---- inputs ----------------------------------------------------------------------------------------
def _specs(case, seed):
    """Width, height, bit depth and search range of every pair."""
    if not case["mixed"]:
        return [(case["width"], case["height"], case["bitdepth"], case["search_range"])] * case["pairs"]
    # the shapes belong to the case, the samples to the seed: the same call signature for every seed
    rng = random.Random(1000 + case["pairs"])
    return [(*rng.choice(MIXED_SHAPES), rng.choice([8, 10]), rng.choice([2, 2, 4])) for _ in range(case["pairs"])]


def _make_pair(gen, w, h, bitdepth, chroma):
    """(reference, distorted) frames: two tuples of three planes on the GPU."""
    dev, maxv = "cuda", (1 << bitdepth) - 1
    scale = maxv / 255.0
    sx, sy = (0 if chroma == 444 else 1), (1 if chroma == 420 else 0)
    nby, nbx = -(-h // 16), -(-w // 16)
    shift_y = torch.randint(-2, 3, (nby, nbx), generator=gen, device=dev)
    shift_x = torch.randint(-2, 3, (nby, nbx), generator=gen, device=dev)
    par = torch.rand(15, generator=gen, device=dev, dtype=torch.float64).tolist()
    dtype = torch.uint8 if bitdepth <= 8 else torch.uint16
    ref, dist = [], []
    for c in range(3):
        ph, pw = (h >> sy, w >> sx) if c else (h, w)
        ax, ay, fx, fy, ang = par[5 * c:5 * c + 5]
        yy = torch.linspace(0, 1, ph, device=dev)[:, None]
        xx = torch.linspace(0, 1, pw, device=dev)[None, :]
        base = 0.16 + (0.12 + 0.16 * ax) * xx + (0.12 + 0.16 * ay) * yy
        base = base + 0.06 * torch.sin(2 * math.pi * ((0.5 + 2.5 * fx) * xx + (0.5 + 2.5 * fy) * yy + ang))
        r = base * maxv + torch.randn(ph, pw, generator=gen, device=dev) * (12.0 * scale)
        r = r.round().clamp_(0, maxv)
        iy, ix = torch.arange(ph, device=dev), torch.arange(pw, device=dev)
        by, bx = (iy << (sy if c else 0)) >> 4, (ix << (sx if c else 0)) >> 4
        dy = shift_y[by][:, bx] >> (sy if c else 0)
        dx = shift_x[by][:, bx] >> (sx if c else 0)
        src = ((iy[:, None] + dy).clamp_(0, ph - 1)) * pw + (ix[None, :] + dx).clamp_(0, pw - 1)
        d = r.reshape(-1)[src] + (3.0, -2.0, 2.0)[c] * scale + torch.randn(ph, pw, generator=gen, device=dev) * (2.0 * scale)
        ref.append(r.to(torch.int32).to(dtype))
        dist.append(d.round_().clamp_(0, maxv).to(torch.int32).to(dtype))
    return tuple(ref), tuple(dist)


def _make_mask(gen, w, h):
    """8-bit mask: 16x16 blocks kept with probability 0.6, the rest zero."""
    keep = torch.rand(-(-h // 16), -(-w // 16), generator=gen, device="cuda") < 0.6
    keep[0, 0] = True
    m = keep.repeat_interleave(16, 0).repeat_interleave(16, 1)[:h, :w]
    return (m.to(torch.uint8) * 255).contiguous()


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    frames, masks = [], []
    for w, h, bitdepth, _ in _specs(case, seed):
        frames.append(_make_pair(gen, w, h, bitdepth, case["chroma"]))
        if case["call"].startswith("masked"):
            masks.append(_make_mask(gen, w, h))
    return frames, masks


WHOLE = ["gcd_r2t", "exact", "invalid_pel", "ssd", "cps_sse_r2t", "cps_sse_t2r"]
DECIBELS = [("psnr", "wspsnr"), ("psnr_pic", "wspsnr_pic", "ivpsnr", "ivpsnr_r2t", "ivpsnr_t2r")]
SIMILARITIES = [("ssim", "msssim"), ("ssim_pic", "msssim_pic", "ivssim", "ivssim_r2t", "ivssim_t2r", "ivmsssim", "ivmsssim_r2t", "ivmsssim_t2r")]


def _table(results, fields):
    lists, numbers = fields
    return np.array([[v for k in lists for v in r[k]] + [r[k] for k in numbers] for r in results], dtype=np.float64)


def _tables(results, non_masked=None, whole=True):
    out = {"whole": np.array([[v for k in WHOLE for v in r[k]] for r in results], dtype=np.int64) if whole else None,
           "decibels": _table(results, DECIBELS), "similarities": _table(results, SIMILARITIES)}
    if non_masked is not None:
        out["non_masked"] = np.array(non_masked, dtype=np.int64) if whole else None
    return out


class _State:
    """What a user's program keeps between calls; the handle is closed with it."""

    def __init__(self, case, seed):
        self.frames, self.masks = _inputs(case, seed)
        self.pinned = []
        if case["host"]:
            self.frames = [tuple(self._pin(f) for f in pair) for pair in self.frames]
        specs = _specs(case, seed)
        self.call, self.metrics = case["call"], qm.metric_mask(case["metrics"])
        options = dict(erp=case["erp"], ssim_mode=case["ssim_mode"], ssim_stride=case["ssim_stride"])
        self.ctx = qm.Context(0)
        if self.call in ("pair", "masked"):
            w, h, bitdepth, search_range = specs[0]
            self.handle = qm.Calc(self.ctx, w, h, bitdepth, case["chroma"], search_range=search_range, **options)
        else:
            self.handle = qm.Batch(self.ctx, len(specs), sum(s[0] * s[1] for s in specs), graph=not case["host"],
                                   autotune=not case["host"], **options)
            self.pairs = [dict(frame0=f[0], frame1=f[1], width=s[0], height=s[1], bitdepth=s[2], chroma_format=case["chroma"],
                               search_range=s[3], metrics=self.metrics) for f, s in zip(self.frames, specs)]
        torch.cuda.synchronize()

    def _pin(self, frame):
        host = [p.cpu().pin_memory() for p in frame]
        self.pinned += host
        return tuple(p.numpy() for p in host)

    def __del__(self):
        for h in (getattr(self, "handle", None), getattr(self, "ctx", None)):
            if h is not None:
                h.close()


def prepare(case, seed):
    return _State(case, seed)


def run(state):
    """Every field of the results: whole numbers, decibels and similarities, a row per pair."""
    extra = None
    if state.call == "pair":
        results = [state.handle.compute(*state.frames[0], state.metrics)]
    elif state.call == "masked":
        result, n = state.handle.compute_masked(*state.frames[0], state.masks[0], 8, state.metrics)
        results, extra = [result], [n]
    elif state.call == "masked_batch":
        results, extra = state.handle.compute_masked(state.pairs, state.masks, [8] * len(state.masks))
    else:
        results = state.handle.compute(state.pairs)
    return _tables(results, extra)


# ---- what a pass cannot do without ---------------------------------------------------------------------
def work(case):
    """bytes: every sample of both frames (and the mask) read once. flops: the search's arithmetic, 8 integer
    operations per candidate and direction (three differences, three multiply-adds, an addition, a minimum),
    and 40 operations per similarity window and component, 10 per tap of the Gaussian one."""
    names = set(case["metrics"].split(","))
    cf = {420: 1.5, 422: 2.0, 444: 3.0}[case["chroma"]]
    nbytes = flops = 0.0
    for w, h, bitdepth, r in _specs(case, 0):
        px = w * h
        nbytes += 2 * cf * px * (1 if bitdepth <= 8 else 2)
        if case["call"].startswith("masked"):
            nbytes += px
        if names & {"IVPSNR", "IVSSIM", "IVMSSSIM"}:
            flops += 2 * px * (2 * r + 1) ** 2 * 8
        evaluations = ("SSIM" in names) + 2 * ("IVSSIM" in names) + (4 / 3) * ("MSSSIM" in names) + (8 / 3) * ("IVMSSSIM" in names)
        if case["ssim_mode"] == qm.SSM_BLOCK_AVERAGED:
            flops += evaluations * 3 * (10 * px + 40 * px / 16)
        else:
            flops += evaluations * 3 * (121 * 10 + 40) * px / case["ssim_stride"] ** 2
        flops += 6 * px
    return {"bytes": nbytes, "flops": flops}


# ---- the same values in 64 bits, plain torch -------------------------------------------------------------
CWA = (4, 1, 1, 0)
MS_EXPONENTS = [[1.0], [0.1356, 0.8644], [0.0711, 0.4530, 0.4760], [0.0517, 0.3295, 0.3462, 0.2726],
                [0.0448, 0.2856, 0.3001, 0.2363, 0.1333]]
def _p444(frame, chroma):
    planes = [p.to(torch.int32).to(torch.int64) for p in frame]
    for c in (1, 2):
        if chroma != 444:
            planes[c] = planes[c].repeat_interleave(2, 1)
        if chroma == 420:
            planes[c] = planes[c].repeat_interleave(2, 0)
    return torch.stack(planes)


def _edge_pad(p, r):
    h, w = p.shape[-2:]
    iy = torch.arange(-r, h + r, device=p.device).clamp_(0, h - 1)
    ix = torch.arange(-r, w + r, device=p.device).clamp_(0, w - 1)
    return p[..., iy, :][..., ix]


def _search(test, ref, r, mask=None):
    """The matched sample of `ref` per sample of `test`: first smallest 4:1:1 weighted squared error in raster order."""
    h, w = test.shape[-2:]
    padded = _edge_pad(ref, r)
    pmask = None if mask is None else _edge_pad(mask, r)
    best = torch.full((h, w), 2 ** 31 - 1, dtype=torch.int64, device=test.device)
    pel = torch.zeros_like(test)
    for dy in range(2 * r + 1):
        for dx in range(2 * r + 1):
            cand = padded[:, dy:dy + h, dx:dx + w]
            d = test - cand
            d = d * d
            err = 4 * d[0] + d[1] + d[2]
            better = err < best
            if pmask is not None:
                better &= pmask[dy:dy + h, dx:dx + w] != 0
            best = torch.where(better, err, best)
            pel = torch.where(better, cand, pel)
    return pel


def _db(peak, err):
    return 10.0 * math.log10(peak / err) if err > 0 else 1.7976931348623157e308


def _ws(h):
    y = torch.arange(h, dtype=torch.float64, device="cuda")
    return torch.cos((y - (h / 2 - 0.5)) * math.pi / h)


def _mean4(v):
    return sum(a * b for a, b in zip(v, CWA)) / sum(CWA)


def _gaussian():
    k = np.arange(-5, 6)
    g = np.exp(-(k[:, None] ** 2 + k[None, :] ** 2) / (2 * 1.5 ** 2))
    return (g / g.sum()).astype(np.float32).astype(np.float64)


def _window_means(v, case):
    if case["ssim_mode"] == qm.SSM_BLOCK_AVERAGED:
        return torch.nn.functional.avg_pool2d(v[None, None], 8, 4)[0, 0]
    s, (h, w) = case["ssim_stride"], v.shape
    ny, nx = -(-(h - 10) // s), -(-(w - 10) // s)
    out = torch.zeros(ny, nx, dtype=torch.float64, device=v.device)
    for dy, row in enumerate(_gaussian()):
        for dx, k in enumerate(row):
            out += float(k) * v[dy:dy + (ny - 1) * s + 1:s, dx:dx + (nx - 1) * s + 1:s]
    return out


def _ssim(a, b, maxv, case, luminance=True, weights=None):
    """Mean window similarity of each component of two 4:4:4 pictures."""
    c1, c2 = (0.01 * maxv) ** 2, (0.03 * maxv) ** 2
    out = []
    for p, q in zip(a.to(torch.float64), b.to(torch.float64)):
        mp, mq, pp, qq, pq = (_window_means(v, case) for v in (p, q, p * p, q * q, p * q))
        win = (2 * (pq - mp * mq) + c2) / ((pp - mp * mp) + (qq - mq * mq) + c2)
        if luminance:
            win = win * (2 * mp * mq + c1) / (mp * mp + mq * mq + c1)
        rows = win.sum(1)
        if weights is not None:
            ny = win.shape[0]
            at = (5 + case["ssim_stride"] * torch.arange(ny, device=rows.device)) if case["ssim_mode"] != qm.SSM_BLOCK_AVERAGED \
                else 4 + 4 * torch.arange(ny, device=rows.device)
            wr = weights[at]
            out.append(((rows * wr).sum() / (win.numel() * (wr.sum() / ny))).item())
        else:
            out.append((rows.sum() / win.numel()).item())
    return out


def _msssim(a, b, maxv, case):
    h, w = a.shape[-2:]
    scales = sum(1 for i in range(5) if min(w, h) >= 32 << i)
    score = [1.0] * 3
    for s in range(scales):
        v = _ssim(a, b, maxv, case, luminance=s == scales - 1)
        score = [x * max(y, 0.0) ** MS_EXPONENTS[scales - 1][s] for x, y in zip(score, v)]
        a, b = ((p[:, 0:p.shape[1] // 2 * 2:2, 0:p.shape[2] // 2 * 2:2] + p[:, 0:p.shape[1] // 2 * 2:2, 1:p.shape[2] // 2 * 2:2]
                 + p[:, 1:p.shape[1] // 2 * 2:2, 0:p.shape[2] // 2 * 2:2] + p[:, 1:p.shape[1] // 2 * 2:2, 1:p.shape[2] // 2 * 2:2] + 2) >> 2
                for p in (a, b))
    return score


def _exact_pair(case, spec, frames, mask):
    w, h, bitdepth, r = spec
    names, maxv, area = set(case["metrics"].split(",")), (1 << bitdepth) - 1, w * h
    f0, f1 = (_p444(f, case["chroma"]) for f in frames)
    weights = _ws(h) if case["erp"] else None
    res = {k: [0.0] * 4 for f in (DECIBELS, SIMILARITIES) for k in f[0]}
    res.update({k: 0.0 for f in (DECIBELS, SIMILARITIES) for k in f[1]})
    m = torch.ones(h, w, dtype=torch.int64, device=f0.device) if mask is None else mask.to(torch.int64)
    peak = float(area * maxv * maxv) if mask is None else float(int((m != 0).sum()) * 255 * maxv * maxv)
    row_ssd = ((f0 - f1) ** 2 * m).sum(2)
    fake = _db(float(area * maxv * maxv), 1.0)
    psnr = [_db(peak if mask is None else peak / maxv ** 2 * 255 ** 2, float(v)) for v in row_ssd.sum(1).tolist()]
    psnr = [v if v < 1e300 else fake for v in psnr]
    if "PSNR" in names:
        res["psnr"], res["psnr_pic"] = psnr + [0.0], _mean4(psnr)
    if "WSPSNR" in names:
        v = psnr
        if weights is not None:
            corr = h / weights.sum().item()
            v = [_db(peak, e * corr) for e in (row_ssd.to(torch.float64) * weights).sum(1).tolist()]
            v = [x if x < 1e300 else fake for x in v]
        res["wspsnr"], res["wspsnr_pic"] = v + [0.0], _mean4(v)
    if names & {"IVPSNR", "IVSSIM", "IVMSSSIM"}:
        den = area if mask is None else int((m != 0).sum()) * 255
        lim = math.floor(0.01 * maxv + 0.5)
        sd = ((f1 - f0) * m).sum((1, 2)).tolist()
        g = [max(-lim, min(lim, int(math.copysign(math.floor(abs(v / den) + 0.5), v)))) for v in sd]
        g = torch.tensor(g, device=f0.device)[:, None, None]
        found1 = _search(f0 + g, f1, r, None if mask is None else m)
        found0 = _search(f1 - g, f0, r, None if mask is None else m)
        quality = []
        for d in (f0 + g - found1, f1 - g - found0):
            rows = (d * d * m).sum(2)
            err = (rows.to(torch.float64) * weights).sum(1) if weights is not None else rows.sum(1).to(torch.float64)
            quality.append(_mean4([_db(peak, e if e > 0 else 1.0) for e in err.tolist()] + [0.0]))
        if mask is not None:
            quality = quality[::-1]   # mask mode names the search of the second picture in the first R2T
        if "IVPSNR" in names:
            res["ivpsnr_r2t"], res["ivpsnr_t2r"], res["ivpsnr"] = quality[0], quality[1], min(quality)
        scp1, scp0 = (found1 - g).clamp(0, maxv), (found0 + g).clamp(0, maxv)
        if "IVSSIM" in names:
            t2r = _mean4(_ssim(f0, scp1, maxv, case, weights=weights) + [0.0])
            r2t = _mean4(_ssim(f1, scp0, maxv, case, weights=weights) + [0.0])
            res["ivssim_t2r"], res["ivssim_r2t"], res["ivssim"] = t2r, r2t, min(t2r, r2t)
        if "IVMSSSIM" in names:
            t2r, r2t = (_mean4(_msssim(a, b, maxv, case) + [0.0]) for a, b in ((f0, scp1), (f1, scp0)))
            res["ivmsssim_t2r"], res["ivmsssim_r2t"], res["ivmsssim"] = t2r, r2t, min(t2r, r2t)
    if "SSIM" in names:
        v = _ssim(f0, f1, maxv, case)
        res["ssim"], res["ssim_pic"] = v + [0.0], _mean4(v + [0.0])
    if "MSSSIM" in names:
        v = _msssim(f0, f1, maxv, case)
        res["msssim"], res["msssim_pic"] = v + [0.0], _mean4(v + [0.0])
    return res


def exact(case, seed):
    frames, masks = _inputs(case, seed)
    rows = [_exact_pair(case, spec, frames[i], masks[i] if masks else None) for i, spec in enumerate(_specs(case, seed))]
    return _tables(rows, masks or None, whole=False)
