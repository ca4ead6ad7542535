"""The work a user has this backend do, as measurable cases.

A case is a dict of plain values. Its `kind` is the entry point it goes through:

  stack     Device.stack_dev: one stacking pass over filtered frames in HBM
  plugin    SearchBackend.run(StackPass): the plugin hook, frames on the host
  stage     Device.stage_dev: the preprocessing stage of frames in HBM
  search    Device.search_dev: a whole search, null runs included
  upload    Device.search: the same from frames on the host
  batch     Device.search_batch_dev: a search and its injection copies
  serve     Server.submit / poll: requests of uneven size in flight together

The sizes follow the benchmark workloads (fainttrail_b200/synthetic.py), the
serving configuration they are drawn from (8 to 120 frames, 512 x 512 and up,
0.1 to 3 px/min, 8 to 32 null runs, here towards its smaller requests) and the
tests (frames down to about 100 x 100). Frames are a sky with read and photon
noise, stars of log-uniform flux and a few movers, with a Gaussian PSF; the
stacking passes get filtered frames (unit noise, correlated over the PSF).
"""
import math

import numpy as np
import torch

import fainttrail_b200 as ftb

FWHM_TO_SIGMA = 1.0 / 2.354820045030949
GRID_TOL_PX = 0.125  # the workloads' half-pixel grid step over the span

_open = {}


def _device():
    """The context of this process, opened once as a program would."""
    if "device" not in _open:
        _open["device"] = ftb.Device()
    return _open["device"]


def _server():
    if "server" not in _open:
        _open["server"] = ftb.Server(workers=2)
    return _open["server"]


# --------------------------------------------------------------------------- cases

def listed():
    return [
        # the smallest call: one pass of a test-size sequence (launches and host steps)
        dict(name="stack-smallest", kind="stack", n=12, w=128, h=96, cadence=60.0, lo=0.2, hi=1.1, tracks="linear"),
        # an ordinary pass through the plugin hook, as a host application's own search() makes it
        dict(name="plugin-1k", kind="plugin", n=20, w=1024, h=1024, cadence=60.0, lo=0.2, hi=1.1, tracks="linear"),
        # the headline pass: the full-frame workload's frames and 19,328 motions
        dict(name="stack-fullframe-4k", kind="stack", n=40, w=4096, h=4096, cadence=30.0, lo=0.1, hi=2.0,
             tracks="linear"),
        # many frames on an odd size, a slow mover search (the taller frame stacks' tiles)
        dict(name="stack-120-frames", kind="stack", n=120, w=1201, h=803, cadence=30.0, lo=0.1, hi=0.6,
             tracks="linear"),
        # explicit shift tables of curved tracks (an orbit's arc rather than a straight line)
        dict(name="stack-curved", kind="stack", n=30, w=1000, h=700, cadence=60.0, lo=0.2, hi=0.7, tracks="curved"),
        # the preprocessing of a batched-workload-size sequence, PSF of the workloads
        dict(name="stage-2k", kind="stage", n=40, w=2048, h=2048, cadence=30.0, fwhm=2.5, blank=0),
        # a tall stack with a wide PSF and blank borders that move with the frames
        dict(name="stage-120-wide", kind="stage", n=120, w=1030, h=777, cadence=30.0, fwhm=6.0, blank=6),
        # the smallest preprocessing call
        dict(name="stage-smallest", kind="stage", n=9, w=211, h=133, cadence=60.0, fwhm=2.5, blank=3),
        # the plain whole search: 20 x 1024^2 and 8 null runs
        dict(name="search-plain-1k", kind="search", n=20, w=1024, h=1024, cadence=60.0, lo=0.2, hi=1.1, nulls=8,
             fwhm=2.5, blank=0),
        # a served request's search from host frames: uneven size, PSF width estimated, blank borders
        dict(name="upload-odd", kind="upload", n=33, w=1501, h=1117, cadence=30.0, lo=0.4, hi=0.9, nulls=8, fwhm=0.0,
             blank=5),
        # null calibration and completeness copies in one batch
        dict(name="batch-1k", kind="batch", n=30, w=1024, h=1024, cadence=60.0, lo=0.2, hi=1.1, nulls=6, copies=3,
             objects=50, fwhm=2.5, blank=0),
        # three requests of uneven size submitted together
        dict(name="serve-3", kind="serve", requests=3, n=16, w=800, h=608, cadence=30.0, lo=0.3, hi=1.5, nulls=8,
             fwhm=2.5, blank=0),
    ]


def _span_h(case):
    return (case["n"] - 1) * case["cadence"] / 3600.0


def _motions(case):
    """The search's square velocity lattice inside the annulus, in px/h."""
    dv = 4.0 * GRID_TOL_PX / _span_h(case)
    k = int(math.ceil(case["hi"] * 60.0 / dv))
    a = np.arange(-k, k + 1) * dv
    vx, vy = np.meshgrid(a, a)
    v = np.hypot(vx, vy)
    keep = (v >= max(0.0, case["lo"] * 60.0 - 0.5 * dv)) & (v <= case["hi"] * 60.0 + 0.5 * dv)
    return np.stack([vx[keep], vy[keep]], 1)


def _adds(case):
    return float(len(_motions(case))) * case["n"] * case["w"] * case["h"]


def draw(rng):
    """One more case: sizes log-uniform over the range, odd ones among them, at
    most 4e12 adds (a third of the listed headline pass)."""
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    while True:
        kind = rng.choice(["stack", "stack", "plugin", "stage", "stage", "search", "search", "upload", "batch"])
        c = dict(kind=kind, n=log(8, 120), w=log(100, 3000), h=log(90, 2200), cadence=rng.choice([30.0, 60.0]))
        if kind == "stage":
            if c["n"] * c["w"] * c["h"] <= 2.2e8:
                return dict(c, fwhm=round(rng.uniform(1.8, 6.5), 2), blank=rng.choice([0, 0, 4, 9]))
            continue
        c["lo"] = round(rng.uniform(0.1, 1.5), 2)
        c["hi"] = round(c["lo"] + rng.uniform(0.2, 1.5), 2)
        passes = 1
        if kind in ("stack", "plugin"):
            c["tracks"] = rng.choice(["linear", "linear", "linear", "curved"]) if kind == "stack" else "linear"
        else:
            c["w"], c["h"] = max(c["w"], 200), max(c["h"], 160)
            c["nulls"] = rng.randint(3, 12)
            c["fwhm"] = rng.choice([0.0, 2.5, round(rng.uniform(2.0, 5.0), 2)])
            c["blank"] = rng.choice([0, 0, 5])
            passes += c["nulls"]
            if kind == "batch":
                c["fwhm"] = c["fwhm"] or 2.5
                c["copies"], c["objects"] = rng.randint(1, 3), rng.randint(5, 50)
                passes += c["copies"]
        m = math.pi * ((c["hi"] * 60) ** 2 - (c["lo"] * 60) ** 2) * (_span_h(c) / (4.0 * GRID_TOL_PX)) ** 2
        if 50 <= m <= 60000 and m * c["n"] * c["w"] * c["h"] * passes <= 4e12:
            return c


def work(case):
    """Frames in, results out; one add per pixel, frame, motion and pass."""
    px = float(case["n"]) * case["w"] * case["h"]
    plane = float(case["w"]) * case["h"]
    kind = case["kind"]
    if kind in ("stack", "plugin"):
        return {"bytes": 4.0 * px + 8.0 * plane, "flops": _adds(case)}
    if kind == "stage":
        # frames in, filtered frames out, sky and mask; two separable passes of 2R + 1 taps
        taps = 2 * max(1, math.ceil(3.0 * case["fwhm"] * FWHM_TO_SIGMA)) + 1
        return {"bytes": 8.0 * px + 8.0 * plane, "flops": 4.0 * taps * px}
    if kind == "serve":
        each = [_request(case, k) for k in range(case["requests"])]
        return {"bytes": sum(4.0 * q["n"] * q["w"] * q["h"] + 8.0 * q["w"] * q["h"] for q in each),
                "flops": sum((1 + q["nulls"]) * _adds(q) for q in each)}
    passes = 1 + case["nulls"] + case.get("copies", 0)
    return {"bytes": 4.0 * px + 8.0 * plane * (1 + case.get("copies", 0)), "flops": passes * _adds(case)}


def _request(case, k):
    """The k-th request of a serving case: each a third larger on a side, with more frames."""
    return dict(case, n=case["n"] + 9 * k, w=case["w"] + 272 * k, h=case["h"] + 208 * k,
                hi=round(case["hi"] - 0.3 * k, 2))


# --------------------------------------------------------------------------- inputs

def _times(case):
    mjd = 61337.9 + (np.arange(case["n"]) * case["cadence"] + 0.5 * case["cadence"]) / 86400.0
    return mjd, np.full(case["n"], 0.75 * case["cadence"])


def _t_h(case):
    mjd, _ = _times(case)
    return (mjd - 0.5 * (mjd[0] + mjd[-1])) * 24.0


def _blur(img, sigma, scale):
    """Separable Gaussian by shifted adds (the same in every process)."""
    r = int(math.ceil(4.0 * sigma))
    k = [math.exp(-0.5 * (i / sigma) ** 2) for i in range(-r, r + 1)]
    s = scale / sum(k)
    for dim in (-1, -2):
        acc = torch.zeros_like(img)
        size = img.shape[dim]
        for i, kv in zip(range(-r, r + 1), k):
            a, b = max(0, -i), min(size, size - i)
            if a < b:
                acc.narrow(dim, a, b - a).add_(img.narrow(dim, a + i, b - a), alpha=kv * s)
        img, s = acc, 1.0 / sum(k)
    return img


def _frames(case, seed, filtered=False):
    """Frames (n, h, w) on the GPU: sky frames in ADU, or filtered ones."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    n, w, h = case["n"], case["w"], case["h"]
    sigma = (case.get("fwhm") or 2.5) * FWHM_TO_SIGMA
    noise = 1.0 if filtered else math.sqrt(1100.0)
    t = _t_h(case)
    # movers and stars as one list of (frame, pixel, flux) impulses, duplicates summed here
    stars = 0 if filtered else max(5, w * h // 20000)
    sx, sy = rng.integers(0, w, stars), rng.integers(0, h, stars)
    sf = np.exp(rng.uniform(math.log(2e3), math.log(2e6), stars))
    movers = 5
    snr = rng.uniform(6.0, 12.0, movers)
    flux = snr / math.sqrt(n) * noise * (1.0 if filtered else math.sqrt(4.0 * math.pi) * sigma)
    rate = 60.0 * rng.uniform(case.get("lo", 0.2), case.get("hi", 1.1), movers)
    pa = rng.uniform(0, 2 * math.pi, movers)
    mx = rng.uniform(0.1, 0.9, movers) * w
    my = rng.uniform(0.1, 0.9, movers) * h
    image = torch.zeros((h, w), device="cuda")
    if stars:
        at, inv = np.unique(sy * w + sx, return_inverse=True)
        image.view(-1)[torch.from_numpy(at).cuda()] = torch.from_numpy(np.bincount(inv, sf).astype(np.float32)).cuda()
        image = _blur(image, sigma, 1.0)
    frames = torch.empty((n, h, w), device="cuda")
    for i in range(n):
        imp = torch.zeros((h, w), device="cuda")
        x = np.rint(mx + rate * np.cos(pa) * t[i]).astype(np.int64)
        y = np.rint(my + rate * np.sin(pa) * t[i]).astype(np.int64)
        ok = (x >= 0) & (x < w) & (y >= 0) & (y < h)
        at, inv = np.unique(y[ok] * w + x[ok], return_inverse=True)
        if len(at):
            imp.view(-1)[torch.from_numpy(at).cuda()] = torch.from_numpy(
                np.bincount(inv, flux[ok]).astype(np.float32)).cuda()
        g = torch.randn((h, w), generator=gen, device="cuda")
        if filtered:
            # white noise and a matched source, both through the filter: unit noise, unit peak
            k2 = 4.0 * math.pi * sigma * sigma
            frames[i] = _blur(g, sigma, math.sqrt(k2)) + _blur(imp, math.sqrt(2.0) * sigma, k2)
        else:
            level = 1000.0 * (1.0 + 0.01 * float(rng.standard_normal()))
            frames[i] = g.mul_(noise).add_(level).add_(image).add_(_blur(imp, sigma, 1.0))
    blank = case.get("blank", 0)
    for i in range(n if blank else 0):  # borders a registration leaves blank, drifting over the sequence
        a, b = (i * blank) // n, blank - (i * blank) // n
        frames[i, :, :a] = float("nan")
        frames[i, :, w - b:] = float("nan")
        frames[i, :b // 2, :] = float("nan")
    return frames


def _subtracted(case, seed):
    f = _frames(case, seed)
    for i in range(case["n"]):
        f[i] -= torch.nanmedian(f[i, ::7, ::5])
    return f


def _lround(x):
    t = np.trunc(x)
    return (t + np.sign(x) * (np.abs(x - t) >= 0.5)).astype(np.int32)


def _shifts(case, seed):
    """Shift tables (motion, frame): straight tracks, or each with a curvature of
    its own (up to a tenth of its rate over half the span)."""
    v, t = _motions(case), _t_h(case)
    px, py = v[:, :1] * t, v[:, 1:] * t
    if case["tracks"] == "curved":
        rng = np.random.default_rng(seed + 1)
        half = 0.5 * _span_h(case)
        a = rng.uniform(-0.1, 0.1, (len(v), 2)) * np.hypot(v[:, :1], v[:, 1:]) / half
        px, py = px + a[:, :1] * t * t, py + a[:, 1:] * t * t
    return np.ascontiguousarray(_lround(px)), np.ascontiguousarray(_lround(py))


def _min_count(case):
    return max(3, math.ceil(0.7 * case["n"]))


def _params(case):
    return dict(vmin_pxh=case["lo"] * 60.0, vmax_pxh=case["hi"] * 60.0, grid_tol_px=GRID_TOL_PX, fwhm_px=case["fwhm"],
                null_runs=case["nulls"])


def _copies(case, seed):
    rng = np.random.default_rng(seed + 2)
    sets = []
    for _ in range(case["copies"]):
        q = case["objects"]
        rate = 60.0 * rng.uniform(case["lo"], case["hi"], q)
        pa = rng.uniform(0, 2 * math.pi, q)
        flux = rng.uniform(2.0, 8.0, q) / math.sqrt(case["n"]) * math.sqrt(1100.0) * math.sqrt(4.0 * math.pi) * (
            case["fwhm"] * FWHM_TO_SIGMA)
        x = rng.uniform(24, case["w"] - 24, q)
        y = rng.uniform(24, case["h"] - 24, q)
        sets.append([tuple(map(float, o)) for o in zip(x, y, rate * np.cos(pa), rate * np.sin(pa), flux)])
    return sets


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, device=_device())
    n, w, h = case["n"], case["w"], case["h"]
    if kind == "stack":
        pitch = (w + 3) // 4 * 4  # rows on 16 bytes, as the entry point wants
        s["frames"] = torch.zeros((n, h, pitch), device="cuda")
        s["frames"][:, :, :w] = _frames(case, seed, filtered=True)
        s["dx"], s["dy"] = _shifts(case, seed)
        s["max_snr"] = torch.empty((h, w), device="cuda")
        s["best_v"] = torch.empty((h, w), dtype=torch.int32, device="cuda")
    elif kind == "plugin":
        s["backend"] = ftb.make_backend("b200", s["device"])
        s["frames"] = _frames(case, seed, filtered=True).cpu().numpy()
        s["velocities"] = _motions(case)
    elif kind == "stage":
        s["frames"] = _subtracted(case, seed)
        s["filtered"] = torch.zeros_like(s["frames"])
        s["sky"] = torch.zeros((h, w), device="cuda")
        s["mask"] = torch.zeros((h, w), device="cuda")
    elif kind == "serve":
        s["server"] = _server()
        s["requests"] = [(q, _frames(q, seed + 100 * k).cpu().numpy())
                         for k, q in enumerate(_request(case, k) for k in range(case["requests"]))]
    else:
        s["frames"] = _frames(case, seed)
        if kind == "upload":
            s["frames"] = s["frames"].cpu().numpy()
        if kind == "batch":
            s["copies"] = _copies(case, seed)
    return s


# --------------------------------------------------------------------------- one pass

def _filled(a, shape):
    """`a` at the start of an array of a fixed shape (lists differ in length from field to field)."""
    out = np.zeros(shape)
    out[tuple(slice(0, k) for k in a.shape)] = a
    return out


def _result(r, case, nulls=True):
    """What a search gives its user, as arrays."""
    rows = np.array([c[0] for c in r["candidates"]]).reshape(-1, 17)
    out = dict(threshold=r["threshold"], max_snr=r["max_snr"], best_v=r["best_v"], found=len(rows),
               candidates=_filled(rows, (300, 17)), tracks=_filled(r["track_points"], (300, case["n"], 5)))
    return dict(out, null_peaks=_filled(r["null_peaks"], (20000 * case["nulls"],)), fwhm=r["fwhm"]) if nulls else out


def run(state):
    case, dev = state["case"], state["device"]
    kind = case["kind"]
    if kind == "serve":
        server = state["server"]
        tickets = [server.submit(f, *_times(q), **_params(q)) for q, f in state["requests"]]
        return [_result(server.poll(t), q) for t, (q, _) in zip(tickets, state["requests"])]
    n, w, h = case["n"], case["w"], case["h"]
    f = state["frames"]
    if kind == "stack":
        dev.stack_dev(f.data_ptr(), w, h, f.shape[2], n, state["dx"], state["dy"], _min_count(case),
                      state["max_snr"].data_ptr(), state["best_v"].data_ptr())
        return dict(max_snr=state["max_snr"], best_v=state["best_v"])
    if kind == "plugin":
        r = state["backend"].run(ftb.StackPass(f, t_h=_t_h(case), velocities=state["velocities"],
                                               min_count=_min_count(case)))
        return dict(max_snr=r.max_snr, best_v=r.best_v)
    if kind == "stage":
        r = dev.stage_dev(f.data_ptr(), w, h, w, n, _t_h(case), case["fwhm"], d_filtered=state["filtered"].data_ptr(),
                          d_static_sky=state["sky"].data_ptr(), d_mask=state["mask"].data_ptr())
        return dict(filtered=state["filtered"], sky=state["sky"], mask=state["mask"], sigma=r["sigma"], cr=r["cr"])
    if kind == "search":
        return _result(dev.search_dev(f.data_ptr(), w, h, w, n, *_times(case), **_params(case)), case)
    if kind == "upload":
        return _result(dev.search(f, *_times(case), **_params(case)), case)
    if kind == "batch":
        base, copies = dev.search_batch_dev(f.data_ptr(), w, h, w, n, *_times(case), state["copies"], **_params(case))
        return dict(base=_result(base, case), copies=[_result(c, case, nulls=False) for c in copies])
    raise ValueError("unknown kind %r" % kind)


# --------------------------------------------------------------------------- 64 bits

def _exact_stack(frames, dx, dy, min_count):
    """max over motions of (sum of the covering frames) / sqrt(their number); 0 where none is defined."""
    n, h, w = frames.shape
    f = frames.double()
    best = torch.full((h, w), -math.inf, dtype=torch.float64, device=f.device)
    X, Y = torch.arange(w, device=f.device), torch.arange(h, device=f.device)
    tx, ty = torch.from_numpy(dx).to(f.device), torch.from_numpy(dy).to(f.device)
    for j in range(dx.shape[0]):
        acc = torch.zeros((h, w), dtype=torch.float64, device=f.device)
        for i in range(n):
            a, b = int(dx[j, i]), int(dy[j, i])
            x0, x1, y0, y1 = max(0, -a), min(w, w - a), max(0, -b), min(h, h - b)
            if x0 < x1 and y0 < y1:
                acc[y0:y1, x0:x1] += f[i, y0 + b:y1 + b, x0 + a:x1 + a]
        inx = ((X[None] + tx[j][:, None] >= 0) & (X[None] + tx[j][:, None] < w)).double()
        iny = ((Y[None] + ty[j][:, None] >= 0) & (Y[None] + ty[j][:, None] < h)).double()
        c = iny.t() @ inx
        torch.maximum(best, torch.where(c >= min_count, acc / c.clamp(min=1.0).sqrt(), -math.inf), out=best)
    return torch.where(torch.isfinite(best), best, 0.0)


def _step(w, h, border):
    usable = max(0, w - 2 * border) * max(0, h - 2 * border)
    return max(1, int(math.sqrt(usable / 200000.0))) if usable else 0


def _sigma(frame, border, mask=None):
    """1.4826 times the median absolute deviation of a frame's sample grid."""
    h, w = frame.shape
    st = _step(w, h, border)
    if not st:
        return 0.0
    v = frame[border:h - border:st, border:w - border:st]
    ok = torch.isfinite(v)
    if mask is not None:
        ok &= mask[border:h - border:st, border:w - border:st] != 0
    v = v[ok]
    if v.numel() < 3:
        return 0.0
    mid = lambda x: 0.5 * float((x[(x.numel() - 1) // 2] + x[x.numel() // 2]))  # noqa: E731
    return 1.4826 * mid((v - mid(v.sort().values)).abs().sort().values)


def _middle(sv, m):
    """The median of the first m of the sorted values along dim 0."""
    lo = ((m - 1).clamp(min=0) // 2).unsqueeze(0)
    hi = (m // 2).clamp(max=sv.shape[0] - 1).unsqueeze(0)
    return 0.5 * (sv.gather(0, lo) + sv.gather(0, hi))[0]


def _exact_stage(frames, fwhm):
    """The preprocessing stage in 64 bits, frames in time order."""
    n, h, w = frames.shape
    v = frames.double()
    fin = torch.isfinite(v)
    e = max(1, int(n / 8.0 + 0.5))
    m_all = fin.sum(0)
    sv, order = torch.where(fin, v, math.inf).sort(dim=0, stable=True)
    known = m_all >= max(5, int(0.6 * n))
    sky = torch.where(known, _middle(sv, m_all), math.nan)
    pos = torch.empty_like(order).scatter_(0, order, torch.arange(n, device=v.device).view(-1, 1, 1).expand_as(order))
    del order
    res = torch.empty_like(v)
    ranks = torch.arange(n, device=v.device).view(-1, 1, 1)
    inside = ranks < m_all.unsqueeze(0)
    for r in range(n):
        kept = inside.clone()
        kept.scatter_(0, pos[max(0, r - e):r + e + 1], False)
        m = kept.sum(0)
        cum = kept.cumsum(0, dtype=torch.int16)
        lo = (cum < (m - 1).unsqueeze(0) // 2 + 1).sum(0, keepdim=True).clamp(max=n - 1)
        hi = (cum < m.unsqueeze(0) // 2 + 1).sum(0, keepdim=True).clamp(max=n - 1)
        out = 0.5 * (sv.gather(0, lo) + sv.gather(0, hi))[0]
        st = torch.where(m >= 5, out, sky)
        res[r] = torch.where(fin[r] & known, v[r] - st, math.nan)
    del sv, pos, inside
    sigma = np.array([_sigma(res[i], 2) or 1.0 for i in range(n)])
    sg = torch.from_numpy(sigma).to(v.device).view(-1, 1, 1)
    fin = torch.isfinite(res)
    dev = torch.where(fin, res.abs() / sg, math.inf).sort(dim=0).values
    c = fin.sum(0)
    scatter = torch.where(c < n // 2, 1e9, 1.4826 * _middle(dev, c))
    del dev
    dil = max(1, int(0.5 * fwhm + 0.5))
    bad = (scatter > 2.5).double()[None, None]
    mask = 1.0 - torch.nn.functional.max_pool2d(bad, 2 * dil + 1, 1, dil)[0, 0]
    s = fwhm * FWHM_TO_SIGMA
    R = max(1, math.ceil(3.0 * s))
    k = [math.exp(-0.5 * i * i / (s * s)) for i in range(-R, R + 1)]
    norm = 1.0 / sum(x * x for x in k)
    ratio = 0.5 * math.exp(-0.5 / (s * s))
    weight = torch.where(scatter > 1.5, scatter, 1.0)
    out = torch.empty_like(v)
    border = math.ceil(3 * s) + 1
    for i in range(n):
        z = torch.where((mask != 0) & fin[i], res[i] / sigma[i] / weight, 0.0)
        flag = torch.zeros_like(z, dtype=torch.bool)
        core = z[1:-1, 1:-1]
        near = 0.25 * (z[1:-1, :-2] + z[1:-1, 2:] + z[:-2, 1:-1] + z[2:, 1:-1])
        flag[1:-1, 1:-1] = (core >= 5.0) & ~(near >= ratio * core)
        around = torch.nn.functional.max_pool2d(flag.double()[None, None], 3, 1, 1)[0, 0] > 0
        z = torch.where(flag | (around & (z > 2.5)), 0.0, z).clamp(-8.0, 8.0)
        for dim, scale in ((-1, 1.0), (-2, norm)):
            acc, size = torch.zeros_like(z), z.shape[dim]
            for q, kv in zip(range(-R, R + 1), k):
                a, b = max(0, -q), min(size, size - q)
                if a < b:
                    acc.narrow(dim, a, b - a).add_(z.narrow(dim, a + q, b - a), alpha=kv * scale)
            z = acc
        g = _sigma(z, border, mask)
        out[i] = z / g if g > 0 else z
    return dict(filtered=out, sky=sky, mask=mask, sigma=sigma, cr=None)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("stack", "plugin"):
        if len(_motions(case)) * case["n"] > 200000 or _adds(case) > 2e11:
            return None  # over about 20 seconds in 64 bits
        frames = _frames(case, seed, filtered=True)
        dx, dy = _shifts(dict(case, tracks=case.get("tracks", "linear")), seed)
        return dict(max_snr=_exact_stack(frames, dx, dy, _min_count(case)), best_v=None)
    if kind == "stage":
        if case["n"] * case["w"] * case["h"] > 1.8e8:
            return None
        return _exact_stage(_subtracted(case, seed), case["fwhm"])
    return None  # a whole search's maps: too many passes for 64 bits
