"""The work that users of this framework have it do, as measurable cases over its public entry points.

listed(): the cases; draw(rng): one more of the same ranges; prepare(case, seed): what a program holds before the call;
run(state): one call, its whole outputs; work(case): the bytes and operations the call cannot do without;
exact(case, seed): the same outputs in float64 by plain torch on the device (a restatement of the method that shares
no code with the framework: python/optflow_ref's phaseflow.py, poc.py, interp.py, strain.py, track.py).

Inputs are speckle pairs of the synthetic generator under a smooth random field, with noise and 8-bit levels, as the
tests and the benchmark use them.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "optflow-soil_b200"))

from optflow_b200 import Config, Engine, api, net, synth  # noqa: E402

OUTS = ("ux", "uy", "conf", "exx", "eyy", "exy", "gmax", "vol", "raw_ux", "raw_uy", "valid")
DEV = "cuda:0"


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest whole pair: a 128 px patch, where launches and latency are the cost
        dict(name="pair_128", kind="pair", w=128, h=128, order=1, mask=False, init=False, freeze=0),
        # a 256 px pair from a start field: what every leg of the CPU-sized example sequence does after the first
        dict(name="pair_256_init", kind="pair", w=256, h=256, order=1, mask=False, init=True, freeze=0),
        # an ROI crop as a user cuts it: odd sides, a mask
        dict(name="pair_333x191_roi", kind="pair", w=333, h=191, order=1, mask=True, init=False, freeze=0),
        # the quadratic shape function at a common size
        dict(name="pair_512_order2", kind="pair", w=512, h=512, order=2, mask=False, init=False, freeze=0),
        # a frame of a 1080p clip at scale 2, ROI and frozen pre-warp: the footing clip's settings
        dict(name="pair_960x540_roi", kind="pair", w=960, h=540, order=1, mask=True, init=False, freeze=3),
        # an ordinary square pair
        dict(name="pair_1024", kind="pair", w=1024, h=1024, order=1, mask=False, init=False, freeze=0),
        # a large ragged crop: neither side has a convenient transform length
        dict(name="pair_1367x911", kind="pair", w=1367, h=911, order=1, mask=False, init=False, freeze=0),
        # the benchmark's size with its ROI: the largest pair
        dict(name="pair_2048_roi", kind="pair", w=2048, h=2048, order=1, mask=True, init=False, freeze=0),
        # the fine stage by itself on host planes (a tiling or stereo driver's call)
        dict(name="refine_640x480", kind="refine", w=640, h=480, order=1, freeze=0),
        # a batch of uneven pairs in one call, sizes of the uneven batch of the benchmarks
        dict(name="batch_uneven", kind="batch", sizes="1024x768,512x1024,256x512,768x768,1536x512"),
        # a short chain sequence of 256 px frames, the CPU-sized example
        dict(name="sequence_256", kind="sequence", w=256, h=256, frames=5),
        # one training step (forward and backward) of the coarse network at its training size
        dict(name="net_train_16x256", kind="train", w=256, h=256, batch=16),
    ]


def _log_size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    k = rng.random()
    if k < 0.7:  # single pairs, any sides
        w, h = _log_size(rng, 80, 2048), _log_size(rng, 80, 2048)
        if rng.random() < 0.3:  # standard sides
            w = rng.choice([128, 256, 320, 480, 512, 640, 720, 768, 960, 1024, 1280, 1536, 1920])
            h = rng.choice([128, 256, 240, 360, 480, 512, 540, 600, 720, 768, 1024, 1080])
        if min(w, h) < 192:  # strips: the coarse stage's windows are at most 64 px a side
            w, h = min(w, 380), min(h, 380)
        order = 2 if rng.random() < 0.15 and w * h <= 1 << 20 else 1
        return dict(kind="pair", w=w, h=h, order=order, mask=rng.random() < 0.4, init=rng.random() < 0.25,
                    freeze=rng.choice([0, 0, 3]))
    if k < 0.8:
        return dict(kind="refine", w=_log_size(rng, 100, 1100), h=_log_size(rng, 100, 1100), order=1,
                    freeze=rng.choice([0, 3]))
    if k < 0.87:
        sides = [(256, 512, 768)] * 4 + [(768, 1024)]
        return dict(kind="batch", sizes=",".join(f"{rng.choice(s)}x{rng.choice(s)}" for s in sides))
    if k < 0.94:
        return dict(kind="sequence", w=_log_size(rng, 120, 400), h=_log_size(rng, 120, 400), frames=rng.randint(3, 5))
    return dict(kind="train", w=8 * rng.randint(16, 40), h=8 * rng.randint(16, 40), batch=rng.choice([4, 8, 16]))


# ---------------------------------------------------------------- inputs
_session = {}


def _engine():
    """The program's engine and stream, made once."""
    if not _session:
        _session["engine"] = Engine(0)
        _session["stream"] = torch.cuda.Stream(DEV)
    return _session["engine"]


def _field(w, h, rng, scale=1.0):
    """A smooth random field that comes to rest at the frame, as soil does at the walls of its box."""
    length = min(128.0, 0.5 * min(w, h))
    grid, gx0, gy0 = synth.gp_grid(h, w, length, scale * length / 12.0, rng)
    rest = []
    for n, g0, k in ((h, gy0, grid.shape[1]), (w, gx0, grid.shape[2])):
        x = g0 + 16.0 * np.arange(k)
        rest.append(np.clip(np.minimum(x, n - 1 - x) / (0.25 * n), 0.0, 1.0))
    grid = grid * np.outer(np.sin(0.5 * np.pi * rest[0]), np.sin(0.5 * np.pi * rest[1]))
    return synth.Field(c=(w / 2, h / 2), grid=grid, gx0=gx0, gy0=gy0, gh=16.0)


def _frames(w, h, seed, n=2):
    """n speckle frames (float32, 8-bit levels) under the field grown frame by frame, and the last frame's field."""
    rng = np.random.default_rng([seed, w, h, n])
    p = synth.make_pattern(h, w, seed=int(rng.integers(1 << 31)), rmin=1.5, rmax=2.5)
    state = rng.bit_generator.state
    out, f = [], None
    for k in range(n):
        if k:
            rng.bit_generator.state = state
            f = _field(w, h, rng, k / (n - 1))
        img = synth.render(p, h, w, f, engine=_engine())
        out.append(synth.degrade(img, seed=int(seed) * 101 + k, noise=0.01, bits=8))
    return out, f


def _mask(case, w, h):
    return synth.rect_roi(h, w, 0.1 * w, 0.1 * h, 0.9 * w, 0.9 * h) if case.get("mask") else None


def _start(field, w, h, seed):
    """A start field as a program has it: the motion to within a pixel."""
    u, v = field.displacement(h, w)
    rng = np.random.default_rng(seed)
    yy, xx = np.mgrid[0:h, 0:w]
    d = [0.4 * np.sin(2 * np.pi * (xx / w * rng.uniform(1, 3) + yy / h * rng.uniform(1, 3))) for _ in range(2)]
    return (u + d[0]).astype(np.float32), (v + d[1]).astype(np.float32)


def _config(case):
    return Config(shape_order=case.get("order", 1), prewarp_freeze_at=case.get("freeze", 0))


def _inputs(case, seed):
    """Host inputs of a case: dict of numpy arrays (and lists of them)."""
    kind = case["kind"]
    if kind == "batch":
        items = []
        for i, s in enumerate(case["sizes"].split(",")):
            w, h = map(int, s.split("x"))
            fr, _ = _frames(w, h, seed * 16 + i)
            items.append(tuple(fr))
        return dict(items=items)
    w, h = case["w"], case["h"]
    if kind == "sequence":
        return dict(frames=_frames(w, h, seed, case["frames"])[0])
    if kind == "train":
        i1, i2, tg, mk = [], [], [], []
        for i in range(case["batch"]):
            fr, f = _frames(w, h, seed * 64 + i)
            t, m = net.cell_target(f, h, w)
            i1.append(fr[0]), i2.append(fr[1]), tg.append(t), mk.append(m)
        return dict(i1=np.stack(i1), i2=np.stack(i2), target=np.stack(tg), mask=np.stack(mk),
                    params=net.load_weights())
    fr, f = _frames(w, h, seed)
    d = dict(i1=fr[0], i2=fr[1], mask=_mask(case, w, h), init=None)
    if case.get("init") or kind == "refine":
        d["init"] = _start(f, w, h, seed)
    return d


def prepare(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    s = dict(kind=kind, engine=_engine(), stream=_session["stream"], cfg=_config(case))
    if kind == "pair":
        up = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
        s.update(i1=up(d["i1"]), i2=up(d["i2"]), mask=up(d["mask"]),
                 init=None if d["init"] is None else tuple(up(a) for a in d["init"]))
    elif kind == "train":
        for k in ("i1", "i2", "target", "mask"):
            s[k] = torch.from_numpy(d[k]).to(DEV)
        if "net" not in _session:
            _session["net"] = net.CoarseNet(0, d["params"])
        s["net"] = _session["net"]
        s["grads"] = torch.empty(d["params"].size, dtype=torch.float32, device=DEV)
    else:
        s.update(d)
    torch.cuda.synchronize()
    return s


def _planes(r):
    o = dict(ux=r.ux, uy=r.uy, conf=r.conf, raw_ux=r.raw_ux, raw_uy=r.raw_uy, valid=r.valid)
    o.update({k: r.strain[n] for k, n in (("exx", "Exx"), ("eyy", "Eyy"), ("exy", "Exy"), ("gmax", "gmax"), ("vol", "vol"))})
    return o


def run(s):
    kind, eng, cfg = s["kind"], s["engine"], s["cfg"]
    if kind == "pair":
        return api.track_pair_device(s["i1"], s["i2"], cfg, mask=s["mask"], init=s["init"], stream=s["stream"], engine=eng)
    if kind == "refine":
        f = api.refine(s["i1"], s["i2"], s["init"][0], s["init"][1], cfg, engine=eng)
        return dict(ux=f.ux, uy=f.uy, conf=f.conf, resid=f.resid, low=f.low)
    if kind == "batch":
        return [_planes(r) for r in api.track_pairs(s["items"], cfg, engine=eng)]
    if kind == "sequence":
        return [_planes(r) for _, r in api.track_sequence(s["frames"], cfg, engine=eng)]
    loss, flow, grads = s["net"].gradients(s["i1"], s["i2"], s["target"], s["mask"], grads=s["grads"], stream=s["stream"])
    return dict(loss=loss, flow=flow, grads=grads)


# ---------------------------------------------------------------- what a call cannot do without
def _fine_flops(w, h, order, outer=8, inner=2, filters=12):
    lg = math.log2((w + 64) * (h + 64))
    fft = 2.5 * lg * (1 + 2 * filters) * (w + 64) * (h + 64) / (w * h)  # a real transform in, the complex ones out
    mom = {1: (15 + 26) * 33 + 250, 2: (29 + 62) * 33 + 1300}[order] * 2
    acc = filters * (16 * 4 + 30) * 2 + 2 * (16 * 4 + 20) * 2
    ref = 2.5 * lg * (1 + 6 * filters)
    return w * h * (outer * (fft + 2 * 33 * 4 + 60 + inner * (acc + mom)) + ref)


def _pair_work(w, h, order, extra):
    poc = 1.25 * (w * h / 256) * 1.5 * 3 * 5 * 64 * 64 * 12  # windows of both levels, three transforms each
    return dict(bytes=w * h * (49 + extra), flops=_fine_flops(w, h, order) + poc + w * h * 11 * 15 * 4)


def work(case):
    kind = case["kind"]
    if kind == "pair":
        return _pair_work(case["w"], case["h"], case["order"], (1 if case["mask"] else 0) + (8 if case["init"] else 0))
    if kind == "refine":
        return dict(bytes=case["w"] * case["h"] * 33, flops=_fine_flops(case["w"], case["h"], case["order"]))
    if kind == "batch":
        ws = [_pair_work(*map(int, s.split("x")), 1, 0) for s in case["sizes"].split(",")]
        return {k: sum(x[k] for x in ws) for k in ("bytes", "flops")}
    if kind == "sequence":
        one = _pair_work(case["w"], case["h"], 1, 0)
        return {k: (case["frames"] - 1) * v for k, v in one.items()}
    px, n = case["w"] * case["h"], case["batch"]
    macs = 2 * (9 * 16 / 4 + 9 * 16 * 32 / 16 + 2 * 9 * 32 * 32 / 64) + (121 * 32 + 9 * (160 * 64 + 64 * 64 + 64 * 32 + 32 * 16)) / 64
    return dict(bytes=n * px * (8 + 17 / 64) + 3 * 4 * 175648, flops=n * px * macs * 6)


# ---------------------------------------------------------------- the method in float64 (plain torch)
PAD, Z = 32, math.sqrt(3.0) - 2.0
F64 = torch.float64


def _mirror(i, n):
    p = 2 * (n - 1)
    i = i.abs() % p
    return torch.where(i >= n, p - i, i)


def _spline(c):
    """Cubic B-spline coefficients along both axes (mirror boundaries, the 21-sample causal start)."""
    for _ in range(2):
        c = (c * 6.0).transpose(0, 1).contiguous()  # lines along dim 1
        n = c.shape[1]
        # the two recursions as one dense solve per line: a lower and an upper bidiagonal factor
        k = torch.arange(n, device=c.device)
        d = (k[:, None] - k[None, :]).to(F64)
        low = torch.where(d >= 0, Z ** d.clamp(min=0), torch.zeros((), dtype=F64, device=c.device))
        hz = min(n, 21)
        low[:, 1:hz] += (Z ** k.to(F64))[:, None] * (Z ** k[1:hz].to(F64))[None, :]
        up = torch.where(d <= 0, -Z * Z ** (-d).clamp(min=0), torch.zeros((), dtype=F64, device=c.device))
        g = Z / (Z * Z - 1.0)
        up[:, n - 1] = Z ** (n - 1 - k).to(F64) * g
        up[:, n - 2] += Z ** (n - 1 - k).to(F64) * g * Z
        m = (up @ low).T
        c = c @ m.to(c.dtype)
    return c


def _weights(t):
    return ((1 - t) ** 3 / 6, (3 * t ** 3 - 6 * t * t + 4) / 6, (-3 * t ** 3 + 3 * t * t + 3 * t + 1) / 6, t ** 3 / 6)


def _taps(x, y, h, w):
    x, y = x.clamp(0, w - 1), y.clamp(0, h - 1)
    fx, fy = x.floor(), y.floor()
    wx, wy = _weights(x - fx), _weights(y - fy)
    xi = [_mirror(fx.long() + k - 1, w) for k in range(4)]
    yi = [_mirror(fy.long() + k - 1, h) for k in range(4)]
    return wx, wy, xi, yi


def _sample(c, taps):
    wx, wy, xi, yi = taps
    w, flat, out = c.shape[1], c.reshape(-1), 0
    for j in range(4):
        out = out + wy[j] * sum(wx[k] * flat[yi[j] * w + xi[k]] for k in range(4))
    return out


def _gauss(sigma):
    r = int(4 * sigma + 0.5)
    t = torch.arange(-r, r + 1, dtype=F64)
    k = torch.exp(-0.5 * (t / sigma) ** 2)
    return (k / k.sum()).tolist()


def _corr(a, taps, axis, edge=True):
    r, n = len(taps) // 2, a.shape[axis]
    if edge:
        i = torch.arange(-r, n + r, device=a.device).clamp(0, n - 1)
        p = a.index_select(axis, i)
    else:
        p = torch.nn.functional.pad(a, (r, r, 0, 0) if axis == 1 else (0, 0, r, r))
    out = torch.zeros_like(a)
    for t, k in enumerate(taps):
        if k != 0.0:
            out += k * p.narrow(axis, t, n)
    return out


def _blur(a, sigma):
    k = _gauss(sigma)
    return _corr(_corr(a, k, 0), k, 1)


def _median(v):
    s = v.reshape(-1).sort().values
    n = s.numel()
    return s[n // 2] if n % 2 else (s[n // 2 - 1] + s[n // 2]) / 2


def _reflect(a):
    h, w = a.shape
    yi = _mirror(torch.arange(-PAD, h + PAD, device=a.device), h)
    xi = _mirror(torch.arange(-PAD, w + PAD, device=a.device), w)
    return a[yi][:, xi]


def _bank(h, w, c):
    fy = torch.fft.fftfreq(h, dtype=F64, device=DEV)[:, None] * 2 * math.pi
    fx = torch.fft.fftfreq(w, dtype=F64, device=DEV)[None, :] * 2 * math.pi
    s_hp = c.dc_cut * c.lam * max(c.scales) / (2 * math.pi)
    hp = 1 - torch.exp(-(fx * fx + fy * fy) * s_hp ** 2 / 2)
    out = []
    for s in c.scales:
        w0 = 2 * math.pi / (c.lam * s)
        b = c.bandwidth * w0
        for k in range(c.n_orient):
            th = math.pi * k / c.n_orient
            out.append(hp * torch.exp(-((fx - w0 * math.cos(th)) ** 2 + (fy - w0 * math.sin(th)) ** 2) / (2 * b * b)))
    return fx, fy, out


def _solve(M, b, n):
    """Cholesky of n x n systems given as planes: the solutions and the pixels where it exists."""
    M, ok = dict(M), None
    for j in range(n):
        d = M[j, j] - sum((M[j, k] ** 2 for k in range(j)), torch.zeros((), dtype=F64, device=DEV))
        good = torch.isfinite(d) & (d > 0)
        ok = good if ok is None else ok & good
        l = torch.sqrt(torch.where(good, d, torch.ones_like(d)))
        M[j, j] = l
        for i in range(j + 1, n):
            s = M[i, j]
            for k in range(j):
                s = s - M[i, k] * M[j, k]
            M[i, j] = s / l
    outs = []
    for r in b:
        r = list(r)
        for i in range(n):
            for k in range(i):
                r[i] = r[i] - M[i, k] * r[k]
            r[i] = r[i] / M[i, i]
        for i in reversed(range(n)):
            for k in range(i + 1, n):
                r[i] = r[i] - M[k, i] * r[k]
            r[i] = r[i] / M[i, i]
        outs.append(r)
    return outs, ok


def _local_solve(sums, ux, uy, c):
    kw = _gauss(c.sigma_w)
    r = len(kw) // 2
    taps = [[k * (t - r) ** p for t, k in enumerate(kw)] for p in range(5)]
    ycache, cache = {}, {}

    def mom(src, px, py):
        if (src, py) not in ycache:
            ycache[src, py] = _corr(sums[src], taps[py], 0)
        if (src, px, py) not in cache:
            cache[src, px, py] = _corr(ycache[src, py], taps[px], 1)
        return cache[src, px, py]

    pw = [(0, 0), (1, 0), (0, 1)] + ([(2, 0), (1, 1), (0, 2)] if c.shape_order == 2 else [])
    unk = [(q, *pw[i]) for i in range(len(pw)) for q in (0, 1)]
    n = len(unk)
    M = {(i, j): mom(unk[i][0] + unk[j][0], unk[i][1] + unk[j][1], unk[i][2] + unk[j][2])
         for i in range(n) for j in range(i + 1)}
    b = [mom(3 + q, px, py) for q, px, py in unk]
    e = M[0, 0] + M[1, 1]
    ok = (e > 1e-9 * _median(e) + 1e-30) & (M[0, 0] * M[1, 1] - M[1, 0] ** 2 > 1e-3 * e * e)
    ridge = 1e-12 * sum(M[i, i] for i in range(n)) / n
    A = {k: (v + ridge if k[0] == k[1] else v) for k, v in M.items()}
    (th,), good = _solve(A, [b], n)
    ok = ok & good
    for t in th:
        ok = ok & torch.isfinite(t)
    fit = sum(t * q for t, q in zip(th, b))
    resid = torch.sqrt((mom(5, 0, 0) - fit).clamp(min=0) / (mom(6, 0, 0) + 1e-30))
    zero = torch.zeros_like(e)
    slope = [torch.where(ok, t, zero) for t in th[2:6]]
    return (torch.where(ok, th[0], ux), torch.where(ok, th[1], uy), e,
            torch.where(ok, resid, torch.full_like(resid, math.pi)), slope)


def _confidence(energy, resid, c):
    tex = (energy / (0.25 * _median(energy) + 1e-30)).clamp(max=1.0)
    return tex * torch.exp(-(resid / c.phase_tol) ** 2)


def _column_nearest(src):
    """Per pixel the row of the nearest source pixel of its column (the smaller row on ties); far rows without one."""
    h = src.shape[0]
    far = 1 << 20
    r = torch.arange(h, device=src.device)[:, None]
    up = torch.where(src, r, torch.full_like(r, -far)).cummax(0).values
    dn = torch.where(src, r, torch.full_like(r, 2 * far)).flip(0).cummin(0).values.flip(0)
    return torch.where(dn - r < r - up, dn, up)


def _within(src, limit):
    """Pixels no further than limit from a source pixel."""
    h, w = src.shape
    v = _column_nearest(src) - torch.arange(h, device=src.device)[:, None]
    v2 = (v * v).clamp(max=1 << 30)
    best = torch.full_like(v2, 1 << 30)
    for dx in range(-int(limit), int(limit) + 1):
        lo, hi = max(0, dx), min(w, w + dx)
        if hi > lo:
            t = best[:, lo - dx:hi - dx]
            torch.minimum(t, v2[:, lo:hi] + dx * dx, out=t)
    return best.to(F64).sqrt() <= limit


def _prewarp(ux, uy, slope, low, c):
    if bool(low.any()):
        ok = ~_within(low, c.auto_edge_guard_px())
        if bool(ok.any()) and not bool(ok.all()):
            w = ok.shape[1]
            row = _column_nearest(ok)
            ys, xs = torch.nonzero(~ok, as_tuple=True)
            cols = torch.arange(w, device=ok.device)
            ux0, uy0, ux, uy = ux, uy, ux.clone(), uy.clone()
            for i in range(0, ys.numel(), 1 << 14):
                y, x = ys[i:i + (1 << 14)], xs[i:i + (1 << 14)]
                d2 = (row[y] - y[:, None]) ** 2 + (cols[None, :] - x[:, None]) ** 2
                col = (d2 * w + cols).argmin(1)  # the smallest distance, then the smallest column
                r = row[y, col]
                dx, dy = (x - col).to(F64), (y - r).to(F64)
                ux[y, x] = ux0[r, col] + slope[0][r, col] * dx + slope[2][r, col] * dy
                uy[y, x] = uy0[r, col] + slope[1][r, col] * dx + slope[3][r, col] * dy
    return _blur(ux, c.sigma_s), _blur(uy, c.sigma_s)


def _refine64(i1, i2, ux, uy, c):
    h, w = i1.shape
    fx, fy, bank = _bank(h + 2 * PAD, w + 2 * PAD, c)
    S = torch.fft.fft2(_reflect(i1))
    cut = lambda a: a[PAD:PAD + h, PAD:PAD + w]  # noqa: E731
    ref = []
    for G in bank:
        P = S * G
        r, rx, ry = (cut(torch.fft.ifft2(q)) for q in (P, 1j * P * fx, 1j * P * fy))
        a2 = r.abs() ** 2 + 1e-12
        ref.append((r, (r.conj() * rx).imag / a2, (r.conj() * ry).imag / a2, a2.sqrt()))
    c2 = _spline(i2)
    yy, xx = (a.to(F64) for a in torch.meshgrid(torch.arange(h, device=DEV), torch.arange(w, device=DEV), indexing="ij"))
    low = frozen = slope = energy = resid = None
    for it in range(c.outer_iters):
        if it == 0:
            sx, sy = _blur(ux, c.sigma_s), _blur(uy, c.sigma_s)
        else:
            k = c.prewarp_freeze_at
            low = frozen if k >= 1 and it > k else _confidence(energy, resid, c) < c.conf_min
            if k >= 1 and it == k:
                frozen = low
            sx, sy = _prewarp(ux, uy, slope, low, c)
        S2 = torch.fft.fft2(_reflect(_sample(c2, _taps(xx + sx, yy + sy, h, w))))
        csx, csy = _spline(sx), _spline(sy)
        resp = [_spline(torch.fft.ifft2(S2 * G)) for G in bank]
        for _ in range(c.inner_iters):
            tx, ty = xx + ux, yy + uy
            px, py = tx - sx, ty - sy
            for _ in range(2):
                t = _taps(px, py, h, w)
                px, py = tx - _sample(csx, t), ty - _sample(csy, t)
            t = _taps(px + PAD, py + PAD, h + 2 * PAD, w + 2 * PAD)
            a = [torch.zeros_like(ux) for _ in range(7)]
            for (r1, gx, gy, amp), R in zip(ref, resp):
                r2 = _sample(R, t)
                wk = amp * r2.abs()
                cc = (r1 * r2.conj()).angle() + gx * ux + gy * uy
                for i, v in enumerate((gx * gx, gx * gy, gy * gy, gx * cc, gy * cc, cc * cc)):
                    a[i] += wk * v
                a[6] += wk
            ux, uy, energy, resid, slope = _local_solve(a, ux, uy, c)
    conf = _confidence(energy, resid, c).clamp(0, 1)
    b = 4.0 * c.sigma_w if c.edge_guard_px() > 0 else 0.0
    tx, ty = xx + ux, yy + uy
    own = torch.minimum(torch.minimum(xx, yy), torch.minimum(w - 1 - xx, h - 1 - yy))
    rep = (own >= b) & (tx >= b) & (ty >= b) & (w - 1 - tx >= b) & (h - 1 - ty >= b)
    return ux, uy, torch.where(rep, conf, torch.zeros_like(conf)), resid


def _poc_grid(a, b, xs, ys, wy, wx, iu, iv):
    H, W = a.shape
    hann = lambda n: 0.5 - 0.5 * torch.cos(2 * math.pi * torch.arange(n, dtype=F64, device=DEV) / n)  # noqa: E731
    wnd = hann(wy)[:, None] * hann(wx)[None, :]
    fy = torch.fft.fftfreq(wy, dtype=F64, device=DEV).abs()[:, None]
    fx = torch.fft.fftfreq(wx, dtype=F64, device=DEV).abs()[None, :]
    lp = ((fy <= 0.25) & (fx <= 0.25)).to(F64)
    Y, X = torch.meshgrid(ys, xs, indexing="ij")
    y, x = Y.reshape(-1), X.reshape(-1)
    dx, dy = iu.reshape(-1).clone(), iv.reshape(-1).clone()
    pk, live = torch.zeros_like(dx), torch.ones_like(dx, dtype=torch.bool)
    ry, rx = torch.arange(wy, device=DEV)[None, :, None], torch.arange(wx, device=DEV)[None, None, :]

    def windows(img, y0, x0):
        v = img[y0[:, None, None] + ry, x0[:, None, None] + rx]
        return (v - v.mean((1, 2), keepdim=True)) * wnd

    for _ in range(3):
        ox, oy = dx.round().long(), dy.round().long()
        y0, x0 = y - wy // 2 + oy, x - wx // 2 + ox
        inside = (y0 >= 0) & (x0 >= 0) & (y0 + wy <= H) & (x0 + wx <= W)
        pk[live & ~inside] = 0.0
        live = live & inside
        for q in torch.nonzero(live).reshape(-1).split(4096):
            if not len(q):
                break
            A = torch.fft.fft2(windows(a, y[q] - wy // 2, x[q] - wx // 2))
            B = torch.fft.fft2(windows(b, y0[q], x0[q]))
            C = B * A.conj()
            r = torch.fft.fftshift(torch.fft.ifft2(C / (C.abs() + 1e-12) * lp).real, dim=(1, 2)) / lp.mean()
            best = r.reshape(len(q), -1).argmax(1)
            iy, ix = (best // wx).clamp(1, wy - 2), (best % wx).clamp(1, wx - 2)
            n = torch.arange(len(q), device=DEV)

            def parabola(m, c, p):
                den = m - 2 * c + p
                return torch.where(den == 0, torch.zeros_like(den), 0.5 * (m - p) / den)

            c0 = r[n, iy, ix]
            sx, sy = parabola(r[n, iy, ix - 1], c0, r[n, iy, ix + 1]), parabola(r[n, iy - 1, ix], c0, r[n, iy + 1, ix])
            sx, sy = ix - wx // 2 + sx, iy - wy // 2 + sy
            dx[q], dy[q], pk[q] = ox[q] + sx, oy[q] + sy, c0
            live[q] = ~((sx.abs() < 0.5) & (sy.abs() < 0.5))
    return dx.reshape(Y.shape), dy.reshape(Y.shape), pk.reshape(Y.shape)


def _neighbours(v, ok):
    p = torch.nn.functional.pad(torch.where(ok, v, torch.full_like(v, math.nan)), (1, 1, 1, 1), value=math.nan)
    h, w = v.shape
    return torch.stack([p[1 + i:1 + i + h, 1 + j:1 + j + w] for i in (-1, 0, 1) for j in (-1, 0, 1) if i or j])


def _nanmedian(v):
    n = torch.isfinite(v).sum(0)
    s = torch.where(torch.isnan(v), torch.full_like(v, math.inf), v).sort(0).values
    at = lambda k: s.gather(0, k.clamp(0, v.shape[0] - 1)[None])[0]  # noqa: E731
    return 0.5 * (at((n - 1) // 2) + at(n // 2)), n


def _clean(u, v, pk, c, iu, iv):
    valid = pk >= c.poc_peak_min
    out = valid.clone()
    for q in (u, v):
        nb = _neighbours(q, valid)
        med, n = _nanmedian(nb)
        res, _ = _nanmedian((nb - med).abs())
        out &= ~(valid & (n >= 3) & ((q - med).abs() / (res + 0.1) > c.median_thresh))
    if not bool(out.any()):
        return iu, iv
    for _ in range(100):
        if bool(out.all()):
            break
        mu, n = _nanmedian(_neighbours(u, out))
        mv, _ = _nanmedian(_neighbours(v, out))
        fill = ~out & (n > 0)
        u, v, out = torch.where(fill, mu, u), torch.where(fill, mv, v), out | fill
    return u, v


def _grid_sample(u, v, xs, ys, qx, qy):
    def frac(q, nodes):
        if len(nodes) == 1:
            return torch.zeros_like(q), torch.zeros_like(q, dtype=torch.long)
        f = ((q - nodes[0]) / float(nodes[1] - nodes[0])).clamp(0, len(nodes) - 1)
        i = f.floor().long().clamp(max=len(nodes) - 2)
        return f - i, i

    tx, x0 = frac(qx, xs)
    ty, y0 = frac(qy, ys)
    x1, y1 = (x0 + 1).clamp(max=len(xs) - 1), (y0 + 1).clamp(max=len(ys) - 1)
    tx, ty = tx[None, :], ty[:, None]
    return [(1 - ty) * ((1 - tx) * a[y0][:, x0] + tx * a[y0][:, x1]) + ty * ((1 - tx) * a[y1][:, x0] + tx * a[y1][:, x1])
            for a in (u, v)]


def _level_window(h, w, win):
    p2 = lambda n: 1 << (n.bit_length() - 1) if n >= 1 else 0  # noqa: E731
    lh, lw = p2(2 * h // 3), p2(2 * w // 3)
    if win <= lh and win <= lw:
        return win, win
    if h <= w:
        wy = min(win, lh)
        wx = min(lw, max(win, win * win // max(wy, 1)))
    else:
        wx = min(win, lw)
        wy = min(lh, max(win, win * win // max(wx, 1)))
    return (wy, wx) if min(wy, wx) >= 16 else None


def _coarse64(a, b, c, init):
    pyr = [(a, b)]
    L = max(0, math.ceil(math.log2(c.max_disp / (c.poc_win / 4))))
    while L > 0 and _level_window(a.shape[0] >> L, a.shape[1] >> L, c.poc_win) is None:
        L -= 1
    for _ in range(L):
        pyr.append(tuple(_blur(q, 1.0)[::2, ::2].contiguous() for q in pyr[-1]))
    got = None
    for lev in range(L, -1, -1):
        p, q = pyr[lev]
        h, w = p.shape
        wy, wx = (c.poc_win, c.poc_win) if lev == 0 else _level_window(h, w, c.poc_win)
        xs = torch.arange(wx // 2, w - wx // 2 + 1, c.grid_step, device=DEV)
        ys = torch.arange(wy // 2, h - wy // 2 + 1, c.grid_step, device=DEV)
        if got is not None:
            iu, iv = (2.0 * g for g in _grid_sample(*got, xs.to(F64) / 2, ys.to(F64) / 2))
        elif init is not None:
            iu, iv = (g[ys << lev][:, xs << lev] / (1 << lev) for g in init)
        else:
            iu = iv = torch.zeros((len(ys), len(xs)), dtype=F64, device=DEV)
        u, v, pk = _poc_grid(p, q, xs, ys, wy, wx, iu, iv)
        got = (*_clean(u, v, pk, c, iu, iv), xs, ys)
    return got


def _components(b, least):
    """Pixels of 4-connected components of at least `least` pixels (labels spread along whole runs until they rest)."""
    lab = torch.arange(1, b.numel() + 1, device=b.device).reshape(b.shape) * b

    def spread(l, m):
        run = (torch.nn.functional.pad(m, (1, 0))[:, :-1] != m).long()
        run[:, 0] = 1
        ids = run.reshape(-1).cumsum(0) - 1
        top = torch.zeros(int(ids[-1]) + 1, dtype=l.dtype, device=l.device).scatter_reduce_(0, ids, l.reshape(-1), "amax")
        return top[ids].reshape(l.shape) * m

    while True:
        new = spread(spread(lab, b).T.contiguous(), b.T.contiguous()).T.contiguous()
        if torch.equal(new, lab):
            break
        lab = new
    return b & (torch.bincount(lab.reshape(-1), minlength=b.numel() + 1)[lab] >= least)


def _strain64(ux, uy, win):
    ok = torch.isfinite(ux) & torch.isfinite(uy)
    zero = torch.zeros_like(ux)
    m, u0, v0 = ok.to(F64), torch.where(ok, ux, zero), torch.where(ok, uy, zero)
    hw = win // 2
    taps = [[float(t) ** p for t in range(-hw, hw + 1)] for p in range(5)]
    basis = [(0, 0), (1, 0), (0, 1), (2, 0), (1, 1), (0, 2)]
    mom = lambda a, px, py: _corr(_corr(a, taps[py], 0, False), taps[px], 1, False)  # noqa: E731
    seen = {}
    for p in basis:
        for q in basis:
            k = (p[0] + q[0], p[1] + q[1])
            if k not in seen:
                seen[k] = mom(m, *k)
    M = {(i, j): seen[basis[i][0] + basis[j][0], basis[i][1] + basis[j][1]] for i in range(6) for j in range(i + 1)}
    (a, b), good = _solve(M, [[mom(u0, *p) for p in basis], [mom(v0, *p) for p in basis]], 6)
    good = good & (seen[0, 0] >= 0.5 * win * win)
    nan = torch.full_like(ux, math.nan)
    g = [torch.where(good, t, nan) for t in (a[1], a[2], b[1], b[2])]
    dudx, dudy, dvdx, dvdy = g
    exx = dudx + 0.5 * (dudx ** 2 + dvdx ** 2)
    eyy = dvdy + 0.5 * (dudy ** 2 + dvdy ** 2)
    exy = 0.5 * (dudy + dvdx) + 0.5 * (dudx * dudy + dvdx * dvdy)
    return dict(exx=exx, eyy=eyy, exy=exy, gmax=2 * torch.sqrt(((exx - eyy) / 2) ** 2 + exy ** 2),
                vol=(1 + dudx) * (1 + dvdy) - dudy * dvdx - 1)


def _pair64(i1, i2, c, mask=None, init=None):
    up = lambda a: torch.from_numpy(np.asarray(a, np.float64)).to(DEV)  # noqa: E731
    a, b = up(i1), up(i2)
    h, w = a.shape
    ini = None if init is None else tuple(up(q) for q in init)
    u, v, xs, ys = _coarse64(a, b, c, ini)
    qx, qy = torch.arange(w, dtype=F64, device=DEV), torch.arange(h, dtype=F64, device=DEV)
    if ini is None:
        gx, gy = _grid_sample(u, v, xs, ys, qx, qy)
    else:
        cu, cv = (g - q[ys][:, xs] for g, q in zip((u, v), ini))
        gx, gy = (q + g for q, g in zip(ini, _grid_sample(cu, cv, xs, ys, qx, qy)))
    ux, uy, conf, _ = _refine64(a, b, gx, gy, c)
    low = conf < c.conf_min
    guard = c.edge_guard_px()
    src = _components(low, c.edge_guard_min_area_px())
    bad = low
    if mask is not None:
        out = ~torch.from_numpy(np.asarray(mask, bool)).to(DEV)
        bad, src = bad | out, src | out
    bd = torch.minimum(torch.minimum(qx, w - 1 - qx)[None, :], torch.minimum(qy, h - 1 - qy)[:, None])
    bad = bad | _within(src, guard) | (bd < guard)
    nan = torch.full_like(ux, math.nan)
    mx, my = torch.where(bad, nan, ux), torch.where(bad, nan, uy)
    o = dict(ux=mx, uy=my, conf=conf, raw_ux=ux, raw_uy=uy, valid=None)
    o.update(_strain64(mx, my, c.strain_win))
    return o


def _train64(d):
    """Loss, flow and gradient of the coarse network's training loss in float64."""
    conv = torch.nn.functional.conv2d
    layers = [(1, 16, 2, 1, 1), (16, 32, 2, 1, 1), (32, 32, 2, 1, 1), (32, 32, 1, 1, 0), (160, 64, 1, 1, 1),
              (64, 64, 1, 2, 1), (64, 32, 1, 4, 1), (32, 16, 1, 1, 0)]  # in, out, stride, dilation, ReLU
    up = lambda a: torch.from_numpy(np.asarray(a, np.float64)).to(DEV)  # noqa: E731
    params = up(d["params"]).requires_grad_()
    x = torch.cat([up(d["i1"]), up(d["i2"])])
    x = (x - x.mean((1, 2), keepdim=True)) / (x.var((1, 2), unbiased=False, keepdim=True).sqrt() + 1e-6)
    x, at, nb, R = x[:, None], 0, len(d["i1"]), 5
    for l, (ci, co, s, dil, relu) in enumerate(layers):
        kp = (9 * ci + 15) // 16 * 16
        wm = params[at:at + co * kp].reshape(co, kp)[:, :9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
        bias = params[at + co * kp:at + co * kp + co]
        at += co * kp + co
        x = conv(x, wm, bias, stride=s, padding=dil, dilation=dil)
        x = torch.relu(x) if relu else x
        if l == 3:
            f1, f2 = x[:nb], torch.nn.functional.pad(x[nb:], (R, R, R, R))
            h, w = f1.shape[2:]
            corr = torch.stack([(f1 * f2[:, :, i:i + h, j:j + w]).sum(1) / 32 for i in range(11) for j in range(11)], 1)
            x = torch.cat([corr, f1, torch.zeros(nb, 7, h, w, dtype=F64, device=DEV)], 1)
    p, k = torch.softmax(corr, 1), torch.arange(121, device=DEV)
    off = [(k % 11 - R).to(F64), (k // 11 - R).to(F64)]
    flow = torch.stack([8 * (p * o[None, :, None, None]).sum(1) + x[:, i] for i, o in enumerate(off)], -1)
    m = up(d["mask"])
    loss = (torch.sqrt(((flow - up(d["target"])) ** 2).sum(-1) + 0.01) * m).sum() / m.numel()
    loss.backward()
    return dict(loss=float(loss.detach()), flow=flow.detach(), grads=params.grad)


def exact(case, seed):
    d, c, kind = _inputs(case, seed), _config(case), case["kind"]
    if kind == "train":
        return _train64(d)
    with torch.no_grad():
        if kind == "pair":
            return _pair64(d["i1"], d["i2"], c, d["mask"], d["init"])
        if kind == "batch":
            return [_pair64(a, b, c) for a, b in d["items"]]
        if kind == "sequence":  # every leg from frame 0 (its confidence never falls to the reference's threshold)
            out, init = [], None
            for f in d["frames"][1:]:
                out.append(_pair64(d["frames"][0], f, c, init=init))
                init = (out[-1]["raw_ux"].float().cpu().numpy(), out[-1]["raw_uy"].float().cpu().numpy())
            return out
        up = lambda a: torch.from_numpy(np.asarray(a, np.float64)).to(DEV)  # noqa: E731
        ux, uy, conf, resid = _refine64(up(d["i1"]), up(d["i2"]), up(d["init"][0]), up(d["init"][1]), c)
        return dict(ux=ux, uy=uy, conf=conf, resid=resid, low=None)
