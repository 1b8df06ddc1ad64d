"""The work a user of doubleeye_b200 has it do, as timed cases through the public entry
points: dense pairs and batches on the device, dense pairs from host arrays, a frame
under the previous frame's map as a prior, keypoint matching, and the float64 edge-list
solver of the Python module.

Inputs are synthetic scenes made on the GPU from the seed: fractal texture over slanted
planes, the right view by a z-buffered warp with refilled occlusions, gain, offset and
sensor noise.  ``exact`` restates the arithmetic in plain torch: the census, cost,
filter and top-2 are integer arithmetic by definition, everything after them runs in
float64.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from doubleeye_b200 import dense, dense_masda, masda_stereo, sparse

DEV = "cuda"
# Image sizes and disparity counts of the uneven batch, the smallest to the largest.
SHAPES = [(320, 240, 64), (640, 480, 128), (848, 480, 128), (1280, 720, 256),
          (1920, 1080, 256)]


def listed():
    return [
        # One small pair resident on the GPU: the least a call does, launches and latency.
        dict(name="pair_320x240_d64", kind="dense", W=320, H=240, D=64, n=1, iters=8),
        # One live camera frame on the GPU, the plain path.
        dict(name="pair_848x480_d128", kind="dense", W=848, H=480, D=128, n=1, iters=8),
        # The benchmark's batch: 16 frames of as many cameras in one call.
        dict(name="batch16_848x480_d128", kind="dense", W=848, H=480, D=128, n=16, iters=8),
        # Large scenes offline, full disparity range.
        dict(name="batch4_1500x1000_d256", kind="dense", W=1500, H=1000, D=256, n=4, iters=12),
        # A mixed batch of every size in use, some of them odd and ragged.
        dict(name="uneven12", kind="uneven", n=12, mix=7, iters=8),
        # 9x7 census with the exact reverse match and all candidate planes written.
        dict(name="planes_848x480_d64_9x7", kind="dense", W=848, H=480, D=64, n=1, iters=10,
             hw=4, lrc=True, cand=True),
        # One pair from ordinary host arrays with its candidate planes: the command-line
        # tool's call, at the size the reference's article uses.
        dict(name="host_450x375_d60", kind="host", W=450, H=375, D=60, n=1, iters=12,
             cand=True, pinned=False),
        # A batch from and to page-locked host arrays: eight cameras end to end.
        dict(name="host8_848x480_d128", kind="host", W=848, H=480, D=128, n=8, iters=8,
             cand=False, pinned=True),
        # A camera stream: the previous frame's map, its holes filled, limits the search.
        dict(name="prior_848x480_d128", kind="prior", W=848, H=480, D=128, band=2, iters=8),
        # Keypoint matching of one frame, results read back.
        dict(name="sparse_848x480", kind="sparse", W=848, H=480, cell=32, per_cell=6),
        # The Python module's dense problem as an edge list, solved in float64.
        dict(name="edges_450x375_d60", kind="edges", W=450, H=375, D=60, iters=12),
        # The Python module's keypoint problem as a score matrix, solved in float64.
        dict(name="points_1000", kind="points", m=1000, n=1000, W=848, H=480, iters=30),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same kinds and ranges; odd sizes as they come."""
    kind = rng.choice(["dense", "dense", "dense", "uneven", "host", "host", "prior", "sparse",
                       "edges", "points"])
    if kind == "uneven":
        c = dict(kind=kind, n=rng.randint(3, 12), mix=rng.randint(100, 10 ** 6), iters=8)
        while sum(W * H * D for W, H, D in _shapes(c)) > 2.1e9:
            c["n"] -= 1
        return c
    if kind == "sparse":
        W = _log(rng, 320, 1280)
        return dict(kind=kind, W=W, H=int(W * rng.uniform(0.5, 0.75)), cell=rng.choice([24, 32, 40]),
                    per_cell=rng.randint(3, 6))
    if kind == "points":
        return dict(kind=kind, m=_log(rng, 60, 1500), n=_log(rng, 60, 1500), W=848, H=480,
                    iters=rng.randint(10, 30))
    W = _log(rng, 200, 450) if kind == "edges" else _log(rng, 300, 1920)
    H = int(W * rng.uniform(0.5, 0.75))
    if kind == "edges":
        return dict(kind=kind, W=W, H=H, D=rng.randint(16, 60), iters=rng.randint(4, 12))
    D = min(rng.randint(20, 256), W // 2)
    c = dict(kind=kind, W=W, H=H, D=D, iters=rng.choice([0, 8, 8, 12]))
    if kind == "prior":
        return dict(c, band=rng.randint(1, 4), D=min(D, 192), iters=8)
    most = 16 if kind == "dense" else 8
    n = max(1, min(_log(rng, 1, most), int(1.0e9 / (W * H * D))))
    if kind == "host":
        return dict(c, n=n, cand=n == 1, pinned=rng.random() < 0.5)
    if n == 1:
        c.update(hw=rng.choice([3, 3, 4]), lrc=rng.random() < 0.3, cand=rng.random() < 0.3)
    return dict(c, n=n)


def _shapes(case):
    """(W, H, D) of each pair of a dense case."""
    if case["kind"] != "uneven":
        return [(case["W"], case["H"], case["D"])] * case.get("n", 1)
    r, out = random.Random(case["mix"]), []
    for _ in range(case["n"]):
        W, H, D = r.choice(SHAPES)
        odd = r.random() < 0.5
        out.append((W - odd * r.randint(1, 40), H - odd * r.randint(1, 30),
                    D - odd * r.randint(0, 24)))
    return out


# ---- inputs ---------------------------------------------------------------------------

def _texture(H, W, g):
    img = torch.zeros((H, W), device=DEV)
    scale, amp = 1.5, 1.0
    for _ in range(4):
        h, w = int(H / scale) + 3, int(W / scale) + 3
        coarse = torch.randn((1, 1, h, w), generator=g, device=DEV)
        up = torch.nn.functional.interpolate(coarse, size=(int(h * scale) + 1, int(w * scale) + 1),
                                             mode="bilinear", align_corners=True)
        img += amp * up[0, 0, :H, :W]
        scale *= 2.7
        amp *= 0.6
    return 110.0 + 40.0 * (img - img.mean()) / img.std()


def _scene(W, H, D, g, rigid=False):
    """(left, right, disparity) of one scene: 12 slanted planes, or fronto-parallel ones at
    whole disparities (``rigid``)."""
    tex = _texture(H, W, g)
    u = lambda n, lo, hi: lo + (hi - lo) * torch.rand(n, generator=g, device=DEV)  # noqa: E731
    ys = torch.arange(H, device=DEV, dtype=torch.float32)[:, None]
    xs = torch.arange(W, device=DEV, dtype=torch.float32)[None, :]
    px, py = u(12, 0, W), u(12, 0, H)
    d0 = u(12, 0, D - 1)
    gr = u(24, -0.15, 0.15) * (0.0 if rigid else 1.0)
    lab = ((xs[None] - px[:, None, None]) ** 2 + (ys[None] - py[:, None, None]) ** 2).argmin(0)
    disp = d0[lab] + gr[:12][lab] * (xs - px[lab]) + gr[12:][lab] * (ys - py[lab])
    disp = disp.clamp(0, D - 1)
    if rigid:
        disp = disp.round()
    # z-buffered forward warp: the nearest surface wins a right pixel
    xi = torch.arange(W, device=DEV).expand(H, W)
    xr = (xi - disp).round().long()
    ok = (xr >= 0) & (xr < W)
    tgt = (torch.arange(H, device=DEV)[:, None] * W + xr)[ok]
    key = ((disp * 256).long() * 8192 + xi)[ok]
    best = torch.full((H * W,), -1, dtype=torch.int64, device=DEV)
    best.scatter_reduce_(0, tgt, key, "amax")
    src = (best % 8192).reshape(H, W).clamp(0, W - 1)
    right = torch.gather(tex, 1, src)
    right = torch.where(best.reshape(H, W) >= 0, right, _texture(H, W, g))
    gain, off = u(1, 0.95, 1.05), u(1, -5.0, 5.0)
    noise = lambda: 2.0 * torch.randn((H, W), generator=g, device=DEV)  # noqa: E731
    q = lambda t: t.round().clamp(0, 255).to(torch.uint8).contiguous()  # noqa: E731
    return q(tex + noise()), q(right * gain + off + noise()), disp


def _scenes(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return [_scene(W, H, D, g) for W, H, D in _shapes(case)]


def _cfg(case, D):
    return dense.Cfg(dmin=1, dmax=D, iters=case["iters"], lrc=int(case.get("lrc", False)),
                     census_hw=case.get("hw", 3), census_hh=3)


def _prior_map(case, seed):
    """The previous frame's map: a disparity to the nearest quarter pixel with holes."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    L, R, disp = _scene(case["W"], case["H"], case["D"], g)
    rough = 0.4 * torch.randn(disp.shape, generator=g, device=DEV)
    prev = (torch.round(4 * (disp + rough)) / 4).clamp(1, case["D"])
    hole = _texture(case["H"], case["W"], g) > 145.0
    prev[hole] = float("nan")
    return L, R, prev


def _points(case, seed):
    """Keypoints of two views on a quarter-pixel grid with census descriptors: most left
    points have a right one with some descriptor bits flipped, the rest are clutter."""
    r = np.random.default_rng(int(seed))
    m, n = case["m"], case["n"]
    pl = np.stack([r.uniform(70, case["W"], m), r.uniform(4, case["H"] - 4, m)], 1)
    dl = r.integers(0, 1 << 48, m, dtype=np.uint64)
    pr = np.stack([r.uniform(4, case["W"], n), r.uniform(4, case["H"] - 4, n)], 1)
    dr = r.integers(0, 1 << 48, n, dtype=np.uint64)
    k = int(0.7 * min(m, n))
    pr[:k] = pl[:k] - np.stack([r.uniform(1, 60, k), r.normal(0, 0.4, k)], 1)
    flips = np.zeros(k, np.uint64)
    for _ in range(6):
        flips |= np.uint64(1) << r.integers(0, 48, k, dtype=np.uint64)
    dr[:k] = dl[:k] ^ flips
    q = lambda p: (np.round(4 * p) / 4).astype(np.float32)  # noqa: E731
    o = r.permutation(n)
    return q(pl), dl, q(pr)[o], dr[o]


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("dense", "uneven"):
        s["pairs"] = [(L, R, D) for (L, R, _), (_, _, D) in zip(_scenes(case, seed), _shapes(case))]
        s["matcher"] = dense.DenseMatcher(_cfg(case, max(p[2] for p in s["pairs"])))
    elif kind == "host":
        def host(t):
            a = dense.pinned_empty(t.shape, np.uint8) if case["pinned"] else np.empty(t.shape, np.uint8)
            a[:] = t.cpu().numpy()
            return a
        s["pairs"] = [(host(L), host(R)) for L, R, _ in _scenes(case, seed)]
        s["cfg"] = _cfg(case, case["D"])
        if case["pinned"]:
            s["out"] = dense.new_results([(case["H"], case["W"])] * case["n"], case["cand"])
    elif kind == "prior":
        L, R, prev = _prior_map(case, seed)
        s.update(L=L.cpu().numpy(), R=R.cpu().numpy(), prev=prev.cpu().numpy(),
                 cfg=_cfg(case, case["D"]))
    elif kind == "sparse":
        g = torch.Generator(device=DEV)
        g.manual_seed(int(seed))
        s["L"], s["R"], _ = _scene(case["W"], case["H"], 61, g, rigid=True)
        s["matcher"] = sparse.SparseMatcher(
            det=sparse.DetCfg(cell=case["cell"], per_cell=case["per_cell"]),
            cfg=sparse.MatchCfg(max_disparity=64.0))
    elif kind == "edges":
        L, R, _ = _scenes(case, seed)[0]
        s.update(L=L, R=R)
    else:
        s["points"] = _points(case, seed)
    return s


# ---- one pass -------------------------------------------------------------------------

def _partner(assign, m):
    """A left -> right assignment as each left point's partner, -1 where it has none."""
    a = np.full(m, -1, np.int64)
    a[np.fromiter(assign.keys(), np.int64, len(assign))] = np.fromiter(
        assign.values(), np.int64, len(assign))
    return a


def _table(a, n):
    """The first n rows of an array, zeros after its end."""
    t = np.zeros((n,) + a.shape[1:], a.dtype)
    t[:len(a)] = a
    return t


def _slots(case):
    """The most keypoints that the detector's grid gives."""
    return -(-case["W"] // case["cell"]) * -(-case["H"] // case["cell"]) * case["per_cell"]


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("dense", "uneven"):
        if case["n"] == 1:
            return s["matcher"].match(*s["pairs"][0], cand=case.get("cand", False))
        return s["matcher"].match_batch(s["pairs"], cand=case.get("cand", False))
    if kind == "host":
        if case["n"] == 1 and not case["pinned"]:
            res = [dense.run_dense(*s["pairs"][0], s["cfg"], want_cand=case["cand"])]
        else:
            res = dense.run_dense_batch(s["pairs"], s["cfg"], want_cand=case["cand"],
                                        out=s.get("out"))
        return [dict(disp=r.disp, margin=r.margin, conf=r.conf, cand=r.cand) for r in res]
    if kind == "prior":
        fill = dense.fill_holes(s["prev"])
        r = dense.run_dense_prior(s["L"], s["R"], fill, s["cfg"], band=case["band"])
        return dict(fill=fill, disp=r.disp, margin=r.margin, conf=r.conf, cand=r.cand)
    if kind == "sparse":
        h = s["matcher"].to_host(s["matcher"].match_pair(s["L"], s["R"]))
        m = h["matches"]
        got = dict(kl=h["kl"], kr=h["kr"], dl=h["dl"].view(np.int64), dr=h["dr"].view(np.int64),
                   **{f: m[f] for f in m.dtype.names})
        return dict({k: _table(a, _slots(case)) for k, a in got.items()}, matches=len(m),
                    stats=h["stats"])
    if kind == "edges":
        ei, ej, se, mn = dense_masda.dense_problem(s["L"], s["R"], 1, case["D"], device=True)
        got, hist = masda_stereo.masda_sparse(ei, ej, se, mn, mn, iters=case["iters"], eps=0.0)
        return dict(ei=ei, ej=ej, se=se, hist=hist, right=_partner(got, mn))
    S = masda_stereo.build_problem(*s["points"])
    got, hist = masda_stereo.masda(S, iters=case["iters"], eps=0.0)
    return dict(S=S, hist=hist, right=_partner(got, case["m"]))


# ---- what a pass cannot do without ----------------------------------------------------

def work(case):
    """Inputs once, outputs once; integer or float operations of the definition: 37 per
    disparity evaluation (score 11, four filter steps 5 each, packing and top-2 6)."""
    kind = case["kind"]
    if kind in ("dense", "uneven", "host", "prior"):
        px = sum(W * H for W, H, _ in _shapes(case))
        ev = sum(W * H * D for W, H, D in _shapes(case))
        out = 9 + (24 if case.get("cand") or kind == "prior" else 0)
        if kind == "prior":      # a map in, a filled map out; planes of the band only
            return dict(bytes=px * (2 + 8 + out), flops=37.0 * px * (2 * case["band"] + 1))
        return dict(bytes=px * (2 + out), flops=37.0 * ev)
    if kind == "sparse":         # both images; corner test and structure tensor per pixel
        px = case["W"] * case["H"]
        kp = 2 * (px / case["cell"] ** 2) * case["per_cell"]
        return dict(bytes=2 * px + 24 * kp + 28 * kp / 2, flops=2 * px * (32 + 9 * 20))
    if kind == "edges":          # edge list out, node assignment out; 2 sweeps of ~10 each
        W, H, D = case["W"], case["H"], case["D"]
        E = sum((H - 6) * (W - 6 - d) for d in range(1, D + 1))
        return dict(bytes=2 * W * H + 20 * E + 16 * W * H, flops=E * (4.0 + 20 * case["iters"]))
    mn = case["m"] * case["n"]
    return dict(bytes=4.0 * mn + 16 * (case["m"] + case["n"]), flops=8.0 * mn)


# ---- the same in plain torch, float64 after the integer stages ------------------------

NEG = float(np.float32(-1e30))


def _window(img, dy, dx):
    """img shifted so that element (y, x) is img[y + dy, x + dx] (edges wrap, unused)."""
    return torch.roll(img, (-dy, -dx), (0, 1))


def _census(img, hw, hh):
    H, W = img.shape
    v = img.to(torch.int64)
    w = torch.zeros_like(v)
    bit = 0
    for dy in range(-hh, hh + 1):
        for dx in range(-hw, hw + 1):
            if dx or dy:
                w |= (_window(v, dy, dx) < v).to(torch.int64) << bit
                bit += 1
    out = torch.zeros_like(w)
    out[hh:H - hh, hw:W - hw] = w[hh:H - hh, hw:W - hw]
    return out


def _popcount(v):
    t = torch.tensor([bin(i).count("1") for i in range(1 << 16)], device=DEV)
    return sum(t[(v >> s) & 0xFFFF] for s in (0, 16, 32, 48))


def _coefficients(img, cfg):
    """Q15 filter coefficients of |difference to the left / upper neighbour|."""
    f = np.float32
    kk = f(-np.sqrt(f(2.0)) / f(cfg.sigma_s))
    rs = f(f(cfg.sigma_s) / f(cfg.sigma_r))
    e = [math.exp(float(f(kk * f(f(1) + f(rs * f(f(d) / f(255))))))) for d in range(256)]
    lut = torch.tensor([int(min(32767.0, float(f(f(f(v) * f(32768)) + f(0.5))))) for v in e],
                       dtype=torch.int32, device=DEV)
    v = img.to(torch.int64)
    ax, ay = torch.zeros_like(v), torch.zeros_like(v)
    ax[:, 1:] = (v[:, 1:] - v[:, :-1]).abs()
    ay[1:] = (v[1:] - v[:-1]).abs()
    return lut[ax], lut[ay]


def _step(c, f, a):
    return c + ((a * (f - c) + (1 << 14)) >> 15)


def _filtered(L, R, cfg, D, rect=None):
    """The filtered cost volume [H][W][D] (int32).  ``rect``: per plane ylo, yhi, xlo, xhi,
    the filter's extent under a prior."""
    H, W = L.shape
    hw, hh, dmin = cfg.census_hw, cfg.census_hh, cfg.dmin
    cl, cr = _census(L, hw, hh), _census(R, hw, hh)
    ax, ay = _coefficients(L, cfg)
    bits = (2 * hw + 1) * (2 * hh + 1) - 1
    half = bits // 2
    q = lambda a, b: int(a / b)  # noqa: E731  C division
    tbl = torch.tensor([q((half - h) * 16384, half) for h in range(bits + 1)], device=DEV)
    wq, T = int(np.float32(cfg.ad) * np.float32(1024)), max(1, cfg.ad_trunc)
    adt = torch.tensor([16384 - q(2 * 16384 * min(v, T), T) for v in range(256)], device=DEV)
    V = torch.zeros((W, H, D), dtype=torch.int32, device=DEV)
    li, ri = L.to(torch.int64), R.to(torch.int64)
    for k in range(D):
        d = dmin + k
        if W - hw <= hw + d:
            continue
        a, b = slice(hw + d, W - hw), slice(hw, W - hw - d)
        h = _popcount(cl[hh:H - hh, a] ^ cr[hh:H - hh, b])
        m = (li[hh:H - hh, a] - ri[hh:H - hh, b]).abs()
        V[a, hh:H - hh, k] = ((tbl[h] * (1024 - wq) + adt[m] * wq) >> 10).to(torch.int32).T

    def sweep(vol, coef, lo, hi):
        """Forward then backward along dimension 0; lo, hi: each plane's extent there."""
        n = vol.shape[0]
        f = torch.zeros_like(vol[0])
        for i in range(n):
            g = _step(vol[i], f, coef[i][:, None])
            if lo is not None:
                g = torch.where(i == lo, vol[i], g)
                g = torch.where((i >= lo) & (i < hi), g, f)
            f = g
            vol[i] = f if lo is None else torch.where((i >= lo) & (i < hi), f, vol[i])
        for i in range(n - 2, -1, -1):
            g = _step(vol[i], f, coef[i + 1][:, None])
            if lo is not None:
                g = torch.where(i == hi - 1, vol[i], g)
                g = torch.where((i >= lo) & (i < hi), g, f)
            f = g
            vol[i] = f if lo is None else torch.where((i >= lo) & (i < hi), f, vol[i])

    r = rect
    sweep(V, ax.T.contiguous(), r and r[2], r and r[3])
    V = V.permute(1, 0, 2).contiguous()
    if r is None:
        V[:hh] = 0
        V[H - hh:] = 0
    sweep(V, ay, r and r[0], r and r[1])
    return V


def _top2(V, cfg, D, allowed=None):
    """Packed top-2 keys and the winner's neighbour costs per pixel, and the best key per
    right pixel (all int64; 0 = none)."""
    H, W, _ = V.shape
    hw, hh, dmin = cfg.census_hw, cfg.census_hh, cfg.dmin
    k0, k1, nm, np_, rk = (torch.zeros((H, W), dtype=torch.int64, device=DEV) for _ in range(5))
    k = torch.arange(D, device=DEV)
    x = torch.arange(W, device=DEV)[:, None]
    ok = (x - hw - dmin >= k) & (x < W - hw)
    kmax = torch.clamp(x[:, 0] - hw - dmin, max=D - 1)
    xr = (x - dmin - k).clamp(min=0).reshape(-1)
    for y in range(hh, H - hh):
        v = V[y].to(torch.int64)
        good = ok if allowed is None else ok & allowed[y]
        key = torch.where(good, ((v + 32768) << 8) | (255 - k), 0)
        k0[y] = key.amax(1)
        k1[y] = torch.where(key == k0[y][:, None], 0, key).amax(1)
        rk[y].scatter_reduce_(0, xr, key.reshape(-1), "amax")
        kw = 255 - (k0[y] & 255)
        lo = torch.gather(v, 1, (kw - 1).clamp(0, D - 1)[:, None])[:, 0]
        hi = torch.gather(v, 1, (kw + 1).clamp(0, D - 1)[:, None])[:, 0]
        nm[y] = torch.where((k0[y] > 0) & (kw >= 1), lo, -32768)
        np_[y] = torch.where((k0[y] > 0) & (kw + 1 <= kmax), hi, -32768)
    return k0, k1, nm, np_, rk


def _seg_excluding(v, seg, n, neg):
    """Max of the other elements of an element's segment (``neg`` where it is alone)."""
    m1 = torch.full((n,), neg, dtype=v.dtype, device=v.device).scatter_reduce_(0, seg, v, "amax")
    top = v >= m1[seg]
    cnt = torch.zeros(n, dtype=torch.int64, device=v.device).scatter_add_(0, seg, top.long())
    m2 = torch.full((n,), neg, dtype=v.dtype, device=v.device)
    m2.scatter_reduce_(0, seg, torch.where(top, torch.full_like(v, neg), v), "amax")
    return torch.where(top & (cnt[seg] < 2), m2[seg], m1[seg])


def _solved(k0, k1, nm, np_, rk, cfg, subpixel=True):
    """disp, margin and the six candidate planes of every row (float64)."""
    H, W = k0.shape
    dmin = cfg.dmin
    lam, gam, damp = (float(np.float32(v)) for v in (cfg.lambda_, cfg.gamma, cfg.damping))
    keep = 1.0 - damp
    key = torch.stack([k0, k1], -1)
    has = key > 0
    cs = torch.where(has, ((key >> 8) - 32768).double() / 16384.0, NEG)
    cd = 255 - (key & 255)
    x = torch.arange(W, device=DEV)[None, :, None]
    row = torch.arange(H, device=DEV)[:, None, None]
    seg_all = row * W + (x - dmin - cd)
    it = has.reshape(-1).nonzero()[:, 0]                   # items: 2 * pixel + j
    seg, c = seg_all.reshape(-1)[it], cs.reshape(-1)[it]
    two = has[..., 1].reshape(-1)[it // 2]
    inv = torch.full((2 * H * W,), 0, dtype=torch.int64, device=DEV)
    inv[it] = torch.arange(len(it), device=DEV)
    other = inv[it ^ 1]
    alt = torch.where(has[..., 1], cs[..., 1].clamp(min=lam), lam)
    margin = torch.where(has[..., 0], cs[..., 0] - alt, 0.0)
    beta, rho = torch.zeros_like(c), torch.zeros_like(c)
    for _ in range(cfg.iters):
        b = torch.where(two, beta[other].clamp(min=lam), lam)
        rho = keep * (c - b) + damp * rho
        ex = _seg_excluding(rho, seg, H * W, NEG)
        beta = keep * (c - ex.clamp(min=gam)) + damp * beta
    bel = beta + rho - c if cfg.iters > 0 else c
    full = torch.full((2 * H * W,), NEG, dtype=torch.float64, device=DEV)
    full[it] = torch.where(c > lam, bel, NEG)
    full = full.reshape(H * W, 2)
    bj = (full[:, 1] > full[:, 0]).long()
    best = full.gather(1, bj[:, None])[:, 0]
    pix = (best > NEG).nonzero()[:, 0]
    cl = seg_all.reshape(-1, 2).gather(1, bj[:, None])[:, 0][pix]
    top = torch.full((H * W,), NEG, dtype=torch.float64, device=DEV)
    top.scatter_reduce_(0, cl, best[pix], "amax")
    first = torch.full((H * W,), H * W, dtype=torch.int64, device=DEV)
    lead = best[pix] >= top[cl]
    first.scatter_reduce_(0, cl[lead], pix[lead], "amin")
    win = torch.zeros(H * W, dtype=torch.bool, device=DEV)
    win[first[first < H * W]] = True
    win, bj = win.reshape(H, W), bj.reshape(H, W)
    d = (dmin + cd.gather(2, bj[..., None])[..., 0]).double()
    if subpixel:
        cm, cp, c0 = nm.double() / 16384.0, np_.double() / 16384.0, cs[..., 0]
        den = c0 - torch.minimum(cm, cp)
        fit = (nm != -32768) & (np_ != -32768) & (den > 1e-6) & (bj == 0)
        off = (0.5 * (cp - cm) / den.clamp(min=1e-9)).clamp(-0.5, 0.5)
        d = d + torch.where(fit, off, 0.0)
    nan = torch.full_like(d, float("nan"))
    disp = torch.where(win, d, nan)
    # reverse match: the best candidate that names a right pixel, the first on ties
    bc = torch.full((H * W,), NEG, dtype=torch.float64, device=DEV)
    bc.scatter_reduce_(0, seg, c, "amax")
    fi = torch.full((H * W,), 2 * H * W, dtype=torch.int64, device=DEV)
    lead = c >= bc[seg]
    fi.scatter_reduce_(0, seg[lead], it[lead], "amin")
    rev = torch.where(fi < 2 * H * W, cd.reshape(-1)[fi.clamp(max=2 * H * W - 1)], -1).reshape(H, W)
    xr = x[..., 0] - torch.floor(torch.where(win, d, 0.0) + 0.5).long()
    ok = win & (xr >= 0) & (xr < W)
    rv = torch.gather(rev, 1, xr.clamp(0, W - 1))
    lrc2 = torch.where(ok & (rv >= 0), (d - (dmin + rv)).abs(), nan)
    lrc = torch.full_like(d, NEG)
    if cfg.lrc:
        kr = torch.gather(rk, 1, xr.clamp(0, W - 1))
        lrc = torch.where(ok & (kr > 0), (d - (dmin + 255 - (kr & 255))).abs(), nan)
    cand = torch.stack([cs[..., 0], cs[..., 1],
                        torch.where(has[..., 0], (dmin + cd[..., 0]).double(), NEG),
                        torch.where(has[..., 1], (dmin + cd[..., 1]).double(), NEG), lrc, lrc2])
    return disp, margin, cand


def _dense_exact(L, R, cfg, D, cand):
    keys = _top2(_filtered(L, R, cfg, D), cfg, D)
    disp, margin, planes = _solved(*keys, cfg)
    return dict(disp=disp.cpu().numpy(), margin=margin.cpu().numpy(), conf=None,
                cand=planes.cpu().numpy() if cand else None)


def _fill_exact(prev):
    v = prev.double()
    for _ in range(128):
        n = torch.stack([torch.roll(v, 1, 1), torch.roll(v, -1, 1), torch.roll(v, 1, 0),
                         torch.roll(v, -1, 0)])
        fin = torch.isfinite(n)
        cnt = fin.sum(0)
        mean = torch.where(fin, n, 0.0).sum(0) / cnt.clamp(min=1)
        grow = ~torch.isfinite(v) & (cnt > 0)
        if not grow.any():
            break
        v = torch.where(grow, mean, v)
    return torch.where(torch.isfinite(v), v, 0.0)


def _prior_exact(case, seed):
    L, R, prev = _prior_map(case, seed)
    H, W, D, band = case["H"], case["W"], case["D"], case["band"]
    cfg = _cfg(case, D)
    fill = _fill_exact(prev)
    dc = torch.floor(fill.float().double() + 0.5)[..., None]
    d = 1 + torch.arange(D, device=DEV)
    want = (d >= dc - band) & (d <= dc + band)                        # [H][W][D]
    rows, cols = want.any(1), want.any(0)
    ar = lambda n: torch.arange(n, device=DEV)[:, None]  # noqa: E731
    lo = lambda m: torch.where(m, ar(len(m)), len(m)).amin(0)  # noqa: E731
    hi = lambda m: torch.where(m, ar(len(m)), -1).amax(0)  # noqa: E731
    ylo, yhi = (lo(rows) - 8).clamp(min=3), (hi(rows) + 9).clamp(max=H - 3)
    xlo = torch.maximum(lo(cols) - 8, 3 + d)
    xhi = (hi(cols) + 9).clamp(max=W - 3)
    none = (yhi <= ylo) | (xhi - xlo < 2) | (hi(rows) < 0)
    yhi, xhi = torch.where(none, ylo, yhi), torch.where(none, xlo, xhi)
    x = torch.arange(W, device=DEV)[None, :, None]
    x0 = torch.where(want, x, W).amin(1, keepdim=True)                # row intervals
    x1 = torch.where(want, x, -1).amax(1, keepdim=True)
    y = torch.arange(H, device=DEV)[:, None, None]
    inside = (x >= x0) & (x <= x1) & (x >= xlo) & (x < xhi) & (y >= ylo) & (y < yhi) & ~none
    V = _filtered(L, R, cfg, D, (ylo, yhi, xlo, xhi))
    keys = _top2(V, cfg, D, inside)
    disp, margin, planes = _solved(*keys, cfg, subpixel=False)
    return dict(fill=fill.cpu().numpy(), disp=disp.cpu().numpy(), margin=margin.cpu().numpy(),
                conf=None, cand=planes.cpu().numpy())


def _masda64(ei, ej, se, m, n, iters, lam=-0.1, gam=-0.1, damp=0.4):
    beta, rho, hist = torch.zeros_like(se), torch.zeros_like(se), []
    inf = float("-inf")
    for _ in range(iters):
        r = (1 - damp) * (se - _seg_excluding(beta, ei, m, inf).clamp(min=lam)) + damp * rho
        dr = (r - rho).abs().max()
        rho = r
        b = (1 - damp) * (se - _seg_excluding(rho, ej, n, inf).clamp(min=gam)) + damp * beta
        hist.append(max(float(dr), float((b - beta).abs().max())))
        beta = b
    return np.array(hist)


def _edges_exact(case, seed):
    L, R, _ = _scenes(case, seed)[0]
    H, W, D = case["H"], case["W"], case["D"]
    cl, cr = _census(L, 3, 3), _census(R, 3, 3)
    grid = (torch.arange(H, device=DEV)[:, None] * W + torch.arange(W, device=DEV))[3:H - 3]
    ei, ej, se = [], [], []
    for d in range(1, D + 1):
        h = _popcount(cl[3:H - 3, 3 + d:W - 3] ^ cr[3:H - 3, 3:W - 3 - d])
        p = grid[:, 3 + d:W - 3].reshape(-1)
        ei.append(p)
        ej.append(p - d)
        se.append((24.0 - h.double().reshape(-1)) / 24.0)
    ei, ej, se = torch.cat(ei), torch.cat(ej), torch.cat(se)
    hist = _masda64(ei, ej, se.float().double(), H * W, H * W, case["iters"])
    return dict(ei=None, ej=None, se=se, hist=hist, right=None)


def _points_exact(case, seed):
    pl, dl, pr, dr = _points(case, seed)
    h = _popcount(torch.tensor((dl[:, None] ^ dr[None]).view(np.int64), device=DEV)).cpu().numpy()
    dy = pl[:, None, 1].astype(np.float64) - pr[None, :, 1]
    dx = pl[:, None, 0].astype(np.float64) - pr[None, :, 0]
    S = np.where((np.abs(dy) <= 1.5) & (dx >= 1) & (dx <= 60), (24.0 - h) / 24.0 - dy ** 2, -np.inf)
    i, j = np.nonzero(np.isfinite(S))
    t = lambda a: torch.tensor(a, device=DEV)  # noqa: E731
    hist = _masda64(t(i), t(j), t(S[i, j].astype(np.float32).astype(np.float64)), case["m"],
                    case["n"], case["iters"])
    return dict(S=S, hist=hist, right=None)


def _response(img, gw):
    """The smaller eigenvalue of the structure tensor over a gw x gw window (float64)."""
    v = img.double()
    w = lambda dy, dx: _window(v, dy, dx)  # noqa: E731
    gx = (w(-1, 1) - w(-1, -1) + 2 * (w(0, 1) - w(0, -1)) + w(1, 1) - w(1, -1)) / 8
    gy = (w(1, -1) - w(-1, -1) + 2 * (w(1, 0) - w(-1, 0)) + w(1, 1) - w(-1, 1)) / 8
    r = max(1, gw // 2)
    n = (2 * r + 1) ** 2
    s = [sum(_window(t, dy, dx) for dy in range(-r, r + 1) for dx in range(-r, r + 1)) / n
         for t in (gx * gx, gy * gy, gx * gy)]
    return 0.5 * (s[0] + s[1]) - torch.sqrt(0.25 * (s[0] - s[1]) ** 2 + s[2] ** 2)


def _keypoints_exact(img, det):
    """FAST corners, strongest first in their squares, the best of each cell (float64)."""
    H, W = img.shape
    v = img.to(torch.int64)
    ring = [(0, -3), (1, -3), (2, -2), (3, -1), (3, 0), (3, 1), (2, 2), (1, 3), (0, 3), (-1, 3),
            (-2, 2), (-3, 1), (-3, 0), (-3, -1), (-2, -2), (-1, -3)]
    p = torch.stack([_window(v, dy, dx) for dx, dy in ring])
    corner = torch.zeros((H, W), dtype=torch.bool, device=DEV)
    for side in (p > v + det.fast_threshold, p < v - det.fast_threshold):
        run9 = torch.stack([torch.stack([side[(a + b) % 16] for b in range(9)]).all(0)
                            for a in range(16)]).any(0)
        corner |= run9 & (side[::4].sum(0) >= 2)
    b = max(det.border, 5)
    inner = torch.zeros_like(corner)
    inner[b:H - b, b:W - b] = True
    resp = _response(img, det.grad_window)
    c = corner & inner & (resp >= det.min_response)
    idx = c.reshape(-1).nonzero()[:, 0]
    rank = torch.zeros(H * W, dtype=torch.float64, device=DEV)     # higher = stronger
    order = torch.sort(-resp.reshape(-1)[idx], stable=True)[1]
    rank[idx[order]] = torch.arange(len(idx), 0, -1, device=DEV).double()
    rank, r = rank.reshape(1, 1, H, W), det.nms_radius
    kept, left = torch.zeros_like(rank, dtype=torch.bool), rank.clone()
    pool = lambda t: torch.nn.functional.max_pool2d(t, 2 * r + 1, 1, r)  # noqa: E731
    while (left > 0).any():
        new = (left > 0) & (left == pool(left))
        kept |= new
        left = torch.where(pool(new.double()) > 0, 0.0, left)
    ys, xs = kept[0, 0].nonzero(as_tuple=True)
    f = img.double()
    n, s1, s2 = (sum(_window(t, dy, dx) for dy in range(-3, 4) for dx in range(-3, 4))
                 for t in (torch.ones_like(f), f, f * f))          # kept points lie inside
    std = torch.sqrt((s2 / n - (s1 / n) ** 2).clamp(min=0))
    good = std[ys, xs] >= det.min_local_std
    ys, xs = ys[good], xs[good]

    def offset(a, b):
        c2 = a - 2 * resp[ys, xs] + b
        o = 0.5 * (a - b) / torch.where(c2.abs() > 1e-12, c2, 1.0)
        return torch.where((c2.abs() > 1e-12) & (o.abs() <= 0.5), o, 0.0)

    kx = xs + offset(resp[ys, xs - 1], resp[ys, xs + 1])
    ky = ys + offset(resp[ys - 1, xs], resp[ys + 1, xs])
    kp = torch.stack([kx, ky, resp[ys, xs], std[ys, xs]], 1).cpu().numpy()
    cell = ((ys // det.cell) * ((W + det.cell - 1) // det.cell) + xs // det.cell).cpu().numpy()
    o = np.lexsort(((ys * W + xs).cpu().numpy(), -kp[:, 2], cell))
    kp, cell = kp[o], cell[o]
    place = np.arange(len(cell)) - np.searchsorted(cell, cell)
    return kp[place < det.per_cell]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("dense", "uneven", "host"):
        if sum(W * H * D for W, H, D in _shapes(case)) > 2.5e9:
            return None
        cand, got = case.get("cand", False), []
        cfg_D = max(D for _, _, D in _shapes(case))
        for (L, R, _), (_, _, D) in zip(_scenes(case, seed), _shapes(case)):
            got.append(_dense_exact(L, R, _cfg(case, cfg_D), D, cand))
            if kind != "host" and not cand:
                got[-1].pop("cand")
        return got[0] if kind == "dense" and case["n"] == 1 else got
    if kind == "prior":
        return _prior_exact(case, seed)
    if kind == "edges":
        return _edges_exact(case, seed)
    if kind == "points":
        return _points_exact(case, seed)
    # the keypoints; the matches are a choice among them
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    L, R, _ = _scene(case["W"], case["H"], 61, g, rigid=True)
    det = sparse.DetCfg(cell=case["cell"], per_cell=case["per_cell"])
    return {k: _table(_keypoints_exact(i, det), _slots(case)) for k, i in (("kl", L), ("kr", R))}
