"""The prior path's row kernel where the planes' rectangles are short and far apart, so that
each lane walks its own: slanted priors across wide images, rising and falling, planes that
reach both image edges, bands on both sides of where lanes walk together again.  Against
the oracle bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("kind", ["rise", "fall", "steps", "ends"])
@pytest.mark.parametrize("W,H,D,band,kw", [
    (600, 19, 64, 0, {}), (521, 17, 20, 0, dict(lrc=1)), (700, 16, 130, 1, dict(ad_trunc=40)),
    (1100, 15, 256, 0, dict(dmin=3)), (640, 18, 40, 3, {}), (640, 18, 40, 12, {}), (900, 8, 2, 0, {})])
def test_slanted(oracle, W, H, D, band, kw, kind):
    import doubleeye_b200 as de
    rng = np.random.default_rng(W + D + band)
    L = rng.integers(0, 256, (H, W), dtype=np.uint8)
    R = np.roll(L, -max(1, D // 2), 1) ^ rng.integers(0, 4, (H, W), dtype=np.uint8)
    dmin = kw.get("dmin", 1)
    ramp = np.linspace(dmin, dmin + D - 1, W, dtype=np.float32)
    if kind == "fall":
        ramp = ramp[::-1]
    elif kind == "steps":
        ramp = np.roll(np.round(ramp / 5) * 5, W // 3)
    elif kind == "ends":                 # two planes, at the image's edges only
        ramp = np.where(np.arange(W) < 12, dmin, np.where(np.arange(W) >= W - 12, dmin + D - 1, -50))
    prior = np.ascontiguousarray(np.broadcast_to(ramp.astype(np.float32), (H, W)))
    cfg = dict(dmin=dmin, dmax=dmin + D - 1, iters=2)
    cfg.update({k: v for k, v in kw.items() if k != "dmin"})
    r = de.run_dense_prior(L, R, prior, de.Cfg(**cfg), band=band)
    d, m, c = oracle.dense_prior(O.default_cfg(**cfg), L, R, prior, band)
    for a, b in ((r.margin, m), (r.cand, c), (r.disp, d)):
        assert ((a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))).all()
