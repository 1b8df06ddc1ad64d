"""The prior path's row and column kernels at the edges of their shapes, against the
oracle bit for bit: every disparity group with planes left over, rectangles one row or a
few pixels large and clipped by the image, bands that admit one plane and all of them,
and the two sizes of the score table."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def same(a, b):
    return bool(((a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))).all())


def prior_map(kind, W, H, D, rng):
    p = np.full((H, W), max(1, D // 2), np.float32)
    if kind == "ramp":
        p[:] = np.linspace(-3, D + 4, W, dtype=np.float32)[None]
    elif kind == "noise":
        p[:] = rng.integers(0, 4 * (D + 2), (H, W)).astype(np.float32) / 4
    elif kind == "spot":                 # planes that one pixel, or one row, asks for
        p[:] = -100
        p[H // 2, W - 6] = max(1, D - 1)
        p[H - 5, W // 2:] = 1
    elif kind == "corner":
        p[:] = -100
        p[0, 0] = p[H - 1, W - 1] = max(1, D // 3)
    return p


@pytest.mark.parametrize("kind", ["flat", "ramp", "noise", "spot", "corner"])
@pytest.mark.parametrize("W,H,D,band,kw", [
    (40, 20, 1, 0, {}), (70, 33, 31, 1, dict(lrc=1)), (131, 24, 64, 2, dict(ad_trunc=40)),
    (150, 41, 65, 3, {}), (201, 18, 128, 1, dict(lrc=1)), (260, 21, 130, 200, {}),
    (230, 16, 193, 2, dict(ad_trunc=300)), (300, 19, 256, 5, {})])
def test_shapes(oracle, W, H, D, band, kw, kind):
    import doubleeye_b200 as de
    rng = np.random.default_rng(W + H + D)
    L = rng.integers(0, 256, (H, W), dtype=np.uint8)
    R = np.roll(L, -max(1, D // 2), 1) ^ rng.integers(0, 4, (H, W), dtype=np.uint8)
    prior = prior_map(kind, W, H, D, rng)
    cfg = dict(dmin=1, dmax=D, iters=2, **kw)
    r = de.run_dense_prior(L, R, prior, de.Cfg(**cfg), band=band)
    d, m, c = oracle.dense_prior(O.default_cfg(**cfg), L, R, prior, band)
    assert same(r.margin, m) and same(r.cand, c) and same(r.disp, d)
