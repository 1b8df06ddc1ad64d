"""The register row solve at the edges of its launch shapes (rows of 2 and 4 pixels a
thread, the last pixel of a warp and of a row), with right pixels named by one to more
than eight candidates, and the settings that keep the shared-memory solve; against the
oracle bit for bit."""
import numpy as np
import pytest

from oracle.oracle import Oracle, default_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def check(L, R, **kw):
    from doubleeye_b200 import dense
    got = dense.run_dense(L, R, dense.Cfg(**kw))
    disp, margin, cand = Oracle().dense(default_cfg(**kw), L, R)
    for name, a, b in (("disp", got.disp, disp), ("margin", got.margin, margin),
                       *((f"plane {p}", got.cand[p], cand[p]) for p in range(6))):
        same = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))
        assert same.all(), f"{name}: {int((~same).sum())} values differ"


def scene(W, H, D, levels):
    """Random texture of a few grey levels: the fewer, the more candidates share a right
    pixel."""
    rng = np.random.default_rng(W + D + levels)
    L = (rng.integers(0, levels, (H, W)) * (255 // levels)).astype(np.uint8)
    return L, np.roll(L, -min(D // 2, 9), 1)


@pytest.mark.parametrize("iters", [0, 1, 4])
@pytest.mark.parametrize("levels", [1, 2, 40])
@pytest.mark.parametrize("W,D", [(8, 1), (63, 20), (65, 40), (257, 128), (1023, 30), (1025, 30),
                                 (2049, 16)])
def test_row_shapes(W, D, levels, iters):
    check(*scene(W, 9, D, levels), dmin=1, dmax=D, iters=iters)


@pytest.mark.parametrize("kw", [dict(damping=1.5), dict(damping=-0.25), dict(lambda_=-2e6),
                                dict(gamma=-3e6), dict(damping=1.0), dict(damping=0.0),
                                dict(min_margin=0.05), dict(min_ratio=1.2), dict(lrc=1),
                                dict(fit_eq=0), dict(subpixel=0)])
def test_settings(kw):
    check(*scene(130, 12, 40, 6), dmin=1, dmax=40, iters=5, **kw)
