"""The detector's per-cell stage at the edges of its cells, against the oracle bit for bit:
cells larger than the image, ragged last cells, one point a cell and all of them, the
densest suppression, with and without sub-pixel positions and the texture floor."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("W,H", [(16, 16), (33, 47), (129, 128), (200, 131)])
@pytest.mark.parametrize("kw", [
    dict(cell=4, per_cell=1, nms_radius=1), dict(cell=32, per_cell=3), dict(cell=31, per_cell=400,
                                                                            nms_radius=1),
    dict(cell=128, per_cell=4000, nms_radius=1, min_local_std=0.0), dict(cell=128, per_cell=2),
    dict(cell=17, per_cell=5, subpixel=0, min_local_std=30.0, grad_window=7)])
def test_cells(oracle, W, H, kw):
    from doubleeye_b200 import sparse as sp
    rng = np.random.default_rng(W * H)
    img = rng.integers(0, 256, (H, W), dtype=np.uint8)
    det = O.default_det_cfg(border=5, **kw)
    c = sp.DetCfg()
    for f, _ in c._fields_:
        setattr(c, f, getattr(det, f))
    got, want = sp.detect_fast(img, c), oracle.detect_fast(img, det)
    assert got.shape == want.shape and got.tobytes() == want.tobytes()
