"""The tensor-memory column kernel at the edges of its tiles, against the oracle bit for
bit: 32-row blocks (a last block that is full, one row long, all border), the 512 rows
that stay on chip and the ones that go back to the volume, tiles of 4, 2 and 1 columns
that the image does not fill, and the four disparity groups with planes left over."""
import numpy as np
import pytest

from oracle.oracle import Oracle, default_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("W,H,D", [
    (8, 8, 1), (9, 9, 2), (41, 35, 31), (40, 36, 32), (97, 67, 64), (98, 70, 65),
    (150, 38, 128), (151, 99, 100), (200, 40, 129), (210, 34, 192), (230, 33, 193),
    (270, 45, 256), (31, 515, 12), (30, 516, 20), (45, 547, 33), (36, 610, 9), (90, 700, 70)])
@pytest.mark.parametrize("hh,lrc", [(3, 0), (3, 1), (4, 0)])
def test_tile_edges(W, H, D, hh, lrc):
    from doubleeye_b200 import dense
    rng = np.random.default_rng(W * 1000 + H)
    L = rng.integers(0, 256, (H, W), dtype=np.uint8)
    R = np.roll(L, -min(D, 5), 1) ^ rng.integers(0, 8, (H, W), dtype=np.uint8)
    kw = dict(dmin=1, dmax=D, iters=2, census_hw=3, census_hh=hh, lrc=lrc)
    got = dense.run_dense(L, R, dense.Cfg(**kw))
    disp, margin, cand = Oracle().dense(default_cfg(**kw), L, R)
    for name, a, b in (("disp", got.disp, disp), ("margin", got.margin, margin),
                       *((f"plane {p}", got.cand[p], cand[p]) for p in range(6))):
        same = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))
        assert same.all(), f"{name}: {int((~same).sum())} values differ"


@pytest.mark.parametrize("D", [40, 128, 192, 256])
def test_reverse_match_in_batches(D):
    """Pairs that share a launch set take the streaming kernel: the same reverse match."""
    from doubleeye_b200 import dense
    rng = np.random.default_rng(D)
    kw = dict(dmin=1, dmax=D, iters=1, lrc=1)
    pairs = [tuple(rng.integers(0, 256, (H, W), dtype=np.uint8) for _ in range(2))
             for W, H in ((D + 70, 21), (D + 141, 40))]
    for got, (L, R) in zip(dense.run_dense_batch(pairs, dense.Cfg(**kw), want_cand=True), pairs):
        _, _, cand = Oracle().dense(default_cfg(**kw), L, R)
        same = (got.cand.view(np.uint32) == cand.view(np.uint32)) | (np.isnan(got.cand) & np.isnan(cand))
        assert same.all()
