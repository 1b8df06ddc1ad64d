"""The tensor-memory column kernel where a CTA takes three tiles or more and the images have
more than the 512 rows that stay on chip: rings and coefficient buffers that wrap across
tiles, rows that go back to the volume, the reverse match's write-back into them; and a
launch set of unequal heights in one disparity group.  Against the oracle bit for bit."""
import numpy as np
import pytest

from oracle.oracle import Oracle, default_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def images(W, H, D, seed):
    rng = np.random.default_rng(seed)
    L = rng.integers(0, 256, (H, W), dtype=np.uint8)
    return L, np.roll(L, -min(D, 9), 1) ^ rng.integers(0, 8, (H, W), dtype=np.uint8)


def check(got, kw, L, R):
    disp, margin, cand = Oracle().dense(default_cfg(**kw), L, R)
    for name, a, b in (("disp", got["disp"], disp), ("margin", got["margin"], margin),
                       ("cand", got["cand"], cand)):
        same = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))
        assert same.all(), f"{name}: {int((~same).sum())} values differ"


@pytest.mark.parametrize("lrc", [0, 1])
@pytest.mark.parametrize("W,H,D", [(1300, 560, 64), (750, 547, 128), (460, 530, 192), (500, 563, 256)])
def test_spill_and_three_tiles(W, H, D, lrc):
    from doubleeye_b200 import dense
    kw = dict(dmin=1, dmax=D, iters=1, lrc=lrc)
    L, R = images(W, H, D, W + lrc)
    check(vars(dense.run_dense(L, R, dense.Cfg(**kw))), kw, L, R)


@pytest.mark.parametrize("lrc", [0, 1])
@pytest.mark.parametrize("D", [50, 120])
def test_unequal_heights(D, lrc):
    from doubleeye_b200 import _lib, dense
    kw = dict(dmin=1, dmax=D, iters=1, lrc=lrc)
    pairs = [images(W, H, D, H) for W, H in ((420, 41), (430, 545), (410, 200))]
    saved = _lib.get_param("batch_streams")
    try:
        _lib.set_param("batch_streams", 1)         # one launch set, which runs by itself
        got = dense.DenseMatcher(dense.Cfg(**kw)).match_batch(
            [tuple(torch.from_numpy(i).cuda() for i in p) for p in pairs], cand=True)
    finally:
        _lib.set_param("batch_streams", saved)
    for g, (L, R) in zip(got, pairs):
        check({k: v.cpu().numpy() for k, v in g.items()}, kw, L, R)


def test_reverse_match_of_uneven_pairs():
    """One launch set whose pairs differ in size and group: seven small ones in one group
    (two of them without candidates), and one in another."""
    from doubleeye_b200 import _lib, dense
    kw = dict(dmin=30, dmax=90, iters=1, lrc=1)
    sizes = [(36, 20, 0), (200, 9, 0), (37, 50, 0), (330, 41, 0), (30, 8, 0), (101, 77, 0),
             (230, 30, 220), (64, 64, 0)]
    pairs = [images(W, H, 60, W + H) for W, H, _ in sizes]
    saved = _lib.get_param("batch_streams")
    try:
        _lib.set_param("batch_streams", 1)
        got = dense.DenseMatcher(dense.Cfg(**kw)).match_batch(
            [(*(torch.from_numpy(i).cuda() for i in p), d) for p, (_, _, d) in zip(pairs, sizes)],
            cand=True)
    finally:
        _lib.set_param("batch_streams", saved)
    for g, (L, R), (_, _, d) in zip(got, pairs, sizes):
        check({k: v.cpu().numpy() for k, v in g.items()}, dict(kw, dmax=d or 90), L, R)
