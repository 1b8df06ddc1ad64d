"""The keypoint matcher's storage and sort choices at their limits, against the oracle bit
for bit: problems that fit in shared memory and ones that do not, right points in bins,
all on one row, spread over many orders of magnitude, and more than a bin or the shared
copies take; lists of one, two, a few and more than 63 edges."""
import numpy as np
import pytest

from oracle import oracle as O
from test_oracle_sparse import same_bits

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def points(rng, n, W, H, rows=None):
    kp = np.zeros((n, 4), np.float32)
    kp[:, 0] = np.round(rng.uniform(0, W, n) * 4) / 4
    kp[:, 1] = np.round(rng.uniform(0, H, n) * 4) / 4 if rows is None else rng.choice(rows, n)
    kp[:, 2] = rng.uniform(1, 50, n)
    return kp, rng.integers(0, 1 << 48, n, dtype=np.uint64)


@pytest.mark.parametrize("nl,nr,W,H,rows,kw", [
    (0, 5, 60, 40, None, {}), (5, 0, 60, 40, None, {}), (1, 1, 60, 40, [7.0], {}),
    (33, 60, 60, 40, None, {}),                              # one bin and a few
    (70, 90, 300, 40, [11.0], dict(max_candidates=100)),     # one row: lists of up to 90
    (400, 500, 400, 300, [0.0, 1e30, -1e30, 3.0], dict(iterations=5)),   # bitonic
    (500, 1500, 700, 40, None, dict(max_candidates=60, iterations=6)),   # many edges
    (2200, 2100, 800, 400, None, dict(iterations=6, lambda_=-0.1, gamma=-0.1)),
    (300, 11500, 800, 1000, None, dict(iterations=3)),       # beyond the shared copies
    (300, 13600, 800, 1000, None, dict(iterations=3)),       # beyond the bins' scratch
    (9000, 900, 800, 600, None, dict(iterations=3))])        # beyond shared storage
def test_shapes(oracle, nl, nr, W, H, rows, kw):
    from doubleeye_b200 import sparse as sp
    rng = np.random.default_rng(nl + 7 * nr)
    kl, dl = points(rng, nl, W, H, rows)
    kr, dr = points(rng, nr, W, H, rows)
    k = min(nl, nr) // 2                                     # half of them have a partner
    kr[:k, :2] = kl[:k, :2] - np.array([3.0, 0.25], np.float32)
    dr[:k] = dl[:k] ^ np.uint64(5)
    kw = dict(max_disparity=64.0, **kw)
    want, ws = oracle.match_masda(kl, dl, kr, dr, O.default_match_cfg(**kw))
    got, gs = sp.match_masda(kl, dl, kr, dr, sp.MatchCfg(**kw))
    assert same_bits(got, want)
    for f in ("candidates", "iterations_run", "converged", "oscillating"):
        assert gs[f] == (ws[f] if isinstance(ws, dict) else getattr(ws, f)), f
