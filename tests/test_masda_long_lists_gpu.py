"""The one-CTA edge-list solve where a row or a column holds many edges, against the oracle
bit for bit: list lengths on both sides of what a thread takes and of a warp's piece, all
edges in one list, long lists of rows and of columns together, equal scores.  Non-finite
scores, whose changes are NaN, are compared with the grid-wide passes instead, which take
the same problem once unused nodes are added (the oracle's maximum drops a NaN)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def solve(oracle, ei, ej, se, m, n, iters):
    from doubleeye_b200 import masda_stereo as ms
    ei, ej = np.ascontiguousarray(ei, np.int64), np.ascontiguousarray(ej, np.int64)
    a, h = ms.masda_sparse(ei, ej, se, m, n, iters=iters, eps=0.0)
    want, wh = oracle.masda_edges(ei, ej, se, m, n, -0.1, -0.1, iters, 0.4, 0.0)
    got = np.array([a.get(i, -1) for i in range(m)], np.int64)
    assert h.tobytes() == np.asarray(wh).tobytes()
    assert np.array_equal(got, want)


@pytest.mark.parametrize("length", [15, 16, 17, 63, 64, 65, 128, 129, 1000, 4096])
@pytest.mark.parametrize("grid", [0, 6])
@pytest.mark.parametrize("turn", [False, True])
def test_lengths(oracle, length, grid, turn):
    rng = np.random.default_rng(length + grid)
    m, n = max(1, 4096 // length), max(length, 64)
    ei = np.repeat(np.arange(m), length)
    ej = np.concatenate([rng.permutation(n)[:length] for _ in range(m)])
    se = rng.uniform(-0.4, 1.0, len(ei))
    if grid:
        se = np.round(se * grid) / grid
    order = rng.permutation(len(ei))
    ei, ej, se = ei[order], ej[order], se[order]
    if turn:
        ei, ej, m, n = ej, ei, n, m
    solve(oracle, ei, ej, se, m, n, 6)


def test_short_and_long_together(oracle):
    rng = np.random.default_rng(5)
    E, m, n = 4096, 900, 700
    ei = np.minimum((rng.pareto(1.0, E) * 2).astype(int), m - 1)
    ej = np.minimum((rng.pareto(0.7, E) * 2).astype(int), n - 1)
    se = rng.uniform(-0.5, 1.0, E)
    solve(oracle, ei, ej, se, m, n, 9)


@pytest.mark.parametrize("value", [-np.inf, np.inf, np.nan])
def test_non_finite_scores(value):
    from doubleeye_b200 import masda_stereo as ms
    rng = np.random.default_rng(6)
    E, m, n = 4096, 900, 700
    ei = np.minimum((rng.pareto(1.0, E) * 2).astype(np.int64), m - 1)
    ej = np.minimum((rng.pareto(0.7, E) * 2).astype(np.int64), n - 1)
    se = rng.uniform(-0.5, 1.0, E)
    se[::50] = value
    a, ha = ms.masda_sparse(ei, ej, se, m, n, iters=4, eps=0.0)
    b, hb = ms.masda_sparse(ei, ej, se, m + 5000, n + 5000, iters=4, eps=0.0)
    assert a == b
    assert np.array_equal(ha, hb, equal_nan=True)
