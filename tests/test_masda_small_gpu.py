"""The one-CTA edge-list solve against the oracle bit for bit, on both sides of the sizes
that it takes, with repeated edges, equal scores and beliefs, empty rows and columns, a
segment that holds every edge, signed zeros and early convergence."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def solve(oracle, ei, ej, se, m, n, iters, eps=0.0, lam=-0.1, gam=-0.1, damping=0.4):
    from doubleeye_b200 import masda_stereo as ms
    a, h = ms.masda_sparse(ei, ej, se, m, n, lam, gam, iters=iters, damping=damping, eps=eps)
    want, wh = oracle.masda_edges(ei, ej, se, m, n, lam, gam, iters, damping, eps)
    got = np.array([a.get(i, -1) for i in range(m)], np.int64)
    assert h.tobytes() == np.asarray(wh).tobytes()
    assert np.array_equal(got, want)


@pytest.mark.parametrize("E,m,n", [(1, 1, 1), (2, 1, 2), (31, 5, 7), (513, 40, 600), (700, 700, 3),
                                   (4095, 300, 5000), (4096, 3000, 3144), (4097, 300, 300),
                                   (4000, 3000, 3145)])
@pytest.mark.parametrize("grid", [0, 8])
def test_sizes(oracle, E, m, n, grid):
    rng = np.random.default_rng(E + m + grid)
    ei, ej = rng.integers(0, m, E), rng.integers(0, n, E)
    se = rng.uniform(-0.5, 1.0, E)
    if grid:                             # equal scores, repeated edges
        se = np.round(se * grid) / grid
        ei[E // 2:] = ei[:E - E // 2]
    solve(oracle, ei.astype(np.int64), ej.astype(np.int64), se, m, n, 7)


def test_settings(oracle):
    rng = np.random.default_rng(3)
    ei, ej = rng.integers(0, 50, 400).astype(np.int64), rng.integers(0, 60, 400).astype(np.int64)
    se = rng.uniform(-1, 1, 400)
    se[:40] = 0.0
    se[40:80] = -0.0
    for kw in (dict(iters=0), dict(iters=1), dict(iters=200, eps=1e-3), dict(iters=9, damping=0.0),
               dict(iters=9, lam=0.3, gam=0.2), dict(iters=9, lam=0.0, gam=-0.0)):
        solve(oracle, ei, ej, se, 50, 60, **kw)


def test_one_row_holds_all(oracle):
    n = 2000
    solve(oracle, np.zeros(n, np.int64), np.arange(n, dtype=np.int64) % 900,
          np.linspace(-1, 1, n), 1, 900, 5)
