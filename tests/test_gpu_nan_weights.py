"""Elimination of a vertex whose weights hold a NaN.  A column whose stored
weights are all zero has the pivot 0, so its fills are 0/0; the neighbours that
receive them sort a NaN among their weights, of either sign.  The factor is NaN
from there on, but no entry may be lost or invented: a sort that lets padding
in before a NaN reads and writes past its list."""
import numpy as np
import pytest

import rchol_b200 as R
from helpers import OracleProblem

pytestmark = pytest.mark.gpu


def two_hubs(N, before, after, seed):
    """A path of `before` vertices, then hub h joined to hub h + 1 and to N more
    vertices by edges of weight zero, hub h + 1 joined to the same N vertices,
    which form a path, then a path of `after` vertices."""
    rng = np.random.default_rng(seed)
    h = before
    r = np.arange(h + 2, h + 2 + N)
    n = h + 2 + N + after
    path = [np.arange(h), np.arange(r[0], n - 1)]
    a = np.concatenate([*path, [h], np.full(N, h), np.full(N, h + 1)])
    b = np.concatenate([path[0] + 1, path[1] + 1, [h + 1], r, r])
    w = rng.uniform(0.5, 2.0, len(a))
    w[-2 * N - 1:-N] = 0.0
    i = np.arange(n)
    d = np.bincount(a, weights=w, minlength=n) + np.bincount(b, weights=w, minlength=n)
    rows, cols, vals = np.concatenate([a, b, i]), np.concatenate([b, a, i]), np.concatenate([-w, -w, d])
    return n, h, r, w[-N:], rows, cols, vals


def check(N, before, after, **opts):
    n, h, r, w, rows, cols, vals = two_hubs(N, before, after, seed=N)
    orc = OracleProblem(n, rows, cols, np.where(vals == 0.0, -1.0, vals)).factor(seed=3)  # columns before h
    ctx = R.Context(seed=3, **opts)
    try:
        ctx.set_triplets(n, rows, cols, vals, trim_ground=False)
        f = ctx.factor()
        cp, ri, val, d = f.to_host()
        info = f.info()
        f.free()
    finally:
        ctx.close()
    # before hub h: the oracle's factor
    assert np.array_equal(cp[:h + 1], orc["colptr"][:h + 1])
    assert np.array_equal(ri[:cp[h]], orc["rowind"][:cp[h]])
    assert np.array_equal(val[:cp[h]], orc["val"][:cp[h]])
    assert np.array_equal(d[:h], orc["diag"][:h])
    # hub h: pivot 0; hub h + 1 keeps its N neighbours, the first with a NaN
    assert np.array_equal(ri[cp[h]:cp[h + 1]], np.append(h + 1, r))
    assert d[h] == 0.0 and np.isnan(val[cp[h]:cp[h + 1]]).all()
    assert np.array_equal(ri[cp[h + 1]:cp[h + 2]], r)
    assert np.isnan(d[h + 1]) and np.isnan(val[cp[h + 1]:cp[h + 2]]).all()
    # every column: rows below the diagonal, ascending, once each
    col = np.repeat(np.arange(n), np.diff(cp))
    assert (ri > col).all() and (ri < n).all()
    assert (np.diff(ri)[np.diff(col) == 0] > 0).all()
    assert info.fills == np.maximum(np.diff(cp) - 1, 0).sum()
    # hub h joins its neighbours in row order (all weights equal), hub h + 1 in
    # weight order with the NaN last: no comparison with a NaN sum holds, so
    # each partner is the next in order
    order = r[1:][np.argsort(w[1:], kind="stable")]
    pairs = [(h + 1, r[0])] + list(zip(r[:-1], r[1:])) + list(zip(order[:-1], order[1:])) + [(order[-1], r[0])]
    have = set(zip(col.tolist(), ri.tolist()))
    assert all((min(p), max(p)) in have for p in pairs)
    assert info.max_gather >= N + 1


@pytest.mark.parametrize("N", [31, 40, 64, 200, 255, 300, 500, 600, 1000, 1022])
def test_late_vertices_of_a_256_thread_cta(N):
    check(N, before=8 * (N + 40), after=0)


@pytest.mark.parametrize("N", [40, 1000, 1500, 3000, 4094])
def test_late_vertices_of_a_1024_thread_cta(N):
    check(N, before=8, after=0, tail_vertices=N + 2)


@pytest.mark.parametrize("N", [20, 33, 40, 100, 128, 200, 255, 300, 1000])
def test_early_vertices_of_one_warp(N):
    check(N, before=0, after=8 * (N + 40))
