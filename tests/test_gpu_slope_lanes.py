"""The slope solver's lane groups (4 to 32 lanes a level), warps and CTAs per coordinate list, and the sums
over more than 4,096 levels: the residuals are orthogonal to every design column and differ from the
rows by a fit of the design, which is what the projection is."""

import numpy as np
import pytest

import fereg_b200 as fb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels,years,other", [(4097, 3, 40), (900, 8, 30), (500, 9, 60), (300, 17, 25),
                                                (120, 33, 7), (40, 200, 3)])
@pytest.mark.parametrize("e_slopes,r,weighted", [(0, 1, False), (1, 4, True), (2, 5, False), (4, 9, True)])
def test_projection(levels, years, other, e_slopes, r, weighted):
    if years <= 1 + e_slopes:
        pytest.skip("levels with as many parameters as rows: their systems have no bounded condition")
    rng = np.random.default_rng(levels + r)
    n = levels * years
    code0 = np.repeat(np.arange(levels), years).astype(np.uint32)
    code1 = np.concatenate([np.arange(other), rng.integers(0, other, n - other)]).astype(np.uint32)
    xs = [rng.standard_normal(n) for _ in range(e_slopes)]
    z = rng.standard_normal(n)
    w = rng.uniform(0.5, 2.0, n) if weighted else None
    ab = fb.Absorber([code0, code1], [levels, other], w, intercept=[True, True], slopes=[xs, [z]])
    v = rng.standard_normal((n, r)) + 0.1 * (code1 % 5)[:, None]
    pi = ab.row_order()
    rows = np.ascontiguousarray(v[pi])
    res = ab.residualize(rows, tol=1e-13, maxiter=100000, want_coefs=True)
    d = np.empty_like(rows)
    d[pi] = rows
    om = np.ones(n) if w is None else w
    for code, g, slopes in ((code0, levels, xs), (code1, other, [z])):
        for s in [np.ones(n)] + slopes:
            for c in range(r):
                # sums of at most a few thousand terms of unit scale, the solve at tol 1e-13
                assert np.max(np.abs(np.bincount(code, om * s * d[:, c], g))) <= 1e-7
    for c in range(r):
        assert np.max(np.abs(ab.fit_rows(res["coefs"], c) - (v[pi, c] - rows[:, c]))) <= 1e-8
