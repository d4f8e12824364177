"""The covariance of a regression on many rows against numpy with the exact small-sample factors (no
scale taken from the result): rss / (n - k - g) unadjusted, n / (n - k - g) robust, analytic weights
normalized to sum n. At entry counts on both sides of the line between the two kernels of the second
moments."""

import numpy as np
import pytest

import fereg_b200 as fb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 3, 8, 9, 10, 16])
@pytest.mark.parametrize("weighted", [False, True])
def test_covariance(k, weighted):
    n, g = 75_903, 37
    rng = np.random.default_rng(k)
    codes = np.concatenate([np.arange(g), rng.integers(0, g, n - g)]).astype(np.uint32)
    x = rng.standard_normal((n, k)) + 0.1 * codes[:, None]
    y = x @ np.linspace(1.0, -0.5, k) + rng.standard_normal(n) * (1 + 0.2 * np.abs(x[:, 0])) + np.sin(codes)
    w = rng.uniform(0.5, 2.0, n) if weighted else None
    om = w * (n / w.sum()) if weighted else np.ones(n)
    rows = np.ascontiguousarray(np.column_stack([y, x]))
    tot = np.bincount(codes, om, g)
    z = rows - np.column_stack([(np.bincount(codes, om * c, g) / tot)[codes] for c in rows.T])
    zx, zy = z[:, 1:], z[:, 0]
    a = zx.T @ (om[:, None] * zx)
    e = zy - zx @ np.linalg.solve(a, zx.T @ (om * zy))
    ai, df = np.linalg.inv(a), n - k - g
    want = {"unadjusted": ai * float(om @ e**2) / df,
            "robust": ai @ (zx.T @ ((om * e)[:, None] ** 2 * zx)) @ ai * (n / df)}
    sess = fb.Session([codes], [g], w=w, weight_kind="aweight" if weighted else None)
    block = np.ascontiguousarray(rows[sess.row_order()])
    for vce, v in want.items():
        got = np.asarray(sess.ols(block, vce=vce)["V"])[:k, :k]
        # sums of 7.6e4 products of order 1, a condition number below 10
        assert np.max(np.abs(got - v)) <= 1e-10 * np.max(np.abs(v)), vce
