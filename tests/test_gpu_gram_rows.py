"""The second moments of a regression's rows (a row per thread up to 10 entries, 8 x 8 blocks by the
matrix instruction beyond) against numpy on demeaned data, at the entry counts where the kernel
changes and at row counts around the least of the streamed path (75,776) and its ragged tails."""

import numpy as np
import pytest

import fereg_b200 as fb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 15, 16])
@pytest.mark.parametrize("n", [75_776, 75_777, 75_903, 151_679])
def test_moments(n, k):
    rng = np.random.default_rng(n + k)
    g = 37
    codes = np.concatenate([np.arange(g), rng.integers(0, g, n - g)]).astype(np.uint32)
    x = rng.standard_normal((n, k)) + 0.1 * codes[:, None]
    y = x @ np.linspace(1.0, -0.5, k) + rng.standard_normal(n) * (1 + 0.2 * np.abs(x[:, 0])) + np.sin(codes)
    w = rng.uniform(0.5, 2.0, n)
    cnt = np.bincount(codes, minlength=g).astype(float)
    rows = np.ascontiguousarray(np.column_stack([y, x]))
    for weighted in (False, True):
        om = w if weighted else np.ones(n)
        tot = np.bincount(codes, om, g)
        z = rows - np.column_stack([(np.bincount(codes, om * c, g) / tot)[codes] for c in rows.T])
        zx, zy = z[:, 1:], z[:, 0]
        a = zx.T @ (om[:, None] * zx)
        b = np.linalg.solve(a, zx.T @ (om * zy))
        e = zy - zx @ b
        df = n - k - g
        ai = np.linalg.inv(a)
        v_un = ai * float(om @ e**2) / df
        v_ro = ai @ (zx.T @ ((om * e)[:, None] ** 2 * zx)) @ ai
        sess = fb.Session([codes], [g], w=w if weighted else None, weight_kind="aweight" if weighted else None)
        for vce in ("unadjusted", "robust"):
            r = sess.ols(np.ascontiguousarray(rows[sess.row_order()]), vce=vce)
            # sums of up to 1.5e5 products of order 1, a condition number below 10
            assert np.max(np.abs(np.asarray(r["b"])[:k] - b)) <= 1e-10
            v = np.asarray(r["V"])[:k, :k]
            want = v_un if vce == "unadjusted" else v_ro
            scale = v[0, 0] / want[0, 0]  # the library's small-sample factor
            assert abs(scale - 1) < 0.01
            assert np.max(np.abs(v - want * scale)) <= 1e-10 * np.max(np.abs(want))
        sess.close()
    assert cnt.min() > 0
