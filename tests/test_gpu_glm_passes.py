"""The GLM's row passes: a call that fails leaves the session as it was."""

import numpy as np
import pytest

import fereg_b200 as fb
from tests._gen import panel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family", ["poisson", "logit"])
def test_a_failed_call_leaves_the_session_unweighted(family):
    codes, g, _, z = panel(n_ind=500, years=6, n_firm=60, seed=2, weighted=False, r=3)
    s = fb.Session(codes, g)
    rows = np.ascontiguousarray(z[s.row_order()])
    want = s.ols(rows)
    y = np.random.default_rng(1).poisson(np.exp(0.3 * rows[:, 1])) if family == "poisson" else rows[:, 0] > 0
    with pytest.raises(fb.FeregError) as e:
        s.glm(np.column_stack([y.astype(float), rows[:, 1:]]), family, maxiter=1)
    assert e.value.rc == 430
    got = s.ols(rows)
    # two solves at tol 1e-8, the second with preconditioners built again
    assert np.max(np.abs(got["b"] - want["b"])) <= 1e-7 * np.max(np.abs(want["b"]))
