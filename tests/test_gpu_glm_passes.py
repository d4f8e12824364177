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


@pytest.mark.parametrize("family", ["poisson", "logit"])
@pytest.mark.parametrize("n_ind", [1, 7, 25_258, 25_259])  # 6 rows each, around one row a thread
def test_device_blocks_are_read_in_place(family, n_ind):
    import torch

    codes, g, _, z = panel(n_ind=n_ind, years=6, n_firm=None, seed=n_ind, weighted=False, r=3)
    n = 6 * n_ind
    rng = np.random.default_rng(n_ind)
    eta = 0.4 * z[:, 1] - 0.2 * z[:, 2]
    y = rng.poisson(np.exp(eta)) if family == "poisson" else rng.random(n) < 1 / (1 + np.exp(-eta))
    codes, g = [codes[1]], [g[1]]  # the years: every level has rows of both outcomes or more
    y = np.where(np.arange(n) < 6, np.arange(n) % 2, y) if n_ind == 1 else y
    s = fb.Session(codes, g)
    rows = np.ascontiguousarray(np.column_stack([y.astype(float), z[:, 1:]])[s.row_order()])
    try:
        want = s.glm(rows, family)
    except fb.FeregError as e:
        want = e.rc
    for off in (0, 1):
        buf = torch.zeros(n * 3 + 4, dtype=torch.float64, device="cuda")
        view = buf[off : off + n * 3]
        view.copy_(torch.from_numpy(rows).reshape(-1))
        torch.cuda.synchronize()
        try:
            got = s.glm(view.data_ptr(), family, on_device=True, nx=2)
        except fb.FeregError as e:
            got = e.rc
        torch.cuda.synchronize()
        assert np.array_equal(view.cpu().numpy(), rows.reshape(-1))  # left as it was
        if isinstance(want, int):
            assert got == want
        else:
            assert np.array_equal(got["b"], want["b"]) and np.array_equal(got["V"], want["V"])
    if n_ind > 7:  # the slopes the outcomes were drawn with
        b = want["b"]
        assert np.all(np.abs(b - [0.4, -0.2]) < 0.05)
