"""The wild bootstrap's draws do not depend on how they are tiled: tiles whose width is not a multiple of
4 (padded columns) or of 32 (sign words), one draw a tile, and a last tile of another width."""

import numpy as np
import pytest

import fereg_b200 as fb
from tests._gen import panel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [1, 3, 31, 32, 33, 66, 70])
@pytest.mark.parametrize("k,weighted", [(1, False), (3, True)])
def test_draws_do_not_depend_on_the_tile(tile, k, weighted):
    codes, g, w, z = panel(n_ind=700, years=6, n_firm=90, seed=k, weighted=weighted, r=1 + k)
    s = fb.Session(codes, g, [codes[2]], [g[2]], w=w, weight_kind="aweight" if weighted else None)
    rows = np.ascontiguousarray(z[s.row_order()])
    kw = dict(coef=k - 1, reps=99, seed=5, tol=1e-12, maxiter=100000)
    a = s.wildboot(rows, tile=99, **kw)
    b = s.wildboot(rows, tile=tile, **kw)
    assert np.all(np.isfinite(a["t_boot"])) and len(a["t_boot"]) == len(b["t_boot"])
    # solves at tol 1e-12 of columns of unit scale
    assert np.max(np.abs(a["t_boot"] - b["t_boot"])) <= 1e-9 * max(1.0, np.max(np.abs(a["t_boot"])))
    assert a["pvalue"] == b["pvalue"] and a["stat"] == b["stat"]
