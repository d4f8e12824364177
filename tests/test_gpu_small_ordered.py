"""One small block of at most 32 coordinates on cells of one row, without weights (k_small_ordered)
against the oracle's preconditioner: the block's width around half a warp and a warp, a small code held
by several cells of a segment (the subtraction once per cell), lists of several items of 256 entries
with a segment's entries across an item's end, and the line at 33 coordinates. The large block (over
4,096 levels) keeps the cells apart. The tolerance is the parity tests' for the preconditioner (1e-10)."""

import numpy as np
import pytest

import fereg_b200 as fb
from oracle import oracle

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.max(np.abs(a - b))) / max(1.0, float(np.max(np.abs(b))))


@pytest.mark.parametrize("years", [1, 2, 15, 16, 17, 31, 32, 33])
@pytest.mark.parametrize("repeats", [1, 6])
def test_small_ordered(years, repeats):
    rng = np.random.default_rng(years)
    n_ind, per, firms = 5200, 9, 5000
    ind = np.repeat(np.arange(n_ind), per)
    # an individual's firms differ: every cell holds one row
    firm = (ind * 7 + np.tile(np.arange(per), n_ind) * 311) % firms
    year = rng.integers(0, years, n_ind * per)
    if repeats > 1:  # the first cells of every individual share a year
        year = year.reshape(n_ind, per)
        year[:, :repeats] = year[:, :1]
        year = year.ravel()
    year[:years] = np.arange(years)
    codes, g = [c.astype(np.uint32) for c in (ind, year, firm)], [n_ind, years, firms]
    gpu, orc = fb.Absorber(codes, g), oracle.Absorber(codes, g)
    assert gpu.ncells == gpu.n and gpu.m_small == years and gpu.fe1 == 0
    p = orc.apply(rng.standard_normal((gpu.m, 2)))
    assert rel(orc.apply(gpu.precond(p)), orc.apply(orc.precond(p))) <= 1e-10
    z = rng.standard_normal((gpu.n, 2))
    z1, z2 = z.copy(), z.copy()
    gpu.residualize(z1, tol=1e-12, maxiter=100000)
    orc.residualize(z2, tol=1e-12, maxiter=100000)
    assert rel(z1, z2) <= 1e-9
