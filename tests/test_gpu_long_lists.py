"""Segments and coordinate lists longer than a warp tile: the warp-per-tile segment passes, the
CTA-per-tile list passes and their slices, with one row per cell and several (the list pass then reads
the cells' sums), weighted and not, at segment lengths around 32 cells and 128 (one tile), list lengths
around 256 and 2048 entries, and widths around the kernels' column chunks. Against the oracle at the
parity tests' bounds (operator and right-hand side 1e-12, residuals 1e-9)."""

import numpy as np
import pytest

import fereg_b200 as fb
from oracle import oracle

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.max(np.abs(a - b))) / max(1.0, float(np.max(np.abs(b))))


def build(cells, rows_per_cell, occ, weighted, seed):
    """Individuals of `cells` distinct (firm, occ) cells, each of rows_per_cell rows."""
    rng = np.random.default_rng(seed)
    n_ind = max(60, 9000 // cells)
    ind = np.repeat(np.arange(n_ind), cells * rows_per_cell)
    firm = np.repeat(rng.integers(0, 5000, n_ind * cells), rows_per_cell)
    oc = np.repeat(rng.integers(0, occ, n_ind * cells), rows_per_cell)
    keep = np.ones(len(ind), bool)
    if rows_per_cell > 1:  # ragged cells
        keep = rng.random(len(ind)) < 0.8
    codes = [np.unique(c[keep], return_inverse=True)[1].astype(np.uint32) for c in (ind, firm, oc)]
    g = [int(c.max()) + 1 for c in codes]
    w = rng.uniform(0.3, 2.0, len(codes[0])) if weighted else None
    return codes, g, w


@pytest.mark.parametrize("cells", [31, 32, 33, 127, 129, 300])
@pytest.mark.parametrize("rows_per_cell,weighted,r", [(1, False, 3), (1, True, 17), (5, False, 12), (5, True, 33)])
def test_long_segments(cells, rows_per_cell, weighted, r):
    codes, g, w = build(cells, rows_per_cell, 25, weighted, cells * 10 + r)
    gpu, orc = fb.Absorber(codes, g, w), oracle.Absorber(codes, g, w)
    assert gpu.fe1 == orc.fe1
    rng = np.random.default_rng(1)
    p = rng.standard_normal((gpu.m, r))
    assert rel(gpu.apply(p), orc.apply(p)) <= 1e-12
    z = rng.standard_normal((gpu.n, r))
    for a, b in zip(gpu.rhs(z), orc.rhs(z)):
        assert rel(a, b) <= 1e-12
    z1, z2 = z.copy(), z.copy()
    i1 = gpu.residualize(z1, tol=1e-12, maxiter=100000, want_coefs=True)
    orc.residualize(z2, tol=1e-12, maxiter=100000)
    assert rel(z1, z2) <= 1e-9
    assert rel(z[:, 0] - gpu.fit_rows(i1["coefs"], 0), z1[:, 0]) <= 1e-9


@pytest.mark.parametrize("occ", [20, 35, 60, 200])
@pytest.mark.parametrize("rows_per_cell,weighted,r", [(1, False, 2), (1, True, 11), (4, True, 40)])
def test_long_lists(occ, rows_per_cell, weighted, r):
    """Lists of 80,000 / 35 entries and the like: whole lists of a tile and slices of longer ones."""
    codes, g, w = build(9, rows_per_cell, occ, weighted, occ + r)
    gpu, orc = fb.Absorber(codes, g, w), oracle.Absorber(codes, g, w)
    rng = np.random.default_rng(2)
    p = rng.standard_normal((gpu.m, r))
    assert rel(gpu.apply(p), orc.apply(p)) <= 1e-12
    z = rng.standard_normal((gpu.n, r))
    for a, b in zip(gpu.rhs(z), orc.rhs(z)):
        assert rel(a, b) <= 1e-12


def test_weights_back_and_forth():
    """Replayed iterations follow the weight state: weighted, unit, weighted again, device weights."""
    import torch

    codes, g, w = build(40, 1, 25, True, 5)
    gpu, orc = fb.Absorber(codes, g, w), oracle.Absorber(codes, g, w)
    z = np.random.default_rng(3).standard_normal((gpu.n, 4))
    order = gpu.row_order()
    w2 = np.random.default_rng(4).uniform(0.5, 1.5, gpu.n)
    for step in (w[order], None, w2, w[order], None, w2):
        for _ in range(3):  # by launches, then by graphs
            if step is w2:
                gpu.set_weights_device(torch.from_numpy(w2).cuda().data_ptr())
            else:
                gpu.set_weights(step)
            orc.set_weights(step)
            z1, z2 = z.copy(), z.copy()
            gpu.residualize(z1, tol=1e-12, maxiter=100000)
            orc.residualize(z2, tol=1e-12, maxiter=100000)
            assert rel(z1, z2) <= 1e-9
