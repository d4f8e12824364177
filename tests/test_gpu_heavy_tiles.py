"""Segments of many rows: tiles cut by rows, heavy ones taken by a CTA. Few levels (every tile heavy),
one large level among many small ones (heavy and light tiles side by side), segments of more than 128
cells (slices, heavy or not), one term alone and no term at all, weighted and not, at widths around the
kernels' column chunks. Against the oracle at the parity tests' bounds (right-hand side 1e-12, residuals
1e-9), and the time of a sample of few levels against the same rows in many."""

import time

import numpy as np
import pytest

import fereg_b200 as fb
from oracle import oracle

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.max(np.abs(a - b), initial=0.0)) / max(1.0, float(np.max(np.abs(b), initial=0.0)))


def draw(n, levels, share, seed):
    """n rows over the terms' levels, the first level of each with `share` of the rows."""
    rng = np.random.default_rng(seed)
    codes = []
    for g in levels:
        c = rng.integers(0, g, n).astype(np.uint32)
        c[rng.random(n) < share] = 0
        c[:g] = np.arange(g)
        codes.append(c)
    return codes, list(levels)


CASES = {
    "one_level": (1500, [1], 0.0),
    "one_term": (9000, [7], 0.0),
    "one_term_skew": (60000, [900], 0.6),
    "few_levels": (8000, [6, 3], 0.0),
    "few_levels_large": (30000, [40, 25], 0.0),
    "skew": (60000, [700, 40], 0.5),
    "slices": (20000, [20, 300, 2], 0.0),
    "slices_skew": (60000, [1500, 400], 0.4),
}


@pytest.mark.parametrize("weighted,r", [(False, 1), (False, 12), (True, 17), (True, 33)])
@pytest.mark.parametrize("name", list(CASES))
def test_heavy_tiles(name, weighted, r):
    n, levels, share = CASES[name]
    codes, g = draw(n, levels, share, len(name) + r)
    rng = np.random.default_rng(r)
    w = rng.uniform(0.3, 2.0, n) if weighted else None
    gpu, orc = fb.Absorber(codes, g, w), oracle.Absorber(codes, g, w)
    assert gpu.fe1 == orc.fe1
    z = rng.standard_normal((n, r))
    for a, b in zip(gpu.rhs(z), orc.rhs(z)):
        assert rel(a, b) <= 1e-12
    z1, z2 = z.copy(), z.copy()
    i1 = gpu.residualize(z1, tol=1e-12, maxiter=100000, want_coefs=True)
    orc.residualize(z2, tol=1e-12, maxiter=100000)
    assert rel(z1, z2) <= 1e-9
    assert rel(z[:, 0] - gpu.fit_rows(i1["coefs"], 0), z1[:, 0]) <= 1e-9


def test_no_term():
    """No absorbed term: one segment of one cell holds every row."""
    n = 4000
    rng = np.random.default_rng(1)
    rows = rng.standard_normal((n, 4))
    out = fb.Session([], [], n=n).ols(rows)
    X = np.column_stack([rows[:, 1:], np.ones(n)])
    b = np.linalg.lstsq(X, rows[:, 0], rcond=None)[0]
    assert rel(out["b"], b) <= 1e-12


def best_ms(a, z, r):
    best = np.inf
    for _ in range(6):
        t = time.perf_counter()
        a.residualize_device(z.data_ptr(), r)
        best = min(best, time.perf_counter() - t)
    return best * 1e3


def test_few_levels_keep_the_chip_busy():
    """1e6 rows in 1000 levels take the chip's warps as the same rows in 25,000 do: within eight times
    the time (a warp per 128 levels takes sixteen times)."""
    import torch

    n, r = 10**6, 4
    z = torch.zeros(n, r, dtype=torch.float64, device="cuda")
    t = {}
    for g in (1000, 25000):
        a = fb.Absorber([(np.arange(n) % g).astype(np.uint32)], [g])
        t[g] = best_ms(a, z, r)
    assert t[1000] <= 8 * t[25000], t
