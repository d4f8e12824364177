"""Escalation on graphs of many components: a ring of firms, whose slow contraction brings the multigrid
preconditioner, beside islands of a few firms, each of which ends as one coarse node whose diagonal is
round-off. The converged answer must not change: residualized columns match the oracle's (Jacobi or the exact small block, run to a tighter
tolerance) to 1e-8 in the W-norm, on the first solve, which escalates, and on a later one."""

import numpy as np
import pytest

import fereg_b200 as fb
from oracle import oracle

pytestmark = pytest.mark.gpu


def dense(c):
    return np.unique(c, return_inverse=True)[1].astype(np.uint32)


def ring_and_islands(firms_per_island):
    """6000 individuals on a ring of 1499 firms; 1500 islands of 3 individuals with 4 rows each."""
    n1 = 60000
    i = np.arange(n1)
    ind, firm, year = i // 10, i % 1499, i % 10
    rng = np.random.default_rng(firms_per_island)
    j = np.arange(1500 * 12)
    isl = j // 12
    ind = np.concatenate([ind, 6000 + isl * 3 + (j % 12) // 4])
    firm = np.concatenate([firm, 1499 + isl * firms_per_island + rng.integers(0, firms_per_island, len(j))])
    year = np.concatenate([year, rng.integers(0, 10, len(j))])
    return [dense(ind), dense(firm), dense(year)]


@pytest.mark.parametrize("prec", [fb.PREC_F64, fb.PREC_F32_REFINED])
@pytest.mark.parametrize("weights", [None, "uniform", "lognormal"])
@pytest.mark.parametrize("graph", ["islands2", "islands5"])
def test_islands(graph, weights, prec):
    codes = ring_and_islands(int(graph[-1]))
    g = [int(c.max()) + 1 for c in codes]
    n = len(codes[0])
    rng = np.random.default_rng(5)
    w = {None: None, "uniform": rng.uniform(0.5, 2.0, n), "lognormal": np.exp(2 * rng.standard_normal(n))}[weights]
    z = rng.standard_normal((n, 2))
    gpu, orc = fb.Absorber(codes, g, w), oracle.Absorber(codes, g, w)
    order = gpu.row_order()
    z = np.ascontiguousarray(z[order])
    wr = np.ones(n) if w is None else w[order]
    want = z.copy()
    orc.residualize(want, tol=1e-12, maxiter=200000)
    scale = np.sqrt(np.sum(wr[:, None] * want**2, axis=0))
    for _ in range(3):
        got = z.copy()
        info = gpu.residualize(got, tol=1e-10, maxiter=100000, precision=prec)
        assert info["escalated"]
        assert np.max(np.sqrt(np.sum(wr[:, None] * (got - want) ** 2, axis=0)) / scale) <= 1e-8
