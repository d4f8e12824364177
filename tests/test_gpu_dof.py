"""The degrees-of-freedom pass (mobility groups of the FE pairs, terms nested in a cluster) against
the oracle's union-find and a numpy nesting check, at the row counts where the pass changes its
launches (one launch below 2^15 rows, two prefixes and the rest from there on) and around them.
Counts and labels are exact."""

import numpy as np
import pytest

import fereg_b200 as fb
from oracle import oracle

pytestmark = pytest.mark.gpu


def codes_of(n, shape, seed):
    rng = np.random.default_rng(seed)
    ind = np.arange(n) // 7
    year = np.arange(n) % 7
    if shape == "islands":  # firms split into groups of 16 that share no individual
        firm = (ind // 40) * 16 + rng.integers(0, 16, n)
    elif shape == "ring":
        firm = np.arange(n) % max(2, n // 31)
    else:
        firm = rng.integers(0, max(2, n // 50), n)
    if shape == "shuffled":
        p = rng.permutation(n)
        ind, year, firm = ind[p], year[p], firm[p]
    out = [np.unique(c, return_inverse=True)[1].astype(np.uint32) for c in (ind, year, firm)]
    return out, [int(c.max()) + 1 for c in out]


@pytest.mark.parametrize("n", [50, 2**15 - 1, 2**15, 2**15 + 1, 100_003])
@pytest.mark.parametrize("shape", ["islands", "ring", "shuffled"])
def test_dof_table(n, shape):
    codes, g = codes_of(n, shape, n)
    # clusters: pairs of individuals (nests ind), or single firms (nests firm alone)
    for cl in (codes[0] // 2, codes[2]):
        sess = fb.Session(codes, g, [cl], [int(cl.max()) + 1])
        rows = np.ascontiguousarray(np.random.default_rng(1).standard_normal((n, 2)))
        r = sess.ols(rows, vce="cluster", want_groupvar=True)
        nested = [len(np.unique(np.stack([c, cl]), axis=1).T) == m for c, m in zip(codes, g)]
        live = [q for q in range(3) if not nested[q]]
        want = [g[q] if nested[q] else 0 for q in range(3)]
        for q in live if any(nested) else live[1:]:
            want[q] = 1
        for i, a in enumerate(live):
            for b in live[i + 1:]:
                want[b] = max(want[b], oracle.mobility_groups(codes[a], g[a], codes[b], g[b]))
        assert [int(x) for x in r["dof_table"][:, 1]] == want
        assert [bool(x) for x in r["dof_table"][:, 4]] == nested
        _, gv = oracle.mobility_groups(codes[live[0]], g[live[0]], codes[live[1]], g[live[1]], want_groupvar=True)
        assert np.array_equal(r["groupvar"].astype(np.uint32), gv)
