"""The mobility-group labels of repeated calls against the oracle's, on sparse graphs whose union-find
trees are deep when the labels are read (long chains, many components): exact every time."""

import numpy as np
import pytest

import fereg_b200 as fb
from oracle import oracle

pytestmark = pytest.mark.gpu


def graph(shape, seed):
    rng = np.random.default_rng(seed)
    if shape == "sparse":  # 0.6 rows a level: many components of all sizes
        n, ga, gb = 5000, 4000, 4000
        a, b = rng.integers(0, ga, n), rng.integers(0, gb, n)
    elif shape == "chains":  # paths of 50 levels, rows shuffled
        n = 20000
        p = rng.permutation(n)
        a, b = ((p + 1) // 2), (p // 2) + (p // 100)
    else:  # nearly one component
        n = 8600
        a, b = rng.integers(0, 1000, n), rng.integers(0, 3000, n)
    return [np.unique(c, return_inverse=True)[1].astype(np.uint32) for c in (a, b)]


@pytest.mark.parametrize("shape", ["sparse", "chains", "dense"])
def test_labels(shape):
    for seed in range(12):
        codes = graph(shape, seed)
        g = [int(c.max()) + 1 for c in codes]
        _, want = oracle.mobility_groups(codes[0], g[0], codes[1], g[1], want_groupvar=True)
        sess = fb.Session(codes, g)
        rows = np.ascontiguousarray(np.random.default_rng(1).standard_normal((len(codes[0]), 2)))
        for _ in range(6):
            got = sess.ols(rows, firstpair=True, want_groupvar=True, tol=1e-4)["groupvar"]
            assert np.array_equal(got.astype(np.uint32), want)
        sess.close()
