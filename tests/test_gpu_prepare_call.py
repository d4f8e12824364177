"""The sample preparation in one call (fereg_prepare) against its steps' own calls, bit for bit: sparse
and dense ids, interactions, terms that share a factor, GLM separation, no drops, the smallest samples;
and the refusals."""

import numpy as np
import pytest

import fereg_b200 as fb

pytestmark = pytest.mark.gpu


def same(a, b):
    assert np.array_equal(a["alive"], b["alive"]) and a["alive"].dtype == bool
    assert (a["num_singletons"], a["fe_separated"]) == (b["num_singletons"], b["fe_separated"])
    assert len(a["terms"]) == len(b["terms"])
    for (c, g), (d, h) in zip(a["terms"], b["terms"]):
        assert g == h and c.dtype == np.uint32 and np.array_equal(c, d)


@pytest.mark.parametrize("n", [1, 2, 31, 1000, 70_001])
@pytest.mark.parametrize("absorb", [[[0]], [[0], [1]], [[0], [1, 2]], [[2, 0], [1], [0, 1, 2]], [[-1], (0, 1)]])
@pytest.mark.parametrize("opts", [{}, dict(singletons=False), dict(family="poisson"), dict(family="logit", singletons=False),
                                  dict(fw=True)])
def test_prepare_is_its_steps(n, absorb, opts):
    rng = np.random.default_rng(n)
    factors = [np.sort(rng.integers(10**9, 10**10, n)).astype(float) // 30_000 * 1e5, rng.integers(0, 1 + n // 3, n) - 5.0,
               rng.choice([0.5, -0.0, 0.0, 2.25], n)]
    opts = dict(opts)
    if opts.get("family"):
        opts["y"] = (rng.random(n) < 0.4).astype(float)
    if opts.pop("fw", None):
        opts["fw"] = rng.integers(1, 3, n).astype(float)
    steps = dict(fw=None, y=None, family=None, singletons=True)
    steps.update(opts)
    same(fb.prepare(factors, absorb, **opts), fb._prepare_steps(factors, absorb, **steps))


def test_prepare_refusals():
    x = np.arange(10.0)
    with pytest.raises(fb.FeregError) as e:
        fb.prepare([np.where(x == 3, np.nan, x)], [[0]])
    assert e.value.rc == 198
    with pytest.raises(fb.FeregError) as e:
        fb.prepare([x], [[0]], family="poisson")
    assert e.value.rc == 198
    with pytest.raises(IndexError):
        fb.prepare([x], [[1]])
    assert fb.prepare([x], [])["terms"] == []


def test_cluster_code_out_of_range_is_refused():
    codes = [np.repeat(np.arange(50), 4).astype(np.uint32)]
    cl = (np.arange(200) % 7).astype(np.uint32)
    with pytest.raises(fb.FeregError) as e:
        fb.Session(codes, [50], [cl], [6])
    assert e.value.rc == 198
    fb.Session(codes, [50], [cl], [7]).close()
