"""Clusters of a session: grouped on the host up to 4,096 rows and on the device beyond, with the same
covariance on both sides of the line (one to three dimensions against the oracle), out-of-range codes
refused on both, and no kernel spent on the grouping of a small sample."""

import numpy as np
import pytest

import fereg_b200 as fb
from oracle import oracle

pytestmark = pytest.mark.gpu


def sample(n, dims, seed):
    rng = np.random.default_rng(seed)
    g = [max(2, n // 20), 10]
    codes = []
    for levels in g:
        c = rng.integers(0, levels, n).astype(np.uint32)
        c[:levels] = np.arange(levels)
        codes.append(c)
    cl_g = [12, 9, 7][:dims]
    cl = [rng.integers(0, k, n).astype(np.uint32) for k in cl_g]
    return codes, g, cl, cl_g, rng


@pytest.mark.parametrize("dims", [1, 2, 3])
@pytest.mark.parametrize("n", [60, 4095, 4096, 4097, 9000])
def test_cluster_covariance(n, dims):
    codes, g, cl, cl_g, rng = sample(n, dims, n + dims)
    gpu, orc = fb.Session(codes, g, cl, cl_g), oracle.Session(codes, g, cl, cl_g)
    rows = rng.standard_normal((n, 3))
    a, b = gpu.ols(rows, vce="cluster", tol=1e-12), orc.ols(rows, vce="cluster", tol=1e-12)
    assert np.max(np.abs(a["b"] - b["b"])) <= 1e-9 * max(1.0, np.max(np.abs(b["b"])))
    assert np.max(np.abs(a["V"] - b["V"])) <= 1e-9 * max(1e-3, np.max(np.abs(b["V"])))


@pytest.mark.parametrize("n", [4096, 4097])
@pytest.mark.parametrize("dims", [1, 2])
def test_out_of_range_codes_are_refused(n, dims):
    codes, g, cl, cl_g, _ = sample(n, dims, 3)
    cl[-1][n // 2] = cl_g[-1]
    with pytest.raises(fb.FeregError) as e:
        fb.Session(codes, g, cl, cl_g)
    assert e.value.rc == 198


def test_small_samples_spend_no_kernels_on_the_grouping():
    from torch.profiler import ProfilerActivity, profile

    def kernels(dims):
        codes, g, cl, cl_g, _ = sample(300, dims, 5)
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            fb.Session(codes, g, cl, cl_g).close()
        names = [e.name for e in prof.events()]
        return sum("Memcpy" not in x and "Memset" not in x and "cuda" not in x for x in names)

    kernels(0)
    none = kernels(0)
    if none == 0:
        pytest.skip("no kernel trace on this machine")
    assert kernels(3) == none
