"""The serving engine admits requests by an upper estimate of their device memory: what a request holds
at most (the memory pool's high-water mark, one request at a time) stays below it, for requests whose
lists, weights in list order and sums by cell are large against their blocks."""

import ctypes as C

import numpy as np
import pytest

import fereg_b200 as fb

pytestmark = pytest.mark.gpu

USED_MEM_HIGH = 8  # CU_MEMPOOL_ATTR_USED_MEM_HIGH
N = 1_000_000


class PoolMark:
    """The default memory pool's bytes in use: the most since the last reset."""

    def __init__(self):
        self.cu = C.CDLL("libcuda.so.1")
        dev, self.pool = C.c_int(), C.c_void_p()
        assert self.cu.cuDeviceGet(C.byref(dev), 0) == 0
        assert self.cu.cuDeviceGetDefaultMemPool(C.byref(self.pool), dev) == 0

    def most(self):
        v = C.c_uint64()
        assert self.cu.cuMemPoolGetAttribute(self.pool, USED_MEM_HIGH, C.byref(v)) == 0
        return v.value

    def reset(self):
        v = C.c_uint64(0)
        assert self.cu.cuMemPoolSetAttribute(self.pool, USED_MEM_HIGH, C.byref(v)) == 0
        return self.most()


CASES = {
    # name: (model, levels, regressors, weighted)
    "two_terms": ("ols", [100_000, 10], 3, False),
    "small_block_32": ("ols", [500_000, 32], 1, False),
    "five_terms_weighted": ("ols", [100_000, 20_000, 10_000, 300, 10], 1, True),
    "six_terms": ("ols", [100_000, 20_000, 10_000, 300, 200, 10], 1, False),
    "wide_on_repeated_cells": ("ols", [1_000, 400], 59, True),
    "poisson_five_terms": ("poisson", [25_000, 20_000, 10_000, 300, 50], 1, False),
}


@pytest.mark.parametrize("name", list(CASES))
def test_request_stays_below_its_estimate(name):
    model, levels, nx, weighted = CASES[name]
    rng = np.random.default_rng(7)
    codes = []
    for g in levels:
        c = rng.integers(0, g, N).astype(np.uint32)
        c[:g] = np.arange(g)
        codes.append(c)
    cols = list(rng.standard_normal((1 + nx, N)))
    if model == "poisson":
        cols[0] = rng.poisson(1.0, N).astype(float)
    w = rng.uniform(0.5, 2.0, N) if weighted else None
    srv = fb.Server(workers=1)  # starts the driver
    mark = PoolMark()
    base = mark.reset()
    out = srv.wait(srv.submit(model, codes, levels, cols, nx, w=w, weight_kind="aweight" if weighted else None))
    used = mark.most() - base
    srv.close()
    assert out["rc"] == 0, out["msg"]
    assert used <= out["bytes"]
