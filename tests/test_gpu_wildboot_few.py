"""Wild bootstrap in tiles of one to three draws: the block has no padding columns. The draws' statistics
equal those of one wide tile, and a tile of one draw holds a block of one column."""

import ctypes as C

import numpy as np
import pytest

import fereg_b200 as fb

pytestmark = pytest.mark.gpu

N = 40_000


def session(weighted):
    rng = np.random.default_rng(11)
    ind = np.repeat(np.arange(N // 8), 8).astype(np.uint32)
    firm = rng.integers(0, 600, N).astype(np.uint32)
    firm[:600] = np.arange(600)
    cl = (firm % 90).astype(np.uint32)
    w = rng.uniform(0.5, 2.0, N) if weighted else None
    s = fb.Session([ind, firm], [N // 8, 600], [cl], [90], w=w, weight_kind="aweight" if weighted else None)
    return s, rng.standard_normal((N, 3))


@pytest.mark.parametrize("tile,weighted", [(2, False), (4, True), (5, False)])
def test_last_tiles_of_few_draws(tile, weighted):
    s, rows = session(weighted)
    kw = dict(reps=11, seed=3, tol=1e-12)  # the last tile holds the rest: 1 or 3 draws
    one, few = s.wildboot(rows, tile=11, **kw), s.wildboot(rows, tile=tile, **kw)
    assert one["point"] == few["point"]
    assert np.max(np.abs(one["t_boot"] - few["t_boot"])) <= 1e-9 * np.max(np.abs(one["t_boot"]))


def test_one_draw_holds_one_column():
    cu = C.CDLL("libcuda.so.1")
    s, rows = session(False)
    dev, pool = C.c_int(), C.c_void_p()
    assert cu.cuDeviceGet(C.byref(dev), 0) == 0 and cu.cuDeviceGetDefaultMemPool(C.byref(pool), dev) == 0

    def most(tile):
        v = C.c_uint64(0)
        assert cu.cuMemPoolSetAttribute(pool, 8, C.byref(v)) == 0  # CU_MEMPOOL_ATTR_USED_MEM_HIGH
        s.wildboot(rows, tile=tile, reps=4)
        assert cu.cuMemPoolGetAttribute(pool, 8, C.byref(v)) == 0
        return v.value

    most(4)  # the handle's own buffers
    assert most(4) - most(1) >= 3 * 8 * N
