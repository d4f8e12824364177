"""The dense small block's assembly and grounded inverse against the oracle's preconditioner, at the
sizes where the kernels change: tiles of 16 and 64 coordinates, the list assembly where the tiles
would be more work, the one-CTA factor (2, 4, 7 and 10 blocks of 16, up to 160 coordinates) and the
panels beyond, the inverse's register widths (32, 128, 512, 1024). The tolerance is the parity
tests' for the preconditioner (1e-10)."""

import numpy as np
import pytest

import fereg_b200 as fb
from oracle import oracle

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.max(np.abs(a - b))) / max(1.0, float(np.max(np.abs(b))))


@pytest.mark.parametrize("ms", [11, 16, 17, 32, 33, 64, 65, 112, 113, 128, 129, 160, 161, 320, 512, 513, 1000])
@pytest.mark.parametrize("weighted", [False, True])
def test_small_block(ms, weighted):
    rng = np.random.default_rng(ms)
    n_ind, years = 1500, 6
    n = n_ind * years
    ind = np.repeat(np.arange(n_ind), years)
    year = np.tile(np.arange(years), n_ind)
    firm = np.concatenate([np.arange(ms - years), rng.integers(0, ms - years, n - (ms - years))])
    codes = [c.astype(np.uint32) for c in (ind, year, firm)]
    g = [n_ind, years, ms - years]
    w = rng.uniform(0.3, 2.0, n) if weighted else None
    gpu, orc = fb.Absorber(codes, g, w), oracle.Absorber(codes, g, w)
    assert gpu.m_small == ms == gpu.m
    p = rng.standard_normal((gpu.m, 3))
    p = orc.apply(p)  # in the range of the system, where any generalized inverse agrees
    assert rel(orc.apply(gpu.precond(p)), orc.apply(orc.precond(p))) <= 1e-10


@pytest.mark.parametrize("cells", [1, 31, 33, 70])
def test_small_block_one_block(cells):
    """One small block (no cross sums), segments of one to several warps of cells."""
    rng = np.random.default_rng(cells)
    n_ind, F = 900, 40
    ind = np.repeat(np.arange(n_ind), cells)
    firm = rng.integers(0, F, len(ind))
    firm[:F] = np.arange(F)
    codes, g = [ind.astype(np.uint32), firm.astype(np.uint32)], [n_ind, F]
    gpu, orc = fb.Absorber(codes, g), oracle.Absorber(codes, g)
    p = orc.apply(rng.standard_normal((gpu.m, 2)))
    assert rel(orc.apply(gpu.precond(p)), orc.apply(orc.precond(p))) <= 1e-10
