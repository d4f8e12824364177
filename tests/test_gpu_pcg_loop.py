"""The device PCG loop: its vector kernels at the widths where they change (narrow up to 64 columns,
column tiles beyond and for weighted systems with a small block), and the ways a solve's iterations
are issued (a session's first solve by launches, later ones by replayed graphs of four iterations):
the same bits and the same iteration counts, and the iteration cap to the iteration."""

import numpy as np
import pytest

import fereg_b200 as fb
from oracle import oracle
from tests._gen import panel

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.max(np.abs(a - b))) / max(1.0, float(np.max(np.abs(b))))


@pytest.mark.parametrize("r", [1, 4, 13, 60, 64, 65, 130])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n_firm,extra", [(5000, ()), (4200, (40,))])
def test_widths_match_oracle(r, weighted, n_firm, extra):
    codes, g, w, _ = panel(n_ind=6000, years=7, n_firm=n_firm, seed=r, weighted=weighted, extra=extra)
    z = np.random.default_rng(r).standard_normal((len(codes[0]), r)) + 0.3 * (codes[0] % 7)[:, None]
    gpu, orc = fb.Absorber(codes, g, w), oracle.Absorber(codes, g, w)
    z1, z2, z3 = z.copy(), z.copy(), z.copy()
    i1 = gpu.residualize(z1, tol=1e-12, maxiter=100000)
    i3 = gpu.residualize(z3, tol=1e-12, maxiter=100000)
    orc.residualize(z2, tol=1e-12, maxiter=100000)
    assert rel(z1, z2) <= 1e-9  # the parity tests' bound
    assert np.array_equal(z1, z3) and i1["iterations"] == i3["iterations"]


@pytest.mark.parametrize("r,weighted", [(2, False), (5, True), (70, False)])
def test_iteration_cap(r, weighted):
    codes, g, w, _ = panel(n_ind=6000, years=7, n_firm=5000, seed=3, weighted=weighted)
    z = np.random.default_rng(1).standard_normal((len(codes[0]), r))
    gpu = fb.Absorber(codes, g, w)
    its = gpu.residualize(z.copy(), tol=1e-8)["iterations"]
    assert its > 5
    first = z.copy()
    gpu.residualize(first, tol=1e-8, maxiter=its)
    for cap in (its, its + 1):  # graphs by now
        again = z.copy()
        assert gpu.residualize(again, tol=1e-8, maxiter=cap)["iterations"] == its
        assert np.array_equal(first, again)
    for cap in (1, 2, 3, 4, 5, its - 1):
        for h in (gpu, fb.Absorber(codes, g, w)):  # by graphs, and by launches
            with pytest.raises(fb.FeregError) as e:
                h.residualize(z.copy(), tol=1e-8, maxiter=cap)
            assert e.value.rc == 430
