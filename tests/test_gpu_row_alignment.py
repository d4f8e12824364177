"""Wide rows (a multiple of 4 columns) in device memory at every 8-byte offset from a 32-byte boundary:
the 256-bit row accesses take the aligned blocks only, the warp tiles the others, with the same values."""

import numpy as np
import pytest

import fereg_b200 as fb
from tests._gen import panel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [20, 132])
@pytest.mark.parametrize("weighted", [False, True])
def test_offsets(r, weighted):
    import torch

    codes, g, w, z = panel(n_ind=3000, years=7, n_firm=200, seed=r, weighted=weighted, r=r)
    ab = fb.Absorber(codes, g, w)
    rows = np.ascontiguousarray(z[ab.row_order()])
    n = len(rows)
    want = None
    for off in range(4):
        buf = torch.zeros(n * r + 8, dtype=torch.float64, device="cuda")
        view = buf[off : off + n * r]
        assert view.data_ptr() % 32 == 8 * off
        view.copy_(torch.from_numpy(rows).reshape(-1))
        torch.cuda.synchronize()
        info = ab.residualize_device(view.data_ptr(), r, want_coefs=True)
        torch.cuda.synchronize()
        got = (view.cpu().numpy(), info["coefs"])
        assert not buf[:off].any() and not buf[off + n * r :].any()  # nothing beside the block
        if want is None:
            want = got
        for a, b in zip(got, want):  # the same solve; sums of 7 values of unit scale in another order
            assert np.max(np.abs(a - b)) <= 1e-12 * max(1.0, np.max(np.abs(b)))
