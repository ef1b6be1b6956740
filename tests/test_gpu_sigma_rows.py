"""Row sigma (both triangles stored) at the edges of its 256-element chunks and of its grid.

Prefixes of an HCI list give rows of every length from 0 to over 300; sizes go from one
determinant (fewer rows than warps of a block) to several blocks with a ragged last one.
"""
import numpy as np
import pytest

from oracle import oracle as O
from risq_b200 import GpuHam, _capi
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 9, 33, 300, 1025, 6943])
def test_row_sigma_matches_oracle(n):
    import torch

    ints, _, dets, _, diag, _ = H.synthetic_hci(10, 4, 1e-3)
    dets, diag = dets[:n], diag[:n]
    # the fast rule: the legacy one (up to 100 determinants) takes spin-flip-closed sets only
    sp = O.Sparse().build(H.oracle_ham(ints), dets, diag, 0, builder=_capi.BUILDER_FAST)
    rp, cols, vals, _ = sp.export()
    x = np.random.default_rng(n).standard_normal(n)
    ref = sp.mv(x)
    # sum of |H_ij x_j| and the number of terms of every row, for the rounding bounds
    rows = np.repeat(np.arange(n), np.diff(rp))
    mag = np.abs(diag * x)
    np.add.at(mag, rows, np.abs(vals * x[cols]))
    np.add.at(mag, cols, np.abs(vals * x[rows]))
    terms = 2 + np.bincount(rows, minlength=n) + np.bincount(cols, minlength=n)
    with GpuHam(ints) as g:
        g.set_dets(dets, 0, diag)
        for prec in (_capi.FP64, _capi.MIXED):
            g.build(prec, _capi.BUILDER_FAST)
            y = g.matrix_vector_prod(x)
            # both sides sum in FP64 in some order; MIXED values carry at least 2^-46
            assert np.all(np.abs(y - ref) <= (2 * terms * 2.0 ** -53 + 2.0 ** -46) * mag)
        order = np.lexsort((dets[:, 2], dets[:, 0]))  # internal order: by (up, dn)
        xd = torch.tensor(x[order], dtype=torch.float32, device="cuda")
        yd = torch.full_like(xd, float("nan"))
        torch.cuda.synchronize()
        g.sigma_device(xd.data_ptr(), yd.data_ptr(), 1)
        # FP32 values and vector (2^-24 each), products and sums of `terms` addends
        bound = (terms + 3) * 2.0 ** -24 * mag[order]
        assert np.all(np.abs(yd.double().cpu().numpy() - ref[order]) <= bound)
