"""Tiled upper-triangle sigma at the edges of its blocks, windows, groups and row slots.

Sizes: a single determinant, the edges of a 256-row block and of the smallest window, a
set of several panels with a ragged last one, and one whose rows exceed a 64-element slot
within a window.
"""
import numpy as np
import pytest

from oracle import oracle as O
from risq_b200 import GpuHam, _capi
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb,nel,n", [(10, 4, 1), (10, 4, 2), (10, 4, 33), (10, 4, 255), (10, 4, 256), (10, 4, 257),
                                        (10, 4, 1100), (10, 4, 6943), (12, 6, 30925)])
def test_tiled_sigma_matches_oracle(norb, nel, n):
    import torch

    ints, _, dets, _, diag, _ = H.synthetic_hci(norb, nel, 1e-3)
    dets, diag = dets[:n], diag[:n]
    # the fast rule: the legacy one (up to 100 determinants) takes spin-flip-closed sets only
    sp = O.Sparse().build(H.oracle_ham(ints), dets, diag, 0, builder=_capi.BUILDER_FAST)
    rp, cols, vals, _ = sp.export()
    x = np.random.default_rng(n).standard_normal(n)
    ref = sp.mv(x)
    rows = np.repeat(np.arange(n), np.diff(rp))
    mag, sums = np.abs(diag * x), np.zeros(n)
    np.add.at(mag, rows, np.abs(vals * x[cols]))
    np.add.at(mag, cols, np.abs(vals * x[rows]))
    np.add.at(sums, rows, np.abs(vals))
    np.add.at(sums, cols, np.abs(vals))
    terms = 2 + np.bincount(rows, minlength=n) + np.bincount(cols, minlength=n)
    # fixed point: a product is rounded to at least 2^-48 (FP64) or 2^-30 (FP32) of the
    # largest tile sum, which its panel's eight 256-row blocks bound by 8 row sums
    unit = 8 * sums.max(initial=0.0) * np.abs(x).max()
    order = np.lexsort((dets[:, 2], dets[:, 0]))  # internal order: by (up, dn)
    xd = torch.tensor(x[order], dtype=torch.float32, device="cuda")
    with GpuHam(ints) as g:
        g.set_dets(dets, 0, diag)
        for prec in (_capi.FP64_UPPER, _capi.MIXED_UPPER, _capi.FP32_UPPER):
            st = g.build(prec, _capi.BUILDER_FAST)
            assert st["nnz_upper"] == len(vals)
            if prec != _capi.FP32_UPPER:
                y = g.matrix_vector_prod(x)
                assert np.all(np.abs(y - ref) <= (terms * 2.0 ** -52 + 2.0 ** -46) * mag + terms * 2.0 ** -48 * unit)
                assert np.array_equal(y, g.matrix_vector_prod(x))
            if prec != _capi.FP64_UPPER:
                bound = (terms + 4) * 2.0 ** -24 * mag + terms * 2.0 ** -30 * unit
                for reproducible in (False, True):
                    g.set_reproducible(reproducible)
                    yd = torch.full_like(xd, float("nan"))
                    torch.cuda.synchronize()
                    g.sigma_device(xd.data_ptr(), yd.data_ptr(), 1)
                    assert np.all(np.abs(yd.double().cpu().numpy() - ref[order]) <= bound[order])
                g.set_reproducible(False)
        orp, ocols, ovals, _ = g.export_upper()
        assert np.array_equal(orp, rp) and np.array_equal(ocols, cols)
