"""Tiled upper-triangle sigma at the edges of its blocks, windows, groups and row slots.

Sizes: a single determinant, the edges of a 256-row block and of the smallest window, a
set of several panels with a ragged last one, and one whose rows exceed a 64-element slot
within a window.
"""
import numpy as np
import pytest

from oracle import oracle as O
from risq_b200 import GpuHam, _capi
from risq_b200.fcidump import synthetic_integrals
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


@pytest.mark.parametrize("n_alpha,run", [(3001, 3), (4099, 3), (2200, 4)])
def test_wide_fp64_windows_of_sparse_sets(n_alpha, run):
    """Runs of `run` determinants of one alpha string, each connected to the others and hardly
    any to the rest: less than one pair per row and window, hence 4096-column windows."""
    norb, nel = 24, 8
    ints = synthetic_integrals(norb, 3)
    rng = np.random.default_rng(n_alpha)
    rows, seen = [], set()
    while len(seen) < n_alpha:
        up = sum(1 << int(o) for o in rng.choice(norb, nel, replace=False))
        if up in seen:
            continue
        seen.add(up)
        occ = rng.choice(norb, nel + run - 1, replace=False)
        base = sum(1 << int(o) for o in occ[:nel - 1])
        rows += [(up, 0, base | 1 << int(o), 0) for o in occ[nel - 1:]]
    dets = np.array(rows, dtype=np.uint64)[rng.permutation(len(rows))]
    x = rng.standard_normal(len(dets))
    with GpuHam(ints) as g:
        g.set_dets(dets)
        st = g.build(_capi.FP64_UPPER)
        assert st["n_tiles"] > 0 and st["nnz_dense"] > st["nnz_upper"] // 2
        assert st["nnz_upper"] < len(dets) * (((len(dets) + 2047) >> 11) // 2)
        rp, cols, vals, diag = g.export_upper()
        y = g.matrix_vector_prod(x)
        g.build(_capi.FP64_UPPER)
        np.testing.assert_array_equal(g.matrix_vector_prod(x), y)
    sp = O.Sparse().build(H.oracle_ham(ints), dets, diag, 0, builder=_capi.BUILDER_FAST)
    orp, ocols, ovals, _ = sp.export()
    np.testing.assert_array_equal(rp, orp)
    np.testing.assert_array_equal(cols, ocols)
    np.testing.assert_array_equal(vals, ovals)
    ref = sp.mv(x)
    assert np.max(np.abs(y - ref)) <= 1e-11 * np.max(np.abs(ref))
