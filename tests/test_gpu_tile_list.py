"""Upper-triangle storage as pair lists: what a build uses where the padded groups do not fit."""
import numpy as np
import pytest

from oracle import oracle as O
from risq_b200 import GpuHam, _capi
from tests import helpers as H
from tests.test_gpu_memory import full_space

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb,nel,n", [(10, 4, 1), (10, 4, 2), (10, 4, 257), (10, 4, 1100), (10, 4, 2049), (10, 4, 6943),
                                        (12, 6, 30925)])
def test_lists_match_oracle(norb, nel, n, monkeypatch):
    import torch

    ints, _, dets, _, diag, _ = H.synthetic_hci(norb, nel, 1e-3)
    dets, diag = dets[:n], diag[:n]
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
    # fixed point: a product is rounded to 2^-51 (FP64) or 2^-31 (FP32) of twice the largest row
    # or column sum of a tile
    unit = 2 * sums.max(initial=0.0) * np.abs(x).max()
    order = np.lexsort((dets[:, 2], dets[:, 0]))
    xd = torch.tensor(x[order], dtype=torch.float32, device="cuda")
    monkeypatch.setenv("RISQGPU_TEST_TILE_OOM", "1")
    with GpuHam(ints) as g:
        g.set_dets(dets, 0, diag)
        for prec in (_capi.FP64_UPPER, _capi.MIXED_UPPER, _capi.FP32_UPPER):
            st = g.build(prec, _capi.BUILDER_FAST)
            assert st["nnz_upper"] == len(vals)
            assert st["bytes_csr"] == len(vals) * (8 if prec == _capi.FP32_UPPER else 12)
            if prec != _capi.FP32_UPPER:
                y = g.matrix_vector_prod(x)
                assert np.all(np.abs(y - ref) <= (terms * 2.0 ** -52 + 2.0 ** -46) * mag + terms * 2.0 ** -51 * unit)
                assert np.array_equal(y, g.matrix_vector_prod(x))
            if prec != _capi.FP64_UPPER:
                for reproducible in (False, True):
                    g.set_reproducible(reproducible)
                    yd = torch.full_like(xd, float("nan"))
                    torch.cuda.synchronize()
                    g.sigma_device(xd.data_ptr(), yd.data_ptr(), 1)
                    assert np.all(np.abs(yd.double().cpu().numpy() - ref[order]) <= (
                        (terms + 4) * 2.0 ** -24 * mag + terms * 2.0 ** -31 * unit)[order])
                g.set_reproducible(False)
            orp, ocols, ovals, _ = g.export_upper()
            assert np.array_equal(orp, rp) and np.array_equal(ocols, cols)
            np.testing.assert_allclose(ovals, vals, rtol=2.0 ** -24 if prec == _capi.FP32_UPPER else 2.0 ** -47, atol=0)
        er, ec, ev = g.export_rows(np.array([n // 2]))
        want = np.concatenate([cols[rows == n // 2], rows[cols == n // 2]])
        assert np.array_equal(np.sort(ec), np.sort(want))


def test_lists_solve_like_groups(monkeypatch):
    ints, _, dets, coeffs, diag, _ = H.synthetic_hci(10, 4, 1e-3)
    with GpuHam(ints) as g:
        g.set_dets(dets, 0, diag)
        g.build(_capi.FP64_UPPER)
        want = g.davidson(1, coeffs, 1e-4, 1e-8, 500)
        monkeypatch.setenv("RISQGPU_TEST_TILE_OOM", "1")
        g.build(_capi.FP64_UPPER)
        got = g.davidson(1, coeffs, 1e-4, 1e-8, 500)
        assert got.converged and abs(got.eigenvalues[0] - want.eigenvalues[0]) < 1e-9
        g.build(_capi.MIXED_UPPER)
        got = g.davidson(1, coeffs, 1e-4, 1e-8, 500, mode=_capi.MODE_MIXED)
        assert got.converged and abs(got.eigenvalues[0] - want.eigenvalues[0]) < 1e-6


@pytest.mark.parametrize("prec,value", [(_capi.FP64_UPPER, 8), (_capi.MIXED_UPPER, 8), (_capi.FP32_UPPER, 4)])
def test_a_bound_of_plain_lists_is_enough(prec, value):
    """A bound on the handle's memory that holds the pairs with 4 bytes of code each, 32 bytes a
    row, a thirty-second of that and the CSR rows of one panel: accepted, however short the
    rows of a tile are."""
    dets = full_space(12, 6)[:250007]
    with GpuHam(H.synthetic_hci(12, 6, 1e-3)[0]) as g:
        g.set_dets(dets)
        used, _ = g.memory_used()
        nnz = g.build(prec)["nnz_upper"]
        x = np.random.default_rng(0).standard_normal(len(dets))
        y = g.matrix_vector_prod(x) if prec != _capi.FP32_UPPER else None
        free, _ = g.memory_used()
    need = (4 + value) * nnz + 32 * len(dets)
    panel = 1024 * 2 * nnz // len(dets) * 2  # twice the mean: upper rows are longer at the top
    limit = used + 12 * len(dets) + need + max(8 << 20, need // 32) + (4 + value) * panel + (2 << 20)
    with GpuHam(H.synthetic_hci(12, 6, 1e-3)[0]) as g:
        g.set_dets(dets)
        g.set_memory_limit(limit)
        assert g.build(prec)["nnz_upper"] == nnz
        g.set_memory_limit(0)
        if y is not None:
            assert np.max(np.abs(g.matrix_vector_prod(x) - y)) <= 1e-11 * np.max(np.abs(y))
