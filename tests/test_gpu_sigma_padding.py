"""Tiled sigma where the last column window holds fewer columns than a warp has lanes.

Short row slots are padded with zero elements; in a window of fewer than 32 columns some of
them lie beyond it, and must not read what another kernel left in shared memory.
"""
import itertools

import numpy as np
import pytest

from oracle import oracle as O
from risq_b200 import GpuHam, _capi
from risq_b200.fcidump import synthetic_integrals
from tests import helpers as H

pytestmark = pytest.mark.gpu


def narrow_last_window(w):
    """2048 + w determinants of 12 orbitals, 6 electrons a spin: the last w in (up, dn) order
    share the highest up string, and most of the others are connected to them."""
    top = 0b111111000000

    def excited(s, k):
        occ = [o for o in range(12) if s >> o & 1]
        vir = [o for o in range(12) if not s >> o & 1]
        return [s - sum(1 << i for i in a) + sum(1 << j for j in b)
                for a in itertools.combinations(occ, k) for b in itertools.combinations(vir, k)]

    s1, s2 = excited(top, 1), excited(top, 2)
    last = [(top, d) for d in ([top] + s1 + s2)[:w]]
    rest = [(u, top) for u in s1 + s2] + [(u, d) for u in s1 for d in s1] + [(u, d) for u in s2 for d in s1]
    dets = np.zeros((2048 + w, 4), dtype=np.uint64)
    dets[:, 0], dets[:, 2] = zip(*(rest[:2048] + last))
    return dets


@pytest.mark.parametrize("w", [1, 2, 8, 30, 31])
def test_narrow_last_window_matches_oracle(w):
    import torch

    norb = 12
    ints = synthetic_integrals(norb, 1)
    dets = narrow_last_window(w)
    n = len(dets)
    with GpuHam(ints) as g:
        diag = g.ham_diag(dets)
    sp = O.Sparse().build(H.oracle_ham(ints), dets, diag, 0, builder=_capi.BUILDER_FAST)
    rp, cols, vals, _ = sp.export()
    order = np.lexsort((dets[:, 2], dets[:, 0]))  # internal order: by (up, dn)
    rank = np.argsort(order)
    rows = np.repeat(np.arange(n), np.diff(rp))
    lo, hi = np.minimum(rank[rows], rank[cols]), np.maximum(rank[rows], rank[cols])
    assert np.bincount(lo[hi >= 2048] >> 10, minlength=2)[:2].max() >= 64  # a dense FP64 tile
    assert np.bincount(lo[hi >= 2048] >> 8, minlength=8).max() >= 64  # a dense FP32 one
    x = np.random.default_rng(w).standard_normal(n)
    ref = sp.mv(x)
    scale = np.abs(ref).max()
    xd = torch.tensor(x[order], dtype=torch.float32, device="cuda")
    with GpuHam(ints) as g:
        g.set_dets(dets, 0, diag)

        def dirty():
            # kernels that leave NaN bit patterns in shared memory
            g.find_new_dets(x, 1e-3, True)
            for dt in (torch.float64, torch.float32):
                m = torch.full((2048, 2048), float("nan"), dtype=dt, device="cuda")
                m @ m
            torch.cuda.synchronize()

        for prec in (_capi.FP64_UPPER, _capi.MIXED_UPPER, _capi.FP32_UPPER):
            st = g.build(prec, _capi.BUILDER_FAST)
            assert st["nnz_upper"] == len(vals)
            if prec != _capi.FP32_UPPER:
                dirty()
                assert np.abs(g.matrix_vector_prod(x) - ref).max() <= 1e-11 * scale
            if prec != _capi.FP64_UPPER:
                for reproducible in (False, True):
                    g.set_reproducible(reproducible)
                    yd = torch.empty_like(xd)
                    dirty()
                    g.sigma_device(xd.data_ptr(), yd.data_ptr(), 1)
                    assert np.abs(yd.double().cpu().numpy() - ref[order]).max() <= 1e-5 * scale
                g.set_reproducible(False)
